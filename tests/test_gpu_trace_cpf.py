"""The gathered f as a trace buffer: the last step's, also where that step's gather emitted from registers, and
never an older step's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,dims", [("D2Q9", (400, 390)), ("D3Q19", (56, 48, 48))])
@pytest.mark.parametrize("graphs", [True, False])
def test_gathered_f_is_never_stale(lattice, dims, graphs):
    from direbm_gb300._lib import DbmError
    from direbm_gb300.lattices import get
    from direbm_gb300.sim import Instance, Simulation
    from oracle.physics import equilibrium

    rng = np.random.default_rng(2)
    c = np.stack(np.meshgrid(*[np.arange(n) for n in dims], indexing="ij"), -1).reshape(-1, len(dims)).astype(float)
    x = c + rng.uniform(0.2, 0.8, c.shape)
    f = equilibrium(np.ones(len(x)), 0.02 * np.sin(x), get(lattice))

    def sim(dense=True):
        s = Simulation([Instance(dims=dims, tau=0.7)], lattice=lattice, precision="fp32dev", dx=1.0, r_res=1.5,
                       cell=1.0, graphs=graphs, moment_capacity=len(x))
        s.set_dense_stencil(dense)
        s.set_state(None, x, f)
        return s

    def gathered(s):
        p = s.count()
        return s.trace("cpf").cpu().numpy().view(np.float32).reshape(2, get(lattice).Q, s.capacity)[:, :, :p]

    a, b = sim(), sim(dense=False)
    for n in (1, 1, 2):  # the later ones from recorded graphs
        a.step(n)
        b.step(n)
        np.testing.assert_array_equal(gathered(a), gathered(b))
        np.testing.assert_array_equal(gathered(a), gathered(b))
        empty = [s.trace("empty").cpu().numpy().view(np.uint32)[: s.count()] for s in (a, b)]
        np.testing.assert_array_equal(*empty)
    a.set_state(None, x, f)  # without a step, there is no gathered f of this state
    a.step(1)
    a.set_state(None, x, f)
    with pytest.raises(DbmError):
        a.trace("cpf")
    a.step(1)
    b.set_state(None, x, f)
    b.step(1)
    for i, (u, v) in enumerate(zip(a.state_numpy(), b.state_numpy())):
        np.testing.assert_array_equal(u, v)
    np.testing.assert_array_equal(gathered(a), gathered(b))
    for s in (a, b):
        s.step(1)  # goes on from the state that the reading left alone
    for u, v in zip(a.state_numpy(), b.state_numpy()):
        np.testing.assert_array_equal(u, v)
    for s in (a, b):
        s.step_partial(6)
    np.testing.assert_array_equal(gathered(a), gathered(b))
