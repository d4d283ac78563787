"""The gathered f as a trace buffer: right after a partial step, refused (not stale) after a step whose gather
emitted from registers."""

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

    a, b = sim(), sim(dense=False)
    for _ in range(2):  # the second from a recorded graph
        a.step(1)
        b.step(1)
        with pytest.raises(DbmError):
            a.trace("cpf")
    for s in (a, b):
        s.step_partial(6)
    p = a.count()
    read = [s.trace("cpf").cpu().numpy().view(np.float32).reshape(2, get(lattice).Q, s.capacity)[:, :, :p] for s in (a, b)]
    np.testing.assert_array_equal(*read)
    a.step(1)  # intermediates are kept from the first partial step on
    a.trace("cpf")
