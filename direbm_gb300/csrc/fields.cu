// Macroscopic fields on the device: bin moments' mass and momentum onto a regular 2D or 3D grid.
//
// Replaces direbm/fields.py:17-41 (bin_fields, numpy histogram2d with mass and momentum weights)
// without leaving the device, and extends it to 3D (histogramdd's rule on three edge arrays; the
// reference bins in 2D only).  A moment's bin follows numpy's rule for the edge array
// (searchsorted(edges, x, "right") - 1, the last edge belonging to the last bin, values outside
// dropped).  One pass over the moments writes their bin and their mass and momentum; the bins are
// stable-sorted, and each bin's sum runs over its moments in input order -- the order the histogram
// accumulates in -- with no float atomics.
//
// The first pass is bound by FP64 additions (two lanes per clock and SM): 18 of them for D2Q9, where the
// plain sums with their products by 0 and +-1 took 45 and the search for a bin 9 comparisons per axis.
// 1.64 M moments, 320 x 320 bins: this pass 78 (bins alone) -> 84 us, the bins' sums 180 -> 32, the sort 93 -> 70
// (17 key bits in place of 32).
#include <algorithm>

#include "lattice.cuh"
#include "sortscan.cuh"

namespace dbm {

// Evenly spaced edges, as histograms have: a value's bin by proportion (FP32).
struct Guess {
  float e0, scale;
};
__device__ __forceinline__ Guess make_guess(const double* __restrict__ edges, int ne) {
  const float e0 = (float)edges[0];
  return {e0, (float)(ne - 1) / ((float)edges[ne - 1] - e0)};
}

__device__ __forceinline__ int bin_of(const double* __restrict__ edges, int ne, double x, const Guess& gs) {
  const int g = min(max((int)(((float)x - gs.e0) * gs.scale), 0), ne - 2);
  if (x >= edges[g] && x < edges[g + 1]) return g;
  // searchsorted(edges, x, side="right") - 1 with the closed last bin of numpy's histogram
  if (!(x >= edges[0]) || !(x <= edges[ne - 1])) return -1;
  if (x == edges[ne - 1]) return ne - 2;
  int lo = 0, hi = ne;  // first index with edges[i] > x
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (edges[mid] > x) hi = mid; else lo = mid + 1;
  }
  return lo - 1;
}

// Edge arrays of the D axes, and the D momentum outputs.
struct Edges {
  const double* e[3];
  int n[3];
};
struct MomOut {
  double* p[3];
};

// A moment's mass and momentum: 32 bytes, one sector.
struct __align__(16) MassMom {
  double v[4];
};

// Component a of c_k: 0, 1 or -1, or 2 for any other value.
template <int Q>
__host__ __device__ constexpr int unit_c(int k, int a) {
  if constexpr (Q == 7) {
    constexpr int c[7][2] = {{0, 0}, {1, 0}, {2, 2}, {2, 2}, {-1, 0}, {2, 2}, {2, 2}};
    return c[k][a];
  } else if constexpr (Q == 9) {
    constexpr int c[9][2] = {{0, 0}, {1, 0}, {0, 1}, {-1, 0}, {0, -1}, {1, 1}, {-1, 1}, {-1, -1}, {1, -1}};
    return c[k][a];
  } else if constexpr (Q == 13) {
    return k == 0 || a == (k < 5 ? 0 : k < 9 ? 2 : 1) ? 0 : 2;
  } else {
    constexpr int c[19][3] = {{0, 0, 0}, {1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1},
                              {1, 1, 0}, {-1, -1, 0}, {1, -1, 0}, {-1, 1, 0}, {1, 0, 1}, {-1, 0, -1},
                              {1, 0, -1}, {-1, 0, 1}, {0, 1, 1}, {0, -1, -1}, {0, 1, -1}, {0, -1, 1}};
    return c[k][a];
  }
}
template <int Q, int D>
bool unit_c_holds(const LatHost& h) {
  for (int k = 0; k < Q; ++k)
    for (int a = 0; a < D; ++a)
      if (unit_c<Q>(k, a) != 2 && h.c[k][a] != unit_c<Q>(k, a)) return false;
  return true;
}

// sum_k f_k and sum_k f_k c_k, term by term from k = 0, every product and sum rounded; terms with c = 0 and
// products with +-1 are left out, which changes nothing for finite f.  They are chosen at compile time: with
// branches on the velocities the compiler computes both sides.
template <int Q, int D>
__device__ __forceinline__ MassMom mass_mom(const double (&f)[Q], const LatK<Q, D>& L) {
  MassMom r{{0.0, 0.0, 0.0, 0.0}};
  r.v[0] = f[0];
#pragma unroll
  for (int k = 1; k < Q; ++k) r.v[0] = __dadd_rn(r.v[0], f[k]);
#pragma unroll
  for (int a = 0; a < D; ++a) {
    bool any = false;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = unit_c<Q>(k, a);
      if (c == 0) continue;
      const double t = c == 1 ? f[k] : c == -1 ? -f[k] : __dmul_rn(f[k], L.c[k][a]);
      r.v[1 + a] = any ? __dadd_rn(r.v[1 + a], t) : t;
      any = true;
    }
  }
  if ((__double2hiint(r.v[0]) & 0x7ff00000) == 0x7ff00000) {  // not finite: the plain sums (0 x inf)
#pragma unroll
    for (int a = 0; a < D; ++a) {
      double p = 0.0;
#pragma unroll 1
      for (int k = 0; k < Q; ++k) {
        double fk = f[0];
#pragma unroll
        for (int q = 1; q < Q; ++q) fk = q == k ? f[q] : fk;
        p = __dadd_rn(p, __dmul_rn(fk, L.c[k][a]));
      }
      r.v[1 + a] = p;
    }
  }
  return r;
}

template <int Q, int D>
__global__ void __launch_bounds__(256) k_bin_moments(const double* __restrict__ x, const double* __restrict__ f,
                                                     int64_t n, Edges E, uint32_t nbins,
                                                     const __grid_constant__ LatK<Q, D> L,
                                                     uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                     MassMom* __restrict__ mm) {
  __shared__ Guess gs[D];  // conversions to FP32 run on the FP64 units
  if (threadIdx.x < D) gs[threadIdx.x] = make_guess(E.e[threadIdx.x], E.n[threadIdx.x]);
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    // bins are indexed [iz][iy][ix] (image convention of the reference); dropped moments sort last
    uint32_t key = 0;
    bool out = false;
#pragma unroll
    for (int a = D - 1; a >= 0; --a) {
      const int b = bin_of(E.e[a], E.n[a], x[(int64_t)D * i + a], gs[a]);
      out |= b < 0;
      key = key * (uint32_t)(E.n[a] - 1) + (uint32_t)(b < 0 ? 0 : b);
    }
    keys[i] = out ? nbins : key;
    vals[i] = (uint32_t)i;
    if (out) continue;
    double fi[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) fi[k] = f[(int64_t)i * Q + k];
    mm[i] = mass_mom<Q, D>(fi, L);
  }
}

// One thread per bin: binary-search its range in the sorted keys, then sum in sorted order, the moments of
// four items in flight.
template <int D>
__global__ void __launch_bounds__(128) k_bin_sums(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ order,
                                                  int64_t n, const MassMom* __restrict__ mm, int64_t nbins,
                                                  double* __restrict__ mass, MomOut mom) {
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nbins; b += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (keys[mid] < (uint32_t)b) lo = mid + 1; else hi = mid;
    }
    double s[1 + D];
#pragma unroll
    for (int a = 0; a <= D; ++a) s[a] = 0.0;
    for (int64_t j = lo;; j += 4) {
      MassMom it[4];
      bool in[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        in[u] = j + u < n && keys[j + u] == (uint32_t)b;
        if (in[u]) it[u] = mm[order[j + u]];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (in[u]) {
#pragma unroll
          for (int a = 0; a <= D; ++a) s[a] = __dadd_rn(s[a], it[u].v[a]);
        }
      }
      if (!in[3]) break;
    }
    mass[b] = s[0];
#pragma unroll
    for (int a = 0; a < D; ++a) mom.p[a][b] = s[1 + a];
  }
}

// Scratch: two pairs of (key, index) arrays, the moments' records, the sort's.
static char* aligned256(void* p) { return (char*)(((uintptr_t)p + 255) & ~(uintptr_t)255); }
static size_t round256(size_t b) { return (b + 255) / 256 * 256; }

// The binning of n moments in D dimensions.
static int bin_fields_impl(int D, const double* x, const double* f, int64_t n, int lattice, const Edges& E,
                           double* mass, MomOut mom, void* tmp, cudaStream_t s) {
  int64_t nbins = 1;
  for (int a = 0; a < D; ++a) nbins *= (int64_t)(E.n[a] - 1);
  if (nbins >= 0xffffffffLL) {
    set_last_error("bin_fields: too many bins (the bin key is 32-bit)");
    return DBM_ERR_INVALID;
  }
  if (n == 0) {
    DBM_CUDA(cudaMemsetAsync(mass, 0, (size_t)nbins * 8, s));
    for (int a = 0; a < D; ++a) DBM_CUDA(cudaMemsetAsync(mom.p[a], 0, (size_t)nbins * 8, s));
    return DBM_OK;
  }
  const size_t al = round256((size_t)n * 4);
  char* base = aligned256(tmp);
  uint32_t* keys = (uint32_t*)base;
  uint32_t* vals = (uint32_t*)(base + al);
  uint32_t* kalt = (uint32_t*)(base + 2 * al);
  uint32_t* valt = (uint32_t*)(base + 3 * al);
  MassMom* mm = (MassMom*)(base + 4 * al);
  void* rtmp = base + 4 * al + round256((size_t)n * sizeof(MassMom));
  const unsigned grid = std::min<unsigned>(div_up(n, 256), (unsigned)sm_count() * 16);
  const LatHost* lh = lat_host(lattice);
  const unsigned bgrid = (unsigned)std::min<int64_t>(div_up(nbins, 128), (int64_t)sm_count() * 64);
  int bits = 1;  // keys up to nbins (dropped)
  while (bits < 32 && (nbins >> bits)) ++bits;
  return dispatch_lattice(lattice, [&](auto tag) -> int {
    using LT = decltype(tag);
    if (!unit_c_holds<LT::Q, LT::D>(*lh)) { set_last_error("internal: bin_fields' velocities differ"); return DBM_ERR_STATE; }
    auto L = make_latk<LT::Q, LT::D>(*lh, 1.0, 1.0);
    k_bin_moments<LT::Q, LT::D><<<grid, 256, 0, s>>>(x, f, n, E, (uint32_t)nbins, L, keys, vals, mm);
    DBM_LAUNCH_CHECK();
    bool alt = false;
    DBM_TRY(radix_sort_pairs<uint32_t>(keys, vals, kalt, valt, n, nullptr, bits, rtmp, s, &alt));
    k_bin_sums<LT::D><<<bgrid, 128, 0, s>>>(alt ? kalt : keys, alt ? valt : vals, n, mm, nbins, mass, mom);
    DBM_LAUNCH_CHECK();
    return DBM_OK;
  });
}

}  // namespace dbm

using namespace dbm;

extern "C" int64_t dbm_bin_fields_tmp_bytes(int64_t n) {
  if (n < 0) return -1;
  const size_t m = (size_t)std::max<int64_t>(n, 1);
  return (int64_t)(256 + 4 * round256(m * 4) + round256(m * sizeof(MassMom)) + radix_tmp_bytes(n));
}

extern "C" int dbm_bin_fields_f64(const double* x, const double* f, int64_t n, int lattice, const double* ex, int nex,
                                  const double* ey, int ney, double* mass, double* momx, double* momy, void* tmp,
                                  void* stream) {
  const LatHost* lh = lat_host(lattice);
  if (!lh || lh->D != 2 || n < 0 || nex < 2 || ney < 2 || !ex || !ey || !mass || !momx || !momy ||
      (n > 0 && (!x || !f || !tmp)) || n >= 0xffffffffLL) {
    set_last_error("bin_fields: bad arguments");
    return DBM_ERR_INVALID;
  }
  const Edges E{{ex, ey, nullptr}, {nex, ney, 0}};
  return bin_fields_impl(2, x, f, n, lattice, E, mass, MomOut{{momx, momy, nullptr}}, tmp, (cudaStream_t)stream);
}

extern "C" int dbm_bin_fields3_f64(const double* x, const double* f, int64_t n, int lattice, const double* ex, int nex,
                                   const double* ey, int ney, const double* ez, int nez, double* mass, double* momx,
                                   double* momy, double* momz, void* tmp, void* stream) {
  const LatHost* lh = lat_host(lattice);
  if (!lh || lh->D != 3 || n < 0 || nex < 2 || ney < 2 || nez < 2 || !ex || !ey || !ez || !mass || !momx || !momy ||
      !momz || (n > 0 && (!x || !f || !tmp)) || n >= 0xffffffffLL) {
    set_last_error("bin_fields3: bad arguments");
    return DBM_ERR_INVALID;
  }
  const Edges E{{ex, ey, ez}, {nex, ney, nez}};
  return bin_fields_impl(3, x, f, n, lattice, E, mass, MomOut{{momx, momy, momz}}, tmp, (cudaStream_t)stream);
}
