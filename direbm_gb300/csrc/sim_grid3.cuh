// Grid variants of the three window kernels in 3D (FP32 store, 1 < R <= 1.5 cells).
//
// The untiled kernels give each (point, direction) a thread that walks the item ranges of its 16 window
// rows through L1: three dependent loads per hit, 17 of 32 lanes active, and every direction of a brick
// in a block of its own re-reading the region.  Here a block of 512 threads owns a brick of 8 x 8 x 8
// cells and stages the brick and its halo once as a grid: one 16-byte record per cell (offsets and item
// index, an empty cell with offsets outside every window).  It then takes the directions one after the
// other; the per-direction operands (exp(f*) for the refine, (1/sw, f*) for the gather) of the next
// direction are copied into the second of two buffers meanwhile.  A window is 4 x 4 x 4 cells from
// floor(p - cd - R - tiny) (a loop over the exact range for a point within `tiny` of a cell border), a
// row four unrolled candidates without a branch, a miss adding the weight 0; only operands that a hit
// alone needs are loaded by the lanes that hit (22 %).
//
// Sums in 3D take the items of each window cell in cell order.  Cells with further items are few (0.1 %
// to 0.6 % in the flow past a sphere), so a region row is marked when it holds one, and a warp in which
// some lane meets a marked row looks for them after each candidate of that row.  The sums of weights are
// exact, so the weights kernel visits them at the end.  Results are bit-identical to the untiled kernels.  Bricks within reach of an
// obstacle's bounced components are not taken (the host leaves them to the untiled kernels), and bricks
// with more further items than the list takes are deferred to them, as are the gather's bricks of an
// instance with a negative density or an f that is not finite.
// Bound by instruction issue (72 - 88 % of slots) and shared-memory wavefronts (71 - 87 %).  D3Q19, 96^3
// cells with one moment each, ms per launch, untiled / grid: thin + refine 2.97 / 1.13, weights 2.53 /
// 1.02, gather with emit 3.62 / 1.58; after 100 steps (0.4 % of the cells with two items) 2.99 / 1.55,
// 2.55 / 1.32, 3.63 / 2.10.  Flow past a sphere, 1.99 M points: step 25.0 / 10.6 ms.
#pragma once

#include "sim_grid.cuh"

namespace dbm {

constexpr int kBrick3 = 8;  // cells per side of a brick
constexpr int kThreads3 = kBrick3 * kBrick3 * kBrick3;
// Cells of halo on each side: 1 < R <= 1.5 and displacements that keep every window, and the four cells from
// its first one, inside (the host checks; up to R where that is 1.5, so one cell in use).
constexpr int kHalo3 = 3;
constexpr int kW3 = kBrick3 + 2 * kHalo3;
constexpr int kCells3 = kW3 * kW3 * kW3;
// Row and plane strides of the records: eight lanes of a row read one 128-byte line of 16-byte records,
// and rows 16 apart keep a column in its bank.
constexpr int kS3 = 16, kP3 = kW3 * kS3;
constexpr int kMore3 = 128;  // further items of a region, and of a brick's own cells, at most

// Shared memory: records, two planes of `elem` bytes per cell, item indices; the further items' records,
// planes, indices, keys and order; marked rows of each region plane; counters.  The item index of a
// cell with further items is -2 - (place of the first of them in the ordered list), and its first item
// is kept in mfirst there; -1: an empty cell.
struct Grid3Layout {
  int pl, gi, mrec, mpl, mgi, mfirst, key, ord, rows, cnt, total;
  __host__ __device__ constexpr Grid3Layout(int elem)
      : pl(kW3 * kP3 * 16), gi(pl + 2 * kCells3 * elem), mrec((gi + kCells3 * 4 + 15) & ~15), mpl(mrec + kMore3 * 16),
        mgi(mpl + 2 * kMore3 * elem), mfirst(mgi + kMore3 * 4), key(mfirst + kMore3 * 4), ord(key + kMore3 * 4), rows(ord + kMore3 * 2),
        cnt((rows + kW3 * 4 + 15) & ~15), total(cnt + 16) {}
};
constexpr Grid3Layout grid3_layout(int stage) { return Grid3Layout(stage == 0 ? 4 : stage == 2 ? 8 : 0); }

template <int STAGE>
struct Grid3Smem {
  static constexpr Grid3Layout L = grid3_layout(STAGE);
  unsigned char* p;
  __device__ __forceinline__ float4* rec() const { return reinterpret_cast<float4*>(p); }
  template <class T>
  __device__ __forceinline__ T* plane(int b) const { return reinterpret_cast<T*>(p + L.pl) + b * kCells3; }
  __device__ __forceinline__ int* gi() const { return reinterpret_cast<int*>(p + L.gi); }
  __device__ __forceinline__ float4* mrec() const { return reinterpret_cast<float4*>(p + L.mrec); }
  template <class T>
  __device__ __forceinline__ T* mplane(int b) const { return reinterpret_cast<T*>(p + L.mpl) + b * kMore3; }
  __device__ __forceinline__ int* mgi() const { return reinterpret_cast<int*>(p + L.mgi); }
  __device__ __forceinline__ int* mfirst() const { return reinterpret_cast<int*>(p + L.mfirst); }
  __device__ __forceinline__ int* key() const { return reinterpret_cast<int*>(p + L.key); }  // cell << 8 | place
  __device__ __forceinline__ short* ord() const { return reinterpret_cast<short*>(p + L.ord); }
  __device__ __forceinline__ int* rows() const { return reinterpret_cast<int*>(p + L.rows); }
  __device__ __forceinline__ int* cnt() const { return reinterpret_cast<int*>(p + L.cnt); }
};

__device__ __forceinline__ bool region_cell3(const InstK& I, int x, int y, int z, uint32_t* g) {
  const int nx = I.dims[0], ny = I.dims[1], nz = I.dims[2];
  if (I.periodic) {
    while (x < 0) x += nx;
    while (x >= nx) x -= nx;
    while (y < 0) y += ny;
    while (y >= ny) y -= ny;
    while (z < 0) z += nz;
    while (z >= nz) z -= nz;
  } else if (x < 0 || x >= nx || y < 0 || y >= ny || z < 0 || z >= nz) {
    return false;
  }
  *g = I.base + (uint32_t)x + (uint32_t)nx * ((uint32_t)y + (uint32_t)ny * (uint32_t)z);
  return true;
}

// Stages the records of a brick's region (their fourth word from `fourth(item)`, 0 in an empty cell) and
// orders its further items; false (in every thread) when the brick must be deferred.
template <class SM, class Fourth>
__device__ __forceinline__ bool stage_grid3(const InstK& I, const Brick& B, const uint32_t* __restrict__ start,
                                            const float* __restrict__ off, int64_t stride, const SM& S, int many,
                                            Fourth&& fourth) {
  for (int i = threadIdx.x; i < kW3; i += blockDim.x) S.rows()[i] = 0;
  __syncthreads();
  for (int ci = threadIdx.x; ci < kCells3; ci += blockDim.x) {
    const int row = ci / kW3, rx = ci - row * kW3, rz = row / kW3, ry = row - rz * kW3;
    uint32_t g;
    int b = 0, e = 0;
    if (region_cell3(I, B.x0 + rx - kHalo3, B.y0 + ry - kHalo3, B.z0 + rz - kHalo3, &g)) {
      b = (int)start[g];
      e = (int)start[g + 1];
    }
    auto record = [&](int m) {
      const float4 r = make_float4(off[m], off[stride + m], off[2 * stride + m], fourth(m));
      many |= (int)!(r.x + r.y + r.z < 4.f);  // NaN: 0 x it is not 0
      return r;
    };
    S.rec()[row * kS3 + rx] = e > b ? record(b) : make_float4(kEmptyOff, kEmptyOff, kEmptyOff, 0.f);
    S.gi()[ci] = e > b ? b : -1;
    for (int m = b + 1; m < e; ++m) {
      const int q = atomicAdd(S.cnt(), 1);
      if (q >= kMore3 || m - b > 255) {
        many = 1;
        break;
      }
      S.mrec()[q] = record(m);
      S.mgi()[q] = m;
      S.key()[q] = (ci << 8) | (m - b);
      atomicOr(S.rows() + rz, 1 << ry);
    }
  }
  if (__syncthreads_or(many)) return false;
  const int n = *S.cnt();
  if (n > 0) {
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      const int kq = S.key()[q];
      int rank = 0;
      for (int r = 0; r < n; ++r) rank += S.key()[r] < kq ? 1 : 0;
      S.ord()[rank] = (short)q;
      if ((kq & 255) == 1) {
        S.mfirst()[q] = S.gi()[kq >> 8];
        S.gi()[kq >> 8] = -2 - rank;
      }
    }
    __syncthreads();
  }
  return true;
}

// Further items of region cell ci, in order: fn(slot).
template <class SM, class Fn>
__device__ __forceinline__ void cell_more(const SM& S, int n, int ci, Fn&& fn) {
  const int v = S.gi()[ci];
  if (v > -2) return;
#pragma unroll 1
  for (int i = -2 - v; i < n; ++i) {
    const int q = S.ord()[i];
    if (S.key()[q] >> 8 != ci) break;
    fn(q);
  }
}

// Window of one direction: its first cell relative to the reference point's, and its extent.
struct Win3 {
  int lo[3], n[3];
  // bases b[a] = p[a] - cd[a] (or o[a] + cd[a])
  __device__ __forceinline__ void set(const float (&b)[3], float R, float tiny) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = (int)floorf(b[a] - R - tiny);
      n[a] = (int)floorf(b[a] + R + tiny) - lo[a] + 1;
    }
  }
  __device__ __forceinline__ bool fits() const { return n[0] <= 4 && n[1] <= 4 && n[2] <= 4; }
};

// Cuts a window five cells wide on some axis (p - cd within tiny of a cell border) to the first four
// where no candidate of the fifth slab is within R on that axis alone, which holds but for offsets
// within tiny of the border.  eof(axis, offset, cell offset): a candidate's displacement on one axis.
template <class SM, class Eof>
__device__ __forceinline__ void cut_window3(const SM& S, int nmore, const int (&c)[3], float R2, Win3& w, Eof&& eof) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (w.n[a] != 5) continue;
    const int a1 = a == 0 ? 1 : 0, a2 = a == 2 ? 1 : 2;
    const int j = w.lo[a] + 4;
    bool hit = false;
    int q[3];
    q[a] = c[a] + j;
#pragma unroll 1
    for (int u = 0; u < w.n[a2]; ++u)
#pragma unroll 1
      for (int v = 0; v < w.n[a1]; ++v) {
        q[a1] = c[a1] + w.lo[a1] + v;
        q[a2] = c[a2] + w.lo[a2] + u;
        const float4 r = S.rec()[q[2] * kP3 + q[1] * kS3 + q[0]];
        const float e = eof(a, a == 0 ? r.x : a == 1 ? r.y : r.z, j);
        hit |= rn_mul(e, e) <= R2;
      }
    for (int i = 0; i < nmore; ++i) {
      const float4 r = S.mrec()[i];
      const int ci = S.key()[i] >> 8, row = ci / kW3;
      const int at = a == 0 ? ci - row * kW3 : a == 1 ? row % kW3 : row / kW3;
      const float e = eof(a, a == 0 ? r.x : a == 1 ? r.y : r.z, j);
      hit |= at == q[a] && rn_mul(e, e) <= R2;
    }
    if (!hit) w.n[a] = 4;
  }
}

// Candidates of a window in order, for every lane of the warp with `on` (all lanes call):
// one(record, cell index or -1, further slot or -1, cx, cy, cz), the displacement constants from
// cof(axis, cell offset).  MORE: the further items of each cell follow its first.
template <bool MORE, class SM, class Cof, class One>
__device__ __forceinline__ void window3(const SM& S, int nmore, bool on, const int (&c)[3], const Win3& w, Cof&& cof,
                                        One&& one) {
  const bool fits = on && w.fits();
  const unsigned lanes = __ballot_sync(0xffffffffu, fits);
  const int z0 = c[2] + w.lo[2], y0 = c[1] + w.lo[1], x0 = c[0] + w.lo[0];
  if (fits) {
    float cx[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) cx[a] = cof(0, w.lo[0] + a);
    const float4* r0 = S.rec() + z0 * kP3 + y0 * kS3 + x0;
    int i0 = (z0 * kW3 + y0) * kW3 + x0;
#pragma unroll 1
    for (int dz = 0; dz < 4; ++dz) {
      const float cz = cof(2, w.lo[2] + dz);
      unsigned marked = 0;  // rows of this plane in which some lane meets a further item
      if (MORE && nmore) marked = __reduce_or_sync(lanes, ((unsigned)S.rows()[z0 + dz] >> y0) & 15u);
#pragma unroll 1
      for (int dy = 0; dy < 4; ++dy) {
        const float cy = cof(1, w.lo[1] + dy);
        if (!MORE || !((marked >> dy) & 1u)) {
#pragma unroll
          for (int a = 0; a < 4; ++a) one(r0[a], i0 + a, -1, cx[a], cy, cz);
        } else {
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            one(r0[a], i0 + a, -1, cx[a], cy, cz);
            cell_more(S, nmore, i0 + a, [&](int q) { one(S.mrec()[q], -1, q, cx[a], cy, cz); });
          }
        }
        r0 += kS3;
        i0 += kW3;
      }
      r0 += kP3 - 4 * kS3;
      i0 += kW3 * kW3 - 4 * kW3;
    }
  } else if (on) {
#pragma unroll 1
    for (int dz = 0; dz < w.n[2]; ++dz)
#pragma unroll 1
      for (int dy = 0; dy < w.n[1]; ++dy)
#pragma unroll 1
        for (int dx = 0; dx < w.n[0]; ++dx) {
          const int i = ((z0 + dz) * kW3 + y0 + dy) * kW3 + x0 + dx;
          const float ca = cof(0, w.lo[0] + dx), cb = cof(1, w.lo[1] + dy), cc = cof(2, w.lo[2] + dz);
          one(S.rec()[(z0 + dz) * kP3 + (y0 + dy) * kS3 + x0 + dx], i, -1, ca, cb, cc);
          if (MORE) cell_more(S, nmore, i, [&](int q) { one(S.mrec()[q], -1, q, ca, cb, cc); });
        }
  }
}

// Squared displacement of a candidate in the canonical order, plus kTinyD2.
__device__ __forceinline__ float canon_d2_tiny(float ex, float ey, float ez) {
  return rn_add(rn_add(rn_mul(ex, ex), rn_mul(ey, ey)), rn_add(rn_mul(ez, ez), kTinyD2));
}

// The brick's own items beyond one per cell (see GridOwn).
struct GridOwn3 {
  int n, taken;
  int item[kMore3], pos[kMore3];
  __device__ __forceinline__ bool push(int it, int t) {
    const int q = atomicAdd(&n, 1);
    if (q >= kMore3) return false;
    item[q] = it;
    pos[q] = t;
    return true;
  }
  __device__ __forceinline__ bool take(int* it, int* t) {
    if (n == 0) return false;
    const int q = atomicAdd(&taken, 1);
    if (q >= n) return false;
    *it = item[q];
    *t = pos[q];
    return true;
  }
};
// Region coordinates of the brick's cell t.
__device__ __forceinline__ void brick3_cell(int t, int (&c)[3]) {
  c[0] = kHalo3 + (t & (kBrick3 - 1));
  c[1] = kHalo3 + ((t / kBrick3) & (kBrick3 - 1));
  c[2] = kHalo3 + t / (kBrick3 * kBrick3);
}
__device__ __forceinline__ bool brick3_global(const Brick& B, const InstK& I, int t, uint32_t* g) {
  int c[3];
  brick3_cell(t, c);
  const int x = B.x0 + c[0] - kHalo3, y = B.y0 + c[1] - kHalo3, z = B.z0 + c[2] - kHalo3;
  if (x >= I.dims[0] || y >= I.dims[1] || z >= I.dims[2]) return false;
  *g = I.base + (uint32_t)x + (uint32_t)I.dims[0] * ((uint32_t)y + (uint32_t)I.dims[1] * (uint32_t)z);
  return true;
}

__device__ __forceinline__ void copy_async(float* dst, const float* src) { copy4_async(dst, src); }
__device__ __forceinline__ void copy_async(float2* dst, const float2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
// Copies one direction's plane of the region's items: `src` [mcap] of T, into buffer `buf`.
template <class T, class SM>
__device__ __forceinline__ void fetch_plane(const SM& S, int nmore, int buf, const T* __restrict__ src) {
  T* dst = S.template plane<T>(buf);
  T* mdst = S.template mplane<T>(buf);
#pragma unroll 2
  for (int ci = threadIdx.x; ci < kCells3; ci += kThreads3) {
    const int m = S.gi()[ci];
    if (m >= 0) copy_async(dst + ci, src + m);
  }
  for (int q = threadIdx.x; q < nmore; q += kThreads3) {
    copy_async(mdst + q, src + S.mgi()[q]);
    const int key = S.key()[q];
    if ((key & 255) == 1) copy_async(dst + (key >> 8), src + S.mfirst()[q]);
  }
}
__device__ __forceinline__ void fetch_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// ---- thinning + refine --------------------------------------------------------------------------

template <int Q>
__device__ __forceinline__ bool thin_refine_brick(const Args<Q, 3, PF32>& A, const Brick& B, const InstK& I,
                                                  unsigned char* smem) {
  const Grid3Smem<0> S{smem};
  if (threadIdx.x == 0) *S.cnt() = 0;
  if (!stage_grid3(I, B, A.a.start, A.a.off, A.mcap, S, 0, [](int) { return 0.f; })) return false;
  const int nmore = *S.cnt();
  fetch_plane<float>(S, nmore, 0, A.wexp);
  int c[3];
  brick3_cell(threadIdx.x, c);
  uint32_t F = 0;
  const bool valid = brick3_global(B, I, threadIdx.x, &F);

  // thinning: component (m, k) lands in F iff floor(off + cd) == -so on every axis
  uint32_t cnt = 0;
  CSum csum[3];
  float cen[3] = {0.f, 0.f, 0.f};
  if (valid) {
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      int lo[3], nn[3];
      const float cd[3] = {A.L.cdf[k][0], A.L.cdf[k][1], A.L.cdf[k][2]};
#pragma unroll
      for (int a = 0; a < 3; ++a) thin_sources<float>(cd[a], &lo[a], &nn[a]);
#pragma unroll 1
      for (int oz = 0; oz < nn[2]; ++oz)
#pragma unroll 1
        for (int oy = 0; oy < nn[1]; ++oy)
#pragma unroll 1
          for (int ox = 0; ox < nn[0]; ++ox) {
            const int so[3] = {lo[0] + ox, lo[1] + oy, lo[2] + oz};
            const int x = c[0] + so[0], y = c[1] + so[1], z = c[2] + so[2];
            auto land = [&](float4 r) {
              const float o[3] = {r.x, r.y, r.z};
              float t[3];
              bool in = true;
#pragma unroll
              for (int a = 0; a < 3; ++a) {
                t[a] = rn_add(o[a], cd[a]);
                const float lowest = (float)(-so[a]);
                in &= t[a] >= lowest && t[a] < lowest + 1.f;
              }
              if (in) {
                ++cnt;
#pragma unroll
                for (int a = 0; a < 3; ++a) csum[a].add(rn_add((float)so[a], t[a]));
              }
            };
            land(S.rec()[z * kP3 + y * kS3 + x]);
            if (nmore) cell_more(S, nmore, (z * kW3 + y) * kW3 + x, [&](int q) { land(S.mrec()[q]); });
          }
    }
    if (cnt) {
#pragma unroll
      for (int a = 0; a < 3; ++a) cen[a] = csum[a].value() / (float)cnt;
    }
  }
  uint32_t mask = 0;
  float swf = 0.f, sx[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    fetch_wait();
    if (k + 1 < Q) fetch_plane<float>(S, nmore, (k + 1) & 1, A.wexp + (int64_t)(k + 1) * A.mcap);
    const float cd[3] = {A.L.cdf[k][0], A.L.cdf[k][1], A.L.cdf[k][2]};
    const float base[3] = {cen[0] - cd[0], cen[1] - cd[1], cen[2] - cd[2]};
    Win3 w;
    w.set(base, A.R, A.tiny);
    if (cnt > 0)
      cut_window3(S, nmore, c, A.R2, w,
                  [&](int a, float off, int jj) { return rn_add(off, canon_c<float>(jj, cd[a], cen[a])); });
    float dmin = 3.0e38f;
    const float* pw = S.plane<float>(k & 1);
    const float* pm = S.mplane<float>(k & 1);
    window3<true>(S, nmore, cnt > 0, c, w, [&](int a, int j) { return canon_c<float>(j, cd[a], cen[a]); },
                  [&](float4 r, int i, int q, float cx, float cy, float cz) {
                    const float ex = rn_add(r.x, cx), ey = rn_add(r.y, cy), ez = rn_add(r.z, cz);
                    const float d2 = rn_add(rn_add(rn_mul(ex, ex), rn_mul(ey, ey)), rn_mul(ez, ez));
                    dmin = fminf(dmin, d2);
                    float wt = 0.f;  // a miss adds nothing
                    if (d2 <= A.R2) wt = q < 0 ? pw[i] : pm[q];
                    swf = __fadd_rn(swf, wt);
                    sx[0] = __fmaf_rn(wt, ex, sx[0]);
                    sx[1] = __fmaf_rn(wt, ey, sx[1]);
                    sx[2] = __fmaf_rn(wt, ez, sx[2]);
                  });
    if (dmin <= A.R2) mask |= 1u << k;
  }
  if (!valid) return true;
  if (cnt == 0) {
    A.occ[F] = 0u;
    if (A.write_trace) { A.tcnt[F] = 0u; A.mask[F] = 0u; }
    return true;
  }
  const bool moves = __popc(mask) > A.kappa_hard;
  float np[3];
  bool finite = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    np[a] = moves ? cen[a] + sx[a] / swf : cen[a];
    finite &= isfinite(np[a]) && fabsf(np[a]) < 64.f;
  }
  if (!finite) {  // exp(f) underflowed to zero weight: keep the centroid and report it
    atomicOr(A.status, ST_NONFINITE);
#pragma unroll
    for (int a = 0; a < 3; ++a) np[a] = cen[a];
  }
  int sh[3];
  float off[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float fl = floorf(np[a]);
    sh[a] = (int)fl;
    off[a] = np[a] - fl;
    if (off[a] >= 1.f) {
      off[a] = 0.f;
      sh[a] += 1;
    }
  }
  uint32_t Gc;
  const bool inside = cell_at<3>(I, B.x0 + c[0] - kHalo3 + sh[0], B.y0 + c[1] - kHalo3 + sh[1],
                                 B.z0 + c[2] - kHalo3 + sh[2], &Gc);
  if (!inside) atomicOr(A.status, ST_OUT_OF_BOX);
  A.occ[F] = inside ? 1u : 0u;
  A.fkey[F] = inside ? Gc : 0xffffffffu;
#pragma unroll
  for (int a = 0; a < 3; ++a) A.foff[(int64_t)a * A.ncells + F] = off[a];
  if (A.write_trace) {
    A.tcnt[F] = cnt;
    A.mask[F] = mask;
#pragma unroll
    for (int a = 0; a < 3; ++a) A.cen[(int64_t)a * A.ncells + F] = cen[a];
  }
  return true;
}

// ---- weights ------------------------------------------------------------------------------------

template <int Q>
__device__ __forceinline__ bool weights_brick(const Args<Q, 3, PF32>& A, const Brick& B, const InstK& I, int share,
                                              int shares, unsigned char* smem) {
  const Grid3Smem<1> S{smem};
  __shared__ GridOwn3 own;
  if (threadIdx.x == 0) *S.cnt() = own.n = own.taken = 0;
  __syncthreads();
  int t = threadIdx.x, m = 0, m1 = 0, many = 0;
  uint32_t g;
  if (brick3_global(B, I, t, &g)) {
    m = (int)A.a.start[g];
    m1 = (int)A.a.start[g + 1];
  }
  bool has = m1 > m;
  for (int i = m + 1; i < m1 && !many; ++i) many = own.push(i, t) ? 0 : 1;
  if (!__syncthreads_or(has)) return true;  // no moment in the brick
  if (!stage_grid3(I, B, A.b.start, A.b.off, A.ccap, S, many, [](int) { return 0.f; })) return false;
  const int nmore = *S.cnt();
  const float base0 = 768.f * __int_as_float(__float_as_int(A.R) & 0x7f800000);  // see GridWeightSum
  if (!has) has = own.take(&m, &t);
#pragma unroll 1
  while (__any_sync(0xffffffffu, has)) {
    int c[3];
    brick3_cell(t, c);
    float o[3] = {0.f, 0.f, 0.f};
    if (has) {
#pragma unroll
      for (int a = 0; a < 3; ++a) o[a] = A.a.off[(int64_t)a * A.mcap + m];
    }
#pragma unroll 1
    for (int k = share; k < Q; k += shares) {
      const float cd[3] = {A.L.cdf[k][0], A.L.cdf[k][1], A.L.cdf[k][2]};
      const float base[3] = {rn_add(o[0], cd[0]), rn_add(o[1], cd[1]), rn_add(o[2], cd[2])};
      Win3 w;
      w.set(base, A.R, A.tiny);
      if (has)
        cut_window3(S, nmore, c, A.R2, w, [&](int a, float off, int jj) {
          return rn_add(o[a], rn_sub(rn_add((float)(-jj), cd[a]), off));
        });
      GridWeightSum s{base0, 0.f};
      auto one = [&](float4 r, int, int, float bx, float by, float bz) {
        const float ex = rn_add(o[0], rn_sub(bx, r.x)), ey = rn_add(o[1], rn_sub(by, r.y)),
                    ez = rn_add(o[2], rn_sub(bz, r.z));
        s.add(window_weight(-canon_d2_tiny(ex, ey, ez), A.R));
      };
      auto cof = [&](int a, int j) { return rn_add((float)(-j), cd[a]); };
      window3<false>(S, nmore, has, c, w, cof, one);
#pragma unroll 1
      for (int q = 0; q < nmore; ++q) {
        const int ci = S.key()[q] >> 8, row = ci / kW3;
        const int x = ci - row * kW3 - c[0], y = row % kW3 - c[1], z = row / kW3 - c[2];
        if ((unsigned)(x - w.lo[0]) < (unsigned)w.n[0] && (unsigned)(y - w.lo[1]) < (unsigned)w.n[1] &&
            (unsigned)(z - w.lo[2]) < (unsigned)w.n[2])
          one(S.mrec()[q], -1, q, cof(0, x), cof(1, y), cof(2, z));
      }
      if (has) {
        const float sw = __fadd_rn(__fsub_rn(s.hi, base0), s.lo);
        const float inv = sw > 0.f ? 1.f / sw : 0.f;
        const int64_t i = (int64_t)k * A.mcap + m;
        A.sw[i] = inv;
        A.kv[i] = KV<float>{inv, A.a.dev[i]};
      }
    }
    has = has && own.take(&m, &t);
  }
  return true;
}

// ---- gather -------------------------------------------------------------------------------------

template <int Q>
__device__ __forceinline__ bool gather_brick(const Args<Q, 3, PF32>& A, const Brick& B, const InstK& I, int share,
                                             int shares, bool fuse, unsigned char* smem) {
  const Grid3Smem<2> S{smem};
  __shared__ GridOwn3 own;
  if (threadIdx.x == 0) *S.cnt() = own.n = own.taken = 0;
  __syncthreads();
  int t = threadIdx.x, j = 0, j1 = 0, many = 0;
  uint32_t g;
  if (brick3_global(B, I, t, &g)) {
    j = (int)A.b.start[g];
    j1 = (int)A.b.start[g + 1];
  }
  bool has = j1 > j;
  for (int i = j + 1; i < j1 && !many; ++i) many = own.push(i, t) ? 0 : 1;
  if (!__syncthreads_or(has)) return true;  // no control point in the brick
  const bool split = shares > 1;
  const float* rho = A.a.rho;
  if (!stage_grid3(I, B, A.a.start, A.a.off, A.mcap, S, many, [&](int m) { return rho[m]; })) return false;
  const int nmore = *S.cnt();
  if (!has) has = own.take(&j, &t);
  const float2* kvs = reinterpret_cast<const float2*>(A.kv);
  // a round serves one control point per thread; every thread takes part in the copies of each
#pragma unroll 1
  while (__syncthreads_or(has ? 1 : 0)) {
    int c[3];
    brick3_cell(t, c);
    float p[3] = {0.f, 0.f, 0.f};
    if (has) {
#pragma unroll
      for (int a = 0; a < 3; ++a) p[a] = A.b.off[(int64_t)a * A.ccap + j];
    }
    uint32_t empty = 0;
    DF F[Q];
    int buf = 0;
    fetch_plane<float2>(S, nmore, 0, kvs + (int64_t)share * A.mcap);
#pragma unroll 1
    for (int k = share; k < Q; k += shares, buf ^= 1) {
      fetch_wait();
      if (k + shares < Q) fetch_plane<float2>(S, nmore, buf ^ 1, kvs + (int64_t)(k + shares) * A.mcap);
      const float cd[3] = {A.L.cdf[k][0], A.L.cdf[k][1], A.L.cdf[k][2]};
      const float base[3] = {p[0] - cd[0], p[1] - cd[1], p[2] - cd[2]};
      Win3 w;
      w.set(base, A.R, A.tiny);
      if (has)
        cut_window3(S, nmore, c, A.R2, w,
                    [&](int a, float off, int jj) { return rn_add(off, canon_c<float>(jj, cd[a], p[a])); });
      GatherSum s;
      s.clear();
      const float2* pk = S.plane<float2>(buf);
      const float2* pm = S.mplane<float2>(buf);
      window3<true>(S, nmore, has, c, w, [&](int a, int jj) { return canon_c<float>(jj, cd[a], p[a]); },
                    [&](float4 r, int i, int q, float cx, float cy, float cz) {
                      const float ex = rn_add(r.x, cx), ey = rn_add(r.y, cy), ez = rn_add(r.z, cz);
                      const float wgt = window_weight(-canon_d2_tiny(ex, ey, ez), A.R);
                      float2 kv = make_float2(0.f, 0.f);
                      if (wgt > 0.f) kv = q < 0 ? pk[i] : pm[q];
                      s.add(__fmul_rn(wgt, kv.x), r.w, kv.y);
                    });
      const DF Fk = gather_total(A.L.wf[k], A.L.wlo[k], s.hi, s.lo, s.sb);
      if (Fk.hi < A.eps) empty |= 1u << k;
      if (!split) {
        F[k] = Fk;
      } else if (has) {
        A.cpfhi[(int64_t)k * A.ccap + j] = Fk.hi;
        A.cpflo[(int64_t)k * A.ccap + j] = Fk.lo;
      }
    }
    if (split) {
      if (has && empty) atomicOr(A.emask + j, empty);
    } else if (has) {
      A.emask[j] = empty;
      if (fuse && !empty) {
        emit_full<Q>(A, j, F);
      } else {
#pragma unroll
        for (int k = 0; k < Q; ++k) {
          A.cpfhi[(int64_t)k * A.ccap + j] = F[k].hi;
          A.cpflo[(int64_t)k * A.ccap + j] = F[k].lo;
        }
      }
    }
    has = has && own.take(&j, &t);
  }
  return true;
}

// ---- kernels ----------------------------------------------------------------------------------------

// The moments beyond one per cell (noted by the collision) are more than 1 in 32: the region of a brick, 2744
// cells, then holds about 86 of them where it is full, and bricks beyond the list of 128 are common.  Each
// would be staged in vain and wait for the others to finish; the untiled kernels take all bricks instead (a
// cluster of 20 k moments in 64^3 cells: 3006 -> 1494 us a step, 1466 by the untiled kernels' own launches).
template <int Q>
__device__ __forceinline__ bool crowded3(const Args<Q, 3, PF32>& A) {
  return (int64_t)*A.further * 32 > (int64_t)*A.a.count;
}

// Called, not inlined: inline it takes registers from the grid kernel (64^3 cells: 411 -> 505 us).
template <int Q>
__device__ __noinline__ void thin_refine_apart(const Args<Q, 3, PF32>& A, uint32_t F, const InstK& I) {
  thin_refine_cell<Q, 3, PF32>(A, F, I);
}

// STAGE: 0 thin + refine, 1 weights, 2 gather.  In boxes of few bricks gridDim.x / nbricks blocks share a
// brick's directions in weights and gather; the gather then leaves its sums to the emit pass.  As many as run at
// once: blocks beyond that, with nothing to do in a full box, set the others two on an SM (152 bricks:
// weights 287 -> 365 us).  A brick that cannot be staged is thinned by the untiled code in the same
// block (a cell per thread, as there); its weights and gather, where the untiled kernels spread the directions
// over blocks, go to a second launch (k_brick3_fallback).
template <int Q, int STAGE>
__global__ void __launch_bounds__(kThreads3, 2) k_brick3(const __grid_constant__ Args<Q, 3, PF32> A,
                                                        const Brick* __restrict__ bricks, int nbricks,
                                                        int* fb_bricks, int* fb_count, int fuse) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int shares = gridDim.x / nbricks, bi = blockIdx.x / shares, share = blockIdx.x % shares;
  if (crowded3(A)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *fb_count = nbricks;
    return;
  }
  const Brick B = bricks[bi];
  const InstK I = A.inst[B.inst];
  bool ok;
  if constexpr (STAGE == 0) ok = thin_refine_brick<Q>(A, B, I, smem);
  else if constexpr (STAGE == 1) ok = weights_brick<Q>(A, B, I, share, shares, smem);
  // a negative density or an f that is not finite in the instance (noted by the collision): no brick
  else ok = !A.odd_f[B.inst] && gather_brick<Q>(A, B, I, share, shares, fuse != 0, smem);
  if (ok || share > 0) return;
  uint32_t g;
  const bool valid = brick3_global(B, I, threadIdx.x, &g);
  if constexpr (STAGE == 0) {
    if (threadIdx.x == 0) atomicAdd(fb_count, 1);
    if (valid) thin_refine_apart<Q>(A, g, I);
  } else {
    if (threadIdx.x == 0) fb_bricks[atomicAdd(fb_count, 1)] = bi;
    if (STAGE == 2 && fuse && valid)
      for (uint32_t j = A.b.start[g], j1 = A.b.start[g + 1]; j < j1; ++j) A.emask[j] = kEmitLater;
  }
}

// The untiled kernels on the deferred bricks (of a crowded state: on all), each as two bricks of 8 x 8 x 4
// cells (thread t <-> cell t), registers as those kernels (six blocks per SM).  Thin + refine, whose blocks do
// little but for crowded states, has one per unit (handed out one by one: 423 -> 519 us in a cluster of 16 k
// moments in 64^3 cells); weights and gather, with Q times as many units, take the next as they finish one,
// direction by direction.  5 % of 96^3 cells after a step: 29.1 -> 21.9 ms a step, 21.4 by the untiled kernels'
// own launches.
template <int Q, int STAGE>
__global__ void __launch_bounds__(256, 6) k_brick3_fallback(const __grid_constant__ Args<Q, 3, PF32> A,
                                                           const Brick* __restrict__ bricks, int nbricks,
                                                           const int* __restrict__ fb_bricks,
                                                           const int* __restrict__ fb_count, int* ticket) {
  const bool all = crowded3(A);
  if (STAGE == 0 && !all) return;
  const BrickGeo bg{kBrick3, kBrick3, kBrick3 / 2};
  if constexpr (STAGE == 0) {
    Brick B = bricks[blockIdx.x >> 1];
    B.z0 += (int)(blockIdx.x & 1) * (kBrick3 / 2);
    const InstK I = A.inst[B.inst];
    uint32_t F;
    if (brick_cell<3>(B, I, bg, threadIdx.x, &F)) thin_refine_cell<Q, 3, PF32>(A, F, I);
    return;
  }
  const int n = 2 * (all ? nbricks : *fb_count);
  const int64_t units = (int64_t)n * Q;
  __shared__ int s_next;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_next = units > 0 ? atomicAdd(ticket, 1) : 0;
    __syncthreads();
    const int64_t u = s_next;
    if (u >= units) return;
    const int k = (int)(u / n), e = (int)(u - (int64_t)k * n);
    Brick B = bricks[all ? e >> 1 : fb_bricks[e >> 1]];
    B.z0 += (e & 1) * (kBrick3 / 2);
    const InstK I = A.inst[B.inst];
    uint32_t F;
    if (!brick_cell<3>(B, I, bg, threadIdx.x, &F)) continue;
    if constexpr (STAGE == 1) {
      for (uint32_t m = A.a.start[F], m1 = A.a.start[F + 1]; m < m1; ++m) weights_one<Q, 3, PF32>(A, m, k, F, I);
    } else {
      for (uint32_t j = A.b.start[F], j1 = A.b.start[F + 1]; j < j1; ++j) gather_one<Q, 3, PF32>(A, j, k, F, I);
    }
  }
}

// Emits the control points without an empty direction of the bricks near an obstacle, which the untiled gather
// served.
template <int Q>
__global__ void __launch_bounds__(256) k_emit_bricks(const __grid_constant__ Args<Q, 3, PF32> A,
                                                    const Brick* __restrict__ bricks, BrickGeo bg, int nbricks) {
  for (int u = blockIdx.x; u < nbricks; u += gridDim.x) {
    const Brick B = bricks[u];
    const InstK I = A.inst[B.inst];
    uint32_t F;
    if (!brick_cell<3>(B, I, bg, threadIdx.x, &F)) continue;
    for (uint32_t j = A.b.start[F], j1 = A.b.start[F + 1]; j < j1; ++j)
      if (A.emask[j] == 0u) emit_from_cpf<Q>(A, (int)j);
  }
}

}  // namespace dbm
