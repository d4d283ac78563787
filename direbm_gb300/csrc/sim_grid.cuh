// Grid variants of the three tiled window kernels (2D, FP32 store) for displacements that are not
// whole cells, or radii of more than two cells: the reference's parameters (D2Q7, r = dx, cell dx / 4:
// R = 4 cells) and D2Q7 with dx = cell.
//
// The row-segment kernels walk, per (reference point, direction), the item ranges of the window's
// rows: a loop of uneven length with a branch per item, a test for each item's place in its cell and a
// second walk over all rows when any window cell holds two items (nearly always, at 80 cells a window
// and 1-2 % of such cells).  Here a tile's region is staged as a grid, as in the dense kernels
// (sim_dense.cuh, whose staging planes, window weight and sums these use): one record per cell, an
// empty cell with offsets outside every window.  A window is W x W cells from floor(p - cd - R - tiny),
// W = ceil(2 R) + 1, which holds the exact range except for a point within `tiny` of a cell border
// (a loop over the exact range then); the W column displacements are formed once per direction, and a
// row is W unrolled candidates without a branch, a miss adding the weight 0.  At R = 4 that is 81
// candidates for 50 hits, at 12 - 26 instructions each.
//
// All further items of the region's cells are kept in one list ordered by (row, column, place in the
// cell); after a direction's grid pass the window's part of the list follows, in that order, which is
// the row-segment kernels' second pass.  Results are bit-identical to them.  A tile with more further
// items than the list takes goes to the row-segment code, in the same block.
// Bound by instruction issue.  D2Q7, R = 4, 368,640 moments, one per cell, us per launch, row segments /
// grid: thin + refine 828 / 155, weights 371 / 171, gather 1098 / 255, whole step 2490 / 641; after 100
// steps (two-item cells) 3333 / 744.
#pragma once

#include "sim_dense.cuh"

namespace dbm {

// Further items of a tile's region, and of its own cells, at most.
constexpr int kGridMore = 128;

// Shared memory: offsets (float2) of each cell's first item, NP pair planes, NF float planes, the item
// index (gather) and per cell the place of its first further item in the ordered list (-1: none); the
// further items' offsets, planes, indices and keys; the list's row starts.
struct GridLayout {
  int rw, rh, s2, s1, n2, n1;
  int kv, fl, gi, nx, mxy, mkv, mfl, mgi, key, ord, row, cnt, total;
  __host__ __device__ GridLayout(int w, int h, int np, int nf, int idx) : rw(w), rh(h) {
    s2 = (w + 15) & ~15;
    s1 = (w + 31) & ~31;
    n2 = s2 * h;
    n1 = s1 * h;
    kv = n2 * 8;
    fl = kv + np * n2 * 8;
    gi = fl + nf * n1 * 4;
    nx = gi + idx * n2 * 4;
    mxy = nx + ((n2 * 2 + 15) & ~15);
    mkv = mxy + kGridMore * 8;
    mfl = mkv + np * kGridMore * 8;
    mgi = mfl + nf * kGridMore * 4;
    key = mgi + kGridMore * 4;
    ord = key + kGridMore * 4;
    row = ord + kGridMore * 4;
    cnt = row + ((h * 4 + 4 + 15) & ~15);
    total = cnt + 16;
  }
};
// stage 0 thin + refine: exp(f*) (Q floats); 1 weights; 2 gather: rho, and (1/sw, f*) of two directions
__host__ __device__ inline GridLayout grid_layout(int Q, int stage, const TileGeo& G) {
  const Halo& h = stage == 1 ? G.cp : G.mom;
  // one more column and row than the halo: a window narrower than W still reads W cells
  return GridLayout(G.tx + h.xh - h.xl + 1, G.ty + h.yh - h.yl + 1, stage == 2 ? 2 : 0, stage == 0 ? Q : stage == 2 ? 1 : 0,
                    stage == 2 ? 1 : 0);
}

struct GridSmem {
  GridLayout L;
  unsigned char* p;
  template <class T>
  __device__ __forceinline__ T* at(int o) const { return reinterpret_cast<T*>(p + o); }
  __device__ __forceinline__ float2* xy() const { return at<float2>(0); }
  __device__ __forceinline__ float2* kv() const { return at<float2>(L.kv); }
  __device__ __forceinline__ float* fl() const { return at<float>(L.fl); }
  __device__ __forceinline__ int* gi() const { return at<int>(L.gi); }
  __device__ __forceinline__ short* nx() const { return at<short>(L.nx); }
  __device__ __forceinline__ float2* mxy() const { return at<float2>(L.mxy); }
  __device__ __forceinline__ float2* mkv() const { return at<float2>(L.mkv); }
  __device__ __forceinline__ float* mfl() const { return at<float>(L.mfl); }
  __device__ __forceinline__ int* mgi() const { return at<int>(L.mgi); }
  // region row << 20 | column << 8 | place in the cell, of each further item
  __device__ __forceinline__ int* key() const { return at<int>(L.key); }
  __device__ __forceinline__ int* ord() const { return at<int>(L.ord); }  // slots in key order
  __device__ __forceinline__ int* row() const { return at<int>(L.row); }  // [rh + 1] first list place of a row
  __device__ __forceinline__ int* cnt() const { return at<int>(L.cnt); }
};

// Stages the region from (xr0, yr0): put(item, offsets, cell slot (float2 planes), cell slot (float
// planes)) and more(item, offsets, slot) fill the planes of a first and of a further item.  Returns
// false, the same in every thread, when the tile must be deferred.  On true the list is ordered.
template <int NF, class Put, class More>
__device__ __forceinline__ bool stage_grid(const InstK& I, int xr0, int yr0, const uint32_t* __restrict__ start,
                                           const float* __restrict__ off, int64_t stride, const GridSmem& S, int many,
                                           Put&& put, More&& more) {
  const int rw = S.L.rw, cells = rw * S.L.rh;
  for (int ci = threadIdx.x; ci < cells; ci += blockDim.x) {
    const int ry = ci / rw, rx = ci - ry * rw;
    const int i2 = ry * S.L.s2 + rx, i1 = ry * S.L.s1 + rx;
    uint32_t g;
    int b = 0, e = 0;
    if (region_cell(I, xr0 + rx, yr0 + ry, &g)) {
      b = (int)start[g];
      e = (int)start[g + 1];
    }
    S.nx()[i2] = -1;
    if (e > b) {
      const float2 o = make_float2(off[b], off[stride + b]);
      S.xy()[i2] = o;
      many |= (int)!(o.x + o.y < 4.f);  // NaN: 0 x it is not 0
      put(b, o, i2, i1);
      for (int m = b + 1; m < e; ++m) {
        const int q = atomicAdd(S.cnt(), 1);
        if (q >= kGridMore || m - b > 255) {
          many = 1;
          break;
        }
        const float2 om = make_float2(off[m], off[stride + m]);
        S.mxy()[q] = om;
        many |= (int)!(om.x + om.y < 4.f);
        S.key()[q] = (ry << 20) | (rx << 8) | (m - b);
        more(m, om, q);
      }
    } else {
      S.xy()[i2] = make_float2(kEmptyOff, kEmptyOff);
      put(-1, make_float2(0.f, 0.f), i2, i1);
    }
  }
  if (__syncthreads_or(many)) return false;
  const int n = *S.cnt();
  if (n > 0) {  // the same in every thread: order the list by rank (keys are distinct)
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
      const int kq = S.key()[q];
      int rank = 0;
      for (int r = 0; r < n; ++r) rank += S.key()[r] < kq ? 1 : 0;
      S.ord()[rank] = q;
      if ((kq & 255) == 1) S.nx()[(kq >> 20) * S.L.s2 + ((kq >> 8) & 0xfff)] = (short)rank;
    }
    for (int r = threadIdx.x; r <= S.L.rh; r += blockDim.x) {
      int c = 0;
      for (int q = 0; q < n; ++q) c += (S.key()[q] >> 20) < r ? 1 : 0;
      S.row()[r] = c;
    }
    __syncthreads();
  }
  return true;
}

// Further items of region rows [r0, r0 + nr) and columns [c0, c0 + nc), in order: fn(slot, row, column).
template <class Fn>
__device__ __forceinline__ void window_more(const GridSmem& S, int r0, int nr, int c0, int nc, Fn&& fn) {
  const int end = S.row()[r0 + nr];
#pragma unroll 1
  for (int i = S.row()[r0]; i < end; ++i) {
    const int q = S.ord()[i], k = S.key()[q];
    const int c = (k >> 8) & 0xfff;
    if ((unsigned)(c - c0) < (unsigned)nc) fn(q, k >> 20, c);
  }
}

// The tile's own reference points beyond one per cell: offered to threads without one of their own;
// what is left takes another round.
struct GridOwn {
  int n, taken;
  int item[kGridMore], pos[kGridMore];
  __device__ __forceinline__ bool push(int it, int bx, int by) {
    const int q = atomicAdd(&n, 1);
    if (q >= kGridMore) return false;
    item[q] = it;
    pos[q] = (by << 16) | bx;
    return true;
  }
  __device__ __forceinline__ bool take(int* it, int* bx, int* by) {
    if (n == 0) return false;
    const int q = atomicAdd(&taken, 1);
    if (q >= n) return false;
    *it = item[q];
    *bx = pos[q] & 0xffff;
    *by = pos[q] >> 16;
    return true;
  }
};

// Exact running sum of window weights as WeightSum, for R in [2^e, 2^(e+1)): every weight is a multiple
// of 2^(e - 24), `hi` starts at 3 x 2^(e + 8) and the at most 81 + kGridMore rounding errors of half an ulp
// of it add up exactly in `lo`.
struct GridWeightSum {
  float hi, lo;
  __device__ __forceinline__ void add(float w) {
    const float t = __fadd_rn(hi, w);
    lo = __fadd_rn(lo, __fsub_rn(w, __fsub_rn(t, hi)));
    hi = t;
  }
};

// ---- thinning + refine --------------------------------------------------------------------------

template <int Q, int W>
__device__ __forceinline__ bool thin_refine_grid_tile(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                                      const TileGeo& G, unsigned char* smem) {
  const GridSmem S{grid_layout(Q, 0, G), smem};
  const int s2 = S.L.s2, s1 = S.L.s1;
  if (threadIdx.x == 0) *S.cnt() = 0;
  __syncthreads();
  const bool ok = stage_grid<Q>(
      I, T.x0 + G.mom.xl, T.y0 + G.mom.yl, A.a.start, A.a.off, A.mcap, S, 0,
      [&](int m, float2, int, int i1) {
        if (m >= 0) {
#pragma unroll
          for (int k = 0; k < Q; ++k) S.fl()[k * S.L.n1 + i1] = exp(fstar_at<Q, 2, PF32>(A, (uint32_t)m, k));
        }
      },
      [&](int m, float2, int q) {
#pragma unroll
        for (int k = 0; k < Q; ++k) S.mfl()[k * kGridMore + q] = exp(fstar_at<Q, 2, PF32>(A, (uint32_t)m, k));
      });
  if (!ok) return false;
  const int nmore = *S.cnt();

  const int lx = threadIdx.x % G.tx, ly = threadIdx.x / G.tx;
  const int Fx = T.x0 + lx, Fy = T.y0 + ly;
  if (ly >= G.ty || Fx >= I.dims[0] || Fy >= I.dims[1]) return true;
  const uint32_t F = I.base + (uint32_t)Fx + (uint32_t)I.dims[0] * (uint32_t)Fy;
  const int bx = lx - G.mom.xl, by = ly - G.mom.yl;  // region coordinates of F

  // thinning: component (m, k) lands in F iff floor(off + cd) == -so on both axes
  uint32_t cnt = 0;
  CSum csum[2];
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    const float cdx = A.L.cdf[k][0], cdy = A.L.cdf[k][1];
    int lox, nx, loy, ny;
    thin_sources<float>(cdx, &lox, &nx);
    thin_sources<float>(cdy, &loy, &ny);
#pragma unroll 1
    for (int oy = 0; oy < ny; ++oy) {
      const int soy = loy + oy;
      const float fy0 = (float)(-soy), sy = (float)soy;
#pragma unroll 1
      for (int ox = 0; ox < nx; ++ox) {
        const int sox = lox + ox;
        const float sxf = (float)sox;
        auto land = [&](float2 o) {
          const float tx = rn_add(o.x, cdx), ty = rn_add(o.y, cdy);
          if (tx >= -sxf && tx < 1.f - sxf && ty >= fy0 && ty < fy0 + 1.f) {
            ++cnt;
            csum[0].add(rn_add(sxf, tx));
            csum[1].add(rn_add(sy, ty));
          }
        };
        const int rx = bx + sox, ry = by + soy, ci = ry * s2 + rx;
        land(S.xy()[ci]);
        if (nmore) {
          const int cell = (ry << 12) | rx;
          for (int i = S.nx()[ci]; i >= 0 && i < nmore; ++i) {
            const int q = S.ord()[i];
            if (S.key()[q] >> 8 != cell) break;
            land(S.mxy()[q]);
          }
        }
      }
    }
  }
  if (cnt == 0) {
    A.occ[F] = 0u;
    A.fkey[F] = 0xffffffffu;  // read by the placement's neighbourhood search
    if (A.write_trace) {
      A.tcnt[F] = 0u;
      A.mask[F] = 0u;
    }
    return true;
  }
  const float cen[2] = {csum[0].value() / (float)cnt, csum[1].value() / (float)cnt};

  uint32_t mask = 0;
  float swf = 0.f;
  float2 sx = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int k = 0; k < Q; ++k) {
    const float cdx = A.L.cdf[k][0], cdy = A.L.cdf[k][1];
    const float bxr = cen[0] - cdx, byr = cen[1] - cdy;
    const int lox = (int)floorf(bxr - A.R - A.tiny), nx = (int)floorf(bxr + A.R + A.tiny) - lox + 1;
    const int loy = (int)floorf(byr - A.R - A.tiny), ny = (int)floorf(byr + A.R + A.tiny) - loy + 1;
    float dmin = 3.0e38f;  // at or below R2 in the end when any candidate of the direction hit
    auto one = [&](float2 o, const float* wp, float cx, float cy) {
      const float2 e = __fadd2_rn(o, make_float2(cx, cy));
      const float2 e2 = __fmul2_rn(e, e);
      const float d2 = rn_add(e2.x, e2.y);
      dmin = fminf(dmin, d2);
      float wt = 0.f;  // a miss adds nothing
      if (d2 <= A.R2) wt = *wp;
      swf = __fadd_rn(swf, wt);
      sx.x = __fmaf_rn(wt, e.x, sx.x);
      sx.y = __fmaf_rn(wt, e.y, sx.y);
    };
    const float2* o0 = S.xy() + (by + loy) * s2 + bx + lox;
    const float* w0 = S.fl() + k * S.L.n1 + (by + loy) * s1 + bx + lox;
    if (nx <= W && ny <= W) {
      float cx[W];
#pragma unroll
      for (int a = 0; a < W; ++a) cx[a] = canon_c<float>(lox + a, cdx, cen[0]);
#pragma unroll 1
      for (int b = 0; b < ny; ++b, o0 += s2, w0 += s1) {
        const float cy = canon_c<float>(loy + b, cdy, cen[1]);
#pragma unroll
        for (int a = 0; a < W; ++a) one(o0[a], w0 + a, cx[a], cy);
      }
    } else {
#pragma unroll 1
      for (int b = 0; b < ny; ++b, o0 += s2, w0 += s1)
#pragma unroll 1
        for (int a = 0; a < nx; ++a)
          one(o0[a], w0 + a, canon_c<float>(lox + a, cdx, cen[0]), canon_c<float>(loy + b, cdy, cen[1]));
    }
    if (nmore)
      window_more(S, by + loy, ny, bx + lox, nx, [&](int q, int r, int c) {
        one(S.mxy()[q], S.mfl() + k * kGridMore + q, canon_c<float>(c - bx, cdx, cen[0]),
            canon_c<float>(r - by, cdy, cen[1]));
      });
    if (dmin <= A.R2) mask |= 1u << k;
  }
  refine_store<Q>(A, I, F, Fx, Fy, cnt, mask, cen, swf, sx);
  return true;
}

// ---- weights ------------------------------------------------------------------------------------

template <int Q, int W>
__device__ __forceinline__ bool weights_grid_tile(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                                  const TileGeo& G, int shares, unsigned char* smem) {
  const GridSmem S{grid_layout(Q, 1, G), smem};
  const int s2 = S.L.s2;
  __shared__ GridOwn own;
  if (threadIdx.x == 0) *S.cnt() = own.n = own.taken = 0;
  __syncthreads();
  const int lx = threadIdx.x % G.tx, ly = threadIdx.x / G.tx;
  const int Sx = T.x0 + lx, Sy = T.y0 + ly;
  int bx = lx - G.cp.xl, by = ly - G.cp.yl;  // region coordinates of the moment's cell
  int m = 0, m1 = 0, many = 0;
  if (ly < G.ty && Sx < I.dims[0] && Sy < I.dims[1]) {
    const uint32_t g = I.base + (uint32_t)Sx + (uint32_t)I.dims[0] * (uint32_t)Sy;
    m = (int)A.a.start[g];
    m1 = (int)A.a.start[g + 1];
  }
  bool has = m1 > m;
  for (int i = m + 1; i < m1 && !many; ++i) many = own.push(i, bx, by) ? 0 : 1;
  if (!__syncthreads_or(has)) return true;  // no moment in the tile
  if (!stage_grid<0>(I, T.x0 + G.cp.xl, T.y0 + G.cp.yl, A.b.start, A.b.off, A.ccap, S, many,
                     [&](int, float2, int, int) {}, [&](int, float2, int) {}))
    return false;
  const int nmore = *S.cnt();
  // sums of weights from 3 x 2^(e + 8), R in [2^e, 2^(e + 1)) (GridWeightSum)
  const float base0 = 768.f * __int_as_float(__float_as_int(A.R) & 0x7f800000);
  if (!has) has = own.take(&m, &bx, &by);
#pragma unroll 1
  while (has) {
    const float2 o = make_float2(A.a.off[m], A.a.off[A.mcap + m]);
#pragma unroll 1
    for (int k = blockIdx.y; k < Q; k += shares) {
      const float cdx = A.L.cdf[k][0], cdy = A.L.cdf[k][1];
      const float tx = rn_add(o.x, cdx), ty = rn_add(o.y, cdy);
      const int lox = (int)floorf(tx - A.R - A.tiny), nx = (int)floorf(tx + A.R + A.tiny) - lox + 1;
      const int loy = (int)floorf(ty - A.R - A.tiny), ny = (int)floorf(ty + A.R + A.tiny) - loy + 1;
      GridWeightSum s{base0, 0.f};
      auto one = [&](float2 pc, float basex, float basey) {
        const float ex = rn_add(o.x, rn_sub(basex, pc.x)), ey = rn_add(o.y, rn_sub(basey, pc.y));
        s.add(window_weight(-rn_add(rn_mul(ex, ex), rn_add(rn_mul(ey, ey), kTinyD2)), A.R));
      };
      const float2* p0 = S.xy() + (by + loy) * s2 + bx + lox;
      if (nx <= W && ny <= W) {
        float bxv[W];
#pragma unroll
        for (int a = 0; a < W; ++a) bxv[a] = rn_add((float)(-(lox + a)), cdx);
#pragma unroll 1
        for (int b = 0; b < ny; ++b, p0 += s2) {
          const float basey = rn_add((float)(-(loy + b)), cdy);
#pragma unroll
          for (int a = 0; a < W; ++a) one(p0[a], bxv[a], basey);
        }
      } else {
#pragma unroll 1
        for (int b = 0; b < ny; ++b, p0 += s2)
#pragma unroll 1
          for (int a = 0; a < nx; ++a)
            one(p0[a], rn_add((float)(-(lox + a)), cdx), rn_add((float)(-(loy + b)), cdy));
      }
      if (nmore)
        window_more(S, by + loy, ny, bx + lox, nx, [&](int q, int r, int c) {
          one(S.mxy()[q], rn_add((float)(bx - c), cdx), rn_add((float)(by - r), cdy));
        });
      const float sw = __fadd_rn(__fsub_rn(s.hi, base0), s.lo);
      A.sw[(int64_t)k * A.mcap + m] = sw > 0.f ? 1.f / sw : 0.f;
    }
    has = own.take(&m, &bx, &by);
  }
  return true;
}

// ---- gather -------------------------------------------------------------------------------------

__device__ __forceinline__ void copy4_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// One direction's (1/sw, f*) pairs are staged while the previous direction runs (two buffers).
template <int Q, int W>
__device__ __forceinline__ bool gather_grid_tile(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                                 const TileGeo& G, int shares, bool fuse, unsigned char* smem) {
  const GridSmem S{grid_layout(Q, 2, G), smem};
  const int s2 = S.L.s2, s1 = S.L.s1, n2 = S.L.n2;
  __shared__ GridOwn own;
  if (threadIdx.x == 0) *S.cnt() = own.n = own.taken = 0;
  __syncthreads();
  const int lx = threadIdx.x % G.tx, ly = threadIdx.x / G.tx;
  const int Fx = T.x0 + lx, Fy = T.y0 + ly;
  int bx = lx - G.mom.xl, by = ly - G.mom.yl;  // region coordinates of the control point's cell
  int j = 0, j1 = 0, many = 0;
  if (ly < G.ty && Fx < I.dims[0] && Fy < I.dims[1]) {
    const uint32_t g = I.base + (uint32_t)Fx + (uint32_t)I.dims[0] * (uint32_t)Fy;
    j = (int)A.b.start[g];
    j1 = (int)A.b.start[g + 1];
  }
  bool has = j1 > j;
  for (int i = j + 1; i < j1 && !many; ++i) many = own.push(i, bx, by) ? 0 : 1;
  if (!__syncthreads_or(has)) return true;  // no control point in the tile
  if (!stage_grid<1>(
          I, T.x0 + G.mom.xl, T.y0 + G.mom.yl, A.a.start, A.a.off, A.mcap, S, many,
          [&](int m, float2, int i2, int i1) {
            S.gi()[i2] = m;
            S.fl()[i1] = m >= 0 ? A.a.rho[m] : 0.f;
            if (m < 0) S.kv()[i2] = S.kv()[n2 + i2] = make_float2(0.f, 0.f);
          },
          [&](int m, float2, int q) {
            S.mgi()[q] = m;
            S.mfl()[q] = A.a.rho[m];
          }))
    return false;
  const int nmore = *S.cnt();
  const int rw = S.L.rw, cells = rw * S.L.rh;
  const bool split = shares > 1;
  auto fetch = [&](int k, int buf) {
    const float* inv = A.sw + (int64_t)k * A.mcap;
    const float* fk = A.a.dev + (int64_t)k * A.mcap;
    float2* kv = S.kv() + buf * n2;
    float2* mkv = S.mkv() + buf * kGridMore;
    for (int ci = threadIdx.x; ci < cells; ci += blockDim.x) {
      const int ry = ci / rw, i2 = ry * s2 + ci - ry * rw, m = S.gi()[i2];
      if (m >= 0) {
        copy4_async(&kv[i2].x, inv + m);
        copy4_async(&kv[i2].y, fk + m);
      }
    }
    for (int q = threadIdx.x; q < nmore; q += blockDim.x) {
      const int m = S.mgi()[q];
      copy4_async(&mkv[q].x, inv + m);
      copy4_async(&mkv[q].y, fk + m);
    }
  };
  if (!has) has = own.take(&j, &bx, &by);
  // a round serves one control point per thread; every thread takes part in the copies of each
#pragma unroll 1
  while (__syncthreads_or(has ? 1 : 0)) {
    const float2 pp = has ? make_float2(A.b.off[j], A.b.off[A.ccap + j]) : make_float2(0.f, 0.f);
    uint32_t empty = 0;
    DF F[Q];
    int buf = 0;
    fetch(blockIdx.y, 0);
#pragma unroll 1
    for (int k = blockIdx.y; k < Q; k += shares, buf ^= 1) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      if (k + shares < Q) fetch(k + shares, buf ^ 1);
      if (!has) continue;
      const float cdx = A.L.cdf[k][0], cdy = A.L.cdf[k][1];
      const float bxr = pp.x - cdx, byr = pp.y - cdy;
      const int lox = (int)floorf(bxr - A.R - A.tiny), nx = (int)floorf(bxr + A.R + A.tiny) - lox + 1;
      const int loy = (int)floorf(byr - A.R - A.tiny), ny = (int)floorf(byr + A.R + A.tiny) - loy + 1;
      GatherSum s;
      s.clear();
      auto one = [&](float2 o, float rho, float2 kv, float cx, float cy) {
        const float ex = rn_add(o.x, cx), ey = rn_add(o.y, cy);
        const float w = window_weight(-rn_add(rn_mul(ex, ex), rn_add(rn_mul(ey, ey), kTinyD2)), A.R);
        s.add(__fmul_rn(w, kv.x), rho, kv.y);
      };
      const int i0 = (by + loy) * s2 + bx + lox;
      const float2* o0 = S.xy() + i0;
      const float2* kv0 = S.kv() + buf * n2 + i0;
      const float* r0 = S.fl() + (by + loy) * s1 + bx + lox;
      if (nx <= W && ny <= W) {
        float cx[W];
#pragma unroll
        for (int a = 0; a < W; ++a) cx[a] = canon_c<float>(lox + a, cdx, pp.x);
#pragma unroll 1
        for (int b = 0; b < ny; ++b, o0 += s2, kv0 += s2, r0 += s1) {
          const float cy = canon_c<float>(loy + b, cdy, pp.y);
#pragma unroll
          for (int a = 0; a < W; ++a) one(o0[a], r0[a], kv0[a], cx[a], cy);
        }
      } else {
#pragma unroll 1
        for (int b = 0; b < ny; ++b, o0 += s2, kv0 += s2, r0 += s1)
#pragma unroll 1
          for (int a = 0; a < nx; ++a)
            one(o0[a], r0[a], kv0[a], canon_c<float>(lox + a, cdx, pp.x), canon_c<float>(loy + b, cdy, pp.y));
      }
      if (nmore)
        window_more(S, by + loy, ny, bx + lox, nx, [&](int q, int r, int c) {
          one(S.mxy()[q], S.mfl()[q], S.mkv()[buf * kGridMore + q], canon_c<float>(c - bx, cdx, pp.x),
              canon_c<float>(r - by, cdy, pp.y));
        });
      const DF Fk = gather_total(A.L.wf[k], A.L.wlo[k], s.hi, s.lo, s.sb);
      if (Fk.hi < A.eps) empty |= 1u << k;
      if (split) {
        A.cpfhi[(int64_t)k * A.ccap + j] = Fk.hi;
        A.cpflo[(int64_t)k * A.ccap + j] = Fk.lo;
      } else {
        F[k] = Fk;
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
    has = own.take(&j, &bx, &by);
  }
  return true;
}

// ---- kernels ----------------------------------------------------------------------------------------
//
// Weights and gather of few moments: up to gridDim.y blocks share a tile's directions (k = blockIdx.y,
// blockIdx.y + shares, ...), since one block per SM waits on its own loads and sums.  Shares
// (direction_shares): as many as the blocks of the moments' tiles (256 cells, one moment each where the store is full) still run at once, and
// the directions in equal parts.  The gather then leaves its sums to the emit pass.  D2Q7 at R = 4
// cells, 5 k to 30 k moments in 24 k to 63 k cells: weights 93 -> 33 us, gather 167 -> 47.  Every block of a tile
// stages the same items and finds the same fault, and the first takes it to the row segments.

__device__ __forceinline__ void count_deferred(int* fb_count) {
  if (threadIdx.x == 0) atomicAdd(fb_count, 1);
}

// This launch's shares (the moments the step began with); slots 0: one.
template <int Q>
__device__ __forceinline__ int grid_shares(const Args<Q, 2, PF32>& A) {
  return A.share_slots ? min(direction_shares<Q>(*A.a.count, A.share_slots), (int)gridDim.y) : 1;
}


// A tile that cannot be staged goes to the row-segment code at once, in the same block (and shared memory,
// of the larger need): its few tiles are the last to finish, and in a launch of their own they started after
// all others had (a cluster in 512 x 512 cells, 57 k moments, R = 1.5: 545 -> 387 us a step, row segments alone
// 416; R = 4: 1689 -> 1357, 1407).  fb_count: their number.
template <int Q, int W>
__global__ void __launch_bounds__(256, 4) k_thin_refine_grid(const __grid_constant__ Args<Q, 2, PF32> A,
                                                            const Tile2* __restrict__ tiles, const TileGeo G, int ntiles,
                                                            int* fb_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int tb = blockIdx.x; tb < ntiles; tb += gridDim.x) {
    const Tile2 T = tiles[tb];
    const InstK I = A.inst[T.inst];
    if (!thin_refine_grid_tile<Q, W>(A, T, I, G, smem)) {
      count_deferred(fb_count);
      thin_refine_tile<Q, PF32, false>(A, T, I, G, smem);
    }
    __syncthreads();
  }
}

template <int Q, int W>
__global__ void __launch_bounds__(256, 4) k_weights_grid(const __grid_constant__ Args<Q, 2, PF32> A,
                                                        const Tile2* __restrict__ tiles, const TileGeo G, int ntiles,
                                                        int* fb_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int shares = grid_shares<Q>(A);
  if ((int)blockIdx.y >= shares) return;
  for (int tb = blockIdx.x; tb < ntiles; tb += gridDim.x) {
    const Tile2 T = tiles[tb];
    const InstK I = A.inst[T.inst];
    if (!weights_grid_tile<Q, W>(A, T, I, G, shares, smem) && blockIdx.y == 0) {
      count_deferred(fb_count);
      weights_tile<Q, PF32, false>(A, T, I, G, smem);
    }
    __syncthreads();
  }
}

template <int Q, int W>
__global__ void __launch_bounds__(256, 4) k_gather_grid(const __grid_constant__ Args<Q, 2, PF32> A,
                                                       const Tile2* __restrict__ tiles, const TileGeo G, int ntiles,
                                                       int* fb_count, int fuse) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int shares = grid_shares<Q>(A);
  if ((int)blockIdx.y >= shares) return;
  for (int tb = blockIdx.x; tb < ntiles; tb += gridDim.x) {
    const Tile2 T = tiles[tb];
    const InstK I = A.inst[T.inst];
    // a negative density or an f that is not finite in the instance (noted by the collision): no grid tile
    if ((A.odd_f[T.inst] || !gather_grid_tile<Q, W>(A, T, I, G, shares, fuse != 0, smem)) && blockIdx.y == 0) {
      count_deferred(fb_count);
      gather_fallback<Q>(A, T, I, G, fuse != 0, [&] { gather_tile<Q, PF32>(A, T, I, G, smem); });
    }
    __syncthreads();
  }
}

}  // namespace dbm
