// Dense-stencil variants of the three whole-cell window kernels (2D, FP32 store).
//
// With whole-cell displacements (every cd_k an integer, D2Q9 with dx = cell) and R < 2 cells, the
// thinning cell holds at most one control point, so in the ensemble and inverse-problem workloads
// almost every cell holds exactly one moment: all of them at first, and after some steps all but
// ~1 % (a refine move occasionally crosses a cell face, leaving a cell with two items and another
// empty).  A tile's region is therefore staged as a dense grid -- one offset pair per region cell,
// an empty cell holding an offset far outside every window, the second item of a two-item cell in
// a small per-tile overflow list -- and each reference point's window for direction k is a fixed
// 4 x 4 block of cells: the component-cell offsets j with e = off + (j - p) in reach of R are
// floor(p - R - tiny) .. floor(p + R + tiny), at most four values per axis at R = 1.5 except
// within tiny of p = 1/2 (five).  A point whose range is wider takes a loop over its exact range, so
// no access leaves the staged region (its halo covers the exact ranges for any R < 2).
//
// NEAR kernels (dx = cell, 1 <= R < 2: the workloads' case).  Direction k's block is the block of
// cd = 0 shifted by -cd_k, so the three directions of one c_y use the same four rows of six items: a
// row's items are loaded once for the three, e_y^2 is formed once per item, and the three sums run
// side by side.  No candidate branches: a miss gets the weight max(R - d, 0) = 0, which leaves every
// sum unchanged, so the independent chains hide each other's latency where the branching loop ran one
// candidate at a time with 18-23 of 32 lanes active.  Strides are compile-time constants of the tile
// width.  Loops over c_y and over rows stay rolled: unrolled further, the body (48 and 144 candidates)
// outgrows the instruction cache and the gather runs 10-25 % slower.
//
// Results are bit-identical to the row-segment kernels: each sum visits the same hits in the same
// order with the same operations.  The first items of the window's cells come first (window rows
// ascending, then columns ascending), then the second items in the same cell order.  A tile whose
// region holds a cell with three or more items, or more two-item cells than the overflow list takes,
// is handed to the row-segment code (a second, normally empty, launch over the deferred tiles); so
// are the gather's tiles of an instance with a negative density or an f that is not finite (0 x it is not 0).
//
// Bound by instruction issue (thin + refine 88 % of issue slots and 87 % of shared-memory wavefronts,
// weights 78 %, gather 70 %; DRAM 5-10 %).  Ensemble of 15.5 M moments, 16 x 16 tiles, ms per step,
// branching 4 x 4 stencil before / now: thin + refine 2.33 / 1.70, weights 2.92 / 1.66, gather with
// emit 4.51 / 3.50; whole step 10.2 / 7.3, and 11.3 / 9.7 after 100 steps (two-item cells).  One
// 64 x 64 box, whole step: 140 us / 60 us.
#pragma once

#include "sim_tiled.cuh"

namespace dbm {

// Offset stored for an empty cell: every displacement from it is ~1e4 cells, far outside R.
constexpr float kEmptyOff = 1.0e4f;
// Second items of a tile's region (cells holding two items): at most this many per tile.  A cell
// with three or more items, or more two-item cells than this, sends the tile to the fallback.
constexpr int kOvf = 32;

// D2Q9 direction of (c_x, c_y), and the displacements the NEAR kernels are compiled for (the host
// takes them only when the lattice's cd_k are these).
__host__ __device__ constexpr int d2q9_dir(int cx, int cy) {
  constexpr int k[9] = {7, 4, 8, 3, 0, 1, 6, 2, 5};
  return k[3 * (cy + 1) + cx + 1];
}
__host__ __device__ constexpr int d2q9_cx(int k) { return (k == 1 || k == 5 || k == 8) - (k == 3 || k == 6 || k == 7); }
__host__ __device__ constexpr int d2q9_cy(int k) { return (k == 2 || k == 5 || k == 6) - (k == 4 || k == 7 || k == 8); }

// Shared memory of a staged region of rw x rh cells: per cell one float2 (the offsets), NP float2
// planes and NF float planes, a signed char (the overflow slot of its second item, -1: none), the
// same for the kOvf overflow items, their region coordinates and the overflow counter.  Rows are
// padded to 16 float2 (32 floats): lanes of consecutive cells then meet in a bank only when two of
// them read the same column of different rows.
template <int RW, int RH, int NP, int NF>
struct DenseLayout {
  static constexpr int rw = RW, rh = RH;
  static constexpr int s2 = (RW + 15) & ~15, s1 = (RW + 31) & ~31;  // row strides of the float2 and float planes
  static constexpr int n2 = s2 * RH, n1 = s1 * RH;                  // elements of one plane
  static constexpr int kv = n2 * 8, fl = kv + NP * n2 * 8, nx = fl + NF * n1 * 4, oxy = nx + ((n2 + 15) & ~15),
                       okv = oxy + kOvf * 8, ofl = okv + NP * kOvf * 8, ocell = ofl + NF * kOvf * 4,
                       cnt = ocell + kOvf * 4, total = cnt + 16;
};
// The same with the region known at run time.
struct DenseLayoutRt {
  int rw, rh, s2, s1, n2, n1;
  int kv, fl, nx, oxy, okv, ofl, ocell, cnt, total;
  __host__ __device__ DenseLayoutRt(int w, int h, int np, int nf) : rw(w), rh(h) {
    s2 = (w + 15) & ~15;
    s1 = (w + 31) & ~31;
    n2 = s2 * h;
    n1 = s1 * h;
    kv = n2 * 8;
    fl = kv + np * n2 * 8;
    nx = fl + nf * n1 * 4;
    oxy = nx + ((n2 + 15) & ~15);
    okv = oxy + kOvf * 8;
    ofl = okv + np * kOvf * 8;
    ocell = ofl + nf * kOvf * 4;
    cnt = ocell + kOvf * 4;
    total = cnt + 16;
  }
};
// planes: thin + refine exp(f*) (Q floats), weights none, gather rho (1 float) and (1/sw, f*) (Q pairs)
constexpr int ds_pairs(int Q, int stage) { return stage == 2 ? Q : 0; }
constexpr int ds_floats(int Q, int stage) { return stage == 0 ? Q : stage == 2 ? 1 : 0; }
// TX > 0: the NEAR kernels' tile of TX x (256 / TX) cells with 3 cells of halo on each side.
template <int Q, int STAGE, int TX>
struct DenseLayoutOf {
  using type = DenseLayout<TX + 6, 256 / TX + 6, ds_pairs(Q, STAGE), ds_floats(Q, STAGE)>;
  static __device__ __forceinline__ type make(const TileGeo&) { return {}; }
};
template <int Q, int STAGE>
struct DenseLayoutOf<Q, STAGE, 0> {
  using type = DenseLayoutRt;
  static __host__ __device__ __forceinline__ type make(const TileGeo& G) {
    const Halo& h = STAGE == 1 ? G.cp : G.mom;
    return type(G.tx + h.xh - h.xl, G.ty + h.yh - h.yl, ds_pairs(Q, STAGE), ds_floats(Q, STAGE));
  }
};

template <class LT>
struct DenseSmem {
  LT L;
  unsigned char* p;
  template <class T>
  __device__ __forceinline__ T* at(int o) const { return reinterpret_cast<T*>(p + o); }
  __device__ __forceinline__ float2* xy() const { return at<float2>(0); }       // [n2] offsets of the cells' first items
  __device__ __forceinline__ float2* kv() const { return at<float2>(L.kv); }    // [np][n2]
  __device__ __forceinline__ float* fl() const { return at<float>(L.fl); }      // [nf][n1]
  __device__ __forceinline__ signed char* nx() const { return at<signed char>(L.nx); }  // [n2] overflow slot, -1: none
  __device__ __forceinline__ float2* oxy() const { return at<float2>(L.oxy); }  // [kOvf]
  __device__ __forceinline__ float2* okv() const { return at<float2>(L.okv); }  // [np][kOvf]
  __device__ __forceinline__ float* ofl() const { return at<float>(L.ofl); }    // [nf][kOvf]
  // [kOvf] region row << 16 | region column of each overflow item's cell
  __device__ __forceinline__ int* ocell() const { return at<int>(L.ocell); }
  // overflow counter, smallest x and y offset of the region (float bits)
  __device__ __forceinline__ int* novf() const { return at<int>(L.cnt); }
};

// Window positions (b * ncol + a, a < ncol columns, b < nrow rows from region cell (row0, col0))
// whose cell holds a second item, from the tile's overflow list: no per-position test in the
// stencil, and nothing to do in a tile without two-item cells.
template <class SM>
__device__ __forceinline__ uint64_t second_item_mask(const SM& S, int no, int row0, int col0, int nrow,
                                                     int ncol) {
  uint64_t ov = 0;
#pragma unroll 1
  for (int q = 0; q < no; ++q) {
    const int rc = S.ocell()[q];
    const int b = (rc >> 16) - row0, a = (rc & 0xffff) - col0;
    if ((unsigned)b < (unsigned)nrow && (unsigned)a < (unsigned)ncol) ov |= 1ull << (b * ncol + a);
  }
  return ov;
}

// Item range of global cell g: at most two items, else *many is set.
__device__ __forceinline__ void cell_items(const uint32_t* __restrict__ start, uint32_t g, int* b, int* e, int* many) {
  const uint32_t b0 = start[g], e0 = start[g + 1];
  if (e0 - b0 > 2u) {
    *many = 1;
    *b = *e = (int)b0;
  } else {
    *b = (int)b0;
    *e = (int)e0;
  }
}

// Clears a tile's counters; ends with a barrier.
template <class SM>
__device__ __forceinline__ void stage_begin(const SM& S, int* own_counters) {
  if (threadIdx.x == 0) {
    S.novf()[0] = 0;
    S.novf()[1] = S.novf()[2] = 0x7f800000;
    if (own_counters) own_counters[0] = own_counters[1] = own_counters[2] = 0;
  }
  __syncthreads();
}

// Dense staging of region cells [xr0, xr0 + rw) x [yr0, yr0 + rh) of a state (sorted ranges `start`,
// offsets off[stride]): put(item, offsets, float2 planes, stride, slot, float planes, stride, slot)
// fills the planes of one item and returns nonzero if the item cannot be served here; the offsets
// of an empty cell get the empty offset and its other planes 0 (NF, NP: those read whether or not a
// candidate hits).  A cell's second item goes to the next overflow slot.  novf[1], novf[2] end as the
// smallest offsets of the region (the bits of a float >= 0 order as integers).  Returns false, the
// same in every thread, when the tile must be deferred (`many` from the caller, a cell with three or
// more items, a full overflow list, or an item refused by `put`).
template <int NF, int NP, class SM, class Put>
__device__ __forceinline__ bool stage_dense(const InstK& I, int xr0, int yr0, const uint32_t* __restrict__ start,
                                            const float* __restrict__ off, int64_t stride, const SM& S, int many,
                                            Put&& put) {
  const int rw = S.L.rw, cells = rw * S.L.rh;
  int minx = 0x7f800000, miny = 0x7f800000;
  auto offsets = [&](int m) {
    const float2 o = make_float2(off[m], off[stride + m]);
    minx = min(minx, __float_as_int(o.x));
    miny = min(miny, __float_as_int(o.y));
    return o;
  };
  for (int ci = threadIdx.x; ci < cells; ci += blockDim.x) {
    const int ry = ci / rw, rx = ci - ry * rw;
    const int i2 = ry * S.L.s2 + rx, i1 = ry * S.L.s1 + rx;
    uint32_t g;
    int b = 0, e = 0;
    if (region_cell(I, xr0 + rx, yr0 + ry, &g)) cell_items(start, g, &b, &e, &many);
    int nxt = -1;
    if (e - b == 2) {
      const int q = atomicAdd(S.novf(), 1);
      if (q < kOvf) {
        const float2 o = offsets(b + 1);
        S.oxy()[q] = o;
        many |= put(b + 1, o, S.okv(), kOvf, q, S.ofl(), kOvf, q);
        S.ocell()[q] = (ry << 16) | rx;
        nxt = q;
      } else {
        many = 1;
      }
    }
    S.nx()[i2] = (signed char)nxt;
    if (e > b) {
      const float2 o = offsets(b);
      S.xy()[i2] = o;
      many |= put(b, o, S.kv(), S.L.n2, i2, S.fl(), S.L.n1, i1);
    } else {
      S.xy()[i2] = make_float2(kEmptyOff, kEmptyOff);
#pragma unroll
      for (int k = 0; k < NF; ++k) S.fl()[k * S.L.n1 + i1] = 0.f;
#pragma unroll
      for (int k = 0; k < NP; ++k) S.kv()[k * S.L.n2 + i2] = make_float2(0.f, 0.f);
    }
  }
  minx = __reduce_min_sync(0xffffffffu, minx);
  miny = __reduce_min_sync(0xffffffffu, miny);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(S.novf() + 1, minx);
    atomicMin(S.novf() + 2, miny);
  }
  return !__syncthreads_or(many);
}

// The tile's reference points beyond one per cell.  The second items of two-item cells are offered to
// the threads whose own cell is empty (or outside the box): over a run about as many cells hold two
// items as none, so most tiles finish in one pass.  What is left, and points whose window does not
// fit the 4 x 4 block, runs as (item, direction) units spread over the block after the pass, so such
// a point adds one direction's work to nine threads instead of nine directions to one thread (whose
// warp, and with it the block, would wait for it).  Each sum is its own: no result changes.
struct OwnList {
  int n, taken, wide;  // second items, those offered and taken, window exceptions
  int item[512];       // second items from the front, window exceptions from the back
  int pos[512];        // region row << 16 | region column of the item's cell
  __device__ __forceinline__ void put(int q, int it, int bx, int by) {
    item[q] = it;
    pos[q] = (by << 16) | bx;
  }
  // at most one of each per thread: neither part exceeds 256 entries
  __device__ __forceinline__ void push_second(int it, int bx, int by) { put(atomicAdd(&n, 1), it, bx, by); }
  __device__ __forceinline__ void push_wide(int it, int bx, int by) { put(511 - atomicAdd(&wide, 1), it, bx, by); }
  __device__ __forceinline__ bool take(int* it, int* bx, int* by) {
    if (n == 0) return false;
    const int q = atomicAdd(&taken, 1);
    if (q >= n) return false;
    *it = item[q];
    *bx = pos[q] & 0xffff;
    *by = pos[q] >> 16;
    return true;
  }
  // after a barrier: the items left, and the list index of the e-th
  __device__ __forceinline__ int left() const { return n - min(taken, n) + wide; }
  __device__ __forceinline__ int index(int e) const {
    const int s = n - min(taken, n);
    return e < s ? n - s + e : 511 - (e - s);
  }
};

// Stencil origin and width along one axis for reference offset p: j in [lo, lo + n).
__device__ __forceinline__ void stencil_axis(float p, float R, float tiny, int* lo, int* n) {
  *lo = (int)floorf(p - R - tiny);
  *n = (int)floorf(p + R + tiny) - *lo + 1;
}
// Columns that a window's exact range can have: at most 3 up to R = 1, 4 up to 1.5, 5 up to 2 (less the
// margins).  fn(integral constant) of that many.  Boxes with other displacements than one cell, or R < 1, take
// each window by its exact range with them, a thread per point: as units of (point, direction) spread over the
// block their sums left in scattered writes.  1024 x 1024 cells, one moment each, us a step, branching 4 x 4
// stencil / units / now: dx 1, r 0.9 498 / 619 / 448; dx 1, r 0.7 477 / 621 / 447; dx 2, r 1.9 990 / 988 / 804.
template <class Fn>
__device__ __forceinline__ void with_columns(float R, float tiny, Fn&& fn) {
  const float w = 2.f * (R + tiny) + 1e-4f;
  if (w <= 2.f) fn(std::integral_constant<int, 3>{});
  else if (w <= 3.f) fn(std::integral_constant<int, 4>{});
  else fn(std::integral_constant<int, 5>{});
}

// Whether the 4 columns from `lo` hold every hit along one axis: the range is no wider, or it is five
// wide (p within tiny of 1/2 at R = 1.5) and the fifth column's candidates, none of them nearer than
// e5, all miss (rounding is monotone, so the smallest offset gives the smallest |e|).
__device__ __forceinline__ bool block_fits(int n, float e5, float R2) {
  return n <= 4 || (n == 5 && rn_mul(e5, e5) > R2);
}

// -d and max(R - d, 0) for the correctly rounded d = sqrt(d2), given nd2 = -d2.  One Newton step in
// Markstein's form (P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990): with y ~ 1/sqrt(d2), g = d2 y and h = y / 2,
// d = fma(fma(-g, g, d2), h, g); carried negated, so no operand needs a sign change.  Equal to
// __fsqrt_rn for every float in [1e-30, 2e8] (all of them compared).  Zero has no reciprocal root, so
// the callers add kTinyD2 to d2's y part: it changes no sum above 1e-22, and below that d is under
// 1e-11 and R - d is R either way.  d2 = NaN or infinity gives the weight 0 (fmaxf drops the NaN), as
// a miss.  Six instructions against about twelve of __fsqrt_rn, and no branch for special values.
constexpr float kTinyD2 = 1e-30f;
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float window_weight(float nd2, float R) {
  const float y = rsqrt_ftz(-nd2);
  const float gn = __fmul_rn(nd2, y), h = __fmul_rn(y, 0.5f);
  const float nd = __fmaf_rn(__fmaf_rn(gn, gn, nd2), h, gn);
  return fmaxf(__fadd_rn(R, nd), 0.f);
}

// The same for two candidates at once with the paired FP32 operations (each half rounds as the scalar).
__device__ __forceinline__ float2 window_weight2(float2 nd2, float R) {
  const float2 y = make_float2(rsqrt_ftz(-nd2.x), rsqrt_ftz(-nd2.y));
  const float2 gn = __fmul2_rn(nd2, y), h = __fmul2_rn(y, make_float2(0.5f, 0.5f));
  const float2 nd = __ffma2_rn(__ffma2_rn(gn, gn, nd2), h, gn);
  const float2 w = __fadd2_rn(make_float2(R, R), nd);
  return make_float2(fmaxf(w.x, 0.f), fmaxf(w.y, 0.f));
}

// Exact running sum of window weights (R in [1, 2), at most 64 terms).  Every weight rn(R - d) is a
// multiple of 2^-24: for d >= 1/2 so are R and d, and for d < 1/2 the weight exceeds 1/2.  `hi`
// starts at 384 and stays in [256, 512), so it moves in steps of 2^-15, each rounding error is a
// multiple of 2^-24 below 2^-15 and is recovered exactly by one FastTwoSum (|hi| >= w always), and
// their sum in `lo` is exact as well.  value() rounds the exact sum once: the bits of CSum's
// hi + lo, whose parts are exact here too, in four operations per term instead of seven.
struct WeightSum {
  float hi, lo;
  __device__ __forceinline__ void clear() { hi = 384.f, lo = 0.f; }
  __device__ __forceinline__ void add(float w) {
    const float t = __fadd_rn(hi, w);
    lo = __fadd_rn(lo, __fsub_rn(w, __fsub_rn(t, hi)));
    hi = t;
  }
  __device__ __forceinline__ float value() const { return __fadd_rn(__fsub_rn(hi, 384.f), lo); }
};
// Two of them (two directions) at once.
struct WeightSum2 {
  float2 hi, lo;
  __device__ __forceinline__ void clear() { hi = make_float2(384.f, 384.f), lo = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void add(float2 w) {
    const float2 m1 = make_float2(-1.f, -1.f);  // a - b as fma(b, -1, a): one rounding, the same bits
    const float2 t = __fadd2_rn(hi, w);
    lo = __fadd2_rn(lo, __ffma2_rn(__ffma2_rn(hi, m1, t), m1, w));
    hi = t;
  }
  __device__ __forceinline__ float x() const { return __fadd_rn(__fsub_rn(hi.x, 384.f), lo.x); }
  __device__ __forceinline__ float y() const { return __fadd_rn(__fsub_rn(hi.y, 384.f), lo.y); }
};

// ---- thinning + refine --------------------------------------------------------------------------
// Float planes: exp(f*_k) of each item.

// The refined control point of cell F: the move for kappa > kappa_hard, its cell and offsets.
template <int Q>
__device__ __forceinline__ void refine_store(const Args<Q, 2, PF32>& A, const InstK& I, uint32_t F, int Fx, int Fy,
                                             uint32_t cnt, uint32_t mask, const float (&cen)[2], float swf, float2 sx) {
  const int kappa = __popc(mask);
  float np[2];
  if (kappa <= A.kappa_hard) {
    np[0] = cen[0];
    np[1] = cen[1];
  } else {
    np[0] = cen[0] + sx.x / swf;
    np[1] = cen[1] + sx.y / swf;
  }
  bool finite = true;
#pragma unroll
  for (int a = 0; a < 2; ++a) finite &= isfinite(np[a]) && fabsf(np[a]) < 64.f;
  if (!finite) {
    atomicOr(A.status, ST_NONFINITE);
    np[0] = cen[0];
    np[1] = cen[1];
  }
  int sh[2];
  float off[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const float fl = floorf(np[a]);
    sh[a] = (int)fl;
    off[a] = np[a] - fl;
    if (off[a] >= 1.f) {
      off[a] = 0.f;
      sh[a] += 1;
    }
  }
  uint32_t Gc;
  const bool inside = cell_at<2>(I, Fx + sh[0], Fy + sh[1], 0, &Gc);
  if (!inside) atomicOr(A.status, ST_OUT_OF_BOX);
  A.occ[F] = inside ? 1u : 0u;
  A.fkey[F] = inside ? Gc : 0xffffffffu;
  A.foff[F] = off[0];
  A.foff[(int64_t)A.ncells + F] = off[1];
  if (A.write_trace) {
    A.tcnt[F] = cnt;
    A.mask[F] = mask;
    A.cen[F] = cen[0];
    A.cen[(int64_t)A.ncells + F] = cen[1];
  }
}

template <int Q, int TX>
__device__ __forceinline__ bool thin_refine_ds_tile(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                                    const TileGeo& G, unsigned char* smem) {
  using Lay = DenseLayoutOf<Q, 0, TX>;
  const DenseSmem<typename Lay::type> S{Lay::make(G), smem};
  const int s2 = S.L.s2, s1 = S.L.s1;
  __shared__ int s_edge;  // some offset of the region rounds up to the next cell when a cell is added
  if (threadIdx.x == 0) s_edge = 0;
  stage_begin(S, nullptr);
  const bool dense = stage_dense<0, 0>(I, T.x0 + G.mom.xl, T.y0 + G.mom.yl, A.a.start, A.a.off, A.mcap, S, 0,
                                       [&](int m, float2 o, float2*, int, int, float* w, int stride, int slot) {
                                         if (fmaxf(o.x, o.y) > 0.9999999f) s_edge = 1;
#pragma unroll
                                         for (int k = 0; k < Q; ++k)
                                           w[k * stride + slot] = exp(fstar_at<Q, 2, PF32>(A, (uint32_t)m, k));
                                         return (int)!(o.x + o.y < 4.f);  // NaN: 0 x it is not 0
                                       });
  if (!dense) return false;
  const int no = *S.novf();  // second items in the overflow list (at most kOvf in a dense tile)
  const bool edge = s_edge != 0;

  const int lx = threadIdx.x % (TX ? TX : G.tx), ly = threadIdx.x / (TX ? TX : G.tx);
  const int Fx = T.x0 + lx, Fy = T.y0 + ly;
  if (ly >= G.ty || Fx >= I.dims[0] || Fy >= I.dims[1]) return true;
  const uint32_t F = I.base + (uint32_t)Fx + (uint32_t)I.dims[0] * (uint32_t)Fy;
  const int bx = lx - (TX ? -3 : G.mom.xl), by = ly - (TX ? -3 : G.mom.yl);  // region coordinates of F

  // thinning: component (m, k) lands in F iff floor(off + cd) == -so on both axes
  uint32_t cnt = 0;
  CSum csum[2];
  if (TX && !edge) {
    // displacements of one cell: direction k's components come from cell (-c_x, -c_y) and all of them
    // land (an offset of 1 - 2^-24, which rn(off + 1) carries into the next cell, takes the loops below)
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float cdx = (float)d2q9_cx(k), cdy = (float)d2q9_cy(k);
      const int ci = (by - d2q9_cy(k)) * s2 + (bx - d2q9_cx(k));
      auto land = [&](float2 o) {
        ++cnt;
        csum[0].add(rn_sub(rn_add(o.x, cdx), cdx));
        csum[1].add(rn_sub(rn_add(o.y, cdy), cdy));
      };
      const float2 o = S.xy()[ci];
      if (o.x < 2.f) land(o);  // not the empty offset
      if (no && S.nx()[ci] >= 0) land(S.oxy()[S.nx()[ci]]);
    }
  } else {
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
        const int ci = (by + soy) * s2 + (bx + sox);
        land(S.xy()[ci]);
        if (no && S.nx()[ci] >= 0) land(S.oxy()[S.nx()[ci]]);
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

  // refine: the centroid's stencil, shifted by -cd_k per direction.  The weighted sums run through
  // the directions in order, so each candidate's turn is fixed and its offsets are read again for
  // each direction (holding the 6 x 6 of them in registers left two blocks per SM and was slower).
  int jlx, nxs, jly, nys;
  stencil_axis(cen[0], A.R, A.tiny, &jlx, &nxs);
  stencil_axis(cen[1], A.R, A.tiny, &jly, &nys);
  const bool fits = TX &&
                    block_fits(nxs, rn_add(__int_as_float(S.novf()[1]), rn_sub((float)(jlx + 4), cen[0])), A.R2) &&
                    block_fits(nys, rn_add(__int_as_float(S.novf()[2]), rn_sub((float)(jly + 4), cen[1])), A.R2);
  uint32_t mask = 0;
  float swf = 0.f;
  float2 sx = make_float2(0.f, 0.f);
  // one candidate with weight *wp; dmin ends at or below R2 when any candidate of the direction hit
  auto one = [&](float2 o, const float* wp, float ex0, float ey0, float& dmin) {
    const float2 e = __fadd2_rn(o, make_float2(ex0, ey0));
    const float2 e2 = __fmul2_rn(e, e);
    const float d2 = rn_add(e2.x, e2.y);
    dmin = fminf(dmin, d2);
    float wt = 0.f;  // a miss adds nothing
    if (d2 <= A.R2) wt = *wp;
    swf = __fadd_rn(swf, wt);
    sx.x = __fmaf_rn(wt, e.x, sx.x);
    sx.y = __fmaf_rn(wt, e.y, sx.y);
  };
  // the second items of direction k's window, in window order
  auto seconds = [&](int k, int cdx, int cdy, int nrow, int ncol, float& dmin) {
    uint64_t ov = second_item_mask(S, no, by + jly - cdy, bx + jlx - cdx, nrow, ncol);
#pragma unroll 1
    while (ov) {
      const int pos = __ffsll(ov) - 1;
      ov &= ov - 1;
      const int b = pos / ncol, a = pos - b * ncol;
      const int q = S.nx()[(by + jly - cdy + b) * s2 + bx + jlx - cdx + a];
      one(S.oxy()[q], S.ofl() + k * kOvf + q, rn_sub((float)(jlx + a), cen[0]), rn_sub((float)(jly + b), cen[1]), dmin);
    }
  };
  if constexpr (TX > 0) {
    if (fits) {
      float cx[4], cy[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        cx[a] = rn_sub((float)(jlx + a), cen[0]);
        cy[a] = rn_sub((float)(jly + a), cen[1]);
      }
#pragma unroll 1
      for (int k = 0; k < 9; ++k) {
        const int cdx = __float2int_rn(A.L.cdf[k][0]), cdy = __float2int_rn(A.L.cdf[k][1]);
        const float2* o0 = S.xy() + (by + jly - cdy) * s2 + (bx + jlx - cdx);
        const float* w0 = S.fl() + k * S.L.n1 + (by + jly - cdy) * s1 + (bx + jlx - cdx);
        float dmin = 3.0e38f;
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
          for (int a = 0; a < 4; ++a) one(o0[b * s2 + a], w0 + b * s1 + a, cx[a], cy[b], dmin);
        if (no) seconds(k, cdx, cdy, 4, 4, dmin);
        if (dmin <= A.R2) mask |= 1u << k;
      }
    }
  }
  if (TX == 0 || (!fits && A.R > 1.55f)) {
    with_columns(A.R, A.tiny, [&](auto nc) {
      constexpr int NC = nc.value;
      float cx[NC];
#pragma unroll
      for (int a = 0; a < NC; ++a) cx[a] = rn_sub((float)(jlx + a), cen[0]);
#pragma unroll 1
      for (int k = 0; k < Q; ++k) {
        const int cdx = __float2int_rn(A.L.cdf[k][0]), cdy = __float2int_rn(A.L.cdf[k][1]);
        const float2* o0 = S.xy() + (by + jly - cdy) * s2 + (bx + jlx - cdx);
        const float* w0 = S.fl() + k * S.L.n1 + (by + jly - cdy) * s1 + (bx + jlx - cdx);
        float dmin = 3.0e38f;
#pragma unroll 1
        for (int b = 0; b < nys; ++b, o0 += s2, w0 += s1) {
          const float cyb = rn_sub((float)(jly + b), cen[1]);
          float2 o[NC];
#pragma unroll
          for (int a = 0; a < NC; ++a) o[a] = a < nxs ? o0[a] : make_float2(kEmptyOff, kEmptyOff);
#pragma unroll
          for (int a = 0; a < NC; ++a) one(o[a], w0 + a, cx[a], cyb, dmin);
        }
        if (no) seconds(k, cdx, cdy, nys, nxs, dmin);
        if (dmin <= A.R2) mask |= 1u << k;
      }
    });
  } else if (!fits) {  // few points, and rows unrolled here would slow the others (R = 1.5: 118 -> 130 us)
#pragma unroll 1
    for (int k = 0; k < Q; ++k) {
      const int cdx = __float2int_rn(A.L.cdf[k][0]), cdy = __float2int_rn(A.L.cdf[k][1]);
      const int row0 = by + jly - cdy, col0 = bx + jlx - cdx;
      float dmin = 3.0e38f;
#pragma unroll 1
      for (int b = 0; b < nys; ++b) {
        const float cyb = rn_sub((float)(jly + b), cen[1]);
#pragma unroll 1
        for (int a = 0; a < nxs; ++a)
          one(S.xy()[(row0 + b) * s2 + col0 + a], S.fl() + k * S.L.n1 + (row0 + b) * s1 + col0 + a,
              rn_sub((float)(jlx + a), cen[0]), cyb, dmin);
      }
      if (no) seconds(k, cdx, cdy, nys, nxs, dmin);
      if (dmin <= A.R2) mask |= 1u << k;
    }
  }
  refine_store<Q>(A, I, F, Fx, Fy, cnt, mask, cen, swf, sx);
  return true;
}

// ---- weights: per component, 1 / (sum over control points within R of (R - d)) -----------------

// One component: direction k of a moment at offset o in region cell (bx, by); NC: with_columns.
template <int Q, int NC, class SM>
__device__ __forceinline__ void weights_ds_unit(const Args<Q, 2, PF32>& A, const SM& S, int no, int m, int k,
                                                int bx, int by) {
  const float2 o = make_float2(A.a.off[m], A.a.off[A.mcap + m]);
  // control-point offsets u (relative to the component's cell) with a possible hit
  int ulx, nxs, uly, nys;
  stencil_axis(o.x, A.R, A.tiny, &ulx, &nxs);
  stencil_axis(o.y, A.R, A.tiny, &uly, &nys);
  const int cdx = __float2int_rn(A.L.cdf[k][0]), cdy = __float2int_rn(A.L.cdf[k][1]);
  const int row0 = by + uly + cdy, col0 = bx + ulx + cdx;
  CSum sws;
  // branch-free, a row at a time: a miss adds the weight 0
  auto one = [&](float2 pc, float basex, float basey) {
    const float2 q = __fadd2_rn(make_float2(basex, basey), make_float2(-pc.x, -pc.y));
    const float2 e = __fadd2_rn(o, q);
    const float2 e2 = __fmul2_rn(e, e);
    sws.add(window_weight(-rn_add(e2.x, rn_add(e2.y, kTinyD2)), A.R));
  };
#pragma unroll 1
  for (int b = 0; b < nys; ++b) {
    const float2* row = S.xy() + (row0 + b) * S.L.s2 + col0;
    float2 pc[NC];
#pragma unroll
    for (int a = 0; a < NC; ++a) pc[a] = a < nxs ? row[a] : make_float2(kEmptyOff, kEmptyOff);
#pragma unroll
    for (int a = 0; a < NC; ++a) one(pc[a], (float)(-(ulx + a)), (float)(-(uly + b)));
  }
  // then the second items, in window order
  uint64_t ov = no ? second_item_mask(S, no, row0, col0, nys, nxs) : 0u;
#pragma unroll 1
  while (ov) {
    const int pos = __ffsll(ov) - 1;
    ov &= ov - 1;
    const int b = pos / nxs, a = pos - b * nxs;
    one(S.oxy()[S.nx()[(row0 + b) * S.L.s2 + col0 + a]], (float)(-(ulx + a)), (float)(-(uly + b)));
  }
  const float sw = sws.value();
  A.sw[(int64_t)k * A.mcap + m] = sw > 0.f ? 1.f / sw : 0.f;
}

template <int Q, int TX, bool SPLIT>
__device__ __forceinline__ bool weights_ds_tile(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                                const TileGeo& G, unsigned char* smem) {
  using Lay = DenseLayoutOf<Q, 1, TX>;
  const DenseSmem<typename Lay::type> S{Lay::make(G), smem};
  __shared__ OwnList own;
  stage_begin(S, &own.n);
  // the tile's own moments (at most two per cell)
  const int lx = threadIdx.x % (TX ? TX : G.tx), ly = threadIdx.x / (TX ? TX : G.tx);
  const int Sx = T.x0 + lx, Sy = T.y0 + ly;
  int bx = lx - (TX ? -3 : G.cp.xl), by = ly - (TX ? -3 : G.cp.yl);  // region coordinates of the moment's cell
  int m = 0, m1 = 0, many = 0;
  if (ly < G.ty && Sx < I.dims[0] && Sy < I.dims[1])
    cell_items(A.a.start, I.base + (uint32_t)Sx + (uint32_t)I.dims[0] * (uint32_t)Sy, &m, &m1, &many);
  bool has = m1 > m;
  if (m1 - m == 2) own.push_second(m + 1, bx, by);
  const bool dense = stage_dense<0, 0>(I, T.x0 + G.cp.xl, T.y0 + G.cp.yl, A.b.start, A.b.off, A.ccap, S, many,
                                       [&](int, float2, float2*, int, int, float*, int, int) { return 0; });
  if (!dense) return false;
  const int no = *S.novf();  // second items in the overflow list (at most kOvf in a dense tile)
  if (!has) has = own.take(&m, &bx, &by);
  if constexpr (TX == 0) {  // each thread its point's directions, windows by their exact ranges
    with_columns(A.R, A.tiny, [&](auto nc) {
#pragma unroll 1
      for (; has; has = own.take(&m, &bx, &by))
#pragma unroll 1
        for (int k = 0; k < Q; ++k) weights_ds_unit<Q, nc.value>(A, S, no, m, k, bx, by);
    });
    return true;
  }
  if (has) {
    bool fits = false;
    if constexpr (TX > 0) {
      const float2 o = make_float2(A.a.off[m], A.a.off[A.mcap + m]);
      int ulx, uly, nxs, nys;
      stencil_axis(o.x, A.R, A.tiny, &ulx, &nxs);
      stencil_axis(o.y, A.R, A.tiny, &uly, &nys);
      fits = block_fits(nxs, rn_add(o.x, rn_sub((float)(-(ulx + 4)), __int_as_float(S.novf()[1]))), A.R2) &&
             block_fits(nys, rn_add(o.y, rn_sub((float)(-(uly + 4)), __int_as_float(S.novf()[2]))), A.R2);
      if (fits) {
        float bxv[4];  // float(-u) of the stencil columns
#pragma unroll
        for (int a = 0; a < 4; ++a) bxv[a] = (float)(-(ulx + a));
#pragma unroll 1
        for (int cy = SPLIT ? (int)blockIdx.y - 1 : -1; cy <= (SPLIT ? (int)blockIdx.y - 1 : 1); ++cy) {
          // the three directions (c_x, c_y), c_x = d - 1: control-point rows uly + c_y + b, and the
          // component's column a is column a + d of the six from ulx - 1
          WeightSum2 s01;
          WeightSum s2;
          s01.clear();
          s2.clear();
          const float2* row = S.xy() + (by + uly + cy) * S.L.s2 + (bx + ulx - 1);
#pragma unroll 2
          for (int b = 0; b < 4; ++b, row += S.L.s2) {
            const float basey = (float)(-(uly + b));
            float2 pc[6];
            float ey2[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) {
              pc[c] = row[c];
              const float ey = rn_add(o.y, rn_sub(basey, pc[c].y));
              ey2[c] = rn_add(rn_mul(ey, ey), kTinyD2);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
              float nd[3];
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                const float ex = rn_add(o.x, rn_sub(bxv[a], pc[a + d].x));
                nd[d] = -rn_add(rn_mul(ex, ex), ey2[a + d]);
              }
              s01.add(window_weight2(make_float2(nd[0], nd[1]), A.R));
              s2.add(window_weight(nd[2], A.R));
            }
          }
          // second items of the 4 x 6 cells: a miss adds nothing, and the sums are exact, so their
          // order does not matter
#pragma unroll 1
          for (int q = 0; q < no; ++q) {
            const int rc = S.ocell()[q];
            const int ur = (rc >> 16) - by - cy, uc = (rc & 0xffff) - bx;  // row relative to the component's
            if ((unsigned)(ur - uly) >= 4u || (unsigned)(uc - (ulx - 1)) >= 6u) continue;
            const float2 pc = S.oxy()[q];
            const float ey = rn_add(o.y, rn_sub((float)(-ur), pc.y));
            const float ey2 = rn_add(rn_mul(ey, ey), kTinyD2);
            float nd[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const float ex = rn_add(o.x, rn_sub((float)(d - 1 - uc), pc.x));
              nd[d] = -rn_add(rn_mul(ex, ex), ey2);
            }
            s01.add(window_weight2(make_float2(nd[0], nd[1]), A.R));
            s2.add(window_weight(nd[2], A.R));
          }
          const float sw[3] = {s01.x(), s01.y(), s2.value()};
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int k = cy < 0 ? d2q9_dir(d - 1, -1) : cy == 0 ? d2q9_dir(d - 1, 0) : d2q9_dir(d - 1, 1);
            A.sw[(int64_t)k * A.mcap + m] = sw[d] > 0.f ? 1.f / sw[d] : 0.f;
          }
        }
      }
    }
    if (!fits) own.push_wide(m, bx, by);
  }
  __syncthreads();
  const int left = own.left();
#pragma unroll 1
  for (int u = threadIdx.x; u < left * Q; u += blockDim.x) {
    const int k = u / left, q = own.index(u - k * left);
    if (SPLIT && d2q9_cy(k) != (int)blockIdx.y - 1) continue;
    weights_ds_unit<Q, 5>(A, S, no, own.item[q], k, own.pos[q] & 0xffff, own.pos[q] >> 16);
  }
  return true;
}

// ---- gather: per control point and direction ------------------------------------------------------
// Float plane: rho; float2 planes: (1/sw, f*_k).

// Sums of one (control point, direction): rho part compensated, deviation part plain FMA.
struct GatherSum {
  float hi, lo, sb;
  __device__ __forceinline__ void clear() { hi = lo = sb = 0.f; }
  // wgt >= 0 and rho >= 0 (with another density the step takes no dense tile), so hi >= 0 and the larger of
  // (hi, p) leads the FastTwoSum: the exact rounding error, as CSum's TwoSum gives it
  __device__ __forceinline__ void add(float wgt, float rho, float f) {
    const float p = __fmul_rn(wgt, rho);
    const float err = __fmaf_rn(wgt, rho, -p);
    const float a = fmaxf(hi, p), b = fminf(hi, p);
    const float t = __fadd_rn(a, b);
    lo = __fadd_rn(lo, __fsub_rn(b, __fsub_rn(t, a)));
    lo = __fadd_rn(lo, err);
    hi = t;
    sb = __fmaf_rn(wgt, f, sb);
  }
};

__device__ __forceinline__ DF gather_total(float wf, float wlo, float hi, float lo, float sb) {
  return df_add(df_mul(DF{wf, wlo}, df_norm(hi, lo)), DF{sb, 0.f});
}

// One (control point, direction): control point at offset pp in region cell (bx, by); NC: with_columns.
template <int Q, int NC, class SM>
__device__ __forceinline__ DF gather_ds_unit(const Args<Q, 2, PF32>& A, const SM& S, int no, float2 pp, int k,
                                             int bx, int by) {
  int jlx, nxs, jly, nys;
  stencil_axis(pp.x, A.R, A.tiny, &jlx, &nxs);
  stencil_axis(pp.y, A.R, A.tiny, &jly, &nys);
  const int cdx = __float2int_rn(A.L.cdf[k][0]), cdy = __float2int_rn(A.L.cdf[k][1]);
  const int row0 = by + jly - cdy, col0 = bx + jlx - cdx;
  GatherSum s;
  s.clear();
  // branch-free, a row at a time: a miss gets the weight 0
  auto one = [&](float2 o, float rho, float2 kv, float ex0, float ey0) {
    const float2 e = __fadd2_rn(o, make_float2(ex0, ey0));
    const float2 e2 = __fmul2_rn(e, e);
    s.add(__fmul_rn(window_weight(-rn_add(e2.x, rn_add(e2.y, kTinyD2)), A.R), kv.x), rho, kv.y);
  };
#pragma unroll 1
  for (int b = 0; b < nys; ++b) {
    const float cyb = rn_sub((float)(jly + b), pp.y);
    const int i2 = (row0 + b) * S.L.s2 + col0, i1 = (row0 + b) * S.L.s1 + col0;
    float2 o[NC], kv[NC];
    float rho[NC];
#pragma unroll
    for (int a = 0; a < NC; ++a) {
      const bool in = a < nxs;
      o[a] = in ? S.xy()[i2 + a] : make_float2(kEmptyOff, kEmptyOff);
      kv[a] = in ? S.kv()[k * S.L.n2 + i2 + a] : make_float2(0.f, 0.f);
      rho[a] = in ? S.fl()[i1 + a] : 0.f;
    }
#pragma unroll
    for (int a = 0; a < NC; ++a) one(o[a], rho[a], kv[a], rn_sub((float)(jlx + a), pp.x), cyb);
  }
  // then the second items, in window order
  uint64_t ov = no ? second_item_mask(S, no, row0, col0, nys, nxs) : 0u;
#pragma unroll 1
  while (ov) {
    const int pos = __ffsll(ov) - 1;
    ov &= ov - 1;
    const int b = pos / nxs, a = pos - b * nxs;
    const int q = S.nx()[(row0 + b) * S.L.s2 + col0 + a];
    one(S.oxy()[q], S.ofl()[q], S.okv()[k * kOvf + q], rn_sub((float)(jlx + a), pp.x), rn_sub((float)(jly + b), pp.y));
  }
  return gather_total(A.L.wf[k], A.L.wlo[k], s.hi, s.lo, s.sb);
}

// Control point j with all nine sums known and no empty direction: the next moment's density and
// deviations (k_emit's arithmetic).
template <int Q, int D>
__device__ __forceinline__ void emit_full(const Args<Q, D, PF32>& A, int j, const DF (&F)[Q]) {
  DF rho = {0.f, 0.f};
#pragma unroll
  for (int k = 0; k < Q; ++k) rho = df_add(rho, F[k]);
  A.b.rho[j] = df_float(rho);
#pragma unroll
  for (int k = 0; k < Q; ++k)
    A.b.dev[(int64_t)k * A.ccap + j] = df_float(df_add(F[k], df_neg(df_mul(DF{A.L.wf[k], A.L.wlo[k]}, rho))));
}
template <int Q, int D>
__device__ __forceinline__ void emit_from_cpf(const Args<Q, D, PF32>& A, int j) {
  DF F[Q];
#pragma unroll
  for (int k = 0; k < Q; ++k) F[k] = DF{A.cpfhi[(int64_t)k * A.ccap + j], A.cpflo[(int64_t)k * A.ccap + j]};
  emit_full<Q>(A, j, F);
}

// With fuse, a control point without empty directions is emitted here (almost all are; its nine
// sums are in registers: 72 bytes less written and read per point) and k_emit takes the others.
template <int Q, int TX, bool SPLIT>
__device__ __forceinline__ bool gather_ds_tile(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                               const TileGeo& G, bool fuse, unsigned char* smem) {
  using Lay = DenseLayoutOf<Q, 2, TX>;
  const DenseSmem<typename Lay::type> S{Lay::make(G), smem};
  __shared__ OwnList own;
  __shared__ uint32_t own_empty[512];
  stage_begin(S, &own.n);
  // the tile's own control points (at most two per cell)
  const int lx = threadIdx.x % (TX ? TX : G.tx), ly = threadIdx.x / (TX ? TX : G.tx);
  const int Fx = T.x0 + lx, Fy = T.y0 + ly;
  int bx = lx - (TX ? -3 : G.mom.xl), by = ly - (TX ? -3 : G.mom.yl);  // region coordinates of the control point's cell
  int j = 0, j1 = 0, many = 0;
  if (ly < G.ty && Fx < I.dims[0] && Fy < I.dims[1])
    cell_items(A.b.start, I.base + (uint32_t)Fx + (uint32_t)I.dims[0] * (uint32_t)Fy, &j, &j1, &many);
  bool has = j1 > j;
  if (j1 - j == 2) own.push_second(j + 1, bx, by);
  const bool dense = stage_dense<1, Q>(I, T.x0 + G.mom.xl, T.y0 + G.mom.yl, A.a.start, A.a.off, A.mcap, S, many,
                                       [&](int m, float2, float2* kv, int stride, int slot, float* fl, int, int fslot) {
                                         fl[fslot] = A.a.rho[m];
#pragma unroll
                                         for (int k = 0; k < Q; ++k)
                                           if (!SPLIT || d2q9_cy(k) == (int)blockIdx.y - 1)
                                             kv[k * stride + slot] = make_float2(A.sw[(int64_t)k * A.mcap + m],
                                                                               A.a.dev[(int64_t)k * A.mcap + m]);
                                         return 0;
                                       });
  if (!dense) return false;
  const int no = *S.novf();  // second items in the overflow list (at most kOvf in a dense tile)
  if (!has) has = own.take(&j, &bx, &by);
  if constexpr (TX == 0) {  // each thread its point's directions, windows by their exact ranges; no emit
    with_columns(A.R, A.tiny, [&](auto nc) {
#pragma unroll 1
      for (; has; has = own.take(&j, &bx, &by)) {
        const float2 pp = make_float2(A.b.off[j], A.b.off[A.ccap + j]);
        uint32_t empty = 0;
#pragma unroll 1
        for (int k = 0; k < Q; ++k) {
          const DF F = gather_ds_unit<Q, nc.value>(A, S, no, pp, k, bx, by);
          A.cpfhi[(int64_t)k * A.ccap + j] = F.hi;
          A.cpflo[(int64_t)k * A.ccap + j] = F.lo;
          if (F.hi < A.eps) empty |= 1u << k;
        }
        A.emask[j] = empty;
      }
    });
    return true;
  }
  if (has) {
    bool fits = false;
    if constexpr (TX > 0) {
      const float2 pp = make_float2(A.b.off[j], A.b.off[A.ccap + j]);
      int jlx, jly, nxs, nys;
      stencil_axis(pp.x, A.R, A.tiny, &jlx, &nxs);
      stencil_axis(pp.y, A.R, A.tiny, &jly, &nys);
      fits = block_fits(nxs, rn_add(__int_as_float(S.novf()[1]), rn_sub((float)(jlx + 4), pp.x)), A.R2) &&
             block_fits(nys, rn_add(__int_as_float(S.novf()[2]), rn_sub((float)(jly + 4), pp.y)), A.R2);
      if (fits) {
        float cx[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) cx[a] = rn_sub((float)(jlx + a), pp.x);
        const int n2 = S.L.n2;
        // second items anywhere in the 6 x 6 cells around the window, in window order
        uint64_t ov6 = no ? second_item_mask(S, no, by + jly - 1, bx + jlx - 1, 6, 6) : 0u;
        DF F[Q];
#pragma unroll 1
        for (int cy = SPLIT ? (int)blockIdx.y - 1 : -1; cy <= (SPLIT ? (int)blockIdx.y - 1 : 1); ++cy) {
          // the three directions (c_x, c_y), c_x = d - 1: moment rows jly - c_y + b, and the component's
          // column a is column a + 2 - d of the six from jlx - 1
          GatherSum s[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) s[d].clear();
          const int k0 = cy < 0 ? d2q9_dir(-1, -1) : cy == 0 ? d2q9_dir(-1, 0) : d2q9_dir(-1, 1);
          const int k1 = cy < 0 ? d2q9_dir(0, -1) : cy == 0 ? d2q9_dir(0, 0) : d2q9_dir(0, 1);
          const int k2 = cy < 0 ? d2q9_dir(1, -1) : cy == 0 ? d2q9_dir(1, 0) : d2q9_dir(1, 1);
          int i2 = (by + jly - cy) * S.L.s2 + (bx + jlx - 1), i1 = (by + jly - cy) * S.L.s1 + (bx + jlx - 1);
#pragma unroll 2
          for (int b = 0; b < 4; ++b, i2 += S.L.s2, i1 += S.L.s1) {
            const float cyb = rn_sub((float)(jly + b), pp.y);
            const float2* kv0 = S.kv() + i2 + k0 * n2;
            const float2* kv1 = S.kv() + i2 + k1 * n2;
            const float2* kv2 = S.kv() + i2 + k2 * n2;
            float2 o[6];
            float rho[6], ey2[6];
#pragma unroll
            for (int c = 0; c < 6; ++c) {
              o[c] = S.xy()[i2 + c];
              rho[c] = S.fl()[i1 + c];
              const float ey = rn_add(o[c].y, cyb);
              ey2[c] = rn_add(rn_mul(ey, ey), kTinyD2);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                const int c = a + 2 - d;
                const float ex = rn_add(o[c].x, cx[a]);
                const float w = window_weight(-rn_add(rn_mul(ex, ex), ey2[c]), A.R);
                const float2 kv = (d == 0 ? kv0 : d == 1 ? kv1 : kv2)[c];
                s[d].add(__fmul_rn(w, kv.x), rho[c], kv.y);
              }
          }
          // then the second items; a direction whose window does not hold the cell misses
          uint64_t ov = ov6;
#pragma unroll 1
          while (ov) {
            const int pos = __ffsll(ov) - 1;
            ov &= ov - 1;
            const int r = pos / 6, c = pos - r * 6;
            const int q = S.nx()[(by + jly - 1 + r) * S.L.s2 + bx + jlx - 1 + c];
            const float2 o = S.oxy()[q];
            const float rho = S.ofl()[q];
            const float ey = rn_add(o.y, rn_sub((float)(jly - 1 + r + cy), pp.y));
            const float ey2 = rn_add(rn_mul(ey, ey), kTinyD2);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const float ex = rn_add(o.x, rn_sub((float)(jlx - 1 + c + d - 1), pp.x));
              const float2 kv = S.okv()[(d == 0 ? k0 : d == 1 ? k1 : k2) * kOvf + q];
              s[d].add(__fmul_rn(window_weight(-rn_add(rn_mul(ex, ex), ey2), A.R), kv.x), rho, kv.y);
            }
          }
          DF T3[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int k = d == 0 ? k0 : d == 1 ? k1 : k2;
            T3[d] = gather_total(A.L.wf[k], A.L.wlo[k], s[d].hi, s[d].lo, s[d].sb);
          }
          if constexpr (SPLIT) {
            uint32_t empty = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const int k = d == 0 ? k0 : d == 1 ? k1 : k2;
              A.cpfhi[(int64_t)k * A.ccap + j] = T3[d].hi;
              A.cpflo[(int64_t)k * A.ccap + j] = T3[d].lo;
              if (T3[d].hi < A.eps) empty |= 1u << k;
            }
            if (empty) atomicOr(A.emask + j, empty);
          } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              if (cy < 0) F[d2q9_dir(d - 1, -1)] = T3[d];
              else if (cy == 0) F[d2q9_dir(d - 1, 0)] = T3[d];
              else F[d2q9_dir(d - 1, 1)] = T3[d];
            }
          }
        }
        if constexpr (!SPLIT) {
          uint32_t empty = 0;
#pragma unroll
          for (int k = 0; k < Q; ++k)
            if (F[k].hi < A.eps) empty |= 1u << k;
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
      }
    }
    if (!fits) own.push_wide(j, bx, by);
  }
  __syncthreads();
  const int left = own.left();
  if (left == 0) return true;  // the same in every thread
  for (int e = threadIdx.x; e < left; e += blockDim.x) own_empty[e] = 0u;
  __syncthreads();
#pragma unroll 1
  for (int u = threadIdx.x; u < left * Q; u += blockDim.x) {
    const int k = u / left, e = u - k * left, q = own.index(e), i = own.item[q];
    if (SPLIT && d2q9_cy(k) != (int)blockIdx.y - 1) continue;
    const DF F = gather_ds_unit<Q, 5>(A, S, no, make_float2(A.b.off[i], A.b.off[A.ccap + i]), k, own.pos[q] & 0xffff,
                                   own.pos[q] >> 16);
    A.cpfhi[(int64_t)k * A.ccap + i] = F.hi;
    A.cpflo[(int64_t)k * A.ccap + i] = F.lo;
    if (F.hi < A.eps) atomicOr(own_empty + e, 1u << k);
  }
  __syncthreads();
#pragma unroll 1
  for (int e = threadIdx.x; e < left; e += blockDim.x) {
    const uint32_t empty = own_empty[e];
    const int i = own.item[own.index(e)];
    if constexpr (SPLIT) {
      if (empty) atomicOr(A.emask + i, empty);
    } else {
      A.emask[i] = empty;
      if (fuse && !empty) emit_from_cpf<Q>(A, i);
    }
  }
  return true;
}

// ---- kernels ----------------------------------------------------------------------------------------
//
// The dense kernels take the tile list (one block per tile, or persistent over it).  A tile that
// is not dense is appended to a fallback list (fb_tiles, *fb_count, cleared before the launch);
// the matching k_dense_fallback then runs the row-segment code on exactly those tiles.  Keeping the
// two paths in separate kernels keeps the dense kernels' register count (and occupancy) their
// own.  The order of the fallback list is arbitrary, which changes no result: tiles write
// disjoint outputs.

// Resident blocks per SM the dense kernels are compiled for (chosen by timing the ensemble step
// on GB300).
#ifndef DBM_DS_BLOCKS_THIN
#define DBM_DS_BLOCKS_THIN 5
#endif
#ifndef DBM_DS_BLOCKS_WEIGHTS
#define DBM_DS_BLOCKS_WEIGHTS 6
#endif
#ifndef DBM_DS_BLOCKS_GATHER
#define DBM_DS_BLOCKS_GATHER 3
#endif

__device__ __forceinline__ void defer_tile(int tb, int* fb_tiles, int* fb_count) {
  if (threadIdx.x == 0) fb_tiles[atomicAdd(fb_count, 1)] = tb;
}

template <int Q, int TX>
__global__ void __launch_bounds__(256, DBM_DS_BLOCKS_THIN) k_thin_refine_ds(const __grid_constant__ Args<Q, 2, PF32> A,
                                                          const Tile2* __restrict__ tiles, const TileGeo G, int ntiles,
                                                          int* fb_tiles, int* fb_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int tb = blockIdx.x; tb < ntiles; tb += gridDim.x) {
    const Tile2 T = tiles[tb];
    const InstK I = A.inst[T.inst];
    if (!thin_refine_ds_tile<Q, TX>(A, T, I, G, smem)) defer_tile(tb, fb_tiles, fb_count);
    __syncthreads();
  }
}

// SPLIT, for a box of few tiles: the three blocks (tile, blockIdx.y) take the directions with c_y =
// blockIdx.y - 1, since one block per SM waits on its own loads and sums; the gather then leaves its sums
// to the emit pass.  For as many tiles as the three blocks of each still run at once: 64 x 64 cells, ten
// steps, 730 -> 600 us; at 256 x 256, where they would not, one block per tile is as fast.  They stage the same items and find the same fault, and the first defers the tile.
template <int Q, int TX, bool SPLIT>
__global__ void __launch_bounds__(256, DBM_DS_BLOCKS_WEIGHTS) k_weights_ds(const __grid_constant__ Args<Q, 2, PF32> A,
                                                      const Tile2* __restrict__ tiles, const TileGeo G, int ntiles,
                                                      int* fb_tiles, int* fb_count) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int tb = blockIdx.x; tb < ntiles; tb += gridDim.x) {
    const Tile2 T = tiles[tb];
    const InstK I = A.inst[T.inst];
    if (!weights_ds_tile<Q, TX, SPLIT>(A, T, I, G, smem) && (!SPLIT || blockIdx.y == 0))
      defer_tile(tb, fb_tiles, fb_count);
    __syncthreads();
  }
}

template <int Q, int TX, bool SPLIT>
__global__ void __launch_bounds__(256, TX ? DBM_DS_BLOCKS_GATHER : 4) k_gather_ds(const __grid_constant__ Args<Q, 2, PF32> A,
                                                     const Tile2* __restrict__ tiles, const TileGeo G, int ntiles,
                                                     int* fb_tiles, int* fb_count, int fuse) {
  extern __shared__ __align__(16) unsigned char smem[];
  for (int tb = blockIdx.x; tb < ntiles; tb += gridDim.x) {
    const Tile2 T = tiles[tb];
    const InstK I = A.inst[T.inst];
    // a negative density or an f that is not finite in the instance (noted by the collision): no dense tile
    if ((A.odd_f[T.inst] || !gather_ds_tile<Q, TX, SPLIT>(A, T, I, G, fuse != 0, smem)) && (!SPLIT || blockIdx.y == 0))
      defer_tile(tb, fb_tiles, fb_count);
    __syncthreads();
  }
}

// A deferred tile's gather: sets its control points' empty masks and runs `gather`.  With fuse the masks start
// as kEmitLater, by which k_emit knows the points that nothing has emitted: emitting them here, from the sums
// just written, cost the kernel its registers (1024 x 1024 cells at R = 1.9, most tiles deferred:
// gather and emit 2583 us a step with it, 1683 without).
template <int Q, class Fn>
__device__ __forceinline__ void gather_fallback(const Args<Q, 2, PF32>& A, const Tile2& T, const InstK& I,
                                                const TileGeo& G, bool fuse, Fn&& gather) {
  const int lx = threadIdx.x % G.tx, ly = threadIdx.x / G.tx;
  if (ly < G.ty && T.x0 + lx < I.dims[0] && T.y0 + ly < I.dims[1]) {
    const uint32_t g = I.base + (uint32_t)(T.x0 + lx) + (uint32_t)I.dims[0] * (uint32_t)(T.y0 + ly);
    for (uint32_t j = A.b.start[g], je = A.b.start[g + 1]; j < je; ++j) A.emask[j] = fuse ? kEmitLater : 0u;
  }
  __syncthreads();
  gather();
}

// Row-segment passes over the deferred tiles (persistent grid; nothing to do when the list is
// empty).  STAGE: 0 thin + refine, 1 weights, 2 gather.
template <int Q, int STAGE>
__global__ void __launch_bounds__(256) k_dense_fallback(const __grid_constant__ Args<Q, 2, PF32> A,
                                                       const Tile2* __restrict__ tiles, const TileGeo G,
                                                       const int* __restrict__ fb_tiles,
                                                       const int* __restrict__ fb_count, int fuse) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = *fb_count;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const Tile2 T = tiles[fb_tiles[i]];
    const InstK I = A.inst[T.inst];
    if constexpr (STAGE == 0) {
      thin_refine_tile<Q, PF32, true>(A, T, I, G, smem);
    } else if constexpr (STAGE == 1) {
      weights_tile<Q, PF32, true>(A, T, I, G, smem);
    } else {
      gather_fallback<Q>(A, T, I, G, fuse != 0, [&] { gather_ts_tile<Q>(A, T, I, G, smem); });
    }
    __syncthreads();
  }
}

}  // namespace dbm
