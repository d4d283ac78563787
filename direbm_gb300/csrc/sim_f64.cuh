// Window sums of the FP64 store: candidates by FP32, hits in FP64.
//
// GB300 runs FP64 at two lanes per clock and SM, and an instruction costs the same 64 cycles of a
// scheduler's FP64 unit however few lanes are active.  So no FP64 instruction is spent on a candidate that
// misses, and none where few lanes need it: a thread first walks its window in FP32 (the items' packed
// float copies, bounds with margins far above the rounding) and lists the items within r plus a margin;
// then it runs down the list, one canonical FP64 test and sum per entry, so the lanes of a warp work on a
// hit each.  The FP64 decisions, sums and their order are those of the plain loops bit for bit.
//
// What is left is ~18 FP64 operations per hit (displacement 3 D - 1 + D, root 7.5, weight and sum 3).
// Before, a candidate cost its displacement and bound in FP64 (5 to 8 operations) and a warp waited for its
// lane with the most of them.  128 x 128 cells, D2Q9, R 1.5, a step: thin + refine 353 -> 144 us, weights
// 437 -> 86, gather 425 -> 80.  D3Q19, 65 k points: 4.9 -> 1.5 ms, 8.1 -> 1.7, 5.5 -> 1.7.  The FP64 units
// are busy 70 to 74 % of the time.
#pragma once

#include "sim.cuh"

namespace dbm {

constexpr int kNearCap = 96;   // listed candidates of a thread; a longer window is worked off in parts
constexpr int kNearFlush = 32; // the refine works its lists off once some lane holds more than this

struct NearList {
  int n = 0;
  int m[kNearCap];
  short4 s[kNearCap];  // cell displacement less ctr, direction
};

// The cell displacement nearest to a direction's.  Listed displacements are relative to it (or its
// opposite), so that they are small at any ratio of spacing and cell.
template <int Q, int D>
__device__ __forceinline__ int cd_cells(const LatK<Q, D>& L, int k, int a) {
  return __float2int_rn(L.cdf[k][a]);
}

// rn((j - cd_cells) + cd_k) per direction, axis and small j, formed once per block.
constexpr int kShiftHalf = 8;
template <int Q, int D>
struct ShiftTable {
  double v[Q][D][2 * kShiftHalf];
  __device__ __forceinline__ static double form(const LatK<Q, D>& L, int k, int a, int j) {
    return rn_add((double)j - (double)cd_cells(L, k, a), L.cd[k][a]);
  }
  __device__ __forceinline__ void fill(const LatK<Q, D>& L) {
    double* p = &v[0][0][0];
    for (int i = threadIdx.x; i < Q * D * 2 * kShiftHalf; i += blockDim.x) {
      const int ka = i / (2 * kShiftHalf);
      p[i] = form(L, ka / D, ka % D, i % (2 * kShiftHalf) - kShiftHalf);
    }
  }
  __device__ __forceinline__ double at(const LatK<Q, D>& L, int k, int a, int j) const {
    const int i = j + kShiftHalf;
    return (unsigned)i < (unsigned)(2 * kShiftHalf) ? v[k][a][i] : form(L, k, a, j);
  }
};

// Lists the items (start, pf) that may lie within R of the point r (cell units relative to cell C of I; the
// margins cover the rounding of r at its size), their displacements less ctr, rows ascending, each row's items in cell order; skip(m) drops an item; flush() empties a full list.
template <int D, class Skip, class Flush>
__device__ __forceinline__ void near_items(const InstK& I, const int (&C)[3], const float (&r)[3], float R, int k, const int (&ctr)[3],
                                           const uint32_t* __restrict__ start, const float4* __restrict__ pf,
                                           NearList& L, Skip&& skip, Flush&& flush) {
  const float big = 1e-6f * (fabsf(r[0]) + fabsf(r[1]) + fabsf(r[2]));
  const float t = 1e-3f + big, Rm = R + 1e-4f * (1.f + R) + big, R2m = Rm * Rm;
  int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
#pragma unroll
  for (int a = 0; a < D; ++a) {
    lo[a] = (int)floorf(r[a] - Rm - t);
    hi[a] = (int)floorf(r[a] + Rm + t);
  }
#pragma unroll 1
  for (int sz = lo[2]; sz <= hi[2]; ++sz) {
    const float cz = D == 3 ? (float)sz - r[2] : 0.f;
    const float lz = D == 3 ? axis_lb<float>(cz) : 0.f;
#pragma unroll 1
    for (int sy = lo[1]; sy <= hi[1]; ++sy) {
      const float cy = (float)sy - r[1];
      const float ly = axis_lb<float>(cy);
      const float rem = R2m - ly * ly - lz * lz;
      if (rem < 0.f) continue;
      const float hw = bound_sqrt(rem) + t;
      const int lox = max((int)floorf(r[0] - hw), lo[0]), hix = min((int)floorf(r[0] + hw), hi[0]);
      if (lox > hix) continue;
      row_runs<D>(I, C[0], C[1] + sy, C[2] + sz, lox, hix, [&](uint32_t g0, uint32_t g1, int shift) {
        const uint32_t m1 = start[g1 + 1];
        for (uint32_t m = start[g0]; m < m1; ++m) {
          const float4 it = pf[m];
          const int sx = __float_as_int(it.w) + shift - C[0];  // the cell's x coordinate, an integer
          const float ex = it.x + ((float)sx - r[0]), ey = it.y + cy;
          float d2 = ex * ex + ey * ey;
          if (D == 3) {
            const float ez = it.z + cz;
            d2 += ez * ez;
          }
          if (!(d2 <= R2m) || skip(m)) continue;
          L.m[L.n] = (int)m;
          L.s[L.n] = make_short4((short)(sx - ctr[0]), (short)(sy - ctr[1]), (short)(sz - ctr[2]), (short)k);
          if (++L.n == kNearCap) flush();
        }
      });
    }
  }
}

// Squared displacement of a listed item from reference point p (gather, refine), canonical order.
template <int Q, int D>
__device__ __forceinline__ double listed_d2(const LatK<Q, D>& L, const ShiftTable<Q, D>& T, const PackItem<double>& it,
                                            short4 s, const double (&p)[3], double (&e)[3]) {
  const int k = s.w;
  double c[3] = {0, 0, 0};
  c[0] = rn_sub(T.at(L, k, 0, s.x), p[0]);
  c[1] = rn_sub(T.at(L, k, 1, s.y), p[1]);
  if constexpr (D == 3) c[2] = rn_sub(T.at(L, k, 2, s.z), p[2]);
  const double o[3] = {it.x, it.y, it.z};
  return canon_d2<D, double>(o, c, e);
}
// a <= b for a >= 0, b > 0 or a NaN: the bits of non-negative doubles order as integers.
__device__ __forceinline__ bool le_bits(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) <= (unsigned long long)__double_as_longlong(b);
}

}  // namespace dbm
