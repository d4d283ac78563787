// Stage functions on explicit component arrays (FP32, 2D), the reference's propagation API.
//
// These keep the data layout of direbm/warp/propagation.py (positions (N,2), values (N,),
// directions (N,), moments (M,Q) row-major) so the drop-in Python module can hand them numpy
// arrays the way the reference tests do.  Components here are arbitrary points in an unbounded
// plane, so neighbour queries use a sorted-cell index: the points' bounds are read back first, so that
// the cell keys are as short as the points allow (16 bits in place of 64 for 192 x 192 cells, two radix
// passes in place of eight) and, where the box is not mostly empty, a table of cell starts takes the place
// of binary searches.  The cells of one x column that a query needs are consecutive: one run of items.
// The refine alone waits for nothing: its index is a hashed table (HashIndex).
//
// The radius test is |a - b| with round-to-nearest FP32 steps and no fused multiply-add, so the
// pairs found are the oracle's (oracle/stages.py) bit for bit.  Sums run in a fixed order per
// thread with compensated accumulators: there are no float atomics and results are reproducible.
#include <algorithm>
#include <mutex>

#include "lattice.cuh"
#include "sortscan.cuh"

namespace dbm {

__device__ __forceinline__ float dist32(float ax, float ay, float bx, float by) {
  const float dx = __fsub_rn(ax, bx), dy = __fsub_rn(ay, by);
  return __fsqrt_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)));
}

// Points of the caller's arrays: 4-byte aligned, no wider loads.
__device__ __forceinline__ float2 load2(const float* __restrict__ p, int64_t i) {
  return make_float2(p[2 * i], p[2 * i + 1]);
}
__device__ __forceinline__ void store2(float* __restrict__ p, int64_t i, float2 v) {
  p[2 * i] = v.x;
  p[2 * i + 1] = v.y;
}

__device__ __forceinline__ long long cell_of(float x, float cs) { return (long long)floorf(__fdiv_rn(x, cs)); }

template <int Q>
__global__ void k_disperse(const float* __restrict__ pos_m, const float* __restrict__ f_m, int64_t m,
                           LatK<Q, 2> L, float dx, float* __restrict__ pos_c, float* __restrict__ val_c,
                           int32_t* __restrict__ dir_c) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = pos_m[2 * i], y = pos_m[2 * i + 1];
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int64_t c = i * Q + k;
      pos_c[2 * c] = __fadd_rn(x, __fmul_rn(L.cf[k][0], dx));
      pos_c[2 * c + 1] = __fadd_rn(y, __fmul_rn(L.cf[k][1], dx));
      val_c[c] = f_m[c];
      dir_c[c] = k;
    }
  }
}

// Cells as 32-bit words whose order is the cells'.
__device__ __forceinline__ uint32_t cell_word(long long i) { return (uint32_t)((unsigned long long)i + 2147483648ULL); }

// Bounds of the points' cells: (min x, min y, ~max x, ~max y), all set to ones before.
__global__ void __launch_bounds__(256) k_bounds(const float* __restrict__ pos, int64_t n, float cs,
                                                uint32_t* __restrict__ bounds) {
  uint32_t lo[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const uint32_t c = cell_word(cell_of(pos[2 * i + a], cs));
      lo[a] = min(lo[a], c);
      lo[2 + a] = min(lo[2 + a], ~c);
    }
  }
  __shared__ uint32_t s_lo[4];
  if (threadIdx.x < 4) s_lo[threadIdx.x] = 0xffffffffu;
  __syncthreads();
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const uint32_t w = __reduce_min_sync(0xffffffffu, lo[a]);
    if ((threadIdx.x & 31) == 0) atomicMin(&s_lo[a], w);
  }
  __syncthreads();
  if (threadIdx.x < 4) atomicMin(&bounds[threadIdx.x], s_lo[threadIdx.x]);
}

// A sorted-cell index over n points (cell size cs).  Key of a cell: dense, dx * ny + dy from the lower
// bounds; else dx << by | dy.
struct PointIndex {
  uint32_t minx = 0, miny = 0, maxx = 0xffffffffu, maxy = 0xffffffffu;
  uint32_t ny = 0;           // dense: cells along y (0: not dense)
  int by = 32;
  uint32_t n = 0;
  uint64_t* keys = nullptr;   // sorted cell keys [n]
  uint32_t* order = nullptr;  // point index in sorted order [n]
  uint32_t* start = nullptr;  // dense: first item of each cell [cells + 1]

  __device__ __forceinline__ uint64_t key(uint32_t wx, uint32_t wy) const {
    return ny ? (uint64_t)(wx - minx) * ny + (wy - miny) : ((uint64_t)(wx - minx) << by) | (wy - miny);
  }
  __device__ __forceinline__ uint32_t lower(uint64_t k) const {  // first item with a key >= k
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (keys[mid] < k) lo = mid + 1; else hi = mid;
    }
    return lo;
  }
  // body(j) for the items of column wx, rows [wy0, wy1], in sorted order
  template <class F>
  __device__ __forceinline__ void run(uint32_t wx, uint32_t wy0, uint32_t wy1, F&& body) const {
    wy0 = max(wy0, miny);
    wy1 = min(wy1, maxy);
    if (wy0 > wy1) return;
    const uint64_t k0 = key(wx, wy0), k1 = k0 + (wy1 - wy0);
    if (ny) {
      const uint32_t e = start[k1 + 1];
      for (uint32_t j = start[k0]; j < e; ++j) body(j);
    } else {
      for (uint32_t j = lower(k0); j < n && keys[j] <= k1; ++j) body(j);
    }
  }
};

// Cells along one axis within 1 + m of the quotient f, m above the rounding of the quotients and of the
// distance (relative 2^-22), at most two away; from 2^40 on, an infinite quotient included, where floats lie
// further apart than dx, its own.
__device__ __forceinline__ void near_cells(float f, long long* lo, long long* hi) {
  const long long c = (long long)floorf(f);
  *lo = *hi = c;
  if (fabsf(f) < 1.0995116e12f) {
    const float m = 1.f + 1e-6f * (2.f + fabsf(f));
    *lo = max((long long)floorf(f - m), c - 2);
    *hi = min((long long)floorf(f + m), c + 2);
  }
}

// body(j) for every item of ix that may lie within dx (its cell size) of (x, y), columns ascending, then
// rows: three columns of three rows but for a query at a cell's edge.
template <class F>
__device__ __forceinline__ void near_points(const PointIndex& ix, float x, float y, float dx, F&& body) {
  const float fx = __fdiv_rn(x, dx), fy = __fdiv_rn(y, dx);
  if (ix.n == 0) return;
  long long x0, x1, y0, y1;
  near_cells(fx, &x0, &x1);
  near_cells(fy, &y0, &y1);
  const uint32_t wy0 = cell_word(y0), wy1 = cell_word(y1);
  for (long long c = x0;; ++c) {
    const uint32_t wx = cell_word(c);
    if (wx >= ix.minx && wx <= ix.maxx) {
      if (wy0 <= wy1) {
        ix.run(wx, wy0, wy1, body);
      } else {  // the rows wrap around the word
        ix.run(wx, wy0, 0xffffffffu, body);
        ix.run(wx, 0u, wy1, body);
      }
    }
    if (c == x1) break;
  }
}

__global__ void k_keys(const float* __restrict__ pos, int64_t n, float cs, PointIndex ix) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    ix.keys[i] = ix.key(cell_word(cell_of(pos[2 * i], cs)), cell_word(cell_of(pos[2 * i + 1], cs)));
    ix.order[i] = (uint32_t)i;
  }
}

// One search per cell: a walk over the keys would leave a long gap between two clusters to one thread.
__global__ void k_cell_starts(PointIndex ix, int64_t ncells) {
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c <= ncells; c += (int64_t)gridDim.x * blockDim.x)
    ix.start[c] = ix.lower((uint64_t)c);
}

__global__ void k_heads(const uint64_t* __restrict__ keys, int64_t n, uint32_t* __restrict__ flags) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

// Sequential FP32 centroid per run, in sorted order (propagation.py:54-68); rank: heads before an item.
__global__ void k_centroid(const float* __restrict__ pos_c, PointIndex ix, const uint32_t* __restrict__ rank,
                           float* __restrict__ cp) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ix.n; i += gridDim.x * blockDim.x) {
    const uint64_t key = ix.keys[i];
    if (i > 0 && ix.keys[i - 1] == key) continue;
    float sx = 0.f, sy = 0.f;
    uint32_t j = i;
    do {
      const float2 q = load2(pos_c, ix.order[j]);
      sx = __fadd_rn(sx, q.x);
      sy = __fadd_rn(sy, q.y);
    } while (++j < ix.n && ix.keys[j] == key);
    const float n = (float)(j - i);
    store2(cp, rank[i], make_float2(__fdiv_rn(sx, n), __fdiv_rn(sy, n)));
  }
}

// The temporaries' own stream-ordered pool, one per device.  Up to 64 MB stay with it between calls: the
// default pool gives every page back at each synchronisation and maps it again on the next call.
constexpr uint64_t kPoolKeep = 64ull << 20;
static int stage_pool(cudaMemPool_t* out) {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  DBM_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_last_error("device %d: out of range", dev); return DBM_ERR_STATE; }
  std::lock_guard<std::mutex> lock(mu);
  if (!pools[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    DBM_CUDA(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = kPoolKeep;
    DBM_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    pools[dev] = pool;
  }
  *out = pools[dev];
  return DBM_OK;
}

// Stream-ordered temporaries of one call, cut from one allocation (`bytes`: an upper bound of their sum).
struct Arena {
  cudaStream_t s;
  char* base = nullptr;
  size_t used = 0, bytes;
  Arena(cudaStream_t st, size_t b) : s(st), bytes(b) {}
  template <class T>
  int get(T** p, int64_t count) {
    if (!base) {
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
      DBM_CUDA(cudaStreamIsCapturing(s, &cap));
      cudaMemPool_t pool = nullptr;
      if (cap == cudaStreamCaptureStatusNone) DBM_TRY(stage_pool(&pool));  // a captured graph owns its memory
      void* q = nullptr;
      const cudaError_t e = pool ? cudaMallocFromPoolAsync(&q, bytes, pool, s) : cudaMallocAsync(&q, bytes, s);
      if (e != cudaSuccess) { set_last_error("stage temporaries: %s", cudaGetErrorString(e)); return DBM_ERR_CUDA; }
      base = (char*)q;
    }
    const size_t sz = ((size_t)std::max<int64_t>(count, 1) * sizeof(T) + 255) / 256 * 256;
    if (sz > bytes - used) { set_last_error("internal: a stage call's temporaries exceed their bound"); return DBM_ERR_STATE; }
    *p = (T*)(base + used);
    used += sz;
    return DBM_OK;
  }
  ~Arena() {
    if (base) cudaFreeAsync(base, s);
  }
};

// The most cells of a table of starts for n points, and the bytes of an index with its packed items.
static uint64_t max_cells(int64_t n) { return 4 * (uint64_t)n + 65536; }
static size_t index_bytes(int64_t n, bool starts) {
  const size_t m = (size_t)std::max<int64_t>(n, 1);
  return m * (8 + 4 + 8 + 4 + 16 + 4) + radix_tmp_bytes(n) + (starts ? (size_t)(max_cells(n) + 1) * 4 : scan_tmp_bytes(n)) +
         12 * 256;
}

static unsigned grid_for(int64_t n) { return std::min<unsigned>(div_up(std::max<int64_t>(n, 1), 256), (unsigned)sm_count() * 16); }

static int bit_length(uint64_t v) {
  int b = 0;
  while (b < 64 && (v >> b)) ++b;
  return b;
}

// Bounds of one or two point sets (n > 0) on the host; false while the stream is being captured, which
// allows no read-back.
struct PointSet {
  const float* pos;
  int64_t n;
  float cs;
};
static int read_bounds(const PointSet* sets, int nsets, Arena& ar, uint32_t (*bounds)[4], bool* known) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  DBM_CUDA(cudaStreamIsCapturing(ar.s, &cap));
  *known = cap == cudaStreamCaptureStatusNone;
  if (!*known) return DBM_OK;
  uint32_t* d = nullptr;
  DBM_TRY(ar.get(&d, 4 * nsets));
  DBM_CUDA(cudaMemsetAsync(d, 0xff, (size_t)nsets * 16, ar.s));
  for (int i = 0; i < nsets; ++i) {
    const unsigned g = std::min<unsigned>(div_up(sets[i].n, 1024), (unsigned)sm_count() * 2);
    k_bounds<<<g, 256, 0, ar.s>>>(sets[i].pos, sets[i].n, sets[i].cs, d + 4 * i);
    DBM_LAUNCH_CHECK();
  }
  DBM_CUDA(cudaMemcpyAsync(bounds, d, (size_t)nsets * 16, cudaMemcpyDeviceToHost, ar.s));
  DBM_CUDA(cudaStreamSynchronize(ar.s));
  return DBM_OK;
}

// starts: the index serves neighbour queries (else only its order is used).
static int build_index(const PointSet& p, const uint32_t (&bounds)[4], bool known, bool starts, Arena& ar,
                       PointIndex* ix) {
  cudaStream_t s = ar.s;
  const int64_t n = p.n;
  uint64_t* k_alt;
  uint32_t* v_alt;
  char* rtmp;
  DBM_TRY(ar.get(&ix->keys, n));
  DBM_TRY(ar.get(&ix->order, n));
  DBM_TRY(ar.get(&k_alt, n));
  DBM_TRY(ar.get(&v_alt, n));
  DBM_TRY(ar.get(&rtmp, (int64_t)radix_tmp_bytes(n)));
  ix->n = (uint32_t)n;
  int bits = 64;
  uint64_t cells = 0;
  if (known) {
    ix->minx = bounds[0];
    ix->miny = bounds[1];
    ix->maxx = ~bounds[2];
    ix->maxy = ~bounds[3];
    const uint64_t nx = (uint64_t)(ix->maxx - ix->minx) + 1, ny = (uint64_t)(ix->maxy - ix->miny) + 1;
    ix->by = bit_length(ny - 1);
    bits = bit_length(nx - 1) + ix->by;
    // a table of at most four cells per point (plus a little): mostly empty boxes are searched instead
    if (nx < (1u << 31) && ny < (1u << 31) && nx * ny <= max_cells(n)) {
      cells = nx * ny;
      ix->ny = (uint32_t)ny;
      bits = bit_length(cells - 1);
    }
  }
  k_keys<<<grid_for(n), 256, 0, s>>>(p.pos, n, p.cs, *ix);
  DBM_LAUNCH_CHECK();
  bool alt = false;
  DBM_TRY(radix_sort_pairs<uint64_t>(ix->keys, ix->order, k_alt, v_alt, n, nullptr, bits, rtmp, s, &alt));
  if (alt) {
    ix->keys = k_alt;
    ix->order = v_alt;
  }
  if (ix->ny && starts) {
    DBM_TRY(ar.get(&ix->start, (int64_t)cells + 1));
    k_cell_starts<<<grid_for((int64_t)cells + 1), 256, 0, s>>>(*ix, (int64_t)cells);
    DBM_LAUNCH_CHECK();
  }
  return DBM_OK;
}

// Components in index order: position, value (expf of it for the refine), direction or weight sum.
__global__ void k_pack_comps(const float* __restrict__ pos_c, const float* __restrict__ val_c,
                             const int32_t* __restrict__ dir_c, const uint32_t* __restrict__ order, uint32_t n,
                             int as_weight, float4* __restrict__ items) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const uint32_t c = order[j];
    const float2 q = load2(pos_c, c);
    const float v = val_c[c];
    items[j] = make_float4(q.x, q.y, as_weight ? expf(v) : v, __int_as_float(dir_c[c]));
  }
}
__global__ void k_pack_points(const float* __restrict__ pos, PointIndex ix, float2* __restrict__ items) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < ix.n; j += gridDim.x * blockDim.x)
    items[j] = load2(pos, ix.order[j]);
}

// The refine's index, which needs no look at the bounds and so leaves the call asynchronous: a table of
// buckets, one per four components or so, bucket = S column + row modulo its size 2^bits with S near 0.618 of
// it, so that the rows which a query needs of one column are consecutive and those of the at most five columns
// lie apart (1 to 4 times S is at least 0.13 of the table from 0; a query has at most five rows): no component
// is met twice, and the distance sorts out those of other cells.  Blocks of 2^16 columns and rows are displaced
// against each other, for points whose cells are multiples of a large power of two; a query across a border
// of blocks (away from the origin, where boxes begin) takes a component only in its own cell's turn.
struct HashIndex {
  int bits = 0;
  uint32_t n = 0;
  uint32_t* order = nullptr;  // component of each place, by bucket, then in input order
  uint32_t* start = nullptr;  // first place of each bucket [2^bits + 1]

  __host__ __device__ __forceinline__ uint32_t mask() const { return (1u << bits) - 1u; }
  __device__ __forceinline__ uint32_t bucket(uint32_t wx, uint32_t wy) const {
    const uint32_t S = (0x9E3779B9u >> (32 - bits)) | 1u;
    return (wx * S + wy + block(wx) * 0x85EBCA6Bu + block(wy) * 0xC2B2AE35u) & mask();
  }
  static __device__ __forceinline__ uint32_t block(uint32_t w) { return (w + 0x4DB7u) >> 16; }
};

__global__ void k_hash_keys(const float* __restrict__ pos, HashIndex ix, float cs, uint32_t* __restrict__ keys) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ix.n; i += gridDim.x * blockDim.x) {
    const float2 q = load2(pos, i);
    keys[i] = ix.bucket(cell_word(cell_of(q.x, cs)), cell_word(cell_of(q.y, cs)));
    ix.order[i] = i;
  }
}
__global__ void k_hash_starts(const uint32_t* __restrict__ keys, HashIndex ix) {
  const uint32_t nb = ix.mask() + 1u;
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= nb; c += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = ix.n;
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (keys[mid] < c) lo = mid + 1; else hi = mid;
    }
    ix.start[c] = lo;
  }
}

static int hash_bits(int64_t n) {
  int b = 8;
  while (b < 31 && (4ll << b) < n) ++b;
  return b;
}
static size_t hash_bytes(int64_t n) {
  const size_t m = (size_t)std::max<int64_t>(n, 1);
  return m * (4 * 4 + 16) + radix_tmp_bytes(n) + (((size_t)1 << hash_bits(n)) + 1) * 4 + 8 * 256;
}
static int build_hash(const float* pos, int64_t n, float cs, Arena& ar, HashIndex* ix) {
  cudaStream_t s = ar.s;
  uint32_t *keys, *k_alt, *v_alt;
  char* rtmp;
  ix->n = (uint32_t)n;
  ix->bits = hash_bits(n);
  DBM_TRY(ar.get(&keys, n));
  DBM_TRY(ar.get(&ix->order, n));
  DBM_TRY(ar.get(&k_alt, n));
  DBM_TRY(ar.get(&v_alt, n));
  DBM_TRY(ar.get(&rtmp, (int64_t)radix_tmp_bytes(n)));
  DBM_TRY(ar.get(&ix->start, (1ll << ix->bits) + 1));
  k_hash_keys<<<grid_for(n), 256, 0, s>>>(pos, *ix, cs, keys);
  DBM_LAUNCH_CHECK();
  bool alt = false;
  DBM_TRY(radix_sort_pairs<uint32_t>(keys, ix->order, k_alt, v_alt, n, nullptr, ix->bits, rtmp, s, &alt));
  if (alt) {
    keys = k_alt;
    ix->order = v_alt;
  }
  k_hash_starts<<<grid_for((1ll << ix->bits) + 1), 256, 0, s>>>(keys, *ix);
  DBM_LAUNCH_CHECK();
  return DBM_OK;
}

// body(it) for the components within dx of p, columns ascending, then rows, then in input order.
template <class F>
__device__ __forceinline__ void hash_hits(const HashIndex& ix, const float4* __restrict__ items, float2 p, float dx,
                                          F&& body) {
  if (ix.n == 0) return;
  long long x0, x1, y0, y1;
  near_cells(__fdiv_rn(p.x, dx), &x0, &x1);
  near_cells(__fdiv_rn(p.y, dx), &y0, &y1);
  const uint32_t wx0 = cell_word(x0), wy0 = cell_word(y0), cols = (uint32_t)(x1 - x0), rows = (uint32_t)(y1 - y0);
  auto within = [&](float4 it) { return dist32(it.x, it.y, p.x, p.y) <= dx; };
  if (ix.block(wx0) == ix.block(wx0 + cols) && ix.block(wy0) == ix.block(wy0 + rows)) {
    for (uint32_t c = 0; c <= cols; ++c) {
      const uint32_t b = ix.bucket(wx0 + c, wy0), b1 = min(b + rows, ix.mask()), over = b + rows - b1;
      for (uint32_t j = ix.start[b], e = ix.start[b1 + 1u]; j < e; ++j) {
        const float4 it = items[j];
        if (within(it)) body(it);
      }
      for (uint32_t j = 0, e = ix.start[over]; j < e; ++j) {  // around the table's end
        const float4 it = items[j];
        if (within(it)) body(it);
      }
    }
  } else {
    for (uint32_t c = 0; c <= cols; ++c)
      for (uint32_t r = 0; r <= rows; ++r) {
        const uint32_t b = ix.bucket(wx0 + c, wy0 + r);
        for (uint32_t j = ix.start[b], e = ix.start[b + 1u]; j < e; ++j) {
          const float4 it = items[j];
          if (within(it) && cell_word(cell_of(it.x, dx)) == wx0 + c && cell_word(cell_of(it.y, dx)) == wy0 + r) body(it);
        }
      }
  }
}

// 205 k points, 258 k components: 200 us by searches (16 dependent loads per cell, 25 cells), 40 by either table;
// the call from 30 k moments (210 k components) 125 us with the read-back of the bounds, 105 without.
__global__ void k_refine(const float* __restrict__ cp, int64_t p, const float4* __restrict__ items, HashIndex ix,
                         float dx, int kappa_hard, float* __restrict__ out) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < p; r += (int64_t)gridDim.x * blockDim.x) {
    const float2 q = load2(cp, r);
    uint32_t mask = 0;
    CSum sw, sx, sy;
    hash_hits(ix, items, q, dx, [&](float4 it) {
      mask |= 1u << __float_as_int(it.w);
      sw.add(it.z);
      sx.add_prod(it.z, it.x);
      sy.add_prod(it.z, it.y);
    });
    if (__popc(mask) <= kappa_hard) {
      store2(out, r, q);
    } else {
      const float s = sw.value();
      store2(out, r, make_float2(sx.value() / s, sy.value() / s));
    }
  }
}

// Resampling, first walk: the weight sum of each component over the control points within dx (166 -> 25 us).
__global__ void k_comp_sw(const float4* __restrict__ comps, uint32_t nc, const float2* __restrict__ cps, PointIndex cpi,
                          float dx, float* __restrict__ sw_out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nc; i += gridDim.x * blockDim.x) {
    const float4 q = comps[i];
    CSum sw;
    near_points(cpi, q.x, q.y, dx, [&](uint32_t j) {
      const float2 c = cps[j];
      const float d = dist32(c.x, c.y, q.x, q.y);
      if (d <= dx) sw.add(__fsub_rn(dx, d));
    });
    sw_out[i] = sw.value();
  }
}

// Second walk, in place of the reference's scatter with float atomics (propagation.py:156-186): every
// control point gathers (dx - d)/sw * f of the components with sw > 0 within dx, direction by direction, in
// index order.  A thread's sums lie in shared memory ([Q][256], its own column), since the direction of the
// next component is not known; writing a record per pair, sorting and summing the records took 0.65 ms for
// 4.6 M pairs where this takes 0.04.
template <int Q>
__global__ void __launch_bounds__(256) k_cp_gather(const float2* __restrict__ cps, PointIndex cpi,
                                                   const float4* __restrict__ comps, const float* __restrict__ sw,
                                                   PointIndex ci, float dx, float eps, uint32_t* __restrict__ emask,
                                                   float* __restrict__ out_pos, float* __restrict__ out_f) {
  __shared__ float s_hi[Q][256], s_lo[Q][256];
  const int t = threadIdx.x;
  for (uint32_t i = blockIdx.x * blockDim.x + t; i < cpi.n; i += gridDim.x * blockDim.x) {
    const float2 p = cps[i];
#pragma unroll
    for (int q = 0; q < Q; ++q) s_hi[q][t] = s_lo[q][t] = 0.f;
    uint32_t seen = 0;
    near_points(ci, p.x, p.y, dx, [&](uint32_t j) {
      const float4 it = comps[j];
      const float d = dist32(p.x, p.y, it.x, it.y);
      if (!(d <= dx)) return;
      const float s = sw[j];
      const uint32_t k = (uint32_t)__float_as_int(it.w);
      if (!(s > 0.f) || k >= (uint32_t)Q) return;
      const float v = __fmul_rn(__fdiv_rn(__fsub_rn(dx, d), s), it.z);
      if ((seen >> k) & 1u) {
        CSum a;
        a.hi = s_hi[k][t];
        a.lo = s_lo[k][t];
        a.add(v);
        s_hi[k][t] = a.hi;
        s_lo[k][t] = a.lo;
      } else {
        seen |= 1u << k;
        s_hi[k][t] = v;
      }
    });
    const uint32_t r = cpi.order[i];
    uint32_t em = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float v = __fadd_rn(s_hi[q][t], s_lo[q][t]);
      if (v < eps) em |= 1u << q;
      out_f[(int64_t)r * Q + q] = v;
    }
    emask[i] = em;
    store2(out_pos, r, p);
  }
}

// Empty directions from the rest state, judged on the masks before the fill.
template <int Q>
__global__ void __launch_bounds__(256) k_cp_fill(const float2* __restrict__ cps, PointIndex cpi,
                                                 const uint32_t* __restrict__ emask, const float* __restrict__ f_rest,
                                                 float dx, float* __restrict__ out_f) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cpi.n; i += gridDim.x * blockDim.x) {
    const uint32_t em = emask[i];
    if (!em) continue;
    const float2 p = cps[i];
    CSum sw[Q];
    near_points(cpi, p.x, p.y, dx, [&](uint32_t j) {
      const uint32_t both = emask[j] & em;
      if (!both) return;
      const float2 o = cps[j];
      const float d = dist32(o.x, o.y, p.x, p.y);
      if (d <= dx) {
        const float w = __fsub_rn(dx, d);
#pragma unroll
        for (int q = 0; q < Q; ++q)
          if ((both >> q) & 1u) sw[q].add(w);
      }
    });
    const uint32_t r = cpi.order[i];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const float s = sw[q].value();
      if (((em >> q) & 1u) && s > 0.f) out_f[(int64_t)r * Q + q] = (dx / s) * f_rest[q];
    }
  }
}

}  // namespace dbm

using namespace dbm;

// Points are indexed in 32 bits, with room for a grid's stride above the last.
constexpr int64_t kMaxPoints = 1ll << 31;

static int check_2d(int lattice) {
  const LatHost* h = lat_host(lattice);
  if (!h || h->D != 2) {
    set_last_error("stage functions take a 2D lattice (got id %d)", lattice);
    return DBM_ERR_INVALID;
  }
  return DBM_OK;
}

extern "C" {

int dbm_disperse_f32(const float* pos_m, const float* f_m, int64_t m, int lattice, float dx, float* pos_c,
                     float* val_c, int32_t* dir_c, void* stream) {
  DBM_TRY(check_2d(lattice));
  if (m < 0 || (m > 0 && (!pos_m || !f_m || !pos_c || !val_c || !dir_c))) {
    set_last_error("disperse: bad arguments");
    return DBM_ERR_INVALID;
  }
  if (m == 0) return DBM_OK;
  return dispatch_lattice(lattice, [&](auto tag) -> int {
    using LT = decltype(tag);
    if constexpr (LT::D == 2) {
      auto L = make_latk<LT::Q, 2>(*lat_host(lattice), 1.0, 1.0);
      k_disperse<LT::Q><<<grid_for(m), 256, 0, (cudaStream_t)stream>>>(pos_m, f_m, m, L, dx, pos_c, val_c, dir_c);
      DBM_LAUNCH_CHECK();
    }
    return DBM_OK;
  });
}

int dbm_create_control_points_f32(const float* pos_c, int64_t nc, float cs, float* cp_pos, int64_t* p_out,
                                  void* stream) {
  if (nc < 0 || !p_out || (nc > 0 && (!pos_c || !cp_pos)) || !(cs > 0.f) || nc >= 0x7fffffffLL) {
    set_last_error("create_control_points: bad arguments");
    return DBM_ERR_INVALID;
  }
  *p_out = 0;
  if (nc == 0) return DBM_OK;
  cudaStream_t s = (cudaStream_t)stream;
  uint32_t nu = 0;
  {
    Arena ar(s, index_bytes(nc, false) + 256);
    PointIndex ix;
    const PointSet pts{pos_c, nc, cs};
    uint32_t bounds[1][4];
    bool known = false;
    DBM_TRY(read_bounds(&pts, 1, ar, bounds, &known));
    DBM_TRY(build_index(pts, bounds[0], known, false, ar, &ix));
    uint32_t *flags, *d_nu;
    char* stmp;
    DBM_TRY(ar.get(&flags, nc));
    DBM_TRY(ar.get(&d_nu, 1));
    DBM_TRY(ar.get(&stmp, (int64_t)scan_tmp_bytes(nc)));
    k_heads<<<grid_for(nc), 256, 0, s>>>(ix.keys, nc, flags);
    DBM_LAUNCH_CHECK();
    DBM_TRY(scan_exclusive_u32(flags, flags, nc, nullptr, d_nu, stmp, s));
    k_centroid<<<grid_for(nc), 256, 0, s>>>(pos_c, ix, flags, cp_pos);
    DBM_LAUNCH_CHECK();
    DBM_CUDA(cudaMemcpyAsync(&nu, d_nu, 4, cudaMemcpyDeviceToHost, s));
  }
  DBM_CUDA(cudaStreamSynchronize(s));
  *p_out = nu;
  return DBM_OK;
}

int dbm_refine_control_points_f32(const float* cp, int64_t p, const float* pos_c, const float* val_c,
                                  const int32_t* dir_c, int64_t nc, float dx, int kappa_hard, float* new_pos,
                                  void* stream) {
  if (p < 0 || nc < 0 || nc > kMaxPoints || !(dx > 0.f) || (p > 0 && (!cp || !new_pos)) ||
      (nc > 0 && (!pos_c || !val_c || !dir_c))) {
    set_last_error("refine_control_points: bad arguments");
    return DBM_ERR_INVALID;
  }
  if (p == 0) return DBM_OK;
  cudaStream_t s = (cudaStream_t)stream;
  Arena ar(s, hash_bytes(nc));
  HashIndex ix;
  float4* items = nullptr;
  if (nc > 0) {
    DBM_TRY(build_hash(pos_c, nc, dx, ar, &ix));
    DBM_TRY(ar.get(&items, nc));
    k_pack_comps<<<grid_for(nc), 256, 0, s>>>(pos_c, val_c, dir_c, ix.order, ix.n, 1, items);
    DBM_LAUNCH_CHECK();
  }
  k_refine<<<grid_for(p), 256, 0, s>>>(cp, p, items, ix, dx, kappa_hard, new_pos);
  DBM_LAUNCH_CHECK();
  return DBM_OK;
}

int dbm_resample_f32(const float* pos_c, const float* val_c, const int32_t* dir_c, int64_t nc, const float* cp,
                     int64_t p, float dx, const float* f_rest, int lattice, float eps, float* out_pos, float* out_f,
                     void* stream) {
  DBM_TRY(check_2d(lattice));
  if (p < 0 || nc < 0 || p > kMaxPoints || nc > kMaxPoints || !(dx > 0.f) ||
      (p > 0 && (!cp || !out_pos || !out_f || !f_rest)) ||
      (nc > 0 && (!pos_c || !val_c || !dir_c))) {
    set_last_error("resample: bad arguments");
    return DBM_ERR_INVALID;
  }
  if (p == 0) return DBM_OK;
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  DBM_CUDA(cudaStreamIsCapturing(s, &cap));
  if (nc > 0 && cap != cudaStreamCaptureStatusNone) {  // as ever: the call waits for the stream
    set_last_error("resample: the call synchronises and cannot be captured");
    return DBM_ERR_STATE;
  }
  return dispatch_lattice(lattice, [&](auto tag) -> int {
    using LT = decltype(tag);
    if constexpr (LT::D == 2) {
      constexpr int Q = LT::Q;
      Arena ar(s, index_bytes(p, true) + index_bytes(nc, true) + 256);
      PointIndex cpi, ci;
      const PointSet sets[2] = {{cp, p, dx}, {pos_c, nc, dx}};
      uint32_t bounds[2][4];
      bool known = false;
      DBM_TRY(read_bounds(sets, nc > 0 ? 2 : 1, ar, bounds, &known));
      float2* cps;
      float4* comps = nullptr;
      float* sw = nullptr;
      uint32_t* em;
      DBM_TRY(build_index(sets[0], bounds[0], known, true, ar, &cpi));
      DBM_TRY(ar.get(&cps, p));
      DBM_TRY(ar.get(&em, p));
      k_pack_points<<<grid_for(p), 256, 0, s>>>(cp, cpi, cps);
      DBM_LAUNCH_CHECK();
      if (nc > 0) {
        DBM_TRY(build_index(sets[1], bounds[1], known, true, ar, &ci));
        DBM_TRY(ar.get(&comps, nc));
        DBM_TRY(ar.get(&sw, nc));
        k_pack_comps<<<grid_for(nc), 256, 0, s>>>(pos_c, val_c, dir_c, ci.order, ci.n, 0, comps);
        DBM_LAUNCH_CHECK();
        k_comp_sw<<<grid_for(nc), 256, 0, s>>>(comps, (uint32_t)nc, cps, cpi, dx, sw);
        DBM_LAUNCH_CHECK();
      }
      k_cp_gather<Q><<<grid_for(p), 256, 0, s>>>(cps, cpi, comps, sw, ci, dx, eps, em, out_pos, out_f);
      DBM_LAUNCH_CHECK();
      k_cp_fill<Q><<<grid_for(p), 256, 0, s>>>(cps, cpi, em, f_rest, dx, out_f);
      DBM_LAUNCH_CHECK();
    }
    return DBM_OK;
  });
}

}  // extern "C"
