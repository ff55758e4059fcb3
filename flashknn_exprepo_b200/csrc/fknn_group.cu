// Neighbour feature grouping: the gather that follows the kNN in point
// networks (Pointcept's pointops.grouping,
// Pointcept/libs/pointops/functions/grouping.py:36-60, called by
// knn_query_and_group, .../functions/utils.py:5-18).
//
// Forward: out[i, j, :] = [xyz[t] - new_xyz[i] | feat[t]] for t = idx[i, j]
// (the xyz part only with with_xyz); an index below 0 is padding and gives a
// zero row.  Every warp stores contiguous runs (rows of float4s, rows staged in
// shared memory or single words, by width and row count): a bandwidth-bound
// copy whose only re-read is the gathered feature row, served from L2 for the
// rows that neighbours share.
//
// Backward: grad_feat[t] = sum of grad_out[i, j, feat part] over the entries
// with idx[i, j] = t, grad_xyz[t] the same over the xyz part and
// grad_new_xyz[i] = -sum_j of the xyz part of row (i, j) over the valid j.
// The reference-side sums are made deterministic the same way as the
// distance backward (fknn_backward.cu): a counting sort of the entries by
// neighbour index, then one warp per support point that orders its segment
// by entry number and adds the rows in that order, so every output channel
// is summed in a fixed order -- no floating-point atomics.
#include <climits>
#include <cstdint>

#include "fknn_common.cuh"
#include "fknn_internal.h"
#include "fknn_sort.cuh"
#include "fknn_backward.h"
#include "fknn_group.h"

namespace fknn {

namespace {

constexpr uint32_t kNoEntry = 0xffffffffu;

__device__ __forceinline__ bool entry_ok(int32_t t, int64_t n, int* status) {
  if (t < 0) return false;
  if (t >= n) {
    raise_status(status, kStatusTable);
    return false;
  }
  return true;
}

}  // namespace

// ------------------------------------------------------------------ forward
// Bound by the output stream: m*k*(c+3)*4 bytes written once, the feature
// rows re-read from L2.

// Rows of whole aligned float4s (no xyz, c % 4 == 0): a group of tpr lanes
// (a power of two, tpr >= c/4 up to 32) copies one row, so a warp writes
// 32/tpr consecutive rows as one contiguous run; the row loop is unrolled so
// several independent gathers are in flight per thread.  Stores stream past
// L2 (st.global.cs): the output is written once and not re-read here.
__global__ void __launch_bounds__(256)
    kg_forward(const float* __restrict__ feat, int64_t n, int c, const int32_t* __restrict__ idx,
               int64_t rows, int tpr, float* __restrict__ out, int* status) {
  chain_wait();
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const int q4 = c >> 2;
  const int sub = threadIdx.x & (tpr - 1);
  const int64_t row_stride = stride / tpr;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / tpr; r < rows;
       r += row_stride) {
    const int32_t t = idx[r];
    const bool ok = entry_ok(t, n, sub == 0 ? status : nullptr);
    const float4* src = reinterpret_cast<const float4*>(feat + static_cast<int64_t>(t) * c);
    float4* dst = reinterpret_cast<float4*>(out) + r * q4;
    for (int q = sub; q < q4; q += tpr) __stcs(dst + q, ok ? __ldg(src + q) : zero);
  }
}

// Rows that are not whole float4s (the xyz part makes them c+3 floats wide):
// a warp gathers R consecutive rows (R % 4 == 0, so the run starts 16-byte
// aligned whatever the width) into its shared-memory slice -- 16-byte loads
// when the feature rows allow it -- and stores the run as float4s.  One
// word per thread, the row found by a 64-bit division, was bound by those
// instructions instead: 3.2 million rows of 3 + 64 floats (858 MB written)
// took 638 us; this takes 232 us (3.7 TB/s written; with streaming stores 271 us).
__global__ void __launch_bounds__(256)
    kg_forward_staged(const float* __restrict__ feat, int64_t n, int c,
                      const int32_t* __restrict__ idx, int64_t rows, int k,
                      const float* __restrict__ xyz, const float* __restrict__ new_xyz, int off,
                      int R, int tpr, float* __restrict__ out, int* status) {
  chain_wait();
  extern __shared__ __align__(16) float kg_smem[];
  const int lane = threadIdx.x & 31;
  const int cw = c + off;
  float* sm = kg_smem + static_cast<int64_t>(threadIdx.x >> 5) * R * cw;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  const int64_t groups = (rows + R - 1) / R;
  int64_t g = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  auto load_idx = [&](int64_t at) {
    return lane < R && at * R + lane < rows ? __ldg(idx + at * R + lane) : -1;
  };
  int32_t t_next = load_idx(g);
  for (; g < groups; g += warps) {
    const int64_t r0 = g * R;
    const int nr = rows - r0 < R ? static_cast<int>(rows - r0) : R;
    int32_t t = t_next;
    if (!entry_ok(t, n, status)) t = -1;
    t_next = load_idx(g + warps);  // in flight while this run is gathered and stored
    if (off) {  // R <= 8: one (row, axis) per lane
      const int r = lane / 3, a = lane - 3 * r;
      const int32_t tr = __shfl_sync(kFull, t, r);
      if (r < nr) {
        const int64_t i = static_cast<uint32_t>(r0 + r) / static_cast<uint32_t>(k);
        sm[r * cw + a] = tr < 0 ? 0.f
                                : __fsub_rn(__ldg(xyz + 3 * static_cast<int64_t>(tr) + a),
                                            __ldg(new_xyz + 3 * i + a));
      }
    }
    if (tpr) {  // whole float4s of features: tpr lanes per row
      const int q4 = c >> 2;
      const int sub = lane & (tpr - 1);
      const int step = 32 / tpr;
#pragma unroll 4
      for (int rr = 0; rr < R; rr += step) {
        const int r = rr + lane / tpr;
        const int32_t tr = __shfl_sync(kFull, t, r);
        const float4* src = reinterpret_cast<const float4*>(feat + static_cast<int64_t>(tr) * c);
        float* dst = sm + r * cw + off;
        if (r < nr)
          for (int q = sub; q < q4; q += tpr) {
            const float4 v = tr < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldg(src + q);
            dst[4 * q] = v.x;
            dst[4 * q + 1] = v.y;
            dst[4 * q + 2] = v.z;
            dst[4 * q + 3] = v.w;
          }
      }
    } else {
      for (int r = 0; r < nr; ++r) {
        const int32_t tr = __shfl_sync(kFull, t, r);
        const float* src = feat + static_cast<int64_t>(tr) * c;
        for (int q = lane; q < c; q += 32) sm[r * cw + off + q] = tr < 0 ? 0.f : __ldg(src + q);
      }
    }
    __syncwarp();
    const int words = nr * cw;
    float* dst = out + r0 * cw;
    for (int w = lane; w < (words >> 2); w += 32)
      reinterpret_cast<float4*>(dst)[w] = reinterpret_cast<const float4*>(sm)[w];
    if (lane < (words & 3)) dst[(words & ~3) + lane] = sm[(words & ~3) + lane];
    __syncwarp();
  }
}

// Any alignment: one warp per row, one word per lane.
__global__ void __launch_bounds__(256)
    kg_forward_rows(const float* __restrict__ feat, int64_t n, int c,
                    const int32_t* __restrict__ idx, int64_t rows, int k,
                    const float* __restrict__ xyz, const float* __restrict__ new_xyz, int off,
                    float* __restrict__ out, int* status) {
  chain_wait();
  const int lane = threadIdx.x & 31;
  const int cw = c + off;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
       r < rows; r += warps) {
    const int32_t t = idx[r];
    const bool ok = entry_ok(t, n, lane == 0 ? status : nullptr);
    for (int col = lane; col < cw; col += 32) {
      float v = 0.f;
      if (ok) {
        if (col < off)
          v = __fsub_rn(xyz[3 * static_cast<int64_t>(t) + col], new_xyz[3 * (r / k) + col]);
        else
          v = __ldg(feat + static_cast<int64_t>(t) * c + (col - off));
      }
      __stcs(out + r * cw + col, v);
    }
  }
}

// Narrow rows, flat over the output: thread t writes words t, t + threads, ...,
// so a warp's stores are one run and neighbouring lanes read one feature row.
// words < 2^31 (the caller launches slabs of rows); the row and the query each
// come from a multiplication (fast_div).  A row of one word or a few leaves
// most lanes of the two kernels above idle: 1.6 million rows took 111 us with
// one channel and 113 us with six, this takes 13 and 25 us.
__global__ void __launch_bounds__(256)
    kg_forward_words(const float* __restrict__ feat, int64_t n, int c,
                     const int32_t* __restrict__ idx, uint32_t words, FastDiv by_width,
                     uint32_t row0, FastDiv by_k, const float* __restrict__ xyz,
                     const float* __restrict__ new_xyz, int off, float* __restrict__ out,
                     int* status) {
  chain_wait();
  const uint32_t cw = static_cast<uint32_t>(c + off);
  const uint32_t stride = gridDim.x * blockDim.x;
#pragma unroll 4
  for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += stride) {
    const uint32_t r = fast_div(w, by_width);
    const int col = static_cast<int>(w - r * cw);
    const int32_t t = __ldg(idx + r);
    float v = 0.f;
    if (entry_ok(t, n, col == 0 ? status : nullptr)) {
      if (col >= off) {
        v = __ldg(feat + static_cast<int64_t>(t) * c + (col - off));
      } else {
        const int64_t i = fast_div(row0 + r, by_k);
        v = __fsub_rn(__ldg(xyz + 3 * static_cast<int64_t>(t) + col), __ldg(new_xyz + 3 * i + col));
      }
    }
    __stcs(out + w, v);
  }
}

// ----------------------------------------------------------------- backward

// count[t] = entries naming support point t.
__global__ void __launch_bounds__(256)
    kg_count(const int32_t* __restrict__ idx, int64_t total, int64_t n,
             uint32_t* __restrict__ count, int* status) {
  chain_wait();
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t t = idx[e];
    if (entry_ok(t, n, status)) atomicAdd(&count[t], 1u);
  }
}

__global__ void __launch_bounds__(256)
    kg_scatter(const int32_t* __restrict__ idx, int64_t total, int64_t n,
               uint32_t* __restrict__ cursor, uint32_t* __restrict__ seg) {
  chain_wait();
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t t = idx[e];
    if (t < 0 || t >= n) continue;
    seg[atomicSub(&cursor[t], 1u) - 1u] = static_cast<uint32_t>(e);
  }
}

// Ascending bitonic sort of one value per lane across the warp.
__device__ __forceinline__ uint32_t warp_sort_u32(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const uint32_t o = __shfl_xor_sync(kFull, v, stride);
      const bool up = (lane & size) == 0;        // ascending block
      const bool low = (lane & stride) == 0;      // lower partner
      v = (low == up) ? min(v, o) : max(v, o);
    }
  }
  return v;
}

template <int V>
struct Vec;
template <>
struct Vec<1> {
  using T = float;
  __device__ static T zero() { return 0.f; }
  __device__ static T add(T a, T b) { return __fadd_rn(a, b); }
};
template <>
struct Vec<2> {
  using T = float2;
  __device__ static T zero() { return make_float2(0.f, 0.f); }
  __device__ static T add(T a, T b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
};

// One warp per support point: its entries in ascending order, each row of
// grad_out added channel by channel in that order.  V channels per lane (2
// when the rows are whole float2s) and NC column blocks of 32*V channels, so
// rows of up to 32*V*NC channels are read in one walk over the entries.  Bound
// by reading grad_out once, at random rows.  Rows of several blocks: the rows
// of eight entries are loaded before they are added, in order, so 8*NC loads
// are in flight per lane; walking the entries again for every 32 channels,
// 3.2 million rows of 3 + 64 floats (858 MB) took 321 us, one walk with four
// rows in flight 296 us, with eight 218 us.  Rows of one block keep few loads
// in flight whatever the unroll, so warps count instead: four rows at a time
// in 32 registers (eight CTAs per SM).  The whole backward of 1.6 million
// rows, segments of 16, takes 90 us with 2 channels (eight rows in 63
// registers: 115) and 133 us with 64 (150).
template <int V, int NC>
__global__ void __launch_bounds__(256, NC == 1 ? 8 : (V == 1 ? 4 : 3))
    kg_support(const float* __restrict__ grad_out, int c, int with_xyz,
               const uint32_t* __restrict__ start, const uint32_t* __restrict__ seg, int64_t n,
               float* __restrict__ grad_feat, float* __restrict__ grad_xyz, int accumulate_xyz) {
  chain_wait();
  using VT = typename Vec<V>::T;
  constexpr int kRows = 8, kAhead = 8;
  const int lane = threadIdx.x & 31;
  const int off = with_xyz ? 3 : 0;
  const int cw = c + off;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t p = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
       p < n; p += warps) {
    const uint32_t s = start[p], len = start[p + 1] - s;
    // Entries of a short segment sorted across the lanes; a long one is
    // walked by repeated selection of the next larger entry.
    uint32_t mine = kNoEntry;
    if (len <= 32) mine = warp_sort_u32(lane < static_cast<int>(len) ? seg[s + lane] : kNoEntry);
    for (int c0 = 0; c0 < cw; c0 += 32 * V * NC) {
      VT acc[NC];
#pragma unroll
      for (int b = 0; b < NC; ++b) acc[b] = Vec<V>::zero();
      auto load = [&](uint32_t e, VT (&v)[NC]) {
        const float* row = grad_out + static_cast<int64_t>(e) * cw;
#pragma unroll
        for (int b = 0; b < NC; ++b) {
          const int col = c0 + (b * 32 + lane) * V;
          v[b] = col < cw ? *reinterpret_cast<const VT*>(row + col) : Vec<V>::zero();
        }
      };
      auto add = [&](const VT (&v)[NC]) {
#pragma unroll
        for (int b = 0; b < NC; ++b) acc[b] = Vec<V>::add(acc[b], v[b]);
      };
      if (len <= 32 && NC == 1) {
        const int col = c0 + lane * V;
        const bool live = col < cw;
        const float* at = grad_out + col;
        auto row = [&](uint32_t e) {
          return *reinterpret_cast<const VT*>(at + static_cast<int64_t>(e) * cw);
        };
        uint32_t r = 0;
        for (; r + 4 <= len; r += 4) {
          const uint32_t e0 = __shfl_sync(kFull, mine, r), e1 = __shfl_sync(kFull, mine, r + 1);
          const uint32_t e2 = __shfl_sync(kFull, mine, r + 2), e3 = __shfl_sync(kFull, mine, r + 3);
          if (live) {
            const VT v0 = row(e0), v1 = row(e1), v2 = row(e2), v3 = row(e3);
            acc[0] = Vec<V>::add(Vec<V>::add(Vec<V>::add(Vec<V>::add(acc[0], v0), v1), v2), v3);
          }
        }
        for (; r < len; ++r) {
          const uint32_t e = __shfl_sync(kFull, mine, r);
          if (live) acc[0] = Vec<V>::add(acc[0], row(e));
        }
      } else if (len <= 32) {
        for (uint32_t r = 0; r < len; r += kRows) {
          VT v[kRows][NC];
#pragma unroll
          for (int u = 0; u < kRows; ++u)
            if (r + u < len) load(__shfl_sync(kFull, mine, r + u), v[u]);
#pragma unroll
          for (int u = 0; u < kRows; ++u)
            if (r + u < len) add(v[u]);
        }
      } else {
        // The two smallest entries from `next` on, per pass over the segment:
        // as unsigned differences the ones before it wrap to above every entry
        // (entries are below 2^31).  Bound by the passes' loads (latency):
        // kAhead at a time, the backward of 800 thousand entries on 64 points
        // takes 68 ms with 3 channels, one entry a pass and one load at a time
        // 715 ms.
        uint32_t next = 0;
        for (uint32_t r = 0; r < len; r += 2) {
          uint32_t g0 = kNoEntry, g1 = kNoEntry, t = lane;
          const uint32_t* at = seg + s + lane;
          auto take = [&](uint32_t v) {
            g1 = min(g1, max(g0, v));
            g0 = min(g0, v);
          };
#pragma unroll 1
          for (; t + 32 * (kAhead - 1) < len; t += 32 * kAhead, at += 32 * kAhead) {
            uint32_t v[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) v[u] = __ldg(at + 32 * u);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) take(v[u] - next);
          }
#pragma unroll 1
          for (; t < len; t += 32, at += 32) take(__ldg(at) - next);
          const uint32_t first = __reduce_min_sync(kFull, g0);
          const uint32_t second = __reduce_min_sync(kFull, g0 == first ? g1 : g0);
          VT v[NC];
          load(next + first, v);
          add(v);
          if (r + 1 < len) {
            load(next + second, v);
            add(v);
          }
          next += second + 1;
        }
      }
#pragma unroll
      for (int b = 0; b < NC; ++b) {
        const int col = c0 + (b * 32 + lane) * V;
        if (col >= cw) continue;
        if constexpr (V == 1) {
          if (col < off) {
            if (grad_xyz) {
              float* g = grad_xyz + 3 * p + col;
              *g = accumulate_xyz ? __fadd_rn(*g, acc[b]) : acc[b];
            }
          } else {
            grad_feat[p * c + (col - off)] = acc[b];
          }
        } else {  // no xyz part: channel col of the row is channel col of feat
          *reinterpret_cast<VT*>(grad_feat + p * c + col) = acc[b];
        }
      }
    }
  }
}

// grad_new_xyz[i] = -sum_j over valid entries of the xyz part of row (i, j),
// j ascending.  A warp takes 32 / kp queries (kp: k rounded up to a power of
// two, at most 32), one row per lane, so the 12 bytes of 32 rows are in
// flight at once; each query's lane 0 then subtracts its rows in order.  One
// thread per query, one row in flight at a time, took 85 us for 3.2 million
// rows of 268 bytes; this takes 70 us.
__global__ void __launch_bounds__(256)
    kg_query(const float* __restrict__ grad_out, int c, const int32_t* __restrict__ idx,
             int64_t m, int k, int64_t n, int kp, float* __restrict__ grad_new_xyz,
             int accumulate) {
  chain_wait();
  const int lane = threadIdx.x & 31;
  const int sub = lane & (kp - 1);
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t i = warp * (32 / kp) + lane / kp;
  const int cw = c + 3;
  float g[3] = {0.f, 0.f, 0.f};
  for (int j0 = 0; j0 < k; j0 += kp) {
    const int j = j0 + sub;
    float v[3] = {0.f, 0.f, 0.f};
    bool ok = false;
    if (i < m && j < k) {
      const int32_t t = idx[i * k + j];
      ok = t >= 0 && t < n;
      if (ok) {
        const float* row = grad_out + (i * k + j) * cw;
#pragma unroll
        for (int a = 0; a < 3; ++a) v[a] = __ldg(row + a);
      }
    }
    const uint32_t valid = __ballot_sync(kFull, ok) >> (lane - sub);
    for (int r = 0; r < kp; ++r) {
      const bool take = (valid >> r) & 1u;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float x = __shfl_sync(kFull, v[a], r, kp);
        if (take) g[a] = __fsub_rn(g[a], x);
      }
    }
  }
  if (i >= m || sub != 0) return;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    grad_new_xyz[3 * i + a] = accumulate ? __fadd_rn(grad_new_xyz[3 * i + a], g[a]) : g[a];
}

// --------------------------------------------------------------- host side

namespace {

struct GBufs {
  Meta* meta;
  uint32_t* count;
  uint32_t* start;
  uint32_t* cursor;
  uint32_t* tiles;
  uint32_t* seg;
};

GBufs glayout(void* ws, int64_t rows, int64_t n, size_t* bytes) {
  Arena a(ws);
  GBufs b{};
  b.meta = a.take<Meta>(1);
  b.count = a.take<uint32_t>(n);
  b.start = a.take<uint32_t>(n + 1);
  b.cursor = a.take<uint32_t>(n);
  b.tiles = a.take<uint32_t>(segment_tiles(n));
  b.seg = a.take<uint32_t>(rows);
  if (bytes) *bytes = a.used + 256;
  return b;
}

inline int capped_blocks(int64_t threads) {
  const int64_t b = ceil_div(threads > 0 ? threads : 1, 256);
  return static_cast<int>(b < 148 * 32 ? b : 148 * 32);
}

inline int capped_warp_blocks(int64_t rows) {
  const int64_t b = ceil_div(rows > 0 ? rows : 1, 8);  // 8 warps per 256-thread block
  return static_cast<int>(b < 148 * 16 ? b : 148 * 16);
}

}  // namespace

size_t group_workspace_bytes(int64_t rows, int64_t n) {
  size_t bytes = 0;
  glayout(nullptr, rows, n, &bytes);
  return bytes;
}

int run_group_forward(const GroupArgs& g, void* ws, size_t ws_bytes, cudaStream_t s,
                      int* launches) {
  size_t need = 0;
  GBufs b = glayout(ws, g.m * g.k, g.n, &need);
  if (ws_bytes < need) return FKNN_ERR_WORKSPACE;
  cudaError_t e = cudaMemsetAsync(b.meta, 0, sizeof(Meta), s);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return FKNN_ERR_CUDA;
  }
  const int64_t rows = g.m * g.k;
  int nl = 0;
  if (rows > 0) {
    const int off = g.with_xyz ? 3 : 0, cw = g.c + off;
    const bool out16 = reinterpret_cast<uintptr_t>(g.out) % 16 == 0;
    const bool feat4 = g.c % 4 == 0 && reinterpret_cast<uintptr_t>(g.feat) % 16 == 0;
    int tpr = 0;  // lanes per row of float4 features
    if (feat4) {
      tpr = 1;
      while (tpr < 32 && tpr < g.c / 4) tpr <<= 1;
    }
    // Rows per warp of the staged path: 8 while a CTA's eight slices stay
    // within 40 KB (five CTAs per SM), 4 up to the 48 KB that need no opt-in;
    // wider rows amortise the per-row work by themselves.
    const int R = cw <= 160 ? 8 : (cw <= 384 ? 4 : 0);
    // Staged runs pay where a feature row fills a good part of a warp's loads
    // and there are enough rows for its warps.  Float4 features from 16
    // channels up: with xyz, 1.6 million rows take 66 us (word by word 74) at
    // 16 channels, but 60 (46) at 8.  Other features from 57 up: 960 thousand
    // rows take 105 us (word by word 111) at 57 channels and 111 (97) at 49.
    // Fewer rows leave warps without a run, and each run is a longer chain of
    // loads: 960 rows of 3 + 16 take 6.4 us (4.6 word by word), 16 thousand
    // rows of 3 + 97 take 14.1 us (8.5 by warps of one row).
    const bool wide = g.c > 56;
    const bool staged = out16 && R && (feat4 ? g.c >= 16 && rows >= 4096 : wide && rows >= 65536);
    if (feat4 && out16 && !off) {
      launch_chained(kg_forward, capped_blocks(rows * tpr), 256, 0, s, g.feat, g.n, g.c, g.idx,
                     rows, tpr, g.out, &b.meta->status);
    } else if (staged) {
      launch_chained(kg_forward_staged, capped_warp_blocks(ceil_div(rows, R)), 256,
                     sizeof(float) * 8 * R * cw, s, g.feat, g.n, g.c, g.idx, rows, g.k, g.xyz,
                     g.new_xyz, off, R, tpr, g.out, &b.meta->status);
    } else if (wide) {
      launch_chained(kg_forward_rows, capped_warp_blocks(rows), 256, 0, s, g.feat, g.n, g.c, g.idx,
                     rows, g.k, g.xyz, g.new_xyz, off, g.out, &b.meta->status);
    } else {
      const int64_t slab = INT32_MAX / cw;  // rows per launch
      for (int64_t r0 = 0; r0 < rows; r0 += slab) {
        const int64_t words = (rows - r0 < slab ? rows - r0 : slab) * cw;
        if (r0 > 0) ++nl;
        launch_chained(kg_forward_words, capped_blocks(words), 256, 0, s, g.feat, g.n, g.c,
                       g.idx + r0, static_cast<uint32_t>(words),
                       make_fast_div(static_cast<uint32_t>(cw)), static_cast<uint32_t>(r0),
                       make_fast_div(static_cast<uint32_t>(g.k)), g.xyz, g.new_xyz, off,
                       g.out + r0 * cw, &b.meta->status);
      }
    }
    ++nl;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return FKNN_ERR_CUDA;
  }
  if (launches) *launches = nl;
  return FKNN_OK;
}

int run_group_backward(const GroupArgs& g, void* ws, size_t ws_bytes, cudaStream_t s,
                       int* launches) {
  size_t need = 0;
  GBufs b = glayout(ws, g.m * g.k, g.n, &need);
  if (ws_bytes < need) return FKNN_ERR_WORKSPACE;
  const int64_t rows = g.m * g.k;
  cudaError_t e = cudaMemsetAsync(b.meta, 0, sizeof(Meta), s);
  if (e == cudaSuccess && g.n > 0) e = cudaMemsetAsync(b.count, 0, sizeof(uint32_t) * g.n, s);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return FKNN_ERR_CUDA;
  }
  int nl = 0;
  if (g.n > 0 && g.grad_feat) {
    const int64_t eb = ceil_div(rows > 0 ? rows : 1, 256);
    const int eblocks = static_cast<int>(eb < 8192 ? eb : 8192);
    if (rows > 0) {
      launch_chained(kg_count, eblocks, 256, 0, s, g.idx, rows, g.n, b.count, &b.meta->status);
      ++nl;
    }
    nl += launch_segment_starts(b.count, g.n, b.tiles, &b.meta->n_groups, b.start, b.cursor, s);
    if (rows > 0) {
      launch_chained(kg_scatter, eblocks, 256, 0, s, g.idx, rows, g.n, b.cursor, b.seg);
      ++nl;
    }
    const bool v2 = !g.with_xyz && g.c % 2 == 0 &&
                    reinterpret_cast<uintptr_t>(g.grad_out) % 8 == 0 &&
                    reinterpret_cast<uintptr_t>(g.grad_feat) % 8 == 0;
    const int cw = g.c + (g.with_xyz ? 3 : 0);
    const int blocks = static_cast<int>(ceil_div(cw, v2 ? 64 : 32));  // of channels
    auto support = [&](auto kernel) {
      launch_chained(kernel, capped_warp_blocks(g.n), 256, 0, s, g.grad_out, g.c, g.with_xyz,
                     b.start, b.seg, g.n, g.grad_feat, g.grad_xyz, g.accumulate_xyz);
    };
    if (v2)
      blocks <= 1 ? support(kg_support<2, 1>) : support(kg_support<2, 2>);
    else
      blocks <= 1   ? support(kg_support<1, 1>)
      : blocks == 2 ? support(kg_support<1, 2>)
                    : support(kg_support<1, 3>);
    ++nl;
  }
  if (g.with_xyz && g.grad_new_xyz && g.m > 0) {
    int kp = 1;
    while (kp < 32 && kp < g.k) kp <<= 1;
    launch_chained(kg_query, static_cast<int>(ceil_div(g.m, 256 / kp)), 256, 0, s, g.grad_out, g.c,
                   g.idx, g.m, g.k, g.n, kp, g.grad_new_xyz, g.accumulate_new_xyz);
    ++nl;
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return FKNN_ERR_CUDA;
  }
  if (launches) *launches = nl;
  return FKNN_OK;
}

}  // namespace fknn
