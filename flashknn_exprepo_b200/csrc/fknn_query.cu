// Persistent grid-kNN query kernel for sm_100a.
//
// Semantics follow the reference production kernel
// (FlashKNN/csrc/flash_knn_query_dynamic_load.cu:469-652): every query gets
// the exact K smallest FP32 squared distances among the points of the 27
// candidate runs of its group, strict acceptance d < cut_r2, ascending output,
// (pad index, +inf) padding.  Equal distances are ordered by the lower index
// (the reference leaves their order to its network layout).
//
// Execution model (B200-first, not the reference's block-per-parent loop):
//   * persistent CTAs; each warp pulls work items from a device queue
//     (atomicAdd on Meta::queue_head);
//   * packed item: up to 32 consecutive queries from up to 16 consecutive
//     groups, one query per lane.  Each group's 27 runs are staged into the
//     warp's shared-memory tile, one 16-byte cp.async per record (the runs
//     are short: a bulk copy each, issued lane after lane, took longer).
//     Each group's candidates are then counting-sorted (32 buckets of squared
//     distance) by distance to the centre of the group's queries, so every
//     lane meets near candidates first and stops at the first bucket whose
//     lower distance bound exceeds its current K-th distance (triangle
//     inequality, with a safety margin for FP32 rounding).  The candidates
//     are taken in blocks, sorted and merged into the lane's list as 32-bit
//     keys (select_blocks);
//   * chunked item: one group with more candidates than a tile; G lanes per
//     query split its candidates, streamed tile by tile by non-multicast
//     cp.async.bulk copies on the warp's mbarrier, and the G partial
//     lists are merged with xor-shuffle bitonic merges;
//   * results come from packed u64 keys (distance bits << 32 | index), so
//     ordering is exact including ties; rows are written straight to the caller's
//     row / index space.
#include <algorithm>
#include <cfloat>
#include <mutex>
#include <vector>

#include "fknn_common.cuh"
#include "fknn_networks.cuh"
#include "fknn_internal.h"

namespace fknn {

// Larger than every key (the distance bits of a key are those of a finite
// float) and, read as a double, +inf: see key_less.
constexpr uint64_t kEmpty = 0x7ff0000000000000ull;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr int kBuckets = 32;
constexpr int kMaxOrderedGroup = 4096;  // queries: larger chunked groups keep record order

// One group of the current packed item (shared memory, per warp).
struct __align__(16) GroupSlot {
  int seg;    // first tile slot of the group's candidates
  int len;    // number of candidates
  int a, b;   // the group's query range inside the item (query-record positions)
};

// A lane's group while its query is scanned.
struct LaneGroup {
  int len;                   // candidates to scan
  const uint16_t* srt;       // their tile positions in bucket order
  const uint16_t* bstart;    // first of every bucket
  float inv_w2;              // 1 / bucket width in squared distance
  float rq;                  // distance of the query to the group's centre (a little above)
  float eps;                 // absolute margin of the early-exit bound
};

// Staging buffers per warp (the autotuner's depth axis: 1 or 2).
constexpr int kMaxStaging = 2;

// Slots for the sorted tile positions of an item's groups: each group's start
// is a multiple of 8, so eight positions are one 16-byte load.
__host__ __device__ constexpr size_t sorted_slots(int T) {
  return static_cast<size_t>(T) + 8 * kMaxGroupsPerItem;
}

// Bytes of one warp's shared-memory region: `depth` staging buffers of T
// records (tile, group slots, flag) and one set of sort scratch.
__host__ __device__ constexpr size_t warp_smem_bytes(int T, int depth) {
  return ((static_cast<size_t>(depth) *
               (static_cast<size_t>(T) * 16 + kMaxGroupsPerItem * sizeof(GroupSlot) + 32) +
           sorted_slots(T) * 2 + static_cast<size_t>(T) * 2 +
           kMaxGroupsPerItem * (kBuckets + 1) * 2 + kBuckets * 4 + 127) /
          128) *
         128;
}

__device__ __forceinline__ uint64_t key_min(uint64_t a, uint64_t b) {
  return key_less(a, b) ? a : b;
}

__device__ __forceinline__ uint64_t make_key(float d, float w) {
  return (static_cast<uint64_t>(__float_as_uint(d)) << 32) |
         static_cast<uint32_t>(__float_as_int(w));
}

// Insert x into the ascending list L, dropping the largest entry.  Slot j
// becomes min(L[j], max(x, L[j-1])): every slot is computed from the old
// list, so the network has no serial dependency.  x == kEmpty is a no-op.
template <int KCAP>
__device__ __forceinline__ void list_insert(uint64_t (&L)[KCAP], uint64_t x) {
#pragma unroll
  for (int j = KCAP - 1; j >= 1; --j) {
    const bool cj = key_less(x, L[j]);
    const bool cm = key_less(x, L[j - 1]);
    L[j] = cj ? (cm ? L[j - 1] : x) : L[j];
  }
  L[0] = key_min(x, L[0]);
}

template <int KCAP>
__device__ __forceinline__ void cas(uint64_t (&L)[KCAP], int i, int j, bool ascending) {
  const uint64_t a = L[i], b = L[j];
  const bool sw = ascending ? key_less(b, a) : key_less(a, b);
  L[i] = sw ? b : a;
  L[j] = sw ? a : b;
}

template <int KCAP>
__device__ __forceinline__ void bitonic_clean_ascending(uint64_t (&L)[KCAP]) {
#pragma unroll
  for (int st = KCAP / 2; st > 0; st >>= 1) {
#pragma unroll
    for (int j = 0; j < KCAP; ++j)
      if ((j & st) == 0) cas<KCAP>(L, j, j + st, true);
  }
}

__device__ __forceinline__ uint64_t shfl_xor_u64(uint64_t v, int mask) {
  const uint32_t lo = __shfl_xor_sync(kFull, static_cast<uint32_t>(v), mask);
  const uint32_t hi = __shfl_xor_sync(kFull, static_cast<uint32_t>(v >> 32), mask);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Keep the KCAP smallest of this lane's list and the list of lane ^ mask.
template <int KCAP>
__device__ __forceinline__ void merge_with_lane(uint64_t (&L)[KCAP], int mask) {
  if constexpr (KCAP == 1) {
    L[0] = key_min(L[0], shfl_xor_u64(L[0], mask));
  } else {
#pragma unroll
    for (int j = 0; j < KCAP / 2; ++j) {
      const uint64_t a = L[j], b = L[KCAP - 1 - j];
      const uint64_t pa = shfl_xor_u64(b, mask);  // partner's L[KCAP-1-j]
      const uint64_t pb = shfl_xor_u64(a, mask);  // partner's L[j]
      L[j] = key_min(a, pa);
      L[KCAP - 1 - j] = key_min(b, pb);
    }
    bitonic_clean_ascending<KCAP>(L);
  }
}

// Acceptance of a candidate at squared distance d (>= +0 or NaN): d < cut_r2
// and d no larger than the current K-th.  For non-negative floats the order
// of the bit patterns is the order of the values, so d < cut_r2 is
// bits(d) <= bits(cut_r2) - 1 and both tests fold into one unsigned
// threshold min(K-th bits, cut_limit).  NaN and +inf lie above every limit.
// cut_r2 <= 0 (or NaN) accepts nothing: queries then take no candidate.
__device__ __forceinline__ bool cut_accepts_any(float cut_r2) { return cut_r2 > 0.f; }

__device__ __forceinline__ uint32_t cut_limit(float cut_r2) {
  return __float_as_uint(cut_r2) - 1u;  // valid when cut_accepts_any(cut_r2)
}

__device__ __forceinline__ uint32_t kth_limit(uint64_t last, uint32_t cut_lim) {
  return min(static_cast<uint32_t>(last >> 32), cut_lim);
}

__device__ __forceinline__ int ceil_log2(int v) { return v <= 1 ? 0 : 32 - __clz(v - 1); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(kFull, v, s);
  return v;
}

// Warp-wide minimum / maximum of a float in one instruction (NaN: ignored).
__device__ __forceinline__ float redux_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ float redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, s));
  return v;
}

// A little above sqrt(d): d * rsqrt(d) is within a few ulp of it, far inside
// the 1e-4 margin.  d >= FLT_MIN keeps a distance of 0 (a query on a support
// point) or a subnormal one bounded from above, and +inf gives NaN, which
// skips no bucket.
__device__ __forceinline__ float sqrt_above(float d) {
  const float m = fmaxf(d, FLT_MIN);
  return m * rsqrtf(m) * 1.0001f;
}

// First sorted position whose bucket cannot hold a candidate closer than the
// lane's current K-th distance `kth`.  Buckets are uniform in the squared
// distance to the group's centre: a candidate in bucket b lies at least
// sqrt(b*w2) from the centre, hence at least sqrt(b*w2) - rq from the
// query; buckets with b*w2 > (rq + sqrt(thr))^2 (plus margins) are skipped.
__device__ __forceinline__ int stop_position(float kth, const LaneGroup& s) {
  const float reach = s.rq + sqrt_above(kth) + s.eps;
  const float lim = reach * reach * s.inv_w2;
  if (!(lim < static_cast<float>(kBuckets - 1))) return s.len;
  return s.bstart[static_cast<int>(lim) + 1];
}

// The work item a warp takes next, fetched while it finishes the current one:
// the queue's atomic, then the item's descriptor, are in flight meanwhile.
// The pop comes late in an item, so that a warp never holds an item it is far
// from starting while others run out.
struct NextItem {
  bool wanted;  // false: the item is taken elsewhere (staging depth 2)
  int popped;   // lane 0
  int item;
  int4 it;
  int gs, ge, row;  // lane's group: query range and runs row (garbage past the item's groups)
  __device__ __forceinline__ void pop(Meta* meta) {
    if (wanted && (threadIdx.x & 31) == 0) popped = atomicAdd(&meta->queue_head, 1);
  }
  __device__ __forceinline__ void load(const QueryLaunch& a, int n_items) {
    if (!wanted) return;
    item = __shfl_sync(kFull, popped, 0);
    if (item < n_items) it = a.items[item];
  }
  // The groups of a well-formed item, one per lane (stage_item checks it).
  __device__ __forceinline__ void load_groups(const QueryLaunch& a, int n_items, int n_groups) {
    if (!wanted || item >= n_items) return;
    const int lane = threadIdx.x & 31;
    const int g = it.z + lane;
    if (it.z >= 0 && it.z < n_groups && lane < (it.w & 0xffff) && g < n_groups) {
      gs = a.group_start[g];
      ge = a.group_end[g];
      row = a.group_row ? a.group_row[g] : g;
    }
  }
};

// Order-preserving 32-bit keys of the packed scan: the squared distance's
// bits with the low ones replaced by the candidate's tile position, so a compare-exchange is a min and a max.
constexpr uint32_t kNone32 = ~0u;
constexpr uint32_t kInfBits = 0x7f800000u;

// Merges the ascending block X into the ascending list L, keeping the KCAP
// smallest; dropped = the smallest key ever left out.
template <int KCAP, int B>
__device__ __forceinline__ void merge_block(uint32_t (&L)[KCAP], const uint32_t (&X)[B],
                                            uint32_t& dropped) {
  constexpr int o = KCAP - B;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    const uint32_t l = L[o + j], x = X[B - 1 - j];
    L[o + j] = min(l, x);
    dropped = min(dropped, max(l, x));
  }
#pragma unroll
  for (int st = KCAP / 2; st > 0; st >>= 1) {
#pragma unroll
    for (int j = 0; j < KCAP; ++j)
      if ((j & st) == 0) cas_up<KCAP>(L, j, j + st);
  }
}

// Adds the candidates of one truncated distance, srt[0, end), to the list by
// their exact keys: the repair of an ambiguous k-th entry (select_blocks).  32
// positions are tested first, then every lane inserts its own next member, so
// the insertions number the largest lane's members instead of one for every
// candidate that some lane of the warp takes.  Where every query is such a
// one (a lattice of 262 thousand points, 216 candidates) the call takes 197 us
// at K=16 and 815 at K=64, inserting as the scan meets members 272 and 1747.
// A second pass of the block selection over the class, with whole keys,
// took 199 and 1127.
template <int KCAP, typename DistBits>
__device__ __forceinline__ void add_class(uint64_t (&E)[KCAP], const uint16_t* srt, int end,
                                          uint32_t cls, uint32_t pos_mask, uint32_t cut_lim,
                                          const DistBits& dist_bits) {
#pragma unroll 1
  for (int t0 = 0; __any_sync(kFull, t0 < end); t0 += 32) {
    uint32_t hits = 0u;  // members among srt[t0, t0 + 32)
#pragma unroll 1
    for (int h = 0; h < 32 && t0 + h < end; h += 8) {
      const uint4 p = *reinterpret_cast<const uint4*>(srt + t0 + h);
      const uint32_t pw[4] = {p.x, p.y, p.z, p.w};
      uint32_t m = 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float4 c;
        const uint32_t d = dist_bits((u & 1) ? pw[u >> 1] >> 16 : pw[u >> 1] & 0xffffu, c);
        if (d <= cut_lim && (d & ~pos_mask) == cls) m |= 1u << u;
      }
      hits |= m << h;
    }
    while (__any_sync(kFull, hits != 0u)) {
      uint64_t x = kEmpty;
      if (hits) {
        float4 c;
        const uint32_t d = dist_bits(srt[t0 + __ffs(hits) - 1], c);
        x = make_key(__uint_as_float(d), c.w);
        hits &= hits - 1u;
      }
      list_insert<KCAP>(E, x);
    }
  }
}

// The same out of line, the list in local memory, so that its registers do not
// add to the scan's: lists of 64 took 602 us inline over 262 thousand points
// without ties, 529 so; short lists gain nothing from it.
template <int KCAP>
__device__ __noinline__ void add_class_apart(uint64_t* list, const float4* tile,
                                             const uint16_t* srt, int end, uint32_t cls,
                                             uint32_t pos_mask, uint32_t cut_lim, float qx,
                                             float qy, float qz) {
  auto dist_bits = [&](uint32_t pos, float4& c) {
    c = tile[pos];
    return __float_as_uint(sq_dist(c.x, c.y, c.z, qx, qy, qz));
  };
  uint64_t E[KCAP];
#pragma unroll
  for (int j = 0; j < KCAP; ++j) E[j] = list[j];
  add_class<KCAP>(E, srt, end, cls, pos_mask, cut_lim, dist_bits);
#pragma unroll
  for (int j = 0; j < KCAP; ++j) list[j] = E[j];
}

// The lane's KCAP smallest candidates as exact keys (distance bits << 32 |
// index), ascending; entries from k on may be left out.
//
// Bound by instruction issue.  The scan sorts blocks of B candidates as
// 32-bit keys and merges each block into the list (a minimum and a maximum
// per compare-exchange), in place of one warp-wide 64-bit insertion per
// accepted candidate of any lane: 309 -> 180 warp instructions per query at
// K=16.  The first block goes through the same loop as the rest (no
// separate fill): the code the warps share has to stay small, since straight
// copies of it made instruction fetch the first stall (2.8 of 10 cycles per
// instruction).  With the staging, the sort and a shorter construction the
// whole call over the 16-cloud batch (1.46 million queries, K=16) went from
// 861 to 553 us, over 700 thousand queries at K=32 from 880 to 476 us, over 300
// thousand at K=64 from 1182 to 455 us.  Short lists gain the same way: 300
// thousand queries at K=3 125 -> 98 us, 700 thousand at K=1 323 -> 302 us.  The
// keys drop the low 9 or 10 bits of the distance, so the exact keys of the list
// are computed at the end and neighbours that the truncation left in the
// wrong order are exchanged; a lane whose k-th entry shares its truncated
// distance with a candidate it left out collects the candidates of that one
// truncated distance again, with exact keys (add_class).
template <int KCAP, typename DistBits>
__device__ __forceinline__ void select_blocks(uint64_t (&E)[KCAP], const LaneGroup& g, int k,
                                              uint32_t pos_mask, uint32_t cut_lim,
                                              DistBits& dist_bits, const QueryLaunch& a,
                                              int n_items, uint32_t none, NextItem& next,
                                              const float4* tile, const float4& q) {
  constexpr int B = KCAP <= 16 ? 8 : 16;
  constexpr int M = KCAP < B ? KCAP : B;  // of a block that the list can take
  const uint16_t* srt = g.srt;
  uint32_t L[KCAP];
  uint32_t dropped = kNone32, last = kNone32;
#pragma unroll
  for (int j = 0; j < KCAP; ++j) L[j] = kNone32;
  int stop = min(g.len, stop_position(__uint_as_float(cut_lim), g));
#pragma unroll 1
  for (int t0 = 0; __any_sync(kFull, t0 < stop); t0 += B) {
    uint32_t X[B];
#pragma unroll
    for (int h = 0; h < B; h += 8) {  // eight positions per 16-byte load
      uint4 p = make_uint4(none, none, none, none);
      if (t0 + h < stop) p = *reinterpret_cast<const uint4*>(srt + t0 + h);
      const uint32_t pw[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        float4 c;
        const uint32_t pos = (u & 1) ? pw[u >> 1] >> 16 : pw[u >> 1] & 0xffffu;
        X[h + u] = (dist_bits(pos, c) & ~pos_mask) | pos;
      }
    }
    sort_network<B, 0, B>(X);
    if (__any_sync(kFull, X[0] < last)) {
      uint32_t Y[M];
#pragma unroll
      for (int j = 0; j < M; ++j) Y[j] = X[j];
      if (M < B) dropped = min(dropped, X[M % B]);
      merge_block<KCAP, M>(L, Y, dropped);
      last = L[KCAP - 1];
      if (k < KCAP) {
#pragma unroll
        for (int j = 0; j < KCAP - 1; ++j)
          if (j == k - 1) last = L[j];
      }
      stop = min(stop, stop_position(__uint_as_float(min(last | pos_mask, cut_lim)), g));
    } else {
      dropped = min(dropped, X[0]);
    }
  }
  next.pop(a.meta);
  // Exact keys.  Candidates outside the cut (NaN: no candidate) went through
  // the list like the others, behind every one inside; they end here, and so
  // do the entries of an ambiguous k-th truncated distance.
  const bool ambiguous =
      (last & ~pos_mask) <= cut_lim && ((dropped ^ last) & ~pos_mask) == 0u;
  const uint32_t limit = ambiguous ? last & ~pos_mask : kInfBits;
#pragma unroll
  for (int j = 0; j < KCAP; ++j) {
    E[j] = kEmpty;
    if (L[j] < limit) {
      float4 c;
      const uint32_t d = dist_bits(L[j] & pos_mask, c);
      if (d <= cut_lim) E[j] = make_key(__uint_as_float(d), c.w);
    }
  }
  next.load(a, n_items);
  while (true) {
    bool sorted = true;
#pragma unroll
    for (int j = 0; j + 1 < KCAP; ++j) sorted = sorted && !key_less(E[j + 1], E[j]);
    if (__all_sync(kFull, sorted)) break;
#pragma unroll
    for (int j = 0; j + 1 < KCAP; j += 2) cas_up<KCAP>(E, j, j + 1);
#pragma unroll
    for (int j = 1; j + 1 < KCAP; j += 2) cas_up<KCAP>(E, j, j + 1);
  }
  if (__any_sync(kFull, ambiguous)) {
    const int end = ambiguous ? stop : 0;
    if constexpr (KCAP <= 16) {
      add_class<KCAP>(E, srt, end, limit, pos_mask, cut_lim, dist_bits);
    } else {
      uint64_t list[KCAP];
#pragma unroll
      for (int j = 0; j < KCAP; ++j) list[j] = E[j];
      add_class_apart<KCAP>(list, tile, srt, end, limit, pos_mask, cut_lim, q.x, q.y, q.z);
#pragma unroll
      for (int j = 0; j < KCAP; ++j) E[j] = list[j];
    }
  }
}

template <typename IdxT, int KCAP, bool EXACT>
__device__ __forceinline__ void write_row(const QueryLaunch& a, const uint64_t (&L)[KCAP], int row,
                                          int k) {
  if (row < 0 || row >= a.n_rows) {
    raise_status(&a.meta->status, kStatusTable);
    return;
  }
  int64_t pad;
  switch (a.pad_mode) {
    case kPadArray64: pad = static_cast<const int64_t*>(a.pad)[row]; break;
    case kPadArray32: pad = static_cast<const int32_t*>(a.pad)[row]; break;
    case kPadMinusOne: pad = -1; break;
    default: pad = row; break;
  }
  IdxT* io = static_cast<IdxT*>(a.idx_out) + static_cast<int64_t>(row) * k;
  float* dout = a.dist_out + static_cast<int64_t>(row) * k;
  if (EXACT && (KCAP % 4) == 0 && a.vec_ok) {
#pragma unroll
    for (int j = 0; j < KCAP; j += 4) {
      float4 dv;
      IdxT iv[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint64_t e = L[j + t];
        const bool empty = e == kEmpty;
        iv[t] = empty ? static_cast<IdxT>(pad) : static_cast<IdxT>(static_cast<int32_t>(e));
        reinterpret_cast<float*>(&dv)[t] =
            empty ? __int_as_float(0x7f800000) : __uint_as_float(static_cast<uint32_t>(e >> 32));
      }
      *reinterpret_cast<float4*>(dout + j) = dv;
      if constexpr (sizeof(IdxT) == 4) {
        *reinterpret_cast<int4*>(io + j) = make_int4(iv[0], iv[1], iv[2], iv[3]);
      } else {
        *reinterpret_cast<longlong2*>(io + j) = make_longlong2(iv[0], iv[1]);
        *reinterpret_cast<longlong2*>(io + j + 2) = make_longlong2(iv[2], iv[3]);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < KCAP; ++j) {
      if (j < k) {
        const uint64_t e = L[j];
        const bool empty = e == kEmpty;
        io[j] = empty ? static_cast<IdxT>(pad) : static_cast<IdxT>(static_cast<int32_t>(e));
        dout[j] = empty ? __int_as_float(0x7f800000) : __uint_as_float(static_cast<uint32_t>(e >> 32));
      }
    }
  }
}

// A run from the caller's tables, emptied (and reported) when it leaves the
// support records.
__device__ __forceinline__ int2 checked_run(const QueryLaunch& a, int2 run) {
  if (run.y < 0 || run.x < 0 || static_cast<int64_t>(run.x) + run.y > a.n_support) {
    raise_status(&a.meta->status, kStatusTable);
    run.y = 0;
  }
  return run;
}

__device__ __forceinline__ int2 load_run(const QueryLaunch& a, int row, int lane) {
  int2 run = make_int2(0, 0);
  if (lane < kNeighbours) run = a.runs[static_cast<int64_t>(row) * kNeighbours + lane];
  return checked_run(a, run);
}

// Record of query qi of a chunked item (queries q0 .. q0+qn-1 of group g0):
// the group's queries taken in octant-major order around their centroid
// (the packer cuts a chunked group into consecutive items from its first
// query, so the item covering positions [q0 - start, q0 - start + qn) of
// that order takes those queries), so every query belongs to exactly one
// item and an item's queries are close together.  A group the item holds
// whole, or one of more than kMaxOrderedGroup queries, keeps record order.
// qlist: 32 ints of scratch; hist: 8 counters.  Kept out of line so its
// registers do not add to the packed path's.
__device__ __noinline__ int ordered_query_row(const float4* __restrict__ qrec,
                                              const int32_t* __restrict__ group_start,
                                              const int32_t* __restrict__ group_end, int g0,
                                              int q0, int qn, int qi, bool active, int* qlist,
                                              uint32_t* hist) {
  const int lane = threadIdx.x & 31;
  const int gq0 = group_start[g0], gq1 = group_end[g0];
  const int nqg = gq1 - gq0;
  if (!(nqg > qn && nqg <= kMaxOrderedGroup && q0 >= gq0 && q0 + qn <= gq1))
    return q0 + qi;
  float gx = 0.f, gy = 0.f, gz = 0.f;
  for (int t = lane; t < nqg; t += 32) {
    const float4 v = qrec[gq0 + t];
    gx += v.x;
    gy += v.y;
    gz += v.z;
  }
  const float inv = 1.f / static_cast<float>(nqg);
  gx = warp_sum(gx) * inv;
  gy = warp_sum(gy) * inv;
  gz = warp_sum(gz) * inv;
  auto octant = [&](int t) {
    const float4 v = qrec[gq0 + t];
    return (v.x > gx ? 1 : 0) | (v.y > gy ? 2 : 0) | (v.z > gz ? 4 : 0);
  };
  if (lane < 8) hist[lane] = 0u;
  __syncwarp();
  for (int t = lane; t < nqg; t += 32) atomicAdd(&hist[octant(t)], 1u);
  __syncwarp();
  const uint32_t h = lane < 8 ? hist[lane] : 0u;
  const uint32_t off = static_cast<uint32_t>(warp_inclusive_scan(static_cast<int>(h))) - h;
  __syncwarp();
  if (lane < 8) hist[lane] = off;  // running position of each octant
  __syncwarp();
  const int first = q0 - gq0;
  for (int t0 = 0; t0 < nqg; t0 += 32) {
    const int t = t0 + lane;
    const int o = t < nqg ? octant(t) : 8;
    const uint32_t peers = __match_any_sync(kFull, o);
    int pos = -1;
    if (o < 8) pos = static_cast<int>(hist[o]) + __popc(peers & lanemask_lt());
    __syncwarp();
    if (o < 8 && lane == __ffs(peers) - 1) hist[o] += __popc(peers);
    if (pos >= first && pos < first + qn) qlist[pos - first] = gq0 + t;
    __syncwarp();
  }
  const int row = active ? qlist[qi] : q0 + qi;
  __syncwarp();
  return row;
}

// Register budget per list length (CTAs have at most 256 threads).  The
// 16-entry kernels' 96 registers fit the 20 resident warps per SM that the
// default tile's shared memory allows: on the 16-cloud batch (1.46 million
// queries, K=16, whole call) 80 registers took 5 % longer and 72 12 %; lists
// of 8 (700 thousand queries) with 64 registers instead of 80 5 %; lists of
// 32 with 112 instead of 128 7 %, with 120 4 %.
template <int KCAP>
constexpr int query_max_regs() {
  return KCAP <= 8 ? 80 : (KCAP <= 16 ? 96 : (KCAP <= 32 ? 128 : 224));
}

// A chunked item: one group with more candidates than a tile.  Out of line,
// so its registers do not add to the packed path's.  Returns the mbarrier's
// next phase, or -1 after a bounded wait gave up (status raised; the warp
// waited once more, bounded, for its copies, and raised kStatusCopyInFlight
// if they still had not landed).
template <int KCAP, bool EXACT, typename IdxT>
__device__ __noinline__ int chunked_item(const QueryLaunch& a, int T, int min_cands_per_lane,
                                         int q0, int qn, int g0, int k, float4* tile,
                                         uint32_t* hist, uint64_t* bar, uint32_t phase) {
  const int lane = threadIdx.x & 31;
  // One group with more candidates than a tile, up to 32 of its queries,
  // G lanes per query.  Phase A scans the first runs (the group's own
  // cell first) until they hold 2K candidates; the G partial lists of a
  // query are then merged, so every query knows its K-th distance over
  // those candidates, an upper bound of its final K-th.  A later
  // candidate can only enter the top-K of some query q if its distance to
  // the queries' centroid c is at most |q - c| + K-th(q) <= R + D (R, D:
  // the item's largest), so phase B scans, tile by tile, only the
  // candidates inside that sphere (with a margin for FP32 rounding).
  const int row = a.group_row ? a.group_row[g0] : g0;
  const int2 run = load_run(a, row, lane);
  const int incl = warp_inclusive_scan(run.y);
  const int total = __shfl_sync(kFull, incl, 31);
  const int run_off = incl - run.y;
  int lg = 5 - ceil_log2(qn);
  while (lg > 0 && (total >> lg) < min_cands_per_lane) --lg;
  const int G = 1 << lg;
  const int qi = lane >> lg, sub = lane & (G - 1);
  const bool active = qi < qn;
  const bool takes = active && cut_accepts_any(a.cut_r2);
  // The packer cuts the group's queries into items in record order: take
  // them instead in octant-major order
  // (ordered_query_row), so an item's queries are close together and the
  // phase-B sphere below stays small.
  const int qrow = ordered_query_row(a.qrec, a.group_start, a.group_end, g0, q0, qn, qi, active,
                                     reinterpret_cast<int*>(tile), hist);
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (active) q = a.qrec[qrow];
  // phase A: whole runs until 2K candidates (all of them when fewer)
  const uint32_t long_enough = __ballot_sync(kFull, lane < kNeighbours && incl >= 2 * KCAP);
  const int a_end = long_enough ? __shfl_sync(kFull, incl, __ffs(long_enough) - 1) : total;
  // centroid of the item's queries and their largest distance to it
  const bool head = active && sub == 0;
  const float inv_qn = 1.f / static_cast<float>(qn);
  const float cx = warp_sum(head ? q.x : 0.f) * inv_qn;
  const float cy = warp_sum(head ? q.y : 0.f) * inv_qn;
  const float cz = warp_sum(head ? q.z : 0.f) * inv_qn;
  const float qx = q.x - cx, qy = q.y - cy, qz = q.z - cz;
  const float rq = sqrtf(warp_max(head ? qx * qx + qy * qy + qz * qz : 0.f));
  uint64_t L[KCAP];
#pragma unroll
  for (int j = 0; j < KCAP; ++j) L[j] = kEmpty;
  const uint32_t cut_lim = cut_limit(a.cut_r2);
  uint32_t thr = cut_lim, qthr = cut_lim;
  bool timed_out = false;
  float rad2 = 0.f;
  // Stage the candidates [lo, hi) of the concatenated runs tile by tile;
  // with `filter`, keep those within sqrt(rad2) of the centroid.
  auto scan_range = [&](int lo_c, int hi_c, bool filter) {
    for (int c0 = lo_c; c0 < hi_c && !timed_out; c0 += T) {
      const int c1 = min(hi_c, c0 + T);
      __syncwarp();
      fence_proxy_async_smem();  // earlier generic reads of the tile precede the copies
      if (lane == 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(c1 - c0) * 16u);
      __syncwarp();
      const int lo = max(run_off, c0), hi = min(run_off + run.y, c1);
      if (hi > lo)
        bulk_copy_g2s(tile + (lo - c0), a.srec + run.x + (lo - run_off),
                      static_cast<uint32_t>(hi - lo) * 16u, bar);
      if (!mbar_wait_bounded(bar, phase, kWaitLimit)) {
        timed_out = true;
        break;
      }
      phase ^= 1u;
      int cnt = c1 - c0;
      if (filter) {  // compact the tile to the candidates inside the sphere
        int m = 0;
        for (int t0 = 0; t0 < cnt; t0 += 32) {
          const int t = t0 + lane;
          bool keep = false;
          float4 c = q;
          if (t < cnt) {
            c = tile[t];
            // NaN keeps the candidate: one query with a NaN coordinate makes the
            // centroid NaN, and the item's other queries still need them all
            const float dx = c.x - cx, dy = c.y - cy, dz = c.z - cz;
            keep = !(dx * dx + dy * dy + dz * dz > rad2);
          }
          // in place: the kept records move towards the front, never past
          // the ones still to be read; a vote orders no memory, so the warp
          // barrier keeps this step's reads before its stores
          const uint32_t b = __ballot_sync(kFull, keep);
          __syncwarp();
          if (keep) tile[m + __popc(b & lanemask_lt())] = c;
          m += __popc(b);
        }
        __syncwarp();
        cnt = m;
      }
      for (int i0 = 0; i0 < cnt; i0 += G) {
        const int i = i0 + sub;
        const bool ok = takes && i < cnt;
        const float4 c = ok ? tile[i] : q;
        const float d = sq_dist(c.x, c.y, c.z, q.x, q.y, q.z);
        const uint32_t db = __float_as_uint(d);
        const bool acc = ok && db <= thr;
        if (__any_sync(kFull, acc)) {
          list_insert<KCAP>(L, acc ? make_key(d, c.w) : kEmpty);
          thr = min(kth_limit(L[KCAP - 1], cut_lim), qthr);
        }
      }
    }
  };
  scan_range(0, a_end, false);
  if (!timed_out && a_end < total) {
    for (int m = 1; m < G; m <<= 1) merge_with_lane<KCAP>(L, m);
    qthr = kth_limit(L[KCAP - 1], cut_lim);  // the query's bound (same in its G lanes)
    thr = qthr;
    if (sub != 0) {  // its candidates now live in lane sub == 0 only
#pragma unroll
      for (int j = 0; j < KCAP; ++j) L[j] = kEmpty;
    }
    const float d2 = warp_max(active ? __uint_as_float(qthr) : 0.f);
    const float mag = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) + rq;
    const float rad = (rq + sqrtf(d2)) * 1.00001f + mag * 4e-6f + 1e-30f;
    rad2 = rad * rad * 1.00001f;
    scan_range(a_end, total, rad2 <= 3.0e38f);
  }
  if (timed_out) {  // no copy was issued after the wait that gave up
    if (lane == 0) raise_status(&a.meta->status, kStatusTimeout);
    const bool landed = mbar_wait_bounded(bar, phase, kWaitLimit);  // let them land
    if (!__all_sync(kFull, landed) && lane == 0)
      raise_status(&a.meta->status, kStatusCopyInFlight);
    return -1;
  }
  for (int m = 1; m < G; m <<= 1) merge_with_lane<KCAP>(L, m);
  if (active && sub == 0) write_row<IdxT, KCAP, EXACT>(a, L, __float_as_int(q.w), k);
  return static_cast<int>(phase);
}

// Shared memory of one staging buffer of a warp: the candidate tile and one
// record past it that no distance accepts (NaN coordinates), the item's group
// slots and a flag word (1 = the item's groups overflowed the
// tile, which only a malformed item can cause).
__host__ __device__ constexpr size_t buffer_bytes(int T) {
  return static_cast<size_t>(T) * 16 + kMaxGroupsPerItem * sizeof(GroupSlot) + 32;
}

// One warp's shared memory: `depth` staging buffers (at buf0 + b * stride)
// and their mbarriers, then the sort scratch shared by the buffers.
struct WarpSmem {
  unsigned char* buf0;
  size_t stride;
  int T;
  uint64_t* bars;
  uint16_t* srt16;
  uint16_t* tmp16;
  uint16_t* bstart;
  uint32_t* hist;
  __device__ __forceinline__ float4* tile(int b) const {
    return reinterpret_cast<float4*>(buf0 + b * stride);
  }
  __device__ __forceinline__ GroupSlot* slots(int b) const {
    return reinterpret_cast<GroupSlot*>(buf0 + b * stride + static_cast<size_t>(T) * 16 + 16);
  }
  __device__ __forceinline__ int* flags(int b) const {
    return reinterpret_cast<int*>(slots(b) + kMaxGroupsPerItem);
  }
  __device__ __forceinline__ uint64_t* bar(int b) const { return bars + b; }
};

__device__ __forceinline__ WarpSmem warp_smem(unsigned char* smem_raw, int T, int depth) {
  const int warp = threadIdx.x >> 5;
  WarpSmem w;
  w.buf0 = smem_raw + 128 + static_cast<size_t>(warp) * warp_smem_bytes(T, depth);
  w.stride = buffer_bytes(T);
  w.T = T;
  w.bars = reinterpret_cast<uint64_t*>(smem_raw) + warp * kMaxStaging;
  w.srt16 = reinterpret_cast<uint16_t*>(w.buf0 + static_cast<size_t>(depth) * buffer_bytes(T));
  w.tmp16 = w.srt16 + sorted_slots(T);
  w.bstart = w.tmp16 + T;
  w.hist = reinterpret_cast<uint32_t*>(w.bstart + kMaxGroupsPerItem * (kBuckets + 1));
  return w;
}

// Checks work item `it` and, for a packed item, issues the copies of its
// groups' candidate runs into buffer b (the caller commits and waits for
// them) and records the groups in the buffer's slots.  Returns 1 when copies
// were issued, 0 for a chunked item (it streams its own tiles), -1 for a
// malformed item (status raised, nothing to do).
__device__ __forceinline__ int stage_item(const QueryLaunch& a, const NextItem& x, int n_groups, int T,
                                          const WarpSmem& w, int b) {
  const int lane = threadIdx.x & 31;
  const int4 it = x.it;
  const int q0 = it.x, qn = it.y, g0 = it.z, gn = it.w & 0xffff;
  const bool chunked = (it.w & kItemChunked) != 0;
  if (q0 < 0 || qn < 1 || qn > 32 || static_cast<int64_t>(q0) + qn > a.n_qrec || g0 < 0 ||
      gn < 1 || gn > kMaxGroupsPerItem || g0 + gn > n_groups || (chunked && gn != 1)) {
    if (lane == 0) raise_status(&a.meta->status, kStatusTable);
    return -1;
  }
  if (chunked) return 0;
  int ga = 0, gb = 0, grow = 0;
  if (lane < gn) {
    grow = x.row;
    ga = max(x.gs, q0);
    gb = max(ga, min(x.ge, q0 + qn));
  }
  // The runs of two groups ahead are in flight while a group's copies are
  // issued.
  auto fetch = [&](int gi) {
    const int row = __shfl_sync(kFull, grow, gi & 31);
    return gi < gn && lane < kNeighbours
               ? __ldg(a.runs + static_cast<int64_t>(row) * kNeighbours + lane)
               : make_int2(0, 0);
  };
  int2 run = fetch(0), run1 = fetch(1);
  float4* tile = w.tile(b);
  int* base = reinterpret_cast<int*>(w.hist);  // one per non-empty run
  int seg = 0;
  bool overflow = false;
#pragma unroll 1
  for (int gi = 0; gi < gn; ++gi) {
    const int2 run2 = fetch(gi + 2);
    const int ga_ = __shfl_sync(kFull, ga, gi), gb_ = __shfl_sync(kFull, gb, gi);
    int len = 0;
    if (gb_ > ga_ && !overflow) {
      run = checked_run(a, run);
      // A tile is full long before 27 runs of the support's size could wrap the
      // sum (caller tables over 80 million points).
      run.y = min(run.y, T + 1);
      const int incl = warp_inclusive_scan(run.y);
      const int first = incl - run.y;
      len = __shfl_sync(kFull, incl, 31);
      if (seg + len > T) {
        overflow = true;
        len = 0;
      } else {
        const uint32_t filled = __ballot_sync(kFull, run.y > 0);
        if (run.y > 0) base[__popc(filled & lanemask_lt())] = run.x - first;
        __syncwarp();
        // 32 records a step, one per lane: a lane's run is the last one that
        // starts at or before its record
        int before = -1;
#pragma unroll 1
        for (int t0 = 0; t0 < len; t0 += 32) {
          const int at = first - t0;
          const uint32_t starts =
              __reduce_or_sync(kFull, run.y > 0 && at >= 0 && at < 32 ? 1u << at : 0u);
          const int r = before + __popc(starts & (lanemask_lt() | (1u << lane)));
          before += __popc(starts);
          if (t0 + lane < len)
            copy_16_async(tile + seg + t0 + lane, a.srec + (base[r] + t0 + lane));
        }
        __syncwarp();
      }
    }
    if (lane == 0) {
      GroupSlot s;
      s.seg = seg;
      s.len = len;
      s.a = ga_;
      s.b = overflow ? ga_ : gb_;
      w.slots(b)[gi] = s;
    }
    seg += len;
    run = run1;
    run1 = run2;
  }
  if (lane == 0) *w.flags(b) = overflow ? 1 : 0;
  return 1;
}

// A packed item whose copies into buffer b have landed: up to 32 queries of
// up to 16 groups, one query per lane (see the file comment).  q is the
// lane's query record; the next item is fetched before the results are
// written.
template <int KCAP, bool EXACT, typename IdxT>
__device__ __forceinline__ void packed_item(const QueryLaunch& a, const int4& it, const float4& q,
                                            const WarpSmem& w, int b, int n_items,
                                            int n_groups, NextItem& next) {
  const int lane = threadIdx.x & 31;
  Meta* meta = a.meta;
  const int qn = it.y, gn = it.w & 0xffff;
  const float4* tile = w.tile(b);
  uint32_t* hist = w.hist;
  const int k = a.k;
  if (*w.flags(b)) {  // the packer bounds every item by the tile; report a broken item
    if (lane == 0) raise_status(&meta->status, kStatusTable);
    next.pop(meta);
    next.load(a, n_items);
    next.load_groups(a, n_items, n_groups);
    return;
  }
  // Per group: centre of its queries' box, distance buckets, counting sort of
  // its candidates' tile positions.  Kept short rather than unrolled, with
  // the box from six reductions instead of a centroid from fifteen shuffles:
  // unrolled by two or four the whole call at K=32 took 533 / 552 us, as here
  // 510 us (700 thousand queries).
  const int p = it.x + lane;
  LaneGroup mine{0, w.srt16, w.bstart, 1.f, 0.f, 0.f};
  bool mapped = false;
  uint16_t* srt = w.srt16;
#pragma unroll 1
  for (int gi = 0; gi < gn; ++gi) {
    const GroupSlot s = w.slots(b)[gi];
    if (s.b <= s.a) continue;
    const bool member = p >= s.a && p < s.b;  // a subset of the item's qn lanes
    const float inf = __int_as_float(kInfBits);
    const float cx = 0.5f * (redux_min(member ? q.x : inf) + redux_max(member ? q.x : -inf));
    const float cy = 0.5f * (redux_min(member ? q.y : inf) + redux_max(member ? q.y : -inf));
    const float cz = 0.5f * (redux_min(member ? q.z : inf) + redux_max(member ? q.z : -inf));
    const float4* seg = tile + s.seg;
    // The buckets' range: the largest squared distance to the centre among
    // 32 evenly spaced candidates (the last bucket takes all beyond).
    float far2 = 0.f;
    if (s.len > 0) {
      const float4 c = seg[(lane * s.len) >> 5];
      far2 = fmaxf(far2, sq_dist(c.x, c.y, c.z, cx, cy, cz));
    }
    far2 = __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(far2)));
    const float inv_w2 = far2 > 0.f ? __fdividef(kBuckets / 1.0001f, far2) : 1.f;
    hist[lane] = 0u;  // kBuckets == 32: one bucket per lane
    __syncwarp();
    // Bucket of every candidate and its rank inside the bucket.
#pragma unroll 1
    for (int t = lane; t < s.len; t += 32) {
      const float4 c = seg[t];
      const float d2 = sq_dist(c.x, c.y, c.z, cx, cy, cz);
      const int bkt = min(static_cast<int>(d2 * inv_w2), kBuckets - 1);
      const uint32_t r = atomicAdd(&hist[bkt], 1u);
      w.tmp16[t] = static_cast<uint16_t>((bkt << 10) | r);
    }
    __syncwarp();
    const uint32_t h = hist[lane];
    const uint32_t hi = static_cast<uint32_t>(warp_inclusive_scan(static_cast<int>(h)));
    uint16_t* bs = w.bstart + gi * (kBuckets + 1);
    bs[lane] = static_cast<uint16_t>(hi - h);
    if (lane == 31) bs[kBuckets] = static_cast<uint16_t>(hi);
    __syncwarp();
#pragma unroll 1
    for (int t = lane; t < s.len; t += 32) {
      const uint32_t v = w.tmp16[t];
      srt[bs[v >> 10] + (v & 1023u)] = static_cast<uint16_t>(s.seg + t);
    }
    if (lane < ((-s.len) & 7)) srt[s.len + lane] = static_cast<uint16_t>(w.T);  // no candidate
    if (member) {
      const float dx = q.x - cx, dy = q.y - cy, dz = q.z - cz;
      const float mag = fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) + sqrt_above(far2);
      mapped = true;
      mine.len = cut_accepts_any(a.cut_r2) ? s.len : 0;
      mine.srt = srt;
      mine.bstart = bs;
      mine.inv_w2 = inv_w2;
      mine.rq = sqrt_above(dx * dx + dy * dy + dz * dz);
      mine.eps = mag * 4e-6f + 1e-30f;
    }
    srt += (s.len + 7) & ~7;
    __syncwarp();
  }

  // One query per lane.
  if (lane < qn && !mapped) raise_status(&meta->status, kStatusTable);
  const uint32_t cut_lim = cut_limit(a.cut_r2);
  // Squared distance bits of the candidate at tile position pos.
  auto dist_bits = [&](uint32_t pos, float4& c) {
    c = tile[pos];
    return __float_as_uint(sq_dist(c.x, c.y, c.z, q.x, q.y, q.z));
  };
  uint64_t L[KCAP];
  const uint32_t none = static_cast<uint32_t>(w.T) * 0x10001u;  // the tile's empty record
  select_blocks<KCAP>(L, mine, k, w.T <= 512 ? 511u : 1023u, cut_lim, dist_bits, a, n_items, none,
                      next, tile, q);
  next.load_groups(a, n_items, n_groups);
  if (lane < qn && mapped) write_row<IdxT, KCAP, EXACT>(a, L, __float_as_int(q.w), k);
  __syncwarp();
}

// The persistent query kernel.  Each warp pulls items from the queue; with
// `depth` 2 it stages the next item's candidate runs into its second buffer
// before it scans the current one, so those copies are in flight while it
// computes.
template <int KCAP, bool EXACT, typename IdxT>
__global__ void __maxnreg__(query_max_regs<KCAP>())
    k_query(const __grid_constant__ QueryLaunch a, int T, int min_cands_per_lane, int depth) {
  chain_wait();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const WarpSmem w = warp_smem(smem_raw, T, depth);
  Meta* meta = a.meta;
  if (lane == 0) {
    const float nan = __int_as_float(0x7fffffff);
    for (int b = 0; b < depth; ++b) {
      mbar_init(w.bar(b), 1);
      w.tile(b)[T] = make_float4(nan, nan, nan, 0.f);
    }
    mbar_init_fence();
  }
  __syncwarp();
  uint32_t phase = 0u;  // bit b: the parity to wait for on buffer b's barrier
  const int n_items = meta->n_items;
  const int n_groups = *a.group_count_ptr;

  auto stage = [&](const NextItem& x, int b) {
    const int staged = x.item < n_items ? stage_item(a, x, n_groups, T, w, b) : -1;
    copy_async_commit();
    return staged;
  };
  int buf = 0;
  NextItem cur{true, 0, 0, make_int4(0, 0, 0, 0), 0, 0, 0};
  cur.pop(meta);
  cur.load(a, n_items);
  cur.load_groups(a, n_items, n_groups);
  int staged = stage(cur, buf);
  while (cur.item < n_items) {
    NextItem next{true, 0, n_items, make_int4(0, 0, 0, 0), 0, 0, 0};
    int next_staged = -1;
    if (depth > 1) {  // the next item's copies fly while this one is scanned
      next.pop(meta);
      next.load(a, n_items);
      next.load_groups(a, n_items, n_groups);
      next_staged = stage(next, buf ^ 1);
      next.wanted = false;
    }
    const int4 it = cur.it;
    if (staged == 1) {
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane < it.y) q = a.qrec[it.x + lane];  // in flight during the wait
      if (depth > 1)
        copy_async_wait<1>();
      else
        copy_async_wait<0>();
      __syncwarp();
      packed_item<KCAP, EXACT, IdxT>(a, it, q, w, buf, n_items, n_groups, next);
    } else {
      if (staged == 0) {
        const int nxt = chunked_item<KCAP, EXACT, IdxT>(a, T, min_cands_per_lane, it.x, it.y, it.z,
                                                        a.k, w.tile(buf), w.hist, w.bar(buf),
                                                        (phase >> buf) & 1u);
        if (nxt < 0) break;  // a bounded wait gave up: its own copies were waited for
        phase = (phase & ~(1u << buf)) | (static_cast<uint32_t>(nxt) << buf);
      }
      next.pop(meta);
      next.load(a, n_items);
      next.load_groups(a, n_items, n_groups);
    }
    if (depth > 1)
      buf ^= 1;
    else
      next_staged = stage(next, buf);
    cur = next;
    cur.wanted = true;
    staged = next_staged;
  }
  copy_async_wait<0>();  // none in flight when the warp leaves
  __syncwarp();
}

// ------------------------------------------------------------------ host

QueryShape resolve_shape(const fknn_config* cfg) {
  QueryShape s{4, 448, 8, 0, 1};
  if (cfg) {
    if (cfg->warps_per_cta) s.warps_per_cta = cfg->warps_per_cta;
    if (cfg->tile_records) s.tile_records = cfg->tile_records;
    if (cfg->min_candidates_per_lane) s.min_candidates_per_lane = cfg->min_candidates_per_lane;
    s.ctas_per_sm = cfg->ctas_per_sm;
    if (cfg->staging_depth) s.staging_depth = cfg->staging_depth;
  }
  return s;
}

bool shape_valid(const QueryShape& s) {
  const bool warps_ok = s.warps_per_cta == 1 || s.warps_per_cta == 2 ||
                        s.warps_per_cta == 4 || s.warps_per_cta == 8;
  const bool depth_ok = s.staging_depth >= 1 && s.staging_depth <= kMaxStaging;
  return warps_ok && depth_ok && s.tile_records >= 64 && s.tile_records <= 1024 &&
         s.tile_records % 32 == 0 && s.min_candidates_per_lane >= 1 &&
         s.ctas_per_sm >= 0 && s.ctas_per_sm <= 32 &&
         128 + static_cast<size_t>(s.warps_per_cta) *
                   warp_smem_bytes(s.tile_records, s.staging_depth) <=
             227 * 1024;
}

namespace {

template <int KCAP, bool EXACT, typename IdxT>
int launch_t(const QueryLaunch& q, const QueryShape& shape, cudaStream_t s) {
  auto kern = k_query<KCAP, EXACT, IdxT>;
  const int threads = shape.warps_per_cta * 32;
  const size_t smem = 128 + static_cast<size_t>(shape.warps_per_cta) *
                               warp_smem_bytes(shape.tile_records, shape.staging_depth);
  // Device properties and occupancy are resolved once per (device, shape) and
  // cached, so a launch inside a CUDA graph capture issues nothing but the
  // kernel itself.  The cache is shared by all host threads under a mutex,
  // and the kernel's dynamic shared-memory limit is raised once per device
  // to the device's opt-in maximum (less the kernel's static shared memory),
  // so a launch with one shape never lowers the limit under a concurrent
  // launch with a larger one.
  struct Cached {
    int dev, threads, per_sm, sms;
    size_t smem;
  };
  static std::mutex mu;
  static std::vector<Cached> cache;
  static std::vector<int> raised;  // devices whose limit is raised
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  Cached use{};
  {
    std::lock_guard<std::mutex> lock(mu);
    bool found = false;
    for (const Cached& c : cache)
      if (c.dev == dev && c.threads == threads && c.smem == smem) {
        use = c;
        found = true;
      }
    if (!found) {
      Cached c{dev, threads, 0, 0, smem};
      e = cudaDeviceGetAttribute(&c.sms, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
      if (std::find(raised.begin(), raised.end(), dev) == raised.end()) {
        int optin = 0;
        e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        if (e != cudaSuccess) return e;
        cudaFuncAttributes fa{};
        e = cudaFuncGetAttributes(&fa, kern);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 optin - static_cast<int>(fa.sharedSizeBytes));
        if (e != cudaSuccess) return e;
        raised.push_back(dev);
      }
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c.per_sm, kern, threads, smem);
      if (e != cudaSuccess) return e;
      if (c.per_sm < 1) c.per_sm = 1;
      cache.push_back(c);
      use = c;
    }
  }
  const int per_sm = shape.ctas_per_sm > 0 ? shape.ctas_per_sm : use.per_sm;
  const int grid = use.sms * per_sm;
  const int slot = profile_start(s);
  launch_chained(kern, grid, threads, smem, s, q, shape.tile_records, shape.min_candidates_per_lane,
      shape.staging_depth);
  e = cudaGetLastError();
  profile_stop(slot, s);
  return e;
}

template <int KCAP>
int launch_k(const QueryLaunch& q, const QueryShape& shape, cudaStream_t s) {
  const bool exact = q.k == KCAP;
  if (q.idx_bits == 64)
    return exact ? launch_t<KCAP, true, int64_t>(q, shape, s)
                 : launch_t<KCAP, false, int64_t>(q, shape, s);
  return exact ? launch_t<KCAP, true, int32_t>(q, shape, s)
               : launch_t<KCAP, false, int32_t>(q, shape, s);
}

}  // namespace

int launch_query(const QueryLaunch& q, const QueryShape& shape, cudaStream_t s) {
  if (q.k <= 1) return launch_k<1>(q, shape, s);
  if (q.k <= 2) return launch_k<2>(q, shape, s);
  if (q.k <= 4) return launch_k<4>(q, shape, s);
  if (q.k <= 8) return launch_k<8>(q, shape, s);
  if (q.k <= 16) return launch_k<16>(q, shape, s);
  if (q.k <= 32) return launch_k<32>(q, shape, s);
  return launch_k<64>(q, shape, s);
}

}  // namespace fknn
