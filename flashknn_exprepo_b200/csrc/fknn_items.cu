// Work items of the query kernel.
//
// A query group is a set of queries (contiguous in the query-record array)
// that share one candidate set: the 27 runs of a parent cell.  Items pack
// up to 32 consecutive queries -- possibly from several consecutive groups --
// so that every lane of a warp owns one query, as long as the candidates of
// all groups in the item fit one shared-memory tile.  Groups with more
// candidates than a tile become "chunked" items of up to 32 queries that
// stream their candidates tile by tile.
//
// Packing is a sequential greedy pass over the groups in order; it runs in
// parallel over segments of consecutive groups (one warp each; the segment
// length follows the group count, see pack_segment_len), each walked twice:
// to count its items, and to write them where one atomic per CTA placed them.
// Items therefore keep the order of the groups inside a segment; the order of
// the segments does not matter.  A count kernel, a scan of the counts and a
// write kernel took 9.4 us for a small cube and 33 us for 1.46 million
// queries.  With this and three launches fewer in the construction the whole
// call takes 71 instead of 87 us on the cube (16 thousand queries, issued
// back to back) and 557 instead of 574 us on 1.46 million.
#include <climits>

#include "fknn_common.cuh"
#include "fknn_internal.h"

namespace fknn {

// cands[g] = number of candidate records of group g (sum of its 27 runs);
// a group without candidates sets kStatusNoCandidates; a sum beyond 32 bits is
// reported and counts as none, which the query kernel's own sum then meets as
// an overfull tile.  meta->pair_total
// receives the sum of queries x candidates (one atomic per block)
// where it is wanted (pairs_wanted).
__global__ void __launch_bounds__(256)
    k_group_cands(const int2* __restrict__ runs, const int32_t* __restrict__ group_row,
                  const int* group_count_ptr, int32_t* __restrict__ cands,
                  const int32_t* __restrict__ group_start, const int32_t* __restrict__ group_end,
                  int pairs, Meta* meta) {
  chain_wait();
  __shared__ unsigned long long s_pairs[8];
  unsigned long long my_pairs = 0ull;
  const int n_groups = *group_count_ptr;
  for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < n_groups;
       g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t row = group_row ? group_row[g] : g;
    const int2* r = runs + row * kNeighbours;
    int64_t sum = 0;
#pragma unroll
    for (int j = 0; j < kNeighbours; ++j) sum += max(r[j].y, 0);
    if (sum > INT_MAX) {  // caller tables only: cells do not overlap
      raise_status(&meta->status, kStatusTable);
      sum = 0;
    }
    const int total = static_cast<int>(sum);
    cands[g] = total;
    if (pairs)
      my_pairs += static_cast<unsigned long long>(total) * max(group_end[g] - group_start[g], 0);
    if (total == 0) raise_status(&meta->status, kStatusNoCandidates);
  }
  if (!pairs) return;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) my_pairs += __shfl_xor_sync(kFull, my_pairs, d);
  if ((threadIdx.x & 31) == 0) s_pairs[threadIdx.x >> 5] = my_pairs;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) my_pairs += s_pairs[w];
    if (my_pairs) atomicAdd(&meta->pair_total, my_pairs);
  }
}

// Queries of a chunked item of a group with c candidates.  Below a full
// item's worth of queries per resident warp (max_qc < 32, chunked_query_cap)
// max_qc.  In a larger problem an item's time grows with c, and smaller items
// stream the candidates more often, so an item is cut only where it would
// run on after the others have ended.  `share` = candidates that an average
// lane meets in the whole call (pairs of query and candidate over the resident
// lanes): a full item of c = share keeps its warp busy for the average warp's
// whole time.  Groups of usual size (c up to 3/2 of the mean over the queries)
// carry most of the work and are cut to that time; groups far above it to a
// quarter, since a few of them decide when the call ends.  Never below
// kChunkedFull candidates or to fewer than kChunkedFew queries.  K=16, whole
// call, full items / every group above 2,048 candidates cut in inverse
// proportion / this rule: a LiDAR scan of 115 thousand points with 40 cm cells
// (up to 13 thousand candidates) 404 / 282 / 277 us, one of 800 thousand 2993 /
// 3168 / 2481; 500 thousand uniform points of 20 thousand candidates 2511 /
// 3248 / 1940, 400 thousand on a sheet of 12 thousand 2070 / 2749 / 1571 (the
// first figure with an earlier scan kernel, 1.3 times slower by itself).  One
// limit for all groups: half a share 5 to 12 % slower on scans of 400
// thousand, a quarter up to 15 % on uniform points.
constexpr float kChunkedFull = 2048.f;
constexpr int kChunkedFew = 8;
__device__ __forceinline__ int chunked_queries(int max_qc, int c, float typical, float share) {
  const float cf = static_cast<float>(c);
  const float full = fmaxf(cf <= typical ? share : 0.25f * share, kChunkedFull);
  if (cf <= full || max_qc < 32) return max_qc;
  return max(static_cast<int>(static_cast<float>(max_qc) * full / cf), kChunkedFew);
}

// One warp per segment of consecutive groups.  Item = (q_start, q_count,
// g_first, g_count | flags).
// The segment's group ranges and candidate counts are loaded once (one
// group per lane); every lane then walks the greedy pass with the same
// values, lane 0 writes packed items and the whole warp writes the items of a
// group that makes many by itself (chunked, or queries for several full
// items): 300 thousand queries in 27 cells of 100 points took 587 us item by
// item.
// An item's queries are consecutive records: a group that does not start
// where the one before it ended starts a new item.
// Caller tables can be malformed: a group whose query range leaves
// [0, n_queries] is reported and skipped, and no item is written at or past
// `capacity` (overlapping ranges could otherwise ask for more items than the
// buffer holds; *n_items, which starts at 0, is clamped to match).
static_assert(kPackSegment <= 32, "one group per lane");
__global__ void __launch_bounds__(256)
    k_pack(const int32_t* __restrict__ group_start, const int32_t* __restrict__ group_end,
           const int32_t* __restrict__ cands, const int* group_count_ptr, int tile, int max_q,
           int max_qc, int64_t n_queries, int64_t capacity, float typical_scale,
           float share_scale, Meta* meta, int4* __restrict__ items) {
  chain_wait();
  int* n_items = &meta->n_items;
  int* status = &meta->status;
  const float pairs = static_cast<float>(meta->pair_total);
  const float typical = pairs * typical_scale, share = pairs * share_scale;
  __shared__ uint32_t s_count[8];
  __shared__ uint32_t s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_groups = *group_count_ptr;
  const int seg_len = pack_segment_len(n_groups);
  const int64_t n_segs = (n_groups + seg_len - 1) / seg_len;
  for (int64_t seg0 = static_cast<int64_t>(blockIdx.x) * 8; seg0 < n_segs;
       seg0 += static_cast<int64_t>(gridDim.x) * 8) {
    const int64_t g_begin = (seg0 + warp) * seg_len;
    const int64_t g_lim = g_begin + seg_len;
    const int64_t g_end = g_lim < n_groups ? g_lim : n_groups;
    const int n_here = g_end > g_begin ? static_cast<int>(g_end - g_begin) : 0;
    int my_gs = 0, my_ge = 0, my_c = 0;
    if (lane < n_here) {
      my_gs = group_start[g_begin + lane];
      my_ge = group_end[g_begin + lane];
      my_c = cands[g_begin + lane];
    }
    // The greedy walk: put(slot, q0, qn, g0, gn, flags, lane that writes) for
    // every item; returns the number of items.
    auto walk = [&](bool write, uint32_t out) {
      uint32_t count = 0;
      int cur_q0 = 0, cur_qn = 0, cur_g0 = 0, cur_gn = 0, cur_c = 0;
      auto put = [&](uint32_t slot, int q0, int qn, int g0, int gn, int flags) {
        if (static_cast<int64_t>(out) + slot < capacity)
          items[out + slot] = make_int4(q0, qn, g0, gn | flags);
        else
          raise_status(status, kStatusTable);
      };
      auto flush = [&]() {
        if (cur_gn > 0) {
          if (write && lane == 0) put(count, cur_q0, cur_qn, cur_g0, cur_gn, 0);
          ++count;
        }
        cur_qn = cur_gn = cur_c = 0;
      };
      for (int j = 0; j < n_here; ++j) {
        const int g = static_cast<int>(g_begin) + j;
        const int gs = __shfl_sync(kFull, my_gs, j), ge = __shfl_sync(kFull, my_ge, j);
        const int c = __shfl_sync(kFull, my_c, j);
        if (gs < 0 || ge > n_queries) {
          if (write && lane == 0) raise_status(status, kStatusTable);
          continue;
        }
        if (ge <= gs) continue;
        if (c > tile) {  // streams its candidates: items of its own
          flush();
          const int qc = chunked_queries(max_qc, c, typical, share);
          const int n_it = (ge - gs + qc - 1) / qc;
          if (write)
            for (int t = lane; t < n_it; t += 32) {
              const int q = gs + t * qc;
              put(count + t, q, min(qc, ge - q), g, 1, kItemChunked);
            }
          count += n_it;
          continue;
        }
        int pos = gs;
        while (pos < ge) {
          // An item spans the groups [cur_g0, g]: groups without queries
          // inside that span still count, because the kernel walks the span.
          if (cur_gn > 0 && (cur_c + c > tile || cur_qn >= max_q || pos != cur_q0 + cur_qn ||
                             g - cur_g0 + 1 > kMaxGroupsPerItem))
            flush();
          if (cur_gn == 0) {
            if (ge - pos >= 2 * max_q) {  // whole items, written by the warp
              const int whole = (ge - pos) / max_q;
              if (write)
                for (int t = lane; t < whole; t += 32)
                  put(count + t, pos + t * max_q, max_q, g, 1, 0);
              count += whole;
              pos += whole * max_q;
              continue;
            }
            cur_q0 = pos;
            cur_g0 = g;
          }
          const int take = min(ge - pos, max_q - cur_qn);
          cur_qn += take;
          cur_gn = g - cur_g0 + 1;
          cur_c += c;
          pos += take;
        }
      }
      flush();
      return count;
    };
    const uint32_t count = walk(false, 0u);
    if (lane == 0) s_count[warp] = count;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t total = 0;
      for (int i = 0; i < 8; ++i) total += s_count[i];
      s_base = total ? atomicAdd(reinterpret_cast<unsigned*>(n_items), total) : 0u;
      if (static_cast<int64_t>(s_base) + total > capacity)
        atomicMin(reinterpret_cast<unsigned*>(n_items), static_cast<unsigned>(capacity));
    }
    __syncthreads();
    uint32_t out = s_base;
    for (int i = 0; i < warp; ++i) out += s_count[i];
    walk(true, out);
    __syncthreads();  // before the next segments' counts
  }
}

// Queries per packed item.  A large problem fills every lane (32); a small
// one -- fewer than 16 queries per resident query warp -- is cut into about
// one item per resident warp (at least 4 queries each), so its few items do
// not leave most warps idle while each one runs the whole scan.
int item_query_cap(int64_t n_queries) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
      sms = v;
    if (sms <= 0) return 32;
  }
  const int64_t warps = static_cast<int64_t>(sms) * 20;  // resident at the default shape
  if (n_queries >= warps * 16) return 32;
  const int64_t cap = ceil_div(n_queries > 0 ? n_queries : 1, warps);
  return static_cast<int>(cap < 4 ? 4 : (cap > 32 ? 32 : cap));
}

// Query warps resident on the current device at the default launch shape; 0
// where the device does not tell.
int64_t resident_warps() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
    return 0;
  return static_cast<int64_t>(sms) * 20;
}

// Only calls of a full item's worth of queries per warp cut chunked items by
// their share of the work (chunked_queries).
bool pairs_wanted(int64_t n_queries) { return n_queries >= resident_warps() * 32; }

// Queries per chunked item (a group whose candidates exceed a tile: every
// query scans many of them).  An item of q queries gives each query 32 / q
// lanes.  A problem with fewer than 32 queries per resident query warp is
// cut into about two items per warp (at least 4 queries each), so a dense
// but small problem spreads every query's scan over several lanes instead
// of one lane walking all its candidates (the DeLA levels of 3.7k-72k points
// are faster so); larger ones start from full items (chunked_queries).
int chunked_query_cap(int64_t n_queries, int64_t warps) {
  if (warps == 0 || n_queries >= warps * 32) return 32;
  const int64_t cap = ceil_div(n_queries > 0 ? n_queries : 1, 2 * warps);
  return static_cast<int>(cap < 4 ? 4 : (cap > 32 ? 32 : cap));
}

int launch_items(const int2* runs, const int32_t* group_start, const int32_t* group_end,
                 const int32_t* group_row, const int* group_count_ptr, int64_t max_groups, int tile,
                 int32_t* cands, Meta* meta, int4* items, cudaStream_t s, int64_t n_queries,
                 bool cands_ready) {
  if (max_groups <= 0) return 0;
  // grids for the host-side bound, capped: the device count drives the loops
  const int64_t gb = ceil_div(max_groups, 256);
  const int gblocks = static_cast<int>(gb < 2048 ? gb : 2048);
  const int64_t sb = ceil_div(pack_segments(max_groups), 8);  // 8 warps per block
  const int sblocks = static_cast<int>(sb < 2048 ? sb : 2048);
  if (!cands_ready)  // else the caller's run kernel wrote cands[g] already
    launch_chained(k_group_cands, gblocks, 256, 0, s, runs, group_row, group_count_ptr, cands,
                   group_start, group_end, pairs_wanted(n_queries) ? 1 : 0, meta);
  const int64_t capacity = static_cast<int64_t>(items_capacity(max_groups, n_queries));
  const int64_t warps = resident_warps();
  launch_chained(k_pack, sblocks, 256, 0, s, group_start, group_end, cands, group_count_ptr, tile,
                 item_query_cap(n_queries), chunked_query_cap(n_queries, warps), n_queries, capacity,
                 n_queries > 0 ? 1.5f / static_cast<float>(n_queries) : 0.f,
                 warps > 0 ? 1.f / static_cast<float>(warps * 32) : 1.f, meta, items);
  return cands_ready ? 1 : 2;
}

size_t items_capacity(int64_t max_groups, int64_t n_queries) {
  // every item holds at least one query, and no query is in two
  const int64_t a = n_queries + max_groups + 32;
  return static_cast<size_t>(a);
}

}  // namespace fknn
