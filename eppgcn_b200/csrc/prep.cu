// One-time execution-path preparation for sm_100a: path marking, stable
// compaction of the marked edges and splitting of the active rows into parts.
//
// The two scans (compaction ranks, part offsets) are single-pass chained scans:
// a tile takes its id from an atomic ticket (so every predecessor of a waiting
// tile has already started), publishes its aggregate in a 64-bit descriptor and
// looks back over its predecessors' descriptors.  Every wait is bounded; when
// the bound is hit the kernel records EPP_ERR_SCAN_TIMEOUT, releases its
// successors and returns.  A three-kernel mode (counts, scan, scatter) that
// never waits is kept as the fallback and as a cross-check.
#include "common.cuh"

namespace epp {
namespace {

constexpr int kScanThreads = 512;
constexpr int kScanWarps = kScanThreads / kWarp;
constexpr int kCompactItems = 8;                                  // per thread
constexpr int kCompactTile = kScanThreads * kCompactItems;        // 4096 edges
constexpr int kSplitItems = 4;
constexpr int kSplitTile = kScanThreads * kSplitItems;            // 2048 vertices
constexpr int kOneWaveTiles = 148 * 4;                            // that fit onto the chip together
constexpr int kMaxPolls = 1 << 21;                                // bounded look-back wait

enum ScanMode { kLookback = 0, kCountOnly = 1, kGivenOffsets = 2 };

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Exclusive prefix (fields a, b) of tile `tile`; called by all lanes of one warp.
// Publishes the tile's aggregate first and its inclusive prefix afterwards.
__device__ void chained_lookback(unsigned long long *desc, ScanHeader *hdr, int *status, int tile,
                                 unsigned agg_a, unsigned agg_b, unsigned &ex_a, unsigned &ex_b) {
  const int lane = threadIdx.x & 31;
  volatile unsigned long long *vdesc = desc;
  volatile int *verr = &hdr->error;
  if (tile == 0) {
    if (lane == 0) vdesc[0] = tile_pack(kTilePrefix, agg_a, agg_b);
    ex_a = ex_b = 0;
    return;
  }
  if (lane == 0) vdesc[tile] = tile_pack(kTileAggregate, agg_a, agg_b);
  unsigned long long sum = 0;   // packed fields, state bits stay zero
  int window_top = tile - 1;
  bool failed = false;
  while (true) {
    const int p = window_top - lane;
    unsigned long long w = tile_pack(kTilePrefix, 0, 0);   // lanes before tile 0 end the search
    if (p >= 0) {
      int polls = 0;
      w = vdesc[p];
      while (tile_state(w) == kTileEmpty) {
        if (++polls > kMaxPolls || *verr != EPP_OK) { failed = true; break; }
        if (polls > 16) __nanosleep(polls > 1024 ? 256 : 32);
        w = vdesc[p];
      }
    }
    if (__any_sync(kFull, failed)) break;
    const unsigned done = __ballot_sync(kFull, tile_state(w) == kTilePrefix);
    // lanes up to and including the nearest predecessor that holds a full prefix
    const unsigned take = done ? ((2u << (__ffs(done) - 1)) - 1u) : kFull;
    unsigned long long v = ((take >> lane) & 1u) ? (w & 0x3fffffffffffffffull) : 0ull;
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
    sum += v;
    if (done) break;
    window_top -= kWarp;
  }
  if (__any_sync(kFull, failed)) {
    if (lane == 0) {
      atomicExch(&hdr->error, EPP_ERR_SCAN_TIMEOUT);
      atomicExch(status, EPP_ERR_SCAN_TIMEOUT);
      vdesc[tile] = tile_pack(kTilePrefix, 0, 0);   // let successors go; the result is void
    }
    ex_a = ex_b = 0;
    return;
  }
  ex_a = tile_a(sum);
  ex_b = tile_b(sum);
  if (lane == 0) vdesc[tile] = tile_pack(kTilePrefix, ex_a + agg_a, ex_b + agg_b);
}

// Block-wide exclusive scan of one (a, b) pair per thread over kScanThreads
// threads; returns the thread's exclusive prefix and the block totals.
__device__ __forceinline__ void block_scan_pair(unsigned a, unsigned b, unsigned &ex_a, unsigned &ex_b,
                                                unsigned &tot_a, unsigned &tot_b,
                                                unsigned (*s_warp)[2]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned ia = a, ib = b;
#pragma unroll
  for (int off = 1; off < kWarp; off <<= 1) {
    const unsigned ta = __shfl_up_sync(kFull, ia, off), tb = __shfl_up_sync(kFull, ib, off);
    if (lane >= off) { ia += ta; ib += tb; }
  }
  if (lane == kWarp - 1) { s_warp[warp][0] = ia; s_warp[warp][1] = ib; }
  __syncthreads();
  if (warp == 0) {
    unsigned wa = lane < kScanWarps ? s_warp[lane][0] : 0, wb = lane < kScanWarps ? s_warp[lane][1] : 0;
    unsigned sa = wa, sb = wb;
#pragma unroll
    for (int off = 1; off < kWarp; off <<= 1) {
      const unsigned ta = __shfl_up_sync(kFull, sa, off), tb = __shfl_up_sync(kFull, sb, off);
      if (lane >= off) { sa += ta; sb += tb; }
    }
    if (lane < kScanWarps) { s_warp[lane][0] = sa - wa; s_warp[lane][1] = sb - wb; }
    if (lane == kWarp - 1) { s_warp[kScanWarps][0] = sa; s_warp[kScanWarps][1] = sb; }
  }
  __syncthreads();
  ex_a = s_warp[warp][0] + ia - a;
  ex_b = s_warp[warp][1] + ib - b;
  tot_a = s_warp[kScanWarps][0];
  tot_b = s_warp[kScanWarps][1];
}

// ---------------------------------------------------------------------------
// path marking
// ---------------------------------------------------------------------------
// A warp takes 32 consecutive groups: their ids and bounds in one coalesced load each, then all of their edges together,
// 128 at a time.  One group per eight lanes left every edge behind a chain of three dependent loads with a handful of
// edges to hide them.  BITS: the source mask as one bit per vertex, an eighth of the bytes to gather from (140 KB for
// 1.13 M vertices: L1 holds it).  13 M edges: 148 us before, 97 now (121 with the bits in shared memory: one block of 32
// warps per SM hides less).  The group of an edge was searched for among 32 ends, five shuffles per 32 edges; counting the
// ends in front of it takes a third of that: 68 -> 52 us where issue is the bound (first and last step).
constexpr int kMaskUnroll = 4;

template <bool BITS>
__device__ __forceinline__ bool in_mask(const unsigned char *bytes, const unsigned *bits, int v) {
  if (BITS) return (__ldg(bits + (v >> 5)) >> (v & 31)) & 1u;
  return bytes[v] != 0;
}

__global__ void __launch_bounds__(256) pack_mask_kernel(const unsigned char *__restrict__ mask, int n, unsigned *bits) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned word = __ballot_sync(kFull, v < n && mask[v] != 0);
  if ((threadIdx.x & 31) == 0 && v < n) bits[v >> 5] = word;
}

template <bool BITS>
__global__ void __launch_bounds__(256) mask_forward_kernel(
    const int *__restrict__ ids, const int *__restrict__ part_ptr, const int *__restrict__ edge_list,
    const unsigned char *__restrict__ src_mask, const unsigned *__restrict__ src_bits, unsigned char *ngh_mask,
    int *__restrict__ back_edge_mask, int *__restrict__ node_degs, int num_parts, bool is_last, int row_offset,
    const ClockMark mark_time) {
  if (blockIdx.x == 0 && threadIdx.x == 0) clock_begin(mark_time);
  const int lane = threadIdx.x & 31;
  const long long first = ((static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kWarp;
  if (first >= num_parts) return;
  const long long g = first + lane;
  const bool has = g < num_parts;
  const int r = has ? __ldg(ids + g) : 0;
  const int beg = __ldg(part_ptr + (has ? g : num_parts)), end = __ldg(part_ptr + (has ? g + 1 : num_parts));
  const bool mark = has && !is_last && end > beg && in_mask<BITS>(src_mask, src_bits, r + row_offset);
  const int all_beg = __shfl_sync(kFull, beg, 0), all_end = __shfl_sync(kFull, end, kWarp - 1);
  const bool some_empty = __any_sync(kFull, has && end == beg);
  int count = 0;
  for (int base = all_beg; base < all_end; base += min(kMaskUnroll * kWarp, all_end - base)) {
    int c[kMaskUnroll];
    bool hit[kMaskUnroll];
#pragma unroll
    for (int u = 0; u < kMaskUnroll; ++u) {
      const int at = u * kWarp + lane;
      c[u] = at < all_end - base ? __ldg(edge_list + base + at) : -1;
    }
#pragma unroll
    for (int u = 0; u < kMaskUnroll; ++u) hit[u] = c[u] >= 0 && in_mask<BITS>(src_mask, src_bits, c[u]);
#pragma unroll
    for (int u = 0; u < kMaskUnroll; ++u) {
      if (u * kWarp >= all_end - base) break;
      const int e0 = base + u * kWarp;
      // this lane's group covers bits [lo, hi) of the 32 edges
      const int lo = min(max(beg - e0, 0), kWarp), hi = min(max(end - e0, 0), kWarp);
      const unsigned below_hi = hi >= kWarp ? kFull : (1u << hi) - 1u, below_lo = lo >= kWarp ? kFull : (1u << lo) - 1u;
      count += __popc(__ballot_sync(kFull, hit[u]) & below_hi & ~below_lo);
      // the group of this lane's edge: as many groups end at or before it.  Their ends as bits, where no two coincide;
      // else the first group whose end lies behind the edge, by search.
      const int e = e0 + lane;
      int owner = 0;
      if (!some_empty) {
        const unsigned ends = __reduce_or_sync(kFull, hi > 0 && hi < kWarp ? 1u << hi : 0u);
        owner = min(__popc(__ballot_sync(kFull, hi == 0)) + __popc(ends & ((2u << lane) - 1u)), kWarp - 1);
      } else {
#pragma unroll
        for (int step = kWarp / 2; step >= 1; step >>= 1)
          if (__shfl_sync(kFull, end, owner + step - 1) <= e) owner += step;
      }
      const int row = __shfl_sync(kFull, r, owner);
      const bool marks = __shfl_sync(kFull, static_cast<int>(mark), owner) != 0;
      if (hit[u]) back_edge_mask[e] = row;
      if (marks && c[u] >= 0) ngh_mask[c[u]] = 1;      // looking first costs more: 97 -> 104 us
    }
  }
  if (count) atomicAdd(node_degs + r, count);
  if (mark) ngh_mask[r + row_offset] = 1;
  if (threadIdx.x == 0) clock_end(mark_time);
}

// ---------------------------------------------------------------------------
// stable compaction of (edge_mask, col) pairs with edge_mask != -1
// ---------------------------------------------------------------------------
struct CompactArgs {
  const int *mask;
  int *out_id, *out_edge;
  ScanHeader *hdr;
  unsigned long long *desc;
  int *valid_len, *status;
};
constexpr int kBatch = 16;
struct CompactBatch {               // lists that share `col`, one per blockIdx.y
  CompactArgs list[kBatch];
  const int *col;
  int length, num_tiles;
};

// A kept pair goes behind the kept pairs before it; a dropped one writes a zero as far from the end as there are dropped
// ones before it, which fills the tail without a pass that would have to wait for the count.
template <int MODE>
__global__ void __launch_bounds__(kScanThreads) compact_mask_kernel(const CompactBatch batch) {
  const CompactArgs &a = batch.list[blockIdx.y];
  const int *__restrict__ mask = a.mask;
  const int *__restrict__ col = batch.col;
  int *__restrict__ out_id = a.out_id;
  int *__restrict__ out_edge = a.out_edge;
  const int length = batch.length, num_tiles = batch.num_tiles;
  ScanHeader *hdr = a.hdr;
  unsigned long long *desc = a.desc;
  __shared__ unsigned s_warp[kScanWarps + 1][2];
  __shared__ unsigned s_base;
  __shared__ int s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int tile = blockIdx.x;
  if (MODE == kLookback) {
    if (threadIdx.x == 0) s_tile = static_cast<int>(atomicAdd(&hdr->ticket, 1u));
    __syncthreads();
    tile = s_tile;
  }
  const long long base = static_cast<long long>(tile) * kCompactTile + warp * (kWarp * kCompactItems);
  int m[kCompactItems];
  unsigned ballots[kCompactItems];
  unsigned count = 0;
#pragma unroll
  for (int k = 0; k < kCompactItems; ++k) {
    const long long idx = base + k * kWarp + lane;
    m[k] = idx < length ? __ldg(mask + idx) : -1;
    ballots[k] = __ballot_sync(kFull, m[k] != -1);
    count += __popc(ballots[k]);
  }
  int c[kCompactItems];              // on their way while the tile looks back
  if (MODE != kCountOnly) {
#pragma unroll
    for (int k = 0; k < kCompactItems; ++k) c[k] = m[k] != -1 ? __ldg(col + base + k * kWarp + lane) : 0;
  }
  // warp totals -> exclusive warp offsets (count is warp-uniform)
  if (lane == 0) s_warp[warp][0] = count;
  __syncthreads();
  if (warp == 0) {
    const unsigned w = lane < kScanWarps ? s_warp[lane][0] : 0;
    unsigned s = w;
#pragma unroll
    for (int off = 1; off < kWarp; off <<= 1) {
      const unsigned t = __shfl_up_sync(kFull, s, off);
      if (lane >= off) s += t;
    }
    const unsigned total = __shfl_sync(kFull, s, kWarp - 1);
    if (lane < kScanWarps) s_warp[lane][0] = s - w;
    unsigned ex = 0, unused = 0;
    if (MODE == kLookback) {
      chained_lookback(desc, hdr, a.status, tile, total, 0u, ex, unused);
    } else if (MODE == kCountOnly) {
      if (lane == 0) desc[tile] = tile_pack(0, total, 0);
    } else {
      ex = tile_a(desc[tile]);
    }
    if (lane == 0) {
      s_base = ex;
      if (MODE != kCountOnly && tile == num_tiles - 1) *a.valid_len = static_cast<int>(ex + total);
    }
  }
  if (MODE == kCountOnly) return;
  __syncthreads();
  unsigned offset = s_base + s_warp[warp][0];
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int k = 0; k < kCompactItems; ++k) {
    const long long idx = base + k * kWarp + lane;
    const unsigned dst = offset + __popc(ballots[k] & lt);      // kept pairs before this one
    if (m[k] != -1) {
      out_id[dst] = m[k];
      out_edge[dst] = c[k];
    } else if (idx < length) {
      const long long at = length - 1 - (idx - dst);
      out_id[at] = 0;
      out_edge[at] = 0;
    }
    offset += __popc(ballots[k]);
  }
}

// Exclusive scan of packed tile totals, one block per list; the lists' arrays lie `stride` words apart.
__global__ void __launch_bounds__(1024) scan_tiles_kernel(unsigned long long *desc, int num_tiles, size_t stride) {
  desc += blockIdx.x * stride;
  __shared__ unsigned long long s_warp[33];
  __shared__ unsigned long long s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int base = 0; base < num_tiles; base += 1024) {
    const int i = base + threadIdx.x;
    const unsigned long long v = i < num_tiles ? desc[i] : 0ull;
    unsigned long long s = v;
#pragma unroll
    for (int off = 1; off < kWarp; off <<= 1) {
      const unsigned long long t = __shfl_up_sync(kFull, s, off);
      if (lane >= off) s += t;
    }
    if (lane == 31) s_warp[warp] = s;
    __syncthreads();
    if (warp == 0) {
      const unsigned long long w = s_warp[lane];
      unsigned long long ws = w;
#pragma unroll
      for (int off = 1; off < kWarp; off <<= 1) {
        const unsigned long long t = __shfl_up_sync(kFull, ws, off);
        if (lane >= off) ws += t;
      }
      s_warp[lane] = ws - w;
      if (lane == 31) s_warp[32] = ws;
    }
    __syncthreads();
    if (i < num_tiles) desc[i] = s_carry + s_warp[warp] + s - v;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += s_warp[32];
    __syncthreads();
  }
}

// Self-test of the bounded wait: makes the first ticket 1, so tile 0 -- whose
// descriptor the look-back of tile 1 needs -- never exists.
__global__ void skip_first_ticket_kernel(ScanHeader *hdr) { hdr->ticket = 1u; }

// ---------------------------------------------------------------------------
// splitting active rows into parts
// ---------------------------------------------------------------------------
struct SplitArgs {
  const int *node_deg;
  int *part_pointer, *part2node;
  ScanHeader *hdr;
  unsigned long long *desc;
  int *num_parts, *status;
  int part_size, out_len, part2node_len;
  const int *part_size_dev;          // where it lies, or NULL: part_size
};
struct SplitBatch {                 // one list per blockIdx.y
  SplitArgs list[kBatch];
  int num_nodes, num_tiles;
};

// Zero-fills a list's part pointers behind the closing one.
__global__ void __launch_bounds__(256) zero_tail_kernel(const SplitBatch batch) {
  const SplitArgs &a = batch.list[blockIdx.y];
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(*a.num_parts) + 1 + static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
       i < a.out_len; i += stride)
    a.part_pointer[i] = 0;
}

template <int MODE>
__global__ void __launch_bounds__(kScanThreads) split_parts_kernel(const SplitBatch batch) {
  const SplitArgs &a = batch.list[blockIdx.y];
  const int *__restrict__ node_deg = a.node_deg;
  int *__restrict__ part_pointer = a.part_pointer;
  int *__restrict__ part2node = a.part2node;
  const int num_nodes = batch.num_nodes, num_tiles = batch.num_tiles;
  const int part_size = a.part_size_dev ? __ldg(a.part_size_dev) : a.part_size, out_len = a.out_len, part2node_len = a.part2node_len;
  ScanHeader *hdr = a.hdr;
  unsigned long long *desc = a.desc;
  __shared__ unsigned s_warp[kScanWarps + 1][2];
  __shared__ unsigned s_cpre[kSplitTile + 1];
  __shared__ unsigned s_epre[kSplitTile];
  __shared__ unsigned s_base[2];
  __shared__ int s_tile;
  int tile = blockIdx.x;
  if (MODE == kLookback) {
    if (threadIdx.x == 0) s_tile = static_cast<int>(atomicAdd(&hdr->ticket, 1u));
    __syncthreads();
    tile = s_tile;
  }
  const long long v0 = static_cast<long long>(tile) * kSplitTile + threadIdx.x * kSplitItems;
  unsigned cnt[kSplitItems], deg[kSplitItems];
  unsigned tc = 0, td = 0;
#pragma unroll
  for (int i = 0; i < kSplitItems; ++i) {
    const long long v = v0 + i;
    const int d = v < num_nodes ? __ldg(node_deg + v) : 0;
    deg[i] = d > 0 ? static_cast<unsigned>(d) : 0u;
    cnt[i] = d > 0 ? static_cast<unsigned>((d - 1) / part_size + 1) : 0u;
    tc += cnt[i];
    td += deg[i];
  }
  unsigned ec, ed, tot_c, tot_d;
  block_scan_pair(tc, td, ec, ed, tot_c, tot_d, s_warp);
  if (MODE != kCountOnly) {
#pragma unroll
    for (int i = 0; i < kSplitItems; ++i) {
      s_cpre[threadIdx.x * kSplitItems + i] = ec;
      s_epre[threadIdx.x * kSplitItems + i] = ed;
      ec += cnt[i];
      ed += deg[i];
    }
    if (threadIdx.x == 0) s_cpre[kSplitTile] = tot_c;
  }
  if (threadIdx.x < kWarp) {
    unsigned ex_c = 0, ex_d = 0;
    if (MODE == kLookback) {
      chained_lookback(desc, hdr, a.status, tile, tot_c, tot_d, ex_c, ex_d);
    } else if (MODE == kCountOnly) {
      if (threadIdx.x == 0) desc[tile] = tile_pack(0, tot_c, tot_d);
    } else {
      ex_c = tile_a(desc[tile]);
      ex_d = tile_b(desc[tile]);
    }
    if (threadIdx.x == 0) { s_base[0] = ex_c; s_base[1] = ex_d; }
  }
  if (MODE == kCountOnly) return;
  __syncthreads();
  const unsigned pc = s_base[0], pe = s_base[1];
  // One thread per output slot: find the owning vertex in the tile by binary
  // search over the exclusive part counts (vertices without parts are skipped
  // because they share their successor's prefix).  A warp takes a contiguous
  // stretch of slots; where vertices have several parts each, the owner of a
  // lane's next slot, 32 further on, is a few steps away from the last one
  // (11 M parts of one edge: 77 us by searching every slot, 34 by walking).
  if (part_size == 1 && !part2node) {      // a part is an edge: its pointer is its place (3 x 1.13 M vertices, size 1: 99 us by search, 38)
    for (unsigned j = threadIdx.x; j < tot_c; j += kScanThreads) {
      const long long slot = static_cast<long long>(pc) + j;
      if (slot < out_len) part_pointer[slot] = static_cast<int>(pe + j);
    }
  }
  const unsigned per_warp = (tot_c + kScanThreads - 1) / kScanThreads * kWarp;
  const unsigned stop = part_size == 1 && !part2node ? 0u : min(tot_c, (threadIdx.x / kWarp + 1) * per_warp);
  const bool walk = tot_c >= 4u * kSplitTile;
  int lo = -1;
  for (unsigned j = threadIdx.x / kWarp * per_warp + threadIdx.x % kWarp; j < stop; j += kWarp) {
    if (walk && lo >= 0) {
      while (s_cpre[lo + 1] <= j) ++lo;
    } else {
      lo = 0;
      int hi = kSplitTile;                // largest v with s_cpre[v] <= j
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_cpre[mid] <= j) lo = mid; else hi = mid;
      }
    }
    const unsigned k = j - s_cpre[lo];
    const long long slot = static_cast<long long>(pc) + j;
    if (slot < out_len) part_pointer[slot] = static_cast<int>(pe + s_epre[lo] + k * static_cast<unsigned>(part_size));
    if (part2node && slot < part2node_len) part2node[slot] = tile * kSplitTile + lo;     // the part's vertex
  }
  if (tile == num_tiles - 1 && threadIdx.x == 0) {
    const long long slot = static_cast<long long>(pc) + tot_c;
    if (slot < out_len) part_pointer[slot] = static_cast<int>(pe + tot_d);
    *a.num_parts = static_cast<int>(pc + tot_c);
  }
}

// Row lengths of a CSR, the input of the part splitting when it builds the forward groups.
__global__ void __launch_bounds__(256) row_lengths_kernel(const int *__restrict__ row_ptr, int num_nodes, int *deg) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < num_nodes) deg[v] = __ldg(row_ptr + v + 1) - __ldg(row_ptr + v);
}

struct CountBatch {                 // one array per blockIdx.y
  const int *values[kBatch];
  int *count[kBatch];
  long long length;
};
__global__ void __launch_bounds__(256) count_nonzero_kernel(const CountBatch batch) {
  const int *__restrict__ v = batch.values[blockIdx.y];
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  int c = 0;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < batch.length; i += stride)
    c += __ldg(v + i) != 0;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) c += __shfl_xor_sync(kFull, c, off);
  __shared__ int s[8];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int i = 0; i < 8; ++i) t += s[i];
    if (t) atomicAdd(batch.count[blockIdx.y], t);
  }
}

inline int tail_grid(long long length) {
  long long b = ceil_div_ll(length, 256);
  return static_cast<int>(b < 1 ? 1 : (b > 148 * 8 ? 148 * 8 : b));
}

}  // namespace
}  // namespace epp

using namespace epp;

static int launch_marking(const int *ids, const int *part_ptr, const int *edge_list, const unsigned char *src_mask,
                          const unsigned *src_bits, unsigned char *ngh_mask, int *back_edge_mask, int *node_degs,
                          int num_parts, int is_last, int row_offset, cudaStream_t s) {
  EPP_REQUIRE(num_parts >= 0 && row_offset >= 0, "negative size");
  if (num_parts == 0) return EPP_OK;
  EPP_REQUIRE(ids && part_ptr && edge_list && src_mask && back_edge_mask && node_degs, "null pointer");
  EPP_REQUIRE(is_last || ngh_mask, "ngh_mask is required before the last step");
  const unsigned blocks = static_cast<unsigned>(ceil_div_ll(num_parts, 256));
  if (src_bits)
    mask_forward_kernel<true><<<blocks, 256, 0, s>>>(ids, part_ptr, edge_list, src_mask, src_bits, ngh_mask, back_edge_mask,
                                                     node_degs, num_parts, is_last != 0, row_offset, take_mark());
  else
    mask_forward_kernel<false><<<blocks, 256, 0, s>>>(ids, part_ptr, edge_list, src_mask, nullptr, ngh_mask,
                                                      back_edge_mask, node_degs, num_parts, is_last != 0, row_offset, take_mark());
  EPP_CHECK_LAUNCH("mask_forward_kernel");
  return EPP_OK;
}

EPP_EXPORT int eppgcn_mask_forward(const int *ids, const int *part_ptr, const int *edge_list,
                                   const unsigned char *src_mask, unsigned char *ngh_mask,
                                   int *back_edge_mask, int *node_degs,
                                   int num_parts, int is_last, int row_offset,
                                   int blockx, int blocky, void *stream) {
  (void)blockx; (void)blocky;
  return launch_marking(ids, part_ptr, edge_list, src_mask, nullptr, ngh_mask, back_edge_mask, node_degs, num_parts, is_last,
                        row_offset, static_cast<cudaStream_t>(stream));
}

EPP_EXPORT int eppgcn_mask_forward_packed(const int *ids, const int *part_ptr, const int *edge_list,
                                          const unsigned char *src_mask, int num_sources, unsigned *bits,
                                          unsigned char *ngh_mask, int *back_edge_mask, int *node_degs, int num_parts,
                                          int is_last, int row_offset, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(num_sources >= 0, "negative size");
  if (num_parts <= 0 || num_sources == 0)
    return launch_marking(ids, part_ptr, edge_list, src_mask, nullptr, ngh_mask, back_edge_mask, node_degs, num_parts,
                          is_last, row_offset, s);
  EPP_REQUIRE(src_mask && bits, "null pointer");
  pack_mask_kernel<<<static_cast<unsigned>(ceil_div_ll(num_sources, 256)), 256, 0, s>>>(src_mask, num_sources, bits);
  EPP_CHECK_LAUNCH("pack_mask_kernel");
  return launch_marking(ids, part_ptr, edge_list, src_mask, bits, ngh_mask, back_edge_mask, node_degs, num_parts, is_last,
                        row_offset, s);
}

static size_t scan_scratch_bytes(long long tiles) {
  return sizeof(ScanHeader) + sizeof(unsigned long long) * static_cast<size_t>(tiles < 1 ? 1 : tiles);
}

EPP_EXPORT size_t eppgcn_compact_scratch_bytes(int length) {
  return scan_scratch_bytes(ceil_div_ll(length < 0 ? 0 : length, kCompactTile));
}

EPP_EXPORT size_t eppgcn_split_scratch_bytes(int num_nodes) {
  return scan_scratch_bytes(ceil_div_ll(num_nodes < 0 ? 0 : num_nodes, kSplitTile));
}

// {count, status} of a list start from zero: one memset where they are neighbours.
static int clear_results(int *count, int *status, cudaStream_t s) {
  if (status == count + 1) {
    EPP_CUDA_TRY(cudaMemsetAsync(count, 0, 2 * sizeof(int), s));
  } else {
    EPP_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(int), s));
    EPP_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), s));
  }
  return EPP_OK;
}

static CompactArgs compact_args(const int *mask, int *out_id, int *out_edge, void *scratch, int *valid_len, int *status) {
  ScanHeader *hdr = static_cast<ScanHeader *>(scratch);
  return CompactArgs{mask, out_id, out_edge, hdr, reinterpret_cast<unsigned long long *>(hdr + 1), valid_len, status};
}

EPP_EXPORT int eppgcn_compact_mask(const int *edge_mask, const int *col_idx, int *out_id, int *out_edge,
                                   int length, void *scratch, size_t scratch_bytes,
                                   int *valid_len_dev, int *status_dev, int mode, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(length >= 0, "negative length");
  EPP_REQUIRE(valid_len_dev && status_dev, "null result pointer");
  EPP_REQUIRE(mode >= 0 && mode <= 2, "mode must be 0, 1 or 2");
  EPP_REQUIRE(mode != 2 || length > kCompactTile, "the wait self-test needs more than one tile of input");
  if (const int rc = clear_results(valid_len_dev, status_dev, s); rc != EPP_OK) return rc;
  if (length == 0) return EPP_OK;
  EPP_REQUIRE(edge_mask && col_idx && out_id && out_edge && scratch, "null pointer");
  EPP_REQUIRE(scratch_bytes >= eppgcn_compact_scratch_bytes(length), "scratch too small");
  EPP_REQUIRE(reinterpret_cast<uintptr_t>(scratch) % 8 == 0, "scratch must be 8-byte aligned");
  const int tiles = static_cast<int>(ceil_div_ll(length, kCompactTile));
  CompactBatch b{};
  b.list[0] = compact_args(edge_mask, out_id, out_edge, scratch, valid_len_dev, status_dev);
  b.col = col_idx;
  b.length = length;
  b.num_tiles = tiles;
  EPP_CUDA_TRY(cudaMemsetAsync(scratch, 0, scan_scratch_bytes(tiles), s));
  if (mode == 0) {
    compact_mask_kernel<kLookback><<<tiles, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("compact_mask_kernel<lookback>");
  } else if (mode == 2) {
    // tile ids 1 .. tiles-1 are handed out; tile 1 looks back at a descriptor nobody writes, its
    // bounded wait runs out, the error word is set and every other tile leaves as soon as it sees it
    skip_first_ticket_kernel<<<1, 1, 0, s>>>(b.list[0].hdr);
    EPP_CHECK_LAUNCH("skip_first_ticket_kernel");
    compact_mask_kernel<kLookback><<<tiles - 1, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("compact_mask_kernel<lookback, wait self-test>");
  } else {
    compact_mask_kernel<kCountOnly><<<tiles, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("compact_mask_kernel<count>");
    scan_tiles_kernel<<<1, 1024, 0, s>>>(b.list[0].desc, tiles, 0);
    EPP_CHECK_LAUNCH("scan_tiles_kernel");
    compact_mask_kernel<kGivenOffsets><<<tiles, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("compact_mask_kernel<scatter>");
  }
  return EPP_OK;
}

static size_t list_scratch_bytes(long long tiles) { return (scan_scratch_bytes(tiles) + 255) / 256 * 256; }

EPP_EXPORT size_t eppgcn_compact_masks_scratch_bytes(int lists, int length) {
  return lists < 1 ? 0 : static_cast<size_t>(lists) * list_scratch_bytes(ceil_div_ll(length < 0 ? 0 : length, kCompactTile));
}

EPP_EXPORT int eppgcn_compact_masks(int lists, const int *const *edge_masks, const int *col_idx, const int *const *node_degs,
                                    int *const *out_ids, int *const *out_edges, int length, int num_nodes, void *scratch,
                                    size_t scratch_bytes, int *results_dev, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(lists >= 0 && lists <= kBatch && length >= 0 && num_nodes >= 0, "bad size (at most 16 lists)");
  if (lists == 0) return EPP_OK;
  EPP_REQUIRE(edge_masks && node_degs && out_ids && out_edges && results_dev, "null pointer");
  EPP_REQUIRE(length == 0 || (col_idx && scratch), "null pointer");
  EPP_REQUIRE(scratch_bytes >= eppgcn_compact_masks_scratch_bytes(lists, length), "scratch too small");
  EPP_REQUIRE(reinterpret_cast<uintptr_t>(scratch) % 8 == 0, "scratch must be 8-byte aligned");
  const int tiles = static_cast<int>(ceil_div_ll(length, kCompactTile));
  CompactBatch b{};
  CountBatch n{};
  b.col = col_idx;
  b.length = length;
  b.num_tiles = tiles;
  n.length = num_nodes;
  for (int i = 0; i < lists; ++i) {
    EPP_REQUIRE((length == 0 || (edge_masks[i] && out_ids[i] && out_edges[i])) && (num_nodes == 0 || node_degs[i]), "null pointer");
    b.list[i] = compact_args(edge_masks[i], out_ids[i], out_edges[i], static_cast<char *>(scratch) + i * list_scratch_bytes(tiles),
                             results_dev + 4 * i, results_dev + 4 * i + 1);
    n.values[i] = node_degs[i];
    n.count[i] = results_dev + 4 * i + 2;
  }
  EPP_CUDA_TRY(cudaMemsetAsync(results_dev, 0, sizeof(int) * 4 * lists, s));
  if (length > 0) {
    EPP_CUDA_TRY(cudaMemsetAsync(scratch, 0, lists * list_scratch_bytes(tiles), s));
    // Tiles that all start at once look back over each other in one launch.  Where there are more, waiting for the tiles
    // before costs more than counting first and reading the masks twice (3 x 13 M edges: 227 us, 169).
    if (static_cast<long long>(tiles) * lists <= kOneWaveTiles) {
      compact_mask_kernel<kLookback><<<dim3(tiles, lists), kScanThreads, 0, s>>>(b);
      EPP_CHECK_LAUNCH("compact_mask_kernel<lookback, batch>");
    } else {
      compact_mask_kernel<kCountOnly><<<dim3(tiles, lists), kScanThreads, 0, s>>>(b);
      EPP_CHECK_LAUNCH("compact_mask_kernel<count, batch>");
      scan_tiles_kernel<<<lists, 1024, 0, s>>>(b.list[0].desc, tiles, list_scratch_bytes(tiles) / sizeof(unsigned long long));
      EPP_CHECK_LAUNCH("scan_tiles_kernel");
      compact_mask_kernel<kGivenOffsets><<<dim3(tiles, lists), kScanThreads, 0, s>>>(b);
      EPP_CHECK_LAUNCH("compact_mask_kernel<scatter, batch>");
    }
  }
  if (num_nodes > 0) {
    count_nonzero_kernel<<<dim3(tail_grid(num_nodes), lists), 256, 0, s>>>(n);
    EPP_CHECK_LAUNCH("count_nonzero_kernel<batch>");
  }
  return EPP_OK;
}

// ---------------------------------------------------------------------------
// Compaction without any allocation by anyone.
//
// Some hosts cannot give this library scratch memory at call time: a process
// that handed the whole device to its own pool at start-up and runs without
// headroom, a latency-critical thread that must never hit the device-wide
// synchronisation cudaMalloc/cudaFree imply, or an embedding application that
// forbids device allocation after initialisation.  For them the tile
// descriptors of the single-pass scan live in this fixed array instead of a
// caller-supplied buffer.  It is part of the library image: every GPU that
// loads the library holds these bytes until the process exits.
// ---------------------------------------------------------------------------
constexpr int kStaticCompactMaxLength = 1 << 26;   // 67,108,864 edges
constexpr size_t kStaticCompactBytes =
    sizeof(epp::ScanHeader) + sizeof(unsigned long long) * (kStaticCompactMaxLength / epp::kCompactTile);   // 131,328 B
static __device__ __align__(256) unsigned char g_static_compact_scratch[kStaticCompactBytes];

// In host code `g_static_compact_scratch` is only a handle for the runtime, not
// a device address; the address is looked up once per device, with that device
// current, and cached.
static int static_compact_scratch_address(void **ptr) {
  constexpr int kMaxDevices = 64;
  static void *cached[kMaxDevices] = {nullptr};
  int dev = 0;
  EPP_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) {
    set_error("device ordinal %d is beyond the %d devices this entry point tracks", dev, kMaxDevices);
    return EPP_ERR_TOO_LARGE;
  }
  if (!cached[dev]) {
    void *p = nullptr;
    EPP_CUDA_TRY(cudaGetSymbolAddress(&p, g_static_compact_scratch));
    if (!p || reinterpret_cast<uintptr_t>(p) % 256 != 0) {
      set_error("static scratch symbol resolved to an unusable address");
      return EPP_ERR_CUDA;
    }
    cached[dev] = p;
  }
  *ptr = cached[dev];
  return EPP_OK;
}

EPP_EXPORT int eppgcn_compact_mask_static(const int *edge_mask, const int *col_idx, int *out_id, int *out_edge,
                                          int length, int *valid_len_dev, int *status_dev, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(length >= 0, "negative length");
  EPP_REQUIRE(valid_len_dev && status_dev, "null result pointer");
  if (length > kStaticCompactMaxLength) {
    set_error("eppgcn_compact_mask_static handles at most %d edges per call, got %d; "
              "use eppgcn_compact_mask with caller-provided scratch", kStaticCompactMaxLength, length);
    return EPP_ERR_TOO_LARGE;
  }
  void *scratch = nullptr;
  const int rc = static_compact_scratch_address(&scratch);
  if (rc != EPP_OK) return rc;
  if (const int rz = clear_results(valid_len_dev, status_dev, s); rz != EPP_OK) return rz;
  if (length == 0) return EPP_OK;
  EPP_REQUIRE(edge_mask && col_idx && out_id && out_edge, "null pointer");
  const int tiles = static_cast<int>(ceil_div_ll(length, kCompactTile));
  CompactBatch b{};
  b.list[0] = compact_args(edge_mask, out_id, out_edge, scratch, valid_len_dev, status_dev);
  b.col = col_idx;
  b.length = length;
  b.num_tiles = tiles;
  // The array keeps the previous call's ticket, error word and descriptors:
  // everything this call will read has to start from zero again.
  EPP_CUDA_TRY(cudaMemsetAsync(scratch, 0, scan_scratch_bytes(tiles), s));
  compact_mask_kernel<kLookback><<<tiles, kScanThreads, 0, s>>>(b);
  EPP_CHECK_LAUNCH("compact_mask_kernel<lookback, static scratch>");
  return EPP_OK;
}

static SplitArgs split_args(const int *node_deg, int part_size, int *part_pointer, int out_len, int *part2node,
                            int part2node_len, void *scratch, int *num_parts, int *status) {
  ScanHeader *hdr = static_cast<ScanHeader *>(scratch);
  return SplitArgs{node_deg, part_pointer, part2node, hdr, reinterpret_cast<unsigned long long *>(hdr + 1), num_parts, status,
                   part_size, out_len, part2node_len};
}

// One list in either mode; the scratch is cleared here.
static int launch_split(const SplitArgs &a, int num_nodes, int mode, cudaStream_t s) {
  SplitBatch b{};
  b.list[0] = a;
  b.num_nodes = num_nodes;
  b.num_tiles = static_cast<int>(ceil_div_ll(num_nodes, kSplitTile));
  EPP_CUDA_TRY(cudaMemsetAsync(a.hdr, 0, scan_scratch_bytes(b.num_tiles), s));
  if (mode == 0) {
    split_parts_kernel<kLookback><<<b.num_tiles, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("split_parts_kernel<lookback>");
  } else {
    split_parts_kernel<kCountOnly><<<b.num_tiles, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("split_parts_kernel<count>");
    scan_tiles_kernel<<<1, 1024, 0, s>>>(a.desc, b.num_tiles, 0);
    EPP_CHECK_LAUNCH("scan_tiles_kernel");
    split_parts_kernel<kGivenOffsets><<<b.num_tiles, kScanThreads, 0, s>>>(b);
    EPP_CHECK_LAUNCH("split_parts_kernel<scatter>");
  }
  return EPP_OK;
}

static int zero_split_tails(const SplitBatch &b, int lists, int longest, cudaStream_t s) {
  if (longest == 0) return EPP_OK;
  zero_tail_kernel<<<dim3(tail_grid(longest), lists), 256, 0, s>>>(b);
  EPP_CHECK_LAUNCH("zero_tail_kernel");
  return EPP_OK;
}

EPP_EXPORT size_t eppgcn_split_lists_scratch_bytes(int lists, int num_nodes) {
  return lists < 1 ? 0 : static_cast<size_t>(lists) * list_scratch_bytes(ceil_div_ll(num_nodes < 0 ? 0 : num_nodes, kSplitTile));
}

// part_sizes: on the host, or -- one of the two -- in device memory, `size_stride` ints apart.
static int split_lists(int lists, const int *const *node_degs, int num_nodes, const int *part_sizes, const int *part_sizes_dev,
                       int size_stride, int *const *part_pointers, int out_len, void *scratch, int *results_dev,
                       int result_stride, cudaStream_t s) {
  SplitBatch b{};
  b.num_nodes = num_nodes;
  b.num_tiles = static_cast<int>(ceil_div_ll(num_nodes, kSplitTile));
  for (int i = 0; i < lists; ++i) {
    EPP_REQUIRE(node_degs[i] && part_pointers[i] && (!part_sizes || part_sizes[i] >= 1), "null pointer or part size < 1");
    b.list[i] = split_args(node_degs[i], part_sizes ? part_sizes[i] : 0, part_pointers[i], out_len, nullptr, 0,
                           static_cast<char *>(scratch) + i * list_scratch_bytes(b.num_tiles), results_dev + result_stride * i,
                           results_dev + result_stride * i + 1);
    if (!part_sizes) b.list[i].part_size_dev = part_sizes_dev + size_stride * i;
  }
  EPP_CUDA_TRY(cudaMemsetAsync(scratch, 0, lists * list_scratch_bytes(b.num_tiles), s));
  split_parts_kernel<kLookback><<<dim3(b.num_tiles, lists), kScanThreads, 0, s>>>(b);
  EPP_CHECK_LAUNCH("split_parts_kernel<lookback, batch>");
  return zero_split_tails(b, lists, out_len, s);
}

EPP_EXPORT int eppgcn_split_lists(int lists, const int *const *node_degs, int num_nodes, const int *part_sizes,
                                  int *const *part_pointers, int out_len, void *scratch, size_t scratch_bytes,
                                  int *results_dev, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(lists >= 0 && lists <= kBatch && num_nodes >= 1 && out_len >= 1, "bad size (at most 16 lists)");
  if (lists == 0) return EPP_OK;
  EPP_REQUIRE(node_degs && part_sizes && part_pointers && scratch && results_dev, "null pointer");
  EPP_REQUIRE(scratch_bytes >= eppgcn_split_lists_scratch_bytes(lists, num_nodes), "scratch too small");
  EPP_REQUIRE(reinterpret_cast<uintptr_t>(scratch) % 8 == 0, "scratch must be 8-byte aligned");
  EPP_CUDA_TRY(cudaMemsetAsync(results_dev, 0, sizeof(int) * 2 * lists, s));
  return split_lists(lists, node_degs, num_nodes, part_sizes, nullptr, 0, part_pointers, out_len, scratch, results_dev, 2, s);
}

// The part size of every list from its counts, as eppgcn_map_back_part_size and the bucket rule give it, at least 1.
// results: {valid, status, active, size, ...} per list.
__global__ void part_sizes_kernel(int *results, int stride, int lists, int rule, int constant) {
  const int i = threadIdx.x;
  if (i >= lists) return;
  int *const r = results + i * stride;
  const int valid = r[0], active = r[2];
  int size = constant;
  if (rule == EPP_PART_SIZE_MAP && active > 0) {      // rounded like the host's sum: no fused multiply-add
    const double degree = __ddiv_rn(static_cast<double>(valid), static_cast<double>(active));
    double sum = __dadd_rn(0.65538, __dmul_rn(1.67431e-5, static_cast<double>(active)));
    sum = __dadd_rn(sum, __dmul_rn(-2.24342e-6, static_cast<double>(valid)));
    sum = __dadd_rn(sum, __dmul_rn(0.63641, degree));
    size = static_cast<int>(round(sum));
  } else if (rule == EPP_PART_SIZE_BUCKET) {
    const int d = valid / max(active, 1);
    size = d < 4 ? 4 : d < 16 ? 8 : d < 64 ? 16 : d < 256 ? 32 : 64;
  }
  r[3] = max(size, 1);
}

EPP_EXPORT size_t eppgcn_prepare_lists_scratch_bytes(int lists, int length, int num_nodes) {
  return eppgcn_compact_masks_scratch_bytes(lists, length) + eppgcn_split_lists_scratch_bytes(lists, num_nodes);
}

EPP_EXPORT int eppgcn_prepare_lists(int lists, const int *const *edge_masks, const int *col_idx, const int *const *node_degs,
                                    int *const *out_ids, int *const *out_edges, int length, int num_nodes, int rule, int constant,
                                    int *const *part_pointers, int out_len, void *scratch, size_t scratch_bytes,
                                    int *results_dev, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(lists >= 0 && lists <= kBatch && num_nodes >= 1 && length >= 1 && out_len >= 1, "bad size (at most 16 lists)");
  if (lists == 0) return EPP_OK;
  EPP_REQUIRE(rule == EPP_PART_SIZE_CONSTANT || rule == EPP_PART_SIZE_MAP || rule == EPP_PART_SIZE_BUCKET, "unknown rule");
  EPP_REQUIRE(part_pointers && scratch && results_dev, "null pointer");
  EPP_REQUIRE(scratch_bytes >= eppgcn_prepare_lists_scratch_bytes(lists, length, num_nodes), "scratch too small");
  const size_t compact_bytes = eppgcn_compact_masks_scratch_bytes(lists, length);
  int *const split_results = results_dev + 4 * lists;
  if (const int rc = eppgcn_compact_masks(lists, edge_masks, col_idx, node_degs, out_ids, out_edges, length, num_nodes, scratch,
                                          compact_bytes, results_dev, stream);
      rc != EPP_OK)
    return rc;
  EPP_CUDA_TRY(cudaMemsetAsync(split_results, 0, sizeof(int) * 2 * lists, s));
  part_sizes_kernel<<<1, kBatch, 0, s>>>(results_dev, 4, lists, rule, constant);
  EPP_CHECK_LAUNCH("part_sizes_kernel");
  return split_lists(lists, node_degs, num_nodes, nullptr, results_dev + 3, 4, part_pointers, out_len,
                     static_cast<char *>(scratch) + compact_bytes, split_results, 2, s);
}

EPP_EXPORT int eppgcn_split_parts(const int *node_deg, int num_nodes, int part_size, int *part_pointer,
                                  int out_len, void *scratch, size_t scratch_bytes, int *num_parts_dev,
                                  int *status_dev, int mode, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(num_nodes >= 0 && out_len >= 0, "negative size");
  EPP_REQUIRE(part_size >= 1, "back part size must be >= 1");
  EPP_REQUIRE(num_parts_dev && status_dev, "null result pointer");
  EPP_REQUIRE(mode == 0 || mode == 1, "mode must be 0 or 1");
  if (const int rc = clear_results(num_parts_dev, status_dev, s); rc != EPP_OK) return rc;
  EPP_REQUIRE(out_len == 0 || part_pointer, "null pointer");
  if (num_nodes == 0) {
    if (out_len) EPP_CUDA_TRY(cudaMemsetAsync(part_pointer, 0, sizeof(int) * static_cast<size_t>(out_len), s));
    return EPP_OK;
  }
  EPP_REQUIRE(node_deg && scratch, "null pointer");
  EPP_REQUIRE(scratch_bytes >= eppgcn_split_scratch_bytes(num_nodes), "scratch too small");
  EPP_REQUIRE(reinterpret_cast<uintptr_t>(scratch) % 8 == 0, "scratch must be 8-byte aligned");
  SplitBatch b{};
  b.list[0] = split_args(node_deg, part_size, part_pointer, out_len, nullptr, 0, scratch, num_parts_dev, status_dev);
  if (const int rc = launch_split(b.list[0], num_nodes, mode, s); rc != EPP_OK) return rc;
  return zero_split_tails(b, 1, out_len, s);
}

EPP_EXPORT int eppgcn_count_nonzero(const int *values, int length, int *count_dev, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(length >= 0 && count_dev, "bad argument");
  EPP_CUDA_TRY(cudaMemsetAsync(count_dev, 0, sizeof(int), s));
  if (length == 0) return EPP_OK;
  EPP_REQUIRE(values, "null pointer");
  CountBatch n{};
  n.values[0] = values;
  n.count[0] = count_dev;
  n.length = length;
  count_nonzero_kernel<<<tail_grid(length), 256, 0, s>>>(n);
  EPP_CHECK_LAUNCH("count_nonzero_kernel");
  return EPP_OK;
}

// ---------------------------------------------------------------------------
// Neighbour groups on the device.  build_part (EPPGCN.cpp:186-227) and the
// part splitting compute the same thing from different inputs: a vertex with d
// edges yields ceil(d / part_size) consecutive pieces of its edge range.  With
// the row lengths of the CSR as "node degrees", the splitting kernel's part
// pointers are the group pointers (edge offsets equal CSR offsets), and the
// vertex it finds for every slot is part2Node.
// ---------------------------------------------------------------------------
EPP_EXPORT size_t eppgcn_build_part_scratch_bytes(int num_nodes) {
  const size_t n = num_nodes < 0 ? 0 : static_cast<size_t>(num_nodes);
  return (eppgcn_split_scratch_bytes(num_nodes) + 255) / 256 * 256 + sizeof(int) * (n + 1);
}

EPP_EXPORT int eppgcn_build_part(const int *row_ptr, int num_nodes, int part_size, int *part_ptr, int part_ptr_len,
                                 int *part2node, int part2node_len, void *scratch, size_t scratch_bytes,
                                 int *num_parts_dev, int *status_dev, int mode, void *stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  EPP_REQUIRE(num_nodes >= 0 && part_ptr_len >= 0 && part2node_len >= 0, "negative size");
  EPP_REQUIRE(part_size >= 1, "part size must be >= 1");
  EPP_REQUIRE(num_parts_dev && status_dev, "null result pointer");
  EPP_REQUIRE(mode == 0 || mode == 1, "mode must be 0 or 1");
  if (const int rc = clear_results(num_parts_dev, status_dev, s); rc != EPP_OK) return rc;
  EPP_REQUIRE(part_ptr_len == 0 || part_ptr, "null pointer");
  EPP_REQUIRE(part2node_len == 0 || part2node, "null pointer");
  if (num_nodes == 0) {
    if (part_ptr_len) EPP_CUDA_TRY(cudaMemsetAsync(part_ptr, 0, sizeof(int) * static_cast<size_t>(part_ptr_len), s));
    return EPP_OK;
  }
  EPP_REQUIRE(row_ptr && scratch, "null pointer");
  EPP_REQUIRE(scratch_bytes >= eppgcn_build_part_scratch_bytes(num_nodes), "scratch too small");
  EPP_REQUIRE(reinterpret_cast<uintptr_t>(scratch) % 8 == 0, "scratch must be 8-byte aligned");
  const size_t scan_bytes = (eppgcn_split_scratch_bytes(num_nodes) + 255) / 256 * 256;
  int *deg = reinterpret_cast<int *>(static_cast<char *>(scratch) + scan_bytes);
  row_lengths_kernel<<<static_cast<unsigned>(ceil_div_ll(num_nodes, 256)), 256, 0, s>>>(row_ptr, num_nodes, deg);
  EPP_CHECK_LAUNCH("row_lengths_kernel");
  return launch_split(split_args(deg, part_size, part_ptr, part_ptr_len, part2node, part2node_len, scratch, num_parts_dev,
                                 status_dev),
                      num_nodes, mode, s);
}
