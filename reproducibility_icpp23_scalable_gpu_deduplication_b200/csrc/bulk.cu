// Bulk build of a baseline's tree digests and digest map.
//
// A baseline starts from an empty map and puts every node's digest into it.  Inserted one by one
// (leaf.cu, forest.cu) each is a read, a claim and an update of a random 32-byte slot: 9 to 13 G
// inserts per second on this device whatever the table's size, 8.4 of the 11 ms of a 4 GiB
// baseline at 128 B chunks.  The digests of a tree do not depend on its labels, so here the leaf
// stage only hashes, and then
//   tree_hash   hashes every inner node, 7 levels per launch;
//   part_*      partitions all (digest, node) pairs by the table range their home slot lies in:
//               one counting pass, then one or two scatter passes;
//   build       makes each range of the table in shared memory and writes it out once, empty slots
//               included (the table is not cleared before).
// All of it streams: per node 16 bytes read twice, 20 written and read once per scatter pass, and
// the table written once.  Whole baselines at 128 B chunks: 4 GiB 11.1, now 6.4 ms; 64 MiB 380, now
// 220 us.  Of the 4 GiB's 4.2 ms here the writing of the 8.6 GB table takes 2.2 and the scatter
// passes 1.35.
//
// All copies of a digest fall to one table range and so to one CTA of the build, which is what bounds
// contents of few, scattered values; the one-by-one inserts meet in one slot there, and are no faster
// to speak of at the worst of them.  Baselines at 128 B chunks, one by one and in bulk, ms: 4 GiB,
// random 11.6 and 6.4; 10 % of the chunks zero 17.6 and 11.3, 50 % 30.6 and 19.8; chunks that repeat
// with period 1, 2, 3, 16 and 1000: 45.9 and 19.4, 34.9 and 33.7, 24.8 and 21.5, 14.6 and 14.1, 11.8
// and 9.6; period 2 at 64 MiB 0.74 and 0.75, in a list of 512 MiB 2.59 and 2.70.
//
// The result is the map the one-by-one inserts leave (src/tree_approach.cpp:54-94, 116-145,
// 218-224 in sequential order): an entry is owned by its lowest leaf, else by its lowest
// first-occurrence parent by (height, index), else by its lowest other parent.  Build cannot know
// which parents are first occurrences, as that follows from the duplicates among the leaves it is
// finding; it gives every parent that priority, marks the parents that lost their entry to another
// parent, and phase 2 settles both (bulk_settle in forest.cu): a parent that is no first occurrence
// takes its real priority, and a marked one that is becomes the owner.  Leaves that lose to a
// lower leaf are shifted duplicates, and build labels them so ("Choose first occurrences", :100-114).
#include "bulk.cuh"
#include "hash.cuh"

namespace b2d {

constexpr uint32_t BULK_RANGE = 16384;      // slots per table range (one build step: 64 KB of indexes)
constexpr uint32_t BULK_MAX_RANGES = 32768; // counted in shared memory (128 KB)
constexpr uint32_t BULK_FAN = 64;           // ranges per bucket of the first scatter of two
constexpr uint32_t BULK_ONE_PASS = 256;     // up to so many ranges, one scatter pass
constexpr uint32_t COUNT_THREADS = 1024;
constexpr uint32_t PART_THREADS = 512;
constexpr uint32_t PART_TILE = 2048;
constexpr uint32_t PART_CTAS = 4;          // resident CTAs per SM
constexpr uint32_t PART_DIGITS = 512;       // buckets of one scatter pass
constexpr uint32_t BUILD_THREADS = 512;
constexpr uint32_t BUILD_CTAS = 2;         // resident CTAs per SM
constexpr uint32_t BUILD_IN = 4;           // entries per thread in flight
constexpr uint32_t BUILD_OUT = 8;          // pieces written per thread and step
constexpr uint32_t NO_ENTRY = 0xffffffffu;

__device__ __forceinline__ void bulk_stamp(const BulkArgs& a) {
  if (a.stamp && blockIdx.x == 0 && threadIdx.x == 0) *a.stamp = device_time_ns();
}
// a node whose entry is inserted once every range is written (probing left the range; the EMPTY
// pattern); more than one per chunk would take digests that are no hash of anything
__device__ __forceinline__ void bulk_overflow(const BulkArgs& a, uint32_t node) {
  const uint32_t at = atomicAdd(a.over_count, 1u);
  if (at < a.n) a.overflow[at] = node;
  else set_error(a.st, DERR_MAP_FULL, 1);
}
__device__ __forceinline__ uint32_t range_of(const BulkArgs& a, const Key128& k) {
  return (uint32_t)(map_home(k, a.map.cap) / BULK_RANGE);
}
__device__ __forceinline__ Key128 node_key(const BulkArgs& a, uint64_t i) {
  return reinterpret_cast<const Key128*>(a.tree)[a.first_node + i];
}
// kept out of the ranges: the EMPTY pattern (it has a slot of its own), a list's zero digests (a
// chunk equal to the zeroed list is FIXED and never inserted), and nodes known to have lost their
// entry to a neighbour of equal digest
__device__ __forceinline__ bool lost_before(const BulkArgs& a, uint64_t i) {
  const uint32_t node = a.first_node + (uint32_t)i;
  return node >= a.n - 1u ? a.leaflab[node - (a.n - 1u)] == SHIFT_DUPL
                          : ((a.lost[node >> 5] >> (node & 31u)) & 1u) != 0u;
}
__device__ __forceinline__ bool left_out(const BulkArgs& a, const Key128& k, bool lost) {
  return lost || key_is_empty_pattern(k) || (a.list && k.lo == 0ull && k.hi == 0ull);
}

// ------------------------------------------------------------------ inner digests
// A node whose digest equals its left neighbour's on the same level has lost its entry to it: it
// is marked and left out of the partition.  Runs of equal chunks (zero pages) would otherwise put
// all their nodes into one range: 0.4 M of them kept one CTA of the build busy for 1 ms.
__device__ __forceinline__ void mark_lost(const BulkArgs& a, uint32_t node) {
  atomicOr(&a.lost[node >> 5], 1u << (node & 31u));
  *a.lost_any = 1;
}
// stores the digest of inner node x; `left`: the digest of node x - 1 of the same level, if known
__device__ __forceinline__ void put_inner(const BulkArgs& a, uint64_t x, const Digest& d, const Digest& left,
                                          bool has_left) {
  a.tree[x] = d;
  if (digest_zero(d)) *a.zero_exists = 1;
  if (has_left && digest_eq(d, left)) mark_lost(a, (uint32_t)x);
}
__device__ __forceinline__ Digest shfl_digest_up(const Digest& d, uint32_t delta) {
  Digest r;
#pragma unroll
  for (int q = 0; q < 4; q++) r.w[q] = __shfl_up_sync(0xffffffffu, d.w[q], delta);
  return r;
}
// digest of node x above two nodes of level `in` (already in the tree), or of the leaf x
__device__ __forceinline__ Digest above(const BulkArgs& a, uint64_t x, bool& inner) {
  inner = x < (uint64_t)a.n - 1u;
  return inner ? hash_pair(a.kind, a.tree[2 * x + 1], a.tree[2 * x + 2]) : a.tree[x];
}

// The two levels above level `in` >= 2: four nodes per lane from memory, three hashes in
// registers, so every lane has work throughout.  They hold three quarters of the inner nodes; by
// the shuffles of tree_hash_kernel the first levels of a 2^25-leaf tree took 377 us.  Nodes that
// are leaves (level D-1 of a tree whose chunk count is not a power of two) keep their digest.
__global__ void __launch_bounds__(256) tree_hash2_kernel(BulkArgs a, uint32_t in) {
  griddep_enter();
  bulk_stamp(a);
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t tasks = 1ull << (in - 2u), warps = (tasks + 31u) / 32u;
  for (uint64_t w = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; w < warps;
       w += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint64_t t = 32u * w + lane;
    const bool act = t < tasks;
    const uint64_t x = (1ull << (in - 1u)) - 1ull + 2u * t, y = (1ull << (in - 2u)) - 1ull + t;
    const Digest zero = Digest{{0u, 0u, 0u, 0u}};
    Digest d0 = zero, d1 = zero, dy = zero;
    bool in0 = false, in1 = false;
    if (act) {
      d0 = above(a, x, in0);
      d1 = above(a, x + 1u, in1);
      dy = hash_pair(a.kind, d0, d1);
    }
    const Digest l1 = shfl_digest_up(d1, 1), ly = shfl_digest_up(dy, 1);
    const uint32_t l1_in = __shfl_up_sync(0xffffffffu, (uint32_t)in1, 1);
    if (act) {
      if (in0) put_inner(a, x, d0, l1, lane > 0u && l1_in);
      if (in1) put_inner(a, x + 1u, d1, d0, in0);
      put_inner(a, y, dy, ly, lane > 0u);
    }
  }
}

// One warp per subtree of 2^k nodes at level `in` (k <= 7), hashed up to its root: the 2^(k-1)
// nodes above two to a lane from memory, the next level in registers, the rest by shuffles.
constexpr uint32_t HASH_LEVELS = 7;
__global__ void __launch_bounds__(256) tree_hash_kernel(BulkArgs a, uint32_t in, uint32_t k) {
  griddep_enter();
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t tasks = 1ull << (in - k);
  for (uint64_t t = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; t < tasks;
       t += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    uint64_t first = (1ull << (in - 1u)) - 1ull + (t << (k - 1u));   // the subtree's nodes at level in - 1
    const uint32_t width = 1u << (k - 1u);
    Digest d[2];
#pragma unroll
    for (uint32_t j = 0; j < 2; j++) {
      const uint32_t i = 2u * lane + j;
      const uint64_t x = first + i;
      d[j] = Digest{{0u, 0u, 0u, 0u}};
      if (i >= width) continue;
      d[j] = hash_pair(a.kind, a.tree[2 * x + 1], a.tree[2 * x + 2]);
      put_inner(a, x, d[j], d[0], j > 0u);
    }
    if (width < 2u) continue;
    first = (first - 1ull) >> 1;
    Digest dg = Digest{{0u, 0u, 0u, 0u}};
    if (lane < width / 2u) dg = hash_pair(a.kind, d[0], d[1]);
    const Digest lg = shfl_digest_up(dg, 1);
    if (lane < width / 2u) put_inner(a, first + lane, dg, lg, lane > 0u);
    for (uint32_t w = width / 4u, s = 0; w >= 1u; w >>= 1, s++) {
      first = (first - 1ull) >> 1;
      Digest rd;
#pragma unroll
      for (int q = 0; q < 4; q++) rd.w[q] = __shfl_down_sync(0xffffffffu, dg.w[q], 1u << s);
      const uint32_t i = lane >> (s + 1u);
      if ((lane & ((2u << s) - 1u)) == 0u && i < w) {
        dg = hash_pair(a.kind, dg, rd);
        put_inner(a, first + i, dg, dg, false);
      }
    }
  }
}

// ------------------------------------------------------------------ partition
__global__ void __launch_bounds__(COUNT_THREADS) part_count_kernel(BulkArgs a) {
  extern __shared__ uint32_t cnt[];
  griddep_enter();
  bulk_stamp(a);
  for (uint32_t i = threadIdx.x; i < a.ranges; i += blockDim.x) cnt[i] = 0;
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  constexpr int U = 6;   // loads in flight per thread
  for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i0 < a.count; i0 += U * stride) {
    Key128 k[U];
    bool lost[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
      lost[j] = true;
      if (i0 + j * stride < a.count) {
        k[j] = node_key(a, i0 + j * stride);
        lost[j] = lost_before(a, i0 + j * stride);
      }
    }
#pragma unroll
    for (int j = 0; j < U; j++)
      if (!lost[j] && !left_out(a, k[j], false)) atomicAdd(&cnt[range_of(a, k[j])], 1u);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < a.ranges; i += blockDim.x)
    if (cnt[i]) atomicAdd(&a.start[i], cnt[i]);
}

// one CTA: range starts (exclusive), the scatter passes' allocation counters, and the first pass's
// buckets' tile offsets for the second
__global__ void __launch_bounds__(1024) part_scan_kernel(BulkArgs a) {
  __shared__ uint32_t sh[33];
  griddep_enter();
  const uint32_t per = (a.ranges + 1023u) / 1024u;
  const uint32_t b = threadIdx.x * per;
  uint32_t sum = 0;
  for (uint32_t i = b; i < b + per && i < a.ranges; i++) sum += a.start[i];
  uint32_t tot;
  uint32_t at = block_excl_scan(sum, sh, &tot);
  for (uint32_t i = b; i < b + per && i < a.ranges; i++) {
    const uint32_t c = a.start[i];
    a.start[i] = at;
    a.alloc[i] = at;
    at += c;
  }
  if (threadIdx.x == 0) a.start[a.ranges] = tot;
  __syncthreads();
  if (a.buckets == 0) return;
  uint32_t carry = 0;
  for (uint32_t t0 = 0; t0 < a.buckets; t0 += 1024u) {
    const uint32_t t = t0 + threadIdx.x;
    uint32_t tiles = 0;
    if (t < a.buckets) {
      const uint32_t lo = a.start[t * BULK_FAN];
      const uint32_t hi = a.start[(t + 1u) * BULK_FAN < a.ranges ? (t + 1u) * BULK_FAN : a.ranges];
      tiles = (hi - lo + PART_TILE - 1u) / PART_TILE;
      a.alloc1[t] = lo;
    }
    uint32_t tt;
    const uint32_t e = block_excl_scan(tiles, sh, &tt);
    if (t < a.buckets) a.tile_beg[t] = carry + e;
    carry += tt;
  }
  if (threadIdx.x == 0) a.tile_beg[a.buckets] = carry;
}

// One scatter pass over tiles of PART_TILE entries.  The tile's entries are ranked per bucket with
// shared atomics (order within a bucket does not matter), laid out bucket after bucket in shared
// memory, and written from there, so each bucket's entries leave as one run.
//   PASS 0: nodes straight into their ranges (few ranges)
//   PASS 1: nodes into buckets of BULK_FAN ranges
//   PASS 2: a bucket's entries into its ranges
template <int PASS>
__global__ void __launch_bounds__(PART_THREADS, PART_CTAS) part_scatter_kernel(BulkArgs a) {
  extern __shared__ __align__(16) uint8_t part_smem[];
  Key128* keys = reinterpret_cast<Key128*>(part_smem);
  uint32_t* ids = reinterpret_cast<uint32_t*>(keys + PART_TILE);
  uint32_t* cnt = ids + PART_TILE;        // per bucket: entries of the tile
  uint32_t* off = cnt + PART_DIGITS;      // exclusive offsets in the tile
  uint32_t* gpos = off + PART_DIGITS;     // where the bucket's run goes
  uint32_t* sh = gpos + PART_DIGITS;      // 33 words
  griddep_enter();
  constexpr uint32_t PER = PART_TILE / PART_THREADS;
  const Key128* in_k = PASS == 2 ? a.key1 : nullptr;
  const uint32_t* in_i = PASS == 2 ? a.id1 : nullptr;
  Key128* out_k = PASS == 1 ? a.key1 : a.key2;
  uint32_t* out_i = PASS == 1 ? a.id1 : a.id2;
  const uint32_t tiles = PASS == 2 ? a.tile_beg[a.buckets] : (uint32_t)((a.count + PART_TILE - 1u) / PART_TILE);
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    uint64_t beg;
    uint32_t len, base = 0, digits;   // digit d of this tile: range or bucket base + d
    uint32_t* alloc = PASS == 1 ? a.alloc1 : a.alloc;
    if (PASS == 2) {
      uint32_t lo = 0, hi = a.buckets;   // bucket with tile_beg[b] <= tile < tile_beg[b + 1]
      while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a.tile_beg[mid] <= tile) lo = mid; else hi = mid;
      }
      base = lo * BULK_FAN;
      const uint32_t last = base + BULK_FAN < a.ranges ? base + BULK_FAN : a.ranges;
      digits = last - base;
      beg = (uint64_t)a.start[base] + (uint64_t)(tile - a.tile_beg[lo]) * PART_TILE;
      const uint64_t left = a.start[last] - beg;
      len = left < PART_TILE ? (uint32_t)left : PART_TILE;
    } else {
      beg = (uint64_t)tile * PART_TILE;
      len = a.count - beg < PART_TILE ? (uint32_t)(a.count - beg) : PART_TILE;
      digits = PASS == 1 ? a.buckets : a.ranges;
    }
    for (uint32_t i = threadIdx.x; i < digits; i += blockDim.x) cnt[i] = 0;
    __syncthreads();
    Key128 k[PER];
    uint32_t place[PER];   // bucket (high half) and rank in it
    bool lost[PER];
#pragma unroll
    for (uint32_t j = 0; j < PER; j++) {
      const uint32_t i = threadIdx.x + j * PART_THREADS;
      place[j] = NO_ENTRY;
      lost[j] = false;
      if (i >= len) continue;
      k[j] = PASS == 2 ? in_k[beg + i] : node_key(a, beg + i);
      if (PASS != 2) lost[j] = lost_before(a, beg + i);
    }
#pragma unroll
    for (uint32_t j = 0; j < PER; j++) {
      const uint32_t i = threadIdx.x + j * PART_THREADS;
      if (i >= len) continue;
      if (PASS != 2 && left_out(a, k[j], lost[j])) {
        // the EMPTY pattern: inserted with the overflows, into its own slot
        if (key_is_empty_pattern(k[j])) bulk_overflow(a, a.first_node + (uint32_t)(beg + i));
        continue;
      }
      const uint32_t r = range_of(a, k[j]);
      const uint32_t d = PASS == 1 ? r / BULK_FAN : r - base;
      place[j] = d << 16 | atomicAdd(&cnt[d], 1u);
    }
    __syncthreads();
    const uint32_t c = threadIdx.x < digits ? cnt[threadIdx.x] : 0u;   // digits <= PART_DIGITS <= threads
    const uint32_t g = c ? atomicAdd(&alloc[base + threadIdx.x], c) : 0u;   // on its way during the scan
    uint32_t total;
    const uint32_t e = block_excl_scan(c, sh, &total);
    if (threadIdx.x < digits) {
      off[threadIdx.x] = e;
      gpos[threadIdx.x] = g;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < PER; j++)
      if (place[j] != NO_ENTRY) {
        const uint32_t i = threadIdx.x + j * PART_THREADS;
        const uint32_t p = off[place[j] >> 16] + (place[j] & 0xffffu);
        keys[p] = k[j];
        ids[p] = PASS == 2 ? in_i[beg + i] : a.first_node + (uint32_t)(beg + i);
      }
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < total; p += PART_THREADS) {
      const Key128 kk = keys[p];
      const uint32_t r = range_of(a, kk);
      const uint32_t d = PASS == 1 ? r / BULK_FAN : r - base;
      const uint32_t at = gpos[d] + (p - off[d]);
      out_k[at] = kk;
      out_i[at] = ids[p];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ table ranges
// which of two nodes with equal digests was inserted first in the sequential order: leaves by
// index, then parents by height and index
__device__ __forceinline__ unsigned long long node_value(const BulkArgs& a, uint32_t node) {
  const bool leaf = node >= a.n - 1u;
  return map_pack(((unsigned long long)(leaf ? 0u : 1u + a.D - node_level(node)) << 32) | node, a.cur);
}
// the node that lost an entry to another one
__device__ __forceinline__ void bulk_lost(const BulkArgs& a, uint32_t loser, uint32_t winner, const Key128& k) {
  if (loser >= a.n - 1u) {
    // a zero digest's chunks are all FIXED
    if (k.lo != 0ull || k.hi != 0ull) a.leaflab[loser - (a.n - 1u)] = SHIFT_DUPL;
  } else if (winner < a.n - 1u) {
    mark_lost(a, loser);
  }
}

__global__ void __launch_bounds__(BUILD_THREADS, BUILD_CTAS) build_kernel(BulkArgs a) {
  extern __shared__ __align__(16) uint32_t tab[];   // per slot: index of its entry
  __shared__ uint32_t claimed;
  griddep_enter();
  for (uint32_t r = blockIdx.x; r < a.ranges; r += gridDim.x) {
    const uint64_t slot0 = (uint64_t)r * BULK_RANGE;
    const uint32_t slots = a.map.cap - slot0 < BULK_RANGE ? (uint32_t)(a.map.cap - slot0) : BULK_RANGE;
    const uint32_t beg = a.start[r], end = a.start[r + 1u];
    for (uint32_t i = threadIdx.x; i < BULK_RANGE / 4u; i += blockDim.x)
      reinterpret_cast<uint4*>(tab)[i] = make_uint4(NO_ENTRY, NO_ENTRY, NO_ENTRY, NO_ENTRY);
    if (threadIdx.x == 0) claimed = 0;
    __syncthreads();
    uint32_t mine = 0;
    for (uint32_t i0 = beg + threadIdx.x; i0 < end; i0 += BUILD_IN * BUILD_THREADS) {
     Key128 kk[BUILD_IN];
     uint32_t nodes[BUILD_IN];
#pragma unroll
     for (uint32_t j = 0; j < BUILD_IN; j++)
       if (i0 + j * BUILD_THREADS < end) {
         kk[j] = a.key2[i0 + j * BUILD_THREADS];
         nodes[j] = a.id2[i0 + j * BUILD_THREADS];
       }
#pragma unroll
     for (uint32_t j = 0; j < BUILD_IN; j++) {
      const uint32_t i = i0 + j * BUILD_THREADS;
      if (i >= end) break;
      const Key128 k = kk[j];
      const uint32_t node = nodes[j];
      uint32_t s = (uint32_t)(map_home(k, a.map.cap) - slot0);
      for (;;) {
        if (s == slots) {   // past the range: inserted once every range is written
          bulk_overflow(a, node);
          break;
        }
        uint32_t cur = *reinterpret_cast<volatile uint32_t*>(&tab[s]);
        if (cur == NO_ENTRY) {
          cur = atomicCAS(&tab[s], NO_ENTRY, i);
          if (cur == NO_ENTRY) {
            mine++;
            break;
          }
        }
        const Key128 ck = a.key2[cur];
        if (ck.lo != k.lo || ck.hi != k.hi) {
          s++;
          continue;
        }
        const uint32_t other = a.id2[cur];
        if (node_value(a, other) < node_value(a, node)) {
          bulk_lost(a, node, other, k);
          break;
        }
        if (atomicCAS(&tab[s], cur, i) == cur) {
          bulk_lost(a, other, node, k);
          break;
        }
      }
     }
    }
    atomicAdd(&claimed, mine);
    __syncthreads();
    if (threadIdx.x == 0 && claimed) atomicAdd(a.map.size, (unsigned long long)claimed);
    // 16-byte pieces: a slot's key, then its value and padding; the entries' loads of BUILD_OUT
    // pieces per thread are in flight together
    uint4* out = reinterpret_cast<uint4*>(map_key(a.map, slot0));
    for (uint32_t p0 = threadIdx.x; p0 < 2u * slots; p0 += BUILD_OUT * BUILD_THREADS) {
      uint4 v[BUILD_OUT];
#pragma unroll
      for (uint32_t j = 0; j < BUILD_OUT; j++) {
        const uint32_t p = p0 + j * BUILD_THREADS;
        v[j] = make_uint4(NO_ENTRY, NO_ENTRY, NO_ENTRY, NO_ENTRY);
        if (p >= 2u * slots) continue;
        const uint32_t i = tab[p >> 1];
        if (i == NO_ENTRY) continue;
        if ((p & 1u) == 0u) v[j] = reinterpret_cast<const uint4*>(a.key2)[i];
        else v[j].x = a.id2[i];
      }
#pragma unroll
      for (uint32_t j = 0; j < BUILD_OUT; j++) {
        const uint32_t p = p0 + j * BUILD_THREADS;
        if (p >= 2u * slots) continue;
        if ((p & 1u) && v[j].x != NO_ENTRY) {   // N < 2^32 - 1: no node id is all ones
          const unsigned long long val = node_value(a, v[j].x);
          v[j].x = (uint32_t)val;
          v[j].y = (uint32_t)(val >> 32);
        }
        out[p] = v[j];
      }
    }
    __syncthreads();
  }
}

// entries whose probing left their range, and the EMPTY pattern
__global__ void __launch_bounds__(256) overflow_kernel(BulkArgs a) {
  griddep_enter();
  const uint32_t count = *a.over_count < a.n ? *a.over_count : a.n;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const uint32_t node = a.overflow[i];
    const Digest d = a.tree[node];
    const unsigned long long v = node_value(a, node);
    const MapRef ref = map_insert_packed(a.map, d, v, a.st);
    unsigned long long prev = ref.prev;
    if (ref.found && !ref.inserted) {
      // the extra slot's insert has merged its value already
      if (!key_is_empty_pattern(digest_key(d))) prev = atomicMin(map_val(a.map, ref.slot), v);
    }
    if (prev == MAP_EMPTY) continue;
    const uint32_t other = (uint32_t)prev;
    if (prev < v) bulk_lost(a, node, other, digest_key(d));
    else if (v < prev) bulk_lost(a, other, node, digest_key(d));
  }
}

// ------------------------------------------------------------------ host side
bool bulk_plan(uint32_t n, uint64_t cap, int list, uint64_t diff_bytes, BulkPlan& p) {
  p.count = list ? n : 2ull * n - 1ull;
  const uint64_t ranges = (cap + BULK_RANGE - 1u) / BULK_RANGE;
  if (n < (list ? BULK_MIN_LIST : BULK_MIN_TREE) || ranges > BULK_MAX_RANGES) return false;
  p.ranges = (uint32_t)ranges;
  p.buckets = ranges <= BULK_ONE_PASS ? 0u : (uint32_t)((ranges + BULK_FAN - 1u) / BULK_FAN);
  // entries of the last scatter pass, and of the first one of two
  uint64_t at = 0;
  auto take = [&](uint64_t bytes) {
    const uint64_t o = at;
    at += (bytes + 15u) / 16u * 16u;
    return o;
  };
  p.key2 = take(16 * p.count);
  p.id2 = take(4 * p.count);
  p.key1 = p.id1 = at;
  if (p.buckets) {
    p.key1 = take(16 * p.count);
    p.id1 = take(4 * p.count);
  }
  if (at > diff_bytes) return false;
  // counters and marks in 4 bytes per chunk (as much as one region list), the zeroed ones first
  at = 0;
  p.start = take(4ull * (p.ranges + 1u));
  p.over_count = take(16);
  p.lost = take((2ull * n + 31u) / 32u * 4u);
  p.zeroed_bytes = at;
  p.alloc = take(4ull * p.ranges);
  p.alloc1 = take(4ull * (p.buckets + 1u));
  p.tile_beg = take(4ull * (p.buckets + 1u));
  return at <= 4ull * n;
}

cudaError_t launch_bulk(const BulkArgs& args, int sm_count, cudaStream_t stream, uint32_t* launches) {
  BulkArgs a = args;
  cudaError_t e = cudaSuccess;
  uint32_t c = 0;
  // Large builds' kernels are launched the ordinary way: with the next kernel's CTAs let in while the
  // one before drains, its resident grid fills the SMs unevenly and late, and as each CTA has its
  // fixed share, all wait for the last (4 GiB: scatter passes 750 and 750 against 720 and 620 us,
  // build 2.75 against 2.16 ms).  Small ones are bound by the launches themselves.  Whole build, early
  // and ordinary launches, us: 2^16 chunks 56 and 68, 2^18 76 and 82, 2^19 115 and 125, 2^20 183 and
  // 192, 2^21 344 and 342, 2^22 587 and 580, 2^23 1159 and 1156, 2^24 2180 and 2128, 2^25 4500 and 4390.
  const bool early = a.n < (1u << 21);
#define B2D_LD(...)                                              \
  if ((e = launch_early(early, __VA_ARGS__)) != cudaSuccess) return e; \
  c++;
  if (!a.list) {
    uint32_t in = a.D;   // >= 15
    const uint64_t want = ((1ull << (in - 2u)) + 255u) / 256u, cap = (uint64_t)sm_count * 6u;   // resident CTAs
    B2D_LD(tree_hash2_kernel, (uint32_t)(want < cap ? want : cap), 256, 0, stream, a, in)
    a.stamp = nullptr;
    for (in -= 2u; in > 0;) {
      const uint32_t k = in < HASH_LEVELS ? in : HASH_LEVELS;
      const uint64_t want = ((1ull << (in - k)) + 7u) / 8u, cap = (uint64_t)sm_count * 8u;
      B2D_LD(tree_hash_kernel, (uint32_t)(want < cap ? want : cap), 256, 0, stream, a, in, k)
      in -= k;
    }
  }
  const size_t csm = sizeof(uint32_t) * a.ranges;
  const size_t psm = (sizeof(Key128) + sizeof(uint32_t)) * PART_TILE + sizeof(uint32_t) * (3u * PART_DIGITS + 33u);
  const size_t bsm = sizeof(uint32_t) * BULK_RANGE;
  struct {
    const void* k;
    size_t sm;
  } attr[] = {{(const void*)part_count_kernel, sizeof(uint32_t) * BULK_MAX_RANGES},
              {(const void*)part_scatter_kernel<0>, psm},
              {(const void*)part_scatter_kernel<1>, psm},
              {(const void*)part_scatter_kernel<2>, psm},
              {(const void*)build_kernel, bsm}};
  for (auto& q : attr)
    if ((e = cudaFuncSetAttribute(q.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)q.sm)) != cudaSuccess) return e;
  const uint32_t sms = (uint32_t)sm_count;
  const uint64_t tiles = (a.count + PART_TILE - 1u) / PART_TILE;
  auto grid = [&](uint64_t want, uint64_t cap) { return (uint32_t)(want < cap ? (want ? want : 1u) : cap); };
  B2D_LD(part_count_kernel, grid(tiles, sms), COUNT_THREADS, csm, stream, a)
  a.stamp = nullptr;
  B2D_LD(part_scan_kernel, 1, 1024, 0, stream, a)
  if (a.buckets == 0) {
    B2D_LD(part_scatter_kernel<0>, grid(tiles, PART_CTAS * sms), PART_THREADS, psm, stream, a)
  } else {
    B2D_LD(part_scatter_kernel<1>, grid(tiles, PART_CTAS * sms), PART_THREADS, psm, stream, a)
    B2D_LD(part_scatter_kernel<2>, grid(tiles, PART_CTAS * sms), PART_THREADS, psm, stream, a)
  }
  B2D_LD(build_kernel, grid(a.ranges, BUILD_CTAS * sms), BUILD_THREADS, bsm, stream, a)
  B2D_LD(overflow_kernel, 8, 256, 0, stream, a)
#undef B2D_LD
  *launches = c;
  return cudaSuccess;
}

}  // namespace b2d
