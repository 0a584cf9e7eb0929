// Diff assembly on the device: the reference's collect_diff (src/tree_approach.cpp:511-710).
//
// Output order is the reference's sequential order (what its atomics produce with one
// thread): region roots by (level descending, node ascending); the repeat table by
// checkpoint id; shifted-duplicate entries stably bucketed by source checkpoint.
//   1. diff_count  per CTA: region roots of each kind and the chunks under the first ones
//   2. diff_write  the root lists in that order, with each first region's chunk offset
//   3. diff_shift  source NodeID of every shifted root, per-range counts by source checkpoint;
//                  the last CTA to finish lays the diff out (bucket starts, repeat table, header)
//   4. diff_emit   stable bucket scatter of the shifted entries, the first-occurrence list and
//                  the 16-byte vectorised data gather, side by side
// Four launches: a checkpoint of a few MiB is bound by the chain of dependent launches, not by
// their work (twelve launches took 36 us of a 1 MiB checkpoint's 130 us).
// Diff layout (include/utils.hpp:29-37, src/tree_approach.cpp:777-780):
//   [header 32 B][u32 first node x F][(u32 ckpt, u32 count) x P][(u32 node, u32 prev) x S][data]
// It is placed `delta` bytes into the device buffer so the data section is 16-byte aligned.
#include "copy.cuh"
#include "dedup_kernels.cuh"
#include "map.cuh"
#include "scan.cuh"

namespace b2d {

constexpr uint32_t COMPACT_THREADS = 512;

// Every kernel below is a body over a virtual grid (bid of nb CTAs) with two launchers: one
// handle's launch (the CUDA grid) and a segmented launch over many handles' diff assembly in
// one grid, where CTA b belongs to the handle h with beg[h] <= b < beg[h+1] (batched form).
__device__ __forceinline__ uint32_t seg_locate(const SegGrid& s, uint32_t& bid, uint32_t& nb) {
  uint32_t lo = 0, hi = s.n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (s.beg[mid] <= blockIdx.x) lo = mid; else hi = mid;
  }
  bid = blockIdx.x - s.beg[lo];
  nb = s.beg[lo + 1] - s.beg[lo];
  return lo;
}
constexpr uint32_t SHIFT_GRID = 296;    // at most 2 x 148 ranges for the shifted-entry passes
constexpr uint32_t SHIFT_THREADS = 256;
constexpr uint32_t EMIT_THREADS = 256;

// Region roots are flagged in `push`: 2 bits per node (PUSH_FIRST = 1, PUSH_SHIFT = 2), 16 nodes
// per 32-bit word, zero-padded to a multiple of 64 nodes, all-zero between checkpoints.  Node x
// sits at position y = x + 1, so level L occupies [2^L, 2^(L+1)) and every 16-byte group of 64
// flags from the second on lies within one level: walking the groups level by level from the
// deepest, each level ascending, then the six levels of the first group, meets the roots in the
// canonical order.  List diffs keep node order (their roots are single leaves), so their walk is
// plainly ascending from the first leaf's group.
constexpr uint32_t PUSH_GROUP = 64;   // nodes per 16-byte load
__device__ __forceinline__ uint4 ld_push16(const uint8_t* push, uint64_t g) {
  return reinterpret_cast<const uint4*>(push)[g];
}
struct GroupWalk {
  uint32_t total;   // groups walked
  uint32_t first;   // node order: the first group; canonical order: 2^(level of the deepest group)
  uint32_t deep;    // canonical order: groups of the deepest level
  bool node_order;
};
__device__ __forceinline__ GroupWalk group_walk(const DiffArgs& a) {
  GroupWalk w;
  const uint32_t groups = (uint32_t)(((uint64_t)a.N >> 6) + 1u);   // positions 1 .. N
  w.node_order = a.node_order != 0;
  if (w.node_order) {
    w.first = a.n >> 6;   // position of chunk 0's leaf: n
    w.total = groups - w.first;
    w.deep = 0;
  } else {
    w.total = groups;
    w.first = groups > 1u ? 1u << (31u - __clz(groups - 1u)) : 0u;
    w.deep = groups > 1u ? groups - w.first : 0u;
  }
  return w;
}
// group at step p of the walk
__device__ __forceinline__ uint32_t walk_group(const GroupWalk& w, uint32_t p) {
  if (w.node_order || p < w.deep) return w.first + p;
  const uint32_t t = w.first - (p - w.deep);   // 2^L .. 1 over the levels above the deepest
  if (t < 2u) return 0u;
  return 3u * (1u << (31u - __clz(t - 1u))) - t;
}
// one bit (the low bit of each 2-bit field) per node flagged first / shifted
__device__ __forceinline__ uint32_t push_first_bits(uint32_t w) { return w & ~(w >> 1) & 0x55555555u; }
__device__ __forceinline__ uint32_t push_shift_bits(uint32_t w) { return (w >> 1) & ~w & 0x55555555u; }
__device__ __forceinline__ uint32_t first_count(const uint4& v) {
  return __popc(push_first_bits(v.x)) + __popc(push_first_bits(v.y)) + __popc(push_first_bits(v.z)) +
         __popc(push_first_bits(v.w));
}
__device__ __forceinline__ uint32_t shift_count(const uint4& v) {
  return __popc(push_shift_bits(v.x)) + __popc(push_shift_bits(v.y)) + __popc(push_shift_bits(v.z)) +
         __popc(push_shift_bits(v.w));
}
// chunks under the first-occurrence roots of a group
__device__ __forceinline__ uint32_t group_chunks(const DiffArgs& a, uint32_t g, const uint4& v, uint32_t cf) {
  if (cf == 0) return 0u;
  if (g > 0) {   // one level: full subtrees all hold 2^k chunks
    const uint32_t k = a.D - (31u - __clz(g)) - 6u;
    if ((((uint64_t)g + 1u) << (6u + k)) <= (uint64_t)a.N + 1u) return cf << k;
  }
  uint32_t c = 0;
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 4; k++)
    for (uint32_t m = push_first_bits(w[k]); m; m &= m - 1u)
      c += node_span(PUSH_GROUP * g + 16u * k + ((__ffs(m) - 1u) >> 1) - 1u, a.N, a.D).count;
  return c;
}

__device__ __forceinline__ void diff_count_body(const DiffArgs& a, uint32_t bid, uint32_t nb, uint32_t bcap) {
  __shared__ uint32_t sh[COMPACT_THREADS / 32 + 1];
  const GroupWalk w = group_walk(a);
  uint64_t beg, end;
  cta_range(w.total, bid, nb, beg, end);
  uint32_t cf = 0, cs = 0, ct = 0;
  // two independent loads per thread per iteration
  for (uint64_t p = beg + threadIdx.x; p < end; p += 2ull * blockDim.x) {
    const uint32_t g0 = walk_group(w, (uint32_t)p);
    const bool two = p + blockDim.x < end;
    const uint32_t g1 = two ? walk_group(w, (uint32_t)p + blockDim.x) : g0;
    const uint4 v0 = ld_push16(a.push, g0);
    const uint4 v1 = two ? ld_push16(a.push, g1) : make_uint4(0, 0, 0, 0);
    if (v0.x | v0.y | v0.z | v0.w) {
      const uint32_t f = first_count(v0);
      cf += f;
      cs += shift_count(v0);
      ct += group_chunks(a, g0, v0, f);
    }
    if (v1.x | v1.y | v1.z | v1.w) {
      const uint32_t f = first_count(v1);
      cf += f;
      cs += shift_count(v1);
      ct += group_chunks(a, g1, v1, f);
    }
  }
  const uint32_t tf = block_reduce_sum(cf, sh);
  const uint32_t ts = block_reduce_sum(cs, sh);
  const uint32_t tt = block_reduce_sum(ct, sh);
  if (threadIdx.x == 0) {
    a.partial2[3 * bid] = tf;
    a.partial2[3 * bid + 1] = ts;
    a.partial2[3 * bid + 2] = tt;
  }
  // the per-checkpoint bucket counts start at zero
  if (bid == 0)
    for (uint32_t t = threadIdx.x; t < bcap; t += blockDim.x) a.hist[t] = 0u;
}
__global__ void __launch_bounds__(COMPACT_THREADS) diff_count_kernel(DiffArgs a0, uint32_t bcap) {
  griddep_enter();
  if (blockIdx.x == 0 && threadIdx.x == 0) a0.stamps->diff = device_time_ns();
  diff_count_body(with_round(a0), blockIdx.x, gridDim.x, bcap);
}
__global__ void __launch_bounds__(COMPACT_THREADS) diff_count_seg(SegGrid s) {
  uint32_t bid, nb;
  const uint32_t h = seg_locate(s, bid, nb);
  diff_count_body(with_round(s.args[h]), bid, nb, s.bcap[h]);
}

// Lists of first / shifted roots and the first regions' chunk offsets; clears the flags it
// consumed.  Each CTA adds up the counts of the CTAs before it.  Each thread owns one 64-node
// group of a tile, so one block scan covers COMPACT_THREADS * 64 = 32768 nodes, which keeps both
// 16-bit halves of the packed counts exact.
__device__ __forceinline__ void diff_write_body(const DiffArgs& a, uint32_t bid, uint32_t nb) {
  __shared__ uint32_t sh[COMPACT_THREADS / 32 + 1];
  const GroupWalk w = group_walk(a);
  uint64_t beg, end;
  cta_range(w.total, bid, nb, beg, end);
  uint32_t bf = 0, bs = 0, bt = 0;
  for (uint32_t i = threadIdx.x; i < bid; i += blockDim.x) {
    bf += a.partial2[3 * i];
    bs += a.partial2[3 * i + 1];
    bt += a.partial2[3 * i + 2];
  }
  bf = block_reduce_sum(bf, sh);
  bs = block_reduce_sum(bs, sh);
  bt = block_reduce_sum(bt, sh);
  if (bid == nb - 1u && threadIdx.x == 0) {
    a.meta->F = bf + a.partial2[3 * bid];
    a.meta->S = bs + a.partial2[3 * bid + 1];
    a.meta->T = bt + a.partial2[3 * bid + 2];
  }
  for (uint64_t t0 = beg; t0 < end; t0 += COMPACT_THREADS) {
    const uint64_t p = t0 + threadIdx.x;
    const uint32_t g = p < end ? walk_group(w, (uint32_t)p) : 0u;
    const uint4 v = p < end ? ld_push16(a.push, g) : make_uint4(0, 0, 0, 0);
    const bool nz = (v.x | v.y | v.z | v.w) != 0u;
    uint32_t cf = 0, cs = 0, ct = 0;
    if (nz) {
      cf = first_count(v);
      cs = shift_count(v);
      ct = group_chunks(a, g, v, cf);
    }
    if (!__syncthreads_or(nz)) continue;
    uint32_t tot, tott;
    const uint32_t ex = block_excl_scan((cf << 16) | cs, sh, &tot);
    const uint32_t et = block_excl_scan(ct, sh, &tott);
    // Groups with many roots of one level over full subtrees (runs of list chunks above all) are
    // written by the whole warp, two nodes per lane, so stores cover whole sectors.
    const uint32_t height = g > 0 ? a.D - (31u - __clz(g)) - 6u : 0u;
    const bool dense = cf + cs >= 8u && g > 0 &&
                       (w.node_order || (((uint64_t)g + 1u) << (6u + height)) <= (uint64_t)a.N + 1u);
    for (uint32_t todo = __ballot_sync(0xffffffffu, dense); todo; todo &= todo - 1u) {
      const uint32_t l = __ffs(todo) - 1u, lane = threadIdx.x & 31u;
      const uint32_t ws[4] = {__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l),
                              __shfl_sync(0xffffffffu, v.z, l), __shfl_sync(0xffffffffu, v.w, l)};
      const uint32_t k = w.node_order ? 0u : __shfl_sync(0xffffffffu, height, l);
      uint32_t of = bf + __shfl_sync(0xffffffffu, ex >> 16, l), os = bs + __shfl_sync(0xffffffffu, ex & 0xffffu, l);
      uint32_t x = PUSH_GROUP * __shfl_sync(0xffffffffu, g, l) + 2u * lane - 1u;
      const uint32_t ot = bt + __shfl_sync(0xffffffffu, et, l);
      const uint32_t mine = lane >> 3, below = (1u << (4u * (lane & 7u))) - 1u;
      uint32_t pf = 0, word = ws[0];
#pragma unroll
      for (uint32_t q = 0; q < 4; q++) {
        if (q == mine) word = ws[q];
        const uint32_t m = q < mine ? ~0u : q == mine ? below : 0u;
        pf += __popc(push_first_bits(ws[q]) & m);
        os += __popc(push_shift_bits(ws[q]) & m);
      }
      of += pf;
      uint32_t o = ot + (pf << k);
#pragma unroll
      for (uint32_t q = 0; q < 2; q++, x++) {
        const uint32_t flag = word >> (4u * (lane & 7u) + 2u * q) & 3u;
        if (flag == PUSH_FIRST) {
          a.first_list[of] = x;
          a.region_off[of] = o;
          of++;
          o += 1u << k;
        } else if (flag == PUSH_SHIFT) {
          a.shift_list[os++] = x;
        }
      }
    }
    if (dense) {
      reinterpret_cast<uint4*>(a.push)[g] = make_uint4(0, 0, 0, 0);
    } else if (nz) {
      uint32_t of = bf + (ex >> 16), os = bs + (ex & 0xffffu), ot = bt + et;
      auto emit = [&](uint32_t word, uint32_t base) {   // the roots of one 16-flag word, ascending
        for (uint32_t m = push_first_bits(word); m; m &= m - 1u) {
          const uint32_t x = base + ((__ffs(m) - 1u) >> 1);
          a.first_list[of] = x;
          a.region_off[of] = ot;
          ot += node_span(x, a.N, a.D).count;
          of++;
        }
        for (uint32_t m = push_shift_bits(word); m; m &= m - 1u) a.shift_list[os++] = base + ((__ffs(m) - 1u) >> 1);
      };
      const uint32_t ws[4] = {v.x, v.y, v.z, v.w};
      if (g > 0 || w.node_order) {
#pragma unroll
        for (int k = 0; k < 4; k++) emit(ws[k], PUSH_GROUP * g + 16u * k - 1u);
      } else {   // positions 1 .. 63: levels 5 .. 0, each ascending
        emit(ws[2], 31u);
        emit(ws[3], 47u);
        emit(ws[1], 15u);
        emit(ws[0] & 0xffff0000u, ~0u);
        emit(ws[0] & 0x0000ff00u, ~0u);
        emit(ws[0] & 0x000000f0u, ~0u);
        emit(ws[0] & 0x0000000cu, ~0u);
      }
      reinterpret_cast<uint4*>(a.push)[g] = make_uint4(0, 0, 0, 0);
    }
    bf += tot >> 16;
    bs += tot & 0xffffu;
    bt += tott;
  }
}
__global__ void __launch_bounds__(COMPACT_THREADS) diff_write_kernel(DiffArgs a0) {
  griddep_enter();
  diff_write_body(with_round(a0), blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(COMPACT_THREADS) diff_write_seg(SegGrid s) {
  uint32_t bid, nb;
  const uint32_t h = seg_locate(s, bid, nb);
  diff_write_body(with_round(s.args[h]), bid, nb);
}

// ---------------------------------------------------------------- shifted duplicates, layout
// Source checkpoints are counted in buckets relative to the last baseline, which emptied the
// map: no entry is older, and a handle that has taken thousands of checkpoints sorts its entries
// into as many buckets as its chain is long.
__device__ __forceinline__ uint32_t bucket_count(const DiffArgs& a, uint32_t bcap) {
  return a.rs->buckets <= bcap ? a.rs->buckets : bcap;
}

// one CTA: bucket starts, repeat table, per-range scatter bases, header, byte layout.  The counts
// come from other CTAs of the same launch, so they are read past L1.
__device__ __forceinline__ void layout_body(const DiffArgs& a, uint32_t B, uint32_t g) {
  __shared__ uint32_t sh[33];
  __shared__ uint32_t carry_start, carry_rows;
  if (threadIdx.x == 0) { carry_start = 0; carry_rows = 0; }
  __syncthreads();
  const DevMeta m0 = *a.meta;
  // count P first so the table position is known
  for (uint32_t t0 = 0; t0 < B; t0 += blockDim.x) {
    const uint32_t t = t0 + threadIdx.x;
    const uint32_t h = t < B ? __ldcg(&a.hist[t]) : 0u;
    uint32_t tot_h;
    const uint32_t eh = block_excl_scan(h, sh, &tot_h);
    const uint32_t tot_r = (uint32_t)__syncthreads_count(h != 0u);
    if (t < B) a.bucket_start[t] = carry_start + eh;
    __syncthreads();
    if (threadIdx.x == 0) { carry_start += tot_h; carry_rows += tot_r; }
    __syncthreads();
  }
  const uint32_t P = carry_rows;
  const uint64_t F = m0.F, S = m0.S, T = m0.T;
  const uint64_t meta_bytes = 4 * F + 8 * (uint64_t)P + 8 * S;
  const uint32_t delta = (uint32_t)((16u - ((32u + meta_bytes) & 15u)) & 15u);
  const uint64_t first_off = delta + 32ull;
  const uint64_t count_off = first_off + 4 * F;
  const uint64_t shift_off = count_off + 8ull * P;
  const uint64_t data_off = shift_off + 8 * S;
  // repeat table rows (ckpt id, count) in ascending id order (:656-665)
  __shared__ uint32_t row_carry;
  if (threadIdx.x == 0) row_carry = 0;
  __syncthreads();
  for (uint32_t t0 = 0; t0 < B; t0 += blockDim.x) {
    const uint32_t t = t0 + threadIdx.x;
    const uint32_t h = t < B ? __ldcg(&a.hist[t]) : 0u;
    uint32_t tot_r;
    const uint32_t er = block_excl_scan(h ? 1u : 0u, sh, &tot_r);
    if (h) {
      uint32_t* row = reinterpret_cast<uint32_t*>(a.diff + count_off + 8ull * (row_carry + er));
      row[0] = a.baseline_id + t;
      row[1] = h;
    }
    __syncthreads();
    if (threadIdx.x == 0) row_carry += tot_r;
    __syncthreads();
  }
  // per-range scatter bases: bucket start + counts of earlier ranges.  `partial` is
  // bucket-major (partial[t * g + range]); one warp scans one bucket's g range counts.
  {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t t = warp; t < B; t += nw) {
      uint32_t carry = a.bucket_start[t];
      uint32_t* row = a.partial + (uint64_t)t * g;
#pragma unroll 4
      for (uint32_t j = 0; j < g; j += 32) {
        const uint32_t b = j + lane;
        const uint32_t v = b < g ? __ldcg(&row[b]) : 0u;
        const uint32_t inc = warp_incl_scan(v);
        if (b < g) row[b] = carry + inc - v;
        carry += __shfl_sync(0xffffffffu, inc, 31);
      }
    }
  }
  if (threadIdx.x == 0) {
    uint32_t* h32 = reinterpret_cast<uint32_t*>(a.diff + delta);
    h32[0] = a.baseline_id;                 // ref_id
    h32[1] = a.cur;                         // chkpt_id
    h32[2] = (uint32_t)a.len;               // datalen (u64, little endian)
    h32[3] = (uint32_t)(a.len >> 32);
    h32[4] = a.cs;                          // chunk_size
    h32[5] = (uint32_t)F;                   // num_first_ocur
    h32[6] = P;                             // num_prior_chkpts
    h32[7] = (uint32_t)S;                   // num_shift_dupl
    DevMeta* m = a.meta;
    m->P = P;
    m->delta = delta;
    m->first_off = first_off;
    m->count_off = count_off;
    m->shift_off = shift_off;
    m->data_off = data_off;
    m->diff_len = 32ull + meta_bytes + T * a.cs;
    m->map_size = *a.map.size;
  }
}
// Source NodeID of each shifted root (:572-580, :672-674) and per-range counts by checkpoint, one
// range per CTA of the first `ranges`; the one of them that finishes last lays the diff out.
// collect_diff keeps a first-occurrence region only when the map names it as the owner of its
// digest (:548-556); the labelling guarantees it, so that is checked here by the other CTAs.
__device__ __forceinline__ void diff_shift_body(const DiffArgs& a, uint32_t bid, uint32_t nb, uint32_t bcap,
                                                uint32_t ranges) {
  if (bid >= ranges) {
    const uint32_t F = a.meta->F;
    for (uint64_t i = (bid - ranges) * (uint64_t)blockDim.x + threadIdx.x; i < F;
         i += (uint64_t)(nb - ranges) * blockDim.x) {
      const uint32_t node = a.first_list[i];
      const uint64_t slot = map_find(a.map, a.tree[node]);
      if (slot > a.map.cap || map_node(a.map, slot) != node || map_tree(a.map, slot) != a.cur)
        set_error(a.st, DERR_INTERNAL, 20);
    }
    return;
  }
  nb = ranges;
  const uint32_t B = bucket_count(a, bcap);
  extern __shared__ uint32_t hs[];
  __shared__ uint32_t last;
  uint64_t beg, end;
  for (uint32_t t = threadIdx.x; t < B; t += blockDim.x) hs[t] = 0;
  __syncthreads();
  cta_range(a.meta->S, bid, nb, beg, end);
  for (uint64_t i = beg + threadIdx.x; i < end; i += blockDim.x) {
    const uint32_t node = a.shift_list[i];
    const uint64_t slot = map_find(a.map, a.tree[node]);
    uint32_t pn = 0, pt = 0;
    if (slot <= a.map.cap) {
      pn = map_node(a.map, slot);
      pt = map_tree(a.map, slot) - a.baseline_id;
    } else {
      set_error(a.st, DERR_INTERNAL, 30);
    }
    if (pt >= B) {
      set_error(a.st, DERR_INTERNAL, 31);
      pt = 0;
    }
    a.sprev[i] = pn;
    a.skey[i] = pt;
    atomicAdd(&hs[pt], 1u);
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < B; t += blockDim.x) {
    const uint32_t v = hs[t];
    a.partial[(uint64_t)t * nb + bid] = v;
    if (v) atomicAdd(&a.hist[t], v);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&a.meta->done, 1u) == nb - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  layout_body(a, B, nb);
}
__global__ void __launch_bounds__(SHIFT_THREADS) diff_shift_kernel(DiffArgs a0, uint32_t bcap, uint32_t ranges) {
  griddep_enter();
  diff_shift_body(with_round(a0), blockIdx.x, gridDim.x, bcap, ranges);
}
__global__ void __launch_bounds__(SHIFT_THREADS) diff_shift_seg(SegGrid s) {
  uint32_t bid, nb;
  const uint32_t h = seg_locate(s, bid, nb);
  diff_shift_body(with_round(s.args[h]), bid, nb, s.bcap[h], s.gs[h]);
}

// stable scatter of one range of the shifted entries: a warp walks it in order; run: B words of
// the warp's own
__device__ __forceinline__ void shift_write_range(const DiffArgs& a, uint32_t range, uint32_t ranges, uint32_t B,
                                                  uint32_t* run) {
  const uint32_t lane = threadIdx.x & 31u;
  uint64_t beg, end;
  cta_range(a.meta->S, range, ranges, beg, end);
  if (beg >= end) return;
  for (uint32_t t = lane; t < B; t += 32) run[t] = a.partial[(uint64_t)t * ranges + range];
  __syncwarp();
  const uint64_t shift_off = a.meta->shift_off;
  // UNR groups of 32 entries per pass: their loads are issued together (they do
  // not depend on the running bucket positions), then the groups are placed in order
  constexpr uint32_t UNR = 4;
  for (uint64_t t0 = beg; t0 < end; t0 += 32ull * UNR) {
    uint32_t key[UNR], node[UNR], prev[UNR];
#pragma unroll
    for (uint32_t u = 0; u < UNR; u++) {
      const uint64_t i = t0 + 32ull * u + lane;
      const bool act = i < end;
      key[u] = act ? a.skey[i] : 0xffffffffu;
      node[u] = act ? a.shift_list[i] : 0u;
      prev[u] = act ? a.sprev[i] : 0u;
    }
#pragma unroll
    for (uint32_t u = 0; u < UNR; u++) {
      const bool act = t0 + 32ull * u + lane < end;
      const uint32_t peers = __match_any_sync(0xffffffffu, key[u]);
      const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
      uint32_t pos = 0;
      if (act) pos = run[key[u]] + rank;
      __syncwarp();
      if (act && rank == 0) run[key[u]] += __popc(peers);
      __syncwarp();
      if (act) {
        uint32_t* e = reinterpret_cast<uint32_t*>(a.diff + shift_off + 8ull * pos);
        e[0] = node[u] - a.id_bias;
        e[1] = prev[u] - a.id_bias;
      }
    }
  }
}
// ---------------------------------------------------------------- data gather
// A 16-byte unit of the data section whose source reaches past the buffer's end (zeros, :643-645), where
// chunks and buffer are 16-byte aligned: a unit then lies within one region.  One byte after another: a
// kernel has the registers of what it calls, 124 with the routine below.
__device__ __noinline__ void gather_end_unit(const uint8_t* data, uint64_t len, uint64_t s, uint4* dst) {
  uint64_t lo = 0, hi = 0;
#pragma unroll 1
  for (uint32_t b = 0; b < 16u && s + b < len; b++) {
    const uint64_t v = (uint64_t)data[s + b] << (8u * (b & 7u));
    if (b < 8u) lo |= v;
    else hi |= v;
  }
  *dst = make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
// a 16-byte unit of the data section that a region ends in, or whose source reaches past the
// buffer's end: byte by byte, region r holding its first byte
struct GatherBytes {
  const uint8_t* data;
  uint64_t len, cs, total;   // buffer length, chunk size, bytes of the data section
  const uint32_t *region_off, *first_list;
  uint32_t F, n, N, D;
};
__device__ __noinline__ void gather_unit_bytes(GatherBytes a, uint8_t* dst, uint64_t unit, uint32_t r) {
  const uint64_t pos0 = 16ull * unit;
  auto start_of = [&](uint32_t i) { return i < a.F ? (uint64_t)a.region_off[i] * a.cs : ~0ull; };
  // source byte minus data-section byte, within region r
  auto shift_of = [&](uint32_t i) {
    return (node_span(a.first_list[i], a.N, a.D).first - (a.n - 1u)) * a.cs - start_of(i);
  };
  uint64_t shift = shift_of(r), next = start_of(r + 1u);
  uint8_t t[16];
  // the bytes' loads do not wait for one another (one at a time, a unit took 16 memory round trips)
#pragma unroll
  for (uint32_t b = 0; b < 16u; b++) {
    const uint64_t pos = pos0 + b;
    while (pos >= next) {
      r++;
      shift = shift_of(r);
      next = start_of(r + 1u);
    }
    const uint64_t s = pos + shift;
    t[b] = pos < a.total && s < a.len ? __ldg(a.data + s) : 0u;
  }
  if (pos0 + 16u <= a.total) {
    uint4 v;
    memcpy(&v, t, 16);
    *reinterpret_cast<uint4*>(dst + pos0) = v;
  } else {
#pragma unroll
    for (uint32_t b = 0; b < 16u; b++)
      if (pos0 + b < a.total) dst[pos0 + b] = t[b];
  }
}

// Data section.  The chunks of a region lie one after another in the buffer, so the section is a
// sequence of byte runs.  Each warp owns an equal share of the section's 16-byte units and copies
// it lane after lane over consecutive units, GATHER_UNROLL per lane in flight, whatever the region
// boundaries: many regions are a few chunks long.  The starts and sources of 32 regions at a time
// are held one per lane, and each unit finds its region among them by a five-step shuffle search,
// so no load waits on another.  Where one region covers a whole step of the warp the search is
// left out and the warp streams to the region's end: a 4 GiB baseline, one region, was bound by
// the search's instructions (2.40 ms, now 1.36 ms; a plain copy of the same bytes takes 1.35 ms).
// Chunk sizes or buffers that are not 16-byte aligned take the same path with shifted loads
// (load_unit): with one thread per chunk and byte copies, 1000 B chunks of a 150 MB buffer at an
// 8-byte offset took 331 us per increment of 5 % and the whole series 2.40 ms, now 0.94 ms.
#ifndef B2D_GATHER_UNROLL
#define B2D_GATHER_UNROLL 4
#endif
template <bool ALIGNED>
__device__ __forceinline__ void gather_body(const DiffArgs& a, uint32_t bid, uint32_t nb) {
  constexpr uint32_t U = B2D_GATHER_UNROLL;
  const DevMeta m = *a.meta;
  uint8_t* dst_base = a.diff + m.data_off;
  uint32_t* first_meta = reinterpret_cast<uint32_t*>(a.diff + m.first_off);
  const uint64_t gtid = bid * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t nthr = (uint64_t)nb * blockDim.x;
  for (uint64_t i = gtid; i < m.F; i += nthr) first_meta[i] = a.first_list[i] - a.id_bias;
  if (m.T == 0) return;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t total = m.T * a.cs;
  const uint32_t F = m.F;
  uint64_t u0, u1;
  cta_range((total + 15u) / 16u, (uint32_t)(gtid >> 5), (uint32_t)(nthr >> 5), u0, u1);
  if (u0 >= u1) return;
  uint4* dst = reinterpret_cast<uint4*>(dst_base);
  // largest r with region_off[r] <= the first unit's chunk (region_off[0] = 0)
  uint32_t r = warp_lower_bound(a.region_off, F, 16ull * u0 / a.cs + 1u) - 1u;
  uint64_t u = u0;
  while (u < u1) {
    // regions r .. r + 31, one per lane, as byte positions relative to unit u; a step covers at
    // most 1 GiB, so positions fit 32 bits and a start beyond the step is never met
    const uint64_t pos0 = 16ull * u;
    const uint32_t rl = r + lane;
    const bool has = rl < F;
    const uint64_t off = has ? (uint64_t)a.region_off[rl] * a.cs : total;
    uint64_t src0 = 0;   // buffer byte that data-section byte pos0 would come from
    if (has) {
      const NodeSpan sp = node_span(a.first_list[rl], a.N, a.D);
      const uint64_t chunk = sp.first - (a.n - 1u);
      if (chunk + sp.count > a.n) set_error(a.st, DERR_INTERNAL, 40);
      src0 = chunk * a.cs - off + pos0;   // wraps where the region starts later: only sums are used
    }
    const uint64_t relw = off > pos0 ? off - pos0 : 0ull;
    const uint32_t rel = relw > 0xfffffff0ull ? 0xfffffff0u : (uint32_t)relw;
    const uint64_t bend = r + 32u < F ? (uint64_t)a.region_off[r + 32u] * a.cs : total;
    const uint64_t brel = bend - pos0;
    uint32_t next = __shfl_down_sync(0xffffffffu, rel, 1);   // where this lane's region ends
    if (lane == 31u) next = brel > 0xfffffff0ull ? 0xfffffff0u : (uint32_t)brel;
    uint64_t uend = (bend + 15u) / 16u;
    if (uend > u1) uend = u1;
    if (uend > u + (1u << 26)) uend = u + (1u << 26);
    const uint32_t units = (uint32_t)(uend - u);
    // regions that follow one another in the buffer too (a list's runs of chunks) are one run
    const uint64_t src_first = __shfl_sync(0xffffffffu, src0, 0);   // by every lane: not inside the || below
    if (__all_sync(0xffffffffu, !has || src0 == src_first))
      next = brel > 0xfffffff0ull ? 0xfffffff0u : (uint32_t)brel;
    auto region_of = [&](uint32_t pos) {   // largest j with region start j <= pos
      uint32_t j = 0;
#pragma unroll
      for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t o = __shfl_sync(0xffffffffu, rel, j + step);
        if (o <= pos) j += step;
      }
      return j;
    };
    for (uint32_t b = 0; b < units;) {
      {   // one region over the warp's next whole steps: stream to its end
        const uint32_t j = region_of(16u * b);
        const uint32_t end = __shfl_sync(0xffffffffu, next, j);
        uint64_t s = __shfl_sync(0xffffffffu, src0, j) + 16ull * b;
        const uint64_t room = s < a.len ? (a.len - s) / 16u : 0ull;   // units before the buffer's end
        uint32_t whole = (end / 16u < units ? end / 16u : units) - b;
        if (whole > room) whole = (uint32_t)room;
        if (whole >= 32u * U) {
          s += 16ull * lane;
          uint4* d = dst + u + b + lane;
          b += whole / (32u * U) * (32u * U);
          for (uint32_t left = whole / (32u * U); left; left--) {
            uint4 v[U];
#pragma unroll
            for (uint32_t i = 0; i < U; i++)
              v[i] = ALIGNED ? __ldg(reinterpret_cast<const uint4*>(a.data + s + 512u * i))
                             : load_unit(a.data, a.len, s + 512u * i);
#pragma unroll
            for (uint32_t i = 0; i < U; i++) d[32u * i] = v[i];
            s += 512u * U;
            d += 32u * U;
          }
          continue;
        }
      }
      uint4 v[U];
      uint32_t st = 0;   // bit i: unit i is this lane's to store
#pragma unroll
      for (uint32_t i = 0; i < U; i++) {
        const uint32_t g = b + lane + 32u * i;
        const bool act = g < units;
        const uint32_t pos = act ? 16u * g : 16u * b;
        const uint32_t j = region_of(pos);
        const uint32_t end = __shfl_sync(0xffffffffu, next, j);
        const uint64_t s = __shfl_sync(0xffffffffu, src0, j) + pos;
        if (!act) continue;
        if (pos + 16u <= end && s < a.len && a.len - s >= 16u) {
          st |= 1u << i;
          v[i] = ALIGNED ? __ldg(reinterpret_cast<const uint4*>(a.data + s)) : load_unit(a.data, a.len, s);
        } else if (ALIGNED) {
          gather_end_unit(a.data, a.len, s, dst + u + g);
        } else {
          gather_unit_bytes(GatherBytes{a.data, a.len, a.cs, total, a.region_off, a.first_list, F, a.n, a.N, a.D},
                            dst_base, u + g, r + j);
        }
      }
#pragma unroll
      for (uint32_t i = 0; i < U; i++)
        if ((st >> i) & 1u) dst[u + b + lane + 32u * i] = v[i];
      b += 32u * U;
    }
    u = uend;
    if (16ull * uend >= bend) r += 32u;   // else a step's limit: the same regions go on
  }
}

// ---------------------------------------------------------------- scatter and gather, one launch
// CTAs below shift_ctas(ranges, B) scatter the shifted entries, one range per warp; the others
// write the first-occurrence list and the data.  Both need only the layout.
__host__ __device__ __forceinline__ uint32_t shift_warps(uint32_t bcap) {   // ranges per CTA: 8 KB of positions
  const uint32_t w = 2048u / (bcap ? bcap : 1u);
  return w < 1u ? 1u : (w > EMIT_THREADS / 32u ? EMIT_THREADS / 32u : w);
}
__host__ __device__ __forceinline__ uint32_t shift_ctas(uint32_t ranges, uint32_t bcap) {
  const uint32_t w = shift_warps(bcap);
  return (ranges + w - 1u) / w;
}
template <bool ALIGNED>
__device__ __forceinline__ void diff_emit_body(const DiffArgs& a, uint32_t bid, uint32_t nb, uint32_t bcap,
                                               uint32_t ranges) {
  extern __shared__ uint32_t run[];
  const uint32_t nbs = shift_ctas(ranges, bcap);
  if (bid >= nbs) {
    gather_body<ALIGNED>(a, bid - nbs, nb - nbs);
    return;
  }
  const uint32_t warp = threadIdx.x >> 5, warps = shift_warps(bcap);
  const uint32_t range = bid * warps + warp;
  if (warp < warps && range < ranges) shift_write_range(a, range, ranges, bucket_count(a, bcap), run + warp * bcap);
}
template <bool ALIGNED>
__global__ void __launch_bounds__(EMIT_THREADS, 2) diff_emit_kernel(DiffArgs a0, uint32_t bcap, uint32_t ranges) {
  griddep_enter();
  diff_emit_body<ALIGNED>(with_round(a0), blockIdx.x, gridDim.x, bcap, ranges);
  // the last CTA hands the checkpoint's state to the host: a copy enqueued behind this kernel
  // took 10 us of a small checkpoint
  if (a0.state_host == nullptr) return;
  __shared__ uint32_t last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&a0.meta->emitted, 1u) == gridDim.x - 1u;
    if (last) {
      a0.stamps->end = device_time_ns();
      __threadfence();
    }
  }
  __syncthreads();
  if (last)
    for (uint32_t i = threadIdx.x; i < a0.state_words; i += blockDim.x) a0.state_host[i] = __ldcg(a0.state + i);
}
// Four CTAs per SM (64 registers): a batch's diffs are gathered in short runs, a chunk to a few
// hundred, that wait on memory, and with two CTAs an increment of 256 buffers (13 GB, 10 % changed)
// spent 1607 us here, with four 1108.  The single launch keeps two: one run over a whole 4 GiB
// baseline streams at 1.36 ms with two and 1.5 with four.
template <bool ALIGNED>
__global__ void __launch_bounds__(EMIT_THREADS, ALIGNED ? 4 : 2) diff_emit_seg(SegGrid s) {
  uint32_t bid, nb;
  const uint32_t h = seg_locate(s, bid, nb);
  __shared__ DiffArgs a;
  for (uint32_t i = threadIdx.x; i < sizeof(DiffArgs) / 4u; i += blockDim.x)
    reinterpret_cast<uint32_t*>(&a)[i] = reinterpret_cast<const uint32_t*>(s.args + h)[i];
  __syncthreads();
  diff_emit_body<ALIGNED>(a, bid, nb, s.bcap[h], s.gs[h]);
}

static uint32_t grid_for(uint64_t units, uint64_t per_cta, uint32_t cap) {
  const uint64_t g = (units + per_cta - 1) / per_cta;
  return g < 1 ? 1u : (g > cap ? cap : (uint32_t)g);
}

// grids follow the buffer size (host-known bounds: F, S <= n), so a small buffer is not charged
// for hundreds of idle CTAs per launch; large buffers get the full grids
DiffGrids diff_grids(const DiffArgs& a, uint32_t bcap, int sm_count) {
  DiffGrids r;
  r.g = grid_for(((uint64_t)a.N + 64u) / 64u, 512, COMPACT_GRID);   // ~1 64-node load per thread
  // shifted-entry ranges: the layout scans every range's count per bucket in one CTA, so fewer,
  // longer ranges (<= 296) keep it short; the scatter walks each range with one warp
  r.gs = grid_for(a.n, 8192, SHIFT_GRID);
  r.gc = r.gs + grid_for(a.n, 4096, (uint32_t)sm_count * 8u);
  // two waves of resident CTAs for the gather, four from 2 GiB on, where the one run of a baseline gains
  // what increments lose.  Diff assembly with two and four, baselines and increments (5 % in runs of
  // 32 chunks of 128 B), us: 32 MiB 31 and 36, 22 and 29; 128 MiB 63 and 67, 25 and 32; 512 MiB 195 and
  // 189, 35 and 44; 2 GiB 734 and 697, 87 and 96; 4 GiB baseline 1540 and 1450
  const uint64_t bytes = (uint64_t)a.n * a.cs;
  r.ge = shift_ctas(r.gs, bcap) + grid_for(bytes, 32768, (uint32_t)sm_count * (bytes >> 31 ? 8u : 4u));
  // 16-byte aligned source units; both kinds write a 16-byte aligned data section
  r.variant = (a.cs % 16u == 0) && ((reinterpret_cast<uintptr_t>(a.data) & 15u) == 0) ? 0 : 1;
  return r;
}

uint32_t diff_emit_smem(uint32_t bcap) { return (uint32_t)sizeof(uint32_t) * shift_warps(bcap) * bcap; }

cudaError_t launch_collect_diff_batch(const DiffBatch& b, cudaStream_t stream, uint32_t* launches) {
  if (b.max_bcap > MAX_BUCKETS || b.base.n == 0) return cudaErrorInvalidValue;
  SegGrid s = b.base;
  uint32_t c = 0;
  s.beg = b.beg_g;   diff_count_seg<<<b.tot_g, COMPACT_THREADS, 0, stream>>>(s); c++;
  s.beg = b.beg_g;   diff_write_seg<<<b.tot_g, COMPACT_THREADS, 0, stream>>>(s); c++;
  s.beg = b.beg_gc;  diff_shift_seg<<<b.tot_gc, SHIFT_THREADS, sizeof(uint32_t) * b.max_bcap, stream>>>(s); c++;
  for (int v = 0; v < GATHER_VARIANTS; v++) {
    if (!b.tot_emit[v]) continue;
    s.beg = b.beg_emit[v];
    if (v == 0) diff_emit_seg<true><<<b.tot_emit[v], EMIT_THREADS, b.max_emit_smem, stream>>>(s);
    else diff_emit_seg<false><<<b.tot_emit[v], EMIT_THREADS, b.max_emit_smem, stream>>>(s);
    c++;
  }
  if (launches) *launches = c;
  return cudaGetLastError();
}

cudaError_t launch_collect_diff(const DiffArgs& a, uint32_t bcap, int sm_count, cudaStream_t stream) {
  const DiffGrids dg = diff_grids(a, bcap, sm_count);
  // bcap is a capacity; each kernel reads the checkpoint's bucket count from rs
  if (bcap > MAX_BUCKETS) return cudaErrorInvalidValue;
  // one kernel after another, each launched to overlap its start with its predecessor's end
  // (launch_dependent)
  cudaError_t e = launch_dependent(diff_count_kernel, dg.g, COMPACT_THREADS, 0, stream, a, bcap);
  if (e == cudaSuccess) e = launch_dependent(diff_write_kernel, dg.g, COMPACT_THREADS, 0, stream, a);
  if (e == cudaSuccess)
    e = launch_dependent(diff_shift_kernel, dg.gc, SHIFT_THREADS, sizeof(uint32_t) * bcap, stream, a, bcap, dg.gs);
  if (e == cudaSuccess)
    e = launch_dependent(dg.variant == 0 ? diff_emit_kernel<true> : diff_emit_kernel<false>, dg.ge, EMIT_THREADS,
                         diff_emit_smem(bcap), stream, a, bcap, dg.gs);
  return e;
}

}  // namespace b2d
