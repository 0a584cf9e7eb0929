// Restart kernel arguments (see restart.cu).
#pragma once
#include "common.cuh"
#include "dedup_kernels.cuh"

namespace b2d {

// One diff's lookups, dense over the leaves of the restarted checkpoint.  An entry means
// something only where its bit in flag[c] is set (the flags are cleared for each diff, the
// arrays are not):
//   dist[c] (flag bit 0) : chunk offset of leaf c inside the diff's data section (u32, like
//                          the reference, which computes some of these offsets in wrapping u32
//                          arithmetic)
//   rep[c]  (flag bit 1) : source NodeID of shifted leaf c
constexpr uint8_t R_HAS_DIST = 1, R_HAS_REP = 2;
struct RestartSlot {
  uint32_t* dist;
  uint2* rep;
  uint8_t* flag;
};

// expansion of one diff's region lists
struct RestartArgs {
  const uint8_t* diff;     // one diff (header at offset 0 of this pointer)
  uint64_t diff_size;
  uint64_t first_off, count_off, shift_off, data_off;   // byte offsets from `diff`
  uint32_t F, P, S;
  uint32_t cur_id;         // chkpt_id of this diff's header
  uint64_t datalen;        // this diff's header datalen
  uint32_t cs;             // this diff's header chunk size
  uint32_t n, N;           // chunks / nodes of the checkpoint being restarted
  int is_main;
  uint8_t* out;            // restart buffer (device)
  uint64_t out_len;        // datalen of the checkpoint being restarted
  uint2* node_list;        // n: NodeID each chunk named by the main diff still comes from
  uint8_t* mflag;          // n: chunk named by the main diff
  RestartSlot slot;        // this diff's lookups
  const unsigned long long* cum;   // inclusive shift counts per checkpoint id (ncum entries)
  uint32_t ncum;
  // per list (0: first-occurrence regions, 1: shifted regions; the two may share memory where one
  // list is expanded before the other is scanned)
  uint32_t* offs[2];       // per entry: exclusive offset of its first chunk
  uint32_t* rstart[2];     // per entry: leftmost leaf of the region's node
  uint32_t* partial[2];    // SCAN_GRID
  unsigned long long* total[2];
  uint32_t* pstart;        // per shift entry: leftmost leaf of the source node
  uint32_t* rtree;         // per shift entry: source checkpoint id
  DevStatus* st;
  // added to every node id read from the diff: list-approach diffs name chunks, which the
  // restart handles as the leaves n-1+c of the same heap (0 for tree diffs)
  uint32_t id_bias;
  // chunk copies (set by launch_restart_diff): piece width in bytes (16/8/4, dividing the chunk
  // size and the alignment of `out` and of the data section; 0: one lane copies a whole chunk),
  // pieces per chunk and its log2 (0xff when not a power of two)
  uint32_t width, per, per_log2;
};

// Older diffs resolved by one walk over the chunks, newest first.
constexpr uint32_t RESTART_WINDOW = 8;
constexpr uint64_t RESTART_SLOT_BYTES = 8ull << 30;   // memory for the window slots of one restart
constexpr uint64_t RESTART_HOST_BYTES = 256ull << 20; // the same, and for the copies, of host diffs
struct RestartWalk {
  uint32_t count;          // diffs in this window
  int dense;               // node_list holds every chunk's NodeID (an earlier window wrote it)
  int last;                // no window follows (node_list is not written back)
  uint32_t main_cur;       // main diff's id: chunks it does not name start at (leaf, main_cur - 1)
  uint32_t n, N, cs;
  uint8_t* out;
  uint64_t out_len;
  uint2* node_list;
  const uint8_t* mflag;
  DevStatus* st;
  uint32_t width, per, per_log2;
  const uint8_t* data[RESTART_WINDOW];      // data sections
  uint64_t data_len[RESTART_WINDOW];        // bytes in each data section
  uint64_t datalen[RESTART_WINDOW];         // each header's datalen
  uint32_t cur[RESTART_WINDOW];             // each header's chkpt_id
  RestartSlot slot[RESTART_WINDOW];
};

// The diffs expanded together by launch_restart_diffs: the main diff and a window, or a window.
struct RestartSet {
  uint32_t count;
  RestartArgs a[RESTART_WINDOW + 1];
};

// The one first-occurrence region (if any) whose root spans two leaf depths (chunk count not a
// power of two), found on the device after the region offsets are known.
struct StraddleInfo {
  int present;
  uint32_t root, region_off, lo, hi;
};
// roots that can span two depths: the common ancestors of the last inner node (n-2) and the
// first leaf of level D-1 (n-1), computed on the host from n alone
struct StraddleQuery {
  uint32_t count;
  uint32_t anc[32];
};
StraddleQuery straddle_query(uint32_t n);

// fills a.cum (device) from the repeat table of the device-resident diff a.diff
cudaError_t launch_restart_cum(const RestartArgs& a, cudaStream_t s);
// Expands one diff: clears the flags of a.slot (for the main diff also a.mflag), fills the
// slot, and for the main diff fills node_list and copies the chunks it resolves itself.  `sd`
// is device memory for the straddling-region record of this diff.
cudaError_t launch_restart_diff(const RestartArgs& a, StraddleInfo* sd, int sm_count, cudaStream_t s);
// The same for several diffs with a scratch of their own each (lists, slots, cum), in one launch
// per step instead of nine per diff: a restart of 1 GiB from five diffs spent 250 of its 940 us
// between 45 small launches.  Fills every a.cum itself; the flags of all slots are cleared by the
// caller.  `sd` has one record per diff.
cudaError_t launch_restart_diffs(const RestartSet& set, StraddleInfo* sd, int sm_count, cudaStream_t s);
int restart_diffs_launches(uint32_t n, bool list);   // kernels of one call
// header_t of a diff (include/utils.hpp:29-37) from its eight words, and the offsets that follow from
// it; false where it does not fit a diff of `size` bytes
struct DiffHeader {
  uint32_t ref_id, chkpt_id;
  uint64_t datalen;
  uint32_t cs, F, P, S;
  uint64_t first_off, count_off, shift_off, data_off;
};
__host__ __device__ inline bool parse_header(const uint32_t* w, uint64_t size, DiffHeader& h) {
  h.ref_id = w[0];
  h.chkpt_id = w[1];
  h.datalen = (uint64_t)w[2] | ((uint64_t)w[3] << 32);
  h.cs = w[4];
  h.F = w[5];
  h.P = w[6];
  h.S = w[7];
  h.first_off = 32;
  h.count_off = h.first_off + 4ull * h.F;
  h.shift_off = h.count_off + 8ull * h.P;
  h.data_off = h.shift_off + 8ull * h.S;
  return h.data_off <= size && h.cs > 0 && h.datalen > 0;
}
// The chain of diffs idx, idx - 1, ... (at most `count`, of 32 bytes and more) as far as their headers
// carry it: the headers' words to `out`, 8 each, how many to `seen` (pinned host memory).
constexpr uint32_t RESTART_HEADERS = 64;
struct RestartHeaders {
  uint32_t count;
  int idx;
  const uint8_t* diff[RESTART_HEADERS];
  uint64_t size[RESTART_HEADERS];
};
cudaError_t launch_restart_headers(const RestartHeaders& h, uint32_t* out, uint32_t* seen, cudaStream_t s);
// resolves the chunks owed by the window's diffs and copies them
cudaError_t launch_restart_walk(const RestartWalk& w, int sm_count, cudaStream_t s);

}  // namespace b2d
