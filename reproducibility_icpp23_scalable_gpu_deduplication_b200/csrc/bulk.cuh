// Bulk build of a baseline's tree digests and digest map (bulk.cu).
#pragma once
#include "dedup_kernels.cuh"
#include "scan.cuh"

namespace b2d {

// Smallest chunk counts that are built in bulk: below them the build's launches cost more than the
// inserts they replace.  Whole baselines of 128 B chunks, bulk against one by one: trees of 2^15
// chunks 123 and 131 us, 2^17 138 and 182 us, 2^19 229 and 368 us; lists, which have no inner
// digests to insert, of 2^18 chunks 167 and 157 us, 2^19 204 and 222 us.
constexpr uint32_t BULK_MIN_TREE = 1u << 15;
constexpr uint32_t BULK_MIN_LIST = 1u << 19;

struct BulkArgs {
  Digest* tree;
  uint8_t* leaflab;
  MapView map;
  DevStatus* st;
  uint32_t n, N, D, cur;
  int kind, list;
  uint32_t first_node;   // entries are the nodes first_node .. first_node + count - 1
  uint64_t count;
  uint32_t ranges;       // of the table
  uint32_t buckets;      // of the first scatter pass; 0: one pass
  uint32_t* start;       // ranges + 1: entry counts, then starts (zeroed)
  uint32_t* alloc;       // ranges
  uint32_t* alloc1;      // buckets
  uint32_t* tile_beg;    // buckets + 1
  Key128 *key1, *key2;   // entries after the first and the last scatter pass
  uint32_t *id1, *id2;
  uint32_t* overflow;    // nodes whose probing left their range
  uint32_t* over_count;  // (zeroed)
  uint32_t* lost;        // bit per node: lost its entry to another parent (zeroed)
  int* lost_any;
  int* zero_exists;
  unsigned long long* stamp;   // where the build's first launch records its start
};

// where the build's arrays lie: byte offsets into the diff buffer (key*, id*; it is free until the
// diff is assembled) and into a scratch of 4 bytes per chunk (the rest; its first zeroed_bytes must
// be zero).  The overflow list is another 4 bytes per chunk.
struct BulkPlan {
  uint64_t count;
  uint32_t ranges, buckets;
  uint64_t key1, key2, id1, id2;
  uint64_t zeroed_bytes, start, over_count, lost, alloc, alloc1, tile_beg;
};
// false: this tree and table are not built in bulk: too few chunks, more than BULK_MAX_RANGES table
// ranges, or entries that do not fit the diff buffer (40 bytes per chunk of a tree in one scatter pass,
// 80 in two, of the buffer's 16 + chunk size: from 24 and from 64 byte chunks on; lists half of that)
bool bulk_plan(uint32_t n, uint64_t cap, int list, uint64_t diff_bytes, BulkPlan& p);
cudaError_t launch_bulk(const BulkArgs& a, int sm_count, cudaStream_t stream, uint32_t* launches);

}  // namespace b2d
