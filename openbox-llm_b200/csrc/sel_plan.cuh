// Index structures of a selection block list, as the tcgen05 selection kernels walk them.
//
// A selection list names blocks of 16, 32 or 64 tokens; the kernels work on 64-token key tiles.
// For every (batch, kv head) unit and key tile: the queries that list one of the tile's blocks
// (ascending, each once) with the 16-token column groups of the tile they attend, and for every
// (query, slot) the position of that pair, -1 where the slot is empty or an earlier slot of the
// query already names the tile.  Every unit owns its own range of pairs, offsets and work items, so
// that the builders of different units do not wait for one another.
#pragma once

#include "common.cuh"

namespace nsa {

// Pair entry: query position in the low 24 bits, column groups (bit i: keys 16 i .. 16 i + 15 of
// the tile) above them.
constexpr int kPairPosBits = 24;
constexpr uint32_t kPairPosMask = (1u << kPairPosBits) - 1u;

// The block-outer selection kernels take one work item per CTA: a key tile of one unit and a chunk
// of at most kSelChunkTiles of its row tiles.  A tile that many queries list (an attention-sink
// block, a forced initial block) becomes several items, so no single CTA walks its whole list.
constexpr int kSelChunkTiles = 128;

struct SelPlanHeader {
  unsigned long long union_tiles;   // distinct (query tile, key tile) pairs of the query-outer kernel
  unsigned long long pairs;         // pairs over all units
  unsigned long long repeats;       // not 0: some query names a block of 16 or 32 tokens more than once
  unsigned long long pad[29];
};

// device pointers into a plan buffer
struct SelPlan {
  SelPlanHeader* hdr;
  int32_t* n_items;        // [units]
  int4* items;             // [units][max_items]: unit, key tile, first row tile, chunks of the tile
  int32_t* offsets;        // [units][n_ktiles + 1]: first pair of a key tile; unit u starts at u * T * S
  int32_t* pairs;          // [units * T * S]
  int32_t* pair_of_slot;   // [units][T][S]
  int max_items;
};

struct SelPlanLayout {
  size_t hdr, n_items, items, offsets, pairs, pos, scratch, total;
  int n_ktiles, max_items, chunk_words, n_chunks;
};
SelPlanLayout sel_plan_layout(int units, int T, int S, int nq);
SelPlan sel_plan_at(const void* base, const SelPlanLayout& l);
int sel_plan_build(const int32_t* block_idx, void* base, const SelPlanLayout& l, int units, int T, int S,
                   int block_size, int nq, int nq_union, cudaStream_t st);

}  // namespace nsa
