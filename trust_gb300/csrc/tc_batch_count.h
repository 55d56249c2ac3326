// tc_batch_count.h — host interface of the batch counting kernel (tc_batch_count.cu).
#pragma once
#include "tc_common.cuh"

namespace tc {

struct BatchCountArgs {
  const int64_t *beg;
  const int32_t *adj;
  const int *lists;          // every degree class's rows, at ctl->class_off
  TcControl *ctl;            // the combined block: list sizes and offsets, queue heads, count
  const int *graph_of;       // graph of every row
  const int64_t *graph_vbeg; // graph g's ids: [graph_vbeg[g], graph_vbeg[g + 1])
  unsigned long long *graph_counts;
  int *huge_tables;          // spill tables of rows above the CTA class: huge_blocks of 2^huge_log2 ints
  int huge_log2, huge_blocks;
  int warp_words;            // shared-memory words per warp (>= 128, multiple of 4)
  int table_bytes;           // shared memory of the tables (a multiple of 16)
  int chunk;                 // steps per queue claim
};

// The most words per warp with which four CTAs of eight warps stay resident on an SM.
int batch_count_warp_words(int *words);
// Resident CTAs per SM with table_bytes of tables (0: too much shared memory); the SM's other memory becomes L1.
int batch_count_occupancy(int threads, bool bitmaps, size_t table_bytes, int *blocks_per_sm);
int launch_batch_count(const BatchCountArgs &a, int blocks, int threads, bool bitmaps, cudaStream_t st);

}  // namespace tc
