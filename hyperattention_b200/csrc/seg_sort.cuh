// Batches of segment sorts (keys of at most 8 bits).
#pragma once
#include "common.cuh"

namespace ha {

struct SortJob {
  const int32_t* codes;
  int32_t* out;
  int n, span, seg_off, seg_len, parts;      // as ha_seg_sort; parts = n / span
  int segs, chunks;                          // segments; chunks of a segment
  int first, first_seg;                      // first chunk / segment of the job in the batch
};
struct SortJobs {
  static constexpr int MAX = 48;
  int count = 0, longest = 0;
  uint32_t* hist = nullptr;
  SortJob job[MAX];
  static bool fits(int seg_len, int key_bits);
  void add(const int32_t* codes, int rows, int n, int span, int seg_off, int seg_len, int32_t* out);
  // workspace: ha_seg_sort_workspace_bytes of every sort of the batch, added up, is more than enough
  int run(uint32_t* workspace, cudaStream_t st);
};

}  // namespace ha
