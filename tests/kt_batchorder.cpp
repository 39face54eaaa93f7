// kt_batchorder.cpp -- TEST-ONLY host build of kt_batch_order.h.
#include "../kerrtracecpp2_b200/csrc/kt_batch_order.h"

extern "C" {
// rank[i] of every whole chunk, frame after frame; returns the classes.
int bo_ranks(int n_frames, const uint64_t* sizes, uint32_t* rank) {
  std::vector<uint32_t> store;
  const kt::BatchOrder o = kt::make_batch_order(std::vector<uint64_t>(sizes, sizes + n_frames), &store);
  for (uint32_t w = 0; w < o.first_chunk()[n_frames]; ++w) {
    const uint32_t k = kt::count_at_most(o.first_chunk(), o.n_frames + 1, w) - 1;
    rank[w] = 0;
    for (uint32_t c0 = 0; c0 < 3; ++c0)  // dealt as to lanes
      rank[w] += kt::chunk_rank(o, k, w - o.first_chunk()[k], c0, 3);
  }
  return (int)o.n_classes;
}
}
