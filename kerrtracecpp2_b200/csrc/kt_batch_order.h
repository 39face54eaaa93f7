// kt_batch_order.h -- where a batch group's chunks of 32 rays go
// (launch_batch_order): tables built on the host, the rank of a chunk on
// either side.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#if defined(__CUDACC__)
#define KT_BO __host__ __device__ inline
#else
#define KT_BO inline
#endif

namespace kt {

// The tables, n_words 32-bit words at `words` (host or device).  Frames with
// equally many whole chunks form a class: chunks of such frames are compared
// with others' once for all of them, so that a rank costs as many steps as
// there are frame sizes, not frames.
struct BatchOrder {
  const uint32_t* words = nullptr;
  size_t n_words = 0;
  uint32_t n_frames = 0, n_classes = 0;
  // whole chunks before frame k; n_frames + 1 of them
  KT_BO const uint32_t* first_chunk() const { return words; }
  // rays beyond whole chunks before frame k; n_frames + 1
  KT_BO const uint32_t* rest() const { return words + n_frames + 1; }
  // the frames by class, in order within one
  KT_BO const uint32_t* members() const { return rest() + n_frames + 1; }
  // whole chunks of a class' frames (not zero, ascending)
  KT_BO const uint32_t* chunks() const { return members() + n_frames; }
  // a class' first member; n_classes + 1
  KT_BO const uint32_t* first_member() const { return chunks() + n_classes; }
};

// The tables of frames of sizes[k] rays (at most 2^31 in all), on the host;
// the result's words are those of `store`.
inline BatchOrder make_batch_order(const std::vector<uint64_t>& sizes, std::vector<uint32_t>* store) {
  const uint32_t nf = (uint32_t)sizes.size();
  std::vector<uint32_t> members(nf), chunks, first;
  for (uint32_t k = 0; k < nf; ++k) members[k] = k;
  std::stable_sort(members.begin(), members.end(),
                   [&](uint32_t a, uint32_t b) { return sizes[a] / 32 < sizes[b] / 32; });
  for (uint32_t i = 0; i < nf; ++i) {
    const uint32_t c = (uint32_t)(sizes[members[i]] / 32);
    if (c != 0 && (chunks.empty() || chunks.back() != c)) {
      chunks.push_back(c);
      first.push_back(i);
    }
  }
  first.push_back(nf);
  store->clear();
  for (int what = 0; what < 2; ++what) {
    uint32_t sum = 0;
    for (uint32_t k = 0; k < nf; ++k) {
      store->push_back(sum);
      sum += (uint32_t)(what == 0 ? sizes[k] / 32 : sizes[k] % 32);
    }
    store->push_back(sum);
  }
  store->insert(store->end(), members.begin(), members.end());
  store->insert(store->end(), chunks.begin(), chunks.end());
  store->insert(store->end(), first.begin(), first.end());
  BatchOrder o;
  o.words = store->data();
  o.n_words = store->size();
  o.n_frames = nf;
  o.n_classes = (uint32_t)chunks.size();
  return o;
}

// How many i in [0, n) have a[i] <= v (a ascending).
KT_BO uint32_t count_at_most(const uint32_t* a, uint32_t n, uint32_t v) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (a[mid] <= v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Chunks that go before chunk j of frame k among the frames of the classes
// c0, c0 + step, ...: chunk i of a frame m with F_m chunks does when
// (i + 1/2) / F_m < (j + 1/2) / F_k, or equal and m < k.  With N = (2 j + 1)
// F_m these i are the odd t = 2 i + 1 with t F_k < N (or = N).
KT_BO uint32_t chunk_rank(const BatchOrder& o, uint32_t k, uint32_t j, uint32_t c0, uint32_t step) {
  const uint64_t Fk = o.first_chunk()[k + 1] - o.first_chunk()[k];
  uint32_t rank = 0;
  for (uint32_t c = c0; c < o.n_classes; c += step) {
    const uint64_t N = (2 * (uint64_t)j + 1) * o.chunks()[c];
    const uint32_t first = o.first_member()[c], n = o.first_member()[c + 1] - first;
    const uint64_t q = N / Fk, r = N % Fk;
    const uint32_t below = (uint32_t)((q - (r == 0 ? 1 : 0) + 1) / 2);  // odd t <= (N - 1) / F_k
    rank += n * below;
    if (r == 0 && (q & 1u)) rank += count_at_most(o.members() + first, n, k) - (Fk == o.chunks()[c] ? 1 : 0);
  }
  return rank;
}

}  // namespace kt
