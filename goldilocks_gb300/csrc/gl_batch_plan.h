// Host-side rules of a batch of polynomials that need no CUDA (gl_batch.cu).
#pragma once
#include <algorithm>
#include <utility>
#include <vector>

#include "../../include/goldilocks_gpu.h"

// Whether two polynomials of the batch share memory (length 1 is a no-op and
// touches none).  A list in address order, as a packed pool's is, is one walk.
inline bool gl_batch_shares_memory(const gl_poly *polys, uint64_t count) {
  const auto first = [&](uint64_t i) { return (uint64_t)(uintptr_t)polys[i].data; };
  bool ordered = true;
  uint64_t end = 0;
  for (uint64_t i = 0; i < count && ordered; i++) {
    if (polys[i].len <= 1) continue;
    ordered = first(i) >= end;
    end = first(i) + 8 * polys[i].len;
  }
  if (ordered) return false;
  std::vector<std::pair<uint64_t, uint64_t>> spans;  // [first, end) in bytes
  for (uint64_t i = 0; i < count; i++)
    if (polys[i].len > 1) spans.push_back({first(i), first(i) + 8 * polys[i].len});
  std::sort(spans.begin(), spans.end());
  for (size_t i = 1; i < spans.size(); i++)
    if (spans[i].first < spans[i - 1].second) return true;
  return false;
}

// The order in which the polynomials of a batch that share memory are
// transformed, one after another: those marked in `plain` (lengths the bucket
// kernels are not built for) in list order, then by (length, direction), equal
// ones in list order -- the order of the buckets' kernels in one stream.
inline std::vector<uint64_t> gl_batch_order(const gl_poly *polys, uint64_t count, const std::vector<bool> &plain) {
  std::vector<uint64_t> order(count);
  for (uint64_t i = 0; i < count; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](uint64_t a, uint64_t b) {
    if (plain[a] || plain[b]) return plain[a] && !plain[b];
    return std::make_pair(polys[a].len, polys[a].dir) < std::make_pair(polys[b].len, polys[b].dir);
  });
  return order;
}

// What a captured bucket graph is kept under: its kernel nodes, their tables
// and the kernels chosen for its SMs belong to one device.
struct gl_bucket_key {
  int device;
  std::vector<std::pair<uint64_t, int>> sig;  // (len, dir) per item, bucket order
  bool operator<(const gl_bucket_key &o) const { return device != o.device ? device < o.device : sig < o.sig; }
};

// The launches of a bucket graph, as items [first, end): a bucket's items in one
// launch, or in several of `most` (a launch has them on grid.y) items or fewer.
inline std::vector<std::pair<size_t, size_t>> gl_bucket_runs(const std::vector<std::pair<uint64_t, int>> &sig,
                                                             size_t most) {
  std::vector<std::pair<size_t, size_t>> runs;
  for (size_t j = 0, end; j < sig.size(); j = end) {
    for (end = j + 1; end < sig.size() && end - j < most && sig[end] == sig[j];) end++;
    runs.push_back({j, end});
  }
  return runs;
}
