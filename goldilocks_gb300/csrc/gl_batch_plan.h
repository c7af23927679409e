// Host-side rules of a batch of polynomials that need no CUDA (gl_batch.cu).
#pragma once
#include <algorithm>
#include <utility>
#include <vector>

#include "../../include/goldilocks_gpu.h"

// Whether two polynomials of the batch share memory (length 1 is a no-op and
// touches none).  A list in address order, as a packed pool's is, is one walk;
// any other is sorted into about two cells of the address range per polynomial
// first (1 024 in random order: std::sort alone took 28 us of a 920 us batch).
inline bool gl_batch_shares_memory(const gl_poly *polys, uint64_t count) {
  const auto first = [&](uint64_t i) { return (uint64_t)(uintptr_t)polys[i].data; };
  bool ordered = true;
  uint64_t lo = ~0ull, hi = 0, last = 0, total = 0, n = 0;
  for (uint64_t i = 0; i < count; i++) {
    if (polys[i].len <= 1) continue;
    const uint64_t end = first(i) + 8 * polys[i].len;
    ordered = ordered && first(i) >= last;
    last = end;
    lo = std::min(lo, first(i));
    hi = std::max(hi, end);
    total += 8 * polys[i].len;
    n++;
  }
  if (ordered) return false;
  if (total > hi - lo) return true;
  int shift = 0;
  while ((hi - lo) >> shift >= 2 * n) shift++;
  std::vector<uint32_t> at(((hi - lo) >> shift) + 2, 0);  // where each cell starts
  for (uint64_t i = 0; i < count; i++)
    if (polys[i].len > 1) at[((first(i) - lo) >> shift) + 1]++;
  for (size_t c = 1; c < at.size(); c++) at[c] += at[c - 1];
  std::vector<std::pair<uint64_t, uint64_t>> spans(n);  // [first, end) in bytes
  for (uint64_t i = 0; i < count; i++)
    if (polys[i].len > 1) spans[at[(first(i) - lo) >> shift]++] = {first(i), first(i) + 8 * polys[i].len};
  for (size_t c = 0, a = 0; c + 1 < at.size(); a = at[c++])  // at[c] is now where cell c ends
    if (at[c] > a + 1) std::sort(spans.begin() + a, spans.begin() + at[c]);
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
