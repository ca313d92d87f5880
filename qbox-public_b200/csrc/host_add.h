// Adding a block that arrives in pieces to a caller's array, on the host.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

namespace qbx {

// dst[i] += scale * x[i] for i < n.  If a piece of x fails to come, dst gets the
// values it had back (kept in old, n of them) and the piece's code is returned
// (0: added).  fetch(slot, first, count, &x) gives the address of `count` values
// from `first` on, valid until the slot's next call, or returns a code.  Each of
// the slots is served by a thread of its own, where there is one to be had.
template <typename Fetch>
int add_all_or_nothing(size_t n, size_t piece, int slots, double scale, double* old, double* dst,
                       const Fetch& fetch) {
  const size_t pieces = (n + piece - 1) / piece;
  std::vector<char> added(pieces, 0);
  std::vector<std::thread> threads;
  threads.reserve(slots);
  std::atomic<int> code{0};
  auto count = [&](size_t i) { return std::min(piece, n - i * piece); };
  auto serve = [&](int slot) {
    for (size_t i = slot; i < pieces && code == 0; i += slots) {
      const size_t first = i * piece, m = count(i);
      const double* x = nullptr;
      const int c = fetch(slot, first, m, &x);
      int none = 0;
      if (c) {
        code.compare_exchange_strong(none, c);
        return;
      }
      double *d = dst + first, *o = old + first;
      added[i] = 1;
      for (size_t k = 0; k < m; k++) {
        const double v = d[k];
        o[k] = v;
        d[k] = v + scale * x[k];
      }
    }
  };
  int served = 1;   // this thread serves slot 0 and those without a thread
  try {
    for (; served < slots; served++) threads.emplace_back(serve, served);
  } catch (const std::exception&) {
  }
  serve(0);
  for (int t = served; t < slots; t++) serve(t);
  for (std::thread& t : threads) t.join();
  for (size_t i = 0; code && i < pieces; i++)
    if (added[i]) std::memcpy(dst + i * piece, old + i * piece, count(i) * sizeof(double));
  return code;
}

}  // namespace qbx
