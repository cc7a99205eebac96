// Every arc of a vertex's range is walked once by one of its lanes, up to the
// largest arc ids, where a lane's step past the end passes 2^31.
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include "cgc_arcs.h"

template <int W>
void check(int32_t first, int32_t past) {
  int64_t seen = 0;
  for (int lane = 0; lane < W; ++lane) {
    int steps = 0;
    for (cgc::ArcWalk<W> a(first, past, lane); a.on(); a.step(), ++steps) {
      const int64_t at = a.at;
      if (at < first || at >= past || (at - first) % W != lane || steps > (past - first) / W) {
        std::printf("W %d range [%d, %d) lane %d: arc %lld\n", W, first, past, lane, (long long)at);
        std::exit(1);
      }
      ++seen;
    }
  }
  if (seen != (int64_t)past - first) {
    std::printf("W %d range [%d, %d): %lld arcs\n", W, first, past, (long long)seen);
    std::exit(1);
  }
}

int main() {
  for (int32_t past : {100, 2147483646, 2147483647})
    for (int32_t count : {0, 1, 3, 4, 15, 16, 17, 33, 64}) {
      check<4>(past - count, past);
      check<8>(past - count, past);
      check<16>(past - count, past);
    }
  std::puts("arc walk ok");
}
