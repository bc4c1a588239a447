// Two host threads move data through the library's copy threads at once (two devices'
// transfers), each over its own buffers; exit status 1 when a byte is not the one sent.
#include <math.h>

#include "../../klft_b200/csrc/hostio.cu"

#include <cstdio>

int main() {
  constexpr size_t n = (3u << 20) + 40;
  int bad[2] = {0, 0};
  auto work = [&](int id) {
    std::vector<char> src(n), dst(n);
    std::vector<double> sq(40000);
    for (int round = 0; round < 400 && !bad[id]; ++round) {
      std::memset(src.data(), 1 + (id * 97 + round) % 250, n);
      std::memset(dst.data(), 0, n);
      klft::par_memcpy(dst.data(), src.data(), n, round & 1);
      bad[id] |= std::memcmp(dst.data(), src.data(), n) != 0;
      klft::par_range(sq.size(), [&](size_t a, size_t b) {
        for (size_t i = a; i < b; ++i) sq[i] = (double)(i + round) * (id + 1);
      });
      for (size_t i = 0; i < sq.size(); ++i) bad[id] |= sq[i] != (double)(i + round) * (id + 1);
    }
  };
  std::thread t0(work, 0), t1(work, 1);
  t0.join();
  t1.join();
  std::printf("%d %d\n", bad[0], bad[1]);
  return bad[0] || bad[1];
}
