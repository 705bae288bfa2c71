// wavefront_pool (wavefront.h): the pool of a pass of n samples, by default and
// with a tuned size.
#include "host_cuda.h"

#include <cstdio>

#include "../../prender_gb300/csrc/wavefront.h"

using namespace pr;

int main() {
  int bad = 0;
  auto is = [&](unsigned int got, unsigned int want, const char* what) {
    if (got != want) printf("%s: %u, not %u\n", what, got, want);
    bad += got != want;
  };
  // the tuner's frames: twice the largest candidate in samples, every candidate as it is
  for (bool sss : {false, true})
    for (unsigned int tuned : {1u << 19, 1u << 20, 1u << 21, 1u << 22}) {
      is(wavefront_pool(2ull << 22, tuned, sss), tuned, "a candidate");
      is(wavefront_pool(64ull << 20, tuned, sss), tuned, "a tuned frame");
      is(wavefront_pool(1, tuned, sss), 8192, "one sample");
      is(wavefront_pool(3000000, tuned, sss), tuned < 3014656u ? tuned : 3014656u, "fewer samples than slots");
    }
  for (bool sss : {false, true}) {
    is(wavefront_pool(1, 0, sss), 8192, "one sample");
    is(wavefront_pool(8193, 0, sss), 16384, "two groups");
    is(wavefront_pool(1u << 19, 0, sss), 1u << 19, "all at once");
    is(wavefront_pool((1u << 19) + 1, 0, sss), 1u << 19, "the smallest share");
    is(wavefront_pool(3145728, 0, sss), sss ? 786432u : 1572864u, "a share");
    is(wavefront_pool(64ull << 20, 0, sss), sss ? kWfSpareSlots : kWfMaxSlots, "the largest");
  }
  return bad != 0;
}
