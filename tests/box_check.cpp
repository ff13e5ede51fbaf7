// The rules of the shared-memory boxes (ibm_box.h), over every extent they meet.
#include <cstdio>

#include "ibm_box.h"

using namespace ibmk;

struct Tap { int b[3]; };

static int fail(const char *what, long a, long b, long c, long d) {
  std::printf("%s: %ld %ld %ld %ld\n", what, a, b, c, d);
  return 1;
}

int main() {
  // a block's shared memory: 227 KB, of which 2 KB for the kernels' own variables
  if ((BOX_MOST + SPREAD_PRE) * 4 + 2048 > 227 * 1024 || BOX_MOST % 4) return fail("limit", BOX_MOST, 0, 0, 0);
  // a box's taps lie in its cells
  for (int nx = 4; nx <= 60; ++nx)
    for (int ny = 4; ny <= 40; ny += 3)
      for (int nz = 4; nz <= 40; nz += 5)
        for (int x0 = -3; x0 <= 4; ++x0)
          for (int I = 512; I <= 514; I += 2) {
            const int bg[8] = {0, 0, x0, 7, 2, nx, ny, nz};
            const BoxLay B(bg, I);
            const Tap lo = {{x0, 7, 2}}, hi = {{x0 + nx - 1, 7 + ny - 1, 2 + nz - 1}};
            if (I % 4 == 0 && (B.pitch % 4 || (B.x0 - B.sh) % 4)) return fail("layout", nx, ny, nz, x0);
            if (B.off(lo, bg) < 0 || B.off(hi, bg) >= B.cells || B.off(hi, bg) % B.pitch < nx - 1)
              return fail("tap", nx, ny, nz, x0);
          }
  // spheres with shells of d cells: where the largest box in quads fits the
  // largest capacity, every box of theirs fits the capacity they get, and no
  // larger one is asked for than that box and a cell an axis take
  for (double d = 1.; d < 90.; d += 0.07)
    for (double ay = 0.5; ay < 2.1; ay += 0.5) {
      const double span[3] = {d, d * ay, d / ay};
      const int cap = box_capacity(span), e[3] = {(int)d + 4, (int)(d * ay) + 4, (int)(d / ay) + 4};
      if (cap < BOX_LEAST || cap > BOX_MOST || cap % 4) return fail("capacity", cap, 0, 0, 0);
      const bool fits = (e[0] + 6l) / 4 * 4 * e[1] * e[2] <= BOX_MOST;
      if (cap > std::max((long)BOX_LEAST, (e[0] + 7l) / 4 * 4 * (e[1] + 1) * (e[2] + 1))) return fail("large", cap, e[0], e[1], e[2]);
      for (int x0 = 0; x0 < 4; ++x0)
        for (int less = 0; less < 8 && fits; ++less) {
          const int bg[8] = {0, 0, x0, 0, 0, e[0] - (less & 1), e[1] - (less >> 1 & 1), e[2] - (less >> 2)};
          if (!BoxLay(bg, 512).ok(cap, 512, 512)) return fail("too small", bg[5], bg[6], bg[7], cap);
        }
    }
  std::printf("boxes ok\n");
  return 0;
}
