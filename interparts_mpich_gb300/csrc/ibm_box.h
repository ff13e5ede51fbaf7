// ibm_box.h -- the mixed form's shared-memory boxes: their layout and how much
// shared memory a context's boxes get.  Plain C++ apart from the qualifiers, so
// that a host program can check the rules (tests/box_check.cpp).
#pragma once
#include <algorithm>
#include <cmath>

#ifdef __CUDACC__
#define IBM_BOX_FN __host__ __device__ __forceinline__
#else
#define IBM_BOX_FN inline
#endif

namespace ibmk {

constexpr int SPREAD_PRE = 2048;  // points of a sphere whose values are staged beside its box
constexpr int BOX_LEAST = 8192;   // cells: 32 KB
constexpr int BOX_SOME = 40960;   // 160 KB
// 216 KB: what SPREAD_PRE values and the kernels' own variables leave of the 227
// KB a block may have
constexpr int BOX_MOST = 55296;

// A (particle, component) box from its record bg (k_ibm_box_geom): the copy in
// shared memory.  With I a multiple of 4 the rows hold the aligned quads of
// x-cells that cover them (a quad never straddles the periodic wrap), so that
// whole quads move; else the rows alone.
struct BoxLay {
  int x0, y0, z0, nbx, nby, nbz;  // first cell (x, y not wrapped) and extents
  int sh, pitch, cells;           // cells before x0 in a row, row length, size
  IBM_BOX_FN BoxLay(const int *bg, int I) {
    x0 = bg[0] + bg[2]; y0 = bg[1] + bg[3]; z0 = bg[4];
    nbx = bg[5]; nby = bg[6]; nbz = bg[7];
    const bool quads = (I & 3) == 0;
    sh = quads ? x0 & 3 : 0;
    pitch = quads ? (sh + nbx + 3) & ~3 : nbx;
    cells = pitch * nby * nbz;
  }
  // usable: fits cap and narrower than half the periodic domain (so relative
  // indices are unambiguous)
  IBM_BOX_FN bool ok(long cap, int I, int J) const {
    return nbx > 0 && (long)pitch * nby * nbz <= cap && nbx < I / 2 && nby < J / 2;
  }
  // offset of tap (0,0,0) of a point (make_cs origin, relative in x and y)
  template <typename S> IBM_BOX_FN int off(const S &s, const int *bg) const {
    return ((s.b[2] - bg[4]) * nby + (s.b[1] - bg[3])) * pitch + (s.b[0] - bg[2]) + sh;
  }
};

// Cells of shared memory for the boxes of a context whose largest sphere's shell
// is span[d] cells wide along axis d.  Its points' origins lie on at most
// floor(span) + 2 cells of an axis, their stencils on two more: where that box
// fits in quads, all do, and they get what the largest takes (a cell of room an
// axis).  A sphere that does not fit works on the field itself, tap by tap, and
// wants the L1 cache; smaller ones beside it get 160 KB.  A forcing loop at 256^3
// with spheres of 31 to 32 dx (343): 1516 us at 160 KB, where none of their boxes
// fits, 1022 so; of 12 to 40 (216): 807, with 216 KB 943.
inline int box_capacity(const double *span) {
  auto cells = [&](long more) {
    auto ext = [&](int d) { return (long)std::floor(span[d]) + more; };
    return (ext(0) + 3 + 3) / 4 * 4 * ext(1) * ext(2);
  };
  const long most = cells(4) <= BOX_MOST ? BOX_MOST : BOX_SOME;
  return (int)std::min(most, std::max((long)BOX_LEAST, cells(5)));
}

}  // namespace ibmk
