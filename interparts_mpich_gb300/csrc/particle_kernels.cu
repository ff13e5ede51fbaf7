// particle_kernels.cu -- rigid-sphere side of the substep on one rank:
// intgr_over_sphere (intgr_over_sphere.f90:12-625), the collision /
// lubrication pass with its integer contact lists (intgr_nwtn_eulr.f90:326-605,
// collisions.f90:10-438), the Newton-Euler update (:607-667), sumrk3
// (:1586-1669), the periodic wrap and neighbour flags (:702-714, :1051-1090)
// and the new Lagrangian points (:1438-1485).
//
// Compiled without FMA contraction: these are few, sequential-per-particle
// operations whose roundings are kept equal to the reference so that the
// integer contact lists (firstc/qmax) come out identical.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"

namespace ibmk {

#define PF(f) b.pf[(long)(f) * np + p]
#define CFA(f, q) b.cf[((long)(f) * np + p) * nq + (q)]

// ---------------------------------------------------------------------------
// intgr_over_sphere.  One block per particle; the self-neighbour copies of a
// particle near the periodic edges integrate the wrapped part of the box
// (intgr_over_sphere.f90:84-112 and :298-313).  type 1 = volume, type 2 =
// integral of u (intu..), type 3 = integral of r x u (intomx..), type 23 =
// types 2 and 3 in one sweep (they read the same fields).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void copy_shift_sphere(int nbrecv, double lx, double ly, double &x, double &y) {
  switch (nbrecv) {
    case 1: x = x + lx; break;
    case 2: x = x + lx; y = y - ly; break;
    case 3: y = y - ly; break;
    case 4: x = x - lx; y = y - ly; break;
    case 5: x = x - lx; break;
    case 6: x = x - lx; y = y + ly; break;
    case 7: y = y + ly; break;
    case 8: x = x + lx; y = y + ly; break;
    default: break;
  }
}

// corner signed-distance fraction of a cell cut by the sphere surface
// (intgr_over_sphere.f90:357-374): sum of the positive signed distances over
// the sum of their magnitudes, corners in the reference's order
__device__ __forceinline__ double corner_fraction(double radius, double dxm2, double dxp2, double dym2, double dyp2,
                                                  double dzm2, double dzp2) {
  double sg[8];
  sg[0] = radius - sqrt(dxm2 + dym2 + dzm2);
  sg[1] = radius - sqrt(dxm2 + dyp2 + dzm2);
  sg[2] = radius - sqrt(dxp2 + dyp2 + dzm2);
  sg[3] = radius - sqrt(dxp2 + dym2 + dzm2);
  sg[4] = radius - sqrt(dxm2 + dym2 + dzp2);
  sg[5] = radius - sqrt(dxm2 + dyp2 + dzp2);
  sg[6] = radius - sqrt(dxp2 + dyp2 + dzp2);
  sg[7] = radius - sqrt(dxp2 + dym2 + dzp2);
  double sum1 = 0., sum2 = 0.;
  for (int cp = 0; cp < 8; ++cp) {
    if (sg[cp] > 0.) sum1 = sum1 + sg[cp];
    sum2 = sum2 + fabs(sg[cp]);
  }
  return sum1 / sum2;
}

// FP32 corner fraction (mixed form): the same expression in single
// precision, with the hardware's approximate square root and reciprocal
// (relative errors of a few 1e-7, below the FP32 rounding of the squared
// distances they act on); its decisions at the surface are continuous in
// the distances
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float corner_fraction_f(float radius, float dxm2, float dxp2, float dym2, float dyp2,
                                                  float dzm2, float dzp2) {
  float sg[8];
  sg[0] = radius - sqrt_approx(dxm2 + dym2 + dzm2);
  sg[1] = radius - sqrt_approx(dxm2 + dyp2 + dzm2);
  sg[2] = radius - sqrt_approx(dxp2 + dyp2 + dzm2);
  sg[3] = radius - sqrt_approx(dxp2 + dym2 + dzm2);
  sg[4] = radius - sqrt_approx(dxm2 + dym2 + dzp2);
  sg[5] = radius - sqrt_approx(dxm2 + dyp2 + dzp2);
  sg[6] = radius - sqrt_approx(dxp2 + dyp2 + dzp2);
  sg[7] = radius - sqrt_approx(dxp2 + dym2 + dzp2);
  float sum1 = 0.f, sum2 = 0.f;
#pragma unroll
  for (int cp = 0; cp < 8; ++cp) {
    sum1 += fmaxf(sg[cp], 0.f);
    sum2 += fabsf(sg[cp]);
  }
  return __fdividef(sum1, sum2);
}

// Sums of one velocity component over the cells of the sphere's box.  Block
// (p, comp, slice of the lines); a thread owns whole i-lines (fixed j, k), so
// the lever arms ry, rz of the torque are constant along its line and only
//   S0 = sum f*w,  Sx = sum rx*f*w
// accumulate per cell (error-free products and sums on the FP32 pipes).  w = 1
// for cells inside radin or with all corners inside, 0 with all corners
// outside, else the corner fraction, classified and evaluated in FP32 (the
// mixed forms).
// Bound by instruction issue, most of it the corner fractions: a warp pays for
// one wherever any of its lines is cut.  So the lines are ordered by their
// distance from the axis (bins of equal area): the 32 lines of a warp enter and
// leave the sphere together, and lines that miss it are left out.  The order
// within a bin is arbitrary, so the line sums go to shared memory and are added
// up in the order of the lines: the result does not depend on it.  FP64 is left
// to the box and the tables, an axis per lane and per warp, with conversions on
// the integer pipe.  1000 spheres of 16 dx: 122 -> 68 us, 94.7 -> 47.9 million
// instructions (lines in their own order, 256 threads, FP64 sums).
// Output: b.red[np + ((p*slices + slice)*3 + comp)*3 + {0,1,2}] = {S0, torque_a,
// torque_b} without the dVeul factor (k_sphere_final).
constexpr int SF_T = 128;    // threads
constexpr int SF_L = 512;    // lines ordered at a time
constexpr int SF_BINS = 64;
__global__ void __launch_bounds__(SF_T, 8) k_sphere_int(Geo g, PartGeo pg, PartBuffers b, const float *__restrict__ u,
                                                        const float *__restrict__ v, const float *__restrict__ w) {
  constexpr int AX = 128;
  const int np = pg.np;
  const int p = blockIdx.x, comp = blockIdx.y;
  const int ms = b.mslv[p];
  if (ms <= 0) return;
  __shared__ double s_c[3];
  __shared__ float s_thr[3];
  __shared__ int s_box[6];                // low and number of cells along each axis
  __shared__ float node[3][AX + 1];       // squared distances of the cell faces from the centre
  __shared__ float2 arm[3][AX];           // rx, ry, rz of the cell centres, FP32 pairs
  __shared__ int bin[SF_BINS + 1];        // lines in a bin, then its next free entry
  __shared__ unsigned short ord[SF_L];
  __shared__ float4 res[SF_L];            // line sums S0, Sx
  __shared__ float st[192];
  __shared__ double tot[3];
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const float *F = comp == 0 ? u : (comp == 1 ? v : w);
  const int *nbf = b.nb + (long)p * 9;
  // the three sums in double-float across the lines
  float A0h = 0.f, A0l = 0.f, TAh = 0.f, TAl = 0.f, TBh = 0.f, TBl = 0.f;
  // lever arms per component: ta += la * f*w, tb += lb * f*w with
  // comp 0: (rz, -ry), comp 1: (-rz, rx), comp 2: (ry, -rx)
  // copies nb = 0..8 (x/y images)
  for (int nb = 0; nb < 9; ++nb) {
    if (nb > 0 && nbf[nb] != 1) continue;
    __syncthreads();  // previous copy done with the tables and the box
    if (threadIdx.x < 3) {
      const int ax = threadIdx.x;
      int nbrecv = nb;
      if (nb > 0) { nbrecv = nb + 4; if (nbrecv > 8) nbrecv -= 8; }
      double cx = PF(PF_X), cy = PF(PF_Y);
      if (nb > 0) copy_shift_sphere(nbrecv, g.lx, g.ly, cx, cy);
      const double c = ax == 0 ? cx : (ax == 1 ? cy : PF(PF_Z));
      const double di = ax == 0 ? g.dxi : (ax == 1 ? g.dyi : g.dzi), rad = p_rad(pg, p);
      const int n = ax == 0 ? g.I : (ax == 1 ? g.J : g.K);
      const int low = max(fnint((c - rad) * di - 2.), 1), high = min(fnint((c + rad) * di + 2.), n);
      s_c[ax] = c;
      s_box[ax] = low;
      s_box[3 + ax] = high - low + 1;
      if (ax == 0) {
        const double radin = rad - 2. * g.dx;  // the particle's own radius when polydisperse
        s_thr[0] = (float)(radin * radin);
        s_thr[1] = (float)p_rthr(pg, p);
        s_thr[2] = (float)rad;
      }
    }
    __syncthreads();
    const int ilow = s_box[0], jlow = s_box[1], klow = s_box[2], ni = s_box[3], nj = s_box[4], nk = s_box[5];
    const float radin2f = s_thr[0], rthrf = s_thr[1], radiusf = s_thr[2];
    if (ni <= 0 || nj <= 0 || nk <= 0) continue;
    if (ni > AX || nj > AX || nk > AX) {  // sphere wider than the axis tables: flag, skip
      if (threadIdx.x == 0) atomicExch(&b.err[3], 1);
      continue;
    }
    // per-axis corner distances and cell-centre offsets, in the reference's
    // expressions (intgr_over_sphere.f90:335-508): warp ax forms those of axis ax
    if (wq < 3) {
      const double c = s_c[wq], d = wq == 0 ? g.dx : (wq == 1 ? g.dy : g.dz);
      const int low = s_box[wq], n = s_box[3 + wq];
      for (int t = lane; t <= n; t += 32) {
        const double xc = f2d_rn((float)(low + t) - 0.5f) * d;  // cell centre
        const double x = comp == wq ? xc : f2d_rn((float)(low + t - 1)) * d;
        const double q = x - c;
        float f;
        int rem;
        if (!d2f_int(q * q, f, rem)) f = 0.f;  // below 2^-126
        node[wq][t] = f;
        if (t < n) {
          float h, l;
          if (!d2df_int(xc - c, h, l)) h = l = 0.f;  // below 2^-74, far under the rounding of xc
          arm[wq][t] = make_float2(h, l);
        }
      }
    }
    const int nlines = nj * nk, per = (nlines + gridDim.z - 1) / gridDim.z;
    const int lbeg = blockIdx.z * per, lend = min(lbeg + per, nlines);
    const FastDiv rowdiv(nj);
    const float binscale = (float)SF_BINS / fmaxf(rthrf, radin2f);
    const long row0 = fidx(g, ilow - 1, 0, 0);
    for (int l0 = lbeg; l0 < lend; l0 += SF_L) {
      const int nl = min(SF_L, lend - l0);
      __syncthreads();  // tables in place, the last lines' sums read
      if (threadIdx.x <= SF_BINS) bin[threadIdx.x] = 0;
      __syncthreads();
      int mine[SF_L / SF_T];  // bins of the thread's lines, -1: misses the sphere
#pragma unroll
      for (int e = 0; e < SF_L / SF_T; ++e) {
        const int q = threadIdx.x + e * SF_T;
        mine[e] = -1;
        if (q < nl) {
          const int tk = rowdiv(l0 + q, nj), tj = l0 + q - tk * nj;
          const float ym = node[1][tj], yp = node[1][tj + 1], zm = node[2][tk], zp = node[2][tk + 1];
          const float ymin = fminf(ym, yp) + fminf(zm, zp);
          if (ymin < rthrf || yp + zp < radin2f) {
            mine[e] = min((int)(ymin * binscale), SF_BINS - 1);
            atomicAdd(&bin[mine[e]], 1);
          } else {
            res[q] = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      }
      __syncthreads();
      if (wq == 0) {  // first entries of the bins
        const int c0 = bin[2 * lane], c1 = bin[2 * lane + 1];
        int x = c0 + c1;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(~0u, x, o);
          if (lane >= o) x += y;
        }
        bin[2 * lane] = x - c0 - c1;
        bin[2 * lane + 1] = x - c1;
        if (lane == 31) bin[SF_BINS] = x;
      }
      __syncthreads();
#pragma unroll
      for (int e = 0; e < SF_L / SF_T; ++e)
        if (mine[e] >= 0) ord[atomicAdd(&bin[mine[e]], 1)] = (unsigned short)(threadIdx.x + e * SF_T);
      __syncthreads();
      const int nact = bin[SF_BINS];
      for (int a = threadIdx.x; a < nact; a += SF_T) {
        const int q = ord[a], tk = rowdiv(l0 + q, nj), tj = l0 + q - tk * nj;
        const float ym = node[1][tj], yp = node[1][tj + 1], zm = node[2][tk], zp = node[2][tk + 1];
        const float yzp = yp + zp;
        const float ymin = fminf(ym, yp) + fminf(zm, zp);
        const float ymax = fmaxf(ym, yp) + fmaxf(zm, zp);
        const float *Fl = F ? F + row0 + fidx(g, 0, jlow + tj - 1, klow + tk) : nullptr;
        // line sums: leading parts by error-free sums, their errors apart
        float s0 = 0.f, e0 = 0.f, sx = 0.f, ex = 0.f;
        float xm, xp = node[0][0];
        for (int ti = 0; ti < ni; ++ti) {
          xm = xp;
          xp = node[0][ti + 1];
          const bool in = xp + yzp < radin2f;
          if (!in && fminf(xm, xp) + ymin >= rthrf) continue;  // outside
          float ph = Fl ? Fl[ti] : 1.f, pe = 0.f;
          if (!in && !(fmaxf(xm, xp) + ymax < rthrf)) {
            const float wgt = corner_fraction_f(radiusf, xm, xp, ym, yp, zm, zp);
            two_prod(ph, wgt, ph, pe);
          }
          float s, e;
          two_sum(s0, ph, s, e);
          s0 = s;
          e0 += e + pe;
          if (comp != 0) {
            const float2 r = arm[0][ti];
            float qh, ql;
            two_prod(ph, r.x, qh, ql);
            ql = fmaf(ph, r.y, fmaf(pe, r.x, ql));
            two_sum(sx, qh, s, e);
            sx = s;
            ex += e + ql;
          }
        }
        float4 o;
        o.x = s0 + e0;
        o.y = e0 - (o.x - s0);
        o.z = sx + ex;
        o.w = ex - (o.z - sx);
        res[q] = o;
      }
      __syncthreads();
      // the line sums into the thread's double-float totals
      for (int q = threadIdx.x; q < nl; q += SF_T) {
        const float4 o = res[q];
        if (o.x == 0.f && o.z == 0.f) continue;
        const int tk = rowdiv(l0 + q, nj), tj = l0 + q - tk * nj;
        const float2 ry = arm[1][tj], rz = arm[2][tk];
        float qh, ql;
        df_add(A0h, A0l, o.x, o.y, A0h, A0l);
        if (comp == 0) {
          df_mul(o.x, o.y, rz.x, rz.y, qh, ql);
          df_add(TAh, TAl, qh, ql, TAh, TAl);
          df_mul(o.x, o.y, ry.x, ry.y, qh, ql);
          df_add(TBh, TBl, -qh, -ql, TBh, TBl);
        } else if (comp == 1) {
          df_mul(o.x, o.y, rz.x, rz.y, qh, ql);
          df_add(TAh, TAl, -qh, -ql, TAh, TAl);
          df_add(TBh, TBl, o.z, o.w, TBh, TBl);
        } else {
          df_mul(o.x, o.y, ry.x, ry.y, qh, ql);
          df_add(TAh, TAl, qh, ql, TAh, TAl);
          df_add(TBh, TBl, -o.z, -o.w, TBh, TBl);
        }
      }
    }
  }
  float h[3] = {A0h, TAh, TBh}, l[3] = {A0l, TAl, TBl};
  block_sum3_df2(h, l, st, tot);
  if (threadIdx.x < 3)
    b.red[np + (((long)p * gridDim.z + blockIdx.z) * 3 + comp) * 3 + threadIdx.x] = tot[threadIdx.x];
}

// The plain form of the same sums, FP64.  Bound by FP64 issue, most of it the
// square roots of the cut cells' corner distances: each corner belongs to up
// to eight cells, so the signed distances R - |x - c| are formed once per grid
// node (in the reference's expression, only within a cell diagonal of the
// surface, compacted into full warps) and a cut cell reads its eight from
// shared memory.  Classification as in the mixed form, by FP32 screening of
// the squared corner distances with a relative margin (1e-5) far above its
// rounding; a cell that the screen leaves open is evaluated, which gives
// exactly 1 or 0 where all its corners lie on one side.
// A block takes the planes of slice blockIdx.z of the box, a slab of nodes at a
// time (ncap doubles of shared memory, small enough for five blocks an SM: the
// phases of one overlap the others'; a sphere too wide for two node planes
// forms its corner distances cell by cell).  1000 spheres of 16 dx: 1063 ->
// 542 us (a warp per row of cells in place of a thread per line: 682), 519 with
// the set-up spread over lanes and warps; one sphere 82 -> 27 us.
constexpr int SI_T = 128, SI_AX = 128, SI_QCAP = 1024, SI_NODES = 16384;
__global__ void __launch_bounds__(SI_T, 5) k_sphere_int_d(Geo g, PartGeo pg, PartBuffers b, const double *__restrict__ u,
                                                      const double *__restrict__ v, const double *__restrict__ w,
                                                      int ncap) {
  // [ncap] signed distances, then the node queue of ncap / 2 entries
  extern __shared__ __align__(16) double s_node[];
  int *nqueue = reinterpret_cast<int *>(s_node + ncap);
  const int np = pg.np, p = blockIdx.x, comp = blockIdx.y, nsl = gridDim.z;
  if (b.mslv[p] <= 0) return;
  __shared__ double s_c[3], s_rad, s_radin2, s_rthr;
  __shared__ float s_thr[5];
  __shared__ int s_box[6];  // ilow, ni, jlow, nj, klow, nk
  __shared__ double sx2[SI_AX + 1], sy2[SI_AX + 1], sz2[SI_AX + 1], srx[SI_AX], sry[SI_AX], srz[SI_AX];
  __shared__ float fx[SI_AX + 1], fy[SI_AX + 1], fz[SI_AX + 1];
  __shared__ int queue[SI_QCAP];
  __shared__ int qn, nn;
  __shared__ double red[3][SI_T / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    const double rad = p_rad(pg, p), rth = p_rthr(pg, p);  // the particle's own when polydisperse
    const double radin = rad - 2. * g.dx, diag = 1.001 * sqrt(g.dx * g.dx + g.dy * g.dy + g.dz * g.dz);
    const double lo = rad > diag ? rad - diag : 0.;
    s_rad = rad;
    s_rthr = rth;
    s_radin2 = radin * radin;
    s_thr[0] = (float)(s_radin2 * (1. + 1e-5));
    s_thr[1] = (float)(rth * (1. - 1e-5));
    s_thr[2] = (float)(rth * (1. + 1e-5));
    s_thr[3] = (float)(lo * lo * (1. - 1e-5));
    s_thr[4] = (float)((rad + diag) * (rad + diag) * (1. + 1e-5));
  }
  __syncthreads();
  const double radius = s_rad, radin2 = s_radin2, rthr = s_rthr, dx = g.dx, dy = g.dy, dz = g.dz;
  const float radin2_hi = s_thr[0], rthr_lo = s_thr[1], rthr_hi = s_thr[2], band_lo = s_thr[3], band_hi = s_thr[4];
  // below the margin of radin^2 (a radius under two cells: radin2 is of the
  // wrong side, but so it is in the reference's test)
  const float radin2_lo = (float)(radin2 * (1. - 1e-5));
  const double *F = comp == 0 ? u : (comp == 1 ? v : w);
  const int *nbf = b.nb + (long)p * 9;
  // ta += la f w, tb += lb f w with comp 0: (rz, -ry), 1: (-rz, rx), 2: (ry, -rx)
  double a0 = 0., ta = 0., tb = 0.;
  const int nzs = pg.zper ? 3 : 1;  // periodic z: each copy also at z -+ lz
  for (int nbz = 0; nbz < 9 * nzs; ++nbz) {
    const int nb = nbz / nzs, zs = nbz - nb * nzs;
    if (nb > 0 && nbf[nb] != 1) continue;
    __syncthreads();  // previous copy done with the tables and the box
    if (threadIdx.x < 3) {  // an axis each: in one thread's chain the set-up of one sphere took 31 us, so 27
      const int ax = threadIdx.x;
      int nbrecv = nb;
      if (nb > 0) { nbrecv = nb + 4; if (nbrecv > 8) nbrecv -= 8; }
      double cx = PF(PF_X), cy = PF(PF_Y);
      const double cz = PF(PF_Z) + (zs == 1 ? -pg.lz : (zs == 2 ? pg.lz : 0.));
      if (nb > 0) copy_shift_sphere(nbrecv, g.lx, g.ly, cx, cy);
      const double c = ax == 0 ? cx : (ax == 1 ? cy : cz), di = ax == 0 ? g.dxi : (ax == 1 ? g.dyi : g.dzi);
      const int low = max(fnint((c - radius) * di - 2.), 1);
      const int high = min(fnint((c + radius) * di + 2.), ax == 0 ? g.I : (ax == 1 ? g.J : g.K));
      s_c[ax] = c;
      s_box[2 * ax] = low;
      s_box[2 * ax + 1] = high - low + 1;
    }
    __syncthreads();
    const int ilow = s_box[0], ni = s_box[1], jlow = s_box[2], nj = s_box[3], klow = s_box[4], nk = s_box[5];
    if (ni <= 0 || nj <= 0 || nk <= 0) continue;
    if (ni > SI_AX || nj > SI_AX || nk > SI_AX) {  // sphere wider than the axis tables: flag, skip
      if (threadIdx.x == 0) atomicExch(&b.err[3], 1);
      continue;
    }
    // squared distances of the node planes and cell-centre offsets, in the
    // reference's expressions (intgr_over_sphere.f90:335-508); a cell's upper
    // face and the next one's lower face have the same expression's value
    // (warp ax those of axis ax)
    if (wid < 3) {
      const double c = s_c[wid], d = wid == 0 ? dx : (wid == 1 ? dy : dz);
      const int low = s_box[2 * wid], n = s_box[2 * wid + 1];
      double *x2 = wid == 0 ? sx2 : (wid == 1 ? sy2 : sz2), *rc = wid == 0 ? srx : (wid == 1 ? sry : srz);
      float *f2 = wid == 0 ? fx : (wid == 1 ? fy : fz);
      for (int t = lane; t <= n; t += 32) {
        const double xc = f2d_rn((float)(low + t) - 0.5f) * d;  // cell centre
        const double q = (comp == wid ? xc : f2d_rn((float)(low + t - 1)) * d) - c;
        x2[t] = q * q;
        f2[t] = (float)x2[t];
        if (t < n) rc[t] = xc - c;
      }
    }
    const int per = (nk + nsl - 1) / nsl, z0 = blockIdx.z * per, z1 = min(nk, z0 + per);
    const int ex = ni + 1, ep = ex * (nj + 1);  // nodes of a row, of a plane
    const int ring = ncap / ep;                 // node planes held, in turn
    const bool nodes = ring >= 2;
    const int slab = nodes ? ring - 1 : nk;
    const long row0 = fidx(g, ilow - 1, 0, 0);
    auto direct = [&](int ti, int tj, int tk) {  // corner fraction without the node table
      if (sx2[ti + 1] + sy2[tj + 1] + sz2[tk + 1] < radin2) return 1.;
      const double mind2 = fmin(sx2[ti], sx2[ti + 1]) + fmin(sy2[tj], sy2[tj + 1]) + fmin(sz2[tk], sz2[tk + 1]);
      if (mind2 >= rthr) return 0.;
      return corner_fraction(radius, sx2[ti], sx2[ti + 1], sy2[tj], sy2[tj + 1], sz2[tk], sz2[tk + 1]);
    };
    int slot0 = 0;  // slot of plane zb (a slab is a plane short of the ring)
    for (int zb = z0; zb < z1; zb += slab, slot0 = slot0 ? slot0 - 1 : ring - 1) {
      const int ze = min(z1, zb + slab);  // cell planes zb..ze-1, node planes zb..ze
      auto node = [&](int ti, int tj, int tk) -> double & {
        int q = slot0 + tk - zb;
        if (q >= ring) q -= ring;
        return s_node[q * ep + tj * ex + ti];
      };
      if (threadIdx.x == 0) { qn = 0; nn = 0; }
      __syncthreads();
      if (nodes) {
        // the nodes within a diagonal of the surface, a warp a row (plane zb
        // is the last slab's uppermost)
        for (int t0 = 0; t0 < ex; t0 += 32) {
          const int ti = t0 + lane;
          const float xf = ti < ex ? fx[ti] : 4.f * band_hi;
          for (int tk = zb == z0 ? zb : zb + 1; tk <= ze; ++tk) {
            const float zf = fz[tk];
            for (int tj = wid; tj <= nj; tj += SI_T / 32) {
              const float d2 = fy[tj] + zf + xf;
              const bool near = d2 >= band_lo && d2 <= band_hi;
              const unsigned m = __ballot_sync(0xffffffffu, near);
              if (!m) continue;
              int at = 0;
              if (lane == 0) at = atomicAdd(&nn, __popc(m));
              at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
              if (near) {
                if (at < ncap / 2) nqueue[at] = ti | (tj << 8) | (tk << 16);
                else node(ti, tj, tk) = radius - sqrt_newton(sx2[ti] + sy2[tj] + sz2[tk]);
              }
            }
          }
        }
      }
      // cells surely inside, a thread a line (fixed j, k: opposite lever arms
      // rx cancel within its sum, the others come in once); the open ones go
      // to the queue
      const int nlines = nj * (ze - zb);
      for (int L = threadIdx.x; L < nlines; L += SI_T) {
        const int lk = L / nj, tj = L - lk * nj, tk = zb + lk;
        const float ymin = fminf(fy[tj], fy[tj + 1]) + fminf(fz[tk], fz[tk + 1]);
        const float ymax = fmaxf(fy[tj], fy[tj + 1]) + fmaxf(fz[tk], fz[tk + 1]);
        const float yzp = fy[tj + 1] + fz[tk + 1];
        const double *f = F ? F + row0 + fidx(g, 0, jlow + tj - 1, klow + tk) : nullptr;
        double s0 = 0., sx = 0.;
        float xm, xp = fx[0];
        for (int ti = 0; ti < ni; ++ti) {
          xm = xp;
          xp = fx[ti + 1];
          const float d2 = xp + yzp;
          if (!(d2 <= radin2_hi) && fminf(xm, xp) + ymin > rthr_hi) continue;  // outside
          double fv;
          if (d2 < radin2_lo || fmaxf(xm, xp) + ymax < rthr_lo) {
            fv = f ? f[ti] : 1.;
          } else {
            const int q = atomicAdd(&qn, 1);
            if (q < SI_QCAP) {
              queue[q] = ti | (tj << 8) | (tk << 16) | (d2 <= radin2_hi ? 1 << 24 : 0);
              continue;
            }
            fv = (f ? f[ti] : 1.) * direct(ti, tj, tk);  // queue full
          }
          s0 += fv;
          if (comp != 0) sx = fma(srx[ti], fv, sx);
        }
        a0 += s0;
        if (comp == 0) { ta = fma(srz[tk], s0, ta); tb = fma(-sry[tj], s0, tb); }
        else if (comp == 1) { ta = fma(-srz[tk], s0, ta); tb += sx; }
        else { ta = fma(sry[tj], s0, ta); tb -= sx; }
      }
      __syncthreads();
      const int nnode = min(nn, ncap / 2);
      for (int q = threadIdx.x; q < nnode; q += SI_T) {
        const int e = nqueue[q], ti = e & 0xff, tj = (e >> 8) & 0xff, tk = e >> 16;
        node(ti, tj, tk) = radius - sqrt_newton(sx2[ti] + sy2[tj] + sz2[tk]);
      }
      __syncthreads();
      const int nq = min(qn, SI_QCAP);
      for (int q = threadIdx.x; q < nq; q += SI_T) {
        const int e = queue[q], ti = e & 0xff, tj = (e >> 8) & 0xff, tk = (e >> 16) & 0xff;
        const double fv = F ? F[row0 + fidx(g, ti, jlow + tj - 1, klow + tk)] : 1.;
        double frac;
        if (!nodes || (e >> 24)) {  // (or within the margin of radin^2)
          frac = direct(ti, tj, tk);
        } else {
          // positive part over magnitude, (S + A) / 2A: S = A inside, -A outside
          const double *n0 = &node(ti, tj, tk), *n1 = &node(ti, tj, tk + 1);
          const double c0 = n0[0], c1 = n0[1], c2 = n0[ex], c3 = n0[ex + 1], c4 = n1[0], c5 = n1[1], c6 = n1[ex],
                       c7 = n1[ex + 1];
          const double S = ((c0 + c1) + (c2 + c3)) + ((c4 + c5) + (c6 + c7));
          const double A = ((fabs(c0) + fabs(c1)) + (fabs(c2) + fabs(c3))) + ((fabs(c4) + fabs(c5)) + (fabs(c6) + fabs(c7)));
          frac = div_newton(0.5 * (S + A), A);
        }
        const double fw = fv * frac;
        const double rx = srx[ti], ry = sry[tj], rz = srz[tk];
        a0 += fw;
        if (comp == 0) { ta = fma(rz, fw, ta); tb = fma(-ry, fw, tb); }
        else if (comp == 1) { ta = fma(-rz, fw, ta); tb = fma(rx, fw, tb); }
        else { ta = fma(ry, fw, ta); tb = fma(-rx, fw, tb); }
      }
      __syncthreads();
    }
  }
  double s3[3] = {a0, ta, tb};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s3[q] += __shfl_down_sync(0xffffffffu, s3[q], d);
    if (lane == 0) red[q][wid] = s3[q];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double x = 0.;
    for (int q = 0; q < SI_T / 32; ++q) x += red[threadIdx.x][q];
    b.red[np + (((long)p * nsl + blockIdx.z) * 3 + comp) * 3 + threadIdx.x] = x;
  }
}

// Totals of the sphere integrals, a warp per particle; nsl: slices per
// (particle, component), summed in order.  With substep set it is the step
// into Newton-Euler as well: the state of the last substep is saved (new ->
// old, intgr_nwtn_eulr.f90:77-118; the integrals are the only part of it that
// changes before the collision pass) and the first collision iteration's
// snapshot taken, two launches fewer.
__device__ __forceinline__ void snapshot_particle(const PartGeo &pg, PartBuffers &b, int p, int iter, int lane);
__global__ void __launch_bounds__(128) k_sphere_final(PartGeo pg, PartBuffers b, int type, int substep, int nsl) {
  const int np = pg.np, nq = pg.nq;
  const int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (p >= np) return;
  const int ms = b.mslv[p];
  if (substep) {
    if (ms > 0) {
      for (int f = PF_X + lane; f <= PF_COLTZ; f += 32) PF(f + (PF_OX - PF_X)) = PF(f);
      for (int e = lane; e < (CF_DWT - CF_DX + 1) * nq; e += 32) {
        const int f = CF_DX + e / nq, q = e % nq;
        CFA(f + (CF_ODX - CF_DX), q) = CFA(f, q);
      }
    }
    snapshot_particle(pg, b, p, 0, lane);
    __syncwarp();
  }
  if (ms == 0) return;
  const double dV = pg.dVeul;
  double s = 0.;  // lane 3 c + q: quantity q = S0, ta, tb of component c
  if (ms > 0 && lane < 9) {
    const double *part = b.red + np + (long)p * 9 * nsl + lane;
    s = part[0];
    for (int z = 1; z < nsl; ++z) s += part[9 * z];
  }
  // lanes 0..2: the linear integral of component c and the torque component c
  const int c = lane < 3 ? lane : 0;
  const double A = __shfl_sync(0xffffffffu, s, 3 * c);
  // torques: (1, ta) + (2, ta), (0, ta) + (2, tb), (0, tb) + (1, tb)
  const double ta = __shfl_sync(0xffffffffu, s, c == 0 ? 4 : (c == 1 ? 1 : 2));
  const double tb = __shfl_sync(0xffffffffu, s, c == 0 ? 7 : (c == 1 ? 8 : 5));
  if (lane >= 3) return;
  if (type == 1 && lane == 0) b.red[p] = A * dV;  // volume of the u-cells (intgr_over_sphere.f90:607-622)
  if (type == 1 || type == 2 || type == 23) PF(PF_INTU + c) = A * dV;
  if (type == 3 || type == 23) PF(PF_INTOMX + c) = (ta + tb) * dV;
}

template <typename T>
void launch_sphere_integrals(cudaStream_t s, const Geo &g, const PartGeo &pg, PartBuffers b, const T *u, const T *v,
                             const T *w, int type, bool substep) {
  if (pg.np == 0) return;
  const bool unit = type == 1;  // volume: integrate w = 1 (F == nullptr)
  u = unit ? nullptr : u; v = unit ? nullptr : v; w = unit ? nullptr : w;
  // few particles: several blocks share a (particle, component)
  const int nsl = sphere_slices(pg.np);
  const dim3 grid(pg.np, 3, nsl);
  if constexpr (sizeof(T) == 4) {
    k_sphere_int<<<grid, SF_T, 0, s>>>(g, pg, b, u, v, w);
  } else {
    // nodes of the largest sphere's box: a slab of up to 24 KB (five blocks an
    // SM), two planes at least (up to 128 KB)
    const long ep = (long)(std::ceil(2. * pg.rmax * g.dxi) + 7.) * (long)(std::ceil(2. * pg.rmax * g.dyi) + 7.);
    const int ncap = (int)(2 * ep <= 3072 ? 3072 : (2 * ep <= SI_NODES ? 2 * ep : 0));
    k_sphere_int_d<<<grid, SI_T, (size_t)ncap * (sizeof(double) + 2), s>>>(g, pg, b, u, v, w, ncap);
  }
  k_sphere_final<<<(pg.np + 3) / 4, 128, 0, s>>>(pg, b, type, substep ? 1 : 0, nsl);
}
int sphere_set_smem_limits() {
  return cudaFuncSetAttribute(k_sphere_int_d, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              SI_NODES * (int)(sizeof(double) + 2)) == cudaSuccess ? 0 : -1;
}
template void launch_sphere_integrals<double>(cudaStream_t, const Geo &, const PartGeo &, PartBuffers,
                                              const double *, const double *, const double *, int, bool);
template void launch_sphere_integrals<float>(cudaStream_t, const Geo &, const PartGeo &, PartBuffers, const float *,
                                             const float *, const float *, int, bool);

// ---------------------------------------------------------------------------
// collisions / lubrication (collisions.f90).  Only the normal contact force
// and the normal lubrication force are applied (collisions.f90:199-205,
// 430-432); the tangential history is still evolved and stored.
// ---------------------------------------------------------------------------
// the scalar normal lubrication force f1 of lubrication (collisions.f90:222-438)
__device__ __noinline__ double d_lub_f1(const PartGeo &pg, double pu, double pv, double pw, int idq, double nx, double ny,
                           double nz, double eps, double u_nb, double v_nb, double w_nb, double coeff_f) {
  const double u1a = pu * nx + pv * ny + pw * nz;
  const double u1b = u_nb * nx + v_nb * ny + w_nb * nz;
  double f1;
  if (idq > pg.np) {
    double a11;
    if (eps < 0.001) a11 = pg.a11_sat_pw;
    else a11 = -(1. / eps) + 1. / 5. * log(eps) + 1. / 21. * eps * log(eps) - .9713;
    f1 = (a11 * u1a);
    f1 = coeff_f * (f1 - (pg.a11_ini_pw * u1a));
  } else {
    double a11a, a11b;
    if (eps < 0.001) { a11a = pg.a11a_sat_pp; a11b = pg.a11b_sat_pp; }
    else {
      const double a11 = -(1. / 4. * pow(eps, -1.)) + 9. / 40. * log(eps) + 3. / 112. * eps * log(eps);
      a11a = a11 - .995;
      a11b = -a11 + .350;
    }
    f1 = (a11a * u1a + a11b * u1b);
    f1 = coeff_f * (f1 - (pg.a11a_ini_pp * u1a + pg.a11b_ini_pp * u1b));
  }
  return f1;
}
__device__ void d_lubrication(const PartGeo &pg, double pu, double pv, double pw, int idq, double nx, double ny,
                              double nz, double eps, double u_nb, double v_nb, double w_nb, double coeff_f,
                              double &cfx, double &cfy, double &cfz) {
  const double f1 = d_lub_f1(pg, pu, pv, pw, idq, nx, ny, nz, eps, u_nb, v_nb, w_nb, coeff_f);
  cfx = cfx + f1 * nx;
  cfy = cfy + f1 * ny;
  cfz = cfz + f1 * nz;
}

// Polydisperse pair constants (init.f90:137-241 with the pair's effective
// mass ratiorho vp vq / (vp + vq), or ratiorho vp for a wall, and the
// lubrication prefactor 6 pi nu Re of the equivalent radius Re), as the
// oracle's pair_consts forms them
struct PairC {
  double kn, kt, etan, etat, muc, coeff_f;
};
__device__ PairC pair_consts(const PartGeo &pg, double vp, double vq, double re) {
  const double me = vq > 0. ? pg.ratiorho * vp * vq / (vp + vq) : pg.ratiorho * vp, mt = 2. / 7. * me;
  PairC k;
  k.kn = pg.pc_an * me / pg.pc_b;
  k.kt = pg.pc_at * mt / pg.pc_b;
  k.etan = pg.pc_en * me / pg.pc_ndt;
  k.etat = pg.pc_et * mt / pg.pc_ndt;
  k.muc = 0.;
  k.coeff_f = 6. * IBM_PI * pg.visc * re;
  return k;
}

struct PState {  // the particle's own state held in registers by the collision thread
  double u, v, w, omx, omy, omz, colfx, colfy, colfz;
};

__device__ __noinline__ void d_collisions(const PartGeo &pg, PartBuffers &b, int p, PState &S, int qq, int idq, double dist,
                             double deltax, double deltay, double deltaz, double u_nb, double v_nb, double w_nb,
                             double omx_nb, double omy_nb, double omz_nb, double dtsub, double rkab) {
  const int np = pg.np, nq = pg.nq;
  const double radius = p_rad(pg, p);
  // polydisperse: the partner's radius in its own rotation term (a wall: 0)
  const double rq = pg.poly ? (idq <= np ? pg.prad[idq - 1] : 0.) : radius;
  const double nx = deltax / dist, ny = deltay / dist, nz = deltaz / dist;
  double deltan, kn, etan, kt, etat, muc;
  if (pg.poly) {
    const bool wall = idq > np;
    const PairC k = pair_consts(pg, pg.pvol[p], wall ? 0. : pg.pvol[idq - 1], radius);
    deltan = (wall ? radius : radius + rq) - dist;
    kn = k.kn; kt = k.kt; etan = k.etan; etat = k.etat; muc = k.muc;
  } else if (idq <= np) {
    deltan = 2 * radius - dist; kn = pg.kn_ss; kt = pg.kt_ss; etan = pg.etan_ss; etat = pg.etat_ss; muc = pg.muc_ss;
  } else {
    deltan = radius - dist; kn = pg.kn_sw; kt = pg.kt_sw; etan = pg.etan_sw; etat = pg.etat_sw; muc = pg.muc_sw;
  }
  const double dun = (S.u + (S.omy * radius * nz) - (S.omz * radius * ny)) -
                     (u_nb + (omy_nb * rq * (-nz)) - (omz_nb * rq * (-ny)));
  const double dvn = (S.v - (S.omx * radius * nz) + (S.omz * radius * nx)) -
                     (v_nb - (omx_nb * rq * (-nz)) + (omz_nb * rq * (-nx)));
  const double dwn = (S.w + (S.omx * radius * ny) - (S.omy * radius * nx)) -
                     (w_nb + (omx_nb * rq * (-ny)) - (omy_nb * rq * (-nx)));
  const double vabs = dun * nx + dvn * ny + dwn * nz;
  const double fxn = -(kn * (deltan * nx)) - etan * (vabs * nx);
  const double fyn = -(kn * (deltan * ny)) - etan * (vabs * ny);
  const double fzn = -(kn * (deltan * nz)) - etan * (vabs * nz);
  const double dut = dun - vabs * nx, dvt = dvn - vabs * ny, dwt = dwn - vabs * nz;
  const double vtabs = sqrt(dut * dut + dvt * dvt + dwt * dwt);
  const int q = qq - 1;
  const double odx = CFA(CF_ODX, q), ody = CFA(CF_ODY, q), odz = CFA(CF_ODZ, q);
  const double distold = sqrt(odx * odx + ody * ody + odz * odz);
  double nxold, nyold, nzold;
  if (distold == 0) { nxold = nx; nyold = ny; nzold = nz; }
  else { nxold = odx / distold; nyold = ody / distold; nzold = odz / distold; }
  double dxt, dyt, dzt;
  if (b.firstc[(long)p * nq + q] == idq) {
    double hx = ny * nzold - nyold * nz;
    double hy = nz * nxold - nzold * nx;
    double hz = nx * nyold - nxold * ny;
    const double aa = sqrt(hx * hx + hy * hy + hz * hz);
    const double cc = cos(asin(aa));
    const double bb = 1. - cc;
    if (aa == 0.) { hx = 0.; hy = 0.; hz = 0.; }
    else { hx = hx / aa; hy = hy / aa; hz = hz / aa; }
    const double h11 = bb * (hx * hx) + cc, h12 = bb * hx * hy - aa * hz, h13 = bb * hx * hz + aa * hy;
    const double h21 = bb * hx * hy + aa * hz, h22 = bb * (hy * hy) + cc, h23 = bb * hy * hz - aa * hx;
    const double h31 = bb * hx * hz - aa * hy, h32 = bb * hy * hz + aa * hx, h33 = bb * (hz * hz) + cc;
    const double oxt = CFA(CF_ODXT, q), oyt = CFA(CF_ODYT, q), ozt = CFA(CF_ODZT, q);
    const double out_ = CFA(CF_ODUT, q), ovt = CFA(CF_ODVT, q), owt = CFA(CF_ODWT, q);
    dxt = oxt * h11 + oyt * h21 + ozt * h31 + 0.5 * dtsub * rkab * (dut + out_ * h11 + ovt * h21 + owt * h31);
    dyt = oxt * h12 + oyt * h22 + ozt * h32 + 0.5 * dtsub * rkab * (dvt + out_ * h12 + ovt * h22 + owt * h32);
    dzt = oxt * h13 + oyt * h23 + ozt * h33 + 0.5 * dtsub * rkab * (dwt + out_ * h13 + ovt * h23 + owt * h33);
  } else {
    CFA(CF_PSI, q) = vtabs / fabs(vabs);
    dxt = 0.; dyt = 0.; dzt = 0.;
  }
  double fxt = -(kt * dxt) - (etat * dut);
  double fyt = -(kt * dyt) - (etat * dvt);
  double fzt = -(kt * dzt) - (etat * dwt);
  const double fnabs = sqrt(fxn * fxn + fyn * fyn + fzn * fzn);
  double ftabs = sqrt(fxt * fxt + fyt * fyt + fzt * fzt);
  const double tx = -fxt / ftabs, ty = -fyt / ftabs, tz = -fzt / ftabs;
  if (!(ftabs <= muc * fnabs)) {
    dxt = muc * fnabs * tx / kt;
    dyt = muc * fnabs * ty / kt;
    dzt = muc * fnabs * tz / kt;
  }
  S.colfx = S.colfx + fxn;
  S.colfy = S.colfy + fyn;
  S.colfz = S.colfz + fzn;
  CFA(CF_DX, q) = deltax; CFA(CF_DY, q) = deltay; CFA(CF_DZ, q) = deltaz;
  CFA(CF_DXT, q) = dxt; CFA(CF_DYT, q) = dyt; CFA(CF_DZT, q) = dzt;
  CFA(CF_DUT, q) = dut; CFA(CF_DVT, q) = dvt; CFA(CF_DWT, q) = dwt;
}

__device__ __noinline__ void d_remove_contact(const PartGeo &pg, PartBuffers &b, int p, int i, int &qlast) {
  const int np = pg.np, nq = pg.nq;
  const int a = i - 1, l = qlast - 1;
  int *fc = b.firstc + (long)p * nq, *ofc = b.ofirstc + (long)p * nq;
  if (qlast > 1) {
    fc[a] = fc[l];
    for (int f : {CF_DXT, CF_DYT, CF_DZT, CF_DUT, CF_DVT, CF_DWT}) CFA(f, a) = CFA(f, l);
    ofc[a] = ofc[l];
    for (int f : {CF_ODXT, CF_ODYT, CF_ODZT, CF_ODUT, CF_ODVT, CF_ODWT}) CFA(f, a) = CFA(f, l);
  }
  fc[l] = 0;
  ofc[l] = 0;
  for (int f = CF_DX; f <= CF_DWT; ++f) CFA(f, l) = 0.;
  for (int f = CF_ODX; f <= CF_ODWT; ++f) CFA(f, l) = 0.;
  qlast = qlast - 1;
}
__device__ void d_new_contact(const PartGeo &pg, PartBuffers &b, int p, int slot) {
  const int np = pg.np, nq = pg.nq;
  const int s = slot - 1;
  for (int f = CF_DX; f <= CF_DWT; ++f) CFA(f, s) = 0.;
  for (int f = CF_ODX; f <= CF_ODWT; ++f) CFA(f, s) = 0.;
}

// position of particle copy nb in the collision loop on one rank
// (intgr_nwtn_eulr.f90:223-322, coords=(0,0), dims=(1,1))
__device__ __forceinline__ void copy_shift_coll(int nb, double lx, double ly, double &x, double &y) {
  const double boundleftnb = lx, boundrightnb = 0., boundbacknb = 0., boundfrontnb = ly;
  switch (nb) {
    case 1: if (x < boundleftnb) x = x + lx; break;
    case 2: if (x < boundleftnb) x = x + lx; if (y > boundbacknb) y = y - ly; break;
    case 3: if (y > boundbacknb) y = y - ly; break;
    case 4: if (x > boundrightnb) x = x - lx; if (y > boundbacknb) y = y - ly; break;
    case 5: if (x > boundrightnb) x = x - lx; break;
    case 6: if (x > boundrightnb) x = x - lx; if (y < boundfrontnb) y = y + ly; break;
    case 7: if (y < boundfrontnb) y = y + ly; break;
    case 8: if (x < boundleftnb) x = x + lx; if (y < boundfrontnb) y = y + ly; break;
    default: break;
  }
}
__device__ __forceinline__ double minimg(double a0, double a1, double a2) {
  double m = a0;
  if (fabs(a1) < fabs(m)) m = a1;
  if (fabs(a2) < fabs(m)) m = a2;
  return m;
}

#define COLL_WARPS 4
#define COLL_CAP 64

// snapshot of collision iteration iter (anb(:,0), intgr_nwtn_eulr.f90:153-206),
// a warp per particle.  Each iteration has its own, so that one iteration's
// update can take the next one's while others still read.
__device__ __forceinline__ void snapshot_particle(const PartGeo &pg, PartBuffers &b, int p, int iter, int lane) {
  const int np = pg.np;
  const bool m = b.mslv[p] > 0;
  double v = 0.;
  if (lane < 9) {
    const int f = lane < 3 ? PF_X + lane : (lane < 6 ? PF_U + lane - 3 : PF_OMX + lane - 6);
    v = m ? PF(f) : 0.;
    PF(PF_SX + 9 * iter + lane) = v;
  }
  // FP32 copy of the positions for the candidate filter (w: master flag)
  const float x = (float)v, y = __shfl_sync(0xffffffffu, x, 1), z = __shfl_sync(0xffffffffu, x, 2);
  if (lane == 0) b.pos4[(long)iter * np + p] = make_float4(x, y, z, m ? 1.f : 0.f);
}

// Uniform cell list of the snapshot positions (one block): cell of every
// particle, counts, exclusive scan, scatter, then every cell's items sorted
// ascending.  Cells are at least 1.01 x the filter distance wide, so every
// partner the FP32 filter accepts lies in the 27 cells around the particle's
// own (periodic in x and y, clamped in z).
__device__ __forceinline__ int coll_cell(const PartGeo &pg, float4 x) {
  int cx = (int)floorf(x.x * pg.cix), cy = (int)floorf(x.y * pg.ciy), cz = (int)floorf(x.z * pg.ciz);
  cx = ((cx % pg.ncx) + pg.ncx) % pg.ncx;
  cy = ((cy % pg.ncy) + pg.ncy) % pg.ncy;
  cz = min(max(cz, 0), pg.ncz - 1);
  return (cz * pg.ncy + cy) * pg.ncx + cx;
}
__global__ void __launch_bounds__(1024) k_cell_build(PartGeo pg, PartBuffers b, int iter) {
  b.pos4 += (long)iter * pg.np;
  const int np = pg.np, ncell = pg.ncx * pg.ncy * pg.ncz, tid = threadIdx.x;
  __shared__ int part[1024];
  for (int q = tid; q < ncell; q += 1024) b.cfill[q] = 0;
  __syncthreads();
  for (int p = tid; p < np; p += 1024) {
    const int c = coll_cell(pg, b.pos4[p]);
    b.ccell[p] = c;
    atomicAdd(&b.cfill[c], 1);
  }
  __syncthreads();
  const int per = (ncell + 1023) / 1024, lo = min(tid * per, ncell), hi = min(lo + per, ncell);
  int sum = 0;
  for (int q = lo; q < hi; ++q) sum += b.cfill[q];
  part[tid] = sum;
  __syncthreads();
  for (int off = 1; off < 1024; off <<= 1) {
    const int v = tid >= off ? part[tid - off] : 0;
    __syncthreads();
    part[tid] += v;
    __syncthreads();
  }
  int run = tid ? part[tid - 1] : 0;
  for (int q = lo; q < hi; ++q) {
    const int n = b.cfill[q];
    b.cstart[q] = run;
    b.cfill[q] = run;
    run += n;
  }
  if (tid == 1023) b.cstart[ncell] = part[1023];
  __syncthreads();
  for (int p = tid; p < np; p += 1024) b.citem[atomicAdd(&b.cfill[b.ccell[p]], 1)] = p;
  __syncthreads();
  for (int q = tid; q < ncell; q += 1024) {  // ascending within the cell
    const int e0 = b.cstart[q], e1 = b.cstart[q + 1];
    for (int i = e0 + 1; i < e1; ++i) {
      const int v = b.citem[i];
      int j = i - 1;
      while (j >= e0 && b.citem[j] > v) { b.citem[j + 1] = b.citem[j]; --j; }
      b.citem[j + 1] = v;
    }
  }
}

// the FP32 periodic-distance filter of the candidate search
__device__ __forceinline__ bool coll_near(float4 q, float pxf, float pyf, float pzf, float lxf, float lyf, float thr2) {
  float dxf = fabsf(q.x - pxf);
  float dyf = fabsf(q.y - pyf);
  const float dzf = q.z - pzf;
  dxf = fminf(dxf, fabsf(lxf - dxf));
  dyf = fminf(dyf, fabsf(lyf - dyf));
  return dxf * dxf + dyf * dyf + dzf * dzf < thr2;
}

// One warp per particle.  A coarse FP32 periodic-distance filter selects the
// partners that can interact (lubrication range, contact, or listed in
// firstc), in ascending particle order, from the 27 cells of the cell list
// around the particle or from all particles (few of them, or a grid narrower
// than three cells).  The lanes evaluate 32 (copy, candidate) pairs at a time;
// lane 0 then walks those that have an effect in the reference's (nb, q)
// order for the force sums and the contact bookkeeping, and handles the walls.
// Newton-Euler and sumrk3 run with a lane per component and accumulator: the
// kernel's cost is its FP64 instructions (a warp's in about 16 cycles of its
// SM), and those of one lane cost as much as a warp's.  Each quantity keeps
// the sequential pass's arithmetic.
// 1000 spheres: 44.5 -> 20.5 us an iteration, and the cell list (9 us) and
// snapshot (7 us) kernels beside it gone; one sphere: 26 -> 14.
__global__ void __launch_bounds__(32 * COLL_WARPS) k_collide_update(PartGeo pg, PartBuffers b, int iter, int rkiter,
                                                                   double dt, int scan, double3 gterm) {
  __shared__ int cand[COLL_WARPS][COLL_CAP];
  __shared__ int ncand[COLL_WARPS], nfar[COLL_WARPS];
  __shared__ int fcs[COLL_WARPS][16];  // the particle's first contact partners (nq <= 15 here)
  const int np = pg.np, nq = pg.nq;
  const int wid = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int p = blockIdx.x * COLL_WARPS + wid;
  if (p >= np) return;
  const float4 *pos4 = b.pos4 + (long)iter * np;
  const int SX = PF_SX + 9 * iter, SU = SX + 3, SOM = SX + 6;  // this iteration's snapshot
  if (lane == 0) { ncand[wid] = 0; nfar[wid] = 0; }
  const double radius = p_rad(pg, p);
  const int qmax0 = b.qmax[p];
  const int *fc = b.firstc + (long)p * nq;
  if (lane < qmax0 && lane < 16) fcs[wid][lane] = fc[lane];
  __syncwarp();
  // FP32 filter: a pair interacts below eps = 0.025, within 1.0125 of the sum
  // of the radii (the equivalent radius is at most half of it); 1.02 leaves
  // room for the FP32 positions (polydisperse: with Rmax, a superset).  The
  // list's capacity is held to the wider 1.05.
  const float rsumf = pg.poly ? (float)(radius + pg.rmax) : 2.f * (float)radius;
  const float thr2 = (1.02f * rsumf) * (1.02f * rsumf), far2 = (1.05f * rsumf) * (1.05f * rsumf);
  const float lxf = (float)pg.lx, lyf = (float)pg.ly;
  const float4 pp = pos4[p];
  const float pxf = pp.x, pyf = pp.y, pzf = pp.z;
  auto listed = [&](int id) {
    for (int i = 0; i < qmax0; ++i)
      if ((i < 16 ? fcs[wid][i] : fc[i]) == id) return true;
    return false;
  };
  if (!scan) {
    // cell list: lane t < 27 scans neighbouring cell t; partners in firstc
    // beyond the filter distance are added by the lane of their slot; then
    // the list is sorted ascending (as the full scan produces it)
    if (lane < 27) {
      const int c0 = b.ccell[p];
      const int cx = c0 % pg.ncx, cy = (c0 / pg.ncx) % pg.ncy, cz = c0 / (pg.ncx * pg.ncy);
      const int x = (cx + lane % 3 - 1 + pg.ncx) % pg.ncx, y = (cy + (lane / 3) % 3 - 1 + pg.ncy) % pg.ncy;
      const int z = cz + lane / 9 - 1;
      if (z >= 0 && z < pg.ncz) {
        const int c = (z * pg.ncy + y) * pg.ncx + x;
        for (int t = b.cstart[c]; t < b.cstart[c + 1]; ++t) {
          const int q = b.citem[t];
          const float4 qp = pos4[q];
          if (q == p || qp.w == 0.f || !coll_near(qp, pxf, pyf, pzf, lxf, lyf, far2)) continue;
          if (coll_near(qp, pxf, pyf, pzf, lxf, lyf, thr2)) {
            const int pos = atomicAdd(&ncand[wid], 1);
            if (pos < COLL_CAP) cand[wid][pos] = q;
          } else if (!listed(b.mslv[q])) {
            atomicAdd(&nfar[wid], 1);
          }
        }
      }
    }
    if (lane < qmax0) {
      const int id = fc[lane];
      if (id >= 1 && id <= np) {
        const int q = id - 1;
        const float4 qp = pos4[q];
        if (q != p && qp.w != 0.f && b.mslv[q] == id && !coll_near(qp, pxf, pyf, pzf, lxf, lyf, thr2)) {
          const int pos = atomicAdd(&ncand[wid], 1);
          if (pos < COLL_CAP) cand[wid][pos] = q;
        }
      }
    }
    __syncwarp();
    const int n = min(ncand[wid], COLL_CAP);
    const int v0 = lane < n ? cand[wid][lane] : 0, v1 = lane + 32 < n ? cand[wid][lane + 32] : 0;
    int r0 = 0, r1 = 0;
    for (int i = 0; i < n; ++i) {
      const int w = cand[wid][i];
      r0 += w < v0;
      r1 += w < v1;
    }
    __syncwarp();
    if (lane < n) cand[wid][r0] = v0;
    if (lane + 32 < n) cand[wid][r1] = v1;
    __syncwarp();
  } else {
    // candidates in ascending q: within the collision distance or already in
    // contact; eight slices of 32 per round, loads issued together
    constexpr int SL = 8;
    for (int base = 0; base < np; base += 32 * SL) {
      float4 qp[SL];
#pragma unroll
      for (int u = 0; u < SL; ++u) {
        const int q = base + 32 * u + lane;
        qp[u] = q < np ? pos4[q] : make_float4(0.f, 0.f, 0.f, 0.f);  // w: 1 for masters
      }
#pragma unroll
      for (int u = 0; u < SL; ++u) {
        const int q = base + 32 * u + lane;
        const bool ok = q < np && q != p && qp[u].w != 0.f;
        bool c = ok && coll_near(qp[u], pxf, pyf, pzf, lxf, lyf, thr2);
        if (qmax0 > 0 && ok && !c) c = listed(b.mslv[q]);
        const bool f = ok && !c && coll_near(qp[u], pxf, pyf, pzf, lxf, lyf, far2);
        const unsigned m = __ballot_sync(0xffffffffu, c), mf = __ballot_sync(0xffffffffu, f);
        if (!(m | mf)) continue;
        if (c) {
          const int pos = ncand[wid] + __popc(m & ((1u << lane) - 1u));
          if (pos < COLL_CAP) cand[wid][pos] = q;
        }
        __syncwarp();
        if (lane == 0) { ncand[wid] += __popc(m); nfar[wid] += __popc(mf); }
        __syncwarp();
      }
    }
  }
  int nc = ncand[wid];
  if (nc + nfar[wid] > COLL_CAP) { if (lane == 0) atomicExch(&b.err[0], 1); nc = min(nc, COLL_CAP); }
  if (b.mslv[p] <= 0) {
    if (iter == 0) snapshot_particle(pg, b, p, 1, lane);
    return;
  }
  const int idp = b.mslv[p];
  const double rkab = pg.rkab[rkiter - 1];
  const int itermax = 1;
  PState S;
  S.u = PF(PF_U); S.v = PF(PF_V); S.w = PF(PF_W); S.omx = PF(PF_OMX); S.omy = PF(PF_OMY); S.omz = PF(PF_OMZ);
  S.colfx = 0.; S.colfy = 0.; S.colfz = 0.;
  const double px = PF(PF_X), py = PF(PF_Y), pz = PF(PF_Z);
  int qlast = qmax0;
  int *fcw = b.firstc + (long)p * nq, *ofcw = b.ofirstc + (long)p * nq;
  // (i) other particles, nb-outer / q-inner as in the reference.  Pairs out of
  // lubrication and contact range (with room for the copies' roundings) and
  // not listed have no effect and are passed over.
  const int npair = pg.nb_copies * nc;
  for (int base = 0; base < npair; base += 32) {
    const int k = base + lane;
    int q = 0, idq = 0, lub = 0;
    bool act = false;
    double dist = 0., deltax = 0., deltay = 0., deltaz = 0., nx = 0., ny = 0., nz = 0., f1 = 0.;
    double qu = 0., qv = 0., qw = 0.;
    if (k < npair) {
      const int nb = k / nc, ci = k - nb * nc;
      q = cand[wid][ci];
      idq = b.mslv[q];
      if (idp != idq && idq > 0) {
        double qx = b.pf[(long)SX * np + q], qy = b.pf[(long)(SX + 1) * np + q];
        const double qz = b.pf[(long)(SX + 2) * np + q];
        copy_shift_coll(nb, pg.lx, pg.ly, qx, qy);
        deltaz = qz - pz;
        deltax = minimg(qx - px, qx - pg.lx - px, qx + pg.lx - px);
        deltay = minimg(qy - py, qy - pg.ly - py, qy + pg.ly - py);
        dist = sqrt(deltax * deltax + deltay * deltay + deltaz * deltaz);
        // polydisperse: contact at the sum of the radii, eps and the
        // lubrication prefactor with the equivalent radius (pair_consts)
        const double rqq = p_rad(pg, q);
        const double rsum = pg.poly ? radius + rqq : 2. * radius;
        // (the shifted copies' minimum image can miss the nearest one, so all
        // copies of a partner that may touch count: they can end its contact)
        const float tf = 1.01f * (float)rsum;
        act = dist < 1.02 * rsum || coll_near(pos4[q], pxf, pyf, pzf, lxf, lyf, tf * tf) || listed(idq);
        if (act) {
          nx = deltax / dist; ny = deltay / dist; nz = deltaz / dist;
          const double re = pg.poly ? 2. * radius * rqq / (radius + rqq) : radius;
          const double eps = (dist - rsum) / re;
          qu = b.pf[(long)SU * np + q]; qv = b.pf[(long)(SU + 1) * np + q]; qw = b.pf[(long)(SU + 2) * np + q];
          if ((eps < 0.025) && (eps > 0.)) {
            lub = 1;
            f1 = d_lub_f1(pg, S.u, S.v, S.w, idq, nx, ny, nz, eps, qu, qv, qw,
                          pg.poly ? 6. * IBM_PI * pg.visc * re : pg.coeff_f);
          }
        }
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, act); todo; todo &= todo - 1) {
      const int j = __ffs(todo) - 1;
      const int jq = __shfl_sync(0xffffffffu, q, j), jidq = __shfl_sync(0xffffffffu, idq, j);
      const int jlub = __shfl_sync(0xffffffffu, lub, j);
      const double jdist = __shfl_sync(0xffffffffu, dist, j);
      const double jdx = __shfl_sync(0xffffffffu, deltax, j), jdy = __shfl_sync(0xffffffffu, deltay, j),
                   jdz = __shfl_sync(0xffffffffu, deltaz, j);
      const double jnx = __shfl_sync(0xffffffffu, nx, j), jny = __shfl_sync(0xffffffffu, ny, j),
                   jnz = __shfl_sync(0xffffffffu, nz, j);
      const double jf1 = __shfl_sync(0xffffffffu, f1, j);
      const double jqu = __shfl_sync(0xffffffffu, qu, j), jqv = __shfl_sync(0xffffffffu, qv, j),
                   jqw = __shfl_sync(0xffffffffu, qw, j);
      if (lane != 0) continue;
      if (jlub) {
        S.colfx = S.colfx + jf1 * jnx;
        S.colfy = S.colfy + jf1 * jny;
        S.colfz = S.colfz + jf1 * jnz;
      }
      int qq = 0;
      const int qm = b.qmax[p];
      const double jrsum = pg.poly ? radius + pg.prad[jq] : 2. * radius;
      for (int i = 1; i <= qm; ++i) {
        if (jidq == fcw[i - 1]) {
          if (jdist < jrsum) {
            qq = i;
            d_collisions(pg, b, p, S, qq, jidq, jdist, jdx, jdy, jdz, jqu, jqv, jqw, b.pf[(long)SOM * np + jq],
                         b.pf[(long)(SOM + 1) * np + jq], b.pf[(long)(SOM + 2) * np + jq], dt, rkab);
          } else if (iter == itermax) {
            d_remove_contact(pg, b, p, i, qlast);
          }
        }
      }
      if (qq == 0 && jdist < jrsum) {
        qlast = qlast + 1;
        if (qlast > nq) {  // overflow: flagged, the pair's update skipped
          atomicExch(&b.err[1], 1);
          qlast = nq;
          continue;
        }
        qq = qlast;
        d_new_contact(pg, b, p, qq);
        d_collisions(pg, b, p, S, qq, jidq, jdist, jdx, jdy, jdz, jqu, jqv, jqw, b.pf[(long)SOM * np + jq],
                     b.pf[(long)(SOM + 1) * np + jq], b.pf[(long)(SOM + 2) * np + jq], dt, rkab);
        fcw[qlast - 1] = jidq;
        ofcw[qlast - 1] = jidq;
      }
      b.qmax[p] = qlast;
    }
  }
  // (ii) walls (intgr_nwtn_eulr.f90:503-603), where one lies within the
  // lubrication range 1.075 R (FP32 screen) or is listed
  const int botw = np + 1, topw = np + 2;
  const float wallf = 1.08f * (float)radius;
  if (!pg.zper && (pzf < wallf || (float)pg.lz - pzf < wallf || !isfinite(pzf) || listed(botw) || listed(topw)) &&
      lane == 0) {
    const int qm_w = b.qmax[p];
    for (int qw_ = botw; qw_ <= topw; ++qw_) {
      const int idq = qw_;
      const double deltax = 0., deltay = 0., deltaz = (qw_ - botw) * pg.lz - pz;
      const double dist = sqrt(deltax * deltax + deltay * deltay + deltaz * deltaz);
      const double deltan = radius - dist;
      const double nx = deltax / dist, ny = deltay / dist, nz = deltaz / dist;
      int qq = 0;
      const double eps = -deltan / radius;
      if ((eps < 0.075) && (eps > 0.))
        d_lubrication(pg, S.u, S.v, S.w, idq, nx, ny, nz, eps, 0., 0., 0.,
                      pg.poly ? 6. * IBM_PI * pg.visc * radius : pg.coeff_f, S.colfx, S.colfy, S.colfz);
      for (int i = 1; i <= qm_w; ++i) {
        if (idq == fcw[i - 1]) {
          qq = i;
          if (dist < radius) {
            d_collisions(pg, b, p, S, qq, idq, dist, deltax, deltay, deltaz, 0., 0., 0., 0., 0., 0., dt, rkab);
          } else if (iter == itermax) {
            d_remove_contact(pg, b, p, i, qlast);
          }
        }
      }
      if ((qq == 0) && (dist < radius)) {
        qlast = qlast + 1;
        if (qlast > nq) { atomicExch(&b.err[1], 1); qlast = nq; continue; }
        qq = qlast;
        d_new_contact(pg, b, p, qq);
        d_collisions(pg, b, p, S, qq, idq, dist, deltax, deltay, deltaz, 0., 0., 0., 0., 0., 0., dt, rkab);
        fcw[qlast - 1] = idq;
        ofcw[qlast - 1] = idq;
      }
    }
  }
  if (lane == 0) b.qmax[p] = qlast;
  // Newton-Euler (intgr_nwtn_eulr.f90:611-667): lane c < 3 takes component c
  // of the translation and of the rotation; colflg is reset to 0 first
  const int c = lane < 3 ? lane : 0;
  const double colx = __shfl_sync(0xffffffffu, S.colfx, 0), coly = __shfl_sync(0xffffffffu, S.colfy, 0),
               colz = __shfl_sync(0xffffffffu, S.colfz, 0);
  const double colf = c == 0 ? colx : (c == 1 ? coly : colz);
  const double vol = p_vol(pg, p), rr = pg.ratiorho;  // ap%vol, ap%ratiorho (coordsfp.f90:96-102)
  const double vr = vol * rr;
  const double ou = PF(PF_OU + c);
  // gterm: rkab dt gacc (1 - 1/ratiorho), formed once on the host
  const double nu = ou + ((-1.) * dt * (PF(PF_FXLTOT + c)) / vr + (PF(PF_INTU + c) - PF(PF_OINTU + c)) / vr) +
                    (c == 0 ? gterm.x : (c == 1 ? gterm.y : gterm.z)) + rkab * 0.5 * dt * (colf + PF(PF_OCOLFX + c)) / vr;
  const double nx = PF(PF_OX + c) + rkab * 0.5 * dt * (nu + ou);
  double om = 0.;
  if (pg.rotation) {
    const double mr = p_mi(pg, p) * rr;
    om = PF(PF_OOMX + c) + (-1.) * dt * PF(PF_TQX + c) / mr + (PF(PF_INTOMX + c) - PF(PF_OINTOMX + c)) / mr +
         rkab * 0.5 * dt * (0. + PF(PF_OCOLTX + c)) / mr;
  }
  const double omx = __shfl_sync(0xffffffffu, om, 0), omy = __shfl_sync(0xffffffffu, om, 1),
               omz = __shfl_sync(0xffffffffu, om, 2);
  // sumrk3 (intgr_nwtn_eulr.f90:1586-1669): lane t owns accumulator t.
  // 0..5: -F + (I - Iold)/dt of the forces and torques; 6: nothing (dpdy = 0);
  // 7..12: the collision terms; 13..15: the accelerations; 16..18: unused
  {
    const int t = lane;
    const double nuc = __shfl_sync(0xffffffffu, nu, t >= 13 && t <= 15 ? t - 13 : 0);
    if (t < RK_N) {
      double *r = b.rkp + (long)p * RK_N + t;
      double a = rkiter == 1 ? 0. : *r;
      if (t < 6 || (t >= 13 && t <= 15)) {
        const double num = t < 6 ? PF(PF_INTU + t) - PF(PF_OINTU + t) : nuc - PF(PF_OU + t - 13);
        if (t < 6) a = a + (-1.) * PF(PF_FXLTOT + t);
        a = a + num / dt;
      } else if (t >= 7 && t <= 12) {
        const double col = t == 7 ? colx : (t == 8 ? coly : (t == 9 ? colz : 0.));
        a = a + 0.5 * rkab * (col + PF(PF_OCOLFX + t - 7));
      }
      *r = a;
    }
  }
  __syncwarp();
  if (lane < 3) {
    PF(PF_X + c) = nx;
    PF(PF_U + c) = nu;
    PF(PF_OMX + c) = om;
    PF(PF_COLFX + c) = colf;
    PF(PF_COLTX + c) = 0.;
  }
  if (lane == 0) {
    const double phi = PF(PF_OPHI) + 0.5 * rkab * dt * (omz + PF(PF_OOMZ));
    PF(PF_PHI) = phi;
    // without rotation about x and y the product with the angle's functions
    // is zero for any finite angle
    const double omtheta = (omx == 0. && omy == 0. && isfinite(phi)) ? 0. : (omy * cos(phi)) - (omx * sin(phi));
    PF(PF_OMTHETA) = omtheta;
    PF(PF_THETA) = PF(PF_OTHETA) + rkab * 0.5 * dt * (omtheta + PF(PF_OOMTHETA));
  }
  if (iter == 0) {
    __syncwarp();
    snapshot_particle(pg, b, p, 1, lane);
  }
}

int launch_collide_update(cudaStream_t s, const PartGeo &pg, PartBuffers b, int iter, int rkiter, double dt) {
  if (pg.np == 0) return 0;
  int n = 1;
  // The search over all particles costs np^2 / 32 FP32 tests, the cell list a
  // one-block kernel over particles and cells.  A whole update, all / cell list:
  // spheres of 16 dx at 256^3 (3375 cells) 1000: 140 / 148 us, 1728: 233 / 221,
  // 2197: 282 / 260; of 3.6 dx at 128^3 (35937 cells) 1000: 142 / 258, 2197: 304 /
  // 388, 4096: 615 / 588.  The line lies between the two break-evens.
  const int scan = pg.np <= 2048 || pg.ncx < 3 || pg.ncy < 3;
  if (!scan) { k_cell_build<<<1, 1024, 0, s>>>(pg, b, iter); ++n; }
  const double rkab = pg.rkab[rkiter - 1], f = 1. - (1. / pg.ratiorho);
  const double3 gt = make_double3(rkab * dt * pg.gacc[0] * f, rkab * dt * pg.gacc[1] * f, rkab * dt * pg.gacc[2] * f);
  k_collide_update<<<(pg.np + COLL_WARPS - 1) / COLL_WARPS, 32 * COLL_WARPS, 0, s>>>(pg, b, iter, rkiter, dt, scan, gt);
  return n;
}

// ---------------------------------------------------------------------------
// periodic correction (:702-714), neighbour flags (:1051-1090, one rank) and
// new Lagrangian points with their rigid-body velocity (:1438-1485).
// One block per particle; the compaction of points flagged `isout` keeps the
// reference order.
// FP64 per point: three additions onto the tabulated offsets (twelve operations
// more when the sphere spins); 1000 spheres of 16 dx: 44 -> 24 us.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_ne_finalize(PartGeo pg, PartBuffers b, IbmBuffers ib, int init) {
  const int np = pg.np;
  const int p = blockIdx.x;
  __shared__ double sx, sy, sz, su, sv, sw, somx, somy, somz;
  __shared__ int wcount[32];
  __shared__ int base;
  __shared__ int edge[4];  // high words of the planes where the periodic image changes, x and y
  // init: 0 = after Newton-Euler, 1 = initial set-up (initparticles +
  // coordsfp), 2 = Lagrangian points only (restart with given flags)
  if (threadIdx.x == 0) {
    if (init == 1) b.mslv[p] = p + 1;
    double x = PF(PF_X), y = PF(PF_Y);
    if (b.mslv[p] > 0 && init == 0) {
      if (x > pg.lx) x = x - pg.lx;
      if (x < 0.) x = x + pg.lx;
      if (y > pg.ly) y = y - pg.ly;
      if (y < 0.) y = y + pg.ly;
      PF(PF_X) = x; PF(PF_Y) = y;
      if (pg.zper) {  // periodic z: the same correction along z
        double z = PF(PF_Z);
        if (z > pg.lz) z = z - pg.lz;
        if (z < 0.) z = z + pg.lz;
        PF(PF_Z) = z;
      }
    }
    const double ro = p_rad(pg, p) + pg.offset;
    const double leftb = 0., rightb = pg.lx, frontb = 0., backb = pg.ly;
    int *nbf = b.nb + (long)p * 9;
    if (init != 2) {
    for (int n = 0; n < 9; ++n) nbf[n] = 0;
    double dist;
    if (x > (rightb - ro)) nbf[1] = 1;
    dist = sqrt((rightb - x) * (rightb - x) + (frontb - y) * (frontb - y));
    if (fabs(dist) < ro) nbf[2] = 1;
    if (y < (frontb + ro)) nbf[3] = 1;
    dist = sqrt((leftb - x) * (leftb - x) + (frontb - y) * (frontb - y));
    if (fabs(dist) < ro) nbf[4] = 1;
    if (x < (leftb + ro)) nbf[5] = 1;
    dist = sqrt((leftb - x) * (leftb - x) + (backb - y) * (backb - y));
    if (fabs(dist) < ro) nbf[6] = 1;
    if (y > (backb - ro)) nbf[7] = 1;
    dist = sqrt((rightb - x) * (rightb - x) + (backb - y) * (backb - y));
    if (fabs(dist) < ro) nbf[8] = 1;
    }
    if (init == 0) {
      double *r = b.rkp + (long)p * RK_N;
      r[RK_DOMX] = 0.; r[RK_DOMY] = 0.; r[RK_DOMZ] = 0.;
    }
    sx = x; sy = y; sz = PF(PF_Z); su = PF(PF_U); sv = PF(PF_V); sw = PF(PF_W);
    somx = PF(PF_OMX); somy = PF(PF_OMY); somz = PF(PF_OMZ);
    edge[0] = __double2hiint(0.5 * pg.dx);
    edge[1] = __double2hiint(pg.lx + 0.5 * pg.dx);
    edge[2] = __double2hiint(0.5 * pg.dy);
    edge[3] = __double2hiint(pg.ly + 0.5 * pg.dy);
    base = 0;
  }
  __syncthreads();
  // nl: the per-particle capacity of the Lagrangian arrays; the sphere's
  // own point count and table offset when polydisperse
  const int nl = pg.nl, nlp = p_nl(pg, p), nt = pg.ntab;
  const double *off3 = b.off + p_toff(pg, p);
  const int wid = threadIdx.x / 32, lane = threadIdx.x % 32;
  // isout (periodic image outside 1..I, 1..J): a point within half a domain of it
  // can only be so by a rounding next to one of the two planes 0.5 dx and lx +
  // 0.5 dx, where the image changes.  So the reference's FP64 test is for points
  // within about 2^-20 of such a plane, by the high words of the coordinates (which
  // order like the integers; a negative coordinate is far from both), and for all
  // points of spheres farther out.
  const double rs = 1.01 * p_rad(pg, p);
  const bool inside = sx - rs > -0.4 * pg.lx && sx + rs < 1.4 * pg.lx && sy - rs > -0.4 * pg.ly && sy + rs < 1.4 * pg.ly;
  auto at_plane = [](double x, const int *h) {
    const unsigned q = (unsigned)__double2hiint(x) + 1u;
    return q - (unsigned)h[0] <= 2u || q - (unsigned)h[1] <= 2u;
  };
  const bool spin = !(somx == 0. && somy == 0. && somz == 0.);
  for (int l0 = 0; l0 < nlp; l0 += blockDim.x) {
    const int l = l0 + threadIdx.x;
    bool keep = false;
    double xfploc = 0, yfploc = 0, zfploc = 0, rx = 0, ry = 0, rz = 0;
    if (l < nlp && b.mslv[p] != 0) {
      // offsets from the centre, radfp*st*cp etc. (table, the reference's
      // rounding); they also serve as (xfp - xc) in the point velocities
      rx = off3[l];
      ry = off3[nt + l];
      rz = off3[2 * nt + l];
      xfploc = sx + rx;
      yfploc = sy + ry;
      zfploc = sz + rz;
      bool isout = false;
      if (!inside || at_plane(xfploc, edge) || at_plane(yfploc, edge + 2)) {
        double isperiodx = 0., isperiody = 0.;
        if (xfploc < 0. + 0.5 * pg.dx) isperiodx = 1.;
        if (xfploc >= pg.lx + 0.5 * pg.dx) isperiodx = -1.;
        if (yfploc < 0. + 0.5 * pg.dy) isperiody = 1.;
        if (yfploc >= pg.ly + 0.5 * pg.dy) isperiody = -1.;
        const double coorxfp = (xfploc + isperiodx * pg.lx - 0.) * pg.dxi;
        if (fnint(coorxfp) < 1 || fnint(coorxfp) > pg.I) isout = true;
        const double cooryfp = (yfploc + isperiody * pg.ly - 0.) * pg.dyi;
        if (fnint(cooryfp) < 1 || fnint(cooryfp) > pg.J) isout = true;
      }
      keep = !isout;
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) wcount[wid] = __popc(m);
    __syncthreads();
    int off = base;
    for (int q = 0; q < wid; ++q) off += wcount[q];
    off += __popc(m & ((1u << lane) - 1u));
    if (keep) {
      const long t = (long)p * nl + off;
      ib.xfp[t] = xfploc; ib.yfp[t] = yfploc; ib.zfp[t] = zfploc;
      ib.ul[t] = spin ? su + somy * rz - somz * ry : su;
      ib.vl[t] = spin ? sv + somz * rx - somx * rz : sv;
      ib.wl[t] = spin ? sw + somx * ry - somy * rx : sw;
    }
    __syncthreads();
    if (threadIdx.x == 0) for (int q = 0; q < (int)(blockDim.x / 32); ++q) base += wcount[q];
    __syncthreads();
  }
  if (threadIdx.x == 0) ib.nla[p] = b.mslv[p] != 0 ? base : 0;
}

void launch_ne_finalize(cudaStream_t s, const PartGeo &pg, PartBuffers b, IbmBuffers ib, int init) {
  if (pg.np == 0) return;
  k_ne_finalize<<<pg.np, 256, 0, s>>>(pg, b, ib, init);
}

}  // namespace ibmk
