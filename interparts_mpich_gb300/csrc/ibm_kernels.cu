// ibm_kernels.cu -- multidirect immersed-boundary forcing on the Lagrangian
// points: eulr2lagr (interp_spread.f90:12-228), complagrforces /
// updtlagrforces (forcing.f90:9-391) and lagr2eulr (interp_spread.f90:230-474).
//
// Compiled without FMA contraction so the stencil indices, delta weights and
// point forces follow the reference roundings.
//
// Spreading is incremental: lagr2eulr rebuilds dudtf = dudtold + S(F) with
// the cumulative point force F every pass (zeroing and re-adding the whole
// field).  By linearity of S, dudtf after pass n equals the pass n-1 field
// plus S(F_n - F_{n-1}); the GPU adds only S(dF) over the points' footprint,
// so no full-field pass is needed.  The one plane that the reference never
// refreshes from dwdt, dwdtf(:,:,k1), is zeroed before the first spread of
// a substep so it carries S(F) exactly as in the reference.
#include <cuda_bf16.h>

#include "kernels.cuh"

namespace ibmk {

// The plain form's IBM kernels are bound by FP64 issue (a warp instruction in
// about 18 cycles per SM).  So the weights are formed once per substep, one
// square root per axis and offset (6 a point, 18 with one per node), products
// and sums are fused by hand where the stencil indices and decisions do not
// hang on them, and a thread takes one component of one point: a single sphere
// (719 points at D = 16 dx) still spreads over 34 SMs.  Blocks take the three
// components of the same points in turn, so that their weights come from L2.
//   1000 spheres of 16 dx: stencil 587 -> 202 us, interpolation 427 -> 171,
//   spreading 276 -> 252 (63 M FP64 atomic adds), force sums (last pass) 34
//   one sphere: stencil 35 -> 9 us, interpolation 70 -> 8, spreading 19 -> 6

// delta weights at three consecutive nodes, r1 the signed distance of node 1.
// |r1| <= 1/2: node 1 takes the inner branch of kernel.f90:7-25, nodes 0 and 2
// the outer one, and all share s = sqrt(1 - 3 r1^2); any other r1 (an origin
// clamped at a wall) takes the general form node by node.
__device__ __forceinline__ void delta3wd(double r1, double *w, long n) {
  if (fabs(r1) <= 0.5) {
    const double s = sqrt_newton(fma(-3. * r1, r1, 1.));
    w[0] = (1. / 6.) * (fma(3., r1, 2.) - s);
    w[n] = (1. / 3.) * (1. + s);
    w[2 * n] = (1. / 6.) * (fma(-3., r1, 2.) - s);
  } else {
    w[0] = delta3(r1 - 1.);
    w[n] = delta3(r1);
    w[2 * n] = delta3(r1 + 1.);
  }
}
// periodic images of a coordinate: floor(t / l) without the division where t
// lies in the domain (the quotient of t < l rounds below one)
__device__ __forceinline__ int image(double t, double l) { return t >= 0. && t < l ? 0 : (int)floor(t / l); }

// stencil of one point (interp_spread.f90:76-130), single rank (zstart = 1):
// origins in so, weights in sw (field-major, SW_*)
__global__ void __launch_bounds__(64) k_ibm_stencil(Geo g, PartGeo pg, IbmBuffers b) {
  const int n = pg.np * pg.nl;  // < 2^31 points (checked at create)
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int p = t / pg.nl, l = t - p * pg.nl;
    if (l >= b.nla[p]) continue;
    const double xfp = b.xfp[t], yfp = b.yfp[t], zfp = b.zfp[t];
    double coorxfp = xfp * g.dxi - (double)((long)image(xfp - 0.5 * g.dx, g.lx) * g.I);
    double cooryfp = yfp * g.dyi - (double)((long)image(yfp - 0.5 * g.dy, g.ly) * g.J);
    // periodic z: the image rule of x and y along z (no wall clamps below)
    double coorzfp = g.zper ? zfp * g.dzi - (double)((long)image(zfp - 0.5 * g.dz, g.lz) * g.K) : zfp * g.dzi;
    // Guard: a point outside the grid (or a non-finite position) would index
    // outside the arrays; flag it and park the point at a safe location.
    if (!(coorxfp >= 0. && coorxfp <= g.I + 1.) || !(cooryfp >= 0. && cooryfp <= g.J + 1.) ||
        !(g.zper ? (coorzfp >= 0. && coorzfp <= g.K + 1.) : (coorzfp >= -1. && coorzfp <= g.K + 0.49))) {
      atomicExch(&b.err[2], 1);
      coorxfp = 1.; cooryfp = 1.; coorzfp = 1.5;
    }
    const int ilows = fnint(coorxfp) - 1, jlows = fnint(cooryfp) - 1;
    const int klows = g.zper ? fnint(coorzfp) - 1 : max(fnint(coorzfp) - 1, 1);
    const int ilow = (int)floor(coorxfp), jlow = (int)floor(cooryfp);
    const int klow = g.zper ? (int)floor(coorzfp) : max(min((int)floor(coorzfp), g.K - 2), 1);
    // the staggered origins as offsets from the centred ones (-1..2)
    b.so[t] = make_int4(ilow, jlow, klow, (ilows - ilow + 8) | (jlows - jlow + 8) << 8 | (klows - klow + 8) << 16);
    const long nn = n;
    double *w = b.sw + t;
    delta3wd(1. * (ilows + 1) - coorxfp, w + SW_X * nn, nn);
    delta3wd(1. * (jlows + 1) - cooryfp, w + SW_Y * nn, nn);
    delta3wd(1. * (klows + 1) - coorzfp, w + SW_Z * nn, nn);
    delta3wd(1. * ilow + .5 - coorxfp, w + SW_XH * nn, nn);
    delta3wd(1. * jlow + .5 - cooryfp, w + SW_YH * nn, nn);
    delta3wd(1. * klow + .5 - coorzfp, w + SW_ZH * nn, nn);
  }
}

// component C (0 u, 1 v, 2 w) of point t: offsets of its 3 x 3 x 3 taps along
// each axis (periodic images folded in) and its weights
template <int C> struct Taps {
  int ox[3], oy[3];
  long oz[3];
  double wx[3], wy[3], wz[3];
  __device__ __forceinline__ Taps(const Geo &g, const IbmBuffers &b, long n, int t) {
    const int4 o = b.so[t];
    const int i0 = o.x + (C == 0 ? (o.w & 255) - 8 : 0), j0 = o.y + (C == 1 ? ((o.w >> 8) & 255) - 8 : 0),
              k0 = o.z + (C == 2 ? ((o.w >> 16) & 255) - 8 : 0);
    const double *w = b.sw + t;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      ox[m] = wrapm(i0 + m - 1, g.I);
      oy[m] = wrapm(j0 + m - 1, g.J) * g.I;
      oz[m] = zwrap(g, k0 + m) * g.plane;
      wx[m] = w[((C == 0 ? SW_X : SW_XH) + m) * n];
      wy[m] = w[((C == 1 ? SW_Y : SW_YH) + m) * n];
      wz[m] = w[((C == 2 ? SW_Z : SW_ZH) + m) * n];
    }
  }
};

// blocks of IB_T points, the three components of a chunk in consecutive blocks
constexpr int IB_T = 64;
inline int ibm_blocks(const PartGeo &pg) {
  const long need = 3L * (((long)pg.np * pg.nl + IB_T - 1) / IB_T);
  return (int)(need < 3 * 152 * 32 ? need : 3 * 152 * 32);
}

// eulr2lagr (the separable form of the 27-tap sums of interp_spread.f90:132-154,
// 39 multiply-adds) and the point force of complagrforces / updtlagrforces
template <int C>
__device__ __forceinline__ void interp_points(const Geo &g, const PartGeo &pg, const IbmBuffers &b,
                                              const double *__restrict__ f, double dti, int first) {
  const int n = pg.np * pg.nl;
  const double *U = C == 0 ? b.ul : (C == 1 ? b.vl : b.wl);
  double *I = C == 0 ? b.dudtl : (C == 1 ? b.dvdtl : b.dwdtl), *F = C == 0 ? b.fxl : (C == 1 ? b.fyl : b.fzl);
  for (int t = (int)(blockIdx.x / 3) * IB_T + threadIdx.x; t < n; t += (int)(gridDim.x / 3) * IB_T) {
    const int p = t / pg.nl;
    if (t - p * pg.nl >= b.nla[p]) continue;
    const Taps<C> s(g, b, n, t);
    double acc = 0.;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      double sj = 0.;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double *r = f + s.oz[k] + s.oy[j];
        sj = fma(fma(r[s.ox[2]], s.wx[2], fma(r[s.ox[1]], s.wx[1], r[s.ox[0]] * s.wx[0])), s.wy[j], sj);
      }
      acc = fma(sj, s.wz[k], acc);
    }
    I[t] = acc;
    if (first < 0) continue;  // interpolation only (slip residual)
    const double d = U[t] - acc;
    F[t] = first ? d * dti : fma(d, dti, F[t]);
  }
}
__global__ void __launch_bounds__(IB_T) k_ibm_interp_force(Geo g, PartGeo pg, IbmBuffers b,
                                                           const double *__restrict__ fu,
                                                           const double *__restrict__ fv,
                                                           const double *__restrict__ fw, double dti, int first) {
  const int c = blockIdx.x % 3;
  if (c == 0) interp_points<0>(g, pg, b, fu, dti, first);
  else if (c == 1) interp_points<1>(g, pg, b, fv, dti, first);
  else interp_points<2>(g, pg, b, fw, dti, first);
}

// force and torque sums of one particle per block (complagrforces), after the
// last pass only: each pass's totals replace the ones before.  A fifth warp
// forms cos and sin of the torque's angle meanwhile (two long FP64 chains at the
// end of one thread before): one sphere 12.5 -> 10.3 us.
constexpr int FT_T = 128;
__global__ void __launch_bounds__(FT_T + 32) k_ibm_force_torque(PartGeo pg, IbmBuffers b) {
  __shared__ double red[6][4], trig[2];
  const int p = blockIdx.x, np = pg.np, nla = b.nla[p];
  if (threadIdx.x >= FT_T) {
    if (threadIdx.x < FT_T + 2) {
      const double phi = b.pf[PF_PHI * np + p];
      trig[threadIdx.x - FT_T] = threadIdx.x == FT_T ? cos(phi) : sin(phi);
    }
  } else {
    const double px = b.pf[PF_X * np + p], py = b.pf[PF_Y * np + p], pz = b.pf[PF_Z * np + p];
    double s[6] = {0., 0., 0., 0., 0., 0.};
#pragma unroll 3
    for (int l = threadIdx.x; l < nla; l += FT_T) {
      const long t = (long)p * pg.nl + l;
      const double fx = b.fxl[t], fy = b.fyl[t], fz = b.fzl[t];
      const double rx = b.xfp[t] - px, ry = b.yfp[t] - py, rz = b.zfp[t] - pz;
      s[0] += fx; s[1] += fy; s[2] += fz;
      s[3] = fma(-rz, fy, fma(ry, fz, s[3]));
      s[4] = fma(-rx, fz, fma(rz, fx, s[4]));
      s[5] = fma(-ry, fx, fma(rx, fy, s[5]));
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) s[q] += __shfl_down_sync(0xffffffffu, s[q], d);
      if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = s[q];
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  if (threadIdx.x < 6) {
    const int q = threadIdx.x;
    const double v = ((red[q][0] + red[q][1]) + (red[q][2] + red[q][3])) * p_dvl(pg, p);
    const int f[6] = {PF_FXLTOT, PF_FYLTOT, PF_FZLTOT, PF_TQX, PF_TQY, PF_TQZ};
    b.pf[f[q] * np + p] = v;
    red[q][0] = v;
  }
  __syncwarp();
  if (threadIdx.x == 0) b.pf[PF_TQTHETA * np + p] = (red[4][0] * trig[0]) - (red[3][0] * trig[1]);
}

void launch_ibm_stencil(cudaStream_t s, const Geo &g, const PartGeo &pg, IbmBuffers b) {
  k_ibm_stencil<<<ibm_blocks(pg) / 3, IB_T, 0, s>>>(g, pg, b);
}

void launch_ibm_interp_force(cudaStream_t s, const Geo &g, const PartGeo &pg, IbmBuffers b, const double *fu,
                             const double *fv, const double *fw, double dt, int first) {
  k_ibm_interp_force<<<ibm_blocks(pg), IB_T, 0, s>>>(g, pg, b, fu, fv, fw, 1. / dt, first);
}
void launch_ibm_force_torque(cudaStream_t s, const PartGeo &pg, IbmBuffers b) {
  k_ibm_force_torque<<<pg.np, FT_T + 32, 0, s>>>(pg, b);
}

// lagr2eulr increment: spread dF = (U_l - u~_l)/dt with the terms of
// interp_spread.f90:329-355, F*coeff0*phix*phiy*phiz, the z and y factors
// taken in before the row of three taps (41 FP64 instructions and 27 atomic
// adds a component)
template <int C>
__device__ __forceinline__ void spread_points(const Geo &g, const PartGeo &pg, const IbmBuffers &b,
                                              double *__restrict__ f, double dti, double coeff0_, double dt) {
  const int n = pg.np * pg.nl;
  const double *U = C == 0 ? b.ul : (C == 1 ? b.vl : b.wl), *I = C == 0 ? b.dudtl : (C == 1 ? b.dvdtl : b.dwdtl);
  for (int t = (int)(blockIdx.x / 3) * IB_T + threadIdx.x; t < n; t += (int)(gridDim.x / 3) * IB_T) {
    const int p = t / pg.nl;
    if (t - p * pg.nl >= b.nla[p]) continue;
    const Taps<C> s(g, b, n, t);
    // the particle's own Lagrangian volume when polydisperse
    const double coeff0 = pg.poly ? (pg.pdvl[p] / pg.dVeul) * dt : coeff0_;
    const double d = (U[t] - I[t]) * dti * coeff0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double dk = d * s.wz[k];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double dj = dk * s.wy[j];
        double *r = f + s.oz[k] + s.oy[j];
#pragma unroll
        for (int i = 0; i < 3; ++i) atomicAdd(r + s.ox[i], dj * s.wx[i]);
      }
    }
  }
}
__global__ void __launch_bounds__(IB_T) k_ibm_spread(Geo g, PartGeo pg, IbmBuffers b, double *__restrict__ fu,
                                                     double *__restrict__ fv, double *__restrict__ fw, double dti,
                                                     double coeff0, double dt) {
  const int c = blockIdx.x % 3;
  if (c == 0) spread_points<0>(g, pg, b, fu, dti, coeff0, dt);
  else if (c == 1) spread_points<1>(g, pg, b, fv, dti, coeff0, dt);
  else spread_points<2>(g, pg, b, fw, dti, coeff0, dt);
}
void launch_ibm_spread(cudaStream_t s, const Geo &g, const PartGeo &pg, IbmBuffers b, double *fu, double *fv,
                       double *fw, double dt) {
  const double coeff0 = (pg.dVlagr / pg.dVeul) * dt;
  k_ibm_spread<<<ibm_blocks(pg), IB_T, 0, s>>>(g, pg, b, fu, fv, fw, 1. / dt, coeff0, dt);
}

template <typename T>
__global__ void k_zero_plane(Geo g, T *f, int k) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < g.plane; t += (long)gridDim.x * blockDim.x)
    f[(long)k * g.plane + t] = (T)0;
}
template <typename T>
void launch_zero_plane(cudaStream_t s, const Geo &g, T *f, int k) {
  k_zero_plane<T><<<152, 256, 0, s>>>(g, f, k);
}
template void launch_zero_plane<double>(cudaStream_t, const Geo &, double *, int);
template void launch_zero_plane<float>(cudaStream_t, const Geo &, float *, int);

// |U_l - u~_l| statistics (max, sum of squares, count) over all points,
// using the interpolation stored by the last pass.
__global__ void k_slip_residual(PartGeo pg, IbmBuffers b, double *out) {
  __shared__ double smax[256], ssum[256];
  double mx = 0., sm = 0.;
  const int n = pg.np * pg.nl;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int p = t / pg.nl, l = t - p * pg.nl;
    if (l >= b.nla[p]) continue;
    const double ex = b.ul[t] - b.dudtl[t], ey = b.vl[t] - b.dvdtl[t], ez = b.wl[t] - b.dwdtl[t];
    const double r2 = ex * ex + ey * ey + ez * ez;
    mx = fmax(mx, sqrt(r2));
    sm += r2;
  }
  smax[threadIdx.x] = mx; ssum[threadIdx.x] = sm;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + o]);
      ssum[threadIdx.x] += ssum[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) { out[0] = smax[0]; out[1] = ssum[0]; }
}
void launch_slip_residual(cudaStream_t s, const PartGeo &pg, IbmBuffers b, double *out) {
  k_slip_residual<<<1, 256, 0, s>>>(pg, b, out);
}

// targets of the slots reserved since the last call: (F_final - F0) * dt, the
// correction the plain passes 1.. added after pass 0
__global__ void k_ibm_harvest_targets(IbmBuffers b, HarvestArgs H, double dt) {
  const int lo = H.count[1], hi = min(H.count[0], H.cap);
  for (int h = lo + blockIdx.x * blockDim.x + threadIdx.x; h < hi; h += gridDim.x * blockDim.x) {
    const int t = H.pidx[h];
    const float *f = H.feat + (long)h * 96 + FEAT_F0;
    H.targ[3 * (long)h] = b.fxs[t] * (float)dt - f[0];
    H.targ[3 * (long)h + 1] = b.fys[t] * (float)dt - f[FEAT_PER_COMP];
    H.targ[3 * (long)h + 2] = b.fzs[t] * (float)dt - f[2 * FEAT_PER_COMP];
  }
}
__global__ void k_ibm_harvest_close(HarvestArgs H) {
  if (threadIdx.x == 0 && blockIdx.x == 0) H.count[1] = min(H.count[0], H.cap);
}
void launch_ibm_harvest_targets(cudaStream_t s, IbmBuffers b, const HarvestArgs &H, double dt) {
  k_ibm_harvest_targets<<<152, 256, 0, s>>>(b, H, dt);
  k_ibm_harvest_close<<<1, 32, 0, s>>>(H);
}
// Residual gate.  R = rms |U - u~| over all points after the loop (from the
// per-(particle, component) sums psum[p][c][0]) and R0 = rms of the first
// pass's slip (from rsum).  A plain loop's R/R0 measures how far its Nl
// passes reduce the slip on the current state, per RK stage (the predicted
// field, and with it the slip's pattern, differs between the stages); the
// learned loop of stage s is held to fallback ratio x (that stage's ratio x
// its own R0), i.e. to what the plain passes would reach from the same
// first-pass slip.  Learn state ls (device):
//   [0] R of the last learned loop      [1] plain R/R0 of stage 1 (the last measured)
//   [2] plain loops measured            [3] fallback ratio
//   [4] fallbacks taken                 [5] learned loops
//   [6] R0 of the last learned loop     [7] reference of the last gate
//   [8] fixed reference (> 0 replaces ratio x R0)
//   [9] R0 and [10] R of the last plain loop measured
//   [11], [12] plain R/R0 of stages 2 and 3; [13..15] plain loops measured per stage
// gate = 1 runs the plain passes 2..Nl after the learned correction.
__global__ void __launch_bounds__(1024) k_ibm_res_gate(int n, const double *__restrict__ psum,
                                                       const float *__restrict__ rsum, long npts, double *ls,
                                                       int *gate, int plain, int stage) {
  // per-(particle, component) sums are FP32 accurate (formed in FP32): their
  // totals in FP32 with warp shuffles, FP64 only for the gate's arithmetic
  __shared__ float sm[2][32];
  float acc = 0.f, acc0 = 0.f;
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    acc += (float)psum[3 * (long)q];
    acc0 += rsum[q];
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    acc += __shfl_xor_sync(0xffffffffu, acc, d);
    acc0 += __shfl_xor_sync(0xffffffffu, acc0, d);
  }
  if ((threadIdx.x & 31) == 0) { sm[0][threadIdx.x >> 5] = acc; sm[1][threadIdx.x >> 5] = acc0; }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  // the 32 warps' sums by a warp (not one thread's chain of 64 FP64 adds)
  double tot = sm[0][threadIdx.x], tot0 = sm[1][threadIdx.x];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    tot += __shfl_down_sync(0xffffffffu, tot, d);
    tot0 += __shfl_down_sync(0xffffffffu, tot0, d);
  }
  if (threadIdx.x != 0) return;
  const double R = npts ? sqrt(tot / (double)npts) : 0., R0 = npts ? sqrt(tot0 / (double)npts) : 0.;
  const int cs = stage == 0 ? 1 : 10 + stage, ns = 13 + stage;
  if (plain) {  // the plain passes' reduction of the slip on the current state
    // the latest measurement alone: the reduction drifts as the flow (and
    // the learned forcing's imprint on it) develops, an average lags it
    ls[cs] = R0 > 0. ? R / R0 : 0.;
    ls[ns] += 1.;
    ls[2] += 1.;
    ls[9] = R0;
    ls[10] = R;
    return;
  }
  const double ref = ls[8] > 0. ? ls[8] : (ls[ns] > 0. ? ls[cs] * R0 : 0.);
  ls[0] = R;
  ls[5] += 1.;
  ls[6] = R0;
  ls[7] = ref;
  const int g = (!(R <= ls[3] * ref)) ? 1 : 0;  // NaN falls back too
  *gate = g;
  if (g) ls[4] += 1.;
}
void launch_ibm_residual_gate(cudaStream_t s, const PartGeo &pg, IbmBuffers b, long npts, double *ls, int *gate,
                              int plain, int stage) {
  k_ibm_res_gate<<<1, 1024, 0, s>>>(3 * pg.np, b.psum, b.rsum, npts, ls, gate, plain, stage);
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {  // splitmix64 finaliser
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
__global__ void k_normal_fill(float *__restrict__ y, long n, unsigned seed, unsigned counter) {
  const unsigned long long key = ((unsigned long long)seed << 32) ^ counter;
  for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < n; q += (long)gridDim.x * blockDim.x) {
    const unsigned long long h = mix64(mix64(key * 0x9E3779B97F4A7C15ULL + (unsigned long long)q));
    // two 24-bit uniforms in (0, 1), Box-Muller (one deviate kept)
    const float u1 = ((float)(h & 0xFFFFFF) + 0.5f) * (1.f / 16777216.f);
    const float u2 = ((float)((h >> 24) & 0xFFFFFF) + 0.5f) * (1.f / 16777216.f);
    y[q] = sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
  }
}
void launch_normal_fill(cudaStream_t s, float *y, long n, unsigned seed, unsigned counter) {
  if (n <= 0) return;
  k_normal_fill<<<1216, 256, 0, s>>>(y, n, seed, counter);
}

}  // namespace ibmk
