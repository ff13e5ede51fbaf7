// fluid_kernels.cu -- momentum predictor, velocity correction, boundary
// conditions, layout conversion and the chkdiv/chkdt reductions.
//
// One thread per interior cell; x/y neighbours by periodic wrap, z ghosts
// stored.  All arithmetic follows the reference expression order; FP64
// fused multiply-add contraction is allowed (differences at 1 ulp level).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdint>

#include "kernels.cuh"

namespace ibmk {

// ---------------------------------------------------------------------------
// Momentum predictor: rk1/rk2/rk3 (rk3.f90:13-329) fused with momxp..momzad
// (mom.f90:8-231).  STAGE 1: dudt = u + f1*gradp; dudt += f1*RHS; rhs_old=RHS
// STAGE 2/3: dudt = u + f1*gradp; dudt += (f2*RHS - f3*rhs_old); stage 2
// stores rhs_old = RHS.  The output goes straight into the forcing buffer
// (dudtf == dudt on entry of the IBM loop, main.f90:288-306).
// One thread per cell: the mixed forms' fields of 2^31 cells and more.
// ---------------------------------------------------------------------------
template <typename TU, typename T, int STAGE>
__global__ void __launch_bounds__(256) k_predict(Geo g, const TU *__restrict__ u, const TU *__restrict__ v,
                                                 const TU *__restrict__ w, const TU *__restrict__ p,
                                                 T *__restrict__ ru, T *__restrict__ rv, T *__restrict__ rw,
                                                 T *__restrict__ fu, T *__restrict__ fv, T *__restrict__ fw,
                                                 T f1, T f2, T f3, const double *__restrict__ cb, double bcoef) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z + 1;
  if (i >= g.I || j >= g.J) return;
  // neighbours as 32-bit offsets from one 64-bit cell address (periodic
  // wrap in x and y folded into the offsets)
  const int dip = i + 1 == g.I ? 1 - g.I : 1, dim = i == 0 ? g.I - 1 : -1;
  const int djp = (j + 1 == g.J ? 1 - g.J : 1) * g.I, djm = (j == 0 ? g.J - 1 : -1) * g.I;
  const int PL = g.I * g.J;
  const long c = fidx(g, i, j, k);
  const int ip = dip, im = dim, jp = djp, jm = djm;
  auto at = [&](int di, int dj, int dk) -> long { return c + (di + dj + dk); };
  const int j0 = 0, i0 = 0;
  const int kp = PL, km = -PL;
  const T dxi = (T)g.dxi, dyi = (T)g.dyi, dzi = (T)g.dzi, visc = (T)g.visc;
  const T q = (T)0.25;
  // u-neighbourhood
  const T U0 = (T)u[c], Uip = (T)u[at(ip, j0, 0)], Uim = (T)u[at(im, j0, 0)], Ujp = (T)u[at(i0, jp, 0)],
          Ujm = (T)u[at(i0, jm, 0)];
  const T Ukp = (T)u[c + PL], Ukm = (T)u[c - PL];
  const T V0 = (T)v[c], Vip = (T)v[at(ip, j0, 0)], Vim = (T)v[at(im, j0, 0)], Vjp = (T)v[at(i0, jp, 0)],
          Vjm = (T)v[at(i0, jm, 0)];
  const T Vkp = (T)v[c + PL], Vkm = (T)v[c - PL];
  const T W0 = (T)w[c], Wip = (T)w[at(ip, j0, 0)], Wim = (T)w[at(im, j0, 0)], Wjp = (T)w[at(i0, jp, 0)],
          Wjm = (T)w[at(i0, jm, 0)];
  const T Wkp = (T)w[c + PL], Wkm = (T)w[c - PL];
  // diagonal neighbours
  const T Vipjm = (T)v[at(ip, jm, 0)], Wipkm = (T)w[at(ip, j0, km)];
  const T Uimjp = (T)u[at(im, jp, 0)], Wjpkm = (T)w[at(i0, jp, km)];
  const T Uimkp = (T)u[at(im, j0, kp)], Vjmkp = (T)v[at(i0, jm, kp)];
  // momxad (mom.f90:21-50)
  T ru_new;
  {
    const T uuip = q * (Uip + U0) * (Uip + U0);
    const T uuim = q * (Uim + U0) * (Uim + U0);
    const T uvjp = q * (Ujp + U0) * (Vip + V0);
    const T uvjm = q * (Ujm + U0) * (Vipjm + Vjm);
    const T uwkp = q * (Ukp + U0) * (Wip + W0);
    const T uwkm = q * (Ukm + U0) * (Wipkm + Wkm);
    const T dudxp = (Uip - U0) * dxi, dudxm = (U0 - Uim) * dxi;
    const T dudyp = (Ujp - U0) * dyi, dudym = (U0 - Ujm) * dyi;
    const T dudzp = (Ukp - U0) * dzi, dudzm = (U0 - Ukm) * dzi;
    ru_new = dxi * (-uuip + uuim) + visc * (dudxp - dudxm) * dxi + dyi * (-uvjp + uvjm) +
             visc * (dudyp - dudym) * dyi + dzi * (-uwkp + uwkm) + visc * (dudzp - dudzm) * dzi;
  }
  T rv_new;
  {  // momyad (mom.f90:94-123)
    const T uvip = q * (U0 + Ujp) * (V0 + Vip);
    const T uvim = q * (Uim + Uimjp) * (V0 + Vim);
    const T vvjp = q * (V0 + Vjp) * (V0 + Vjp);
    const T vvjm = q * (V0 + Vjm) * (V0 + Vjm);
    const T wvkp = q * (W0 + Wjp) * (Vkp + V0);
    const T wvkm = q * (Wkm + Wjpkm) * (Vkm + V0);
    const T dvdxp = (Vip - V0) * dxi, dvdxm = (V0 - Vim) * dxi;
    const T dvdyp = (Vjp - V0) * dyi, dvdym = (V0 - Vjm) * dyi;
    const T dvdzp = (Vkp - V0) * dzi, dvdzm = (V0 - Vkm) * dzi;
    rv_new = dxi * (-uvip + uvim) + visc * (dvdxp - dvdxm) * dxi + dyi * (-vvjp + vvjm) +
             visc * (dvdyp - dvdym) * dyi + dzi * (-wvkp + wvkm) + visc * (dvdzp - dvdzm) * dzi;
  }
  T rw_new;
  {  // momzad (mom.f90:170-199)
    const T uwip = q * (W0 + Wip) * (U0 + Ukp);
    const T uwim = q * (W0 + Wim) * (Uim + Uimkp);
    const T vwjp = q * (W0 + Wjp) * (V0 + Vkp);
    const T vwjm = q * (W0 + Wjm) * (Vjm + Vjmkp);
    const T wwkp = q * (W0 + Wkp) * (W0 + Wkp);
    const T wwkm = q * (W0 + Wkm) * (W0 + Wkm);
    const T dwdxp = (Wip - W0) * dxi, dwdxm = (W0 - Wim) * dxi;
    const T dwdyp = (Wjp - W0) * dyi, dwdym = (W0 - Wjm) * dyi;
    const T dwdzp = (Wkp - W0) * dzi, dwdzm = (W0 - Wkm) * dzi;
    rw_new = dxi * (-uwip + uwim) + visc * (dwdxp - dwdxm) * dxi + dyi * (-vwjp + vwjm) +
             visc * (dwdyp - dwdym) * dyi + dzi * (-wwkp + wwkm) + visc * (dwdzp - dwdzm) * dzi;
  }
  // momzbuoy (mom.f90:251), added as rk1..rk3 do (rk3.f90:56-58)
  if (cb) rw_new = (T)(bcoef * (cb[c] + cb[c + PL])) + rw_new;
  // pressure gradient (momxp/momyp/momzp)
  const T P0 = (T)p[c];
  const T gx = -dxi * ((T)p[at(ip, j0, 0)] - P0);
  const T gy = -dyi * ((T)p[at(i0, jp, 0)] - P0);
  const T gz = -dzi * ((T)p[c + PL] - P0);
  T du = U0 + f1 * gx, dv = V0 + f1 * gy, dw = W0 + f1 * gz;
  if (STAGE == 1) {
    du = du + f1 * ru_new;
    dv = dv + f1 * rv_new;
    dw = dw + f1 * rw_new;
  } else {
    du = du + (f2 * ru_new - f3 * ru[c]);
    dv = dv + (f2 * rv_new - f3 * rv[c]);
    dw = dw + (f2 * rw_new - f3 * rw[c]);
  }
  fu[c] = du;
  fv[c] = dv;
  fw[c] = dw;
  if (STAGE != 3) {
    ru[c] = ru_new;
    rv[c] = rv_new;
    rw[c] = rw_new;
  }
}

// FP64 predictor: bound by FP64 issue (one warp instruction in about 18 cycles
// per SM), so the kernel is built around the number of FP64 instructions a
// cell takes.  Every product of interpolated velocities is a flux through one
// face or edge and is formed once, by the cell on its lower side:
//   xx = (u(i+1) + u)^2, yy = (v(j+1) + v)^2, zz = (w(k+1) + w)^2,
//   uv = (u(j+1) + u)(v(i+1) + v), uw = (u(k+1) + u)(w(i+1) + w),
//   vw = (w(j+1) + w)(v(k+1) + v);
// the cells at i+1 and j+1 read it from shared memory, the one at k+1 keeps
// it in registers as the block marches along z.  With the Laplacian as sums
// of opposite neighbours that is 63 to 66 FP64 instructions a cell, against
// about 130 for one thread per cell forming all its fluxes.  256^3, stage 2:
// 4.39 -> 2.22 ms (0.50 T FP64 instructions/s both times).
// A block of tx x ty cells (at most 256) holds planes k and k+1 with a
// one-cell x/y halo (periodic) in shared memory; plane k+2 is in flight in
// registers while k is computed.  The products on the tile's lower halo
// column and row are formed by two of its warps.
struct PredCoef {
  double qx, qy, qz;          // dxi/4, dyi/4, dzi/4 (stage 3: times f2)
  double vx, vy, vz, vc;      // visc dxi^2 .., -2 (vx + vy + vz) (stage 3: times f2)
  double gx, gy, gz;          // -f1 dxi ..
  double f2, mf3;             // f1 (stage 1) or f2, -f3
  double bc;                  // buoyancy factor (stage 3: times f2)
};
template <int STAGE, bool BUOY>
__global__ void __launch_bounds__(256, 2) k_predict_d(Geo g, const double *__restrict__ u, const double *__restrict__ v,
                                                      const double *__restrict__ w, const double *__restrict__ p,
                                                      double *__restrict__ ru, double *__restrict__ rv,
                                                      double *__restrict__ rw, double *__restrict__ fu,
                                                      double *__restrict__ fv, double *__restrict__ fw, PredCoef q,
                                                      const double *__restrict__ cb, int tx, int ty, int kc) {
  extern __shared__ __align__(16) double smd[];
  const int hx = tx + 2, hn = hx * (ty + 2), qx = tx + 1, qn = qx * (ty + 1);
  double *su = smd, *sv = su + 2 * hn, *sw = sv + 2 * hn, *sp = sw + 2 * hn;  // two planes each
  double *qxx = sp + 2 * hn, *qyy = qxx + qn, *quv = qyy + qn, *quw = quv + qn, *qvw = quw + qn;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int i0 = blockIdx.x * tx, j0 = blockIdx.y * ty;
  const int k0 = 1 + blockIdx.z * kc, k1 = min(g.K, k0 + kc - 1);
  const long PL = g.plane;
  // this thread's elements of a haloed plane (at most two)
  int hoff[2];
  bool has[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = tid + e * nt;
    has[e] = t < hn;
    const int y = has[e] ? t / hx : 0, x = has[e] ? t - y * hx : 0;
    const int gi = (i0 - 1 + x + g.I) % g.I, gj = (j0 - 1 + y + g.J) % g.J;
    hoff[e] = gj * g.I + gi;
  }
  double nu[2], nv[2], nw[2], np_[2];
  auto fetch = [&](int kk) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (has[e]) {
        const long o = (long)kk * PL + hoff[e];
        nu[e] = u[o]; nv[e] = v[o]; nw[e] = w[o]; np_[e] = p[o];
      }
  };
  auto commit = [&](int kk) {
    const int b = (kk & 1) * hn;
#pragma unroll
    for (int e = 0; e < 2; ++e)
      if (has[e]) {
        const int t = b + tid + e * nt;
        su[t] = nu[e]; sv[t] = nv[e]; sw[t] = nw[e]; sp[t] = np_[e];
      }
  };
  fetch(k0 - 1);
  commit(k0 - 1);
  fetch(k0);
  commit(k0);
  fetch(k0 + 1);
  __syncthreads();
  const bool cell = tid < tx * ty;
  const int ly = cell ? tid / tx : 0, lx = cell ? tid - ly * tx : 0;
  const int i = i0 + lx, j = j0 + ly;
  const bool in = cell && i < g.I && j < g.J;
  const int ch = (ly + 1) * hx + lx + 1, cq = (ly + 1) * qx + lx + 1;
  // the fluxes through the block's lowest z faces, and the column's values
  double Um, Vm, Wm, U0, V0, W0, uwm, vwm, zzm;
  {
    const int a = ((k0 - 1) & 1) * hn + ch, b = (k0 & 1) * hn + ch;
    Um = su[a]; Vm = sv[a]; Wm = sw[a];
    U0 = su[b]; V0 = sv[b]; W0 = sw[b];
    uwm = (U0 + Um) * (sw[a + 1] + Wm);
    vwm = (sw[a + hx] + Wm) * (V0 + Vm);
    const double z = W0 + Wm;
    zzm = z * z;
  }
  __syncthreads();
  long c = (long)k0 * PL + (long)j * g.I + i;
  for (int k = k0; k <= k1; ++k, c += PL) {
    commit(k + 1);  // over plane k - 1, which no thread reads any more
    __syncthreads();
    if (k < k1) fetch(k + 2);
    const double *uk = su + (k & 1) * hn, *vk = sv + (k & 1) * hn, *wk = sw + (k & 1) * hn, *pk = sp + (k & 1) * hn;
    const double *ukp = su + ((k + 1) & 1) * hn, *vkp = sv + ((k + 1) & 1) * hn, *wkp = sw + ((k + 1) & 1) * hn;
    double Up = 0., Vp = 0., Wp = 0., xx = 0., yy = 0., zz = 0., uv = 0., uw = 0., vw = 0.;
    double au = 0., av = 0., aw = 0., du = 0., dv = 0., dw = 0.;
    if (cell) {
      Up = ukp[ch]; Vp = vkp[ch]; Wp = wkp[ch];
      const double Uip = uk[ch + 1], Ujp = uk[ch + hx], Vip = vk[ch + 1], Vjp = vk[ch + hx], Wip = wk[ch + 1],
                   Wjp = wk[ch + hx];
      const double sx = Uip + U0, sy = Vjp + V0, sz = Wp + W0;
      xx = sx * sx;
      yy = sy * sy;
      zz = sz * sz;
      uv = (Ujp + U0) * (Vip + V0);
      uw = (Up + U0) * (Wip + W0);
      vw = (Wjp + W0) * (Vp + V0);
      qxx[cq] = xx; qyy[cq] = yy; quv[cq] = uv; quw[cq] = uw; qvw[cq] = vw;
      // velocity and pressure gradient, then (stage 3, whose right-hand side
      // is not stored) everything added onto them, else the right-hand side
      // starts from the Laplacian alone
      const double P0 = pk[ch];
      du = fma(q.gx, pk[ch + 1] - P0, U0);
      dv = fma(q.gy, pk[ch + hx] - P0, V0);
      dw = fma(q.gz, sp[((k + 1) & 1) * hn + ch] - P0, W0);
      if (STAGE != 1 && in) {
        du = fma(q.mf3, ru[c], du);
        dv = fma(q.mf3, rv[c], dv);
        dw = fma(q.mf3, rw[c], dw);
      }
      au = STAGE == 3 ? fma(q.vc, U0, du) : q.vc * U0;
      av = STAGE == 3 ? fma(q.vc, V0, dv) : q.vc * V0;
      aw = STAGE == 3 ? fma(q.vc, W0, dw) : q.vc * W0;
      au = fma(q.vx, Uip + uk[ch - 1], fma(q.vy, Ujp + uk[ch - hx], fma(q.vz, Up + Um, au)));
      av = fma(q.vx, Vip + vk[ch - 1], fma(q.vy, Vjp + vk[ch - hx], fma(q.vz, Vp + Vm, av)));
      aw = fma(q.vx, Wip + wk[ch - 1], fma(q.vy, Wjp + wk[ch - hx], fma(q.vz, Wp + Wm, aw)));
      if constexpr (BUOY)
        if (in) aw = fma(q.bc, cb[c] + cb[c + PL], aw);  // momzbuoy
    }
    if (tid < tx) {  // row j0 - 1
      const int a = tid + 1, b = hx + tid + 1;
      const double s = vk[b] + vk[a];
      qyy[tid + 1] = s * s;
      quv[tid + 1] = (uk[b] + uk[a]) * (vk[a + 1] + vk[a]);
      qvw[tid + 1] = (wk[b] + wk[a]) * (vkp[a] + vk[a]);
    }
    const int lh = nt - 1 - tid;
    if (lh < ty) {  // column i0 - 1
      const int a = (lh + 1) * hx, o = (lh + 1) * qx;
      const double s = uk[a + 1] + uk[a];
      qxx[o] = s * s;
      quv[o] = (uk[a + hx] + uk[a]) * (vk[a + 1] + vk[a]);
      quw[o] = (ukp[a] + uk[a]) * (wk[a + 1] + wk[a]);
    }
    __syncthreads();
    if (cell) {
      au = fma(q.qx, qxx[cq - 1] - xx, fma(q.qy, quv[cq - qx] - uv, fma(q.qz, uwm - uw, au)));
      av = fma(q.qx, quv[cq - 1] - uv, fma(q.qy, qyy[cq - qx] - yy, fma(q.qz, vwm - vw, av)));
      aw = fma(q.qx, quw[cq - 1] - uw, fma(q.qy, qvw[cq - qx] - vw, fma(q.qz, zzm - zz, aw)));
      if (in) {
        fu[c] = STAGE == 3 ? au : fma(q.f2, au, du);
        fv[c] = STAGE == 3 ? av : fma(q.f2, av, dv);
        fw[c] = STAGE == 3 ? aw : fma(q.f2, aw, dw);
        if (STAGE != 3) {
          ru[c] = au;
          rv[c] = av;
          rw[c] = aw;
        }
      }
      uwm = uw; vwm = vw; zzm = zz;
      Um = U0; Vm = V0; Wm = W0;
      U0 = Up; V0 = Vp; W0 = Wp;
    }
  }
}

// FP32 predictor with 2.5D blocking: a 32 x 8 column tile marches along z
// through a chunk of planes, keeping the planes k-1, k, k+1 of u, v, w and
// k, k+1 of p (with a one-cell x/y halo, periodic) in shared memory, so each
// field is read from HBM about once.  The terms of k_predict, regrouped (below).
constexpr int PTX = 32, PTY = 8, PHX = PTX + 2, PHY = PTY + 2, PKC = 32;
// BUOY: momzbuoy from the scalar field cb (FP64).  A separate instantiation
// keeps the FP64 buoyancy instructions out of the kernel without a scalar:
// issued under a false predicate they still take FP64 issue slots, which on
// this GPU run at 1/64 of the FP32 rate.
template <int STAGE, bool BUOY>
__global__ void __launch_bounds__(PTX *PTY) k_predict_tiled(Geo g, const float *__restrict__ u,
                                                            const float *__restrict__ v,
                                                            const float *__restrict__ w,
                                                            const float *__restrict__ p, float *__restrict__ ru,
                                                            float *__restrict__ rv, float *__restrict__ rw,
                                                            float *__restrict__ fu, float *__restrict__ fv,
                                                            float *__restrict__ fw, float f1, float f2, float f3,
                                                            const double *__restrict__ cb, double bcoef) {
  __shared__ float su[3][PHY][PHX], sv[3][PHY][PHX], sw[3][PHY][PHX], sp[2][PHY][PHX];
  const int tx = threadIdx.x % PTX, ty = threadIdx.x / PTX;
  const int i0 = blockIdx.x * PTX, j0 = blockIdx.y * PTY;
  const int k0 = 1 + blockIdx.z * PKC, k1 = min(g.K, k0 + PKC - 1);
  const int i = i0 + tx, j = j0 + ty;
  const bool in = i < g.I && j < g.J;
  const int PL = g.I * g.J;  // 32-bit offsets: launched only for fields < 2^31 cells
  // this thread's halo elements (at most two of the PHY*PHX) and their
  // in-plane offsets, periodic in x and y (full wrap: tiles wider than the
  // grid reach beyond one period)
  constexpr int NH = PHY * PHX, NT = PTX * PTY;
  int hoff[2], hyx[2];
  bool has[2];
  for (int q = 0; q < 2; ++q) {
    const int e = threadIdx.x + q * NT;
    has[q] = e < NH;
    const int hy = has[q] ? e / PHX : 0, hx = has[q] ? e - hy * PHX : 0;
    int gi = (i0 - 1 + hx) % g.I, gj = (j0 - 1 + hy) % g.J;
    if (gi < 0) gi += g.I;
    if (gj < 0) gj += g.J;
    hoff[q] = gj * g.I + gi;
    hyx[q] = hy * PHX + hx;
  }
  // next plane in registers (u, v, w, p for each halo element)
  float nu[2], nv[2], nw[2], np_[2];
  auto fetch = [&](int kk) {
    for (int q = 0; q < 2; ++q)
      if (has[q]) {
        const int o = kk * PL + hoff[q];
        nu[q] = u[o]; nv[q] = v[o]; nw[q] = w[o]; np_[q] = p[o];
      }
  };
  auto commit = [&](int kk) {
    for (int q = 0; q < 2; ++q)
      if (has[q]) {
        (&su[kk % 3][0][0])[hyx[q]] = nu[q];
        (&sv[kk % 3][0][0])[hyx[q]] = nv[q];
        (&sw[kk % 3][0][0])[hyx[q]] = nw[q];
        (&sp[kk % 2][0][0])[hyx[q]] = np_[q];
      }
  };
  fetch(k0 - 1);
  commit(k0 - 1);
  fetch(k0);
  commit(k0);
  fetch(k0 + 1);
  const float dxi = (float)g.dxi, dyi = (float)g.dyi, dzi = (float)g.dzi, visc = (float)g.visc;
  const float qdxi = 0.25f * dxi, qdyi = 0.25f * dyi, qdzi = 0.25f * dzi;
  const float vdx2 = visc * dxi * dxi, vdy2 = visc * dyi * dyi, vdz2 = visc * dzi * dzi;
  for (int k = k0; k <= k1; ++k) {
    commit(k + 1);  // slots of k-2 (u, v, w) and k-1 (p) are free
    __syncthreads();
    if (k + 1 <= k1) fetch(k + 2);  // in flight while plane k is computed
    if (in) {
      const int cm = (k - 1) % 3, c0 = k % 3, cp = (k + 1) % 3;
      const int x = tx + 1, y = ty + 1;
      const float U0 = su[c0][y][x], Uip = su[c0][y][x + 1], Uim = su[c0][y][x - 1], Ujp = su[c0][y + 1][x],
                  Ujm = su[c0][y - 1][x], Ukp = su[cp][y][x], Ukm = su[cm][y][x];
      const float V0 = sv[c0][y][x], Vip = sv[c0][y][x + 1], Vim = sv[c0][y][x - 1], Vjp = sv[c0][y + 1][x],
                  Vjm = sv[c0][y - 1][x], Vkp = sv[cp][y][x], Vkm = sv[cm][y][x];
      const float W0 = sw[c0][y][x], Wip = sw[c0][y][x + 1], Wim = sw[c0][y][x - 1], Wjp = sw[c0][y + 1][x],
                  Wjm = sw[c0][y - 1][x], Wkp = sw[cp][y][x], Wkm = sw[cm][y][x];
      const float Vipjm = sv[c0][y - 1][x + 1], Wipkm = sw[cm][y][x + 1];
      const float Uimjp = su[c0][y + 1][x - 1], Wjpkm = sw[cm][y + 1][x];
      const float Uimkp = su[cp][y][x - 1], Vjmkp = sv[cp][y - 1][x];
      // momxad, momyad, momzad (mom.f90:21-50, 94-123, 170-199), the same
      // terms regrouped for the FP32 pipes: each of the three mixed products
      // that two equations share is formed once; q (a + b)^2 - q (c + d)^2
      // as one FMA; the diffusion from neighbour differences, which are
      // exact for neighbouring values within a factor of two.
      const float Puv = (Ujp + U0) * (Vip + V0);  // momx uvjp, momy uvip
      const float Puw = (Ukp + U0) * (Wip + W0);  // momx uwkp, momz uwip
      const float Pvw = (Wjp + W0) * (Vkp + V0);  // momy wvkp, momz vwjp
      float ru_new, rv_new, rw_new;
      {
        const float sp_ = Uip + U0, sm_ = Uim + U0;
        ru_new = qdxi * fmaf(sm_, sm_, -(sp_ * sp_)) + qdyi * ((Ujm + U0) * (Vipjm + Vjm) - Puv) +
                 qdzi * ((Ukm + U0) * (Wipkm + Wkm) - Puw) + vdx2 * ((Uip - U0) - (U0 - Uim)) +
                 vdy2 * ((Ujp - U0) - (U0 - Ujm)) + vdz2 * ((Ukp - U0) - (U0 - Ukm));
      }
      {
        const float sp_ = V0 + Vjp, sm_ = V0 + Vjm;
        rv_new = qdxi * ((Uim + Uimjp) * (V0 + Vim) - Puv) + qdyi * fmaf(sm_, sm_, -(sp_ * sp_)) +
                 qdzi * ((Wkm + Wjpkm) * (Vkm + V0) - Pvw) + vdx2 * ((Vip - V0) - (V0 - Vim)) +
                 vdy2 * ((Vjp - V0) - (V0 - Vjm)) + vdz2 * ((Vkp - V0) - (V0 - Vkm));
      }
      {
        const float sp_ = W0 + Wkp, sm_ = W0 + Wkm;
        rw_new = qdxi * ((W0 + Wim) * (Uim + Uimkp) - Puw) + qdyi * ((W0 + Wjm) * (Vjm + Vjmkp) - Pvw) +
                 qdzi * fmaf(sm_, sm_, -(sp_ * sp_)) + vdx2 * ((Wip - W0) - (W0 - Wim)) +
                 vdy2 * ((Wjp - W0) - (W0 - Wjm)) + vdz2 * ((Wkp - W0) - (W0 - Wkm));
      }
      // pressure gradient (momxp/momyp/momzp)
      const float P0 = sp[k % 2][y][x];
      const float gx = -dxi * (sp[k % 2][y][x + 1] - P0);
      const float gy = -dyi * (sp[k % 2][y + 1][x] - P0);
      const float gz = -dzi * (sp[(k + 1) % 2][y][x] - P0);
      const int c = k * PL + j * g.I + i;
      if constexpr (BUOY) rw_new = (float)(bcoef * (cb[c] + cb[c + PL])) + rw_new;  // momzbuoy
      float du = U0 + f1 * gx, dv = V0 + f1 * gy, dw = W0 + f1 * gz;
      if (STAGE == 1) {
        du = du + f1 * ru_new;
        dv = dv + f1 * rv_new;
        dw = dw + f1 * rw_new;
      } else {
        du = du + (f2 * ru_new - f3 * ru[c]);
        dv = dv + (f2 * rv_new - f3 * rv[c]);
        dw = dw + (f2 * rw_new - f3 * rw[c]);
      }
      fu[c] = du;
      fv[c] = dv;
      fw[c] = dw;
      if (STAGE != 3) {
        ru[c] = ru_new;
        rv[c] = rv_new;
        rw[c] = rw_new;
      }
    }
    __syncthreads();  // slot (k-1) % 3 is reloaded next
  }
}

// The same stage with two x-neighbouring cells per thread in packed FP32x2
// arithmetic (one instruction for both cells; the x neighbours of the pair
// come from three aligned 8-byte shared loads instead of six): 64 x 8 cells
// per block.  Three kernels stage the planes differently and share the
// arithmetic (pair_cells), so that they agree bit for bit:
//   k_predict_quad  rows of 72 cells from x = i0 - 4, loaded as 16-byte
//                   quads through registers one plane ahead (the default);
//   k_predict_pair  rows of 66 cells, one 4-byte load per cell;
//   k_predict_tma   the k_predict_quad rows, copied by the tensor-memory
//                   accelerator into a ring of four planes per field.
constexpr int QTX = 64, QTY = 8, QHY = QTY + 2, QROW = QTX + 4;
constexpr int TBX = QTX + 8, TBY = QTY + 2;  // quad / TMA rows: 72 cells from x = i0 - 4, 10 rows from y = j0 - 1
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 ld2(const float *row, int idx) { return *reinterpret_cast<const float2 *>(row + idx); }
__device__ __forceinline__ float2 mid(float2 a, float2 b) { return make_float2(a.y, b.x); }

struct PairCoef {
  float2 qdxi, qdyi, qdzi, vdx2, vdy2, vdz2, mdxi, mdyi, mdzi, F1, F2, mF3;
  __device__ PairCoef(const Geo &g, float f1, float f2_, float f3) {
    const float dxi = (float)g.dxi, dyi = (float)g.dyi, dzi = (float)g.dzi, visc = (float)g.visc;
    qdxi = f2(0.25f * dxi); qdyi = f2(0.25f * dyi); qdzi = f2(0.25f * dzi);
    vdx2 = f2(visc * dxi * dxi); vdy2 = f2(visc * dyi * dyi); vdz2 = f2(visc * dzi * dzi);
    mdxi = f2(-dxi); mdyi = f2(-dyi); mdzi = f2(-dzi);
    F1 = f2(f1); F2 = f2(f2_); mF3 = f2(-f3);
  }
};
// Planes k-1 (m), k (0), k+1 (p) of u, v, w and k, k+1 of p in shared
// memory, rows of RS cells; the pair's first cell at column x of row y.
struct PairPlanes {
  const float *um, *u0, *up, *vm, *v0, *vp, *wm, *w0, *wp, *p0, *pp;
};
// momxad, momyad, momzad (mom.f90:21-50, 94-123, 170-199), momxp..momzp and
// the rk1..rk3 update of two cells (global index c, c + 1; 32-bit: the
// tiled kernels run on fields of fewer than 2^31 cells)
template <int STAGE, bool BUOY, int RS>
__device__ __forceinline__ void pair_cells(const PairPlanes &P, int x, int y, int c, int PL, const PairCoef &q,
                                           float *__restrict__ ru, float *__restrict__ rv, float *__restrict__ rw,
                                           float *__restrict__ fu, float *__restrict__ fv, float *__restrict__ fw,
                                           const double *__restrict__ cb, double bcoef) {
  auto row = [&](const float *f, int yy) { return f + yy * RS; };
  // u
  const float *ur = row(P.u0, y);
  const float2 U0 = ld2(ur, x), UL = ld2(ur, x - 2), UR = ld2(ur, x + 2);
  const float2 Uip = mid(U0, UR), Uim = mid(UL, U0);
  const float2 Ujp = ld2(row(P.u0, y + 1), x), Ujm = ld2(row(P.u0, y - 1), x);
  const float2 Ukp = ld2(row(P.up, y), x), Ukm = ld2(row(P.um, y), x);
  const float2 Uimjp = mid(ld2(row(P.u0, y + 1), x - 2), Ujp), Uimkp = mid(ld2(row(P.up, y), x - 2), Ukp);
  // v
  const float *vr = row(P.v0, y);
  const float2 V0 = ld2(vr, x), VL = ld2(vr, x - 2), VR = ld2(vr, x + 2);
  const float2 Vip = mid(V0, VR), Vim = mid(VL, V0);
  const float2 Vjp = ld2(row(P.v0, y + 1), x), Vjm = ld2(row(P.v0, y - 1), x);
  const float2 Vkp = ld2(row(P.vp, y), x), Vkm = ld2(row(P.vm, y), x);
  const float2 Vipjm = mid(Vjm, ld2(row(P.v0, y - 1), x + 2)), Vjmkp = ld2(row(P.vp, y - 1), x);
  // w
  const float *wr = row(P.w0, y);
  const float2 W0 = ld2(wr, x), WL = ld2(wr, x - 2), WR = ld2(wr, x + 2);
  const float2 Wip = mid(W0, WR), Wim = mid(WL, W0);
  const float2 Wjp = ld2(row(P.w0, y + 1), x), Wjm = ld2(row(P.w0, y - 1), x);
  const float2 Wkp = ld2(row(P.wp, y), x), Wkm = ld2(row(P.wm, y), x);
  const float2 Wipkm = mid(Wkm, ld2(row(P.wm, y), x + 2)), Wjpkm = ld2(row(P.wm, y + 1), x);
  // the terms of k_predict_tiled in packed arithmetic
  const float2 Puv = mul2(add2(Ujp, U0), add2(Vip, V0));
  const float2 Puw = mul2(add2(Ukp, U0), add2(Wip, W0));
  const float2 Pvw = mul2(add2(Wjp, W0), add2(Vkp, V0));
  auto lap = [&](float2 cc, float2 xp, float2 xm, float2 yp, float2 ym, float2 zp, float2 zm) {
    const float2 dx_ = sub2(sub2(xp, cc), sub2(cc, xm)), dy_ = sub2(sub2(yp, cc), sub2(cc, ym)),
                 dz_ = sub2(sub2(zp, cc), sub2(cc, zm));
    return fma2(q.vdx2, dx_, fma2(q.vdy2, dy_, mul2(q.vdz2, dz_)));
  };
  auto sqd = [&](float2 a, float2 b) { return fma2(a, a, mul2(f2(-1.f), mul2(b, b))); };  // a^2 - b^2
  float2 ru_new, rv_new, rw_new;
  {
    const float2 sp_ = add2(Uip, U0), sm_ = add2(Uim, U0);
    ru_new = fma2(q.qdxi, sqd(sm_, sp_),
                  fma2(q.qdyi, sub2(mul2(add2(Ujm, U0), add2(Vipjm, Vjm)), Puv),
                       fma2(q.qdzi, sub2(mul2(add2(Ukm, U0), add2(Wipkm, Wkm)), Puw),
                            lap(U0, Uip, Uim, Ujp, Ujm, Ukp, Ukm))));
  }
  {
    const float2 sp_ = add2(V0, Vjp), sm_ = add2(V0, Vjm);
    rv_new = fma2(q.qdxi, sub2(mul2(add2(Uim, Uimjp), add2(V0, Vim)), Puv),
                  fma2(q.qdyi, sqd(sm_, sp_),
                       fma2(q.qdzi, sub2(mul2(add2(Wkm, Wjpkm), add2(Vkm, V0)), Pvw),
                            lap(V0, Vip, Vim, Vjp, Vjm, Vkp, Vkm))));
  }
  {
    const float2 sp_ = add2(W0, Wkp), sm_ = add2(W0, Wkm);
    rw_new = fma2(q.qdxi, sub2(mul2(add2(W0, Wim), add2(Uim, Uimkp)), Puw),
                  fma2(q.qdyi, sub2(mul2(add2(W0, Wjm), add2(Vjm, Vjmkp)), Pvw),
                       fma2(q.qdzi, sqd(sm_, sp_), lap(W0, Wip, Wim, Wjp, Wjm, Wkp, Wkm))));
  }
  // pressure gradient (momxp/momyp/momzp)
  const float *pr = row(P.p0, y);
  const float2 P0 = ld2(pr, x);
  const float2 gx = mul2(q.mdxi, sub2(mid(P0, ld2(pr, x + 2)), P0));
  const float2 gy = mul2(q.mdyi, sub2(ld2(row(P.p0, y + 1), x), P0));
  const float2 gz = mul2(q.mdzi, sub2(ld2(row(P.pp, y), x), P0));
  if constexpr (BUOY) {
    rw_new.x = (float)(bcoef * (cb[c] + cb[c + PL])) + rw_new.x;  // momzbuoy
    rw_new.y = (float)(bcoef * (cb[c + 1] + cb[c + 1 + PL])) + rw_new.y;
  }
  float2 du = fma2(q.F1, gx, U0), dv = fma2(q.F1, gy, V0), dw = fma2(q.F1, gz, W0);
  if (STAGE == 1) {
    du = fma2(q.F1, ru_new, du);
    dv = fma2(q.F1, rv_new, dv);
    dw = fma2(q.F1, rw_new, dw);
  } else {
    const float2 ou = *reinterpret_cast<const float2 *>(ru + c), ov = *reinterpret_cast<const float2 *>(rv + c),
                 ow = *reinterpret_cast<const float2 *>(rw + c);
    du = add2(du, fma2(q.F2, ru_new, mul2(q.mF3, ou)));
    dv = add2(dv, fma2(q.F2, rv_new, mul2(q.mF3, ov)));
    dw = add2(dw, fma2(q.F2, rw_new, mul2(q.mF3, ow)));
  }
  *reinterpret_cast<float2 *>(fu + c) = du;
  *reinterpret_cast<float2 *>(fv + c) = dv;
  *reinterpret_cast<float2 *>(fw + c) = dw;
  if (STAGE != 3) {
    *reinterpret_cast<float2 *>(ru + c) = ru_new;
    *reinterpret_cast<float2 *>(rv + c) = rv_new;
    *reinterpret_cast<float2 *>(rw + c) = rw_new;
  }
}

#define PREDICT_ARGS                                                                                          \
  Geo g, const float *__restrict__ u, const float *__restrict__ v, const float *__restrict__ w,               \
      const float *__restrict__ p, float *__restrict__ ru, float *__restrict__ rv, float *__restrict__ rw,    \
      float *__restrict__ fu, float *__restrict__ fv, float *__restrict__ fw, float f1, float f2_, float f3,  \
      const double *__restrict__ cb, double bcoef, int kc

template <int STAGE, bool BUOY>
__global__ void __launch_bounds__(QTX / 2 * QTY, 3) k_predict_pair(PREDICT_ARGS) {
  // row layout: [pad, x = i0 - 1, x = i0 .. i0 + 63, x = i0 + 64, pad]
  __shared__ __align__(16) float su[3][QHY][QROW], sv[3][QHY][QROW], sw[3][QHY][QROW], sp[2][QHY][QROW];
  constexpr int NT = QTX / 2 * QTY, NH = QHY * (QTX + 2), HQ = (NH + NT - 1) / NT;
  const int tx = threadIdx.x % (QTX / 2), ty = threadIdx.x / (QTX / 2);
  const int i0 = blockIdx.x * QTX, j0 = blockIdx.y * QTY;
  const int k0 = 1 + blockIdx.z * kc, k1 = min(g.K, k0 + kc - 1);
  const int i = i0 + 2 * tx, j = j0 + ty;
  const bool in = i < g.I && j < g.J;  // I even: i + 1 < I as well
  const int PL = g.I * g.J;  // 32-bit offsets: launched only for fields < 2^31 cells
  int hoff[HQ], hyx[HQ];
  bool has[HQ];
#pragma unroll
  for (int q = 0; q < HQ; ++q) {
    const int e = threadIdx.x + q * NT;
    has[q] = e < NH;
    const int hy = has[q] ? e / (QTX + 2) : 0, hx = has[q] ? e - hy * (QTX + 2) : 0;
    int gi = (i0 - 1 + hx) % g.I, gj = (j0 - 1 + hy) % g.J;
    if (gi < 0) gi += g.I;
    if (gj < 0) gj += g.J;
    hoff[q] = gj * g.I + gi;
    hyx[q] = hy * QROW + hx + 1;
  }
  float nu[HQ], nv[HQ], nw[HQ], np_[HQ];
  auto fetch = [&](int kk) {
#pragma unroll
    for (int q = 0; q < HQ; ++q)
      if (has[q]) {
        const int o = kk * PL + hoff[q];
        nu[q] = u[o]; nv[q] = v[o]; nw[q] = w[o]; np_[q] = p[o];
      }
  };
  auto commit = [&](int kk) {
#pragma unroll
    for (int q = 0; q < HQ; ++q)
      if (has[q]) {
        (&su[kk % 3][0][0])[hyx[q]] = nu[q];
        (&sv[kk % 3][0][0])[hyx[q]] = nv[q];
        (&sw[kk % 3][0][0])[hyx[q]] = nw[q];
        (&sp[kk % 2][0][0])[hyx[q]] = np_[q];
      }
  };
  fetch(k0 - 1);
  commit(k0 - 1);
  fetch(k0);
  commit(k0);
  fetch(k0 + 1);
  const PairCoef cf(g, f1, f2_, f3);
  for (int k = k0; k <= k1; ++k) {
    commit(k + 1);
    __syncthreads();
    if (k + 1 <= k1) fetch(k + 2);
    if (in) {
      const int cm = (k - 1) % 3, c0 = k % 3, cp = (k + 1) % 3;
      const PairPlanes P{&su[cm][0][0], &su[c0][0][0], &su[cp][0][0], &sv[cm][0][0], &sv[c0][0][0],
                         &sv[cp][0][0], &sw[cm][0][0], &sw[c0][0][0], &sw[cp][0][0], &sp[k % 2][0][0],
                         &sp[(k + 1) % 2][0][0]};
      pair_cells<STAGE, BUOY, QROW>(P, 2 * tx + 2, ty + 1, k * PL + j * g.I + i, PL, cf, ru, rv, rw, fu,
                                    fv, fw, cb, bcoef);
    }
    __syncthreads();
  }
}

// Quads: the block's 18 x 10 quads of a plane (16-byte aligned with I a
// multiple of 4, so that a quad never straddles the periodic wrap, which is
// applied to whole quads) are read by its first 180 threads, one quad of
// each field per thread, into registers one plane ahead.
constexpr int QQX = TBX / 4, NQUAD = QQX * TBY;
template <int STAGE, bool BUOY>
__global__ void __launch_bounds__(QTX / 2 * QTY, 3) k_predict_quad(PREDICT_ARGS) {
  __shared__ __align__(16) float su[3][TBY][TBX], sv[3][TBY][TBX], sw[3][TBY][TBX], sp[2][TBY][TBX];
  const int tx = threadIdx.x % (QTX / 2), ty = threadIdx.x / (QTX / 2);
  const int i0 = blockIdx.x * QTX, j0 = blockIdx.y * QTY;
  const int k0 = 1 + blockIdx.z * kc, k1 = min(g.K, k0 + kc - 1);
  const int i = i0 + 2 * tx, j = j0 + ty;
  const bool in = i < g.I && j < g.J;
  const int PL = g.I * g.J;  // 32-bit offsets: launched only for fields < 2^31 cells
  const bool has = threadIdx.x < NQUAD;
  const int qy = threadIdx.x / QQX, qx = threadIdx.x - qy * QQX;
  const int gx = (((i0 - 4 + 4 * qx) % g.I) + g.I) % g.I, gy = (((j0 - 1 + qy) % g.J) + g.J) % g.J;
  const int qoff = gy * g.I + gx, qsm = qy * TBX + 4 * qx;
  float4 nu, nv, nw, np_;
  auto fetch = [&](int kk) {
    if (has) {
      const int o = kk * PL + qoff;
      nu = __ldg(reinterpret_cast<const float4 *>(u + o));
      nv = __ldg(reinterpret_cast<const float4 *>(v + o));
      nw = __ldg(reinterpret_cast<const float4 *>(w + o));
      np_ = __ldg(reinterpret_cast<const float4 *>(p + o));
    }
  };
  auto commit = [&](int kk) {
    if (has) {
      *reinterpret_cast<float4 *>(&su[kk % 3][0][0] + qsm) = nu;
      *reinterpret_cast<float4 *>(&sv[kk % 3][0][0] + qsm) = nv;
      *reinterpret_cast<float4 *>(&sw[kk % 3][0][0] + qsm) = nw;
      *reinterpret_cast<float4 *>(&sp[kk % 2][0][0] + qsm) = np_;
    }
  };
  fetch(k0 - 1);
  commit(k0 - 1);
  fetch(k0);
  commit(k0);
  fetch(k0 + 1);
  const PairCoef cf(g, f1, f2_, f3);
  for (int k = k0; k <= k1; ++k) {
    commit(k + 1);
    __syncthreads();
    if (k + 1 <= k1) fetch(k + 2);
    if (in) {
      const int cm = (k - 1) % 3, c0 = k % 3, cp = (k + 1) % 3;
      const PairPlanes P{&su[cm][0][0], &su[c0][0][0], &su[cp][0][0], &sv[cm][0][0], &sv[c0][0][0],
                         &sv[cp][0][0], &sw[cm][0][0], &sw[c0][0][0], &sw[cp][0][0], &sp[k % 2][0][0],
                         &sp[(k + 1) % 2][0][0]};
      pair_cells<STAGE, BUOY, TBX>(P, 2 * tx + 4, ty + 1, k * PL + j * g.I + i, PL, cf, ru, rv, rw, fu,
                                   fv, fw, cb, bcoef);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// The quad rows staged by the tensor-memory accelerator: one
// cp.async.bulk.tensor load per field and plane brings the block's 72 x 10
// box (x from i0 - 4, 16-byte aligned) from HBM into shared memory,
// completing on the slot's mbarrier.  Four slots per field hold the planes
// k-1, k, k+1 being read and k+2 in flight; the next load is issued into the
// slot of k-1 once the block has finished reading it.  Box cells outside the
// domain (filled with zeros by the copy) are patched with their periodic
// images by plain loads, fetched one plane ahead into registers.  Measured
// at 256^3 this stages no faster than the quads through registers (the
// waits for the copies stay on the critical path at every prefetch depth
// tried), so it is selectable (IBM_PREDICTOR_TMA), not the default.
// ---------------------------------------------------------------------------
constexpr int TSLOT = ((TBX * TBY * 4 + 127) / 128) * 128 / 4;     // floats per field slot (128-byte aligned)
constexpr int TNS = 4;                                             // slots per field
constexpr int TPATCH = (QTX + 2) * TBY;                            // cells of the box the stencils read
constexpr int TPQ = (TPATCH + QTX / 2 * QTY - 1) / (QTX / 2 * QTY);  // patch cells per thread
constexpr size_t TMA_SMEM = (size_t)TNS * 4 * TSLOT * 4 + 128;
struct TmaFields {
  CUtensorMap u, v, w, p;
};
namespace {
__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool tma_wait(uint64_t *bar, uint32_t parity) {
  for (long it = 0; it < (1L << 22); ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(sm_addr(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_plane(const TmaFields &tm, float *slot, uint64_t *bar, int x, int y, int z) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sm_addr(bar)), "r"(4 * TBX * TBY * 4)
               : "memory");
  const CUtensorMap *m[4] = {&tm.u, &tm.v, &tm.w, &tm.p};
#pragma unroll
  for (int f = 0; f < 4; ++f)
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(sm_addr(slot + f * TSLOT)),
        "l"(reinterpret_cast<uint64_t>(m[f])), "r"(x), "r"(y), "r"(z), "r"(sm_addr(bar))
        : "memory");
}
}  // namespace

template <int STAGE, bool BUOY>
__global__ void __launch_bounds__(QTX / 2 * QTY, 3) k_predict_tma(PREDICT_ARGS, const __grid_constant__ TmaFields tm,
                                                                 int *__restrict__ err) {
  extern __shared__ __align__(128) unsigned char tma_sm[];
  float *sbase = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(tma_sm) + 127) & ~uintptr_t(127));
  __shared__ __align__(8) uint64_t bar[TNS];
  constexpr int NT = QTX / 2 * QTY;
  const int tx = threadIdx.x % (QTX / 2), ty = threadIdx.x / (QTX / 2);
  const int i0 = blockIdx.x * QTX, j0 = blockIdx.y * QTY;
  const int k0 = 1 + blockIdx.z * kc, k1 = min(g.K, k0 + kc - 1);
  const int pfirst = k0 - 1, plast = k1 + 1;  // planes this block reads
  const int i = i0 + 2 * tx, j = j0 + ty;
  const bool in = i < g.I && j < g.J;  // I even: i + 1 < I as well
  const int PL = g.I * g.J;  // 32-bit offsets: launched only for fields < 2^31 cells
  auto sidx = [&](int P) { return (P - pfirst) & (TNS - 1); };
  auto slot_of = [&](int P) { return sbase + sidx(P) * 4 * TSLOT; };
  auto parity_of = [&](int P) { return (uint32_t)(((P - pfirst) / TNS) & 1); };
  if (threadIdx.x == 0) {
    for (int q = 0; q < TNS; ++q) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr(&bar[q])));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int P = pfirst; P <= min(plast, pfirst + TNS - 1); ++P)
      tma_load_plane(tm, slot_of(P), &bar[sidx(P)], i0 - 4, j0 - 1, P);
  // box cells outside the domain that the stencils read: their periodic
  // images by plain loads (none in tiles away from the domain's edges).
  // Thread cell q is e = tid + q NT of the (QTX + 2) x TBY region from x =
  // i0 - 1; bit q of pmask marks the ones outside.
  auto patch_cell = [&](int q, int &hyx, int &off) {
    const int e = threadIdx.x + q * NT;
    const int hy = e / (QTX + 2), hx = e - hy * (QTX + 2) + 3;
    const int gx = i0 - 4 + hx, gy = j0 - 1 + hy;
    hyx = hy * TBX + hx;
    off = (((gy % g.J) + g.J) % g.J) * g.I + ((gx % g.I) + g.I) % g.I;
    return e < TPATCH && (gx < 0 || gx >= g.I || gy < 0 || gy >= g.J);
  };
  unsigned pmask = 0;
#pragma unroll
  for (int q = 0; q < TPQ; ++q) {
    int a, b;
    if (patch_cell(q, a, b)) pmask |= 1u << q;
  }
  const bool edge = __syncthreads_or(pmask != 0) != 0;  // the block patches cells
  float nu[TPQ], nv[TPQ], nw[TPQ], np_[TPQ];
  auto fetch = [&](int P) {
#pragma unroll
    for (int q = 0; q < TPQ; ++q)
      if (pmask & (1u << q)) {
        int a, b;
        patch_cell(q, a, b);
        const int o = P * PL + b;
        nu[q] = u[o]; nv[q] = v[o]; nw[q] = w[o]; np_[q] = p[o];
      }
  };
  auto commit = [&](int P) {
    float *sl = slot_of(P);
#pragma unroll
    for (int q = 0; q < TPQ; ++q)
      if (pmask & (1u << q)) {
        int a, b;
        patch_cell(q, a, b);
        sl[a] = nu[q];
        sl[TSLOT + a] = nv[q];
        sl[2 * TSLOT + a] = nw[q];
        sl[3 * TSLOT + a] = np_[q];
      }
  };
  // bounded wait on plane P, the same outcome in every thread
  bool failed = false;
  auto wait_plane = [&](int P) {
    const bool ok = tma_wait(&bar[sidx(P)], parity_of(P));
    failed = __syncthreads_or(!ok) != 0;
  };
  int issued = min(plast, pfirst + TNS - 1);  // last plane whose load is issued
  int waited = pfirst - 1;                    // last plane waited for
  fetch(pfirst);
  wait_plane(pfirst);
  waited = pfirst;
  if (!failed) {
    commit(pfirst);
    fetch(pfirst + 1);
    wait_plane(pfirst + 1);
    waited = pfirst + 1;
  }
  if (!failed) {
    commit(pfirst + 1);
    fetch(pfirst + 2);
  }
  const PairCoef cf(g, f1, f2_, f3);
  for (int k = k0; k <= k1 && !failed; ++k) {
    wait_plane(k + 1);
    if (failed) break;
    waited = k + 1;
    if (edge) {
      commit(k + 1);
      if (k + 2 <= plast) fetch(k + 2);
      __syncthreads();
    }
    if (in) {
      const float *Sm = slot_of(k - 1), *S0 = slot_of(k), *Sp = slot_of(k + 1);
      const PairPlanes P{Sm, S0, Sp, Sm + TSLOT, S0 + TSLOT, Sp + TSLOT, Sm + 2 * TSLOT, S0 + 2 * TSLOT,
                         Sp + 2 * TSLOT, S0 + 3 * TSLOT, Sp + 3 * TSLOT};
      pair_cells<STAGE, BUOY, TBX>(P, 2 * tx + 4, ty + 1, k * PL + j * g.I + i, PL, cf, ru, rv, rw, fu,
                                   fv, fw, cb, bcoef);
    }
    // the slot of plane k - 1 is free once every thread is past this point;
    // the patches written into it are ordered before the next copy into it
    if (pmask) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && issued < plast) {
      ++issued;
      tma_load_plane(tm, slot_of(issued), &bar[sidx(issued)], i0 - 4, j0 - 1, issued);
    }
  }
  if (failed && threadIdx.x == 0) {
    // a copy did not complete within the limit: flag it, and give the copies
    // still in flight a bounded time to land before the block exits
    atomicExch(err, 1);
    for (int P = waited + 1; P <= issued; ++P) tma_wait(&bar[sidx(P)], parity_of(P));
  }
}

namespace {
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }();
  return fn;
}
// 3-D map of one FP32 cell field (I, J, K + 2), box 72 x 10 x 1
bool encode_field_map(CUtensorMap *m, const Geo &g, const float *f) {
  auto enc = tensor_map_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(f) & 15)) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)g.I, (cuuint64_t)g.J, (cuuint64_t)(g.K + 2)};
  const cuuint64_t strides[2] = {(cuuint64_t)g.I * 4, (cuuint64_t)g.I * g.J * 4};
  const cuuint32_t box[3] = {(cuuint32_t)TBX, (cuuint32_t)TBY, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(f), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
int sm_count() {
  static int nsm = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n;
  }();
  return nsm;
}
// Planes per z chunk of a kernel that marches `tiles` column tiles along z with
// `slots` resident blocks: the split that keeps the block waves fullest, net
// of what a chunk costs in addition (in planes), chunks of at most maxkc planes
int zchunk(int K, int tiles, int slots, int maxkc, double extra) {
  slots = std::max(1, slots);
  const int most = std::min(K, 64);
  int kc = K;
  double best = -1.;
  for (int nz = 1; nz <= most; ++nz) {
    const int kcz = (K + nz - 1) / nz, nb = tiles * ((K + kcz - 1) / kcz);
    if (kcz > maxkc && nz < most) continue;
    const double waves = (double)nb / slots, eff = waves / std::ceil(waves) * kcz / (kcz + extra);
    if (eff > best + 1e-9) { best = eff; kc = kcz; }
  }
  return kc;
}
// the FP32 predictors, nbs resident blocks per SM: two halo planes a chunk
int predict_zchunk(const Geo &g, int nbs, int maxkc) {
  return zchunk(g.K, ((g.I + QTX - 1) / QTX) * ((g.J + QTY - 1) / QTY), sm_count() * nbs, maxkc, 2.);
}
int quad_blocks_per_sm() {
  static int n = [] {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_predict_quad<2, false>, QTX / 2 * QTY, 0) != cudaSuccess)
      return 3;
    return nb > 0 ? nb : 3;
  }();
  return n;
}
int tma_blocks_per_sm() {
  static int n = [] {
    int nb = 0;
    for (auto k : {k_predict_tma<1, false>, k_predict_tma<2, false>, k_predict_tma<3, false>,
                   k_predict_tma<1, true>, k_predict_tma<2, true>, k_predict_tma<3, true>})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TMA_SMEM) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_predict_tma<2, false>, QTX / 2 * QTY, TMA_SMEM) !=
        cudaSuccess)
      return 0;
    return nb;
  }();
  return n;
}
}  // namespace

// The TMA-staged stage: false when it does not apply (rows not a multiple of
// 4 cells, no tensor-map encoder).
bool launch_predict_tma(cudaStream_t s, const Geo &g, int stage, const float *u, const float *v, const float *w,
                        const float *p, float *ru, float *rv, float *rw, float *fu, float *fv, float *fw, float a,
                        float b, float c, const double *cb, double bcoef, int *err) {
  if (!err || g.I % 4 != 0 || g.nfield >= (1L << 31)) return false;
  const int nbs = tma_blocks_per_sm();
  if (nbs <= 0) return false;
  TmaFields tm;
  if (!encode_field_map(&tm.u, g, u) || !encode_field_map(&tm.v, g, v) || !encode_field_map(&tm.w, g, w) ||
      !encode_field_map(&tm.p, g, p))
    return false;
  // at most 24 planes a chunk (measured fastest at 256^3)
  const int kc = predict_zchunk(g, nbs, 24);
  dim3 grd((g.I + QTX - 1) / QTX, (g.J + QTY - 1) / QTY, (g.K + kc - 1) / kc);
  auto go = [&](auto kern) {
    kern<<<grd, QTX / 2 * QTY, TMA_SMEM, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, a, b, c, cb, bcoef, kc, tm, err);
  };
  if (cb) {
    if (stage == 1) go(k_predict_tma<1, true>);
    else if (stage == 2) go(k_predict_tma<2, true>);
    else go(k_predict_tma<3, true>);
  } else {
    if (stage == 1) go(k_predict_tma<1, false>);
    else if (stage == 2) go(k_predict_tma<2, false>);
    else go(k_predict_tma<3, false>);
  }
  return true;
}

// Tiles of the FP64 predictor: equal parts of at most 32 x-cells, then as many
// rows as 256 threads take in equal parts (the kernel's cost is its FP64
// instructions, so cells beyond the grid count in full; coalescing hardly
// does).  z chunks by the block-wave model below; a chunk costs the fluxes
// through its lowest faces and two planes' loads in addition, about 0.4 planes.
void launch_predict_d(cudaStream_t s, const Geo &g, int stage, const double *u, const double *v, const double *w,
                      const double *p, double *ru, double *rv, double *rw, double *fu, double *fv, double *fw,
                      double f1, double f2, double f3, const double *cb, double bcoef) {
  auto parts = [](int n, int most) {
    const int m = (n + most - 1) / most;
    return (n + m - 1) / m;
  };
  const int tx = parts(g.I, 32), ty = parts(g.J, 256 / tx), nt = (tx * ty + 31) / 32 * 32;
  const size_t smem = (size_t)(8 * (tx + 2) * (ty + 2) + 5 * (tx + 1) * (ty + 1)) * sizeof(double);
  PredCoef q;
  const double f = stage == 3 ? f2 : 1.;
  q.qx = f * 0.25 * g.dxi; q.qy = f * 0.25 * g.dyi; q.qz = f * 0.25 * g.dzi;
  q.vx = f * (g.visc * g.dxi * g.dxi); q.vy = f * (g.visc * g.dyi * g.dyi); q.vz = f * (g.visc * g.dzi * g.dzi);
  q.vc = -2. * (q.vx + q.vy + q.vz);
  q.gx = -f1 * g.dxi; q.gy = -f1 * g.dyi; q.gz = -f1 * g.dzi;
  q.f2 = stage == 1 ? f1 : f2;
  q.mf3 = -f3;
  q.bc = f * bcoef;
  const int tiles = ((g.I + tx - 1) / tx) * ((g.J + ty - 1) / ty);
  const int kc = zchunk(g.K, tiles, sm_count() * 2, 64, 0.4);
  dim3 grd((g.I + tx - 1) / tx, (g.J + ty - 1) / ty, (g.K + kc - 1) / kc);
  auto go = [&](auto kern) { kern<<<grd, nt, smem, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, q, cb, tx, ty, kc); };
  if (cb) {
    if (stage == 1) go(k_predict_d<1, true>);
    else if (stage == 2) go(k_predict_d<2, true>);
    else go(k_predict_d<3, true>);
  } else {
    if (stage == 1) go(k_predict_d<1, false>);
    else if (stage == 2) go(k_predict_d<2, false>);
    else go(k_predict_d<3, false>);
  }
}

template <typename TU, typename T>
void launch_predict(cudaStream_t s, const Geo &g, int stage, const TU *u, const TU *v, const TU *w, const TU *p,
                    T *ru, T *rv, T *rw, T *fu, T *fv, T *fw, double f1, double f2, double f3, const double *cb,
                    double bcoef, int kind, int *err) {
  if constexpr (sizeof(T) == 4 && sizeof(TU) == 4) {
    if (g.nfield < (1L << 31)) {
    const float a = (float)f1, b = (float)f2, c = (float)f3;
    if (kind == IBM_PREDICTOR_TMA &&
        launch_predict_tma(s, g, stage, u, v, w, p, ru, rv, rw, fu, fv, fw, a, b, c, cb, bcoef, err))
      return;
    const int kc = predict_zchunk(g, quad_blocks_per_sm(), 64);
    dim3 gq((g.I + QTX - 1) / QTX, (g.J + QTY - 1) / QTY, (g.K + kc - 1) / kc);
    auto goq = [&](auto kern) {
      kern<<<gq, QTX / 2 * QTY, 0, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, a, b, c, cb, bcoef, kc);
    };
    if (g.I % 4 == 0 && (kind == IBM_PREDICTOR_AUTO || kind == IBM_PREDICTOR_TMA)) {
      if (cb) {
        if (stage == 1) goq(k_predict_quad<1, true>);
        else if (stage == 2) goq(k_predict_quad<2, true>);
        else goq(k_predict_quad<3, true>);
      } else {
        if (stage == 1) goq(k_predict_quad<1, false>);
        else if (stage == 2) goq(k_predict_quad<2, false>);
        else goq(k_predict_quad<3, false>);
      }
      return;
    }
    if (g.I % 2 == 0 && kind != IBM_PREDICTOR_CELLS) {
      if (cb) {
        if (stage == 1) goq(k_predict_pair<1, true>);
        else if (stage == 2) goq(k_predict_pair<2, true>);
        else goq(k_predict_pair<3, true>);
      } else {
        if (stage == 1) goq(k_predict_pair<1, false>);
        else if (stage == 2) goq(k_predict_pair<2, false>);
        else goq(k_predict_pair<3, false>);
      }
      return;
    }
    dim3 grd((g.I + PTX - 1) / PTX, (g.J + PTY - 1) / PTY, (g.K + PKC - 1) / PKC);
    auto go = [&](auto kern) { kern<<<grd, PTX * PTY, 0, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, a, b, c, cb, bcoef); };
    if (cb) {
      if (stage == 1) go(k_predict_tiled<1, true>);
      else if (stage == 2) go(k_predict_tiled<2, true>);
      else go(k_predict_tiled<3, true>);
    } else {
      if (stage == 1) go(k_predict_tiled<1, false>);
      else if (stage == 2) go(k_predict_tiled<2, false>);
      else go(k_predict_tiled<3, false>);
    }
    return;
    }
  }
  if constexpr (sizeof(T) == 8) {
    launch_predict_d(s, g, stage, u, v, w, p, ru, rv, rw, fu, fv, fw, f1, f2, f3, cb, bcoef);
  } else {
    dim3 blk(64, 4, 1);
    dim3 grd((g.I + 63) / 64, (g.J + 3) / 4, g.K);
    if (stage == 1)
      k_predict<TU, T, 1><<<grd, blk, 0, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, (T)f1, (T)f2, (T)f3, cb, bcoef);
    else if (stage == 2)
      k_predict<TU, T, 2><<<grd, blk, 0, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, (T)f1, (T)f2, (T)f3, cb, bcoef);
    else
      k_predict<TU, T, 3><<<grd, blk, 0, s>>>(g, u, v, w, p, ru, rv, rw, fu, fv, fw, (T)f1, (T)f2, (T)f3, cb, bcoef);
  }
}
template void launch_predict<double, double>(cudaStream_t, const Geo &, int, const double *, const double *,
                                             const double *, const double *, double *, double *, double *,
                                             double *, double *, double *, double, double, double, const double *,
                                             double, int, int *);
template void launch_predict<float, float>(cudaStream_t, const Geo &, int, const float *, const float *,
                                           const float *, const float *, float *, float *, float *, float *,
                                           float *, float *, double, double, double, const double *, double, int,
                                           int *);

// ---------------------------------------------------------------------------
// Scalar: scalad (scal.f90:11-58) fused with the dcdt update of rk1..rk3
// (rk3.f90:48,78 / 151,188 / 266,300).  STAGE 1: cnext = c + f1*RHS,
// rhs_old = RHS; STAGE 2/3: cnext = c + (f2*RHS - f3*rhs_old), stage 2 stores
// rhs_old = RHS.  cnext becomes cnew after the projection (main.f90:374-376).
// ---------------------------------------------------------------------------
template <typename TU, int STAGE>
__global__ void __launch_bounds__(256) k_scalar_stage(Geo g, const TU *__restrict__ u, const TU *__restrict__ v,
                                                      const TU *__restrict__ w, const double *__restrict__ cf,
                                                      double *__restrict__ rc, double *__restrict__ cnext,
                                                      double kappa, double f1, double f2, double f3) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z + 1;
  if (i >= g.I || j >= g.J) return;
  const long c = fidx(g, i, j, k);
  const long cip = fidx(g, i + 1 == g.I ? 0 : i + 1, j, k), cim = fidx(g, i == 0 ? g.I - 1 : i - 1, j, k);
  const long cjp = fidx(g, i, j + 1 == g.J ? 0 : j + 1, k), cjm = fidx(g, i, j == 0 ? g.J - 1 : j - 1, k);
  const long ckp = c + g.plane, ckm = c - g.plane;
  const double dxi = g.dxi, dyi = g.dyi, dzi = g.dzi;
  const double C0 = cf[c], Cip = cf[cip], Cim = cf[cim], Cjp = cf[cjp], Cjm = cf[cjm], Ckp = cf[ckp], Ckm = cf[ckm];
  const double ucip = 0.5 * (double)u[c] * (Cip + C0);
  const double ucim = 0.5 * (double)u[cim] * (C0 + Cim);
  const double vcjp = 0.5 * (double)v[c] * (Cjp + C0);
  const double vcjm = 0.5 * (double)v[cjm] * (C0 + Cjm);
  const double wckp = 0.5 * (double)w[c] * (Ckp + C0);
  const double wckm = 0.5 * (double)w[ckm] * (C0 + Ckm);
  const double dcdxp = (Cip - C0) * dxi, dcdxm = (C0 - Cim) * dxi;
  const double dcdyp = (Cjp - C0) * dyi, dcdym = (C0 - Cjm) * dyi;
  const double dcdzp = (Ckp - C0) * dzi, dcdzm = (C0 - Ckm) * dzi;
  const double rhs = dxi * (-ucip + ucim) + kappa * (dcdxp - dcdxm) * dxi + dyi * (-vcjp + vcjm) +
                     kappa * (dcdyp - dcdym) * dyi + dzi * (-wckp + wckm) + kappa * (dcdzp - dcdzm) * dzi;
  if (STAGE == 1) cnext[c] = C0 + f1 * rhs;
  else cnext[c] = C0 + (f2 * rhs - f3 * rc[c]);
  if (STAGE != 3) rc[c] = rhs;
}
template <typename TU>
void launch_scalar_stage(cudaStream_t s, const Geo &g, int stage, const TU *u, const TU *v, const TU *w,
                         const double *cf, double *rc, double *cnext, double kappa, double f1, double f2, double f3) {
  dim3 blk(64, 4, 1);
  dim3 grd((g.I + 63) / 64, (g.J + 3) / 4, g.K);
  if (stage == 1) k_scalar_stage<TU, 1><<<grd, blk, 0, s>>>(g, u, v, w, cf, rc, cnext, kappa, f1, f2, f3);
  else if (stage == 2) k_scalar_stage<TU, 2><<<grd, blk, 0, s>>>(g, u, v, w, cf, rc, cnext, kappa, f1, f2, f3);
  else k_scalar_stage<TU, 3><<<grd, blk, 0, s>>>(g, u, v, w, cf, rc, cnext, kappa, f1, f2, f3);
}
template void launch_scalar_stage<double>(cudaStream_t, const Geo &, int, const double *, const double *,
                                          const double *, const double *, double *, double *, double, double,
                                          double, double);
template void launch_scalar_stage<float>(cudaStream_t, const Geo &, int, const float *, const float *, const float *,
                                         const double *, double *, double *, double, double, double, double);

// boundscal (bound.f90:109-171): wall ghost planes of the scalar
__global__ void k_boundscal(Geo g, double *__restrict__ cf, int top_dirichlet, double top, int bot_dirichlet,
                            double bot) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < g.plane; e += (long)gridDim.x * blockDim.x) {
    const long t = (long)(g.K + 1) * g.plane + e, n = (long)g.K * g.plane + e;
    cf[t] = top_dirichlet ? 2 * top - cf[n] : cf[n];
    cf[e] = bot_dirichlet ? 2 * bot - cf[g.plane + e] : cf[g.plane + e];
  }
}
void launch_boundscal(cudaStream_t s, const Geo &g, double *cf, int top_dirichlet, double top, int bot_dirichlet,
                      double bot) {
  k_boundscal<<<(int)std::min<long>(1216, (g.plane + 255) / 256), 256, 0, s>>>(g, cf, top_dirichlet, top,
                                                                               bot_dirichlet, bot);
}

// ---------------------------------------------------------------------------
// correc (correc.f90:11-42) + pnew += p (main.f90:369-371) + bounduvw(unew)
// and boundp(pnew) z-ghosts (bound.f90:11-107).  phi holds the Poisson
// solution on planes 1..K; its Neumann ghost p(k1)=p(kmax) is implied.
// ---------------------------------------------------------------------------
template <typename TF, typename TPh, typename TU>
__global__ void __launch_bounds__(256) k_correc(Geo g, const TF *fu, const TF *fv, const TF *fw,
                                                const TPh *__restrict__ phi, TU *u, TU *v, TU *w,
                                                double *__restrict__ pn, float *__restrict__ pn32, double fi_,
                                                double fj_, double fk_) {
  // fu may alias u (the defect correction updates the state in place: each
  // thread reads and writes only its own cell of u/v/w)
  typedef TU T;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z + 1;
  if (i >= g.I || j >= g.J) return;
  const int ip = i + 1 == g.I ? 0 : i + 1;
  const int jp = j + 1 == g.J ? 0 : j + 1;
  const long PL = g.plane;
  const long c = fidx(g, i, j, k);
  const T fi = (T)fi_, fj = (T)fj_, fk = (T)fk_;
  const T P0 = (T)phi[c];
  const T Pip = (T)phi[fidx(g, ip, j, k)];
  const T Pjp = (T)phi[fidx(g, i, jp, k)];
  if (g.zper) {  // periodic z: p(k1) = p(1); w(kmax) is an unknown; ghost planes are copies
    const T Pkp = (k == g.K) ? (T)phi[c - (long)(g.K - 1) * PL] : (T)phi[c + PL];
    const T un = (T)fu[c] - fi * (Pip - P0);
    const T vn = (T)fv[c] - fj * (Pjp - P0);
    const T wn = (T)fw[c] - fk * (Pkp - P0);
    u[c] = un;
    v[c] = vn;
    w[c] = wn;
    const double pnn = pn[c] + (double)phi[c];
    pn[c] = pnn;
    if (pn32) pn32[c] = (float)pnn;
    const long gh = k == 1 ? c + (long)g.K * PL : (k == g.K ? c - (long)g.K * PL : -1);
    if (gh >= 0) {  // plane 1 -> ghost k1, plane K -> ghost 0
      u[gh] = un;
      v[gh] = vn;
      w[gh] = wn;
      pn[gh] = pnn;
      if (pn32) pn32[gh] = (float)pnn;
    }
    return;
  }
  const T Pkp = (k == g.K) ? P0 : (T)phi[c + PL];
  const T un = (T)fu[c] - fi * (Pip - P0);
  const T vn = (T)fv[c] - fj * (Pjp - P0);
  const T wn = (k == g.K) ? (T)0 : (T)fw[c] - fk * (Pkp - P0);
  u[c] = un;
  v[c] = vn;
  w[c] = wn;
  const double pnn = pn[c] + (double)phi[c];
  pn[c] = pnn;
  if (pn32) pn32[c] = (float)pnn;
  if (k == g.K) {
    const T sg = g.bc_top == IBM_BC_NOSLIP ? (T)-1 : (T)1;
    u[c + PL] = sg * un;
    v[c + PL] = sg * vn;
    pn[c + PL] = pnn;
    if (pn32) pn32[c + PL] = (float)pnn;
  }
  if (k == 1) {
    const T sg = g.bc_bot == IBM_BC_NOSLIP ? (T)-1 : (T)1;
    u[c - PL] = sg * un;
    v[c - PL] = sg * vn;
    w[c - PL] = (T)0;
    pn[c - PL] = pnn;
    if (pn32) pn32[c - PL] = (float)pnn;
  }
}

template <typename TF, typename TPh, typename TU>
void launch_correc(cudaStream_t s, const Geo &g, const TF *fu, const TF *fv, const TF *fw, const TPh *phi, TU *u,
                   TU *v, TU *w, double *pn, float *pn32, double fi, double fj, double fk) {
  dim3 blk(64, 4, 1);
  dim3 grd((g.I + 63) / 64, (g.J + 3) / 4, g.K);
  k_correc<TF, TPh, TU><<<grd, blk, 0, s>>>(g, fu, fv, fw, phi, u, v, w, pn, pn32, fi, fj, fk);
}
template void launch_correc<double, double, double>(cudaStream_t, const Geo &, const double *, const double *,
                                                    const double *, const double *, double *, double *, double *,
                                                    double *, float *, double, double, double);
template void launch_correc<float, float, float>(cudaStream_t, const Geo &, const float *, const float *,
                                                 const float *, const float *, float *, float *, float *, double *,
                                                 float *, double, double, double);

// Mixed form of the same update: FP32 velocity; pnew carried as the
// double-float pair (ph, pl), ph doubling as the FP32 pressure that the
// predictor reads.  fu may alias u (defect correction in place).
__global__ void __launch_bounds__(256) k_correc_mixed(Geo g, const float *fu, const float *fv, const float *fw,
                                                      const float *__restrict__ phi, float *u, float *v, float *w,
                                                      float *__restrict__ ph, float *__restrict__ pl, float fi,
                                                      float fj, float fk) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z + 1;
  if (i >= g.I || j >= g.J) return;
  const int ip = i + 1 == g.I ? 0 : i + 1;
  const int jp = j + 1 == g.J ? 0 : j + 1;
  const long PL = g.plane;
  const long c = fidx(g, i, j, k);
  const float P0 = phi[c];
  const float Pip = phi[fidx(g, ip, j, k)];
  const float Pjp = phi[fidx(g, i, jp, k)];
  const float Pkp = (k == g.K) ? P0 : phi[c + PL];
  const float un = fu[c] - fi * (Pip - P0);
  const float vn = fv[c] - fj * (Pjp - P0);
  const float wn = (k == g.K) ? 0.f : fw[c] - fk * (Pkp - P0);
  u[c] = un;
  v[c] = vn;
  w[c] = wn;
  float sh, sl;
  df_add(ph[c], pl[c], P0, 0.f, sh, sl);
  ph[c] = sh;
  pl[c] = sl;
  if (k == g.K) {
    const float sg = g.bc_top == IBM_BC_NOSLIP ? -1.f : 1.f;
    u[c + PL] = sg * un;
    v[c + PL] = sg * vn;
    ph[c + PL] = sh;
    pl[c + PL] = sl;
  }
  if (k == 1) {
    const float sg = g.bc_bot == IBM_BC_NOSLIP ? -1.f : 1.f;
    u[c - PL] = sg * un;
    v[c - PL] = sg * vn;
    w[c - PL] = 0.f;
    ph[c - PL] = sh;
    pl[c - PL] = sl;
  }
}
// correc with the defect correction folded in: u = u* - f grad(phi1 + phi2)
// and pnew += phi1 + phi2 (double-float), one pass over the fields
__global__ void __launch_bounds__(256) k_correc_mixed2(Geo g, const float *__restrict__ fu,
                                                       const float *__restrict__ fv, const float *__restrict__ fw,
                                                       const float *__restrict__ phi1,
                                                       const float *__restrict__ phi2, float *__restrict__ u,
                                                       float *__restrict__ v, float *__restrict__ w,
                                                       float *__restrict__ ph, float *__restrict__ pl, float fi,
                                                       float fj, float fk) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z + 1;
  if (i >= g.I || j >= g.J) return;
  const int dip = i + 1 == g.I ? 1 - g.I : 1;
  const int djp = (j + 1 == g.J ? 1 - g.J : 1) * g.I;
  const long PL = g.plane;
  const long c = fidx(g, i, j, k);
  const float a0 = phi1[c], b0 = phi2[c];
  const float P0 = a0 + b0;
  const float Pip = phi1[c + dip] + phi2[c + dip];
  const float Pjp = phi1[c + djp] + phi2[c + djp];
  const float Pkp = (k == g.K) ? P0 : phi1[c + PL] + phi2[c + PL];
  const float un = fu[c] - fi * (Pip - P0);
  const float vn = fv[c] - fj * (Pjp - P0);
  const float wn = (k == g.K) ? 0.f : fw[c] - fk * (Pkp - P0);
  u[c] = un;
  v[c] = vn;
  w[c] = wn;
  float sh, sl;
  df_add(ph[c], pl[c], a0, 0.f, sh, sl);
  df_add(sh, sl, b0, 0.f, sh, sl);
  ph[c] = sh;
  pl[c] = sl;
  if (k == g.K) {
    const float sg = g.bc_top == IBM_BC_NOSLIP ? -1.f : 1.f;
    u[c + PL] = sg * un;
    v[c + PL] = sg * vn;
    ph[c + PL] = sh;
    pl[c + PL] = sl;
  }
  if (k == 1) {
    const float sg = g.bc_bot == IBM_BC_NOSLIP ? -1.f : 1.f;
    u[c - PL] = sg * un;
    v[c - PL] = sg * vn;
    w[c - PL] = 0.f;
    ph[c - PL] = sh;
    pl[c - PL] = sl;
  }
}
void launch_correc_mixed2(cudaStream_t s, const Geo &g, const float *fu, const float *fv, const float *fw,
                          const float *phi1, const float *phi2, float *u, float *v, float *w, float *ph, float *pl,
                          double fi, double fj, double fk) {
  dim3 blk(64, 4, 1);
  dim3 grd((g.I + 63) / 64, (g.J + 3) / 4, g.K);
  k_correc_mixed2<<<grd, blk, 0, s>>>(g, fu, fv, fw, phi1, phi2, u, v, w, ph, pl, (float)fi, (float)fj, (float)fk);
}

// The same update four x-cells per thread with 16-byte loads and stores
// (I a multiple of 4): identical arithmetic per cell, a quarter of the
// memory instructions.
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__global__ void __launch_bounds__(256) k_correc_mixed4(Geo g, const float *fu, const float *fv, const float *fw,
                                                       const float *__restrict__ phi, float *u, float *v, float *w,
                                                       float *__restrict__ ph, float *__restrict__ pl, float fi,
                                                       float fj, float fk) {
  const int i0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z + 1;
  if (i0 >= g.I || j >= g.J) return;
  const int jp = j + 1 == g.J ? 0 : j + 1;
  const long PL = g.plane;
  const long c = fidx(g, i0, j, k);
  const float4 P0 = ld4(phi + c);
  const float P4 = phi[fidx(g, i0 + 4 == g.I ? 0 : i0 + 4, j, k)];
  const float4 Pjp = ld4(phi + fidx(g, i0, jp, k));
  const float4 Pkp = (k == g.K) ? P0 : ld4(phi + c + PL);
  const float4 FU = ld4(fu + c), FV = ld4(fv + c);
  const float4 FW = (k == g.K) ? make_float4(0.f, 0.f, 0.f, 0.f) : ld4(fw + c);
  const float p0[4] = {P0.x, P0.y, P0.z, P0.w}, pip[4] = {P0.y, P0.z, P0.w, P4};
  const float pjp[4] = {Pjp.x, Pjp.y, Pjp.z, Pjp.w}, pkp[4] = {Pkp.x, Pkp.y, Pkp.z, Pkp.w};
  const float fu4[4] = {FU.x, FU.y, FU.z, FU.w}, fv4[4] = {FV.x, FV.y, FV.z, FV.w}, fw4[4] = {FW.x, FW.y, FW.z, FW.w};
  const float4 H = ld4(ph + c), Lo = ld4(pl + c);
  const float h4[4] = {H.x, H.y, H.z, H.w}, l4[4] = {Lo.x, Lo.y, Lo.z, Lo.w};
  float un[4], vn[4], wn[4], sh[4], sl[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    un[e] = fu4[e] - fi * (pip[e] - p0[e]);
    vn[e] = fv4[e] - fj * (pjp[e] - p0[e]);
    wn[e] = (k == g.K) ? 0.f : fw4[e] - fk * (pkp[e] - p0[e]);
    df_add(h4[e], l4[e], p0[e], 0.f, sh[e], sl[e]);
  }
  const float4 U = make_float4(un[0], un[1], un[2], un[3]), V = make_float4(vn[0], vn[1], vn[2], vn[3]);
  const float4 W = make_float4(wn[0], wn[1], wn[2], wn[3]);
  const float4 SH = make_float4(sh[0], sh[1], sh[2], sh[3]), SL = make_float4(sl[0], sl[1], sl[2], sl[3]);
  st4(u + c, U);
  st4(v + c, V);
  st4(w + c, W);
  st4(ph + c, SH);
  st4(pl + c, SL);
  if (k == g.K) {
    const float sg = g.bc_top == IBM_BC_NOSLIP ? -1.f : 1.f;
    st4(u + c + PL, make_float4(sg * un[0], sg * un[1], sg * un[2], sg * un[3]));
    st4(v + c + PL, make_float4(sg * vn[0], sg * vn[1], sg * vn[2], sg * vn[3]));
    st4(ph + c + PL, SH);
    st4(pl + c + PL, SL);
  }
  if (k == 1) {
    const float sg = g.bc_bot == IBM_BC_NOSLIP ? -1.f : 1.f;
    st4(u + c - PL, make_float4(sg * un[0], sg * un[1], sg * un[2], sg * un[3]));
    st4(v + c - PL, make_float4(sg * vn[0], sg * vn[1], sg * vn[2], sg * vn[3]));
    st4(w + c - PL, make_float4(0.f, 0.f, 0.f, 0.f));
    st4(ph + c - PL, SH);
    st4(pl + c - PL, SL);
  }
}

void launch_correc_mixed(cudaStream_t s, const Geo &g, const float *fu, const float *fv, const float *fw,
                         const float *phi, float *u, float *v, float *w, float *ph, float *pl, double fi, double fj,
                         double fk) {
  if ((g.I & 3) == 0) {
    dim3 blk(64, 4, 1);
    dim3 grd((g.I / 4 + 63) / 64, (g.J + 3) / 4, g.K);
    k_correc_mixed4<<<grd, blk, 0, s>>>(g, fu, fv, fw, phi, u, v, w, ph, pl, (float)fi, (float)fj, (float)fk);
    return;
  }
  dim3 blk(64, 4, 1);
  dim3 grd((g.I + 63) / 64, (g.J + 3) / 4, g.K);
  k_correc_mixed<<<grd, blk, 0, s>>>(g, fu, fv, fw, phi, u, v, w, ph, pl, (float)fi, (float)fj, (float)fk);
}

// ---------------------------------------------------------------------------
// Layout conversion between the reference host layout (0:i1,0:j1,0:k1) and
// the device layout.  to_dev: dev(i,j,k) = ref(i+1,j+1,k).  to_ref fills the
// x/y ghosts with the periodic values, as bounduvw/boundp leave them.  LO: the
// device field is an FP32 pair dev + lo (the mixed form's pressure).
//
// Bound by memory: a warp walks rows with four loads of a lane in flight, the
// row's offset is formed once, and FP32 values are converted on the integer
// pipe (the conversion instructions issue at the rate of FP64).  A cell per
// thread with three 64-bit divisions and the conversions, and the pressure
// through an FP64 array and a second pass, 512 x 512 x 256: FP32 to_dev 273 us,
// to_ref 385 us, pressure 760 and 757 us; now 116, 132, 168 and 170 (the copy rate: 118
// and 158).  A conversion instruction that is only predicated off for the normal
// values still cost its issue: 143 and 146 us, pressure 378 and 414.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double wide(float f) { return f2d_rn(f); }
__device__ __forceinline__ double wide(double f) { return f; }
template <typename T, bool LO>
__global__ void __launch_bounds__(256) k_ref_to_dev(Geo g, const double *__restrict__ ref, T *__restrict__ dev,
                                                    float *__restrict__ lo) {
  const int lane = threadIdx.x & 31, nrow = g.J * (g.K + 2), I = g.I;
  for (int q = (blockIdx.x * 256 + threadIdx.x) >> 5; q < nrow; q += gridDim.x * 8) {
    const int k = (int)((unsigned)q / (unsigned)g.J), j = q - k * g.J;
    const double *r = ref + 1 + (long)(I + 2) * (j + 1 + (long)(g.J + 2) * k);
    T *d = dev + (long)q * I;
    for (int i0 = lane; i0 < I; i0 += 128) {
      double x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (i0 + 32 * e < I) x[e] = r[i0 + 32 * e];
      bool ok = true;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + 32 * e;
        if (i >= I) break;
        if constexpr (LO) {
          float h, l;
          ok &= d2df_int(x[e], h, l);
          d[i] = h;
          lo[(long)q * I + i] = l;
        } else if constexpr (sizeof(T) == 4) {
          float h;
          int rem;
          ok &= d2f_int(x[e], h, rem);
          d[i] = h;
        } else {
          d[i] = x[e];
        }
      }
      if (sizeof(T) == 4 && !ok) {  // a value out of FP32's normal range: the conversion instructions
#pragma unroll 1
        for (int i = i0; i < I && i < i0 + 128; i += 32) {
          const double y = r[i];
          const float h = (float)y;
          d[i] = h;
          if constexpr (LO) lo[(long)q * I + i] = (float)(y - (double)h);
        }
      }
    }
  }
}
template <typename T, bool LO>
__global__ void __launch_bounds__(256) k_dev_to_ref(Geo g, const T *__restrict__ dev, const float *__restrict__ lo,
                                                    double *__restrict__ ref) {
  const int lane = threadIdx.x & 31, nrow = (g.J + 2) * (g.K + 2), I = g.I;
  for (int q = (blockIdx.x * 256 + threadIdx.x) >> 5; q < nrow; q += gridDim.x * 8) {
    const int k = (int)((unsigned)q / (unsigned)(g.J + 2)), j = wrapm(q - k * (g.J + 2) - 1, g.J);
    const long row = fidx(g, 0, j, k);
    const T *d = dev + row;
    double *r = ref + (long)q * (I + 2);
    for (int i0 = lane; i0 < I + 2; i0 += 128) {
      T x[4];
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + 32 * e;
        if (i < I + 2) {
          const int id = wrapm(i - 1, I);
          x[e] = d[id];
          if constexpr (LO) y[e] = lo[row + id];
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + 32 * e;
        if (i >= I + 2) break;
        if constexpr (LO) r[i] = wide(x[e]) + wide(y[e]);
        else r[i] = wide(x[e]);
      }
    }
  }
}
static int row_blocks(int nrow) { return std::min((nrow + 7) / 8, 8 * sm_count()); }
template <typename T>
void launch_ref_to_dev(cudaStream_t s, const Geo &g, const double *ref, T *dev) {
  k_ref_to_dev<T, false><<<row_blocks(g.J * (g.K + 2)), 256, 0, s>>>(g, ref, dev, nullptr);
}
template <typename T>
void launch_dev_to_ref(cudaStream_t s, const Geo &g, const T *dev, double *ref) {
  k_dev_to_ref<T, false><<<row_blocks((g.J + 2) * (g.K + 2)), 256, 0, s>>>(g, dev, nullptr, ref);
}
void launch_ref_to_dev_df(cudaStream_t s, const Geo &g, const double *ref, float *h, float *l) {
  k_ref_to_dev<float, true><<<row_blocks(g.J * (g.K + 2)), 256, 0, s>>>(g, ref, h, l);
}
void launch_dev_to_ref_df(cudaStream_t s, const Geo &g, const float *h, const float *l, double *ref) {
  k_dev_to_ref<float, true><<<row_blocks((g.J + 2) * (g.K + 2)), 256, 0, s>>>(g, h, l, ref);
}
template void launch_ref_to_dev<double>(cudaStream_t, const Geo &, const double *, double *);
template void launch_ref_to_dev<float>(cudaStream_t, const Geo &, const double *, float *);
template void launch_dev_to_ref<double>(cudaStream_t, const Geo &, const double *, double *);
template void launch_dev_to_ref<float>(cudaStream_t, const Geo &, const float *, double *);

// ---------------------------------------------------------------------------
// Reductions over the grid: chkdiv, chkdt and the wall shear.  One launch each:
// the blocks leave partials in the context's scratch and the last one to
// finish combines them in a fixed order, a partial per lane.  (One thread that
// walked 608 partials took 98 us for chkdiv, 53 us for chkdt and 6 us for the
// shear's 64, longer than the sweeps over a 64^3 grid.)  The counter behind
// the last block's choice wraps back to zero by itself.
// ---------------------------------------------------------------------------
constexpr int RED_BLOCKS = 1216;                // partials of one kind
constexpr int RED_COUNT = 4088;                 // scratch entry of the counters
__device__ __forceinline__ bool red_last(double *scratch, int which) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned *cnt = reinterpret_cast<unsigned *>(scratch + RED_COUNT) + which;
    last = atomicInc(cnt, gridDim.x - 1) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  return last;
}
// Sum over 256 threads, valid in thread 0.
__device__ __forceinline__ double block_sum(double s) {
  __shared__ double sm[8];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(~0u, s, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int q = 1; q < 8; ++q) s += sm[q];
  return s;
}
// Smallest and largest of doubles >= 0 over 256 threads, valid in thread 0.
// Their bits order like the integers, which keeps the FP64 pipe out of it.
__device__ __forceinline__ void block_min_max(double &mn, double &mx) {
  __shared__ long long sn[8], sx[8];
  long long n = __double_as_longlong(mn), x = __double_as_longlong(mx);
  for (int o = 16; o > 0; o >>= 1) {
    n = min(n, __shfl_down_sync(~0u, n, o));
    x = max(x, __shfl_down_sync(~0u, x, o));
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) { sn[threadIdx.x >> 5] = n; sx[threadIdx.x >> 5] = x; }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int q = 1; q < 8; ++q) { n = min(n, sn[q]); x = max(x, sx[q]); }
  mn = __longlong_as_double(n);
  mx = __longlong_as_double(x);
}
// Larger value first, then the smaller index.  Values are kept as the bits of
// a double >= 0 (or of -1: nothing seen), which order like the integers.
__device__ __forceinline__ void max_loc(long long &m, long long &l, long long m2, long long l2) {
  if (m2 > m || (m2 == m && l2 >= 0 && (l < 0 || l2 < l))) { m = m2; l = l2; }
}
__device__ __forceinline__ void block_max_loc(long long &m, long long &l) {
  __shared__ long long sm[8], sl[8];
  for (int o = 16; o > 0; o >>= 1) {
    const long long m2 = __shfl_down_sync(~0u, m, o), l2 = __shfl_down_sync(~0u, l, o);
    max_loc(m, l, m2, l2);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) { sm[threadIdx.x >> 5] = m; sl[threadIdx.x >> 5] = l; }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int q = 1; q < 8; ++q) max_loc(m, l, sm[q], sl[q]);
}
// Chunks of 256 cells of one plane, dealt to the blocks in turn: one uniform
// division a chunk and one 32-bit division a cell.
__host__ __device__ __forceinline__ int red_chunks(const Geo &g) { return (int)((g.plane + 255) / 256); }
static int red_blocks(const Geo &g) {
  const long n = (long)red_chunks(g) * g.K;
  return (int)(n < RED_BLOCKS ? n : RED_BLOCKS);
}

// chkdiv (chkdiv.f90:7-61): sum(div) and (max|div|, first linear index).
template <typename T>
__global__ void __launch_bounds__(256) k_chkdiv(Geo g, const T *__restrict__ u, const T *__restrict__ v,
                                                const T *__restrict__ w, double *scratch, double *out) {
  const int ncp = red_chunks(g);
  const long nq = (long)ncp * g.K;
  double s = 0.;
  long long m = __double_as_longlong(-1.), loc = -1;
  for (long q = blockIdx.x; q < nq; q += gridDim.x) {
    const int kk = (int)(q / ncp), k = kk + 1;
    const int t = (int)(q - (long)kk * ncp) * 256 + (int)threadIdx.x;
    if (t >= g.plane) continue;
    const int j = (int)((unsigned)t / (unsigned)g.I), i = t - j * g.I;
    const long c = (long)k * g.plane + t;
    const double div = (wide(w[c]) - wide(w[c - g.plane])) * g.dzi +
                       (wide(v[c]) - wide(v[fidx(g, i, wrapm(j - 1, g.J), k)])) * g.dyi +
                       (wide(u[c]) - wide(u[fidx(g, wrapm(i - 1, g.I), j, k)])) * g.dxi;
    s += div;
    const long long a = __double_as_longlong(fabs(div));
    if (a > m && a <= 0x7ff0000000000000ll) { m = a; loc = c - g.plane; }  // not a NaN
  }
  double *psum = scratch;
  long long *pmax = reinterpret_cast<long long *>(scratch + RED_BLOCKS), *ploc = pmax + RED_BLOCKS;
  s = block_sum(s);
  block_max_loc(m, loc);
  if (threadIdx.x == 0) { psum[blockIdx.x] = s; pmax[blockIdx.x] = m; ploc[blockIdx.x] = loc; }
  if (!red_last(scratch, 0)) return;
  s = 0.;
  m = __double_as_longlong(-1.);
  loc = -1;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) {
    s += __ldcg(psum + b);
    max_loc(m, loc, __ldcg(pmax + b), __ldcg(ploc + b));
  }
  s = block_sum(s);
  block_max_loc(m, loc);
  if (threadIdx.x == 0) { out[0] = s; out[1] = __longlong_as_double(m); out[2] = (double)loc; }
}
template <typename T>
void launch_chkdiv(cudaStream_t s, const Geo &g, const T *u, const T *v, const T *w, double *scratch, double *out) {
  k_chkdiv<T><<<red_blocks(g), 256, 0, s>>>(g, u, v, w, scratch, out);
}
template void launch_chkdiv<double>(cudaStream_t, const Geo &, const double *, const double *, const double *,
                                    double *, double *);
template void launch_chkdiv<float>(cudaStream_t, const Geo &, const float *, const float *, const float *, double *,
                                   double *);

// chkdt (chkdt.f90:6-273): min over the three staggered components of
// sqrt(3) / S with S = |u|/dx + |v|/dy + |w|/dz.  Only the largest S counts, so
// every component is bounded in FP32 first, and S is formed in FP64 where the
// upper bound reaches the largest lower bound seen: a warp or two of a block.
// (|t| for the sqrt(t^2) of the reference: the same number unless t^2 leaves
// the range.)  Cells whose speed may be under the 1e-12 below which the
// reference takes 99999, and those with an infinity or a NaN, go through its
// formula as it stands.  In FP64 throughout, the kernel was bound by three
// square roots and a division a component: 119 us at 64^3, now 26.
template <typename T>
__global__ void __launch_bounds__(256) k_chkdt(Geo g, const T *__restrict__ u, const T *__restrict__ v,
                                               const T *__restrict__ w, float still, double *scratch, double *out) {
  const int ncp = red_chunks(g);
  const long nq = (long)ncp * g.K;
  const double dxi = g.dxi, dyi = g.dyi, dzi = g.dzi;
  const float dx = (float)dxi, dy = (float)dyi, dz = (float)dzi;
  double m = 899999., most_s = 0.;
  __shared__ unsigned lmax;     // largest lower bound of S in the block (bits of a float >= 0)
  if (threadIdx.x == 0) lmax = 0u;
  __syncthreads();
  bool first = true;
  for (long q = blockIdx.x; q < nq; q += gridDim.x) {
    const int kk = (int)(q / ncp), k = kk + 1;
    const int t = (int)(q - (long)kk * ncp) * 256 + (int)threadIdx.x;
    const bool in = t < g.plane;
    const int j = (int)((unsigned)t / (unsigned)g.I), i = t - j * g.I;
    float ub[3] = {-1.f, -1.f, -1.f}, lb = 0.f;
    bool slow = false;
    T u0, um, v0, vm, w0, wm, v1, v2, w1, w2, u1, u2, w3, w4, u3, u4, v3, v4;
    if (in) {
      const long ip = i + 1 < g.I ? 1 : 1 - g.I, im = i ? -1 : g.I - 1;
      const long jp = j + 1 < g.J ? g.I : g.I - g.plane, jm = j ? -g.I : g.plane - g.I, kp = g.plane;
      const long c = (long)k * g.plane + t;
      const T *pu = u + c, *pv = v + c, *pw = w + c;
      u0 = pu[0]; um = pu[im]; v0 = pv[0]; vm = pv[jm]; w0 = pw[0]; wm = pw[-kp];
      v1 = pv[ip]; v2 = pv[ip + jm]; w1 = pw[ip]; w2 = pw[ip - kp];
      u1 = pu[jp]; u2 = pu[im + jp]; w3 = pw[jp]; w4 = pw[jp - kp];
      u3 = pu[im + kp]; u4 = pu[kp]; v3 = pv[jm + kp]; v4 = pv[kp];
      // a: the component's own velocity, b and c: four neighbours of the others'
      auto bound = [&](int e, T a, float da, T b0, T b1, T b2, T b3, float db, T c0, T c1, T c2, T c3, float dc) {
        const float fa = fabsf((float)a) * da;
        const float x0 = (float)b0, x1 = (float)b1, x2 = (float)b2, x3 = (float)b3;
        const float y0 = (float)c0, y1 = (float)c1, y2 = (float)c2, y3 = (float)c3;
        const float s = fa + 0.25f * (fabsf(x0 + x1 + x2 + x3) * db + fabsf(y0 + y1 + y2 + y3) * dc);
        const float mag = fa + 0.25f * ((fabsf(x0) + fabsf(x1) + fabsf(x2) + fabsf(x3)) * db +
                                        (fabsf(y0) + fabsf(y1) + fabsf(y2) + fabsf(y3)) * dc);
        const float er = 1.e-6f * mag;  // ten FP32 roundings of 2^-24
        ub[e] = s + er;
        lb = fmaxf(lb, s - er);
        slow |= !(s - er > still);
      };
      bound(0, u0, dx, v0, vm, v1, v2, dy, w0, wm, w1, w2, dz);
      bound(1, v0, dy, u0, u1, u2, um, dx, w0, w3, w4, wm, dz);
      bound(2, w0, dz, u0, um, u3, u4, dx, v0, vm, v3, v4, dy);
    }
    const unsigned wl = __reduce_max_sync(~0u, __float_as_uint(lb));
    if ((threadIdx.x & 31) == 0) atomicMax(&lmax, wl);
    if (first) __syncthreads();  // later chunks make do with what is there
    first = false;
    const float most = __uint_as_float(max(wl, *(volatile unsigned *)&lmax));
    if (in && (slow || fmaxf(fmaxf(ub[0], ub[1]), ub[2]) >= most)) {
      auto comp = [&](int e, T a, double da, T b0, T b1, T b2, T b3, double db, T c0, T c1, T c2, T c3, double dc) {
        if (!slow && ub[e] < most) return;
        const double t0 = wide(a), t1 = 0.25 * (wide(b0) + wide(b1) + wide(b2) + wide(b3)),
                     t2 = 0.25 * (wide(c0) + wide(c1) + wide(c2) + wide(c3));
        if (!slow) {
          most_s = fmax(most_s, fabs(t0) * da + fabs(t1) * db + fabs(t2) * dc);
          return;
        }
        const double s0 = t0 * t0, s1 = t1 * t1, s2 = t2 * t2, velo = sqrt(s0 + s1 + s2);
        m = fmin(m, fabs(velo) > 1.e-12 ? sqrt(3.) / (sqrt(s0) * da + sqrt(s1) * db + sqrt(s2) * dc) : 99999.);
      };
      comp(0, u0, dxi, v0, vm, v1, v2, dyi, w0, wm, w1, w2, dzi);
      comp(1, v0, dyi, u0, u1, u2, um, dxi, w0, w3, w4, wm, dzi);
      comp(2, w0, dzi, u0, um, u3, u4, dxi, v0, vm, v3, v4, dyi);
    }
  }
  block_min_max(m, most_s);
  if (threadIdx.x == 0) { scratch[blockIdx.x] = m; scratch[RED_BLOCKS + blockIdx.x] = most_s; }
  if (!red_last(scratch, 1)) return;
  m = 899999.;
  most_s = 0.;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) {
    long long n = __double_as_longlong(m), x = __double_as_longlong(most_s);
    n = min(n, __double_as_longlong(__ldcg(scratch + b)));
    x = max(x, __double_as_longlong(__ldcg(scratch + RED_BLOCKS + b)));
    m = __longlong_as_double(n);
    most_s = __longlong_as_double(x);
  }
  block_min_max(m, most_s);
  if (threadIdx.x == 0) {
    m = fmin(m, 1.65 / (4. * g.visc * (dxi * dxi + dyi * dyi + dzi * dzi)));
    out[0] = most_s > 0. ? fmin(m, sqrt(3.) / most_s) : m;
  }
}
template <typename T>
void launch_chkdt(cudaStream_t s, const Geo &g, const T *u, const T *v, const T *w, double *scratch, double *out) {
  // above this S the speed is certainly over 1e-12
  const float still = (float)(1.01e-12 * std::sqrt(g.dxi * g.dxi + g.dyi * g.dyi + g.dzi * g.dzi));
  k_chkdt<T><<<red_blocks(g), 256, 0, s>>>(g, u, v, w, still, scratch, out);
}
template void launch_chkdt<double>(cudaStream_t, const Geo &, const double *, const double *, const double *,
                                   double *, double *);
template void launch_chkdt<float>(cudaStream_t, const Geo &, const float *, const float *, const float *, double *,
                                  double *);

// wall shear of rk1/rk2/rk3 (rk3.f90:80-103): sum over the wall planes.
template <typename T>
__global__ void __launch_bounds__(256) k_wallshear(Geo g, const T *__restrict__ v, double *scratch, double *out) {
  double s = 0.;
  const long PL = g.plane;
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < PL; t += (long)gridDim.x * blockDim.x) {
    const long top = (long)g.K * PL + t, bot = PL + t;
    s += ((double)v[top + PL] - (double)v[top]) - ((double)v[bot] - (double)v[bot - PL]);
  }
  s = block_sum(s);
  if (threadIdx.x == 0) scratch[blockIdx.x] = s;
  if (!red_last(scratch, 2)) return;
  s = 0.;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) s += __ldcg(scratch + b);
  s = block_sum(s);
  if (threadIdx.x == 0) out[0] = s * (g.visc * g.dzi * (1. / g.dxi) * (1. / g.dyi));
}
template <typename T>
void launch_wallshear(cudaStream_t s, const Geo &g, const T *v, double *scratch, double *out) {
  const int n = red_chunks(g);
  k_wallshear<T><<<n < 256 ? n : 256, 256, 0, s>>>(g, v, scratch, out);
}
template void launch_wallshear<double>(cudaStream_t, const Geo &, const double *, double *, double *);
template void launch_wallshear<float>(cudaStream_t, const Geo &, const float *, double *, double *);

// convert / copy helpers for the mixed form
__global__ void k_d2f(long n, const double *__restrict__ a, float *__restrict__ b) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
    b[t] = (float)a[t];
}
__global__ void k_f2d(long n, const float *__restrict__ a, double *__restrict__ b) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
    b[t] = (double)a[t];
}
void launch_d2f(cudaStream_t s, long n, const double *a, float *b) { k_d2f<<<1216, 256, 0, s>>>(n, a, b); }
void launch_f2d(cudaStream_t s, long n, const float *a, double *b) { k_f2d<<<1216, 256, 0, s>>>(n, a, b); }

}  // namespace ibmk
