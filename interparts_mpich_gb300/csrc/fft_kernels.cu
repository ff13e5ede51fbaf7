// fft_kernels.cu -- pressure Poisson solve of solver2d (solver.f90:43-172):
// real FFT along x fused with fillps (fillps.f90:8-53), complex FFT along y,
// batched Thomas sweep along z with the zero-mode guard, inverse y, inverse x.
//
// The reference transforms with VFFTPACK in half-complex storage; the solve
// is storage independent (each Fourier mode decouples with eigenvalue
// xrt+yrt, initsolver.f90:42-64), so the GPU keeps an ordinary complex
// spectrum S[k][ky][kx], kx = 0..I/2, built from a half-length complex FFT.
//
// FFTs run in shared memory with a Stockham autosort formulation of radix
// 2/3/4 stages (Govindaraju et al., SC'08); twiddles come from a host-built
// table W_M^t = exp(-2*pi*i*t/M).
#include "kernels.cuh"

namespace ibmk {

template <typename T> struct cpx;
template <> struct cpx<double> { typedef double2 t; };
template <> struct cpx<float> { typedef float2 t; };

template <typename C> __device__ __forceinline__ C cmk(decltype(C().x) a, decltype(C().x) b) { C r; r.x = a; r.y = b; return r; }
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return cmk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return cmk<C>(a.x - b.x, a.y - b.y); }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) { return cmk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <typename C> __device__ __forceinline__ C cconj(C a) { return cmk<C>(a.x, -a.y); }
template <typename C> __device__ __forceinline__ C cscale(C a, decltype(C().x) s) { return cmk<C>(a.x * s, a.y * s); }
// multiply by -i (forward) or +i (inverse)
template <typename C> __device__ __forceinline__ C cmi(C a, int inv) { return inv ? cmk<C>(-a.y, a.x) : cmk<C>(a.y, -a.x); }

// small DFTs, forward e^{-2 pi i qr/R} (inverse: conjugate kernel)
template <typename C> __device__ __forceinline__ void dft2(C *v) {
  C a = v[0], b = v[1];
  v[0] = cadd(a, b); v[1] = csub(a, b);
}
template <typename C> __device__ __forceinline__ void dft4(C *v, int inv) {
  C t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
  C t2 = cadd(v[1], v[3]), t3 = cmi(csub(v[1], v[3]), inv);
  v[0] = cadd(t0, t2); v[2] = csub(t0, t2);
  v[1] = cadd(t1, t3); v[3] = csub(t1, t3);
}
template <typename C> __device__ __forceinline__ void dft3(C *v, int inv) {
  typedef decltype(C().x) R;
  const R h = (R)0.5, s3 = (R)0.86602540378443864676372317075294;
  C t1 = cadd(v[1], v[2]);
  C t2 = csub(v[0], cscale(t1, h));
  C t3 = cscale(cmi(csub(v[1], v[2]), inv), s3);
  v[0] = cadd(v[0], t1);
  v[1] = cadd(t2, t3);
  v[2] = csub(t2, t3);
}

// In-place (ping-pong) shared-memory FFT of nseq sequences of length M.
// element m of sequence s lives at buf[s*ss + m*es].  Returns the buffer
// holding the result (a or b).
template <typename C>
__device__ C *fft_smem(C *a, C *b, int M, int nseq, int es, int ss, const FftPlan &pl, const C *__restrict__ tw,
                       int inv) {
  int Ns = 1;
  for (int st = 0; st < pl.nst; ++st) {
    const int R = pl.rad[st];
    const int nb = M / R;
    const int twst = M / (Ns * R);
    for (int t = threadIdx.x; t < nb * nseq; t += blockDim.x) {
      const int sq = t / nb, jb = t - sq * nb;
      const C *src = a + (long)sq * ss;
      C *dst = b + (long)sq * ss;
      const int kk = jb % Ns;
      C v[4];
      for (int r = 0; r < R; ++r) {
        C x = src[(jb + r * nb) * es];
        if (r > 0 && kk > 0) {
          C wt = tw[kk * twst * r];
          if (inv) wt = cconj(wt);
          x = cmul(x, wt);
        }
        v[r] = x;
      }
      if (R == 2) dft2(v);
      else if (R == 4) dft4(v, inv);
      else dft3(v, inv);
      const int idxD = (jb / Ns) * Ns * R + kk;
      for (int r = 0; r < R; ++r) dst[(idxD + r * Ns) * es] = v[r];
    }
    __syncthreads();
    C *t = a; a = b; b = t;
    Ns *= R;
  }
  return a;
}

// Compile-time specialisation of the same Stockham stages for the lengths
// used by the configurations: the index arithmetic (divisions by the
// butterfly count and the sub-transform size) becomes shifts and constant
// multiplies.  Radix order as in the runtime plan: 4s, then 2, then 3.
template <int M, int Ns, typename C>
__device__ __forceinline__ C *fft_stages_ct(C *a, C *b, int nseq, int ss, const C *__restrict__ tw, int inv) {
  if constexpr (Ns >= M) {
    return a;
  } else {
    constexpr int rem = M / Ns;
    constexpr int R = (rem % 4 == 0) ? 4 : ((rem % 2 == 0) ? 2 : 3);
    constexpr int nb = M / R;
    constexpr int twst = M / (Ns * R);
    for (int t = threadIdx.x; t < nb * nseq; t += blockDim.x) {
      const int sq = t / nb, jb = t - sq * nb;
      const C *src = a + (long)sq * ss;
      C *dst = b + (long)sq * ss;
      const int kk = jb % Ns;
      C v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        C x = src[jb + r * nb];
        if (r > 0 && kk > 0) {
          C wt = tw[kk * twst * r];
          if (inv) wt = cconj(wt);
          x = cmul(x, wt);
        }
        v[r] = x;
      }
      if constexpr (R == 2) dft2(v);
      else if constexpr (R == 4) dft4(v, inv);
      else dft3(v, inv);
      const int idxD = (jb / Ns) * Ns * R + kk;
#pragma unroll
      for (int r = 0; r < R; ++r) dst[idxD + r * Ns] = v[r];
    }
    __syncthreads();
    return fft_stages_ct<M, Ns * R, C>(b, a, nseq, ss, tw, inv);
  }
}

// unit-stride sequences (es = 1); lengths without a specialisation use the
// runtime plan
template <typename C>
__device__ C *fft_smem1(C *a, C *b, int M, int nseq, int ss, const FftPlan &pl, const C *__restrict__ tw, int inv) {
  switch (M) {
    case 16: return fft_stages_ct<16, 1, C>(a, b, nseq, ss, tw, inv);
    case 24: return fft_stages_ct<24, 1, C>(a, b, nseq, ss, tw, inv);
    case 32: return fft_stages_ct<32, 1, C>(a, b, nseq, ss, tw, inv);
    case 48: return fft_stages_ct<48, 1, C>(a, b, nseq, ss, tw, inv);
    case 64: return fft_stages_ct<64, 1, C>(a, b, nseq, ss, tw, inv);
    case 96: return fft_stages_ct<96, 1, C>(a, b, nseq, ss, tw, inv);
    case 128: return fft_stages_ct<128, 1, C>(a, b, nseq, ss, tw, inv);
    case 192: return fft_stages_ct<192, 1, C>(a, b, nseq, ss, tw, inv);
    case 256: return fft_stages_ct<256, 1, C>(a, b, nseq, ss, tw, inv);
    case 384: return fft_stages_ct<384, 1, C>(a, b, nseq, ss, tw, inv);
    case 512: return fft_stages_ct<512, 1, C>(a, b, nseq, ss, tw, inv);
    case 768: return fft_stages_ct<768, 1, C>(a, b, nseq, ss, tw, inv);
    default: return fft_smem<C>(a, b, M, nseq, 1, ss, pl, tw, inv);
  }
}

// ---------------------------------------------------------------------------
// Register four-step FFT of the FP32 divergence residual (forward).  N = N1*N2
// with N1 = N2 or 2*N2 and N1 <= 16: a group of N2 threads holds a sequence, thread t the elements
// x[t + N2*n1]; an N1-point DFT in registers, the twiddle W_N^(t*k1), one
// exchange through a padded shared buffer (group-private, __syncwarp only),
// then N2-point DFTs in registers (N1/N2 per thread), written back in
// natural order.  Same DFT as the Stockham stages, other summation order.
// ---------------------------------------------------------------------------
// multiply by exp(-2 pi i m/den) given cos, sin of 2 pi m/den
__device__ __forceinline__ float2 cmulcs(float2 x, float c, float s) {
  return make_float2(x.x * c + x.y * s, x.y * c - x.x * s);
}
// cos, sin of 2 pi m / 16, m = 0..9
__device__ __forceinline__ void w16(int m, float &c, float &s) {
  const float C1 = 0.92387953251128675613f, S1 = 0.38268343236508977173f, R2 = 0.70710678118654752440f;
  const float cs[10] = {1.f, C1, R2, S1, 0.f, -S1, -R2, -C1, -1.f, -C1};
  const float sn[10] = {0.f, S1, R2, C1, 1.f, C1, R2, S1, 0.f, -S1};
  c = cs[m]; s = sn[m];
}
template <int N> __device__ __forceinline__ void dft_reg(float2 *v);
template <> __device__ __forceinline__ void dft_reg<4>(float2 *v) { dft4(v, 0); }
template <> __device__ __forceinline__ void dft_reg<8>(float2 *v) {
  // n = n2 + 2 n1, k = k1 + 4 k2
  float2 a0[4] = {v[0], v[2], v[4], v[6]}, a1[4] = {v[1], v[3], v[5], v[7]};
  dft4(a0, 0);
  dft4(a1, 0);
  float c, s;
  w16(2, c, s); a1[1] = cmulcs(a1[1], c, s);
  a1[2] = cmi(a1[2], 0);
  w16(6, c, s); a1[3] = cmulcs(a1[3], c, s);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) { v[k1] = cadd(a0[k1], a1[k1]); v[k1 + 4] = csub(a0[k1], a1[k1]); }
}
template <> __device__ __forceinline__ void dft_reg<16>(float2 *v) {
  // n = n2 + 4 n1, k = k1 + 4 k2
  float2 a[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) a[n2][n1] = v[n2 + 4 * n1];
    dft4(a[n2], 0);
  }
#pragma unroll
  for (int n2 = 1; n2 < 4; ++n2)
#pragma unroll
    for (int k1 = 1; k1 < 4; ++k1) {
      float c, s;
      w16(n2 * k1, c, s);
      a[n2][k1] = cmulcs(a[n2][k1], c, s);
    }
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    float2 b[4] = {a[0][k1], a[1][k1], a[2][k1], a[3][k1]};
    dft4(b, 0);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = b[k2];
  }
}
// one sequence in shared memory (unit stride) per group of N2 threads;
// ex: group-private exchange buffer of N1*(N2+1) elements.  Every thread of
// the warp must call it (it synchronises the warp).
template <int N1, int N2>
__device__ __forceinline__ void fft_group(float2 *row, float2 *ex, int t, const float2 *__restrict__ tw) {
  constexpr int N = N1 * N2;
  float2 v[N1];
#pragma unroll
  for (int r = 0; r < N1; ++r) v[r] = row[t + N2 * r];
  dft_reg<N1>(v);
#pragma unroll
  for (int k1 = 1; k1 < N1; ++k1)
    if (t > 0) v[k1] = cmul(v[k1], __ldg(&tw[(t * k1) % N]));
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) ex[k1 * (N2 + 1) + t] = v[k1];
  __syncwarp();
#pragma unroll
  for (int q = 0; q < N1 / N2; ++q) {
    const int k1 = t + q * N2;
    float2 w[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) w[n2] = ex[k1 * (N2 + 1) + n2];
    dft_reg<N2>(w);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) row[k1 + N1 * k2] = w[k2];
  }
  __syncwarp();
}
// (N1, N2) of the supported lengths; 0 = use the Stockham stages
__host__ __device__ inline int reg_n2(int N) {
  return N == 16 ? 4 : N == 32 ? 4 : N == 64 ? 8 : N == 128 ? 8 : N == 256 ? 16 : 0;
}

// divergence factors dt/dx, dt/dy, dt/dz as double-float pairs (hi, lo)
struct DivScale {
  float xh, xl, yh, yl, zh, zl;
};

// With phi1 (defect correction, DF): the right-hand side is the divergence
// residual of the corrected velocity u* - f grad(phi1) (correc's FP32
// expressions), formed on the fly instead of read from a stored state.
template <int N1, int N2>
__global__ void __launch_bounds__(128) k_fillps_fftx_r(Geo g, const float *__restrict__ fu,
                                                       const float *__restrict__ fv, float *__restrict__ fw,
                                                       float2 *__restrict__ S, const float2 *__restrict__ twM,
                                                       const float2 *__restrict__ twN, DivScale ds,
                                                       const float *__restrict__ phi1, float cfi, float cfj,
                                                       float cfk) {
  constexpr int M = N1 * N2, ROWS = 128 / N2;
  // group strides padded by 8 elements (64 B): groups sharing a warp start
  // half a bank row apart
  constexpr int RS = M + 8, ES = N1 * (N2 + 1) + 8;
  __shared__ __align__(16) float2 A[ROWS * RS];
  __shared__ float2 EX[ROWS * ES];
  const int row0 = blockIdx.x * ROWS;
  const int nrow = g.J * g.K;
  const float fx_hi = ds.xh, fx_lo = ds.xl, fy_hi = ds.yh, fy_lo = ds.yl, fz_hi = ds.zh, fz_lo = ds.zl;
  const int PL = g.I * g.J;
  // 1. right-hand side, packed z_m = x_{2m} + i x_{2m+1}; four consecutive
  // i per thread with 128-bit loads (I % 4 == 0 on this path)
  constexpr int Q = 2 * M / 4;  // float4 per row
#pragma unroll 4
  for (int q = threadIdx.x; q < ROWS * Q; q += blockDim.x) {
    const int r = q / Q, i0 = (q - r * Q) * 4;
    const int row = row0 + r;
    float val[4] = {0.f, 0.f, 0.f, 0.f};
    if (row < nrow) {
      const int j = row % g.J, k = row / g.J + 1;
      const long c = fidx(g, i0, j, k);
      const float4 w4 = (k == g.K) ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4 *>(fw + c);
      const float4 wm4 = *reinterpret_cast<const float4 *>(fw + c - PL);  // plane 0 holds w(0)=0
      if (k == g.K) *reinterpret_cast<float4 *>(fw + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      const long cjm = c + (j == 0 ? (g.J - 1) * g.I : -g.I);
      const float4 v4 = *reinterpret_cast<const float4 *>(fv + c);
      const float4 vm4 = *reinterpret_cast<const float4 *>(fv + cjm);
      const float4 u4 = *reinterpret_cast<const float4 *>(fu + c);
      const long cim = c + (i0 == 0 ? g.I - 1 : -1);
      const float um1 = fu[cim];
      float wk[4] = {w4.x, w4.y, w4.z, w4.w}, wkm[4] = {wm4.x, wm4.y, wm4.z, wm4.w};
      float vv[4] = {v4.x, v4.y, v4.z, v4.w}, vjm[4] = {vm4.x, vm4.y, vm4.z, vm4.w};
      float uu[4] = {u4.x, u4.y, u4.z, u4.w}, uim[4] = {um1, u4.x, u4.y, u4.z};
      if (phi1) {
        // u - fi (phi(i+1) - phi(i)) etc. as correc stores them (w = 0 on
        // the walls k = K and 0)
        const float4 p4 = *reinterpret_cast<const float4 *>(phi1 + c);
        const float pim = phi1[cim];
        const float pip = phi1[c + (i0 + 4 == g.I ? 4 - g.I : 4)];
        const float4 pjp4 = *reinterpret_cast<const float4 *>(phi1 + c + (j + 1 == g.J ? (1 - g.J) * g.I : g.I));
        const float4 pjm4 = *reinterpret_cast<const float4 *>(phi1 + cjm);
        const float4 pkp4 = (k == g.K) ? p4 : *reinterpret_cast<const float4 *>(phi1 + c + PL);
        const float4 pkm4 = *reinterpret_cast<const float4 *>(phi1 + c - PL);
        const float P[6] = {pim, p4.x, p4.y, p4.z, p4.w, pip};
        const float Pjp[4] = {pjp4.x, pjp4.y, pjp4.z, pjp4.w}, Pjm[4] = {pjm4.x, pjm4.y, pjm4.z, pjm4.w};
        const float Pkp[4] = {pkp4.x, pkp4.y, pkp4.z, pkp4.w}, Pkm[4] = {pkm4.x, pkm4.y, pkm4.z, pkm4.w};
        for (int e = 0; e < 4; ++e) {
          const float P0 = P[e + 1];
          const float un = uu[e] - cfi * (P[e + 2] - P0);
          const float unm = uim[e] - cfi * (P0 - P[e]);
          const float vn = vv[e] - cfj * (Pjp[e] - P0);
          const float vnm = vjm[e] - cfj * (P0 - Pjm[e]);
          const float wn = (k == g.K) ? 0.f : wk[e] - cfk * (Pkp[e] - P0);
          const float wnm = (k == 1) ? 0.f : wkm[e] - cfk * (P0 - Pkm[e]);
          uu[e] = un; uim[e] = unm; vv[e] = vn; vjm[e] = vnm; wk[e] = wn; wkm[e] = wnm;
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // divergence residual in double-float arithmetic: exact differences
        // of the FP32 velocities, products with the split FP64 factors
        float dh, dl, th, tl, sh, sl;
        two_sum(wk[e], -wkm[e], dh, dl);
        df_mul(dh, dl, fz_hi, fz_lo, sh, sl);
        two_sum(vv[e], -vjm[e], dh, dl);
        df_mul(dh, dl, fy_hi, fy_lo, th, tl);
        df_add(sh, sl, th, tl, sh, sl);
        two_sum(uu[e], -uim[e], dh, dl);
        df_mul(dh, dl, fx_hi, fx_lo, th, tl);
        df_add(sh, sl, th, tl, sh, sl);
        val[e] = sh + sl;
      }
    }
    *reinterpret_cast<float4 *>(reinterpret_cast<float *>(A + r * RS) + i0) = make_float4(val[0], val[1], val[2], val[3]);
  }
  __syncthreads();
  const int grp = threadIdx.x / N2, t = threadIdx.x - grp * N2;
  fft_group<N1, N2>(A + grp * RS, EX + grp * ES, t, twM);
  __syncthreads();
  // 2. unpack to X_k, k = 0..M  (X_k = E_k + W_N^k O_k)
  for (int q = threadIdx.x; q < ROWS * (M + 1); q += blockDim.x) {
    const int r = q / (M + 1), kx = q - r * (M + 1);
    const int row = row0 + r;
    if (row >= nrow) continue;
    const float2 Zk = A[r * RS + (kx == M ? 0 : kx)];
    const float2 Zc = cconj(A[r * RS + (kx == 0 ? 0 : M - kx)]);
    const float2 E = cscale(cadd(Zk, Zc), 0.5f);
    const float2 D = csub(Zk, Zc);
    const float2 O = cmk<float2>(D.y * 0.5f, -D.x * 0.5f);  // D/(2i)
    S[(long)row * g.MX + kx] = cadd(E, cmul(__ldg(&twN[kx]), O));
  }
}

// dispatch of the register FFT of the divergence residual for M = I/2
template <int M1, int M2>
bool launch_fftx_r(cudaStream_t s, const Geo &g, const float *fu, const float *fv, float *fw, float2 *S,
                   const float2 *twM, const float2 *twN, double a, double b, double c, const PoissonResid &rs) {
  const int nrow = g.J * g.K;
  constexpr int ROWS = 128 / M2;
  const int grid = (nrow + ROWS - 1) / ROWS;
  // the divergence factors as double-float pairs, split here once rather
  // than in every thread (FP64 issues at a small fraction of the FP32 rate)
  DivScale ds;
  ds.xh = (float)a; ds.xl = (float)(a - (double)ds.xh);
  ds.yh = (float)b; ds.yl = (float)(b - (double)ds.yh);
  ds.zh = (float)c; ds.zl = (float)(c - (double)ds.zh);
  k_fillps_fftx_r<M1, M2><<<grid, 128, 0, s>>>(g, fu, fv, fw, S, twM, twN, ds, rs.phi1, rs.fi, rs.fj, rs.fk);
  return true;
}
bool fftx_r(cudaStream_t s, const Geo &g, const float *fu, const float *fv, float *fw, float2 *S, const float2 *twM,
            const float2 *twN, double a, double b, double c, const PoissonResid &rs) {
  switch (g.I / 2) {
    case 16: return launch_fftx_r<4, 4>(s, g, fu, fv, fw, S, twM, twN, a, b, c, rs);
    case 32: return launch_fftx_r<8, 4>(s, g, fu, fv, fw, S, twM, twN, a, b, c, rs);
    case 64: return launch_fftx_r<8, 8>(s, g, fu, fv, fw, S, twM, twN, a, b, c, rs);
    case 128: return launch_fftx_r<16, 8>(s, g, fu, fv, fw, S, twM, twN, a, b, c, rs);
    case 256: return launch_fftx_r<16, 16>(s, g, fu, fv, fw, S, twM, twN, a, b, c, rs);
    default: return false;
  }
}
bool poisson_fused_residual_ok(const Geo &g) { return reg_n2(g.I / 2) && reg_n2(g.J) && g.I % 4 == 0; }

// ---------------------------------------------------------------------------
// fillps + forward real FFT along x.  One CTA handles ROWS rows (j,k).
// Reads the forced predictor (fu,fv,fw) with the bounduvw(dudt) wall values
// w(0)=w(kmax)=0 applied (and stored back into fw plane K).
// ---------------------------------------------------------------------------
template <typename TIn, typename T, typename TA, bool DF = false>
__global__ void __launch_bounds__(128) k_fillps_fftx(Geo g, FftPlan plx, const TIn *__restrict__ fu,
                                                     const TIn *__restrict__ fv, TIn *__restrict__ fw,
                                                     typename cpx<T>::t *__restrict__ S,
                                                     const typename cpx<T>::t *__restrict__ twM,
                                                     const typename cpx<T>::t *__restrict__ twN, double dtidxi,
                                                     double dtidyi, double dtidzi, int rows) {
  typedef typename cpx<T>::t C;
  extern __shared__ unsigned char smraw[];
  C *A = reinterpret_cast<C *>(smraw);
  const int M = g.I / 2;
  C *B = A + rows * M;
  const int row0 = blockIdx.x * rows;
  const int nrow = g.J * g.K;
  const float fx_hi = (float)dtidxi, fx_lo = (float)(dtidxi - (double)fx_hi);
  const float fy_hi = (float)dtidyi, fy_lo = (float)(dtidyi - (double)fy_hi);
  const float fz_hi = (float)dtidzi, fz_lo = (float)(dtidzi - (double)fz_hi);
  (void)fx_lo; (void)fy_lo; (void)fz_lo;
  // 1. right-hand side, packed z_m = x_{2m} + i x_{2m+1}
  for (int t = threadIdx.x; t < rows * g.I; t += blockDim.x) {
    const int r = t / g.I, i = t - r * g.I;
    const int row = row0 + r;
    T val = 0;
    if (row < nrow) {
      const int j = row % g.J, k = row / g.J + 1;
      const long c = fidx(g, i, j, k);
      if constexpr (DF) {
        // divergence residual in double-float arithmetic: exact differences
        // of the FP32 velocities, products with the split FP64 factors
        const float wk = (k == g.K) ? 0.f : (float)fw[c];
        const float wkm = (float)fw[c - g.plane];
        if (k == g.K) fw[c] = (TIn)0;
        const float vjm = (float)fv[fidx(g, i, j == 0 ? g.J - 1 : j - 1, k)];
        const float uim = (float)fu[fidx(g, i == 0 ? g.I - 1 : i - 1, j, k)];
        float dh, dl, th, tl, sh, sl;
        two_sum(wk, -wkm, dh, dl);
        df_mul(dh, dl, fz_hi, fz_lo, sh, sl);
        two_sum((float)fv[c], -vjm, dh, dl);
        df_mul(dh, dl, fy_hi, fy_lo, th, tl);
        df_add(sh, sl, th, tl, sh, sl);
        two_sum((float)fu[c], -uim, dh, dl);
        df_mul(dh, dl, fx_hi, fx_lo, th, tl);
        df_add(sh, sl, th, tl, sh, sl);
        val = (T)(sh + sl);
      } else {
        // walls: w(kmax) = 0 (bounduvw on dudt), plane 0 holds w(0) = 0;
        // periodic z: w(kmax) is an unknown and w(0) = w(kmax)
        const TA wk = (k == g.K && !g.zper) ? (TA)0 : (TA)fw[c];
        const TA wkm = (TA)fw[(k == 1 && g.zper) ? c + (long)(g.K - 1) * g.plane : c - g.plane];
        if (k == g.K && !g.zper) fw[c] = (TIn)0;
        const TA vjm = (TA)fv[fidx(g, i, j == 0 ? g.J - 1 : j - 1, k)];
        const TA uim = (TA)fu[fidx(g, i == 0 ? g.I - 1 : i - 1, j, k)];
        val = (T)((wk - wkm) * (TA)dtidzi + ((TA)fv[c] - vjm) * (TA)dtidyi + ((TA)fu[c] - uim) * (TA)dtidxi);
      }
    }
    T *Ar = reinterpret_cast<T *>(A + r * M);
    Ar[i] = val;
  }
  __syncthreads();
  C *Z = fft_smem1<C>(A, B, M, rows, M, plx, twM, 0);
  // 2. unpack to X_k, k = 0..M  (X_k = E_k + W_N^k O_k)
  for (int t = threadIdx.x; t < rows * (M + 1); t += blockDim.x) {
    const int r = t / (M + 1), kx = t - r * (M + 1);
    const int row = row0 + r;
    if (row >= nrow) continue;
    const C Zk = Z[r * M + (kx == M ? 0 : kx)];
    const C Zc = cconj(Z[r * M + (kx == 0 ? 0 : M - kx)]);
    const C E = cscale(cadd(Zk, Zc), (T)0.5);
    const C D = csub(Zk, Zc);
    const C O = cmk<C>(D.y * (T)0.5, -D.x * (T)0.5);  // D/(2i)
    const C X = cadd(E, cmul(twN[kx], O));
    S[(long)row * g.MX + kx] = X;
  }
}

// complex FFT along y for a tile of COLS kx-columns of one k-plane, in place.
template <typename T>
__global__ void __launch_bounds__(256) k_ffty(Geo g, FftPlan ply, typename cpx<T>::t *__restrict__ S,
                                              const typename cpx<T>::t *__restrict__ twJ, int cols, int inv) {
  typedef typename cpx<T>::t C;
  extern __shared__ unsigned char smraw[];
  // each column is stored contiguously (row length J+1 to spread the banks),
  // so the Stockham stages access shared memory with unit stride
  const int LD = g.J + 1;
  C *A = reinterpret_cast<C *>(smraw);
  C *B = A + LD * cols;
  const int kx0 = blockIdx.x * cols;
  const int k = blockIdx.y;
  C *plane = S + (long)k * g.J * g.MX;
  for (int t = threadIdx.x; t < g.J * cols; t += blockDim.x) {
    const int jy = t / cols, cx = t - jy * cols;
    const int kx = kx0 + cx;
    A[cx * LD + jy] = (kx < g.MX) ? plane[(long)jy * g.MX + kx] : cmk<C>((T)0, (T)0);
  }
  __syncthreads();
  C *Y = fft_smem1<C>(A, B, g.J, cols, LD, ply, twJ, inv);
  for (int t = threadIdx.x; t < g.J * cols; t += blockDim.x) {
    const int jy = t / cols, cx = t - jy * cols;
    const int kx = kx0 + cx;
    if (kx < g.MX) plane[(long)jy * g.MX + kx] = Y[cx * LD + jy];
  }
}

// Thomas sweep along z for every (kx,ky) (solver.f90:94-134), FP64.  With
// R = dzi^2 r, r the forward value, both sweeps need one factor per (k, |ky|,
// kx), c_k = dzi^2 / den_k (den_k the pivots; 0 in the last plane of the zero
// mode, which is pinned there):
//   R_k = c_k (d_k - R_(k-1)),   X_k = R_k - c_k X_(k+1),   x = X oscale,
// oscale the transforms' scale over dzi^2.
//
// Periodic z (CYC): Sherman-Morrison around the sweep (T: diagonal -2 a2 + xy
// with its two ends changed, off-diagonals a2 = dzi^2; u = (gamma, 0.., 0, a2),
// gamma = -b), the zero mode pinned at its last plane.  Tables behind the c_k:
// z = T^-1 u and gi = 1 / (gamma (1 + z_0 + a2 z_(K-1) / gamma)).  T is
// symmetric, so the factor of the correction, f = (y_0 + a2 y_(K-1) / gamma)
// gamma gi with y = T^-1 r, is (z . r) gi: known after the forward sweep, and
// the back substitution stores y - f z at once.
//
// Bound by the instructions of each thread's chain where columns are few, by
// memory where they are many.  Real and imaginary parts do not meet, so each
// has a thread; the next planes are loaded while the current ones are worked
// on.  64^3 cyclic: 40 -> 22 us, 96 x 108 x 75: 45 -> 19, 384 x 192 x 128:
// 104 -> 78 (a thread per complex column, pivots and dzi^2 apart).
template <bool CYC>
__global__ void __launch_bounds__(64) k_thomas(Geo g, double *__restrict__ S, const double *__restrict__ tab,
                                               double oscale) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int ncol = g.MX * g.J;
  if (e >= 2l * ncol) return;
  const int t = (int)(e >> 1), ky = t / g.MX, kx = t - ky * g.MX;
  const int kyy = ky <= g.J / 2 ? ky : g.J - ky;
  const int sst = 2 * ncol, zst = (g.J / 2 + 1) * g.MX, K = g.K;
  const double *cp = tab + kyy * g.MX + kx, *zp = cp + (long)K * zst;
  double *s = S + e;
  constexpr int PF = 8;
  double v[2][PF], c[2][PF], z[2][CYC ? PF : 1];
  double r = 0., f = 0.;
  // plane k0 + q (forward), k0 - q (backward)
  auto load = [&](int slot, int k0, int dir) {
    const double *sk = s + (long)k0 * sst, *ck = cp + (long)k0 * zst, *zk = zp + (long)k0 * zst;
    const int n = dir > 0 ? K - k0 : k0 + 1;
#pragma unroll
    for (int q = 0; q < PF; ++q)
      if (q < n) {
        v[slot][q] = sk[(long)(dir * q) * sst];
        c[slot][q] = ck[(long)(dir * q) * zst];
        if constexpr (CYC) z[slot][q] = zk[(long)(dir * q) * zst];
      }
  };
  auto fwd = [&](int slot, int k0) {
    double *sk = s + (long)k0 * sst;
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      if (k0 + q >= K) break;
      if constexpr (CYC) f = fma(z[slot][q], v[slot][q], f);
      r = fma(-c[slot][q], r, c[slot][q] * v[slot][q]);
      sk[(long)q * sst] = r;
    }
  };
  auto bwd = [&](int slot, int k0) {
    double *sk = s + (long)k0 * sst;
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      if (k0 - q < 0) break;
      r = fma(-c[slot][q], r, v[slot][q]);
      sk[-(long)q * sst] = CYC ? fma(f, z[slot][q], r * oscale) : r * oscale;
    }
  };
  load(0, 0, 1);
  for (int k0 = 0; k0 < K; k0 += 2 * PF) {
    if (k0 + PF < K) load(1, k0 + PF, 1);
    fwd(0, k0);
    if (k0 + PF >= K) break;
    if (k0 + 2 * PF < K) load(0, k0 + 2 * PF, 1);
    fwd(1, k0 + PF);
  }
  // z . r is in units of the right-hand side, z of the solution's
  if constexpr (CYC) f *= -zp[(long)K * zst] * (g.dzi * g.dzi) * oscale;
  r = 0.;
  load(0, K - 1, -1);
  for (int k0 = K - 1; k0 >= 0; k0 -= 2 * PF) {
    if (k0 - PF >= 0) load(1, k0 - PF, -1);
    bwd(0, k0);
    if (k0 - PF < 0) break;
    if (k0 - 2 * PF >= 0) load(0, k0 - 2 * PF, -1);
    bwd(1, k0 - PF);
  }
}

// The tables of k_thomas<true>, one thread per (kx, |ky|).  The zero mode is
// pinned at its last plane: rows 0..K-2 alone, z = 0 (cp = iv = 0 in row K-1).
// Products are rounded one by one, as on a host.  Formed here rather than there
// and copied (2 K entries a column): a
// context of 64^3 cells is ready 0.6 ms earlier.
__global__ void __launch_bounds__(64) k_cyclic_tables(Geo g, const double *__restrict__ xrt,
                                                      const double *__restrict__ yrt, double *__restrict__ tab) {
  const long nz = (long)(g.J / 2 + 1) * g.MX, col = blockIdx.x * 64l + threadIdx.x;
  if (col >= nz) return;
  const int K = g.K;
  const double a2 = g.dzi * g.dzi, xy = xrt[col % g.MX] + yrt[col / g.MX], bb = -2. * a2 + xy, gamma = -bb;
  const bool zero = xy == 0.;
  double *cp = tab + col, *z = cp + K * nz;
  double c = 0., zz = 0.;
  for (int k = 0; k < K; ++k) {
    const bool last = k == K - 1;
    double den = zero ? bb : (k == 0 ? bb - gamma : (last ? bb - a2 * a2 / gamma : bb));
    den -= __dmul_rn(a2, c);
    const double v = zero && last ? 0. : 1. / den;
    c = a2 * v;
    // forward sweep of T z = u, u = (gamma, 0.., 0, a2)
    zz = zero ? 0. : ((k == 0 ? gamma : (last ? a2 : 0.)) - __dmul_rn(a2, zz)) * v;
    cp[k * nz] = c;
    z[k * nz] = zz;
  }
  const double zl = zz;
  for (int k = K - 2; k >= 0; --k) {
    zz = z[k * nz] - __dmul_rn(cp[k * nz], zz);
    z[k * nz] = zz;
  }
  tab[2 * K * nz + col] = zero ? 0. : 1. / (gamma * (1. + zz + a2 * zl / gamma));
}
void launch_cyclic_tables(cudaStream_t s, const Geo &g, const double *xrt, const double *yrt, double *tab) {
  const long nz = (long)(g.J / 2 + 1) * g.MX;
  k_cyclic_tables<<<(unsigned)((nz + 63) / 64), 64, 0, s>>>(g, xrt, yrt, tab);
}

// The same sweep for the mixed form in double-float arithmetic (pairs of FP32
// with error-free products and sums, ~48 significant bits) on the FP32 pipes;
// GB300 issues FP64 at 1/64 of the FP32 rate.  Table: c_k, formed in FP64 and
// split hi + lo.  The recurrence carries its value in double-float from plane
// to plane; the forward intermediate between the sweeps is kept in the FP32
// spectrum; 1 / dzi^2 (a pair) and the transforms' scale are applied at the
// final FP32 store.  256^3:
// 70 -> 65 us, 512 x 512 x 256: 271 -> 231.
__global__ void __launch_bounds__(64) k_thomas_df(Geo g, float *__restrict__ S, const float2 *__restrict__ tab,
                                                  float iah, float ial, float fscale) {
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const int ncol = g.MX * g.J;
  if (e >= 2l * ncol) return;
  const int t = (int)(e >> 1), ky = t / g.MX, kx = t - ky * g.MX;
  const int kyy = ky <= g.J / 2 ? ky : g.J - ky;
  const int sst = 2 * ncol, zst = (g.J / 2 + 1) * g.MX, K = g.K;
  const float2 *cp = tab + kyy * g.MX + kx;
  float *s = S + e;
  constexpr int PF = 16;
  float v[2][PF];
  float2 c[2][PF];
  float rh = 0.f, rl = 0.f;
  auto load = [&](int slot, int k0, int dir) {
    const float *sk = s + (long)k0 * sst;
    const float2 *ck = cp + (long)k0 * zst;
    const int n = dir > 0 ? K - k0 : k0 + 1;
#pragma unroll
    for (int q = 0; q < PF; ++q)
      if (q < n) {
        v[slot][q] = sk[(long)(dir * q) * sst];
        c[slot][q] = ck[(long)(dir * q) * zst];
      }
  };
  auto fwd = [&](int slot, int k0) {
    float *sk = s + (long)k0 * sst;
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      if (k0 + q >= K) break;
      float h, l;
      df_add(v[slot][q], 0.f, -rh, -rl, h, l);
      df_mul(h, l, c[slot][q].x, c[slot][q].y, rh, rl);
      sk[(long)q * sst] = rh;
    }
  };
  auto out = [&]() { return fmaf(rh, iah, fmaf(rh, ial, rl * iah)) * fscale; };
  auto bwd = [&](int slot, int k0) {
    float *sk = s + (long)k0 * sst;
#pragma unroll
    for (int q = 0; q < PF; ++q) {
      if (k0 - q < 0) break;
      float h, l;
      df_mul(c[slot][q].x, c[slot][q].y, rh, rl, h, l);
      df_add(v[slot][q], 0.f, -h, -l, rh, rl);
      sk[-(long)q * sst] = out();
    }
  };
  load(0, 0, 1);
  for (int k0 = 0; k0 < K; k0 += 2 * PF) {
    if (k0 + PF < K) load(1, k0 + PF, 1);
    fwd(0, k0);
    if (k0 + PF >= K) break;
    if (k0 + 2 * PF < K) load(0, k0 + 2 * PF, 1);
    fwd(1, k0 + PF);
  }
  // the last plane is final, and goes on unrounded
  s[(long)(K - 1) * sst] = out();
  load(0, K - 2, -1);
  for (int k0 = K - 2; k0 >= 0; k0 -= 2 * PF) {
    if (k0 - PF >= 0) load(1, k0 - PF, -1);
    bwd(0, k0);
    if (k0 - PF < 0) break;
    if (k0 - 2 * PF >= 0) load(0, k0 - 2 * PF, -1);
    bwd(1, k0 - PF);
  }
}

// inverse real FFT along x: spectrum row -> phi(i,j,k), k = 1..K
template <typename T>
__global__ void __launch_bounds__(128) k_ifftx(Geo g, FftPlan plx, const typename cpx<T>::t *__restrict__ S,
                                               T *__restrict__ phi, const typename cpx<T>::t *__restrict__ twM,
                                               const typename cpx<T>::t *__restrict__ twN, int rows) {
  typedef typename cpx<T>::t C;
  extern __shared__ unsigned char smraw[];
  C *A = reinterpret_cast<C *>(smraw);
  const int M = g.I / 2;
  C *B = A + rows * M;
  C *X = B + rows * M;  // rows*(M+1) spectrum staging
  const int row0 = blockIdx.x * rows;
  const int nrow = g.J * g.K;
  for (int t = threadIdx.x; t < rows * (M + 1); t += blockDim.x) {
    const int r = t / (M + 1), kx = t - r * (M + 1);
    const int row = row0 + r;
    X[t] = row < nrow ? S[(long)row * g.MX + kx] : cmk<C>((T)0, (T)0);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < rows * M; t += blockDim.x) {
    const int r = t / M, kx = t - r * M;
    const C Xk = X[r * (M + 1) + kx];
    const C Xc = cconj(X[r * (M + 1) + (M - kx)]);
    const C E = cscale(cadd(Xk, Xc), (T)0.5);
    const C O = cmul(cscale(csub(Xk, Xc), (T)0.5), cconj(twN[kx]));
    A[r * M + kx] = cadd(E, cmk<C>(-O.y, O.x));  // E + i O
  }
  __syncthreads();
  C *Z = fft_smem1<C>(A, B, M, rows, M, plx, twM, 1);
  for (int t = threadIdx.x; t < rows * g.I; t += blockDim.x) {
    const int r = t / g.I, i = t - r * g.I;
    const int row = row0 + r;
    if (row >= nrow) continue;
    const int j = row % g.J, k = row / g.J + 1;
    const T *Zr = reinterpret_cast<const T *>(Z + r * M);
    phi[fidx(g, i, j, k)] = Zr[i];
  }
}

// Thomas sweep along z between the forward and inverse transforms
template <typename T>
void launch_thomas(cudaStream_t s, const Geo &g, typename cpx<T>::t *S, const double *zt, const float2 *thomas_df) {
  const long n = 2l * g.MX * g.J;
  // small blocks: the columns spread over the SMs (FP64: each has its own slow
  // pipe)
  const int bs = n < 64 * 1216 ? 32 : 64;
  const unsigned nb = (unsigned)((n + bs - 1) / bs);
  const double oscale = 1.0 / ((double)(g.I / 2) * g.J) / (g.dzi * g.dzi);
  if constexpr (sizeof(T) == 4) {
    const double ia = 1.0 / (g.dzi * g.dzi);
    const float iah = (float)ia;
    k_thomas_df<<<nb, bs, 0, s>>>(g, (float *)S, thomas_df, iah, (float)(ia - (double)iah),
                                  (float)(1.0 / ((double)(g.I / 2) * g.J)));
  } else if (g.zper) {
    k_thomas<true><<<nb, bs, 0, s>>>(g, (double *)S, zt, oscale);
  } else {
    k_thomas<false><<<nb, bs, 0, s>>>(g, (double *)S, zt, oscale);
  }
}

template <typename TIn, typename T>
void launch_poisson(cudaStream_t s, const Geo &g, const FftPlan &plx, const FftPlan &ply, const TIn *fu,
                    const TIn *fv, TIn *fw, void *spec, T *phi, const void *twM, const void *twN, const void *twJ,
                    const double *zt, double dtidxi, double dtidyi, double dtidzi, int *launches, bool res64,
                    const float2 *thomas_df, PoissonHook hook, PoissonResid resid) {
  typedef typename cpx<T>::t C;
  C *S = reinterpret_cast<C *>(spec);
  const int M = g.I / 2;
  const int rows = g.I <= 256 ? 4 : 2;
  const int nrow = g.J * g.K;
  const size_t smx = (size_t)2 * rows * M * sizeof(C);
  // the passes in registers take every transform they have a plan for; the
  // divergence residual (res64) keeps its own first transform
  bool plan;
  if constexpr (sizeof(T) == 4) plan = fft_stage_ok(g);
  else plan = fft_radix_ok<T>(g);
  bool done = false;
  hook(0, 1);
  if constexpr (sizeof(TIn) == sizeof(T)) {
    if (plan && !res64) {
      if constexpr (sizeof(T) == 4) fft_stage_fillps_x(s, g, fu, fv, fw, spec, twM, twN, dtidxi, dtidyi, dtidzi);
      else fft_radix_fillps_x<T>(s, g, fu, fv, fw, spec, twM, twN, dtidxi, dtidyi, dtidzi);
      done = true;
    }
  }
  if constexpr (sizeof(T) == 4 && sizeof(TIn) == 4) {
    if (!done && res64 && poisson_fused_residual_ok(g))
      done = fftx_r(s, g, fu, fv, fw, (float2 *)spec, (const float2 *)twM, (const float2 *)twN, dtidxi, dtidyi, dtidzi,
                    resid);
  }
  if (!done) {
    if (res64 && sizeof(TIn) == 4)
      k_fillps_fftx<TIn, T, float, true><<<(nrow + rows - 1) / rows, 128, smx, s>>>(
          g, plx, fu, fv, fw, S, (const C *)twM, (const C *)twN, dtidxi, dtidyi, dtidzi, rows);
    else if (res64)
      k_fillps_fftx<TIn, T, double><<<(nrow + rows - 1) / rows, 128, smx, s>>>(
          g, plx, fu, fv, fw, S, (const C *)twM, (const C *)twN, dtidxi, dtidyi, dtidzi, rows);
    else
      k_fillps_fftx<TIn, T, TIn><<<(nrow + rows - 1) / rows, 128, smx, s>>>(
          g, plx, fu, fv, fw, S, (const C *)twM, (const C *)twN, dtidxi, dtidyi, dtidzi, rows);
  }
  hook(0, 0);
  const int cols = 8;
  const size_t smy = (size_t)2 * (g.J + 1) * cols * sizeof(C);
  const dim3 gy((g.MX + cols - 1) / cols, g.K);
  auto ffty = [&](int inv) {
    if (!plan) k_ffty<T><<<gy, 256, smy, s>>>(g, ply, S, (const C *)twJ, cols, inv);
    else if constexpr (sizeof(T) == 4) fft_stage_y(s, g, spec, twJ, inv);
    else fft_radix_y<T>(s, g, spec, twJ, inv);
  };
  hook(1, 1);
  ffty(0);
  hook(1, 0);
  hook(2, 1);
  launch_thomas<T>(s, g, S, zt, thomas_df);
  hook(2, 0);
  hook(3, 1);
  ffty(1);
  hook(3, 0);
  hook(4, 1);
  if (plan) {
    if constexpr (sizeof(T) == 4) fft_stage_ix(s, g, spec, phi, twM, twN);
    else fft_radix_ix<T>(s, g, spec, phi, twM, twN);
  } else {
    const size_t smi = (size_t)(2 * rows * M + rows * (M + 1)) * sizeof(C);
    k_ifftx<T><<<(nrow + rows - 1) / rows, 128, smi, s>>>(g, plx, S, phi, (const C *)twM, (const C *)twN, rows);
  }
  hook(4, 0);
  if (launches) *launches += 5;
}

template <typename T>
int poisson_set_smem_limits() {
  int st;
  if constexpr (sizeof(T) == 4) st = fft_stage_set_smem_limits();
  else st = fft_radix_set_smem_limits<T>();
  if (st != 0) return -1;
  cudaError_t e[4];
  e[0] = cudaFuncSetAttribute(k_fillps_fftx<T, T, double>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (sizeof(T) == 4)
    if (cudaFuncSetAttribute(k_fillps_fftx<T, T, float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             200 * 1024) != cudaSuccess)
      return -1;
  e[1] = cudaFuncSetAttribute(k_fillps_fftx<T, T, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  e[2] = cudaFuncSetAttribute(k_ffty<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  e[3] = cudaFuncSetAttribute(k_ifftx<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  for (cudaError_t x : e)
    if (x != cudaSuccess) return -1;
  return 0;
}

template void launch_poisson<double, double>(cudaStream_t, const Geo &, const FftPlan &, const FftPlan &,
                                             const double *, const double *, double *, void *, double *,
                                             const void *, const void *, const void *, const double *, double, double,
                                             double, int *, bool, const float2 *, PoissonHook, PoissonResid);
template void launch_poisson<float, float>(cudaStream_t, const Geo &, const FftPlan &, const FftPlan &,
                                           const float *, const float *, float *, void *, float *, const void *,
                                           const void *, const void *, const double *, double, double, double, int *,
                                           bool, const float2 *, PoissonHook, PoissonResid);
template int poisson_set_smem_limits<double>();
template int poisson_set_smem_limits<float>();

}  // namespace ibmk
