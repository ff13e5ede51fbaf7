// fft_stage_kernels.cu -- the FP32 transforms of the pressure solve: fillps +
// real FFT along x, complex FFT along y, inverse real FFT along x, for lengths
// with up to six radix-4/2/3 stages.
//
// Same stages and roundings as the radix-4/2/3 Stockham stages of fft_smem (4s,
// then 2, then 3s; W_N^m from the table) and, where both lengths are 16, 32,
// 64, 128 or 256, as the four-step scheme of k_fillps_fftx_r: the FP32
// projection leaves a pressure whose rounding noise is far above that of its
// velocities, so another summation order would be another pressure.  What
// changes is where the elements are between the stages: two consecutive stages
// make one pass in registers, the first pass takes its elements from global
// memory (fillps: the divergence formed on the fly) and the last one puts them
// back, so a transform crosses shared memory once or twice instead of once a
// stage plus staging (five to seven times at 384 and 768).  Products are fused
// by hand (cmul), since which of two the compiler fuses depends on the context.
// Bound by L2/HBM traffic and latency: all loads of a butterfly are issued
// together.  Measured, us a launch, the stages (or the four-step kernels they
// replaced at powers of two) -> these:
//   512 x 512 x 256: fillps+x 584 -> 293, y 433 -> 140, inverse x 399 -> 125
//   384 x 384 x 192: fillps+x 254 -> 111, y 146 -> 58, inverse x 178 -> 60
//   256^3 (four-step): fillps+x 73 -> 75, y 44 -> 26, inverse x 37.5 -> 37.2
// (a spectrum read and written once at the copy rate: 79 us at 512 x 512 x 256)
#include <type_traits>

#include "kernels.cuh"

namespace ibmk {
namespace {

// The transforms of two lengths: what a pass may be made of.
enum { M_SMALL = 0, M_BIG = 1, M_FOUR = 2 };  // stages, radices up to 9 / up to 16; the four-step scheme
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a b + c d: one product rounded, the other one fused (first: a b)
__device__ __forceinline__ float dot2(float a, float b, float c, float d, bool first) {
  return first ? fmaf(a, b, __fmul_rn(c, d)) : fmaf(c, d, __fmul_rn(a, b));
}
template <bool FIRST> __device__ __forceinline__ float2 cmul(float2 a, float2 w) {  // FIRST: of the imaginary part
  return make_float2(dot2(a.x, w.x, -a.y, w.y, true), dot2(a.x, w.y, a.y, w.x, FIRST));
}
template <int INV> __device__ __forceinline__ float2 rot(float2 a) {  // times -i (inverse: +i)
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
template <int INV> __device__ __forceinline__ float2 wdir(float2 w) { return INV ? make_float2(w.x, -w.y) : w; }

template <int R, int INV> struct Dft;
template <int INV> struct Dft<1, INV> {
  static __device__ __forceinline__ void run(float2 *) {}
};
template <int INV> struct Dft<2, INV> {
  static __device__ __forceinline__ void run(float2 *v) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b); v[1] = csub(a, b);
  }
};
template <int INV> struct Dft<3, INV> {
  static __device__ __forceinline__ void run(float2 *v) {
    const float s3 = 0.86602540378443864676372317075294f;
    const float2 s = cadd(v[1], v[2]), d = rot<INV>(csub(v[1], v[2]));
    const float2 t = make_float2(fmaf(-0.5f, s.x, v[0].x), fmaf(-0.5f, s.y, v[0].y));
    v[0] = cadd(v[0], s);
    v[1] = make_float2(fmaf(s3, d.x, t.x), fmaf(s3, d.y, t.y));
    v[2] = make_float2(fmaf(-s3, d.x, t.x), fmaf(-s3, d.y, t.y));
  }
};
template <int INV> struct Dft<4, INV> {
  static __device__ __forceinline__ void run(float2 *v) {
    const float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]),
                 t3 = rot<INV>(csub(v[1], v[3]));
    v[0] = cadd(t0, t2); v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3); v[3] = csub(t1, t3);
  }
};
// times exp(-+ 2 pi i m / 16); fuse: bit 0 the real part's first product, bit
// 1 the imaginary part's
template <int INV> __device__ __forceinline__ float2 root(float2 a, int m, int fuse) {
  constexpr float c1 = 0.92387953251128675613f, r2 = 0.70710678118654752440f, s1 = 0.38268343236508977173f;
  const float cs[10] = {1.f, c1, r2, s1, 0.f, -s1, -r2, -c1, -1.f, -c1};
  const float sn[10] = {0.f, s1, r2, c1, 1.f, c1, r2, s1, 0.f, -s1};
  const float c = cs[m], s = sn[m];
  return INV ? make_float2(dot2(a.x, c, -a.y, s, fuse & 1), dot2(a.y, c, a.x, s, fuse & 2))
             : make_float2(dot2(a.x, c, a.y, s, fuse & 1), dot2(a.y, c, -a.x, s, fuse & 2));
}
template <int INV> struct Dft<8, INV> {  // the four-step scheme's: n = n2 + 2 n1, k = k1 + 4 k2
  static __device__ __forceinline__ void run(float2 *v) {
    float2 a[4] = {v[0], v[2], v[4], v[6]}, b[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, INV>::run(a);
    Dft<4, INV>::run(b);
    b[1] = root<INV>(b[1], 2, INV ? 1 : 2);
    b[2] = rot<INV>(b[2]);
    b[3] = root<INV>(b[3], 6, INV ? 1 : 2);
#pragma unroll
    for (int k = 0; k < 4; ++k) { v[k] = cadd(a[k], b[k]); v[k + 4] = csub(a[k], b[k]); }
  }
};
template <int INV> struct Dft<16, INV> {  // n = n2 + 4 n1, k = k1 + 4 k2
  static __device__ __forceinline__ void run(float2 *v) {
    float2 a[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int n = 0; n < 4; ++n) a[b][n] = v[b + 4 * n];
      Dft<4, INV>::run(a[b]);
    }
    // (a[2][2] times -+i: the product with cos = 0 and sin = 1, exact)
#pragma unroll
    for (int b = 1; b < 4; ++b)
#pragma unroll
      for (int k = 1; k < 4; ++k) a[b][k] = b * k == 4 ? rot<INV>(a[b][k]) : root<INV>(a[b][k], b * k, INV ? 1 : (b * k == 2 ? 1 : (b * k == 6 ? 2 : 3)));
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float2 q[4] = {a[0][c], a[1][c], a[2][c], a[3][c]};
      Dft<4, INV>::run(q);
#pragma unroll
      for (int d = 0; d < 4; ++d) v[c + 4 * d] = q[d];
    }
  }
};

// A pass: two consecutive stages of radices R1, R2 (R2 = 1: one stage).  Kinds
// 8 and 9 are the four-step scheme's register DFTs.
template <int R1_, int R2_> struct KindT { static constexpr int R1 = R1_, R2 = R2_, R = R1_ * R2_; };
template <int K> struct Kind;
template <> struct Kind<0> : KindT<4, 4> {};
template <> struct Kind<1> : KindT<4, 2> {};
template <> struct Kind<2> : KindT<4, 3> {};
template <> struct Kind<3> : KindT<4, 1> {};
template <> struct Kind<4> : KindT<2, 3> {};
template <> struct Kind<5> : KindT<2, 1> {};
template <> struct Kind<6> : KindT<3, 3> {};
template <> struct Kind<7> : KindT<3, 1> {};
template <> struct Kind<8> : KindT<16, 1> {};
template <> struct Kind<9> : KindT<8, 1> {};
const int KIND_R1[10] = {4, 4, 4, 4, 2, 2, 3, 3, 16, 8}, KIND_R2[10] = {4, 2, 3, 1, 3, 1, 3, 1, 1, 1};
struct StagePlan {
  int n = 0, kind[3] = {3, 3, 3}, r[3] = {1, 1, 1}, most = 0;
};
inline int kind_of(int r1, int r2) {
  for (int q = 0; q < 10; ++q)
    if (KIND_R1[q] == r1 && KIND_R2[q] == r2) return q;
  return -1;
}
inline void add_pass(StagePlan &p, int kind) {
  p.kind[p.n] = kind;
  p.r[p.n] = KIND_R1[kind] * KIND_R2[kind];
  p.most = p.most > p.r[p.n] ? p.most : p.r[p.n];
  ++p.n;
}
// The stages of length N (4s, 2, 3s) in the fewest passes, and of those ways
// the one whose smallest pass is largest (the threads of a sequence idle
// least); n = 0: more than three passes.
inline StagePlan stage_plan(int N, bool four_step) {
  if (four_step) {
    StagePlan p;
    const int n2 = N == 16 || N == 32 ? 4 : (N == 64 || N == 128 ? 8 : 16);
    add_pass(p, kind_of(N / n2, 1));
    add_pass(p, kind_of(n2, 1));
    return p;
  }
  int st[32], ns = 0;
  while (N % 4 == 0 && ns < 30) { st[ns++] = 4; N /= 4; }
  while (N % 2 == 0 && ns < 30) { st[ns++] = 2; N /= 2; }
  while (N % 3 == 0 && ns < 30) { st[ns++] = 3; N /= 3; }
  StagePlan best;
  if (N != 1 || ns > 6) return best;
  int score = 0;
  for (int m = 0; m < 8; ++m) {  // bit q: pass q takes two stages
    StagePlan p;
    int at = 0, lo = 99;
    for (int q = 0; q < 3 && at < ns; ++q) {
      const int two = (m >> q & 1) && at + 1 < ns;
      const int kd = kind_of(st[at], two ? st[at + 1] : 1);
      if (kd < 0) { at = -1; break; }
      add_pass(p, kd);
      lo = lo < p.r[q] ? lo : p.r[q];
      at += 1 + two;
    }
    if (at != ns || p.n < 2) continue;
    if (!best.n || p.n < best.n || (p.n == best.n && lo > score)) { best = p; score = lo; }
  }
  return best;
}
inline int plan_threads(const StagePlan &pl, int N) {
  int t = 0;
  for (int q = 0; q < pl.n; ++q) t = N / pl.r[q] > t ? N / pl.r[q] : t;
  return t;
}
template <int MODE, typename F> __device__ __forceinline__ void with_kind(int k, F f) {
  if constexpr (MODE == M_FOUR) {
    if (k == 3) f(std::integral_constant<int, 3>{});
    else if (k == 8) f(std::integral_constant<int, 8>{});
    else f(std::integral_constant<int, 9>{});
  } else {
    switch (k) {
      case 1: f(std::integral_constant<int, 1>{}); return;
      case 3: f(std::integral_constant<int, 3>{}); return;
      case 4: f(std::integral_constant<int, 4>{}); return;
      case 5: f(std::integral_constant<int, 5>{}); return;
      case 6: f(std::integral_constant<int, 6>{}); return;
      case 7: f(std::integral_constant<int, 7>{}); return;
      default: break;
    }
    if constexpr (MODE == M_BIG) {
      if (k == 0) f(std::integral_constant<int, 0>{});
      else f(std::integral_constant<int, 2>{});
    }
  }
}

// A sequence of N elements by threads t = 0..T-1.  Butterfly j of a pass of
// radix R after sub-transforms of size Ns takes elements j + m N/R, k = j mod
// Ns, and leaves (j / Ns) Ns R + k + s Ns.  Its first stage's butterfly q takes
// m = q + R2 r with W_(Ns R1)^(k r); the second stage's butterfly r takes the
// r-th outputs with W_(Ns R)^((k + r Ns) q).  FIRST: Ns = 1, k = 0; LAST: Ns R =
// N, k = j.
template <int K, int INV, bool IM, bool FIRST, bool LAST, typename LD, typename ST>
__device__ __forceinline__ void pass(int N, int Ns, int t, int T, const float2 *__restrict__ tw, LD ld, ST st) {
  constexpr int R1 = Kind<K>::R1, R2 = Kind<K>::R2, R = R1 * R2;
  const int nb = N / R;
  if (FIRST) Ns = 1;
  if (LAST) Ns = nb;
  const int ws2 = nb / Ns, ws1 = ws2 * R2;
  for (int j = t; j < nb; j += T) {
    const int a = FIRST ? j : (LAST ? 0 : j / Ns), k = FIRST ? 0 : j - a * Ns;
    float2 v[R];
#pragma unroll
    for (int m = 0; m < R; ++m) v[m] = ld(j + m * nb);
    float2 b[R2][R1];
#pragma unroll
    for (int q = 0; q < R2; ++q) {
#pragma unroll
      for (int r = 0; r < R1; ++r) {
        b[q][r] = v[q + R2 * r];
        if (!FIRST && r > 0) b[q][r] = cmul<IM>(b[q][r], wdir<INV>(__ldg(&tw[k * r * ws1])));
      }
      Dft<R1, INV>::run(b[q]);
    }
#pragma unroll
    for (int r = 0; r < R1; ++r) {
      float2 c[R2];
#pragma unroll
      for (int q = 0; q < R2; ++q) {
        c[q] = b[q][r];
        if (q > 0 && !(FIRST && r == 0)) c[q] = cmul<IM>(c[q], wdir<INV>(__ldg(&tw[(k + r * Ns) * q * ws2])));
      }
      Dft<R2, INV>::run(c);
#pragma unroll
      for (int q = 0; q < R2; ++q) st(a * Ns * R + k + (r + R1 * q) * Ns, c[q]);
    }
  }
}

// Complex FFT along y of COLS neighbouring kx-columns of one plane, in place:
// COLS neighbours of 8 bytes make each access of a butterfly a full 64 or 128
// bytes, in global and (element-major, columns fastest) shared memory.
template <int MODE, int INV, int COLS>
__global__ void __launch_bounds__(MODE ? 256 : 512) k_ffty_stage(Geo g, StagePlan pl, float2 *__restrict__ S,
                                                                const float2 *__restrict__ tw, int T) {
  extern __shared__ __align__(16) unsigned char smq[];
  float2 *A = reinterpret_cast<float2 *>(smq);
  const int N = g.J, col = threadIdx.x % COLS, t = threadIdx.x / COLS;
  const int kx = blockIdx.x * COLS + col;
  const bool ok = kx < g.MX;
  float2 *__restrict__ s = S + (long)blockIdx.y * N * g.MX + (ok ? kx : 0);
  const int MX = g.MX;
  float2 *a = A + col, *b = a;
  with_kind<MODE>(pl.kind[0], [&](auto K) {
    pass<K.value, INV, MODE == M_FOUR, true, false>(N, 1, t, T, tw, [&](int m) { return s[m * MX]; },
                                           [&](int m, float2 x) { a[m * COLS] = x; });
  });
  __syncthreads();
  if (pl.n == 3) {
    b = a + N * COLS;
    with_kind<MODE>(pl.kind[1], [&](auto K) {
      pass<K.value, INV, MODE == M_FOUR, false, false>(N, pl.r[0], t, T, tw, [&](int m) { return a[m * COLS]; },
                                              [&](int m, float2 x) { b[m * COLS] = x; });
    });
    __syncthreads();
  }
  with_kind<MODE>(pl.kind[pl.n - 1], [&](auto K) {
    pass<K.value, INV, MODE == M_FOUR, false, true>(N, 0, t, T, tw, [&](int m) { return b[m * COLS]; },
                                           [&](int m, float2 x) { if (ok) s[m * MX] = x; });
  });
}

// rows of the x transforms in shared memory, padded by one element every 128
// bytes so that a butterfly's strided writes spread over the banks
__host__ __device__ constexpr int xpad(int m) { return m + m / 16; }
__host__ __device__ constexpr int xrow(int M) { return xpad(M) + 1; }

// fillps (fillps.f90:8-53) with the bounduvw(dudt) wall values w(0) =
// w(kmax) = 0 applied (and stored into fw plane K), and the real FFT along x
// of the rows row0..: z_m = x_2m + i x_(2m+1), a complex FFT of M = I/2, then
// X_k = E_k + W_I^k O_k.
template <int MODE>
__global__ void __launch_bounds__(256, 3) k_fillps_fftx_stage(Geo g, StagePlan pl, const float *__restrict__ fu,
                                                           const float *__restrict__ fv, const float *__restrict__ fw,
                                                           float *__restrict__ fwk, float2 *__restrict__ S,
                                                           const float2 *__restrict__ twM,
                                                           const float2 *__restrict__ twN, float sx, float sy, float sz,
                                                           int rows, int T) {
  extern __shared__ __align__(16) unsigned char smq[];
  const int M = g.I / 2, RS = xrow(M);
  float2 *A = reinterpret_cast<float2 *>(smq), *B = A + rows * RS;
  const int row0 = blockIdx.x * rows, nrow = g.J * g.K;
  const int r = threadIdx.x / T, t = threadIdx.x - r * T, row = row0 + r;
  float2 *a = A + r * RS, *b = B + r * RS;
  if (row < nrow) {
    const int k1 = row / g.J, j = row - k1 * g.J, k = k1 + 1;
    const long c = ((long)row + g.J) * g.I, PL = g.plane;
    const bool top = k == g.K && !g.zper;
    const float *u = fu + c, *v = fv + c, *vm = v + (j == 0 ? (long)(g.J - 1) * g.I : -(long)g.I);
    const float *w = fw + c;
    const float *wm = (k == 1 && g.zper) ? w + (long)(g.K - 1) * PL : w - PL;
    auto div = [&](float dw, float dv, float du) {
      return fmaf(du, sx, dot2(dw, sz, dv, sy, true));
    };
    with_kind<MODE>(pl.kind[0], [&](auto K) {
      pass<K.value, 0, MODE == M_FOUR, true, false>(
          M, 1, t, T, twM,
          [&](int m) {
            const int i = 2 * m;
            const float2 w2 = top ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2 *>(w + i);
            const float2 wm2 = *reinterpret_cast<const float2 *>(wm + i), v2 = *reinterpret_cast<const float2 *>(v + i),
                         vm2 = *reinterpret_cast<const float2 *>(vm + i), u2 = *reinterpret_cast<const float2 *>(u + i);
            const float um = u[i == 0 ? g.I - 1 : i - 1];
            return make_float2(div(w2.x - wm2.x, v2.x - vm2.x, u2.x - um), div(w2.y - wm2.y, v2.y - vm2.y, u2.y - u2.x));
          },
          [&](int m, float2 x) { a[xpad(m)] = x; });
    });
    if (top)  // plane K of fw (fwk: the same field; nothing reads that plane here)
      for (int m = t; m < M; m += T) *reinterpret_cast<float2 *>(fwk + c + 2 * m) = make_float2(0.f, 0.f);
  }
  __syncthreads();
  if (pl.n == 3) {
    if (row < nrow)
      with_kind<MODE>(pl.kind[1], [&](auto K) {
        pass<K.value, 0, MODE == M_FOUR, false, false>(M, pl.r[0], t, T, twM, [&](int m) { return a[xpad(m)]; },
                                              [&](int m, float2 x) { b[xpad(m)] = x; });
      });
    __syncthreads();
    float2 *q = a; a = b; b = q;
    q = A; A = B; B = q;
  }
  if (row < nrow)
    with_kind<MODE>(pl.kind[pl.n - 1], [&](auto K) {
      pass<K.value, 0, MODE == M_FOUR, false, true>(M, 0, t, T, twM, [&](int m) { return a[xpad(m)]; },
                                           [&](int m, float2 x) { b[xpad(m)] = x; });
    });
  __syncthreads();
  const int H = M / 2 + 1;  // bins 0..M/2 and their partners M - k, whose E and D are the conjugates
  for (int e = threadIdx.x; e < rows * H; e += blockDim.x) {
    const int rr = e / H, q = e - rr * H;
    if (row0 + rr >= nrow) break;
    const float2 *z = B + rr * RS;
    float2 *o = S + (long)(row0 + rr) * g.MX;
    const float2 zk = z[xpad(q)], zc = z[xpad(q == 0 ? 0 : M - q)];
    const float2 E = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y - zc.y));
    const float2 h = make_float2(0.5f * (zk.x - zc.x), 0.5f * (zk.y + zc.y));
    o[q] = cadd(E, cmul<true>(__ldg(&twN[q]), make_float2(h.y, -h.x)));  // E + W (D / 2i)
    if (M - q != q)
      o[M - q] = cadd(make_float2(E.x, -E.y), cmul<true>(__ldg(&twN[M - q]), make_float2(h.y, h.x)));
  }
}

// inverse real FFT along x: spectrum row -> phi(i,j,k), k = 1..K.  The first
// butterflies form their elements E_k + i O_k from the spectrum (each bin is
// read twice, the second time from cache).
template <int MODE>
__global__ void __launch_bounds__(256, 3) k_ifftx_stage(Geo g, StagePlan pl, const float2 *__restrict__ S,
                                                     float *__restrict__ phi, const float2 *__restrict__ twM,
                                                     const float2 *__restrict__ twN, int rows, int T) {
  extern __shared__ __align__(16) unsigned char smq[];
  const int M = g.I / 2, RS = xrow(M);
  float2 *A = reinterpret_cast<float2 *>(smq), *B = A + rows * RS;
  const int row0 = blockIdx.x * rows, nrow = g.J * g.K;
  const int r = threadIdx.x / T, t = threadIdx.x - r * T, row = row0 + r;
  float2 *a = A + r * RS, *b = B + r * RS;
  if (row < nrow) {
    const float2 *x = S + (long)row * g.MX;
    with_kind<MODE>(pl.kind[0], [&](auto K) {
      pass<K.value, 1, false, true, false>(
          M, 1, t, T, twM,
          [&](int m) {
            const float2 xk = x[m], xc = x[M - m], wn = __ldg(&twN[m]);
            const float2 E = make_float2(0.5f * (xk.x + xc.x), 0.5f * (xk.y - xc.y));
            const float2 O = cmul<false>(make_float2(0.5f * (xk.x - xc.x), 0.5f * (xk.y + xc.y)), wdir<1>(wn));
            return make_float2(E.x - O.y, E.y + O.x);
          },
          [&](int m, float2 v) { b[xpad(m)] = v; });
    });
  }
  __syncthreads();
  if (pl.n == 3) {
    if (row < nrow)
      with_kind<MODE>(pl.kind[1], [&](auto K) {
        pass<K.value, 1, false, false, false>(M, pl.r[0], t, T, twM, [&](int m) { return b[xpad(m)]; },
                                               [&](int m, float2 x) { a[xpad(m)] = x; });
      });
    __syncthreads();
    b = a;
  }
  if (row < nrow) {
    float2 *o = reinterpret_cast<float2 *>(phi + ((long)row + g.J) * g.I);
    with_kind<MODE>(pl.kind[pl.n - 1], [&](auto K) {
      pass<K.value, 1, false, false, true>(M, 0, t, T, twM, [&](int m) { return b[xpad(m)]; },
                                            [&](int m, float2 x) { o[m] = x; });
    });
  }
}

constexpr size_t STAGE_SMEM = 200 * 1024;
// columns of the y transform: a full 128-byte line where one buffer does,
// half of one where three passes take two
constexpr int ycols(int passes) { return passes == 2 ? 16 : 8; }
inline size_t ysmem(const StagePlan &pl, int N) { return (size_t)(pl.n == 2 ? 1 : 2) * N * ycols(pl.n) * sizeof(float2); }
// rows of a block of the x transforms: about 128 threads, 256 at most
inline void xshape(const StagePlan &pl, int M, int &rows, int &T, size_t &smem) {
  T = plan_threads(pl, M);
  if (T > 256) T = 256;
  rows = T >= 128 ? 1 : 128 / T;
  smem = (size_t)2 * rows * xrow(M) * sizeof(float2);
}
inline bool four_len(int N) { return N == 16 || N == 32 || N == 64 || N == 128 || N == 256; }
inline bool four_step(const Geo &g) { return four_len(g.I / 2) && four_len(g.J); }
inline bool stage_plans(const Geo &g, StagePlan &px, StagePlan &py) {
  const bool fs = four_step(g);
  px = stage_plan(g.I / 2, fs);
  py = stage_plan(g.J, fs);
  if (!px.n || !py.n) return false;
  int rows, T;
  size_t smem;
  xshape(px, g.I / 2, rows, T, smem);
  return smem <= STAGE_SMEM && ysmem(py, g.J) <= STAGE_SMEM;
}
template <int MODE, int INV, int COLS>
void ffty_go(cudaStream_t s, const Geo &g, const StagePlan &pl, float2 *S, const float2 *tw) {
  const int cap = (MODE ? 256 : 512) / COLS, t = plan_threads(pl, g.J), T = t < cap ? t : cap;
  k_ffty_stage<MODE, INV, COLS><<<dim3((g.MX + COLS - 1) / COLS, g.K), COLS * T, ysmem(pl, g.J), s>>>(g, pl, S, tw, T);
}
template <int INV> void ffty_dir(cudaStream_t s, const Geo &g, const StagePlan &pl, float2 *S, const float2 *tw) {
  if (four_step(g)) ffty_go<M_FOUR, INV, ycols(2)>(s, g, pl, S, tw);
  else if (pl.n == 2)
    pl.most > 9 ? ffty_go<M_BIG, INV, ycols(2)>(s, g, pl, S, tw) : ffty_go<M_SMALL, INV, ycols(2)>(s, g, pl, S, tw);
  else
    pl.most > 9 ? ffty_go<M_BIG, INV, ycols(3)>(s, g, pl, S, tw) : ffty_go<M_SMALL, INV, ycols(3)>(s, g, pl, S, tw);
}
template <typename F> bool big_smem(F *k) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STAGE_SMEM) == cudaSuccess;
}
template <int MODE> bool stage_limits() {
  return big_smem(k_ffty_stage<MODE, 0, ycols(2)>) && big_smem(k_ffty_stage<MODE, 1, ycols(2)>) &&
         (MODE == M_FOUR || (big_smem(k_ffty_stage<MODE, 0, ycols(3)>) && big_smem(k_ffty_stage<MODE, 1, ycols(3)>))) &&
         big_smem(k_fillps_fftx_stage<MODE>) && big_smem(k_ifftx_stage<MODE>);
}
}  // namespace

bool fft_stage_ok(const Geo &g) {
  StagePlan px, py;
  return stage_plans(g, px, py);
}
void fft_stage_fillps_x(cudaStream_t s, const Geo &g, const float *fu, const float *fv, float *fw, void *spec,
                        const void *twM, const void *twN, double sx, double sy, double sz) {
  const StagePlan pl = stage_plan(g.I / 2, four_step(g));
  int rows, t;
  size_t smem;
  xshape(pl, g.I / 2, rows, t, smem);
  auto go = [&](auto k) {
    k<<<(g.J * g.K + rows - 1) / rows, rows * t, smem, s>>>(g, pl, fu, fv, fw, fw, (float2 *)spec, (const float2 *)twM,
                                                            (const float2 *)twN, (float)sx, (float)sy, (float)sz, rows, t);
  };
  if (four_step(g)) go(k_fillps_fftx_stage<M_FOUR>);
  else if (pl.most > 9) go(k_fillps_fftx_stage<M_BIG>);
  else go(k_fillps_fftx_stage<M_SMALL>);
}
void fft_stage_y(cudaStream_t s, const Geo &g, void *spec, const void *twJ, int inv) {
  const StagePlan pl = stage_plan(g.J, four_step(g));
  if (inv) ffty_dir<1>(s, g, pl, (float2 *)spec, (const float2 *)twJ);
  else ffty_dir<0>(s, g, pl, (float2 *)spec, (const float2 *)twJ);
}
void fft_stage_ix(cudaStream_t s, const Geo &g, const void *spec, float *phi, const void *twM, const void *twN) {
  const StagePlan pl = stage_plan(g.I / 2, four_step(g));
  int rows, t;
  size_t smem;
  xshape(pl, g.I / 2, rows, t, smem);
  auto go = [&](auto k) {
    k<<<(g.J * g.K + rows - 1) / rows, rows * t, smem, s>>>(g, pl, (const float2 *)spec, phi, (const float2 *)twM,
                                                            (const float2 *)twN, rows, t);
  };
  if (four_step(g)) go(k_ifftx_stage<M_FOUR>);
  else if (pl.most > 9) go(k_ifftx_stage<M_BIG>);
  else go(k_ifftx_stage<M_SMALL>);
}
int fft_stage_set_smem_limits() { return stage_limits<M_SMALL>() && stage_limits<M_BIG>() && stage_limits<M_FOUR>() ? 0 : -1; }

}  // namespace ibmk
