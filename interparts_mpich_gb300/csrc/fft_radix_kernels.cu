// fft_radix_kernels.cu -- the FP64 transforms of the pressure solve for lengths
// that factor into two or three radices of {2, 3, 4, 6, 8, 9, 12, 16}: fillps
// + real FFT along x, complex FFT along y, inverse real FFT along x, every
// length up to about a thousand with factors 2 and 3.  (FP32: fft_stage_kernels.cu.)
//
// Stockham order, each butterfly a small DFT in registers.  The first pass
// takes its elements from global memory (fillps: the divergence formed on the
// fly) and the last one puts them back, so a transform of two radices crosses
// shared memory once, one of three radices twice, where the radix-4/2/3
// stages of fft_smem cross it once per stage plus staging (five to seven
// times for 384 and 768).  The first pass has no twiddles and the last one's
// index is the butterfly's own, so neither divides.
// Bound by FP64 issue: a radix-16 butterfly is 160 FP64 instructions, ten per
// element for four binary levels, twiddles 4 each; the real-transform
// (un)packing forms bins k and M - k together.
// Measured, us a launch, radix-4/2/3 stages -> these: 384 x 192 x 128: fillps+x
// 445 -> 421, y 287 -> 211, inverse x 331 -> 308 (0.48 T FP64 instructions/s,
// the pipe's rate); 256^3: fillps+x 833 -> 703 and inverse x 642 -> 487 with the
// threads of a row chosen so that both passes use every lane.
#include <cmath>
#include <type_traits>

#include "kernels.cuh"

namespace ibmk {
namespace {

template <typename T> struct cpx;
template <> struct cpx<double> { typedef double2 t; };
template <typename C> using real_of = decltype(C().x);

template <typename C> __device__ __forceinline__ C mk(real_of<C> a, real_of<C> b) { C r; r.x = a; r.y = b; return r; }
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <typename C> __device__ __forceinline__ C axpy(real_of<C> s, C x, C y) { return mk<C>(fma(s, x.x, y.x), fma(s, x.y, y.y)); }
// times w (inverse: times conj(w))
template <int INV, typename C> __device__ __forceinline__ C twid(C a, C w) {
  return INV ? mk<C>(fma(a.y, w.y, a.x * w.x), fma(-a.x, w.y, a.y * w.x))
             : mk<C>(fma(-a.y, w.y, a.x * w.x), fma(a.x, w.y, a.y * w.x));
}
// times -i (inverse: +i)
template <int INV, typename C> __device__ __forceinline__ C rot(C a) { return INV ? mk<C>(-a.y, a.x) : mk<C>(a.y, -a.x); }

// DFT of R elements in registers, in place, natural order
template <int R, int INV> struct Dft;
template <int INV> struct Dft<2, INV> {
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    const C a = v[0], b = v[1];
    v[0] = cadd(a, b); v[1] = csub(a, b);
  }
};
template <int INV> struct Dft<3, INV> {
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    typedef real_of<C> T;
    const C s = cadd(v[1], v[2]), d = rot<INV>(csub(v[1], v[2]));
    const C t = axpy((T)-0.5, s, v[0]);
    v[0] = cadd(v[0], s);
    v[1] = axpy((T)0.86602540378443864676372317075294, d, t);
    v[2] = axpy((T)-0.86602540378443864676372317075294, d, t);
  }
};
template <int INV> struct Dft<4, INV> {
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    const C t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]), t2 = cadd(v[1], v[3]),
            t3 = rot<INV>(csub(v[1], v[3]));
    v[0] = cadd(t0, t2); v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3); v[3] = csub(t1, t3);
  }
};
// coprime factors: index maps without twiddles (Good, J. R. Stat. Soc. B 20, 1958)
template <int INV> struct Dft<6, INV> {  // n = 3 a + 2 b, k = 3 c + 4 d (mod 6)
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    C p[3] = {v[0], v[2], v[4]}, q[3] = {v[3], v[5], v[1]};
    Dft<3, INV>::run(p);
    Dft<3, INV>::run(q);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      v[(4 * d) % 6] = cadd(p[d], q[d]);
      v[(3 + 4 * d) % 6] = csub(p[d], q[d]);
    }
  }
};
template <int INV> struct Dft<12, INV> {  // n = 3 a + 4 b, k = 9 c + 4 d (mod 12)
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    C p[4][3];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
      for (int b = 0; b < 3; ++b) p[a][b] = v[(3 * a + 4 * b) % 12];
      Dft<3, INV>::run(p[a]);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      C q[4] = {p[0][d], p[1][d], p[2][d], p[3][d]};
      Dft<4, INV>::run(q);
#pragma unroll
      for (int c = 0; c < 4; ++c) v[(9 * c + 4 * d) % 12] = q[c];
    }
  }
};
template <int INV> struct Dft<8, INV> {
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    typedef real_of<C> T;
    const T r = (T)0.70710678118654752440084436210485;
    C a[4] = {v[0], v[2], v[4], v[6]}, b[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, INV>::run(a);
    Dft<4, INV>::run(b);
    v[0] = cadd(a[0], b[0]); v[4] = csub(a[0], b[0]);
    // exp(-+ i pi/4) b1 and exp(-+ 3 i pi/4) b3 with the 1/sqrt(2) in the sums
    const C s = INV ? mk<C>(b[1].x - b[1].y, b[1].y + b[1].x) : mk<C>(b[1].x + b[1].y, b[1].y - b[1].x);
    v[1] = axpy(r, s, a[1]); v[5] = axpy(-r, s, a[1]);
    const C t = rot<INV>(b[2]);
    v[2] = cadd(a[2], t); v[6] = csub(a[2], t);
    const C u = INV ? mk<C>(-b[3].x - b[3].y, b[3].x - b[3].y) : mk<C>(b[3].y - b[3].x, -b[3].x - b[3].y);
    v[3] = axpy(r, u, a[3]); v[7] = axpy(-r, u, a[3]);
  }
};
template <int INV> struct Dft<9, INV> {  // n = b + 3 a, k = c + 3 d
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    typedef real_of<C> T;
    // exp(-2 pi i m / 9), m = 1, 2, 4
    const C w1 = mk<C>((T)0.76604444311897803520239265055542, (T)-0.64278760968653932632264340990726);
    const C w2 = mk<C>((T)0.17364817766693034885171662676931, (T)-0.98480775301220805936674302458952);
    const C w4 = mk<C>((T)-0.93969262078590838405410927732473, (T)-0.34202014332566873304409961468226);
    C a[3][3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
#pragma unroll
      for (int n = 0; n < 3; ++n) a[b][n] = v[b + 3 * n];
      Dft<3, INV>::run(a[b]);
    }
    a[1][1] = twid<INV>(a[1][1], w1);
    a[1][2] = twid<INV>(a[1][2], w2);
    a[2][1] = twid<INV>(a[2][1], w2);
    a[2][2] = twid<INV>(a[2][2], w4);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      C q[3] = {a[0][c], a[1][c], a[2][c]};
      Dft<3, INV>::run(q);
#pragma unroll
      for (int d = 0; d < 3; ++d) v[c + 3 * d] = q[d];
    }
  }
};
template <int INV> struct Dft<16, INV> {  // n = b + 4 a, k = c + 4 d
  template <typename C> static __device__ __forceinline__ void run(C *v) {
    typedef real_of<C> T;
    const T c1 = (T)0.92387953251128675612818318939679, s1 = (T)0.38268343236508977172845998403040;
    const T r = (T)0.70710678118654752440084436210485;
    const C w1 = mk<C>(c1, -s1), w3 = mk<C>(s1, -c1), w9 = mk<C>(-c1, s1);
    C a[4][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
#pragma unroll
      for (int n = 0; n < 4; ++n) a[b][n] = v[b + 4 * n];
      Dft<4, INV>::run(a[b]);
    }
    auto w2 = [&](C x) { return INV ? mk<C>(r * (x.x - x.y), r * (x.y + x.x)) : mk<C>(r * (x.x + x.y), r * (x.y - x.x)); };
    auto w6 = [&](C x) { return INV ? mk<C>(-r * (x.x + x.y), r * (x.x - x.y)) : mk<C>(r * (x.y - x.x), -r * (x.x + x.y)); };
    a[1][1] = twid<INV>(a[1][1], w1);
    a[1][2] = w2(a[1][2]);
    a[1][3] = twid<INV>(a[1][3], w3);
    a[2][1] = w2(a[2][1]);
    a[2][2] = rot<INV>(a[2][2]);
    a[2][3] = w6(a[2][3]);
    a[3][1] = twid<INV>(a[3][1], w3);
    a[3][2] = w6(a[3][2]);
    a[3][3] = twid<INV>(a[3][3], w9);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      C q[4] = {a[0][c], a[1][c], a[2][c], a[3][c]};
      Dft<4, INV>::run(q);
#pragma unroll
      for (int d = 0; d < 4; ++d) v[c + 4 * d] = q[d];
    }
  }
};

// N = r[0] r[1] (r[2]); T threads work on one sequence
struct RadixPlan {
  int n = 0, r[3] = {1, 1, 1}, most = 0;
};
// The fewest passes, then the largest smallest radix (even passes: the
// threads of a sequence idle least).
RadixPlan radix_plan(int N) {
  static const int R[8] = {2, 3, 4, 6, 8, 9, 12, 16};
  RadixPlan best;
  int score = 0;
  auto take = [&](int n, int a, int b, int c) {
    const int lo = n == 2 ? (a < b ? a : b) : (a < b ? (a < c ? a : c) : (b < c ? b : c));
    if (lo <= score) return;
    score = lo;
    best.n = n;
    best.r[0] = a; best.r[1] = b; best.r[2] = c;
    best.most = a > b ? (a > c ? a : c) : (b > c ? b : c);
  };
  for (int a : R)
    for (int b : R)
      if (a * b == N) take(2, a, b, 1);
  if (best.n) return best;
  for (int a : R)
    for (int b : R)
      for (int c : R)
        if (a * b * c == N) take(3, a, b, c);
  return best;
}
// Threads per sequence, lo..hi of them: those that leave the fewest lanes idle.
// A pass of N/R butterflies takes ceil(N/R / T) turns of all T lanes, and FP64
// instructions cost the same with half of the lanes (8 x 16 = 128 elements: a
// quarter is lost with 16 threads, nothing with 8).  Of equal ones the most.
int plan_threads(const RadixPlan &pl, int N, int lo, int hi) {
  int best = 1;
  double least = 1e30;
  for (int t = lo; t <= hi; ++t) {
    double cost = 0.;
    for (int q = 0; q < pl.n; ++q) {
      const int R = pl.r[q], nb = N / R;
      cost += (double)((nb + t - 1) / t) * t * R * (4. + 2.5 * std::log2((double)R));
    }
    if (cost <= least * (1. + 1e-9)) { least = cost < least ? cost : least; best = t; }
  }
  return best;
}
int plan_most(const RadixPlan &pl, int N) {  // one butterfly each in the pass with the most of them
  int t = 0;
  for (int q = 0; q < pl.n; ++q) t = N / pl.r[q] > t ? N / pl.r[q] : t;
  return t;
}

// call f with the radix as a compile-time constant
template <int MAXR, typename F> __device__ __forceinline__ void with_radix(int R, F f) {
  switch (R) {
    case 2: f(std::integral_constant<int, 2>{}); return;
    case 3: f(std::integral_constant<int, 3>{}); return;
    case 4: f(std::integral_constant<int, 4>{}); return;
    case 6: f(std::integral_constant<int, 6>{}); return;
    case 8: f(std::integral_constant<int, 8>{}); return;
    case 9: f(std::integral_constant<int, 9>{}); return;
    default: break;
  }
  if constexpr (MAXR > 9) {
    if (R == 12) f(std::integral_constant<int, 12>{});
    else f(std::integral_constant<int, 16>{});
  }
}

// One pass of a sequence of N elements by threads t = 0..T-1: butterfly j
// reads elements j + r N/R (times the twiddles W_(Ns R)^(k r), k = j mod Ns,
// tw[m] = W_N^m) and writes (j / Ns) Ns R + k + r Ns.
template <int R, int INV, typename C, typename LD, typename ST>
__device__ __forceinline__ void pass_first(int N, int t, int T, LD ld, ST st) {
  const int nb = N / R;
  for (int j = t; j < nb; j += T) {
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(j + r * nb);
    Dft<R, INV>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st(j * R + r, v[r]);
  }
}
template <int R, int INV, typename C, typename LD, typename ST>
__device__ __forceinline__ void pass_mid(int N, int Ns, int t, int T, const C *__restrict__ tw, LD ld, ST st) {
  const int nb = N / R, ws = nb / Ns;
  for (int j = t; j < nb; j += T) {
    const int a = j / Ns, k = j - a * Ns;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(j + r * nb);
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = twid<INV>(v[r], __ldg(&tw[k * r * ws]));
    Dft<R, INV>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st(a * Ns * R + k + r * Ns, v[r]);
  }
}
template <int R, int INV, typename C, typename LD, typename ST>
__device__ __forceinline__ void pass_last(int N, int t, int T, const C *__restrict__ tw, LD ld, ST st) {
  const int nb = N / R;
  for (int j = t; j < nb; j += T) {
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld(j + r * nb);
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = twid<INV>(v[r], __ldg(&tw[j * r]));
    Dft<R, INV>::run(v);
#pragma unroll
    for (int r = 0; r < R; ++r) st(j + r * nb, v[r]);
  }
}

// Complex FFT along y of COLS neighbouring kx-columns of one plane, in place:
// COLS neighbours of 16 bytes make each access of a butterfly a full 64 or
// 128 bytes, in global and (element-major, columns fastest) shared memory.
template <typename C, int MAXR, int INV, int COLS>
__global__ void __launch_bounds__(MAXR > 9 ? 256 : 512) k_ffty_radix(Geo g, RadixPlan pl, C *__restrict__ S,
                                                                     const C *__restrict__ tw, int T) {
  extern __shared__ __align__(16) unsigned char smq[];
  C *A = reinterpret_cast<C *>(smq);
  const int N = g.J, col = threadIdx.x % COLS, t = threadIdx.x / COLS;
  const int kx = blockIdx.x * COLS + col;
  const bool ok = kx < g.MX;
  C *__restrict__ s = S + (long)blockIdx.y * N * g.MX + (ok ? kx : 0);
  const int MX = g.MX;
  C *a = A + col, *b = a;
  with_radix<MAXR>(pl.r[0], [&](auto R) {
    pass_first<R.value, INV, C>(N, t, T, [&](int m) { return s[m * MX]; }, [&](int m, C x) { a[m * COLS] = x; });
  });
  __syncthreads();
  if (pl.n == 3) {
    b = a + N * COLS;
    with_radix<MAXR>(pl.r[1], [&](auto R) {
      pass_mid<R.value, INV, C>(N, pl.r[0], t, T, tw, [&](int m) { return a[m * COLS]; },
                                [&](int m, C x) { b[m * COLS] = x; });
    });
    __syncthreads();
  }
  with_radix<MAXR>(pl.r[pl.n - 1], [&](auto R) {
    pass_last<R.value, INV, C>(N, t, T, tw, [&](int m) { return b[m * COLS]; },
                               [&](int m, C x) { if (ok) s[m * MX] = x; });
  });
}

// rows of the x transforms in shared memory, padded by one element every 128
// bytes so that a butterfly's strided writes spread over the banks
template <typename C> __host__ __device__ constexpr int xpad(int m) { return m + m / (128 / (int)sizeof(C)); }
template <typename C> __host__ __device__ constexpr int xrow(int M) { return xpad<C>(M) + 1; }

// fillps (fillps.f90:8-53) with the bounduvw(dudt) wall values w(0) =
// w(kmax) = 0 applied (and stored into fw plane K), and the real FFT along x
// of the rows row0..: z_m = x_2m + i x_(2m+1), a complex FFT of M = I/2, then
// X_k = E_k + W_I^k O_k for k and M - k together.
template <typename T, int MAXR>
__global__ void __launch_bounds__(256) k_fillps_fftx_radix(Geo g, RadixPlan pl, const T *__restrict__ fu,
                                                           const T *__restrict__ fv, const T *__restrict__ fw,
                                                           T *__restrict__ fwk,
                                                           typename cpx<T>::t *__restrict__ S,
                                                           const typename cpx<T>::t *__restrict__ twM,
                                                           const typename cpx<T>::t *__restrict__ twN, T sx, T sy, T sz,
                                                           int rows, int T_) {
  typedef typename cpx<T>::t C;
  extern __shared__ __align__(16) unsigned char smq[];
  const int M = g.I / 2, RS = xrow<C>(M);
  C *A = reinterpret_cast<C *>(smq), *B = A + rows * RS;
  const int row0 = blockIdx.x * rows, nrow = g.J * g.K;
  const int r = threadIdx.x / T_, t = threadIdx.x - r * T_, row = row0 + r;
  C *a = A + r * RS, *b = B + r * RS;
  if (row < nrow) {
    const int k1 = row / g.J, j = row - k1 * g.J, k = k1 + 1;
    const long c = ((long)row + g.J) * g.I, PL = g.plane;
    const bool top = k == g.K && !g.zper;
    const T *u = fu + c, *v = fv + c, *vm = v + (j == 0 ? (long)(g.J - 1) * g.I : -(long)g.I);
    const T *w = fw + c;
    const T *wm = (k == 1 && g.zper) ? w + (long)(g.K - 1) * PL : w - PL;
    with_radix<MAXR>(pl.r[0], [&](auto R) {
      pass_first<R.value, 0, C>(
          M, t, T_,
          [&](int m) {
            const int i = 2 * m;
            const C w2 = top ? mk<C>((T)0, (T)0) : *reinterpret_cast<const C *>(w + i);
            const C wm2 = *reinterpret_cast<const C *>(wm + i), v2 = *reinterpret_cast<const C *>(v + i),
                    vm2 = *reinterpret_cast<const C *>(vm + i), u2 = *reinterpret_cast<const C *>(u + i);
            const T um = u[i == 0 ? g.I - 1 : i - 1];
            return mk<C>((w2.x - wm2.x) * sz + (v2.x - vm2.x) * sy + (u2.x - um) * sx,
                         (w2.y - wm2.y) * sz + (v2.y - vm2.y) * sy + (u2.y - u2.x) * sx);
          },
          [&](int m, C x) { a[xpad<C>(m)] = x; });
    });
    if (top)  // plane K of fw (fwk: the same field; nothing reads that plane here)
      for (int m = t; m < M; m += T_) *reinterpret_cast<C *>(fwk + c + 2 * m) = mk<C>((T)0, (T)0);
  }
  __syncthreads();
  if (pl.n == 3) {
    if (row < nrow)
      with_radix<MAXR>(pl.r[1], [&](auto R) {
        pass_mid<R.value, 0, C>(M, pl.r[0], t, T_, twM, [&](int m) { return a[xpad<C>(m)]; },
                                [&](int m, C x) { b[xpad<C>(m)] = x; });
      });
    __syncthreads();
    C *q = a; a = b; b = q;
    q = A; A = B; B = q;
  }
  if (row < nrow)
    with_radix<MAXR>(pl.r[pl.n - 1], [&](auto R) {
      pass_last<R.value, 0, C>(M, t, T_, twM, [&](int m) { return a[xpad<C>(m)]; },
                               [&](int m, C x) { b[xpad<C>(m)] = x; });
    });
  __syncthreads();
  const int H = M / 2 + 1;  // bins 0..M/2 and their partners M - k
  for (int e = threadIdx.x; e < rows * H; e += blockDim.x) {
    const int rr = e / H, q = e - rr * H;
    if (row0 + rr >= nrow) break;
    const C *z = B + rr * RS;
    C *o = S + (long)(row0 + rr) * g.MX;
    const C zk = z[xpad<C>(q)], zc = q == 0 ? zk : z[xpad<C>(M - q)];
    const C E = mk<C>(zk.x + zc.x, zk.y - zc.y), D = mk<C>(zk.x - zc.x, zk.y + zc.y);
    const C wn = __ldg(&twN[q]);
    const C h = mk<C>((T)0.5 * wn.x, (T)0.5 * wn.y);
    const C P = mk<C>(fma(D.x, h.y, D.y * h.x), fma(-D.x, h.x, D.y * h.y));  // W (D / 2i)
    o[q] = mk<C>(fma((T)0.5, E.x, P.x), fma((T)0.5, E.y, P.y));
    if (M - q != q) o[M - q] = mk<C>(fma((T)0.5, E.x, -P.x), fma((T)-0.5, E.y, P.y));
  }
}

// inverse real FFT along x: spectrum row -> phi(i,j,k), k = 1..K
template <typename T, int MAXR>
__global__ void __launch_bounds__(256) k_ifftx_radix(Geo g, RadixPlan pl, const typename cpx<T>::t *__restrict__ S,
                                                     T *__restrict__ phi, const typename cpx<T>::t *__restrict__ twM,
                                                     const typename cpx<T>::t *__restrict__ twN, int rows, int T_) {
  typedef typename cpx<T>::t C;
  extern __shared__ __align__(16) unsigned char smq[];
  const int M = g.I / 2, RS = xrow<C>(M);
  C *A = reinterpret_cast<C *>(smq), *B = A + rows * RS;
  const int row0 = blockIdx.x * rows, nrow = g.J * g.K;
  const int r = threadIdx.x / T_, t = threadIdx.x - r * T_, row = row0 + r;
  C *a = A + r * RS, *b = B + r * RS;
  // A_k = E + i O with E = (X_k + conj X_(M-k)) / 2, O = conj(W_k) (X_k - conj
  // X_(M-k)) / 2, and A_(M-k) = conj(E - i O)
  auto half = [&](C xk, C xc, C wn, C &E, C &O) {
    E = mk<C>((T)0.5 * (xk.x + xc.x), (T)0.5 * (xk.y - xc.y));
    const C D = mk<C>(xk.x - xc.x, xk.y + xc.y), h = mk<C>((T)0.5 * wn.x, (T)0.5 * wn.y);
    O = mk<C>(fma(D.y, h.y, D.x * h.x), fma(-D.x, h.y, D.y * h.x));
  };
  // FP64, bound by its instructions: k and M - k together, staged
  const int H = M / 2 + 1;
  for (int e = threadIdx.x; e < rows * H; e += blockDim.x) {
    const int rr = e / H, q = e - rr * H;
    if (row0 + rr >= nrow) break;
    const C *x = S + (long)(row0 + rr) * g.MX;
    C *z = A + rr * RS;
    C E, O;
    half(x[q], x[M - q], __ldg(&twN[q]), E, O);
    z[xpad<C>(q)] = mk<C>(E.x - O.y, E.y + O.x);
    if (q != 0 && M - q != q) z[xpad<C>(M - q)] = mk<C>(E.x + O.y, O.x - E.y);
  }
  __syncthreads();
  if (row < nrow)
    with_radix<MAXR>(pl.r[0], [&](auto R) {
      pass_first<R.value, 1, C>(M, t, T_, [&](int m) { return a[xpad<C>(m)]; },
                                [&](int m, C x) { b[xpad<C>(m)] = x; });
    });
  __syncthreads();
  if (pl.n == 3) {
    if (row < nrow)
      with_radix<MAXR>(pl.r[1], [&](auto R) {
        pass_mid<R.value, 1, C>(M, pl.r[0], t, T_, twM, [&](int m) { return b[xpad<C>(m)]; },
                                [&](int m, C x) { a[xpad<C>(m)] = x; });
      });
    __syncthreads();
    b = a;
  }
  if (row < nrow) {
    C *o = reinterpret_cast<C *>(phi + ((long)row + g.J) * g.I);
    with_radix<MAXR>(pl.r[pl.n - 1], [&](auto R) {
      pass_last<R.value, 1, C>(M, t, T_, twM, [&](int m) { return b[xpad<C>(m)]; }, [&](int m, C x) { o[m] = x; });
    });
  }
}

constexpr size_t RADIX_SMEM = 200 * 1024;
// columns of the y transform: a full 128-byte line where one buffer does,
// half of one where three radices take two
template <typename C> constexpr int ycols(int passes) { return (passes == 2 ? 128 : 64) / (int)sizeof(C); }
template <typename C> size_t ysmem(const RadixPlan &pl, int N) {
  return (size_t)(pl.n == 2 ? 1 : 2) * N * ycols<C>(pl.n) * sizeof(C);
}
// rows of a block of the x transforms: about 128 threads, 256 at most; three
// blocks an SM where there is a choice
template <typename C> void xshape(const RadixPlan &pl, int M, int &rows, int &T, size_t &smem) {
  int hi = plan_most(pl, M);
  if (hi > 256) hi = 256;
  auto need = [&](int t) { return (size_t)2 * (t >= 128 ? 1 : 128 / t) * xrow<C>(M) * sizeof(C); };
  int lo = hi;
  while (lo > 1 && need(lo - 1) <= 72 * 1024) --lo;
  T = plan_threads(pl, M, lo, hi);
  rows = T >= 128 ? 1 : 128 / T;
  smem = need(T);
}
template <typename C> bool radix_fits(const Geo &g, RadixPlan &px, RadixPlan &py) {
  px = radix_plan(g.I / 2);
  py = radix_plan(g.J);
  if (!px.n || !py.n) return false;
  int rows, T;
  size_t smem;
  xshape<C>(px, g.I / 2, rows, T, smem);
  return smem <= RADIX_SMEM && ysmem<C>(py, g.J) <= RADIX_SMEM;
}

template <typename C, int MAXR, int INV, int COLS>
void ffty_go(cudaStream_t s, const Geo &g, const RadixPlan &pl, C *S, const C *tw) {
  const int cap = (MAXR > 9 ? 256 : 512) / COLS, t = plan_most(pl, g.J), T = t < cap ? t : cap;
  k_ffty_radix<C, MAXR, INV, COLS><<<dim3((g.MX + COLS - 1) / COLS, g.K), COLS * T, ysmem<C>(pl, g.J), s>>>(g, pl, S,
                                                                                                          tw, T);
}
template <typename C, int INV> void ffty_dir(cudaStream_t s, const Geo &g, const RadixPlan &pl, C *S, const C *tw) {
  if (pl.n == 2) {
    if (pl.most > 9) ffty_go<C, 16, INV, ycols<C>(2)>(s, g, pl, S, tw);
    else ffty_go<C, 9, INV, ycols<C>(2)>(s, g, pl, S, tw);
  } else {
    if (pl.most > 9) ffty_go<C, 16, INV, ycols<C>(3)>(s, g, pl, S, tw);
    else ffty_go<C, 9, INV, ycols<C>(3)>(s, g, pl, S, tw);
  }
}
template <typename F> bool big_smem(F *k) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RADIX_SMEM) == cudaSuccess;
}
template <typename C, int INV> bool ffty_limits() {
  return big_smem(k_ffty_radix<C, 16, INV, ycols<C>(2)>) && big_smem(k_ffty_radix<C, 9, INV, ycols<C>(2)>) &&
         big_smem(k_ffty_radix<C, 16, INV, ycols<C>(3)>) && big_smem(k_ffty_radix<C, 9, INV, ycols<C>(3)>);
}
}  // namespace

template <typename T> bool fft_radix_ok(const Geo &g) {
  RadixPlan px, py;
  return radix_fits<typename cpx<T>::t>(g, px, py);
}
template <typename T>
void fft_radix_fillps_x(cudaStream_t s, const Geo &g, const T *fu, const T *fv, T *fw, void *spec, const void *twM,
                        const void *twN, double sx, double sy, double sz) {
  typedef typename cpx<T>::t C;
  const RadixPlan pl = radix_plan(g.I / 2);
  int rows, t;
  size_t smem;
  xshape<C>(pl, g.I / 2, rows, t, smem);
  const int grid = (g.J * g.K + rows - 1) / rows;
  auto go = [&](auto k) {
    k<<<grid, rows * t, smem, s>>>(g, pl, fu, fv, fw, fw, (C *)spec, (const C *)twM, (const C *)twN, (T)sx, (T)sy, (T)sz,
                                   rows, t);
  };
  if (pl.most > 9) go(k_fillps_fftx_radix<T, 16>);
  else go(k_fillps_fftx_radix<T, 9>);
}
template <typename T> void fft_radix_y(cudaStream_t s, const Geo &g, void *spec, const void *twJ, int inv) {
  typedef typename cpx<T>::t C;
  const RadixPlan pl = radix_plan(g.J);
  if (inv) ffty_dir<C, 1>(s, g, pl, (C *)spec, (const C *)twJ);
  else ffty_dir<C, 0>(s, g, pl, (C *)spec, (const C *)twJ);
}
template <typename T>
void fft_radix_ix(cudaStream_t s, const Geo &g, const void *spec, T *phi, const void *twM, const void *twN) {
  typedef typename cpx<T>::t C;
  const RadixPlan pl = radix_plan(g.I / 2);
  int rows, t;
  size_t smem;
  xshape<C>(pl, g.I / 2, rows, t, smem);
  const int grid = (g.J * g.K + rows - 1) / rows;
  auto go = [&](auto k) {
    k<<<grid, rows * t, smem, s>>>(g, pl, (const C *)spec, phi, (const C *)twM, (const C *)twN, rows, t);
  };
  if (pl.most > 9) go(k_ifftx_radix<T, 16>);
  else go(k_ifftx_radix<T, 9>);
}
template <typename T> int fft_radix_set_smem_limits() {
  typedef typename cpx<T>::t C;
  const bool ok = ffty_limits<C, 0>() && ffty_limits<C, 1>() && big_smem(k_fillps_fftx_radix<T, 16>) &&
                  big_smem(k_fillps_fftx_radix<T, 9>) && big_smem(k_ifftx_radix<T, 16>) && big_smem(k_ifftx_radix<T, 9>);
  return ok ? 0 : -1;
}
#define FFT_RADIX_INST(T)                                                                                          \
  template bool fft_radix_ok<T>(const Geo &);                                                                      \
  template void fft_radix_fillps_x<T>(cudaStream_t, const Geo &, const T *, const T *, T *, void *, const void *,  \
                                      const void *, double, double, double);                                       \
  template void fft_radix_y<T>(cudaStream_t, const Geo &, void *, const void *, int);                              \
  template void fft_radix_ix<T>(cudaStream_t, const Geo &, const void *, T *, const void *, const void *);         \
  template int fft_radix_set_smem_limits<T>();
FFT_RADIX_INST(double)

}  // namespace ibmk
