// Hand-written mixed-radix 3D FFT for the P3M mesh (sm_100a).
//
// Real mesh [M0][M1][M2] (z fastest) <-> complex half mesh [M0][M1][hp]
// (kz < M2/2+1 used, hp = padded row length).  Forward = exp(-i k x),
// backward = exp(+i k x), both unnormalised, as the reference's FFTW
// plans (fft/fft.cpp:682-696).  Each pass stages a tile of lines in shared
// memory and transforms them there; twiddles come from an FP64-computed
// table rounded to the working precision.  Only forward transforms are
// coded: a backward one swaps real and imaginary parts on its way into and
// out of shared memory.
//
// Lengths N1 N2 with factors of at most 16 (AxisPlan n1, n2: nearly every
// mesh up to 256) transform in place in two register steps; the others run
// Stockham autosort stages with a second buffer (Govindaraju et al. 2008
// formulation).
//
// The x pass is fused with the P3M k-space work that follows the forward
// transform: optimal influence function, k-space energy and pressure-tensor
// sums, and the backward x transforms.  The differentiation i k_d along y
// and z commutes with the x transform, so the x pass emits two spectra only
// (k_x phi and phi); the y pass forms and transforms k_y phi beside phi, and
// the z pass multiplies by k_z.
#pragma once

#include "common.cuh"
#include "p3m_kernels.cuh"

#include <type_traits>

namespace p3mx {

// Block work item of an FFT pass: replica, first item, item count.
struct Blk {
  int rep;
  int a;   // first line / x / y index
  int b;   // line count, or second index (kz tile start)
  int w;   // columns of the kz tile (y and x passes)
};

// Shared-memory position of element i of a staged line: one pad slot per 16
// elements, so the stride-R accesses of the early Stockham stages (and the
// stride-16 transposed loads) fall into distinct banks.
__host__ __device__ inline int pix(int i) { return i + (i >> 4); }
// Line stride (elements) of staged lines of length n: padded length, odd so
// that consecutive lines start in different banks.
__host__ __device__ inline int line_ld(int n) { return (n + ((n - 1) >> 4)) | 1; }

// Copy the twiddle table exp(-2 pi i k / n), k < n, of one axis to shared
// memory (caller synchronises).
template <typename C>
__device__ inline void load_twiddles(C *dst, const C *__restrict__ twtab, AxisPlan const &pl) {
  const C *src = twtab + pl.tw_off;
  for (int k = threadIdx.x; k < pl.n; k += blockDim.x)
    dst[k] = src[k];
}

// cos and sin of 2 pi k / n at compile time: the angle reduced to [0, pi/4]
// in integers, then the Taylor series.
__host__ __device__ constexpr double series_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 12; ++i) {
    t *= -x * x / ((2 * i - 1) * (2 * i));
    s += t;
  }
  return s;
}
__host__ __device__ constexpr double series_sin(double x) {
  double t = x, s = x;
  for (int i = 1; i < 12; ++i) {
    t *= -x * x / ((2 * i) * (2 * i + 1));
    s += t;
  }
  return s;
}
__host__ __device__ constexpr double root_cos(int k, int n) {
  k = ((k % n) + n) % n;
  if (2 * k > n)
    k = n - k;
  // angle 2 pi k / n in [0, pi]
  if (4 * k > n)
    return -root_cos(n - 2 * k, 2 * n);
  if (8 * k > n)
    return series_sin(2.0 * kPi * (n - 4 * k) / (4.0 * n));
  return series_cos(2.0 * kPi * k / n);
}
__host__ __device__ constexpr double root_sin(int k, int n) { return root_cos(4 * k - n, 4 * n); }

// f(integral_constant<int, I>) for I = 0 .. N-1, unrolled.
template <int I, int N, typename F> __device__ __forceinline__ void static_for(F &&f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}

// v * exp(-2 pi i K / N), K and N compile-time.
template <int K, int N, typename C> __device__ __forceinline__ C mul_root(C v) {
  using Real = decltype(v.x);
  constexpr int k = K % N;
  if constexpr (k == 0) {
    return v;
  } else if constexpr (4 * k == N) {
    return C{v.y, -v.x};
  } else if constexpr (2 * k == N) {
    return C{-v.x, -v.y};
  } else if constexpr (4 * k == 3 * N) {
    return C{-v.y, v.x};
  } else {
    constexpr Real c = static_cast<Real>(root_cos(k, N)), s = static_cast<Real>(root_sin(k, N));
    return C{v.x * c + v.y * s, v.y * c - v.x * s};
  }
}

// In-register forward DFT of length R, natural order in and out: 2 and 4
// directly, odd primes from the sums and differences of mirrored inputs,
// 8 and 16 from halves, other composites R = A B as B transforms of length A,
// twiddles, A of length B.
template <typename C, int R> __device__ __forceinline__ void dft(C *v) {
  using Real = decltype(v[0].x);
  if constexpr (R == 2) {
    C const a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    C const s0 = cadd(v[0], v[2]), s1 = csub(v[0], v[2]);
    C const s2 = cadd(v[1], v[3]), s3 = csub(v[1], v[3]);
    C const s3r = C{s3.y, -s3.x};
    v[0] = cadd(s0, s2);
    v[2] = csub(s0, s2);
    v[1] = cadd(s1, s3r);
    v[3] = csub(s1, s3r);
  } else if constexpr (R % 2 == 1 && R % 3 != 0 || R == 3) {
    constexpr int H = (R - 1) / 2;
    C p[H], m[H];
    static_for<0, H>([&](auto j) {
      constexpr int J = decltype(j)::value;
      p[J] = cadd(v[J + 1], v[R - 1 - J]);
      m[J] = csub(v[J + 1], v[R - 1 - J]);
    });
    C const x0 = v[0];
    C sum = x0;
    static_for<0, H>([&](auto j) { sum = cadd(sum, p[decltype(j)::value]); });
    v[0] = sum;
    static_for<1, H + 1>([&](auto kk) {
      constexpr int K = decltype(kk)::value;
      C a = x0, b = C{Real(0), Real(0)};
      static_for<0, H>([&](auto j) {
        constexpr int J = decltype(j)::value;
        constexpr Real c = static_cast<Real>(root_cos((J + 1) * K, R)),
                       s = static_cast<Real>(root_sin((J + 1) * K, R));
        a.x += c * p[J].x;
        a.y += c * p[J].y;
        b.x += s * m[J].x;
        b.y += s * m[J].y;
      });
      // X_K = a - i b, X_{R-K} = a + i b
      v[K] = C{a.x + b.y, a.y - b.x};
      v[R - K] = C{a.x - b.y, a.y + b.x};
    });
  } else if constexpr (R == 8 || R == 16) {
    // halves of even and odd inputs (the fewest live registers)
    constexpr int H = R / 2;
    C e[H], o[H];
    static_for<0, H>([&](auto i) {
      e[decltype(i)::value] = v[2 * decltype(i)::value];
      o[decltype(i)::value] = v[2 * decltype(i)::value + 1];
    });
    dft<C, H>(e);
    dft<C, H>(o);
    static_for<0, H>([&](auto kk) {
      constexpr int K = decltype(kk)::value;
      C const t = mul_root<K, R>(o[K]);
      v[K] = cadd(e[K], t);
      v[K + H] = csub(e[K], t);
    });
  } else {
    constexpr int A = R % 4 == 0 ? 4 : (R % 2 == 0 ? 2 : 3), B = R / A;
    C y[R]; // y[k1 * B + t]
    static_for<0, B>([&](auto tt) {
      constexpr int T = decltype(tt)::value;
      C w[A];
      static_for<0, A>([&](auto mm) { w[decltype(mm)::value] = v[T + B * decltype(mm)::value]; });
      dft<C, A>(w);
      static_for<0, A>([&](auto kk) {
        constexpr int K = decltype(kk)::value;
        y[K * B + T] = mul_root<T * K, R>(w[K]);
      });
    });
    static_for<0, A>([&](auto kk) {
      constexpr int K = decltype(kk)::value;
      dft<C, B>(y + K * B);
      static_for<0, B>([&](auto jj) { v[K + A * decltype(jj)::value] = y[K * B + decltype(jj)::value]; });
    });
  }
}

// Generic (runtime) radix for primes beyond the templated set.
template <typename C>
__device__ inline void dft_dyn(C *v, int R, const C *__restrict__ tw, int n) {
  C out[32];
  int const step = n / R;
  for (int m = 0; m < R; ++m) {
    C acc = v[0];
    for (int r = 1; r < R; ++r) {
      int const e = (r * m) % R;
      acc = cadd(acc, cmul(v[r], tw[e * step]));
    }
    out[m] = acc;
  }
  for (int m = 0; m < R; ++m)
    v[m] = out[m];
}

// Quotient of small non-negative ints (< 2^24) by a runtime divisor via the
// FP32 reciprocal plus one correction step (replaces the ~20-instruction
// integer division in the FFT index maps).
__device__ inline int qdiv(int a, int b, float rb) {
  int q = __float2int_rz(__int2float_rn(a) * rb);
  int const r = a - q * b;
  q += (r >= b) - (r < 0);
  return q;
}

// One Stockham stage over `nlines` lines of length n held in shared memory
// with line stride ld (ld > n pads the lines against bank conflicts).
// Twiddle index r*jm*tstride < n, so no modulo is needed.
template <typename C, int R>
__device__ inline void fft_stage_t(const C *src, C *dst, int n, int ld, int nlines, int Ns,
                                   const C *__restrict__ tw) {
  int const nb = n / R;
  int const total = nb * nlines;
  int const tstride = n / (Ns * R);
  float const rnb = 1.0f / static_cast<float>(nb);
  float const rNs = 1.0f / static_cast<float>(Ns);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int const line = qdiv(t, nb, rnb);
    int const j = t - line * nb;
    C const *s = src + line * ld;
    C *d = dst + line * ld;
    int const jq = qdiv(j, Ns, rNs);
    int const jm = j - jq * Ns;
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      v[r] = s[pix(j + r * nb)];
      if (r > 0 && jm != 0)
        v[r] = cmul(v[r], tw[r * jm * tstride]);
    }
    dft<C, R>(v);
    int const base = jq * Ns * R + jm;
#pragma unroll
    for (int r = 0; r < R; ++r)
      d[pix(base + r * Ns)] = v[r];
  }
}

template <typename C>
__device__ inline void fft_stage_dyn(const C *src, C *dst, int n, int ld, int nlines, int Ns,
                                     int R, const C *__restrict__ tw) {
  int const nb = n / R;
  int const total = nb * nlines;
  int const tstride = n / (Ns * R);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int const line = t / nb;
    int const j = t - line * nb;
    C const *s = src + line * ld;
    C *d = dst + line * ld;
    int const jm = j % Ns;
    C v[32];
    for (int r = 0; r < R; ++r) {
      v[r] = s[pix(j + r * nb)];
      if (r > 0 && jm != 0)
        v[r] = cmul(v[r], tw[r * jm * tstride]);
    }
    dft_dyn(v, R, tw, n);
    int const base = (j / Ns) * Ns * R + jm;
    for (int r = 0; r < R; ++r)
      d[pix(base + r * Ns)] = v[r];
  }
}

// Two-step transform in place, n = N1 N2 (n = t + N2 m, k = k1 + N1 k2):
//   step 1, item (line, t): Y[t][k1] = w_n^(t k1) * DFT_N1 over m of x[t + N2 m],
//           written in place at t + N2 k1;
//   step 2, item (line, k1): X[k1 + N1 k2] = DFT_N2 over t of Y[t][k1]: the
//           lines of a round are read into registers, the block
//           synchronises, then they are written back in natural order.
// n2 / n1 are the other factor (compile-time constants where the caller
// passes them as such, so the strides fold).
// opaque(): the compiler neither hoists the index arithmetic of all factors out
// of a caller's loop nor keeps a step's 16 read addresses in registers for its
// writes (both spill at the passes' register bounds).
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}
// A block takes at most 256 / n2 lines, n2 the smaller factor: step 1 is one
// item per thread.
template <typename C, int N1>
__device__ __forceinline__ void fft_step1(C *a, int nlines, int ld, int n2,
                                          const C *__restrict__ tw) {
  int const it = opaque(threadIdx.x);
  if (it >= nlines * n2)
    return;
  int const l = qdiv(it, n2, 1.0f / static_cast<float>(n2));
  int t = it - l * n2;
  C *s = a + l * ld;
  C v[N1];
#pragma unroll
  for (int m = 0; m < N1; ++m)
    v[m] = s[pix(t + n2 * m)];
  dft<C, N1>(v);
#pragma unroll
  for (int k1 = 1; k1 < N1; ++k1)
    v[k1] = cmul(v[k1], tw[t * k1]);
  t = opaque(t);
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1)
    s[pix(t + n2 * k1)] = v[k1];
}
template <typename C, int N2, bool ONE>
__device__ __forceinline__ void fft_step2(C *a, int nlines, int ld, int n1) {
  int const per = blockDim.x / n1; // lines per round
  int const tid = opaque(threadIdx.x);
  int const lq = qdiv(tid, n1, 1.0f / static_cast<float>(n1)), k1 = tid - lq * n1;
#pragma unroll 1
  for (int l0 = 0; l0 < nlines; l0 += per) {
    bool const act = lq < per && l0 + lq < nlines;
    C *s = a + (l0 + lq) * ld;
    C v[N2];
    if (act) {
#pragma unroll
      for (int t = 0; t < N2; ++t)
        v[t] = s[pix(N2 * k1 + t)];
      dft<C, N2>(v);
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2)
        s[pix(k1 + n1 * k2)] = v[k2];
    }
    if (ONE)
      break;
  }
}
// The two steps for compile-time factors (powers of two): the padded indices
// fold to a base and immediate offsets.  Blocks of 256 threads, one item per
// thread in the first step; a loop around either step made the compiler keep
// addresses live across it (64-84 bytes of spills at 64 registers, now none).
template <typename C, int N1, int N2, bool ONE>
__device__ __forceinline__ void fft_pow2(C *a, int nlines, int ld, const C *__restrict__ tw) {
  unsigned const tid = threadIdx.x;
  if (tid < static_cast<unsigned>(nlines * N2)) {
    int const l = tid / N2, t = tid % N2;
    C *s = a + l * ld + t;
    C v[N1];
#pragma unroll
    for (int m = 0; m < N1; ++m)
      v[m] = s[pix(N2 * m)]; // t < 16 never crosses a pad
    dft<C, N1>(v);
#pragma unroll
    for (int k1 = 1; k1 < N1; ++k1)
      v[k1] = cmul(v[k1], tw[t * k1]);
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1)
      s[pix(N2 * k1)] = v[k1];
  }
  __syncthreads();
  constexpr int per = 256 / N1;
  int const lq = tid / N1, k1 = tid % N1;
#pragma unroll 1
  for (int l0 = 0; l0 < nlines; l0 += per) {
    bool const act = l0 + lq < nlines;
    C *s = a + (l0 + lq) * ld;
    C v[N2];
    if (act) {
      C const *r = s + pix(N2 * k1);
#pragma unroll
      for (int t = 0; t < N2; ++t)
        v[t] = r[t];
      dft<C, N2>(v);
    }
    __syncthreads();
    if (act) {
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2)
        s[k1 + pix(N1 * k2)] = v[k2];
    }
    if (ONE)
      break;
  }
}
#define P3MX_FACTOR_DISPATCH(N, CALL)                                          \
  switch (N) {                                                                 \
  case 2: { constexpr int R = 2; CALL; } break;                                \
  case 3: { constexpr int R = 3; CALL; } break;                                \
  case 4: { constexpr int R = 4; CALL; } break;                                \
  case 5: { constexpr int R = 5; CALL; } break;                                \
  case 6: { constexpr int R = 6; CALL; } break;                                \
  case 7: { constexpr int R = 7; CALL; } break;                                \
  case 8: { constexpr int R = 8; CALL; } break;                                \
  case 9: { constexpr int R = 9; CALL; } break;                                \
  case 10: { constexpr int R = 10; CALL; } break;                              \
  case 12: { constexpr int R = 12; CALL; } break;                              \
  case 14: { constexpr int R = 14; CALL; } break;                              \
  case 15: { constexpr int R = 15; CALL; } break;                              \
  default: { constexpr int R = 16; CALL; } break;                              \
  }
// Forward transform of nlines lines in `a` (element i of line l at
// l*ld + pix(i)); tw = the axis twiddle table (shared memory).  KIND, for all
// lines of a launch: kFftPow2 -- powers of two 32 to 256, in place,
// compile-time factors (without the other factors' code a pass needs no
// spills at four blocks per SM); kFftTwo -- two-factor plans, in place;
// kFftAny -- Stockham stages with `b`, a second buffer of the same size.
// ONE: at most 16 lines, so that a thread has one item per step (no loops, and
// nothing hoisted out of them).  Returns the buffer holding the result.  All threads of the block call it
// behind a barrier; the result is visible when it returns.
constexpr int kFftAny = 0, kFftTwo = 1, kFftPow2 = 2;
template <int KIND, bool ONE, typename C>
__device__ __forceinline__ C *fft_lines(C *a, C *b, int nlines, int ld, AxisPlan const &pl,
                                        const C *__restrict__ tw) {
  if constexpr (KIND == kFftPow2) {
    switch (pl.n) {
    case 32: fft_pow2<C, 8, 4, ONE>(a, nlines, ld, tw); break;
    case 64: fft_pow2<C, 8, 8, ONE>(a, nlines, ld, tw); break;
    case 128: fft_pow2<C, 16, 8, ONE>(a, nlines, ld, tw); break;
    default: fft_pow2<C, 16, 16, ONE>(a, nlines, ld, tw); break;
    }
    __syncthreads();
    return a;
  } else if constexpr (KIND == kFftTwo) {
    P3MX_FACTOR_DISPATCH(pl.n1, (fft_step1<C, R>(a, nlines, ld, pl.n2, tw)))
    __syncthreads();
    P3MX_FACTOR_DISPATCH(pl.n2, (fft_step2<C, R, ONE>(a, nlines, ld, pl.n1)))
    __syncthreads();
    return a;
  } else {
    int const n = pl.n;
    int Ns = 1;
    C *src = a, *dst = b;
    for (int s = 0; s < pl.nstages; ++s) {
      int const R = pl.radix[s];
      switch (R) {
      case 2: fft_stage_t<C, 2>(src, dst, n, ld, nlines, Ns, tw); break;
      case 3: fft_stage_t<C, 3>(src, dst, n, ld, nlines, Ns, tw); break;
      case 4: fft_stage_t<C, 4>(src, dst, n, ld, nlines, Ns, tw); break;
      case 8: fft_stage_t<C, 8>(src, dst, n, ld, nlines, Ns, tw); break;
      case 16: fft_stage_t<C, 16>(src, dst, n, ld, nlines, Ns, tw); break;
      case 5: fft_stage_t<C, 5>(src, dst, n, ld, nlines, Ns, tw); break;
      case 7: fft_stage_t<C, 7>(src, dst, n, ld, nlines, Ns, tw); break;
      default: fft_stage_dyn<C>(src, dst, n, ld, nlines, Ns, R, tw); break;
      }
      __syncthreads();
      Ns *= R;
      C *t = src;
      src = dst;
      dst = t;
    }
    return src;
  }
}

// f(integral_constant<int, kind>) for a runtime kind.
template <typename Fn> inline void fft_pick(int kind, Fn &&f) {
  if (kind == kFftPow2)
    f(std::integral_constant<int, kFftPow2>{});
  else if (kind == kFftTwo)
    f(std::integral_constant<int, kFftTwo>{});
  else
    f(std::integral_constant<int, kFftAny>{});
}

// Blocks per SM of the z and y passes (their registers are sized for it).  Four
// also for two-factor lines, with some spills: three without measured 888 ->
// 916 us (131 072 dipoles), 335 -> 345 us (98 304 ions on 112 x 112 x 144).
template <typename Real> constexpr int kFftBlocks = sizeof(Real) == 4 ? 4 : 2;

// Signed frequency of index i in an axis of m points, the Nyquist index as
// zero (calc_meshift with the differential operator's convention,
// p3m/common.hpp:248-264).
__device__ inline int freq_dop(int i, int m) { return (i == m / 2) ? 0 : (i < m / 2 ? i : i - m); }
template <typename C> __device__ inline C cswap(C v) { return C{v.y, v.x}; }

// ---- pass z, forward: real lines -> complex half lines -----------------
// Two real lines per complex transform: Z = x0 + i x1, then
// X0[k] = (Z[k] + conj Z[n-k]) / 2 and X1[k] = -i (Z[k] - conj Z[n-k]) / 2.
// bk.b real lines per block (an odd last line is paired with zeros).
// The charge mesh exists only as the assignment's tiles: the block sums, for
// every (x, y) line, the 1 to 4 (in wrap corners 9) tile rows that cover it,
// contiguous along z: first the points of each super-brick, four per load,
// then its halo, added to the points of the next one.  Bound by instructions
// (integer ones run at half rate), so the rows of a line are listed once in
// shared memory, and lines, groups and half rows are flat index ranges (a warp
// per line left lanes idle on short lines: 48 small meshes 45 -> 109 us).  At
// 256^3 84 us; from a mesh 54 us, but the mesh cost the assignment its flushes.
// blockIdx.y: charge set (tiles and spectra tile_stride / c_stride apart).
// Shared memory: bk.b/2 staged lines of line_ld(n) (twice that for KIND 0),
// twiddles (n).  Meshes are even, so is bk.b.
constexpr int kZfLines = 64; // most real lines per block
template <typename Real, int KIND>
__global__ void __launch_bounds__(256, kFftBlocks<Real>)
k_fft_z_fwd(const RepGeom *__restrict__ reps, const Blk *__restrict__ blks,
            const Real *__restrict__ tiles, long long tile_stride, const int *__restrict__ cov,
            int E, typename CplxOf<Real>::type *__restrict__ cmesh, long long c_stride,
            const typename CplxOf<Real>::type *__restrict__ twtab) {
  using C = typename CplxOf<Real>::type;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ long long s_row[kZfLines][9];
  __shared__ int s_nrow[kZfLines];
  Blk const bk = blks[blockIdx.x];
  RepGeom const &G = reps[bk.rep];
  int const n = G.mesh[2];
  int const ld = line_ld(n);
  int const nl = bk.b;          // real lines in this block
  int const np = (nl + 1) >> 1; // complex lines
  C *a = reinterpret_cast<C *>(smem_raw);
  C *b = KIND ? nullptr : a + np * ld;
  C *tw = a + (KIND ? 1 : 2) * np * ld;
  tiles += blockIdx.y * tile_stride + G.tl_off;
  cmesh += blockIdx.y * c_stride;
  load_twiddles(tw, twtab, G.plan[2]);
  long long const line0 = bk.a;
  TileMap const tm(G, E);
  if (static_cast<int>(threadIdx.x) < nl) {
    int const M0 = G.mesh[0], M1 = G.mesh[1];
    int const x = static_cast<int>((line0 + threadIdx.x) / M1),
              y = static_cast<int>((line0 + threadIdx.x) % M1);
    int c = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) {
        long long const bx = tm.x(cov[G.cov_off[0] + i * M0 + x]);
        int const by = tm.y(cov[G.cov_off[1] + j * M1 + y]);
        if (bx >= 0 && by >= 0)
          s_row[threadIdx.x][c++] = bx + by;
      }
    s_nrow[threadIdx.x] = c;
  }
  __syncthreads();
  // real line l, element k -> real or imaginary part of slot l/2
  Real *ar = reinterpret_cast<Real *>(a);
  using R4 = typename Real4Of<Real>::type;
  auto row_sum = [&](int l, int z) {
    int const c = s_nrow[l];
    const long long *r = s_row[l];
    const Real *t = tiles + z;
    R4 s = *reinterpret_cast<const R4 *>(t + r[0]);
    if (c == 2) {
      s = tile_add(s, *reinterpret_cast<const R4 *>(t + r[1]));
    } else if (c > 2) {
      // three rows (wrap corners) or four and more
      R4 const u = *reinterpret_cast<const R4 *>(t + r[1]),
               v = *reinterpret_cast<const R4 *>(t + r[2]);
      s = tile_add(s, u);
      if (c == 3) {
        s = tile_add(s, v);
      } else {
        s = tile_add(s, tile_add(v, *reinterpret_cast<const R4 *>(t + r[3])));
        for (int k = 4; k < c; ++k)
          s = tile_add(s, *reinterpret_cast<const R4 *>(t + r[k]));
      }
    }
    return s;
  };
  int const g4 = (n + 3) >> 2;
  int const le = 31 - __clz(E), tz = tm.tz;
  float const rg4 = 1.0f / static_cast<float>(g4);
#pragma unroll 2
  for (int t = threadIdx.x; t < nl * g4; t += 256) {
    // E is a multiple of 4: the four points lie in one super-brick (rows are
    // padded, so the last group may reach past the mesh)
    int const l = qdiv(t, g4, rg4), k = 4 * (t - l * g4);
    R4 const v = row_sum(l, (k >> le) * tz + (k & (E - 1)));
    Real *p = ar + 2 * ((l >> 1) * ld + pix(k)) + (l & 1);
    p[0] = v.x;
    p[2] = v.y;
    if (k + 2 < n) {
      p[4] = v.z;
      p[6] = v.w;
    }
  }
  // halos: group h of super-brick b's, points (b E + len_b + 4 h ...) mod n.
  // The last super-brick's length need not be a multiple of 4: its row
  // segment is then read point by point
  int const halo = G.cao - 1, nb = G.sbn[2], hg = (halo + 3) >> 2;
  int const last = n - (nb - 1) * E; // length of the last super-brick
  int const per = nb * hg;           // halo groups of a line
  float const rper = 1.0f / static_cast<float>(max(per, 1));
  float const rhg = 1.0f / static_cast<float>(max(hg, 1));
  // the halo of the one before the last may reach around the axis to the same
  // points as the last one's: added after it
  bool const around = nb > 1 && last < halo;
  for (int pass = 0; pass < (around ? 2 : 1); ++pass) {
    __syncthreads();
    for (int t = threadIdx.x; t < nl * per; t += 256) {
      int const l = qdiv(t, per, rper), u = t - l * per;
      int const bz = qdiv(u, hg, rhg), h = 4 * (u - bz * hg);
      if (around && (bz == nb - 2) != (pass == 1))
        continue;
      int const len = bz == nb - 1 ? last : E;
      Real v[4];
      if ((len & 3) == 0) {
        R4 const q = row_sum(l, bz * tz + len + h);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
      } else {
        for (int e = 0; e < 4; ++e) {
          v[e] = Real(0);
          if (h + e < halo)
            for (int c = 0; c < s_nrow[l]; ++c)
              v[e] += tiles[s_row[l][c] + bz * tz + len + h + e];
        }
      }
      Real *o = ar + 2 * ((l >> 1) * ld) + (l & 1);
      int const z = bz * E + len + h;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int const zz = z + e >= n ? (z + e) % n : z + e;
        if (h + e < halo)
          o[2 * pix(zz)] += v[e];
      }
    }
  }
  __syncthreads();
  C *res = fft_lines<KIND, false>(a, b, np, ld, G.plan[2], tw);
  int const H = n / 2 + 1;
  int const hp = G.hp;
  // both lines of a slot from one pair of entries
  C *const out = cmesh + G.km_off + line0 * hp;
  float const rhp = 1.0f / static_cast<float>(hp);
#pragma unroll 2
  for (int t = threadIdx.x; t < np * hp; t += 256) {
    int const p = qdiv(t, hp, rhp), k = t - p * hp;
    C v0{Real(0), Real(0)}, v1 = v0;
    if (k < H) {
      C const z = res[p * ld + pix(k)];
      C const zc = res[p * ld + pix(k == 0 ? 0 : n - k)];
      v0 = C{Real(0.5) * (z.x + zc.x), Real(0.5) * (z.y - zc.y)};
      v1 = C{Real(0.5) * (z.y + zc.y), Real(0.5) * (zc.x - z.x)};
    }
    C *q = out + 2 * p * hp + k;
    q[0] = v0;
    q[hp] = v1;
  }
}

// ---- pass y ---------------------------------------------------------------
// Bound by the latency of its row loads, then by instructions; at 256^3 36 us
// forward and 100 us for the three backward spectra (two of them inputs).
// Jobs of a y pass: job k transforms array src[k], times k_y^pw[k], into array
// dst[k].  Array src[k] is read by other jobs unless dst[k] = src[k].  The
// jobs of one tile are neighbouring blocks, so a shared source is read from
// HBM once.
struct YPass {
  int n;
  signed char src[9], dst[9], pw[9];
};
// nf arrays in place
inline YPass y_plain(int nf) {
  YPass p{};
  p.n = nf;
  for (int k = 0; k < nf; ++k)
    p.src[k] = p.dst[k] = static_cast<signed char>(k);
  return p;
}
// backward y pass of the charge fields: k_x phi (array 0, in place), k_y phi
// and phi (arrays 2 and 3) from phi (array 1)
inline YPass y_charge() { return YPass{3, {1, 1, 0}, {2, 3, 0}, {1, 0, 0}}; }
constexpr int kChargeSpectra = 4; // arrays of the charge fields' spectra
// KIND: every replica's y lines transform in place (the host checks).  kscale:
// k_y in units of 2 pi / box (1) or as an integer (0).  Shared memory: tile
// staged lines of line_ld(M1) (two sets for KIND 0), twiddles (M1).
template <typename Real, bool INV, int KIND>
__global__ void __launch_bounds__(256, kFftBlocks<Real>)
k_fft_y(const RepGeom *__restrict__ reps, const Blk *__restrict__ blks,
        typename CplxOf<Real>::type *__restrict__ c0, long long field_stride, const __grid_constant__ YPass job,
        int kscale, int tile, const typename CplxOf<Real>::type *__restrict__ twtab) {
  using C = typename CplxOf<Real>::type;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int const blk = blockIdx.x / job.n, jb = blockIdx.x - blk * job.n;
  Blk const bk = blks[blk];
  RepGeom const &G = reps[bk.rep];
  int const M1 = G.mesh[1];
  int const x = bk.a, kz0 = bk.b;
  int const T = bk.w;
  int const ld = line_ld(M1);
  C *a = reinterpret_cast<C *>(smem_raw);
  C *b = KIND ? nullptr : a + tile * ld;
  C *tw = a + (KIND ? 1 : 2) * tile * ld;
  load_twiddles(tw, twtab, G.plan[1]);
  long long const hp = G.hp;
  // 16 x 16 thread mapping (tile <= 16 columns): column tq, rows yq + 16 i
  int const tq = threadIdx.x & 15, yq = threadIdx.x >> 4;
  bool const col = tq < T;
  long long const base = G.km_off + static_cast<long long>(x) * M1 * hp + kz0;
  const C *src = c0 + field_stride * job.src[jb] + base + min(tq, T - 1);
  C *dst = c0 + field_stride * job.dst[jb] + base + tq;
  int const pw = INV ? job.pw[jb] : 0;
  Real const ks = kscale ? static_cast<Real>(2.0 * kPi * G.box_i[1]) : Real(1);
  // all of a thread's rows in flight at once (up to 16: M1 <= 256 in one
  // round), rows and columns past the tile read a valid one in their place, so
  // that the loads are unconditional (guarded they were not all in flight
  // together: with the spills, the two y passes of 256^3 took 64 + 125 us
  // against 36 + 100); row y = yq + 16 u of column tq lies at tq ld + yq + 17 u
  C *const sl = a + tq * ld + yq;
  int const rows = col ? (M1 - yq + 15) >> 4 : 0;
  long long const step = 16 * hp;
  for (int u0 = 0; u0 < rows; u0 += 16) {
    C v[16];
    int const last = M1 - 1 - 16 * u0;
    const C *p = src + 16 * u0 * hp;
#pragma unroll
    for (int u = 0; u < 16; ++u)
      v[u] = p[min(yq + 16 * u, last) * hp];
#pragma unroll
    for (int u = 0; u < 16; ++u)
      if (u0 + u < rows) {
        C w = INV ? cswap(v[u]) : v[u];
        if (INV && pw > 0) {
          Real const k = static_cast<Real>(freq_dop(yq + 16 * (u0 + u), M1)) * ks;
          Real const f = pw == 2 ? k * k : k;
          w = C{f * w.x, f * w.y};
        }
        sl[17 * (u0 + u)] = w;
      }
  }
  __syncthreads();
  const C *res = fft_lines<KIND, true>(a, b, T, ld, G.plan[1], tw) + tq * ld + yq;
  C *q = dst + yq * hp;
#pragma unroll 4
  for (int u = 0; u < rows; ++u, q += step) {
    C const v = res[17 * u];
    *q = INV ? cswap(v) : v;
  }
}

// ---- pass x fused with the k-space operator -----------------------------
// Per block: one ky, a tile of kz; partials[blk*8 + {E, Pxx, Pxy, Pxz, Pyy,
// Pyz, Pzz, diag}] in FP64 (Hermitian weights 1 for kz = 0, M2/2, else 2).
// Emits two backward-x-transformed spectra: array 0 i k_x phi, array 1 i phi
// (the y and z passes apply k_y and k_z).
// Shared memory: 2 x tile staged lines of line_ld(M0) (phi, k_x phi; 3 x
// for KIND 0: a scratch buffer), twiddles (M0).
// EV: energy / virial partials (a template parameter, so that the
// forces-only instance carries none of their registers).  Bound by instructions:
// 101 us at 256^3 (three backward transforms per mode: 181 us).
template <typename Real, bool EV, int KIND>
__global__ void __launch_bounds__(256, sizeof(Real) == 4 && !EV && KIND ? 3 : 2)
k_fft_x_kspace(const RepGeom *__restrict__ reps, const Blk *__restrict__ blks,
               const typename CplxOf<Real>::type *__restrict__ rho_hat,
               const Real *__restrict__ ginf, typename CplxOf<Real>::type *__restrict__ field0,
               long long field_stride, int tile, int want_fields,
               double *__restrict__ partials,
               const typename CplxOf<Real>::type *__restrict__ twtab) {
  using C = typename CplxOf<Real>::type;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Blk const bk = blks[blockIdx.x];
  RepGeom const &G = reps[bk.rep];
  int const M0 = G.mesh[0], M1 = G.mesh[1], M2 = G.mesh[2];
  int const y = bk.a, kz0 = bk.b;
  int const T = bk.w;
  int const ld = line_ld(M0);
  int const L = tile * ld;
  C *a = reinterpret_cast<C *>(smem_raw);
  C *b = a + L;
  C *c = KIND ? nullptr : b + L;
  C *tw = a + (KIND ? 2 : 3) * L;
  load_twiddles(tw, twtab, G.plan[0]);
  long long const stride_x = static_cast<long long>(M1) * G.hp;
  long long const base = G.km_off + static_cast<long long>(y) * G.hp + kz0;
  // 16 x 16 thread mapping (tile <= 16 columns): column tq, rows xq + 16 i
  int const tq = threadIdx.x & 15, xq = threadIdx.x >> 4;
  bool const col = tq < T;
  for (int x0 = xq; x0 < M0; x0 += 64) {
    C v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      int const x = x0 + 16 * u;
      if (col && x < M0)
        v[u] = rho_hat[base + x * stride_x + tq];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      int const x = x0 + 16 * u;
      if (col && x < M0)
        a[tq * ld + pix(x)] = v[u];
    }
  }
  __syncthreads();
  C *res = fft_lines<KIND, true>(a, b, T, ld, G.plan[0], tw);
  C *fb = (res == a) ? b : a; // k_x phi goes to the free buffer
  // k-space operator
  double const wv[3] = {2.0 * kPi * G.box_i[0], 2.0 * kPi * G.box_i[1],
                        2.0 * kPi * G.box_i[2]};
  double const hai2 = (1.0 / 2.0 / G.alpha) * (1.0 / 2.0 / G.alpha);
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int const kyd = freq_dop(y, M1);
  for (int x = xq; col && x < M0; x += 16) {
    // t fastest across lanes: the influence-function reads are T-contiguous
    int const t = tq;
    int const kz = kz0 + t;
    C const rh = res[t * ld + pix(x)];
    Real const g = ginf[base + x * stride_x + t];
    int const kxd = freq_dop(x, M0), kzd = freq_dop(kz, M2);
    if constexpr (EV) {
      double const wgt = (kz == 0 || kz == M2 / 2) ? 1.0 : 2.0;
      double const ek = wgt * static_cast<double>(g) *
                        (static_cast<double>(rh.x) * rh.x + static_cast<double>(rh.y) * rh.y);
      acc[0] += ek;
      double const kx = kxd * wv[0], ky = kyd * wv[1], kzv = kzd * wv[2];
      double const nsq = kx * kx + ky * ky + kzv * kzv;
      if (nsq != 0.0) {
        double const pr = ek * (-2.0 * (1.0 / nsq + hai2));
        acc[1] += pr * kx * kx;
        acc[2] += pr * kx * ky;
        acc[3] += pr * kx * kzv;
        acc[4] += pr * ky * ky;
        acc[5] += pr * ky * kzv;
        acc[6] += pr * kzv * kzv;
        acc[7] += ek;
      }
    }
    // i phi and i k_x phi, real and imaginary parts swapped for the backward
    // transforms (phi = G rho_hat replaced in place: same thread, same point)
    Real const k = static_cast<Real>(kxd) * static_cast<Real>(wv[0]);
    C const p = C{g * rh.x, -(g * rh.y)};
    res[t * ld + pix(x)] = p;
    fb[t * ld + pix(x)] = C{k * p.x, k * p.y};
  }
  if constexpr (EV) {
    // block reduction of the 8 partial sums (fixed order -> deterministic)
    __shared__ double red[8][32];
    int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double v = acc[k];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, o);
      if (lane == 0)
        red[k][wid] = v;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
      double s = 0.0;
      int const nw = (blockDim.x + 31) >> 5;
      for (int w = 0; w < nw; ++w)
        s += red[threadIdx.x][w];
      partials[static_cast<long long>(blockIdx.x) * 8 + threadIdx.x] = s;
    }
  }
  if (!want_fields)
    return;
  __syncthreads();
  // with KIND 0 the scratch of the second transform is the first's buffer
  // once that is stored
  const C *f0 = fft_lines<KIND, true>(fb, c, T, ld, G.plan[0], tw) + tq * ld + xq;
  int const rows = col ? (M0 - xq + 15) >> 4 : 0;
  C *q = field0 + base + xq * stride_x + tq;
#pragma unroll 4
  for (int u = 0; u < rows; ++u)
    q[u * 16 * stride_x] = cswap(f0[17 * u]);
  if constexpr (!KIND)
    __syncthreads();
  const C *f1 = fft_lines<KIND, true>(res, fb, T, ld, G.plan[0], tw) + tq * ld + xq;
  q += field_stride;
#pragma unroll 4
  for (int u = 0; u < rows; ++u)
    q[u * 16 * stride_x] = cswap(f1[17 * u]);
}

// ---- pass z, backward for 3 field components -> real fields -------------
// Field component d of set blockIdx.y is array arr[3 set + d] times
// k_z^pw[3 set + d].
struct ZPass {
  signed char arr[9], pw[9];
};
inline ZPass z_charge() { return ZPass{{0, 2, 3}, {0, 0, 1}}; }
// Two real outputs per complex transform: slot l < nl carries Ex + i Ey of
// line l, slot nl + j carries Ez of lines 2j and 2j+1.  Each half row is
// extended by Hermitian symmetry with the imaginary parts of the k = 0 and
// k = n/2 entries dropped (c2r semantics), so both packed outputs are real:
// a thread reads entry k of the slot's two half rows and writes entries k and
// n - k (real and imaginary parts swapped: a backward transform).
// Set blockIdx.y writes the field mesh e_stride records further on.
// Shared memory: nl + ceil(nl/2) staged lines of line_ld(n) (twice for
// KIND 0), twiddles (n).  FP32: four blocks per SM -- the block's load, transform
// and store phases do not overlap, so the fourth resident block pays for the
// 64-register bound.  The half rows are read straight into the slots: staging
// them first cost a pass over shared memory and half the lines per block (128^3
// 32 -> 26 us; at 256^3, where the spectra come from HBM, 156 -> 162 us).
constexpr int kZiLines = 128; // most lines per block
template <typename Real, int KIND>
__global__ void __launch_bounds__(256, kFftBlocks<Real>)
k_fft_z_inv3(const RepGeom *__restrict__ reps, const Blk *__restrict__ blks,
             const typename CplxOf<Real>::type *__restrict__ field0, long long field_stride,
             const __grid_constant__ ZPass zp, int kscale, Real *__restrict__ efield, long long e_stride,
             const typename CplxOf<Real>::type *__restrict__ twtab) {
  using C = typename CplxOf<Real>::type;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Blk const bk = blks[blockIdx.x];
  RepGeom const &G = reps[bk.rep];
  int const n = G.mesh[2];
  int const H = n / 2 + 1;
  int const ld = line_ld(n);
  int const nl = bk.b;
  int const nz = (nl + 1) >> 1;
  int const nc = nl + nz;
  long long const line0 = bk.a;
  C *a = reinterpret_cast<C *>(smem_raw);
  C *b = KIND ? nullptr : a + nc * ld;
  C *tw = a + (KIND ? 1 : 2) * nc * ld;
  load_twiddles(tw, twtab, G.plan[2]);
  const C *fsrc = field0 + G.km_off + line0 * G.hp;
  int const set = 3 * blockIdx.y;
  const C *fx = fsrc + field_stride * zp.arr[set], *fy = fsrc + field_stride * zp.arr[set + 1],
          *fz = fsrc + field_stride * zp.arr[set + 2];
  Real const ks = kscale ? static_cast<Real>(2.0 * kPi * G.box_i[2]) : Real(1);
  int const px = zp.pw[set], py = zp.pw[set + 1], pz = zp.pw[set + 2];
  float const rH = 1.0f / static_cast<float>(H);
  long long const hp = G.hp;
  // entry k of the half rows X and Y (times k_z^p0, k_z^p1) into slot j
  auto put = [&](int j, int k, C X, C Y, int p0, int p1) {
    if (p0 | p1) {
      Real const kz = static_cast<Real>(freq_dop(k, n)) * ks;
      Real const f0 = p0 == 0 ? Real(1) : (p0 == 2 ? kz * kz : kz);
      Real const f1 = p1 == 0 ? Real(1) : (p1 == 2 ? kz * kz : kz);
      X = C{f0 * X.x, f0 * X.y};
      Y = C{f1 * Y.x, f1 * Y.y};
    }
    C *s = a + j * ld;
    if (k == 0 || 2 * k == n) {
      // swapped (X.x + i Y.x)
      s[pix(k)] = C{Y.x, X.x};
    } else {
      // X + i Y at k, conj(X) + i conj(Y) at n - k, swapped
      s[pix(k)] = C{X.y + Y.x, X.x - Y.y};
      s[pix(n - k)] = C{Y.x - X.y, X.x + Y.y};
    }
  };
#pragma unroll 4
  for (int t = threadIdx.x; t < nl * H; t += 256) {
    int const j = qdiv(t, H, rH), k = t - j * H;
    put(j, k, fx[j * hp + k], fy[j * hp + k], px, py);
  }
#pragma unroll 2
  for (int t = threadIdx.x; t < nz * H; t += 256) {
    int const j = qdiv(t, H, rH), k = t - j * H;
    const C *r = fz + 2 * j * hp + k;
    put(nl + j, k, r[0], (2 * j + 1 < nl) ? r[hp] : C{Real(0), Real(0)}, pz, pz);
  }
  __syncthreads();
  const C *res = fft_lines<KIND, false>(a, b, nc, ld, G.plan[2], tw);
  // packed field mesh: one (Ex, Ey, Ez, 0) record per mesh point, so the
  // interpolation gathers one 16-byte (FP32) record per stencil point
  // (ghost-padded: every record also goes to its periodic images in the
  // high-side ghost layers of extent epad)
  using R4 = typename Real4Of<Real>::type;
  R4 *out = reinterpret_cast<R4 *>(efield) + blockIdx.y * e_stride + G.re_off;
  int const M1 = G.mesh[1], M0 = G.mesh[0];
  int const P0 = G.epad[0], P1 = G.epad[1], P2 = G.epad[2];
  // per line: its row of the field mesh, and whether it has ghost images along
  // x or y
  __shared__ long long s_row[kZiLines];
  for (int l = threadIdx.x; l < nl; l += 256) {
    int const x = static_cast<int>((line0 + l) / M1), y = static_cast<int>((line0 + l) % M1);
    long long const row = (static_cast<long long>(x) * P1 + y) * P2;
    s_row[l] = (x + M0 < P0 || y + M1 < P1) ? ~row : row;
  }
  __syncthreads();
  float const rn = 1.0f / static_cast<float>(n);
#pragma unroll 2
  for (int t = threadIdx.x; t < nl * n; t += 256) {
    int const l = KIND == kFftPow2 ? t >> (__ffs(n) - 1) : qdiv(t, n, rn), k = t - l * n;
    C const xy = res[l * ld + pix(k)];
    C const zz = res[(nl + (l >> 1)) * ld + pix(k)];
    R4 v;
    v.x = xy.y; // swapped back
    v.y = xy.x;
    v.z = (l & 1) ? zz.x : zz.y;
    v.w = Real(0);
    long long const row = s_row[l];
    if (row >= 0) {
      out[row + k] = v;
      for (int zg = k + n; zg < P2; zg += n)
        out[row + zg] = v;
      continue;
    }
    int const x = static_cast<int>((line0 + l) / M1), y = static_cast<int>((line0 + l) % M1);
    for (int xg = x; xg < P0; xg += M0)
      for (int yg = y; yg < P1; yg += M1) {
        R4 *r = out + (static_cast<long long>(xg) * P1 + yg) * P2;
        for (int zg = k; zg < P2; zg += n)
          r[zg] = v;
      }
  }
}

} // namespace p3mx
