// fft_core.cuh -- FP32 complex FFTs of one line by a group of threads, with
// the line in registers and one shared-memory buffer between the stages.
//
// A length L = R1 R2 R3 (R3 = 1: two stages) is transformed by decimation in
// frequency: thread t holds R1 elements i1 N1 + t (N1 = L / R1), makes their
// R1-point DFT, and the sub-transforms follow over shared memory.  The
// frequencies come out in the order the last stage leaves them: slot
// s = j (L / RL) + t of thread t's output j (RL: the last radix), frequency
// fft_perm(s).  Nothing reorders them: a pointwise factor is stored in slot
// order, and the inverse starts from the same registers.  Every stage
// reads its operands from the places that the same thread writes back to, so
// one buffer and one barrier per exchange are enough.
//
// HALF: the upper half of the input (or of the wanted output) is zero (not
// wanted), as for an image padded to twice its width; the first (last)
// radix-R1 stage is then two R1/2-point DFTs over the lower half.
//
// The short DFTs are the textbook ones: 2, 3, 4 and 5 points written out,
// products of coprime radices by the Good-Thomas index map, others by one
// Cooley-Tukey step.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace pgb {
namespace fft {

// ---- constants at compile time --------------------------------------------
constexpr double kPi = 3.14159265358979323846;
constexpr double c_sin(double x) {  // Taylor series, |x| <= pi
  double t = x, s = x;
  for (int k = 1; k < 24; ++k) {
    t *= -x * x / ((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
constexpr double c_cos(double x) {
  double t = 1, s = 1;
  for (int k = 1; k < 24; ++k) {
    t *= -x * x / ((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
constexpr double c_ang(int num, int den) {  // 2 pi num / den, in (-pi, pi]
  num %= den;
  if (2 * num > den) num -= den;
  return 2 * kPi * num / den;
}
constexpr int c_gcd(int a, int b) { return b == 0 ? a : c_gcd(b, a % b); }
constexpr int c_inv(int a, int m) {  // a^-1 mod m
  for (int x = 0; x < m; ++x)
    if ((a * x) % m == 1 % m) return x;
  return 0;
}

// times S i (S = -1: forward)
template <int S>
__device__ __forceinline__ float2 rot90(float2 a) {
  return S < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}
// times exp(S 2 pi i NUM / DEN)
template <int S, int NUM, int DEN>
__device__ __forceinline__ float2 ctw(float2 a) {
  constexpr int n = NUM % DEN;
  if constexpr (n == 0) return a;
  if constexpr (4 * n == DEN) return rot90<S>(a);
  if constexpr (2 * n == DEN) return make_float2(-a.x, -a.y);
  if constexpr (4 * n == 3 * DEN) return rot90<-S>(a);
  constexpr float c = static_cast<float>(c_cos(c_ang(n, DEN)));
  constexpr float s = static_cast<float>(S * c_sin(c_ang(n, DEN)));
  return make_float2(fmaf(-a.y, s, a.x * c), fmaf(a.y, c, a.x * s));
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * w (S = -1) or a * conj(w) (S = +1)
template <int S>
__device__ __forceinline__ float2 twmul(float2 a, float2 w) {
  return S < 0 ? make_float2(fmaf(-a.y, w.y, a.x * w.x), fmaf(a.y, w.x, a.x * w.y))
               : make_float2(fmaf(a.y, w.y, a.x * w.x), fmaf(a.y, w.x, -a.x * w.y));
}

template <int I, int N, class F>
__device__ __forceinline__ void unroll(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    unroll<I + 1, N>(f);
  }
}

// first factor of a composite radix
constexpr int c_fac(int R) {
  return R == 6 ? 2 : R == 8 ? 2 : R == 9 ? 3 : R == 10 ? 2 : R == 12 ? 4 : R == 15 ? 3 : R == 16 ? 4 : R == 20 ? 4 : R == 18 ? 2 : R == 24 ? 3 : R == 25 ? 5 : R == 30 ? 5 : R == 32 ? 4 : 0;
}

// v[0..R) <- DFT (S = -1) or unscaled inverse DFT (S = +1)
template <int R, int S>
struct Dft {
  static __device__ __forceinline__ void run(float2 (&v)[R]) {
    constexpr int A = c_fac(R), B = R / A;
    static_assert(A > 1 && A * B == R, "unsupported radix");
    float2 m[B][A];
    if constexpr (c_gcd(A, B) == 1) {
      unroll<0, B>([&](auto n2) {
        unroll<0, A>([&](auto n1) { m[n2][n1] = v[(B * n1 + A * n2) % R]; });
        Dft<A, S>::run(m[n2]);
      });
      unroll<0, A>([&](auto k1) {
        float2 c[B];
        unroll<0, B>([&](auto n2) { c[n2] = m[n2][k1]; });
        Dft<B, S>::run(c);
        unroll<0, B>([&](auto k2) {
          v[(B * c_inv(B % A, A) * k1 + A * c_inv(A % B, B) * k2) % R] = c[k2];
        });
      });
    } else {
      unroll<0, B>([&](auto n2) {
        unroll<0, A>([&](auto n1) { m[n2][n1] = v[B * n1 + n2]; });
        Dft<A, S>::run(m[n2]);
      });
      unroll<0, A>([&](auto k1) {
        float2 c[B];
        unroll<0, B>([&](auto n2) { c[n2] = ctw<S, decltype(n2)::value * decltype(k1)::value, R>(m[n2][k1]); });
        Dft<B, S>::run(c);
        unroll<0, B>([&](auto k2) { v[k1 + A * k2] = c[k2]; });
      });
    }
  }
};
template <int S>
struct Dft<1, S> {
  static __device__ __forceinline__ void run(float2 (&)[1]) {}
};
template <int S>
struct Dft<2, S> {
  static __device__ __forceinline__ void run(float2 (&v)[2]) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};
template <int S>
struct Dft<3, S> {
  static __device__ __forceinline__ void run(float2 (&v)[3]) {
    constexpr float h = static_cast<float>(c_sin(kPi / 3));
    const float2 s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const float2 m = make_float2(fmaf(-0.5f, s.x, v[0].x), fmaf(-0.5f, s.y, v[0].y));
    const float2 r = rot90<S>(cscale(d, h));
    v[0] = cadd(v[0], s);
    v[1] = cadd(m, r);
    v[2] = csub(m, r);
  }
};
template <int S>
struct Dft<4, S> {
  static __device__ __forceinline__ void run(float2 (&v)[4]) {
    const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    const float2 c = cadd(v[1], v[3]), d = rot90<S>(csub(v[1], v[3]));
    v[0] = cadd(a, c);
    v[1] = cadd(b, d);
    v[2] = csub(a, c);
    v[3] = csub(b, d);
  }
};
template <int S>
struct Dft<5, S> {
  static __device__ __forceinline__ void run(float2 (&v)[5]) {
    constexpr float c1 = static_cast<float>(c_cos(2 * kPi / 5)), c2 = static_cast<float>(c_cos(4 * kPi / 5));
    constexpr float s1 = static_cast<float>(c_sin(2 * kPi / 5)), s2 = static_cast<float>(c_sin(4 * kPi / 5));
    const float2 a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
    const float2 a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
    const float2 p1 = make_float2(fmaf(c2, a2.x, fmaf(c1, a1.x, v[0].x)), fmaf(c2, a2.y, fmaf(c1, a1.y, v[0].y)));
    const float2 p2 = make_float2(fmaf(c1, a2.x, fmaf(c2, a1.x, v[0].x)), fmaf(c1, a2.y, fmaf(c2, a1.y, v[0].y)));
    const float2 q1 = rot90<S>(make_float2(fmaf(s2, b2.x, s1 * b1.x), fmaf(s2, b2.y, s1 * b1.y)));
    const float2 q2 = rot90<S>(make_float2(fmaf(-s1, b2.x, s2 * b1.x), fmaf(-s1, b2.y, s2 * b1.y)));
    v[0] = cadd(v[0], cadd(a1, a2));
    v[1] = cadd(p1, q1);
    v[4] = csub(p1, q1);
    v[2] = cadd(p2, q2);
    v[3] = csub(p2, q2);
  }
};

// R-point DFT of v[0..R/2) followed by zeros: frequency 2 k + h is the
// R/2-point DFT of v[n] exp(S 2 pi i n h / R).
template <int R, int S>
__device__ __forceinline__ void dft_half_in(float2 (&v)[R]) {
  constexpr int H = R / 2;
  float2 e[H], o[H];
  unroll<0, H>([&](auto n) {
    e[n] = v[n];
    o[n] = ctw<S, decltype(n)::value, R>(v[n]);
  });
  Dft<H, S>::run(e);
  Dft<H, S>::run(o);
  unroll<0, H>([&](auto k) {
    v[2 * k] = e[k];
    v[2 * k + 1] = o[k];
  });
}
// the first R/2 outputs of the R-point DFT of v, in v[0..R/2)
template <int R, int S>
__device__ __forceinline__ void dft_half_out(float2 (&v)[R]) {
  constexpr int H = R / 2;
  float2 e[H], o[H];
  unroll<0, H>([&](auto k) {
    e[k] = v[2 * k];
    o[k] = v[2 * k + 1];
  });
  Dft<H, S>::run(e);
  Dft<H, S>::run(o);
  unroll<0, H>([&](auto n) { v[n] = cadd(e[n], ctw<S, decltype(n)::value, R>(o[n])); });
}

// ---- a length and its stages ------------------------------------------------
// Q1, Q2: strides (complex elements) of the buffer index k1 Q1 + j Q2 + r2,
// the padding with the fewest bank conflicts over the three access patterns.
template <int L_, int R1_, int R2_, int R3_, int Q1_, int Q2_>
struct Len {
  static constexpr int L = L_, R1 = R1_, R2 = R2_, R3 = R3_, Q1 = Q1_, Q2 = Q2_;
  static constexpr int N1 = L / R1;              // threads of stage 1
  static constexpr int RL = R3 > 1 ? R3 : R2;    // radix of the last stage
  static constexpr int NL = L / RL;              // threads of the last stage
  static constexpr int N2 = L / R2;
  static constexpr int T = N1 > NL ? (N1 > N2 ? N1 : N2) : (NL > N2 ? NL : N2);
  static constexpr int SZ = R1 * Q1;             // buffer elements
  static constexpr int TW = L + R2 * R3;         // twiddles: [k1][r], then [k2][r2]
  static_assert(R1 * R2 * R3 == L && R1 % 2 == 0, "bad length");
  static_assert(R3 == 1 || T >= N2, "threads");
};

// Stages of one line.  W: distance between the line's elements in the buffer
// (columns interleaved); `sm` already points at the line's first element.
template <class F, int W, bool HALF>
struct Line {
  static constexpr int R1 = F::R1, R2 = F::R2, R3 = F::R3;

  // v: thread t's inputs i1 N1 + t; o: its outputs, slots j NL + t.  Every
  // thread of the block must call this (barriers); those with ok == false
  // only wait.
  static __device__ __forceinline__ void forward(float2 (&v)[R1], float2 (&o)[F::RL], float2* sm, int t, bool ok,
                                                 const float2* __restrict__ tw) {
    if (ok && t < F::N1) {
      if constexpr (HALF) dft_half_in<R1, -1>(v);
      else Dft<R1, -1>::run(v);
      float2* p = sm + (R3 > 1 ? (t / R3) * F::Q2 + t % R3 : t) * W;
      p[0] = v[0];
      unroll<1, R1>([&](auto k) { p[k * F::Q1 * W] = twmul<-1>(v[k], __ldg(tw + k * F::N1 + t)); });
    }
    __syncthreads();
    if constexpr (R3 > 1) {
      if (ok && t < F::N2) {
        const int k1 = t / R3, r2 = t % R3;
        float2* p = sm + (k1 * F::Q1 + r2) * W;
        float2 u[R2];
        unroll<0, R2>([&](auto j) { u[j] = p[j * F::Q2 * W]; });
        Dft<R2, -1>::run(u);
        p[0] = u[0];
        unroll<1, R2>([&](auto k) { p[k * F::Q2 * W] = twmul<-1>(u[k], __ldg(tw + F::L + k * R3 + r2)); });
      }
      __syncthreads();
    }
    if (ok && t < F::NL) {
      const float2* p = sm + last(t) * W;
      unroll<0, F::RL>([&](auto j) { o[j] = p[j * W]; });
      Dft<F::RL, -1>::run(o);
    }
  }

  // The unscaled inverse from the slots o back to v (HALF: v[0..R1/2) only).
  // The caller keeps the buffer free of other lines' reads before the call.
  static __device__ __forceinline__ void inverse(float2 (&o)[F::RL], float2 (&v)[R1], float2* sm, int t, bool ok,
                                                 const float2* __restrict__ tw) {
    if (ok && t < F::NL) {
      Dft<F::RL, 1>::run(o);
      float2* p = sm + last(t) * W;
      unroll<0, F::RL>([&](auto j) { p[j * W] = o[j]; });
    }
    __syncthreads();
    if constexpr (R3 > 1) {
      if (ok && t < F::N2) {
        const int k1 = t / R3, r2 = t % R3;
        float2* p = sm + (k1 * F::Q1 + r2) * W;
        float2 u[R2];
        u[0] = p[0];
        unroll<1, R2>([&](auto k) { u[k] = twmul<1>(p[k * F::Q2 * W], __ldg(tw + F::L + k * R3 + r2)); });
        Dft<R2, 1>::run(u);
        unroll<0, R2>([&](auto j) { p[j * F::Q2 * W] = u[j]; });
      }
      __syncthreads();
    }
    if (ok && t < F::N1) {
      const float2* p = sm + (R3 > 1 ? (t / R3) * F::Q2 + t % R3 : t) * W;
      v[0] = p[0];
      unroll<1, R1>([&](auto k) { v[k] = twmul<1>(p[k * F::Q1 * W], __ldg(tw + k * F::N1 + t)); });
      if constexpr (HALF) dft_half_out<R1, 1>(v);
      else Dft<R1, 1>::run(v);
    }
  }

  // first element of the last stage's operands of thread t
  static __device__ __forceinline__ int last(int t) {
    if constexpr (R3 > 1) return (t / R2) * F::Q1 + (t % R2) * F::Q2;
    else return t * F::Q1;
  }
};

// Lines per block of the row kernel: about 256 threads and at most 40 KB.
template <class F>
constexpr int rows_per_block() {
  constexpr int by_threads = F::T >= 192 ? 1 : 256 / F::T, by_smem = 5120 / F::SZ;  // 40 KB
  return by_smem < 1 ? 1 : by_threads < by_smem ? by_threads : by_smem;
}

// Groups of threads an output row's coils are dealt to (a block of 256
// threads, of 160 where a line takes two stages and its threads hold more).
// Measured at (length, coils): groups for 512 threads against these,
// 640, 16: 20.4 -> 16.4 us; 768, 24: 54 -> 26; 384, 24: 21.4 -> 15.9;
// 256, 16: 7.7 -> 6.4: smaller blocks leave the tail of the last wave short.
template <class F>
constexpr int coil_groups() {
  constexpr int n = F::R3 > 1 ? 256 : 160;
  return 2 * F::T > n ? 1 : n / F::T;
}

// Groups of T threads, at most `most`, to which an output row's C coils are
// dealt.  With few rows: as many as keep them busy, unless the last turn
// would leave over a tenth of their time unused (16 coils on 3 or 2 groups of
// a 640 line: 26.5 / 21.7 us).  With rows enough for every SM: the fewest that
// make whole warps, which wait for each other least (192^3, 12 coils, groups of
// 16 threads: 10: 596 us, 6: 352, 3: 405, 2: 308, 1: 526).
inline int coil_group_count(int C, int T, int most, int64_t rows) {
  if (rows >= 8192)
    for (int g = 1; g <= most && g <= C; ++g)
      if (g * T % 32 == 0) return g;
  int g = C < most ? C : most;
  while (g > 1 && (C + g - 1) / g * g * 10 > C * 11) --g;
  return g;
}

// The lengths built, X(L, radices, buffer strides), for lines along rows
// (many threads a line, few elements each) and along columns (a thread of
// each of 8 adjacent lines: two stages of large radices trade registers for
// exchanges; 16 coils of 640: 40 us with 10 x 8 x 8, 27.5 us with 20 x 32).
// Even first radix; steps of at most 1.25 between neighbours, so that a
// padded line wastes little.
#define PGB_FFT_ROWS(X)                                                                              \
  X(64, 8, 8, 1, 9, 1) X(80, 8, 10, 1, 11, 1) X(96, 8, 12, 1, 13, 1) X(100, 10, 10, 1, 11, 1)        \
  X(108, 12, 9, 1, 9, 1) X(120, 12, 10, 1, 11, 1) X(128, 8, 16, 1, 17, 1) X(144, 12, 12, 1, 13, 1)   \
  X(160, 10, 16, 1, 17, 1) X(180, 12, 15, 1, 15, 1) X(192, 12, 16, 1, 17, 1) X(216, 6, 6, 6, 54, 9)  \
  X(240, 16, 15, 1, 15, 1) X(256, 16, 16, 1, 17, 1) X(288, 6, 6, 8, 56, 9) X(320, 10, 8, 4, 44, 5)   \
  X(360, 10, 6, 6, 54, 9) X(384, 6, 8, 8, 72, 9) X(400, 10, 10, 4, 60, 5) X(432, 6, 8, 9, 89, 10)    \
  X(480, 6, 8, 10, 90, 10) X(512, 8, 8, 8, 72, 9) X(576, 8, 9, 8, 88, 9) X(600, 6, 10, 10, 122, 11)  \
  X(640, 10, 8, 8, 72, 9) X(720, 8, 9, 10, 90, 10) X(768, 12, 8, 8, 72, 9) X(800, 10, 10, 8, 104, 9) \
  X(900, 10, 9, 10, 90, 10) X(960, 12, 10, 8, 104, 9) X(1024, 16, 8, 8, 72, 9)
#define PGB_FFT_COLS(X)                                                                               \
  X(64, 8, 8, 1, 9, 1) X(80, 8, 10, 1, 11, 1) X(96, 8, 12, 1, 13, 1) X(100, 10, 10, 1, 11, 1)         \
  X(108, 12, 9, 1, 9, 1) X(120, 12, 10, 1, 11, 1) X(128, 8, 16, 1, 17, 1) X(144, 12, 12, 1, 13, 1)    \
  X(160, 10, 16, 1, 17, 1) X(180, 12, 15, 1, 15, 1) X(192, 12, 16, 1, 17, 1) X(216, 12, 18, 1, 19, 1) \
  X(240, 16, 15, 1, 15, 1) X(256, 16, 16, 1, 17, 1) X(288, 16, 18, 1, 19, 1) X(320, 16, 20, 1, 21, 1) \
  X(360, 18, 20, 1, 21, 1) X(384, 16, 24, 1, 25, 1) X(400, 20, 20, 1, 21, 1) X(432, 18, 24, 1, 25, 1) \
  X(480, 20, 24, 1, 25, 1) X(512, 16, 32, 1, 33, 1) X(576, 24, 24, 1, 25, 1) X(600, 24, 25, 1, 25, 1) \
  X(640, 20, 32, 1, 33, 1) X(720, 24, 30, 1, 31, 1) X(768, 24, 32, 1, 33, 1) X(800, 32, 25, 1, 25, 1) \
  X(900, 30, 30, 1, 31, 1) X(960, 30, 32, 1, 33, 1) X(1024, 32, 32, 1, 33, 1)

}  // namespace fft
}  // namespace pgb
