// toep_fft.cu -- the 2-D Toeplitz normal operator in three passes over the
// coil planes, with FFTs of this library.
//
//   out[b] = sum_c conj(S_c) crop(IFFT2(P FFT2(pad(S_c x_b)))) + damp x_b
//
// Reference: _toep/_grog_toep.py:154-209 (per coil: smaps, pad, centred FFT,
// PSF, centred IFFT, crop, conj-smaps accumulate).
//
// The operator is a convolution of the n0 x n1 image with the kernel behind
// the PSF, cropped to the image, so (a) it does not depend on where in the
// padded plane the image lies: it is put at the origin, the centring shifts
// and their index maps drop out; (b) any circulant length L >= 2 n - 1 gives
// the same values once the PSF is resampled to it (exactly, from the kernel's
// lags |l| < n: pgb_toep2d_plan), so prime-factor grids run on smooth
// lengths; (c) only image rows enter and leave the column transforms.
//
//   rows:    U[b,c,q,:]  = FFT_L1(S_c x_b row q)              n0 rows of a plane, not L0
//   columns: U[b,c,:,kx] = crop(IFFT_L0(P FFT_L0(column)))    in place, in registers / shared memory
//   out:     sum over the coils of conj(S_c) crop(IFFT_L1(row))
//
// against expansion, two cuFFT transforms of two passes each, PSF and combine
// over full planes: at 16 coils of 640 x 640 (image 320 x 320) the planes move
// 105 MB instead of 627 MB an application, nearly all of it inside the 126 MB
// L2, and the time is that of the FFT arithmetic and its shared-memory
// exchanges.
//
// The frequency order of U and of the PSF is the slot order of fft_core.cuh.
#include "toep_cols.cuh"

namespace pgb {
namespace fft {

template <class F, bool HALF>
__global__ void __launch_bounds__(F::T* rows_per_block<F>())
    toep_rows_kernel(const float2* __restrict__ x, const float2* __restrict__ smaps, float2* __restrict__ U, int C,
                     int n0, int n1, int64_t units, const float2* __restrict__ tw) {
  __shared__ float2 sm[rows_per_block<F>()][F::SZ];
  grid_wait();
  const int t = threadIdx.x;
  const int64_t unit = static_cast<int64_t>(blockIdx.x) * blockDim.y + threadIdx.y;  // (b, q, c), c fastest
  const bool ok = unit < units;
  const int64_t row = ok ? unit / C : 0;
  const int c = ok ? static_cast<int>(unit - row * C) : 0;
  const int64_t b = row / n0;
  const int q = static_cast<int>(row - b * n0);
  float2 v[F::R1], o[F::RL];
  if (ok && t < F::N1) {
    const float2* xr = x + row * n1;
    const float2* sr = smaps ? smaps + (static_cast<int64_t>(c) * n0 + q) * n1 : nullptr;
    unroll<0, F::R1>([&](auto i) {
      if constexpr (HALF && decltype(i)::value >= F::R1 / 2) return;
      const int e = i * F::N1 + t;
      float2 a = make_float2(0.f, 0.f);
      if (e < n1) {
        a = xr[e];
        if (sr) a = cmul(a, sr[e]);
      }
      v[i] = a;
    });
  }
  Line<F, 1, HALF>::forward(v, o, sm[threadIdx.y], t, ok, tw);
  if (ok && t < F::NL) {
    float2* ur = U + ((b * C + c) * n0 + q) * F::L + t;
    unroll<0, F::RL>([&](auto j) { ur[j * F::NL] = o[j]; });
  }
}

// One image row of one frame per block; its coils are dealt to blockDim.y
// groups of threads, whose partial sums are added in group order: results do
// not vary from run to run.  The next coil's line is loaded before this one's
// stages.
template <class F, bool HALF>
__global__ void __launch_bounds__(F::T* coil_groups<F>())
    toep_out_kernel(const float2* __restrict__ U, const float2* __restrict__ smaps, float2* __restrict__ out, int C,
                    int n0, int n1, const float2* __restrict__ add, float add_scale, const float2* __restrict__ tw) {
  extern __shared__ float2 smo[];  // (groups, max(F::SZ, F::L))
  constexpr int SZ = F::SZ > F::L ? F::SZ : F::L;
  constexpr int NV = HALF ? F::R1 / 2 : F::R1;
  grid_wait();
  const int t = threadIdx.x, g = threadIdx.y, ng = blockDim.y;
  float2* sm = smo + g * SZ;
  const int64_t row = blockIdx.x;
  const int64_t b = row / n0;
  const int q = static_cast<int>(row - b * n0);
  float2 acc[NV], nxt[F::RL];
  unroll<0, NV>([&](auto i) { acc[i] = make_float2(0.f, 0.f); });
  const auto load = [&](int c) {
    if (c < C && t < F::NL) {
      const float2* ur = U + ((b * C + c) * n0 + q) * F::L + t;
      unroll<0, F::RL>([&](auto j) { nxt[j] = ur[j * F::NL]; });
    }
  };
  load(g);
  for (int c0 = 0; c0 < C; c0 += ng) {
    const int c = c0 + g;
    const bool ok = c < C;
    float2 v[F::R1], o[F::RL], sv[NV];
    unroll<0, F::RL>([&](auto j) { o[j] = nxt[j]; });
    if (ok && smaps && t < F::N1) {
      const float2* sr = smaps + (static_cast<int64_t>(c) * n0 + q) * n1;
      unroll<0, NV>([&](auto i) {
        const int e = i * F::N1 + t;
        sv[i] = e < n1 ? sr[e] : make_float2(0.f, 0.f);
      });
    }
    load(c + ng);
    if (c0) __syncthreads();  // the previous coil's last reads
    Line<F, 1, HALF>::inverse(o, v, sm, t, ok, tw);
    if (ok && t < F::N1) {
      unroll<0, NV>([&](auto i) {
        if (smaps) cfma_conj(acc[i], sv[i], v[i]);
        else acc[i] = cadd(acc[i], v[i]);
      });
    }
  }
  __syncthreads();
  if (t < F::N1) {
    unroll<0, NV>([&](auto i) {
      const int e = i * F::N1 + t;
      if (e < n1) sm[e] = acc[i];
    });
  }
  __syncthreads();
  for (int e = g * F::T + t; e < n1; e += ng * F::T) {
    float2 s = smo[e];
    for (int k = 1; k < ng; ++k) s = cadd(s, smo[k * SZ + e]);
    const int64_t i = row * n1 + e;
    if (add) {
      const float2 a = add[i];
      s.x = fmaf(add_scale, a.x, s.x);
      s.y = fmaf(add_scale, a.y, s.y);
    }
    out[i] = s;
  }
}

template <class F, bool HALF>
int launch_rows(const float2* x, const float2* S, float2* U, int64_t B, int C, int n0, int n1, const float2* tw,
                cudaStream_t s) {
  constexpr int FB = rows_per_block<F>();
  const int64_t units = B * n0 * C;
  launch_chained(toep_rows_kernel<F, HALF>, static_cast<unsigned>((units + FB - 1) / FB), dim3(F::T, FB), 0, s, x, S, U,
                 C, n0, n1, units, tw);
  PGB_LAUNCH_CHECK("toep_rows");
  return PGB_OK;
}

template <class F, bool HALF>
int launch_out(const float2* U, const float2* S, float2* out, int64_t B, int C, int n0, int n1, const float2* add,
               float add_scale, const float2* tw, cudaStream_t s) {
  constexpr int GM = coil_groups<F>();
  const int G = coil_group_count(C, F::T, GM, B * n0);
  const size_t smem = sizeof(float2) * (F::SZ > F::L ? F::SZ : F::L) * G;
  auto k = toep_out_kernel<F, HALF>;
  if (smem > 48 * 1024) allow_smem<toep_out_kernel<F, HALF>>(227 * 1024);
  launch_chained(k, static_cast<unsigned>(B * n0), dim3(F::T, G), smem, s, U, S, out, C, n0, n1, add, add_scale, tw);
  PGB_LAUNCH_CHECK("toep_out");
  return PGB_OK;
}

// ---- plan: twiddles and the PSF on the circulant lengths, in slot order ----
struct Radices {
  int L, R1, R2, R3;
};
__device__ __forceinline__ int slot_freq(const Radices& r, int s) {
  if (r.R3 == 1) return s % r.R1 + r.R1 * (s / r.R1);
  const int t = s % (r.R1 * r.R2), k3 = s / (r.R1 * r.R2);
  return t / r.R2 + r.R1 * (t % r.R2) + r.R1 * r.R2 * k3;
}

// exp(-2 pi i k r / L) as Line reads them, from FP64 (axis 0, then axis 1)
__global__ void toep_twiddle_kernel(Radices a, Radices b, float2* __restrict__ tw0, float2* __restrict__ tw1) {
  const Radices r = blockIdx.y ? b : a;
  float2* tw = blockIdx.y ? tw1 : tw0;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int k, n;
  if (r.L == 0) return;
  if (i < r.L) {
    k = (i / (r.L / r.R1)) * (i % (r.L / r.R1)) % r.L;
    n = r.L;
  } else if (i < r.L + r.R2 * r.R3) {
    const int j = i - r.L;
    n = r.R2 * r.R3;
    k = (j / r.R3) * (j % r.R3) % n;
  } else {
    return;
  }
  double s, c;
  sincospi(-2.0 * k / n, &s, &c);
  tw[i] = make_float2(static_cast<float>(c), static_cast<float>(s));
}

// D[k][slot of j] = sum over lags |l| < n of exp(2 pi i l (k / N - j / L)) / N
//                 = sin((2 n - 1) a) / (N sin a),  a = pi (k L - j N) / (N L):
// inverse DFT of length N, the lags wrapped to length L, DFT of length L.
__global__ void toep_dirichlet_kernel(Radices r, int N, int n, double* __restrict__ D) {
  const int64_t NL = static_cast<int64_t>(N) * r.L;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < NL;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int k = static_cast<int>(i / r.L), s = static_cast<int>(i - static_cast<int64_t>(k) * r.L);
    const int64_t d = ((static_cast<int64_t>(k) * r.L - static_cast<int64_t>(slot_freq(r, s)) * N) % NL + NL) % NL;
    const int64_t w = 2 * n - 1;
    D[i] = d == 0 ? static_cast<double>(w) / N
                  : sinpi(static_cast<double>(w * d % (2 * NL)) / NL) / (N * sinpi(static_cast<double>(d) / NL));
  }
}

// T[i][s1][m]: axis 1 of the centred PSF (N0, N1, M) taken to the slots of L1;
// i in FFT order (D == nullptr: L1 == N1, a gather).
__global__ void toep_plan1_kernel(const float* __restrict__ psf, int N0, int N1, int M, Radices r,
                                  const double* __restrict__ D, double* __restrict__ T) {
  const int64_t total = static_cast<int64_t>(N0) * r.L * M;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t is = i / M;
    const int m = static_cast<int>(i - is * M), row = static_cast<int>(is / r.L), s = static_cast<int>(is % r.L);
    const float* p = psf + static_cast<int64_t>((row + N0 / 2) % N0) * N1 * M + m;
    double v = 0.0;
    if (D == nullptr) {
      v = p[static_cast<int64_t>((slot_freq(r, s) + N1 / 2) % N1) * M];
    } else {
      for (int k = 0; k < N1; ++k)
        v = fma(D[static_cast<int64_t>(k) * r.L + s], static_cast<double>(p[static_cast<int64_t>((k + N1 / 2) % N1) * M]), v);
    }
    T[i] = v;
  }
}

// out[s0][x] = scale * axis 0 of T (N0, X) taken to the slots of L0
__global__ void toep_plan0_kernel(const double* __restrict__ T, int N0, int64_t X, Radices r,
                                  const double* __restrict__ D, double scale, float* __restrict__ out) {
  const int64_t total = X * r.L;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int s = static_cast<int>(i / X);
    const int64_t x = i - s * X;
    double v = 0.0;
    if (D == nullptr) {
      v = T[slot_freq(r, s) * X + x];
    } else {
      for (int k = 0; k < N0; ++k) v = fma(D[static_cast<int64_t>(k) * r.L + s], T[k * X + x], v);
    }
    out[i] = static_cast<float>(scale * v);
  }
}

// radices of a built length (along columns: axis 0); L == 0 if it is not built
static Radices radices(int64_t L, bool columns) {
  static const Radices rows[] = {
#define X(L, A, B_, C_, Q, R) {L, A, B_, C_},
      PGB_FFT_ROWS(X)
  };
  static const Radices cols[] = {PGB_FFT_COLS(X)
#undef X
  };
  for (const Radices& r : rows)
    if (r.L == L) return columns ? cols[&r - rows] : r;
  return Radices{0, 1, 1, 1};
}
static const int kLengths[] = {
#define X(L, A, B_, C_, Q, R) L,
    PGB_FFT_ROWS(X)
#undef X
};

}  // namespace fft
}  // namespace pgb

using namespace pgb;
using namespace pgb::fft;

extern "C" {

int pgb_fft_length(int64_t i) {
  const int64_t n = sizeof(kLengths) / sizeof(kLengths[0]);
  return i >= 0 && i < n ? kLengths[i] : 0;
}

int64_t pgb_fft_twiddles(int64_t L) {
  const Radices a = radices(L, true), b = radices(L, false);
  const int64_t x = a.R2 * a.R3, y = b.R2 * b.R3;
  return a.L == 0 ? 0 : L + (x > y ? x : y);
}

int pgb_fft_twiddle_tables(int64_t L0, int64_t L1, void* tw0, void* tw1, void* stream) {
  clear_error();
  const Radices r0 = radices(L0, true), r1 = radices(L1, false);
  PGB_REQUIRE((r0.L || !L0) && (r1.L || !L1), PGB_ERR_UNSUPPORTED, "fft_twiddle_tables: lengths %lld x %lld are not built",
              (long long)L0, (long long)L1);
  PGB_REQUIRE((tw0 || !L0) && (tw1 || !L1), PGB_ERR_INVALID, "fft_twiddle_tables: null pointer");
  toep_twiddle_kernel<<<dim3(16, 2), 128, 0, as_stream(stream)>>>(r0, r1, static_cast<float2*>(tw0),
                                                                  static_cast<float2*>(tw1));
  PGB_LAUNCH_CHECK("fft_twiddle_tables");
  return PGB_OK;
}

int pgb_toep2d_plan(const float* psf, int64_t S, int64_t M, int64_t N0, int64_t N1, int64_t n0, int64_t n1,
                    int64_t L0, int64_t L1, void* work, float* out, void* tw0, void* tw1, void* stream) {
  clear_error();
  PGB_REQUIRE(S >= 0 && M >= 1 && n0 >= 1 && n1 >= 1 && n0 <= N0 && n1 <= N1 && N0 < (1 << 20) && N1 < (1 << 20),
              PGB_ERR_INVALID, "toep2d_plan: invalid sizes");
  const Radices r0 = radices(L0, true), r1 = radices(L1, false);
  PGB_REQUIRE(r0.L && r1.L, PGB_ERR_UNSUPPORTED, "toep2d_plan: lengths %lld x %lld are not built", (long long)L0,
              (long long)L1);
  PGB_REQUIRE((L0 == N0 || L0 >= 2 * n0 - 1) && (L1 == N1 || L1 >= 2 * n1 - 1), PGB_ERR_INVALID,
              "toep2d_plan: circulant length shorter than the kernel");
  PGB_REQUIRE(psf && work && out && tw0 && tw1, PGB_ERR_INVALID, "toep2d_plan: null pointer");
  cudaStream_t s = as_stream(stream);
  toep_twiddle_kernel<<<dim3(16, 2), 128, 0, s>>>(r0, r1, static_cast<float2*>(tw0), static_cast<float2*>(tw1));
  PGB_LAUNCH_CHECK("toep2d_plan(twiddles)");
  double* D0 = static_cast<double*>(work);
  double* D1 = D0 + N0 * L0;
  double* T = D1 + N1 * L1;
  const int m0 = static_cast<int>(N0), m1 = static_cast<int>(N1), mm = static_cast<int>(M);
  if (L0 != N0) toep_dirichlet_kernel<<<grid_for(N0 * L0, 256), 256, 0, s>>>(r0, m0, static_cast<int>(n0), D0);
  if (L1 != N1) toep_dirichlet_kernel<<<grid_for(N1 * L1, 256), 256, 0, s>>>(r1, m1, static_cast<int>(n1), D1);
  for (int64_t k = 0; k < S; ++k) {
    toep_plan1_kernel<<<grid_for(N0 * L1 * M, 256), 256, 0, s>>>(psf + k * N0 * N1 * M, m0, m1, mm, r1,
                                                                 L1 != N1 ? D1 : nullptr, T);
    toep_plan0_kernel<<<grid_for(L0 * L1 * M, 256), 256, 0, s>>>(T, m0, L1 * M, r0, L0 != N0 ? D0 : nullptr,
                                                                 1.0 / (static_cast<double>(L0) * L1),
                                                                 out + k * L0 * L1 * M);
  }
  PGB_LAUNCH_CHECK("toep2d_plan");
  return PGB_OK;
}

int pgb_toep_slots(const double* psf, int64_t L, int64_t X, double scale, float* out, void* stream) {
  clear_error();
  const Radices r = radices(L, true);
  PGB_REQUIRE(r.L, PGB_ERR_UNSUPPORTED, "toep_slots: length %lld is not built", (long long)L);
  PGB_REQUIRE(X >= 0 && (X == 0 || (psf && out)), PGB_ERR_INVALID, "toep_slots: invalid arguments");
  if (X == 0) return PGB_OK;
  toep_plan0_kernel<<<grid_for(X * L, 256), 256, 0, as_stream(stream)>>>(psf, static_cast<int>(L), X, r, nullptr, scale,
                                                                        out);
  PGB_LAUNCH_CHECK("toep_slots");
  return PGB_OK;
}

int pgb_toep2d(const void* x, const void* smaps, const float* psf, void* work, void* out, int64_t B, int64_t C,
               int64_t K, int64_t n0, int64_t n1, int64_t L0, int64_t L1, const void* tw0, const void* tw1, const void* add,
               float add_scale, void* stream) {
  clear_error();
  PGB_REQUIRE(B >= 0 && C >= 1 && n0 >= 1 && n1 >= 1 && n0 <= L0 && n1 <= L1, PGB_ERR_INVALID, "toep2d: invalid sizes");
  if (B == 0) return PGB_OK;
  PGB_REQUIRE(x && psf && work && out && tw0 && tw1, PGB_ERR_INVALID, "toep2d: null pointer");
  // blocks of the passes: rows, and columns (4 a block with components)
  PGB_REQUIRE(L0 <= 4096 && L1 <= 4096 && B < (1 << 28) && C < (1 << 28) && B * C < (int64_t(1) << 31) &&
                  B * C * (K > 0 ? K : 1) * n0 < (int64_t(1) << 31) && B * C * ((L1 + 3) / 4) < (int64_t(1) << 31),
              PGB_ERR_RANGE, "toep2d: too many planes");
  PGB_REQUIRE(K >= 0 && K <= kSubMax, PGB_ERR_UNSUPPORTED, "toep2d: at most %d components", kSubMax);
  const int64_t BC = B * C;
  if (K > 0) B *= K;  // every component is an image
  cudaStream_t s = as_stream(stream);
  const float2* xi = static_cast<const float2*>(x);
  const float2* S = static_cast<const float2*>(smaps);
  float2* U = static_cast<float2*>(work);
  const float2* t0 = static_cast<const float2*>(tw0);
  const float2* t1 = static_cast<const float2*>(tw1);
  const int c = static_cast<int>(C), m0 = static_cast<int>(n0), m1 = static_cast<int>(n1);
  const int l1 = static_cast<int>(L1);
  int st = PGB_ERR_UNSUPPORTED;
  const bool h0 = 2 * n0 <= L0, h1 = 2 * n1 <= L1;  // the upper half of a line is padding
  switch (L1) {
#define X(L, A, B_, C_, Q, R)                                                             \
  case L:                                                                                 \
    st = h1 ? launch_rows<Len<L, A, B_, C_, Q, R>, true>(xi, S, U, B, c, m0, m1, t1, s)    \
            : launch_rows<Len<L, A, B_, C_, Q, R>, false>(xi, S, U, B, c, m0, m1, t1, s);  \
    break;
    PGB_FFT_ROWS(X)
#undef X
  }
  PGB_REQUIRE(st != PGB_ERR_UNSUPPORTED, st, "toep2d: length %lld is not built", (long long)L1);
  if (st) return st;
  st = K == 0 ? toep_cols(U, psf, BC, m0, l1, static_cast<int>(L0), t0, s)
              : toep_sub_cols(U, psf, BC, c, static_cast<int>(K), m0, l1, static_cast<int>(L0), t0, s);
  PGB_REQUIRE(st != PGB_ERR_UNSUPPORTED, st, "toep2d: length %lld is not built", (long long)L0);
  if (st) return st;
  const float2* a = static_cast<const float2*>(add);
  switch (L1) {
#define X(L, A, B_, C_, Q, R)                                                                                       \
  case L:                                                                                                           \
    st = h1 ? launch_out<Len<L, A, B_, C_, Q, R>, true>(U, S, static_cast<float2*>(out), B, c, m0, m1, a, add_scale, t1, s) \
            : launch_out<Len<L, A, B_, C_, Q, R>, false>(U, S, static_cast<float2*>(out), B, c, m0, m1, a, add_scale, t1, s); \
    break;
    PGB_FFT_ROWS(X)
#undef X
  }
  return st;
}

}  // extern "C"
