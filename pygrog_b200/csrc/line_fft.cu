// line_fft.cu -- 2-D and 3-D centred transforms between coil images and
// FFT-order grids on line FFTs, with the coil maps at the image end.
//
//   image to grid: V[b,c] = FFT(pad(S_c x_b))
//   grid to image: out[b] = scale * sum_c conj(S_c) crop(IFFT(V[b,c])) (+ add)
//
// Reference: operator/_sparse_fft.py:574-621, 741-789 (per coil: pad or crop,
// centred transform, maps).
//
// Expansion, a cuFFT transform of two passes and (in the other direction) a
// combine pass move the padded planes five or six times; here the rows that
// are padding never exist, the maps are applied as the image rows are read
// and written, and the planes are written (read) once by the column pass and
// n0 / L0 of them twice by the row pass: at 16 coils of 640 x 640 (image 320)
// 131 MB instead of 328.  In 3-D the middle axis and z are two column passes,
// in place where the image is not padded along them.
#include "line_fft.cuh"
#include "toep_cols.cuh"

namespace pgb {
namespace fft {

// U[b, c, q, :] = FFT of row q of S_c x_b, natural order: the slots pass
// through shared memory once more, so that rows are written whole.
template <class F>
__global__ void __launch_bounds__(F::T* rows_per_block<F>())
    line_rows_kernel(const float2* __restrict__ x, const float2* __restrict__ smaps, float2* __restrict__ U, int C,
                     int n0, Centre ce, int64_t units, const float2* __restrict__ tw) {
  __shared__ float2 smr[rows_per_block<F>()][F::SZ];
  float2* sm = smr[threadIdx.y];
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
    const float2* xr = x + row * ce.n;
    const float2* sr = smaps ? smaps + (static_cast<int64_t>(c) * n0 + q) * ce.n : nullptr;
    unroll<0, F::R1>([&](auto i) {
      const int e = ce.index<F::L>(i * F::N1 + t);
      float2 a = make_float2(0.f, 0.f);
      if (e >= 0 && e < ce.n) {
        a = xr[e];
        if (sr) a = cmul(a, sr[e]);
      }
      v[i] = a;
    });
  }
  Line<F, 1, false>::forward(v, o, sm, t, ok, tw);
  __syncthreads();
  if (ok && t < F::NL) unroll<0, F::RL>([&](auto j) { sm[out_freq<F>(t, j)] = o[j]; });
  __syncthreads();
  if (ok) {
    float2* ur = U + ((b * C + c) * n0 + q) * F::L;
    for (int e = t; e < F::L; e += F::T) ur[e] = sm[e];
  }
}

// One image row of one frame per block, its coils dealt to groups of threads
// and summed in group order (toep_out_kernel), from rows in natural order.
template <class F>
__global__ void __launch_bounds__(F::T* coil_groups<F>())
    line_out_kernel(const float2* __restrict__ U, const float2* __restrict__ smaps, float2* __restrict__ out, int C,
                    int n0, Centre ce, float scale, const float2* __restrict__ add, float add_scale,
                    const float2* __restrict__ tw) {
  extern __shared__ float2 smo[];  // (groups, F::SZ)
  static_assert(F::SZ >= F::L, "a row fits the buffer");
  grid_wait();
  const int t = threadIdx.x, g = threadIdx.y, ng = blockDim.y;
  float2* sm = smo + g * F::SZ;
  const int64_t row = blockIdx.x;
  const int64_t b = row / n0;
  const int q = static_cast<int>(row - b * n0);
  constexpr int NX = (F::L + F::T - 1) / F::T;
  float2 acc[F::R1], nxt[NX];
  unroll<0, F::R1>([&](auto i) { acc[i] = make_float2(0.f, 0.f); });
  const auto load = [&](int c) {
    if (c < C) {
      const float2* ur = U + ((b * C + c) * n0 + q) * F::L;
      unroll<0, NX>([&](auto i) {
        if (i * F::T + t < F::L) nxt[i] = ur[i * F::T + t];
      });
    }
  };
  load(g);
  for (int c0 = 0; c0 < C; c0 += ng) {
    const int c = c0 + g;
    const bool ok = c < C;
    float2 v[F::R1], o[F::RL], sv[F::R1];
    if (c0) __syncthreads();  // the previous coil's last reads
    if (ok) unroll<0, NX>([&](auto i) {
        if (i * F::T + t < F::L) sm[i * F::T + t] = nxt[i];
      });
    if (ok && smaps && t < F::N1) {
      const float2* sr = smaps + (static_cast<int64_t>(c) * n0 + q) * ce.n;
      unroll<0, F::R1>([&](auto i) {
        const int e = ce.index<F::L>(i * F::N1 + t);
        sv[i] = e >= 0 && e < ce.n ? sr[e] : make_float2(0.f, 0.f);
      });
    }
    load(c + ng);
    __syncthreads();
    if (ok && t < F::NL) unroll<0, F::RL>([&](auto j) { o[j] = sm[out_freq<F>(t, j)]; });
    __syncthreads();
    Line<F, 1, false>::inverse(o, v, sm, t, ok, tw);
    if (ok && t < F::N1) {
      unroll<0, F::R1>([&](auto i) {
        if (smaps) cfma_conj(acc[i], sv[i], v[i]);
        else acc[i] = cadd(acc[i], v[i]);
      });
    }
  }
  __syncthreads();
  if (t < F::N1) {
    unroll<0, F::R1>([&](auto i) {
      const int e = ce.index<F::L>(i * F::N1 + t);
      if (e >= 0 && e < ce.n) sm[e] = acc[i];
    });
  }
  __syncthreads();
  for (int e = g * F::T + t; e < ce.n; e += ng * F::T) {
    float2 s = smo[e];
    for (int k = 1; k < ng; ++k) s = cadd(s, smo[k * F::SZ + e]);
    s = cscale(s, scale);
    const int64_t i = row * ce.n + e;
    if (add) {
      const float2 a = add[i];
      s.x = fmaf(add_scale, a.x, s.x);
      s.y = fmaf(add_scale, a.y, s.y);
    }
    out[i] = s;
  }
}

template <class F>
int launch_line_rows(const float2* x, const float2* S, float2* U, int64_t B, int C, int n0, int n1, const float2* tw,
                     cudaStream_t s) {
  constexpr int FB = rows_per_block<F>();
  const int64_t units = B * n0 * C;
  const Centre ce{n1, F::L / 2 - (F::L - n1) / 2};
  launch_chained(line_rows_kernel<F>, static_cast<unsigned>((units + FB - 1) / FB), dim3(F::T, FB), 0, s, x, S, U, C, n0,
                 ce, units, tw);
  PGB_LAUNCH_CHECK("line_rows");
  return PGB_OK;
}

template <class F>
int launch_line_out(const float2* U, const float2* S, float2* out, int64_t B, int C, int n0, int n1, float scale,
                    const float2* add, float add_scale, const float2* tw, cudaStream_t s) {
  constexpr int GM = coil_groups<F>();
  const int G = coil_group_count(C, F::T, GM, B * n0);
  const size_t smem = sizeof(float2) * F::SZ * G;
  auto k = line_out_kernel<F>;
  if (smem > 48 * 1024) allow_smem<line_out_kernel<F>>(227 * 1024);
  const Centre ce{n1, F::L / 2 - (F::L - n1) / 2};
  launch_chained(k, static_cast<unsigned>(B * n0), dim3(F::T, G), smem, s, U, S, out, C, n0, ce, scale, add, add_scale,
                 tw);
  PGB_LAUNCH_CHECK("line_out");
  return PGB_OK;
}

struct Axes {
  int64_t n[3], g[3];  // image and grid, the first 1 in 2-D
  const float2* tw[3];
  int64_t n01, g12;
};

static int line_axes(int64_t B, int64_t C, int ndim, const int64_t* image, const int64_t* grid, const void* const* tw,
                     Axes& a, const char* who) {
  PGB_REQUIRE(B >= 0 && C >= 1 && (ndim == 2 || ndim == 3) && image && grid && tw, PGB_ERR_INVALID, "%s: invalid sizes",
              who);
  for (int d = 0; d < 3; ++d) {
    const int k = d - (3 - ndim);
    a.n[d] = k < 0 ? 1 : image[k];
    a.g[d] = k < 0 ? 1 : grid[k];
    a.tw[d] = k < 0 ? nullptr : static_cast<const float2*>(tw[k]);
    PGB_REQUIRE(a.n[d] >= 1 && a.n[d] <= a.g[d] && (k < 0 || a.tw[d]), PGB_ERR_INVALID, "%s: invalid sizes", who);
    PGB_REQUIRE(a.g[d] <= 4096, PGB_ERR_RANGE, "%s: grid too large", who);
  }
  a.n01 = a.n[0] * a.n[1];
  a.g12 = a.g[1] * a.g[2];
  // blocks of the widest passes: rows, columns of the middle axis (n[0] planes of a coil image), columns of z
  const int64_t middle = a.n[0] * ((a.g[2] + 7) / 8), z = ndim == 3 ? (a.g12 + 7) / 8 : 0;
  const int64_t most = a.n01 > middle ? (a.n01 > z ? a.n01 : z) : (middle > z ? middle : z);
  PGB_REQUIRE(B < (1 << 28) && C < (1 << 28) && B * C < (int64_t(1) << 31) && B * C * most < (int64_t(1) << 31),
              PGB_ERR_RANGE, "%s: too many planes", who);
  return PGB_OK;
}

static int rows_pass(const Axes& a, const float2* x, const float2* S, float2* U, int64_t B, int64_t C, cudaStream_t s) {
  const int c = static_cast<int>(C), m0 = static_cast<int>(a.n01), m1 = static_cast<int>(a.n[2]);
  switch (a.g[2]) {
#define X(L, A, B_, C_, Q, R) \
  case L:                     \
    return launch_line_rows<Len<L, A, B_, C_, Q, R>>(x, S, U, B, c, m0, m1, a.tw[2], s);
    PGB_FFT_ROWS(X)
#undef X
  }
  return PGB_ERR_UNSUPPORTED;
}

static int out_pass(const Axes& a, const float2* U, const float2* S, float2* out, int64_t B, int64_t C, float scale,
                    const float2* add, float add_scale, cudaStream_t s) {
  const int c = static_cast<int>(C), m0 = static_cast<int>(a.n01), m1 = static_cast<int>(a.n[2]);
  switch (a.g[2]) {
#define X(L, A, B_, C_, Q, R) \
  case L:                     \
    return launch_line_out<Len<L, A, B_, C_, Q, R>>(U, S, out, B, c, m0, m1, scale, add, add_scale, a.tw[2], s);
    PGB_FFT_ROWS(X)
#undef X
  }
  return PGB_ERR_UNSUPPORTED;
}

static int middle_pass(const Axes& a, float2* U, float2* V, int64_t BC, bool inverse, cudaStream_t s) {
  return line_cols(U, V, BC * a.n[0], static_cast<int>(a.n[1]), static_cast<int>(a.g[2]), static_cast<int>(a.g[1]), inverse,
                   a.tw[1], s);
}

}  // namespace fft
}  // namespace pgb

using namespace pgb;
using namespace pgb::fft;

extern "C" {

int pgb_line_to_grid(const void* x, const void* smaps, void* work, void* work2, void* grid, int64_t B, int64_t C,
                     int ndim, const int64_t* image, const int64_t* shape, const void* const* tw, void* stream) {
  clear_error();
  Axes a;
  int st = line_axes(B, C, ndim, image, shape, tw, a, "line_to_grid");
  if (st || B == 0) return st;
  PGB_REQUIRE(x && work && grid && (ndim == 2 || work2), PGB_ERR_INVALID, "line_to_grid: null pointer");
  cudaStream_t s = as_stream(stream);
  float2 *U = static_cast<float2*>(work), *V = static_cast<float2*>(ndim == 2 ? grid : work2);
  st = rows_pass(a, static_cast<const float2*>(x), static_cast<const float2*>(smaps), U, B, C, s);
  if (st == PGB_OK) st = middle_pass(a, U, V, B * C, false, s);
  if (st == PGB_OK && ndim == 3)
    st = line_cols(V, static_cast<float2*>(grid), B * C, static_cast<int>(a.n[0]), static_cast<int>(a.g12),
                   static_cast<int>(a.g[0]), false, a.tw[0], s);
  PGB_REQUIRE(st != PGB_ERR_UNSUPPORTED, st, "line_to_grid: a length is not built");
  return st;
}

int pgb_line_to_image(void* grid, const void* smaps, void* work, void* work2, void* out, int64_t B, int64_t C, int ndim,
                      const int64_t* image, const int64_t* shape, const void* const* tw, float scale, const void* add,
                      float add_scale, void* stream) {
  clear_error();
  Axes a;
  int st = line_axes(B, C, ndim, image, shape, tw, a, "line_to_image");
  if (st || B == 0) return st;
  PGB_REQUIRE(grid && work && out && (ndim == 2 || work2), PGB_ERR_INVALID, "line_to_image: null pointer");
  cudaStream_t s = as_stream(stream);
  float2 *U = static_cast<float2*>(work), *V = static_cast<float2*>(grid);
  if (ndim == 3) {
    float2* W = static_cast<float2*>(work2);
    st = line_cols(W, V, B * C, static_cast<int>(a.n[0]), static_cast<int>(a.g12), static_cast<int>(a.g[0]), true, a.tw[0],
                   s);
    V = W;
  }
  if (st == PGB_OK) st = middle_pass(a, U, V, B * C, true, s);
  if (st == PGB_OK)
    st = out_pass(a, U, static_cast<const float2*>(smaps), static_cast<float2*>(out), B, C, scale,
                  static_cast<const float2*>(add), add_scale, s);
  PGB_REQUIRE(st != PGB_ERR_UNSUPPORTED, st, "line_to_image: a length is not built");
  return st;
}

int pgb_toep3d(const void* x, const void* smaps, const float* psf, void* work, void* work2, void* out, int64_t B, int64_t C,
               const int64_t* image, const int64_t* shape, const void* const* tw, const void* add, float add_scale,
               void* stream) {
  clear_error();
  Axes a;
  int st = line_axes(B, C, 3, image, shape, tw, a, "toep3d");
  if (st || B == 0) return st;
  PGB_REQUIRE(x && psf && work && work2 && out, PGB_ERR_INVALID, "toep3d: null pointer");
  cudaStream_t s = as_stream(stream);
  const float2* S = static_cast<const float2*>(smaps);
  float2 *U = static_cast<float2*>(work), *V = static_cast<float2*>(work2);
  st = rows_pass(a, static_cast<const float2*>(x), S, U, B, C, s);
  if (st == PGB_OK) st = middle_pass(a, U, V, B * C, false, s);
  if (st == PGB_OK)  // along z the image may lie anywhere: at the origin, as the column pass has it
    st = toep_cols(V, psf, B * C, static_cast<int>(a.n[0]), static_cast<int>(a.g12), static_cast<int>(a.g[0]), a.tw[0], s);
  if (st == PGB_OK) st = middle_pass(a, U, V, B * C, true, s);
  if (st == PGB_OK)
    st = out_pass(a, U, S, static_cast<float2*>(out), B, C, 1.f, static_cast<const float2*>(add), add_scale, s);
  PGB_REQUIRE(st != PGB_ERR_UNSUPPORTED, st, "toep3d: a length is not built");
  return st;
}

}  // extern "C"
