// grog_expand.cu -- replica expansion with the replicas of a chunk of samples
// taken in the order of their shift operators.
//
//   out[b, co, n*kw + j] = T[idx[n*kw + j]] @ data[b, :, n]
//
// Reference: calib/_grog.py:668-695 (_sparse_full_single: replicate,
// ext.grog_interpolate, copy back), csrc/torch/grog_interp.cpp:39-73.
//
// In sample order (grog_expand_kernel, grog_fused.cu) every replica fetches
// its own C x C operator: 2 KB at 16 coils, 604 MB from L2 for 295 k replicas
// of 50 MB data.  Here a block holds a chunk of samples in shared memory, a
// lane owns a replica, and the lanes of a warp are neighbours in the chunk's
// order by operator (made once per table): most of a warp's loads of operator
// elements are of one address, or a few.  Results of up to 8 coils at a time
// are put back into sample order in shared memory and written in rows.
//
// With one replica a sample, sample n's values may lie anywhere (`src`): the
// gridding of a plan's valid replicas is this kernel and the cell sums
// (cell_sum.cu), its adjoint this kernel on the cells with the transposed
// operators and a sum over each sample's replicas.
//
// The bound is then the FP32 multiply-add rate (4 C^2 a replica) and the
// operator loads, one wavefront per distinct operator of a warp and 16 bytes.
// The expansion's sum over the input coils runs in the same order as in sample
// order: the same bits.
#include "common.cuh"

namespace pgb {

constexpr int kExpThreads = 256;

// 32 aligned bytes of read-only data in one load (sm_100): lanes with operators
// of their own cost a wavefront each per load, so half the loads are half the
// time where operators are hardly shared (10,201 of 8 coils 45.9 -> 39.3 us; 32
// coils 296 -> 262, 24 coils 234 -> 205).
__device__ __forceinline__ void load_sector(const float2* p, float2 (&t)[4]) {
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(t[0].x), "=f"(t[0].y), "=f"(t[1].x), "=f"(t[1].y), "=f"(t[2].x), "=f"(t[2].y), "=f"(t[3].x), "=f"(t[3].y)
      : "l"(p));
}

// One row of an operator times x, in PART partial sums over the input coils.  One:
// the bits of the sample order.  Two: the brick kernels' sums, for the factors.
// Four, for the adjoint of a whole table: shorter chains of FP32 roundings, which
// keep degrid's error at the brick kernels' (2-D, up to 10 coils, ratio of the
// errors against FP64 0.97 on average with four, 1.07 with one).
template <int C, int PART>
__device__ __forceinline__ float2 row_dot(const float2* __restrict__ T, const float2 (&x)[C]) {
  float2 y[PART] = {};
  if constexpr (C % 4 == 0) {
#pragma unroll
    for (int q = 0; q < C / 4; ++q) {
      float2 t[4];
      load_sector(T + 4 * q, t);
#pragma unroll
      for (int j = 0; j < 4; ++j) cfma(y[j % PART], t[j], x[4 * q + j]);
    }
  } else if constexpr (C % 2 == 0) {
#pragma unroll
    for (int q = 0; q < C / 2; ++q) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(T) + q);
      cfma(y[2 * q % PART], make_float2(t.x, t.y), x[2 * q]);
      cfma(y[(2 * q + 1) % PART], make_float2(t.z, t.w), x[2 * q + 1]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < C; ++c) cfma(y[c % PART], __ldg(T + c), x[c]);
  }
  if constexpr (PART == 4) return cadd(cadd(y[0], y[1]), cadd(y[2], y[3]));
  else if constexpr (PART == 2) return cadd(y[0], y[1]);
  else return y[0];
}

// The operators of a table, or (FACT) of two factors, table[e / n] applied first
// and second[e % n] to its result, or the other way round (swap): in turn, where
// the brick kernels do so, since the whole table of smooth coils' factors rounds
// away what they keep (errors up to 3.6 times theirs).  Twice the products, but
// on few operators: 33 k replicas of 8 coils (10,201 operators of 2 x 101
// factors) 26 / 22 us for grid / degrid against 24 / 19 with the whole table,
// 1.2 M of 11 coils in 3-D 400 / 445 against 572 / 643, of 12 coils 481 / 540
// against 444 / 541.
struct ShiftTable {
  const float2* table;
  const float2* second;
  int K, n, swap;
};

template <int C, int PART, bool FACT>
__global__ void __launch_bounds__(kExpThreads, 2)
    grog_expand_sorted_kernel(const float2* __restrict__ data, int64_t N, const int32_t* __restrict__ src,
                              int64_t stride, int kw, const uint32_t* __restrict__ order,
                              const int32_t* __restrict__ ent, ShiftTable tb, float2* __restrict__ out, int NS, int CG) {
  extern __shared__ float2 smem[];
  float2* xs = smem;           // (C, NS) samples
  float2* stage = smem + C * NS;  // (CG, NS * kw) results in sample order
  const int SR = NS * kw;
  const int64_t n0 = static_cast<int64_t>(blockIdx.x) * NS;
  const int ns = static_cast<int>(N - n0 < NS ? N - n0 : NS), nrep = ns * kw;
  const int64_t base = n0 * kw;
  const float2* dat = data + static_cast<int64_t>(blockIdx.y) * C * stride;
  float2* o = out + static_cast<int64_t>(blockIdx.y) * C * N * kw + base;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c = warp; c < C; c += kExpThreads / 32)
    for (int i = lane; i < ns; i += 32) {
      const int64_t at = src ? src[n0 + i] : n0 + i;
      xs[c * NS + i] = at >= 0 && at < stride ? dat[c * stride + at] : make_float2(0.f, 0.f);
    }
  __syncthreads();
  if constexpr (FACT) {  // one replica a sample: its first product takes the sample's place
    for (int i = threadIdx.x; i < nrep; i += kExpThreads) {
      const int l = order[base + i] & 0xffffu, e = ent[base + i];
      float2 x[C];
#pragma unroll
      for (int c = 0; c < C; ++c) x[c] = xs[c * NS + l];
      const int at = e >= 0 && e < tb.K ? (tb.swap ? e % tb.n : e / tb.n) : 0;
      const float2* T = (tb.swap ? tb.second : tb.table) + static_cast<int64_t>(at) * C * C;
#pragma unroll 4
      for (int c = 0; c < C; ++c, T += C) xs[c * NS + l] = row_dot<C, PART>(T, x);
    }
  }
  for (int g0 = 0; g0 < C; g0 += CG) {
    const int ng = min(CG, C - g0);
    for (int i = threadIdx.x; i < nrep; i += kExpThreads) {
      const uint32_t od = order[base + i];  // place in the chunk, sample in the chunk << 16
      const int l = od & 0xffffu, n = od >> 16, e = ent[base + i];
      float2 x[C];
#pragma unroll
      for (int c = 0; c < C; ++c) x[c] = xs[c * NS + n];
      const bool ok = e >= 0 && e < tb.K;
      int at = ok ? e : 0;
      if constexpr (FACT) at = tb.swap ? at / tb.n : at % tb.n;
      const float2* T = (FACT && !tb.swap ? tb.second : tb.table) + (static_cast<int64_t>(at) * C + g0) * C;
#pragma unroll 4  // the operator rows of four coils in flight
      for (int co = 0; co < ng; ++co, T += C) {
        const float2 y = row_dot<C, PART>(T, x);  // in every lane: a branch here would keep the rows' loads apart
        stage[co * SR + l] = ok ? y : make_float2(0.f, 0.f);
      }
    }
    __syncthreads();
    for (int co = 0; co < ng; ++co)
      for (int i = threadIdx.x; i < nrep; i += kExpThreads)
        o[static_cast<int64_t>(g0 + co) * N * kw + i] = stage[co * SR + i];
    __syncthreads();
  }
}

// The order of one chunk per block: bitonic sort of (table index, replica) in
// shared memory; runs += the chunk's runs of one operator.
__global__ void __launch_bounds__(512) grog_expand_order_kernel(const int64_t* __restrict__ idx, int64_t R, int kw, int SR,
                                                                int P, int64_t K, uint32_t* __restrict__ order,
                                                                int32_t* __restrict__ ent, int32_t* __restrict__ runs) {
  extern __shared__ unsigned long long keys[];  // (P), P a power of two
  const int64_t base = static_cast<int64_t>(blockIdx.x) * SR;
  const int n = static_cast<int>(R - base < SR ? R - base : SR);
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    unsigned long long k = ~0ull;
    if (i < n) {
      const int64_t e = idx[base + i];
      k = static_cast<unsigned long long>((e < 0 ? -1 : e >= K ? K : e) + 1) << 16 | i;
    }
    keys[i] = k;
  }
  for (int size = 2; size <= P; size *= 2)
    for (int d = size / 2; d > 0; d /= 2) {
      __syncthreads();
      for (int i = threadIdx.x; i < P / 2; i += blockDim.x) {
        const int a = 2 * i - (i & (d - 1)), b = a + d;
        const unsigned long long x = keys[a], y = keys[b];
        if ((x > y) == ((a & size) == 0)) keys[a] = y, keys[b] = x;
      }
    }
  __syncthreads();
  int mine = 0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long k = keys[i];
    const uint32_t l = static_cast<uint32_t>(k & 0xffffu);
    order[base + i] = l | (l / kw) << 16;
    ent[base + i] = static_cast<int32_t>(static_cast<int64_t>(k >> 16) - 1);
    mine += i == 0 || (keys[i - 1] >> 16) != (k >> 16);
  }
  for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(0xffffffffu, mine, o);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(runs, mine);
}

// out[bc, n] = sum over the sample's replicas v of w_v y[bc, v]  (v ascending
// by sample, ptr: each sample's range)
__global__ void sample_sum_kernel(const float2* __restrict__ y, const int32_t* __restrict__ ptr,
                                  const float* __restrict__ w, float2* __restrict__ out, int64_t N, int64_t V,
                                  int64_t BC) {
  const int64_t n = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const int lo = ptr[n], hi = ptr[n + 1];
  for (int64_t bc = blockIdx.y; bc < BC; bc += gridDim.y) {
    float2 acc = make_float2(0.f, 0.f);
    for (int v = lo; v < hi; ++v) {
      const float2 a = y[bc * V + v];
      acc.x = fmaf(w[v], a.x, acc.x);
      acc.y = fmaf(w[v], a.y, acc.y);
    }
    out[bc * N + n] = acc;
  }
}

// Samples a chunk and coils a pass: two blocks' shared memory on an SM, and
// whole waves of blocks.  (295 k replicas of 16 coils / 820 k of 8 / 420 k of
// 32, with 16-byte loads: 46.8 / 46.0 / 291 us; three blocks of 72 KB 49.3 / 46.0
// / 379, four coils a pass 63.9 / 64.0 / 383: a smaller chunk shares its operators
// less.)
static void expand_shape(int64_t N, int64_t C, int64_t kw, int& ns, int& cg) {
  for (cg = C < 8 ? static_cast<int>(C) : 8; cg >= 1; cg /= 2) {
    const int64_t per = 8 * (C + cg * kw);
    int64_t n = 110 * 1024 / per;
    if (n > 1024) n = 1024;
    if (n * kw > 65536) n = 65536 / kw;
    if (n >= 32) {
      const int64_t wave = 2 * kNumSMs, waves = (N + n * wave - 1) / (n * wave);
      const int64_t even = waves > 0 ? (N + waves * wave - 1) / (waves * wave) : n;
      ns = static_cast<int>(even < 32 ? 32 : even);
      return;
    }
  }
  ns = 0;
  cg = 1;
}

}  // namespace pgb

using namespace pgb;

extern "C" {

int pgb_grog_expand_chunk(int64_t N, int64_t C, int64_t kw) {
  int ns = 0, cg = 1;
  if (N >= 0 && C >= 1 && C <= 32 && kw >= 1 && kw <= 2048) expand_shape(N, C, kw, ns, cg);
  return ns;
}

int pgb_grog_expand_order(const int64_t* idx, int64_t N, int kw, int64_t K, int64_t C, uint32_t* order, int32_t* ent,
                          int32_t* runs, void* stream) {
  clear_error();
  const int ns = pgb_grog_expand_chunk(N, C, kw);
  PGB_REQUIRE(ns > 0, PGB_ERR_UNSUPPORTED, "grog_expand_order: kw=%d too large for the staging tile", kw);
  PGB_REQUIRE(K >= 1 && K < (int64_t(1) << 31) - 1, PGB_ERR_RANGE, "grog_expand_order: table too large");
  if (N == 0) return PGB_OK;
  PGB_REQUIRE(idx && order && ent && runs, PGB_ERR_INVALID, "grog_expand_order: null pointer");
  const int SR = ns * kw;
  int P = 2;
  while (P < SR) P *= 2;
  const size_t smem = sizeof(unsigned long long) * P;
  PGB_REQUIRE(smem <= 227 * 1024, PGB_ERR_UNSUPPORTED, "grog_expand_order: chunk too large");
  const int64_t blocks = (N + ns - 1) / ns;
  PGB_REQUIRE(blocks < (int64_t(1) << 31), PGB_ERR_RANGE, "grog_expand_order: too many samples");
  allow_smem<grog_expand_order_kernel>(227 * 1024);
  grog_expand_order_kernel<<<static_cast<unsigned>(blocks), 512, smem, as_stream(stream)>>>(idx, N * kw, kw, SR, P, K,
                                                                                            order, ent, runs);
  PGB_LAUNCH_CHECK("grog_expand_order");
  return PGB_OK;
}

int pgb_sample_sum(const void* y, const int32_t* ptr, const float* w, void* out, int64_t N, int64_t V, int64_t BC,
                   void* stream) {
  clear_error();
  PGB_REQUIRE(N >= 0 && V >= 0 && BC >= 0, PGB_ERR_INVALID, "sample_sum: negative size");
  if (N == 0 || BC == 0) return PGB_OK;
  PGB_REQUIRE(ptr && out && (V == 0 || (y && w)), PGB_ERR_INVALID, "sample_sum: null pointer");
  const int64_t blocks = (N + 255) / 256;
  PGB_REQUIRE(blocks < (int64_t(1) << 31), PGB_ERR_RANGE, "sample_sum: too many samples");
  sample_sum_kernel<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(BC < 65535 ? BC : 65535)), 256, 0,
                      as_stream(stream)>>>(static_cast<const float2*>(y), ptr, w, static_cast<float2*>(out), N, V, BC);
  PGB_LAUNCH_CHECK("sample_sum");
  return PGB_OK;
}

static int expand_sorted(const void* data, int64_t N, const int32_t* src, int64_t stride, int kw, const uint32_t* order,
                         const int32_t* ent, const void* table, int64_t K, const void* second, int64_t n,
                         int adjoint, int64_t C, int64_t B, void* out, void* stream, const char* who) {
  clear_error();
  if (!src) stride = N;
  PGB_REQUIRE(stride >= 0, PGB_ERR_INVALID, "%s: invalid sizes", who);
  const int cmax = second ? 16 : 32;
  PGB_REQUIRE(C >= 1 && C <= cmax, PGB_ERR_UNSUPPORTED, "%s: ncoils must be 1..%d, got %lld", who, cmax, (long long)C);
  PGB_REQUIRE(N >= 0 && B >= 0 && kw >= 1 && K >= 1 && (!second || (n >= 1 && K % n == 0 && K < (int64_t(1) << 31))),
              PGB_ERR_INVALID, "%s: invalid sizes", who);
  if (N == 0 || B == 0) return PGB_OK;
  PGB_REQUIRE(data && order && ent && table && out, PGB_ERR_INVALID, "%s: null pointer", who);
  PGB_REQUIRE(B <= 65535, PGB_ERR_RANGE, "%s: batch must be <= 65535", who);
  const int align = C % 4 == 0 ? 32 : C % 2 == 0 ? 16 : 8;  // of the operator loads
  PGB_REQUIRE(reinterpret_cast<uintptr_t>(table) % align == 0 && reinterpret_cast<uintptr_t>(second) % align == 0,
              PGB_ERR_INVALID, "%s: table not %d-byte aligned", who, align);
  int ns, cg;
  ns = pgb_grog_expand_chunk(N, C, kw);
  if (ns > 0) expand_shape(N, C, kw, ns, cg);
  PGB_REQUIRE(ns > 0, PGB_ERR_UNSUPPORTED, "%s: kw=%d too large for the staging tile", who, kw);
  const size_t smem = sizeof(float2) * ns * (C + static_cast<int64_t>(cg) * kw);
  const int64_t blocks = (N + ns - 1) / ns;
  PGB_REQUIRE(blocks < (int64_t(1) << 31), PGB_ERR_RANGE, "%s: too many samples", who);
  const dim3 grd(static_cast<unsigned>(blocks), static_cast<unsigned>(B));
  const ShiftTable tb{static_cast<const float2*>(table), static_cast<const float2*>(second),
                      static_cast<int>(K < INT32_MAX ? K : INT32_MAX), static_cast<int>(n), adjoint};
  cudaStream_t s = as_stream(stream);
  const auto go = [&](auto launch) {
    launch(static_cast<const float2*>(data), N, src, stride, kw, order, ent, tb, static_cast<float2*>(out), ns, cg);
  };
#define Y(CC, P, F)                                                              \
  {                                                                              \
    allow_smem<grog_expand_sorted_kernel<CC, P, F>>(227 * 1024);                 \
    go([&](auto... a) { grog_expand_sorted_kernel<CC, P, F><<<grd, kExpThreads, smem, s>>>(a...); }); \
  }
  if (second) {
    switch (C) {
#define X(CC) \
  case CC:    \
    Y(CC, 2, true) break;
      X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)
#undef X
    }
  } else {
    switch (C) {
#define X(CC)                            \
  case CC:                               \
    if (adjoint) Y(CC, 4, false)         \
    else Y(CC, 1, false) break;
      X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20)
      X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31) X(32)
#undef X
    }
  }
#undef Y
  PGB_LAUNCH_CHECK(who);
  return PGB_OK;
}

int pgb_grog_expand_sorted(const void* data, int64_t N, const int32_t* src, int64_t stride, int kw,
                           const uint32_t* order, const int32_t* ent, const void* table, int64_t K, int64_t C, int64_t B,
                           void* out, void* stream) {
  return expand_sorted(data, N, src, stride, kw, order, ent, table, K, nullptr, 0, 0, C, B, out, stream,
                       "grog_expand_sorted");
}

int pgb_grog_shift(const void* data, int64_t M, const int32_t* src, int64_t V, const uint32_t* order, const int32_t* ent,
                   const void* table, int64_t K, const void* second, int64_t n, int adjoint, int64_t C, int64_t B,
                   void* out, void* stream) {
  clear_error();
  PGB_REQUIRE(src || V == 0, PGB_ERR_INVALID, "grog_shift: null pointer");
  return expand_sorted(data, V, src, M, 1, order, ent, table, K, second, n, adjoint, C, B, out, stream,
                       "grog_shift");
}

}  // extern "C"
