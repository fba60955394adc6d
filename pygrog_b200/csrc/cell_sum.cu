// cell_sum.cu -- sparse k-space to grid, cell by cell.
//
//   u[b, c, cell]    = sum over the cell's replicas of w_r y[b, c, r]
//   u[b, k, c, cell] = sum over the cell's replicas of w_r B[k, t_r] y[b, c, r]
//
// Reference: operator/_sparse_fft.py:574-621 (per-coil scatter_add on the
// grid, csrc/torch/sparse_ops.cpp:233-300), gadgets/_subspace.py:311-400 (one
// scatter per coil and component).
//
// Each cell gathers its replicas (lists built once per plan) instead of each
// replica adding to its cell: no atomics, every cell of the grid written
// once, empty ones included (no clearing pass), and the same sum in the same
// order in every run.  Bound: the replicas' sectors from HBM once and the grid
// written once.  A sample's replicas share one or two sectors and go to
// neighbouring cells, so a block takes a brick of cells (16 along x: 128-byte
// stores), in which those sectors meet again in L1.
//
// A thread owns a cell and sums lists of up to kLight replicas.  Longer ones
// (the centre of a radial or spiral trajectory holds thousands in a cell) are
// cut into segments of kSegment for a warp each; those of one segment are
// written at once, the partial sums of the others by a second kernel in list
// order.  With the long lists left to their brick's block, that block alone
// took 4.6 ms of a 192^3 radial scan and 0.125 ms of a 320^2 spiral.
#include "common.cuh"

namespace pgb {

constexpr int kCellThreads = 256;  // cells of a brick
constexpr int kLight = 8;
constexpr int kSegment = 256;

struct CellGrid {
  int g[3];   // extents z, y, x
  int b[3];   // brick
  int nb[3];  // bricks
};

// NK components at once (SUB; otherwise the weight alone), CB coils, the loads
// of NU replicas in flight.  Measured (16 coils, 640 x 640, 295 k replicas /
// 12 coils, 192^3, 7.7 M of 30.7 M replicas, us): CB NU kLight 4 2 8:
// 33.8 / 1137; 4 1 16: 46.7 / 1252; 4 4 16: 40.1 / 1134; 6 2 8: 33.9 / 1205;
// 4 4 4: 42.5 / 1530; atomics per replica after a clearing pass: 85 / 3240.
// NB bricks a block, their ranges loaded together: where most cells are empty a
// block is little more than that latency (153^3, 2 cells of 100 with a replica,
// 4 / 8 / 16 coils: NB 1 61 / 106 / 206 us, 2 55 / 93 / 165, 4 56 / 94 / 169;
// clearing the grid and skipping the empty cells 60 / 101 / 181; 128^3, a
// replica a cell, 8 coils: 183, 187, 202).
template <int NK, int CB, int NU, bool SUB, int NB>
__global__ void __launch_bounds__(kCellThreads)
    cell_sum_kernel(const float2* __restrict__ y, const uint32_t* __restrict__ start, const uint32_t* __restrict__ src,
                    const float* __restrict__ w, const int32_t* __restrict__ tix, const float2* __restrict__ basis,
                    int T, float2* __restrict__ u, CellGrid cg, int B, int C, int K, int64_t R, int64_t G,
                    const int4* __restrict__ seg, int n_seg, float2* __restrict__ part) {
  const int kch = (K + NK - 1) / NK;
  const int c0 = (blockIdx.y / kch) * CB, k0 = (blockIdx.y % kch) * NK;
  const int nc = min(CB, C - c0), nk = min(NK, K - k0);
  // acc += the replicas i, i + step, ... (NU of them, those before e): their
  // loads are issued together
  const auto add = [&](float2(&acc)[NK][CB], const float2* yb, uint32_t i, uint32_t e, uint32_t step) {
    float2 v[NU][CB];
    float ww[NU];
    int t[NU];
#pragma unroll
    for (int q = 0; q < NU; ++q) {
      const uint32_t at = i + q * step;
      uint32_t r = 0xffffffffu;
      ww[q] = 0.f;
      t[q] = 0;
      if (at < e) {
        r = src[at];
        ww[q] = w[at];
        if constexpr (SUB) t[q] = tix[at];
      }
      if constexpr (SUB) {  // no such encoding: the replica adds nothing
        if (static_cast<unsigned>(t[q]) >= static_cast<unsigned>(T)) {
          r = 0xffffffffu;
          t[q] = 0;
        }
      }
      if (r >= R) ww[q] = 0.f;  // past the end, or fewer samples than the plan has
#pragma unroll
      for (int j = 0; j < CB; ++j) v[q][j] = r < R && j < nc ? yb[j * R + r] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < NU; ++q) {
      if constexpr (SUB) {
#pragma unroll
        for (int k = 0; k < NK; ++k) {
          if (k < nk) {
            const float2 c = cscale(__ldg(basis + static_cast<int64_t>(k0 + k) * T + t[q]), ww[q]);
#pragma unroll
            for (int j = 0; j < CB; ++j) cfma(acc[k][j], c, v[q][j]);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < CB; ++j) {
          acc[0][j].x = fmaf(ww[q], v[q][j].x, acc[0][j].x);
          acc[0][j].y = fmaf(ww[q], v[q][j].y, acc[0][j].y);
        }
      }
    }
  };
  const auto store = [&](const float2(&acc)[NK][CB], int b, float2* to, int64_t n, int64_t pos) {
#pragma unroll
    for (int k = 0; k < NK; ++k)
#pragma unroll
      for (int j = 0; j < CB; ++j)
        if (k < nk && j < nc) to[((static_cast<int64_t>(b) * K + k0 + k) * C + c0 + j) * n + pos] = acc[k][j];
  };

  const int seg_blocks = (n_seg + kCellThreads / 32 - 1) / (kCellThreads / 32);
  if (blockIdx.x < seg_blocks) {  // first, as the longest: a segment of a long list per warp
    const int h = blockIdx.x * (kCellThreads / 32) + (threadIdx.x >> 5);
    if (h >= n_seg) return;
    const int4 sg = seg[h];  // {begin, end, grid position + 1 or 0: partial sum h}
    for (int b = blockIdx.z; b < B; b += gridDim.z) {
      const float2* yb = y + (static_cast<int64_t>(b) * C + c0) * R;
      float2 acc[NK][CB] = {};
      for (uint32_t i = static_cast<uint32_t>(sg.x) + (threadIdx.x & 31); i < static_cast<uint32_t>(sg.y); i += 32 * NU)
        add(acc, yb, i, static_cast<uint32_t>(sg.y), 32);
#pragma unroll
      for (int k = 0; k < NK; ++k)
#pragma unroll
        for (int j = 0; j < CB; ++j)
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            acc[k][j].x += __shfl_xor_sync(0xffffffffu, acc[k][j].x, o);
            acc[k][j].y += __shfl_xor_sync(0xffffffffu, acc[k][j].y, o);
          }
      if ((threadIdx.x & 31) == 0) {
        if (sg.z > 0) store(acc, b, u, G, sg.z - 1);
        else store(acc, b, part, n_seg, h);
      }
    }
    return;
  }
  const int bxy = cg.nb[1] * cg.nb[2], bricks = bxy * cg.nb[0];
  const int b0 = (blockIdx.x - seg_blocks) * NB;
  const int lx = threadIdx.x % cg.b[2], ly = threadIdx.x / cg.b[2];
  uint32_t s[NB], e[NB];
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const uint32_t* st = start + static_cast<int64_t>(b0 + q) * kCellThreads + threadIdx.x;
    s[q] = b0 + q < bricks ? st[0] : 0;
    e[q] = b0 + q < bricks ? st[1] : 0xffffffffu;  // no brick: as a long list, left out
  }
#pragma unroll
  for (int q = 0; q < NB; ++q) {
    const int brick = b0 + q;
    const int bz = brick / bxy, by = (brick - bz * bxy) / cg.nb[2], bx = brick % cg.nb[2];
    const int z = bz * cg.b[0] + ly / cg.b[1], yy = by * cg.b[1] + ly % cg.b[1], x = bx * cg.b[2] + lx;
    if (z >= cg.g[0] || yy >= cg.g[1] || x >= cg.g[2] || e[q] - s[q] > kLight) continue;
    for (int b = blockIdx.z; b < B; b += gridDim.z) {
      const float2* yb = y + (static_cast<int64_t>(b) * C + c0) * R;
      float2 acc[NK][CB] = {};
      for (uint32_t i = s[q]; i < e[q]; i += NU) add(acc, yb, i, e[q], 1);
      store(acc, b, u, G, (static_cast<int64_t>(z) * cg.g[1] + yy) * cg.g[2] + x);
    }
  }
}

// u[plane, position] = the sum of a long cell's partial sums (cells: {position,
// first segment, segments}), a warp per cell and plane
__global__ void __launch_bounds__(256) cell_merge_kernel(const float2* __restrict__ part, int n_seg,
                                                         const int4* __restrict__ cells, int n_cells,
                                                         float2* __restrict__ u, int64_t planes, int64_t G) {
  const int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (i >= planes * n_cells) return;
  const int64_t p = i / n_cells;
  const int4 c = cells[i - p * n_cells];
  float2 acc = make_float2(0.f, 0.f);
  for (int k = threadIdx.x & 31; k < c.z; k += 32) acc = cadd(acc, part[p * n_seg + c.y + k]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  if ((threadIdx.x & 31) == 0 && c.z > 0) u[p * G + c.x] = acc;
}

// Slot (brick order) of each replica's cell; the number of slots for replicas
// without a weight or a cell of the grid.
__global__ void cell_key_kernel(const int32_t* __restrict__ cell, const float* __restrict__ w, int64_t R, CellGrid g,
                                int32_t slots, int32_t* __restrict__ key) {
  const int64_t G = static_cast<int64_t>(g.g[0]) * g.g[1] * g.g[2];
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < R;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int c = cell[i];
    int k = slots;
    if (c >= 0 && c < G && w[i] != 0.f) {
      const int yz = c / g.g[2], x = c - yz * g.g[2], z = yz / g.g[1], y = yz - z * g.g[1];
      const int brick = (z / g.b[0] * g.nb[1] + y / g.b[1]) * g.nb[2] + x / g.b[2];
      k = brick * kCellThreads + (z % g.b[0] * g.b[1] + y % g.b[1]) * g.b[2] + x % g.b[2];
    }
    key[i] = k;
  }
}

// The long lists' segments and the cells of several, in any order (a cell's
// segments together); count: {segments, cells}.
__global__ void cell_segment_kernel(const uint32_t* __restrict__ start, int32_t slots, CellGrid g,
                                    int4* __restrict__ seg, int4* __restrict__ cells, int32_t* __restrict__ count) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < slots; s += gridDim.x * blockDim.x) {
    const int lo = static_cast<int>(start[s]), n = static_cast<int>(start[s + 1]) - lo;
    if (n <= kLight) continue;
    const int brick = s / kCellThreads, l = s % kCellThreads, bxy = g.nb[1] * g.nb[2];
    const int z = brick / bxy * g.b[0] + l / (g.b[1] * g.b[2]);
    const int y = brick / g.nb[2] % g.nb[1] * g.b[1] + l / g.b[2] % g.b[1];
    const int pos = (z * g.g[1] + y) * g.g[2] + brick % g.nb[2] * g.b[2] + l % g.b[2];
    const int cuts = (n + kSegment - 1) / kSegment;
    const int at = atomicAdd(count, cuts);
    for (int k = 0; k < cuts; ++k)
      seg[at + k] = make_int4(lo + k * kSegment, lo + min(n, (k + 1) * kSegment), cuts == 1 ? pos + 1 : 0, 0);
    if (cuts > 1) cells[atomicAdd(count + 1, 1)] = make_int4(pos, at, cuts, 0);
  }
}

static int cell_grid(int ndim, const int64_t* shape, CellGrid& g) {
  PGB_REQUIRE((ndim == 2 || ndim == 3) && shape != nullptr, PGB_ERR_INVALID, "cell_sum: ndim must be 2 or 3");
  const int b3[3] = {4, 4, 16}, b2[3] = {1, 16, 16};
  for (int d = 0; d < 3; ++d) {
    const int64_t n = ndim == 3 ? shape[d] : d == 0 ? 1 : shape[d - 1];
    PGB_REQUIRE(n >= 1 && n < (1 << 30), PGB_ERR_INVALID, "cell_sum: invalid grid extent");
    g.g[d] = static_cast<int>(n);
    g.b[d] = ndim == 3 ? b3[d] : b2[d];
    g.nb[d] = (g.g[d] + g.b[d] - 1) / g.b[d];
  }
  return PGB_OK;
}

}  // namespace pgb

using namespace pgb;

extern "C" {

int64_t pgb_cell_slots(int ndim, const int64_t* grid_shape) {
  CellGrid g;
  if (cell_grid(ndim, grid_shape, g)) return -1;
  return static_cast<int64_t>(g.nb[0]) * g.nb[1] * g.nb[2] * kCellThreads;
}

int pgb_cell_keys(const int32_t* cell, const float* w, int64_t R, int ndim, const int64_t* grid_shape, int32_t* key,
                  void* stream) {
  clear_error();
  CellGrid g;
  const int st = cell_grid(ndim, grid_shape, g);
  if (st) return st;
  const int64_t slots = pgb_cell_slots(ndim, grid_shape);
  PGB_REQUIRE(R >= 0 && slots < (int64_t(1) << 31), PGB_ERR_RANGE, "cell_keys: sizes out of range");
  if (R == 0) return PGB_OK;
  PGB_REQUIRE(cell && w && key, PGB_ERR_INVALID, "cell_keys: null pointer");
  cell_key_kernel<<<grid_for(R, 256), 256, 0, as_stream(stream)>>>(cell, w, R, g, static_cast<int32_t>(slots), key);
  PGB_LAUNCH_CHECK("cell_keys");
  return PGB_OK;
}

void pgb_cell_bounds(int64_t n, int64_t* out) {
  out[0] = n / (kLight + 1) + n / kSegment + 1;
  out[1] = n / (kSegment + 1) + 1;
}

int pgb_cell_segments(const uint32_t* start, int ndim, const int64_t* grid_shape, void* seg, void* cells, int32_t* count,
                      void* stream) {
  clear_error();
  CellGrid g;
  const int st = cell_grid(ndim, grid_shape, g);
  if (st) return st;
  const int64_t slots = pgb_cell_slots(ndim, grid_shape);
  PGB_REQUIRE(slots < (int64_t(1) << 31), PGB_ERR_RANGE, "cell_segments: sizes out of range");
  PGB_REQUIRE(start && seg && cells && count, PGB_ERR_INVALID, "cell_segments: null pointer");
  cell_segment_kernel<<<grid_for(slots, 256), 256, 0, as_stream(stream)>>>(
      start, static_cast<int32_t>(slots), g, static_cast<int4*>(seg), static_cast<int4*>(cells), count);
  PGB_LAUNCH_CHECK("cell_segments");
  return PGB_OK;
}

int pgb_cell_sum(const void* y, const uint32_t* start, const uint32_t* src, const float* w, const int32_t* tix,
                 const void* basis, int64_t T, void* u, int64_t B, int64_t C, int64_t K, int64_t R, int ndim,
                 const int64_t* grid_shape, const void* seg, int64_t n_seg, const void* cells, int64_t n_cells,
                 void* part, void* stream) {
  clear_error();
  CellGrid g;
  const int st = cell_grid(ndim, grid_shape, g);
  if (st) return st;
  PGB_REQUIRE(B >= 0 && C >= 0 && K >= 1 && K <= 32 && R >= 0 && T >= 0 && (basis != nullptr ? T >= 1 : K == 1), PGB_ERR_INVALID,
              "cell_sum: invalid sizes (K must be 1..32, T at least 1)");
  if (B == 0 || C == 0) return PGB_OK;
  PGB_REQUIRE(u && start && (y || R == 0) && (!basis || tix), PGB_ERR_INVALID, "cell_sum: null pointer");
  const int64_t G = static_cast<int64_t>(g.g[0]) * g.g[1] * g.g[2];
  const int64_t bricks = static_cast<int64_t>(g.nb[0]) * g.nb[1] * g.nb[2];
  PGB_REQUIRE(n_seg >= 0 && n_cells >= 0 && (n_seg == 0 || seg) && (n_cells == 0 || (cells && part)), PGB_ERR_INVALID,
              "cell_sum: invalid segments");
  const int64_t nx = bricks + (n_seg + kCellThreads / 32 - 1) / (kCellThreads / 32);
  PGB_REQUIRE(n_seg < (int64_t(1) << 31) && n_cells < (int64_t(1) << 31) && nx < (int64_t(1) << 31) && C < (1 << 24) && B < (int64_t(1) << 31), PGB_ERR_RANGE,
              "cell_sum: grid too large");
  const unsigned zb = static_cast<unsigned>(B < 65535 ? B : 65535);
  cudaStream_t s = as_stream(stream);
  if (basis) {
    constexpr int NK = 4, CB = 2, NU = 1;
    const int64_t ny = (C + CB - 1) / CB * ((K + NK - 1) / NK);
    PGB_REQUIRE(ny <= 65535, PGB_ERR_RANGE, "cell_sum: too many coils");
    cell_sum_kernel<NK, CB, NU, true, 1><<<dim3(static_cast<unsigned>(nx), static_cast<unsigned>(ny), zb), kCellThreads, 0, s>>>(
        static_cast<const float2*>(y), start, src, w, tix, static_cast<const float2*>(basis), static_cast<int>(T),
        static_cast<float2*>(u), g, static_cast<int>(B), static_cast<int>(C), static_cast<int>(K), R, G,
        static_cast<const int4*>(seg), static_cast<int>(n_seg), static_cast<float2*>(part));
  } else {
    constexpr int CB = 4, NU = 2;
    const int64_t ny = (C + CB - 1) / CB;
    PGB_REQUIRE(ny <= 65535, PGB_ERR_RANGE, "cell_sum: too many coils");
    // fewer replicas than cells in 3-D: two bricks a block (the comment at the kernel)
    const int nb = ndim == 3 && R < G ? 2 : 1;
    auto k = nb == 2 ? cell_sum_kernel<1, CB, NU, false, 2> : cell_sum_kernel<1, CB, NU, false, 1>;
    const int64_t blocks = nx - bricks + (bricks + nb - 1) / nb;
    k<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(ny), zb), kCellThreads, 0, s>>>(
        static_cast<const float2*>(y), start, src, w, nullptr, nullptr, 0, static_cast<float2*>(u), g,
        static_cast<int>(B), static_cast<int>(C), 1, R, G, static_cast<const int4*>(seg), static_cast<int>(n_seg),
        static_cast<float2*>(part));
  }
  PGB_LAUNCH_CHECK("cell_sum");
  if (n_cells > 0) {
    const int64_t planes = B * K * C, blocks = (planes * n_cells + 7) / 8;
    PGB_REQUIRE(blocks < (int64_t(1) << 31), PGB_ERR_RANGE, "cell_sum: too many long cells");
    cell_merge_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(
        static_cast<const float2*>(part), static_cast<int>(n_seg), static_cast<const int4*>(cells),
        static_cast<int>(n_cells), static_cast<float2*>(u), planes, G);
    PGB_LAUNCH_CHECK("cell_sum(merge)");
  }
  return PGB_OK;
}

}  // extern "C"
