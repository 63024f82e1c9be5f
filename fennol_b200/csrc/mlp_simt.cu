// Species-indexed MLP in float32 on CUDA cores (the plain FP32 form).
//
// Replaces SpeciesIndexNet / FullyConnectedNet (src/fennol/models/misc/nets.py:
// 13-102, 301-426) and the transpose jax.grad builds for the input gradient.
// Rows are grouped by species in 128-row tiles; each tile multiplies by the
// weights of its species.  One launch per layer for a batch of models, with
// fused epilogues:
//   forward  : H = celu(A W + b)
//   head     : e = H3 . w4 + b4 ;  G3 = w4 * celu'(H3)
//   backward : G = (G' W^T) * celu'(H)   (celu' recovered from H itself:
//              1 for H > 0, H/alpha + 1 otherwise)
//   input    : dX (+)= (G1 W1^T) / n_models, model after model
// Every element is one chain of FMAs in increasing k, whatever the tiling.
#include <algorithm>

#include "mlp_common.cuh"

using namespace fnl;

namespace {

// SGEMM tile: 128 x 64 outputs per 128 threads, 8 x 8 each.  Bound by the FP32
// pipe: the products are packed two to an instruction (fma.rn.f32x2, each half
// rounded as a scalar FMA), which takes the pipe as long as two scalar FMAs but
// leaves every other issue slot to the loads and address arithmetic.  64
// columns divide the padded widths (192, 256) without a remainder, and small
// blocks keep several per SM.  6,591 atoms x 8 models (water): layer 2 takes
// 146 us, 35 TFLOP/s, FMA pipe 62 % busy; the whole form 3.2 ms with scalar
// FMAs, 4-byte loads and every AEV column, 0.75 ms now.
constexpr int BM = 128, BN = 64, BK = 16;
constexpr int kThreads = 128;
constexpr int kMaxGroups = 256;

enum Epi { EPI_BIAS_CELU = 0, EPI_DCELU = 1, EPI_SCALE_ACC = 2, EPI_STORE = 3 };

struct GemmArgs {
  const float* A;
  size_t a_model;      // elements between models (0: the same A)
  int lda;
  const float* W;      // group-strided weights
  size_t w_group;      // elements between groups
  int ldw;             // row stride of W
  const float* bias;   // group-strided bias (EPI_BIAS_CELU)
  size_t b_group;
  float* C;
  size_t c_model;
  int ldc;
  const int* tile_species;
  const int* tile_row;
  int n_species;
  int model0, models;  // EPI_SCALE_ACC: the models summed in one block; else blockIdx.z is the model
  float alpha;         // celu alpha
  float scale;         // EPI_SCALE_ACC: C = (first model ? 0 : C) + scale * acc
  int vec;             // every array is 16-byte aligned: four floats per access
  int nk;              // K in steps of 16
  int nn;              // N in steps of 16
  // the 16-column groups of the AEV columns that K (first layer) or N (input
  // gradient) runs over; `all`: every one in turn
  int all;
  unsigned char group[kMaxGroups];
};

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(F2 x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x.v));
  return r;
}
__device__ __forceinline__ void fma2(F2& d, F2 a, F2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d.v) : "l"(a.v), "l"(b.v));
}

__device__ __forceinline__ float4 ld4(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ void st4(float* p, float4 v, bool vec) {
  if (vec) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    p[0] = v.x;
    p[1] = v.y;
    p[2] = v.z;
    p[3] = v.w;
  }
}

// NT = false: C = A @ W with W [K][N] (row stride ldw); K may be gathered
// NT = true : C = A @ W^T with W [N][K] (row stride ldw); N may be gathered
// RB = 2: a block has a whole 128-row tile; RB = 1: half of one (blockIdx.x = 2 tile
// + half), 4 x 8 outputs per thread.
template <bool NT, int EPI, int RB>
__global__ void __launch_bounds__(kThreads, 4) k_sgemm(const __grid_constant__ GemmArgs g) {
  pdl_wait();
  // rows padded by 4 floats: the transposed stores of a warp hit 32 banks, and
  // 16-byte loads stay aligned
  __shared__ __align__(16) float As[2][BK][64 * RB + 4];
  __shared__ __align__(16) float Bs[2][BK][BN + 4];
  const int tile = RB == 2 ? blockIdx.x : blockIdx.x >> 1;
  const int n0 = blockIdx.y * BN;
  const int row0 = g.tile_row[tile] + (RB == 2 ? 0 : 64 * (blockIdx.x & 1));
  const int species = g.tile_species[tile];
  const int tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;  // columns tx*4 and 32 + tx*4, rows ty*4 and 64 + ty*4
  const int m_first = EPI == EPI_SCALE_ACC ? 0 : blockIdx.z, m_end = EPI == EPI_SCALE_ACC ? g.models : m_first + 1;
  auto column = [&](int step) -> int { return (g.all ? step : (int)g.group[step]) * 16; };

  for (int m = m_first; m < m_end; ++m) {
    const int grp = (g.model0 + m) * g.n_species + species;
    const float* __restrict__ A = g.A + (size_t)m * g.a_model + (size_t)row0 * g.lda;
    const float* __restrict__ W = g.W + (size_t)grp * g.w_group;
    F2 acc[4 * RB][4];
#pragma unroll
    for (int a = 0; a < 4 * RB; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b] = pack2(0.f, 0.f);

    // global -> register staging: A 128 rows x 16 k and W 16 x 64 as 16-byte loads
    constexpr int kAhead = RB == 2 ? 1 : 2;  // steps that loads run ahead
    float4 ra_[kAhead][2 * RB], rb_[kAhead][2];
    auto load_tile = [&](int step, float4 (&ra)[2 * RB], float4 (&rb)[2]) {
      const int ka = NT ? step * 16 : column(step);
#pragma unroll
      for (int q = 0; q < 2 * RB; ++q)
        ra[q] = ld4(A + (size_t)((tid >> 2) + 32 * q) * g.lda + ka + (tid & 3) * 4, g.vec);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (!NT) {
          const int k = ka + (tid >> 4) + 8 * q, n = n0 + (tid & 15) * 4;
          rb[q] = n < g.nn * 16 ? ld4(W + (size_t)k * g.ldw + n, g.vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
          const int n = n0 + (tid >> 2) + 32 * q;
          const int wr = EPI >= EPI_SCALE_ACC && n < g.nn * 16 ? column(n >> 4) + (n & 15) : n;
          rb[q] = n < g.nn * 16 ? ld4(W + (size_t)wr * g.ldw + step * 16 + (tid & 3) * 4, g.vec)
                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    };
    auto store_tile = [&](int buf, const float4 (&ra)[2 * RB], const float4 (&rb)[2]) {
#pragma unroll
      for (int q = 0; q < 2 * RB; ++q) {
        const int r = (tid >> 2) + 32 * q, k = (tid & 3) * 4;
        As[buf][k][r] = ra[q].x;
        As[buf][k + 1][r] = ra[q].y;
        As[buf][k + 2][r] = ra[q].z;
        As[buf][k + 3][r] = ra[q].w;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (!NT) {
          *reinterpret_cast<float4*>(&Bs[buf][(tid >> 4) + 8 * q][(tid & 15) * 4]) = rb[q];
        } else {
          const int n = (tid >> 2) + 32 * q, k = (tid & 3) * 4;
          Bs[buf][k][n] = rb[q].x;
          Bs[buf][k + 1][n] = rb[q].y;
          Bs[buf][k + 2][n] = rb[q].z;
          Bs[buf][k + 3][n] = rb[q].w;
        }
      }
    };

    auto multiply = [&](int buf) {
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        float av[4 * RB];
        F2 bv[4];
        *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
        if (RB == 2)
          *reinterpret_cast<float4*>(av + 4 * (RB - 1)) =
              *reinterpret_cast<const float4*>(&As[buf][kk][64 * (RB - 1) + ty * 4]);
        const float4 b0 = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
        const float4 b1 = *reinterpret_cast<const float4*>(&Bs[buf][kk][32 + tx * 4]);
        bv[0] = pack2(b0.x, b0.y);
        bv[1] = pack2(b0.z, b0.w);
        bv[2] = pack2(b1.x, b1.y);
        bv[3] = pack2(b1.z, b1.w);
#pragma unroll
        for (int a = 0; a < 4 * RB; ++a) {
          const F2 aa = pack2(av[a], av[a]);
#pragma unroll
          for (int b = 0; b < 4; ++b) fma2(acc[a][b], aa, bv[b]);
        }
      }
    };
    load_tile(0, ra_[0], rb_[0]);
    store_tile(0, ra_[0], rb_[0]);
    if (kAhead == 2 && g.nk > 1) load_tile(1, ra_[kAhead - 1], rb_[kAhead - 1]);
    __syncthreads();
    for (int kt = 0; kt < g.nk; kt += kAhead) {
#pragma unroll
      for (int h = 0; h < kAhead; ++h) {  // register set h: step kt + h, then step kt + h + kAhead
        const int step = kt + h, buf = step & 1;
        if (step >= g.nk) break;
        if (step + kAhead < g.nk) load_tile(step + kAhead, ra_[h], rb_[h]);
        multiply(buf);
        if (step + 1 < g.nk) store_tile(buf ^ 1, ra_[(h + 1) % kAhead], rb_[(h + 1) % kAhead]);
        __syncthreads();
      }
    }

#pragma unroll
    for (int h = 0; h < 2; ++h) {  // columns n .. n + 3 of each half
      const int n = n0 + 32 * h + tx * 4;
      if (n >= g.nn * 16) continue;
      const int col = EPI == EPI_SCALE_ACC ? column(n >> 4) + (n & 15) : n;
      float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
      if (EPI == EPI_BIAS_CELU) bias = ld4(g.bias + (size_t)grp * g.b_group + n, g.vec);
#pragma unroll
      for (int a = 0; a < 4 * RB; ++a) {
        const int r = row0 + (a < 4 ? ty * 4 + a : 64 + ty * 4 + a - 4);
        float* c = g.C + (size_t)m * g.c_model + (size_t)r * g.ldc + col;
        const float2 v0 = unpack2(acc[a][2 * h]), v1 = unpack2(acc[a][2 * h + 1]);
        float4 o;
        if (EPI == EPI_BIAS_CELU) {
          o = make_float4(celu_f(v0.x + bias.x, g.alpha), celu_f(v0.y + bias.y, g.alpha),
                          celu_f(v1.x + bias.z, g.alpha), celu_f(v1.y + bias.w, g.alpha));
        } else if (EPI == EPI_DCELU) {
          const float4 t = ld4(c, g.vec);
          o = make_float4(v0.x * dcelu_from_h(t.x, g.alpha), v0.y * dcelu_from_h(t.y, g.alpha),
                          v1.x * dcelu_from_h(t.z, g.alpha), v1.y * dcelu_from_h(t.w, g.alpha));
        } else if (EPI == EPI_STORE) {
          o = make_float4(v0.x, v0.y, v1.x, v1.y);
        } else {
          const float4 t = g.model0 + m > 0 ? ld4(c, g.vec) : make_float4(0.f, 0.f, 0.f, 0.f);
          o = make_float4(fmaf(g.scale, v0.x, t.x), fmaf(g.scale, v0.y, t.y), fmaf(g.scale, v1.x, t.z),
                          fmaf(g.scale, v1.y, t.w));
        }
        st4(c, o, g.vec);
      }
    }
  }
}

// dX (+)= scale * (the models' input gradients), model after model; rows of a
// tile x groups of 16 columns, four columns per thread.
__global__ void __launch_bounds__(256) k_dx_sum(const __grid_constant__ GemmArgs g, const float* __restrict__ part,
                                                size_t part_model) {
  pdl_wait();
  const int row0 = g.tile_row[blockIdx.x], N = g.nn * 16;
  for (int k = blockIdx.y * 256 + threadIdx.x; k < BM * N / 4; k += 256 * gridDim.y) {
    const int r = row0 + k / (N / 4), n = k % (N / 4) * 4;
    float* c = g.C + (size_t)r * g.ldc + (g.all ? n >> 4 : (int)g.group[n >> 4]) * 16 + (n & 15);
    float4 t = g.model0 > 0 ? ld4(c, g.vec) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int m = 0; m < g.models; ++m) {
      const float4 v = ld4(part + m * part_model + (size_t)r * N + n, g.vec);
      t = make_float4(fmaf(g.scale, v.x, t.x), fmaf(g.scale, v.y, t.y), fmaf(g.scale, v.z, t.z),
                      fmaf(g.scale, v.w, t.w));
    }
    st4(c, t, g.vec);
  }
}

// Last layer (width dims[3] -> 1) and its transpose: one warp per row, the
// batch's models four at a time with every load in flight (one after the other:
// 33 us for 6,591 rows x 8 models).
__global__ void __launch_bounds__(256) k_head(float* __restrict__ H3, size_t h_model, int n3,
                                              const float* __restrict__ w4, const float* __restrict__ b4,
                                              const int* __restrict__ tile_species, const int* __restrict__ tile_row,
                                              int ntiles, int n_species, int model0, int models, float alpha,
                                              float inv_models, float* __restrict__ e_rows) {
  pdl_wait();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int tile = warp / 128;
  if (tile >= ntiles) return;
  const int r = tile_row[tile] + (warp % 128);
  float total = model0 > 0 ? e_rows[r] : 0.f;
  for (int m0 = 0; m0 < models; m0 += 4) {
    float e[4] = {0.f, 0.f, 0.f, 0.f};
    for (int n0 = 0; n0 < n3; n0 += 192) {
      float hv[4][6], wv[4][6];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (m0 + u >= models) break;
        const float* w = w4 + ((size_t)(model0 + m0 + u) * n_species + tile_species[tile]) * n3;
        const float* h = H3 + (m0 + u) * h_model + (size_t)r * n3;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          const int n = n0 + 32 * k + lane;
          hv[u][k] = n < n3 ? h[n] : 0.f;
          wv[u][k] = n < n3 ? w[n] : 0.f;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (m0 + u >= models) break;
        float* h = H3 + (m0 + u) * h_model + (size_t)r * n3;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          const int n = n0 + 32 * k + lane;
          if (n >= n3) break;
          e[u] = fmaf(hv[u][k], wv[u][k], e[u]);
          h[n] = wv[u][k] * dcelu_from_h(hv[u][k], alpha);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (m0 + u >= models) break;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e[u] += __shfl_xor_sync(0xffffffffu, e[u], o);
      e[u] += b4[(size_t)(model0 + m0 + u) * n_species + tile_species[tile]];
      total = fmaf(e[u], inv_models, total);
    }
  }
  if (lane == 0) e_rows[r] = total;
}

// Models evaluated per launch: as many as give 2,400 blocks of the narrower
// layers (three a tile), four waves of the GPU, so that a nearly empty last wave
// costs little (6,591 atoms x 8 models in two launches of 624 blocks, 1.05 waves:
// 90 us each); the activations in memory stay below those of about 100,000 rows.
constexpr int kLaunchTiles = 800;  // (tile, model) pairs per launch
int models_per_launch(int rows, int n_models) {
  return std::min(n_models, std::max(1, kLaunchTiles / std::max(rows / BM, 1)));
}

// One layer: half tiles where whole ones give the GPU too few blocks to be busy
// (kFewBlocks).  An element's FMAs come in the same order either way.
// Half tiles also load two steps ahead (128 registers hold it).  256 molecules, 1
// model, 56 tiles, whole / half tiles: 256 -> 192 41 / 31 us, 192 -> 160 37 / 28,
// their transposes 43 / 29 and 42 / 35; 1008 -> 256, 448 half blocks of which
// four SMs have one more than the others, 123 / 125.
constexpr int kFewBlocks = 148 * 4;
template <bool NT, int EPI>
int sgemm(int ntiles, int ny, int nz, const GemmArgs& a, cudaStream_t st) {
  if (ntiles * ny * nz >= kFewBlocks)
    FNL_LAUNCH_PDL((k_sgemm<NT, EPI, 2>), dim3(ntiles, ny, nz), dim3(kThreads), 0, st, a);
  else
    FNL_LAUNCH_PDL((k_sgemm<NT, EPI, 1>), dim3(2 * ntiles, ny, nz), dim3(kThreads), 0, st, a);
  return FENNOL_OK;
}

// Few columns of dX on few tiles: a block per model, into the activations that are
// no longer needed (H2), and a sum; 106 blocks that went through 8 models took 176
// us on 6,591 atoms, 848 blocks and the sum 96 us.
bool dx_by_model(int models, int ntiles, int N, const int* d) {
  return models > 1 && ntiles * ((N + BN - 1) / BN) < kFewBlocks && N <= d[2];
}

}  // namespace

// Activations of a launch: those of `rows` or of any fewer rows, which can be
// more (100 tiles go through 8 models at a time, 101 through 7).
size_t fnl_mlp_simt_workspace(int rows, const fennol_mlp_weights* w) {
  const size_t tiles = ((size_t)rows + BM - 1) / BM;
  const size_t most = std::min(tiles * w->n_models, std::max(tiles, (size_t)kLaunchTiles));
  return most * BM * (w->dims[1] + w->dims[2] + w->dims[3]) * sizeof(float);
}

int fnl_mlp_simt_launches(int rows, int ntiles, const fennol_mlp_weights* w, ColumnGroups dg, bool want_dx) {
  const int per = models_per_launch(rows, w->n_models), groups = w->dims[0] / 16;
  int wanted = 0, n = 0;
  for (int g = 0; g < groups; ++g) wanted += groups > kMaxGroups || dg.has(g);
  for (int m0 = 0; m0 < w->n_models; m0 += per) {
    n += 4;  // three layers and the head
    if (!want_dx) continue;
    n += 2;
    if (wanted > 0) n += 1 + dx_by_model(std::min(per, w->n_models - m0), ntiles, 16 * wanted, w->dims);
  }
  return n;
}

int fnl_mlp_simt(int rows, int ntiles, const int* tile_species, const int* tile_row,
                 const fennol_mlp_weights* w, const float* x, ColumnGroups xg, ColumnGroups dg, float* e_rows,
                 float* dx, void* ws, cudaStream_t st) {
  const int* d = w->dims;
  const int per = models_per_launch(rows, w->n_models);
  float* Hs[4] = {nullptr, (float*)ws, nullptr, nullptr};
  Hs[2] = Hs[1] + (size_t)per * rows * d[1];
  Hs[3] = Hs[2] + (size_t)per * rows * d[2];
  const float inv_m = 1.0f / (float)w->n_models;
  // the first layer's K steps and the input gradient's columns
  const int groups = d[0] / 16;
  auto list = [&](GemmArgs& a, const ColumnGroups& cg) -> int {
    if (groups > kMaxGroups || !cg.words) {
      a.all = 1;
      return groups;
    }
    int n = 0;
    for (int k = 0; k < groups; ++k)
      if (cg.has(k)) a.group[n++] = (unsigned char)k;
    return n;
  };
  GemmArgs base{};
  base.tile_species = tile_species;
  base.tile_row = tile_row;
  base.n_species = w->n_species;
  base.alpha = w->celu_alpha;
  base.all = 1;
  uintptr_t bits = (uintptr_t)x | (uintptr_t)dx | (uintptr_t)ws;
  for (int l = 0; l < 3; ++l) bits |= (uintptr_t)w->w32[l] | (uintptr_t)w->b32[l];
  base.vec = (bits & 15) == 0;
  for (int m0 = 0; m0 < w->n_models; m0 += per) {
    const int nm = std::min(per, w->n_models - m0);
    base.model0 = m0;
    base.models = nm;
    // forward layers 1..3
    for (int l = 0; l < 3; ++l) {
      GemmArgs a = base;
      a.A = l == 0 ? x : Hs[l];
      a.a_model = l == 0 ? 0 : (size_t)rows * d[l];
      a.lda = d[l];
      a.W = w->w32[l];
      a.w_group = (size_t)d[l] * d[l + 1];
      a.ldw = d[l + 1];
      a.bias = w->b32[l];
      a.b_group = d[l + 1];
      a.C = Hs[l + 1];
      a.c_model = (size_t)rows * d[l + 1];
      a.ldc = d[l + 1];
      a.nk = d[l] / 16;
      if (l == 0) {
        a.all = 0;
        a.nk = list(a, xg);
        if (a.nk == 0) {  // nothing can be non-zero: one step of zeros
          a.nk = 1;
          a.group[0] = 0;
        }
      }
      a.nn = d[l + 1] / 16;
      if (int err = sgemm<false, EPI_BIAS_CELU>(ntiles, (d[l + 1] + BN - 1) / BN, nm, a, st)) return err;
    }
    // head: energy + G3 (in place of H3)
    FNL_LAUNCH_PDL(k_head, dim3((ntiles * 128 * 32 + 255) / 256), dim3(256), 0, st, Hs[3], (size_t)rows * d[3], d[3],
                   w->w32[3], w->b32[3], tile_species, tile_row, ntiles, w->n_species, m0, nm, w->celu_alpha, inv_m,
                   e_rows);
    if (!dx) continue;  // energies only
    // backward layers 3..2: G_{l} = (G_{l+1} W_{l+1}^T) * celu'(H_l), in place of H_l
    for (int l = 2; l >= 1; --l) {
      GemmArgs a = base;
      a.A = Hs[l + 1];
      a.a_model = (size_t)rows * d[l + 1];
      a.lda = d[l + 1];
      a.W = w->w32[l];
      a.w_group = (size_t)d[l] * d[l + 1];
      a.ldw = d[l + 1];
      a.C = Hs[l];
      a.c_model = (size_t)rows * d[l];
      a.ldc = d[l];
      a.nk = d[l + 1] / 16;
      a.nn = d[l] / 16;
      if (int err = sgemm<true, EPI_DCELU>(ntiles, (d[l] + BN - 1) / BN, nm, a, st)) return err;
    }
    // input gradient dX (+)= G1 W1^T / n_models
    GemmArgs a = base;
    a.A = Hs[1];
    a.a_model = (size_t)rows * d[1];
    a.lda = d[1];
    a.W = w->w32[0];
    a.w_group = (size_t)d[0] * d[1];
    a.ldw = d[1];
    a.C = dx;
    a.ldc = d[0];
    a.scale = inv_m;
    a.nk = d[1] / 16;
    a.all = 0;
    a.nn = list(a, dg);
    if (a.nn == 0) continue;
    const int N = a.nn * 16;
    if (dx_by_model(nm, ntiles, N, d)) {
      GemmArgs p = a;
      p.C = Hs[2];
      p.c_model = (size_t)rows * N;
      p.ldc = N;
      if (int err = sgemm<true, EPI_STORE>(ntiles, (N + BN - 1) / BN, nm, p, st)) return err;
      FNL_LAUNCH_PDL(k_dx_sum, dim3(ntiles, (BM * N / 4 + 255) / 256), dim3(256), 0, st, a, (const float*)Hs[2], (size_t)rows * N);
      continue;
    }
    if (int err = sgemm<true, EPI_SCALE_ACC>(ntiles, (a.nn * 16 + BN - 1) / BN, 1, a, st)) return err;
  }
  return FENNOL_OK;
}
