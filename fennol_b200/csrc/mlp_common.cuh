// Shared pieces of the species-MLP kernels.
#pragma once
#include "common.cuh"

namespace fnl {

// jax.nn.celu(x, alpha) = x if x > 0 else alpha * expm1(x / alpha)
__device__ __forceinline__ float celu_f(float x, float alpha) {
  return x > 0.f ? x : alpha * expm1f(x / alpha);
}

// celu'(z) recovered from h = celu(z): 1 for h > 0, exp(z/alpha) = h/alpha + 1 otherwise.
__device__ __forceinline__ float dcelu_from_h(float h, float alpha) {
  return h > 0.f ? 1.f : h / alpha + 1.f;
}

// Which 16-column groups of the AEV columns a call has to look at (bit g % 64
// of word g / 64: columns [16 g, 16 g + 16)); words == nullptr: all of them.
struct ColumnGroups {
  const unsigned long long* words;
  bool has(int g) const { return !words || ((words[g >> 6] >> (g & 63)) & 1ull) != 0; }
};

}  // namespace fnl

// Entry points of the individual MLP implementations (C++ linkage, internal).
// xg: the input columns that may be non-zero; dg: the dx columns wanted; dx
// NULL: energies only.
size_t fnl_mlp_simt_workspace(int rows, const fennol_mlp_weights* w);
int fnl_mlp_simt(int rows, int ntiles, const int* tile_species, const int* tile_row,
                 const fennol_mlp_weights* w, const float* x, fnl::ColumnGroups xg, fnl::ColumnGroups dg,
                 float* e_rows, float* dx, void* ws, cudaStream_t st);
// The *_launches functions: kernels of one call.
int fnl_mlp_simt_launches(int rows, int ntiles, const fennol_mlp_weights* w, fnl::ColumnGroups dg, bool want_dx);
size_t fnl_mlp_tc_workspace(int precision, int rows, int n_models, const fennol_mlp_weights* w);
int fnl_mlp_tc(int precision, int rows, int ntiles, const int* tile_species, const int* tile_row,
               const fennol_mlp_weights* w, const void* x, const void* x_lo, fnl::ColumnGroups xg,
               fnl::ColumnGroups dg, float* e_rows, float* dx, void* ws, size_t ws_bytes, cudaStream_t st);
int fnl_mlp_tc_launches(int precision, int ntiles, const fennol_mlp_weights* w, bool want_dx);
bool fnl_mlp_fused_supported(int precision, const fennol_mlp_weights* w);
size_t fnl_mlp_fused_workspace(int rows, const fennol_mlp_weights* w);
int fnl_mlp_fused(int precision, int rows, int ntiles, const int* tile_species, const int* tile_row,
                  const fennol_mlp_weights* w, const void* x, const void* x_lo, fnl::ColumnGroups xg,
                  fnl::ColumnGroups dg, float* e_rows, float* dx, void* ws, size_t ws_bytes, cudaStream_t st);
int fnl_mlp_fused_launches(int ntiles, const fennol_mlp_weights* w);
