// Library-level C entry points: version and the MLP dispatcher.
#include "mlp_common.cuh"

extern "C" const char* fennol_version(void) { return "fennol_b200 0.1 (sm_100a)"; }

static bool weights_ok(int precision, const fennol_mlp_weights* w) {
  if (!w || w->n_models < 1 || w->n_species < 1) return false;
  for (int l = 0; l < 4; ++l)
    if (w->dims[l] <= 0 || w->dims[l] % 64 != 0) return false;
  if (w->dims[4] != 1) return false;
  for (int l = 0; l < 4; ++l)
    if (!w->w32[l] || !w->b32[l]) return false;
  if (precision != FENNOL_MLP_FP32) {
    for (int l = 0; l < 3; ++l) {
      if (!w->wt_hi[l] || !w->w_hi[l]) return false;
      if (precision == FENNOL_MLP_BF16X3 && (!w->wt_lo[l] || !w->w_lo[l])) return false;
      if ((precision == FENNOL_MLP_F16X3X1 || precision == FENNOL_MLP_F16X3X2) && !w->wt_lo[l]) return false;
      if (precision == FENNOL_MLP_F16X3X2 && !w->w_lo[l]) return false;
    }
  }
  if ((precision == FENNOL_MLP_F16X3X1 || precision == FENNOL_MLP_F16X3X2) && !w->f16_scale) return false;
  return true;
}

extern "C" size_t fennol_mlp_workspace_bytes(int precision, int rows, int n_models,
                                             const fennol_mlp_weights* w) {
  if (rows < 0 || !w) return 0;
  if (precision == FENNOL_MLP_FP32) return fnl_mlp_simt_workspace(rows, w);
  return fnl_mlp_tc_workspace(precision, rows, n_models, w);
}

namespace {

int energy_grad(int precision, int rows, int ntiles, const int* tile_species, const int* tile_row,
                const fennol_mlp_weights* w, const void* x, const void* x_lo, fnl::ColumnGroups xg,
                fnl::ColumnGroups dg, float* e_rows, float* dx, void* workspace, size_t workspace_bytes,
                void* stream) {
  if (precision < FENNOL_MLP_FP32 || precision > FENNOL_MLP_F16X3X2) return FENNOL_ERR_INVALID;
  if (!weights_ok(precision, w)) return FENNOL_ERR_INVALID;
  if (rows < 0 || ntiles < 0 || rows % 128 != 0 || ntiles * 128 > rows) return FENNOL_ERR_INVALID;
  if (ntiles == 0) return FENNOL_OK;
  if (!tile_species || !tile_row || !x || !e_rows || !workspace) return FENNOL_ERR_INVALID;
  if (workspace_bytes < fennol_mlp_workspace_bytes(precision, rows, w->n_models, w))
    return FENNOL_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (precision == FENNOL_MLP_FP32)
    return fnl_mlp_simt(rows, ntiles, tile_species, tile_row, w, (const float*)x, xg, dg, e_rows, dx, workspace, st);
  if (precision != FENNOL_MLP_BF16 && !x_lo) return FENNOL_ERR_INVALID;
  return fnl_mlp_tc(precision, rows, ntiles, tile_species, tile_row, w, x, x_lo, xg, dg, e_rows, dx, workspace,
                    workspace_bytes, st);
}

}  // namespace

extern "C" int fennol_mlp_energy_grad_groups(int precision, int rows, int ntiles, const int* tile_species,
                                             const int* tile_row, const fennol_mlp_weights* w, const void* x,
                                             const void* x_lo, const unsigned long long* host_x_groups,
                                             const unsigned long long* host_dx_groups, int group_words,
                                             float* e_rows, float* dx, void* workspace, size_t workspace_bytes,
                                             void* stream) {
  if (w && (host_x_groups || host_dx_groups) && (long long)group_words * 64 * 16 < w->dims[0])
    return FENNOL_ERR_INVALID;
  return energy_grad(precision, rows, ntiles, tile_species, tile_row, w, x, x_lo, fnl::ColumnGroups{host_x_groups},
                     fnl::ColumnGroups{host_dx_groups}, e_rows, dx, workspace, workspace_bytes, stream);
}

extern "C" int fennol_mlp_launches(int precision, int rows, int ntiles, const fennol_mlp_weights* w,
                                   const unsigned long long* host_dx_groups, int group_words, int want_dx) {
  if (precision < FENNOL_MLP_FP32 || precision > FENNOL_MLP_F16X3X2 || !weights_ok(precision, w)) return FENNOL_ERR_INVALID;
  if (rows < 0 || ntiles < 0 || rows % 128 != 0 || ntiles * 128ll > rows) return FENNOL_ERR_INVALID;
  if (host_dx_groups && (long long)group_words * 64 * 16 < w->dims[0]) return FENNOL_ERR_INVALID;
  if (ntiles == 0) return 0;
  return precision == FENNOL_MLP_FP32
             ? fnl_mlp_simt_launches(rows, ntiles, w, fnl::ColumnGroups{host_dx_groups}, want_dx != 0)
             : fnl_mlp_tc_launches(precision, ntiles, w, want_dx != 0);
}

extern "C" int fennol_mlp_energy_grad_active(int precision, int rows, int ntiles, const int* tile_species,
                                             const int* tile_row, const fennol_mlp_weights* w, const void* x,
                                             const void* x_lo, unsigned long long active_chunks, float* e_rows,
                                             float* dx, void* workspace, size_t workspace_bytes, void* stream) {
  if (!dx && ntiles != 0) return FENNOL_ERR_INVALID;
  // four column groups per 64-column chunk
  unsigned long long words[4] = {0, 0, 0, 0};
  for (int c = 0; c < 64; ++c)
    if ((active_chunks >> c) & 1ull) words[c / 16] |= 0xFull << (4 * (c % 16));
  const bool dense = !active_chunks || active_chunks == ~0ull || precision == FENNOL_MLP_FP32 ||
                     precision == FENNOL_MLP_BF16X3;
  if (!active_chunks && precision != FENNOL_MLP_FP32 && ntiles > 0) return FENNOL_ERR_INVALID;
  const fnl::ColumnGroups g{dense ? nullptr : words};
  return energy_grad(precision, rows, ntiles, tile_species, tile_row, w, x, x_lo, g, g, e_rows, dx, workspace,
                     workspace_bytes, stream);
}

extern "C" int fennol_mlp_energy_grad(int precision, int rows, int ntiles, const int* tile_species,
                                      const int* tile_row, const fennol_mlp_weights* w, const void* x,
                                      const void* x_lo, float* e_rows, float* dx, void* workspace,
                                      size_t workspace_bytes, void* stream) {
  return fennol_mlp_energy_grad_active(precision, rows, ntiles, tile_species, tile_row, w, x, x_lo, ~0ull, e_rows,
                                       dx, workspace, workspace_bytes, stream);
}
