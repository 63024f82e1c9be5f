// Network sweep of the training-loss parameter gradient, on CUDA cores.
//
// FeNNol trains with jax.value_and_grad over a loss that holds forces
// (src/fennol/training/utils.py:140-525, train_step :508): second-order
// differentiation through SpeciesIndexNet (src/fennol/models/misc/nets.py:
// 13-102, 301-426).  With t = dAEV/dx . dL/dF from the AEV tangent kernel,
// the parameter gradient of the loss is the gradient, per species network f,
// of  sum_rows c_e[row] f(a_row) - <grad_a f(a_row), t_row>  (a = AEV row,
// c_e = dL/dE of the row's system).  This file computes it:
//
//   forward    [z_l; zd_l] = [h_{l-1}; hd_{l-1}] W_l (+ b_l on the z rows)
//              h_l = celu(z_l), hd_l = celu'(z_l) zd_l          (l = 1..3)
//   head       seeds hbar_3 = c_e w4, hdbar_3 = -w4; grad w4 = h_3^T c_e - sum hd_3,
//              grad b4 = sum c_e
//   backward   zbar = celu' hbar + celu'' zd hdbar, zdbar = celu' hdbar
//              grad W_l = [h_{l-1}; hd_{l-1}]^T [zbar_l; zdbar_l], grad b_l = sum zbar_l
//              [hbar_{l-1}; hdbar_{l-1}] = [zbar_l; zdbar_l] W_l^T
//
// A row and its tangent are rows 2r and 2r + 1 of one [2R x d] buffer, so every
// product above is one plain GEMM, and both rows of a pair end in the same
// thread, which applies CELU and its derivatives before it stores (no pass over
// memory of its own).  The first layer reads the AEV rows and the tangents where
// they are.  All species of a batch go through one grouped launch per stage.
// float32 or float64 arithmetic (the sweep's precision); the weight-gradient
// products (K = all rows of a species) are split along K with the partial
// products summed in a fixed order, so the result is deterministic.
//
// 256 molecules (6,242 atoms, float32): 0.7 ms (the two GEMMs of the first layer
// 0.34 ms, 38 TFLOP/s), against 1.45 ms with 128 x 128 tiles of scalar FMAs and
// separate CELU, stacking and column-sum passes (0.3 ms of that in column sums by
// 8 threads a column, 0.1 ms in a 128 x 128 tile for grad w4).
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int kMaxG = 8;   // species per batch
// GEMM tile: 128 x 64 outputs per 128 threads, 8 x 8 each; K slices of 64 bytes.
// Bound by the FP32 (FP64) pipe; float32 products are packed two to an
// instruction, which leaves issue slots to the loads (see mlp_simt.cu).
constexpr int BM = 128, BN = 64, kThreads = 128;
template <typename T>
constexpr int BK = sizeof(T) == 4 ? 16 : 8;

enum Mode { kForward = 0, kHead = 1, kBackward = 2, kWeights = 3 };

// Row m of a paired operand: (m odd ? p1 : p0) + (m / 2) * ld.
template <typename T>
struct Gemm {
  const T* a0[kMaxG];
  const T* a1[kMaxG];
  const T* b0[kMaxG];   // the kernel W, or the paired operand of the weight gradient
  const T* b1[kMaxG];
  T* c[kMaxG];          // z / - / - / weight gradient or its partial products
  T* h[kMaxG];          // [h; hd] (forward), [zbar; zdbar] (backward)
  T* zb[kMaxG];         // [zbar; zdbar] of the last hidden layer (head)
  const T* aux[kMaxG];  // bias (forward), [z; zd] (backward)
  const T* w4[kMaxG];
  const T* c_row[kMaxG];
  int rows2[kMaxG];     // 2 x the species' rows
  int splits[kMaxG];
  int first[kMaxG + 1]; // first block of each group
  int ng, M, N, K, lda, ldb, kper, vec;
  T alpha;
};

template <typename T>
struct Four {
  T v[4];
};
// Four consecutive values of which `valid` exist (zeros for the others).
template <typename T>
__device__ __forceinline__ Four<T> load4(const T* p, int valid, bool vec) {
  Four<T> r;
  if (vec && valid >= 4) {
    if constexpr (sizeof(T) == 4) {
      const float4 q = *reinterpret_cast<const float4*>(p);
      r.v[0] = q.x, r.v[1] = q.y, r.v[2] = q.z, r.v[3] = q.w;
    } else {
      const double2 q0 = *reinterpret_cast<const double2*>(p), q1 = *reinterpret_cast<const double2*>(p + 2);
      r.v[0] = q0.x, r.v[1] = q0.y, r.v[2] = q1.x, r.v[3] = q1.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = k < valid ? p[k] : T(0);
  }
  return r;
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const T* v, int valid, bool vec) {
  if (vec && valid >= 4) {
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
      *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < valid) p[k] = v[k];
  }
}
// shared memory: always aligned and whole
template <typename T>
__device__ __forceinline__ void lds4(const T* p, T* v) {
  const Four<T> r = load4(p, 4, true);
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = r.v[k];
}

template <typename T>
__device__ __forceinline__ void celu3(T z, T alpha, T& h, T& d1, T& d2) {
  const T e = exp((z < T(0) ? z : T(0)) / alpha);
  h = z > T(0) ? z : alpha * (e - T(1));
  d1 = z > T(0) ? T(1) : e;
  d2 = z > T(0) ? T(0) : e / alpha;
}

// acc[8][8] += a[8] b[8]^T
__device__ __forceinline__ void outer(float* acc, const float* a, const float* b) {
  unsigned long long* p = reinterpret_cast<unsigned long long*>(acc);
  unsigned long long bb[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) asm("mov.b64 %0, {%1, %2};" : "=l"(bb[j]) : "f"(b[2 * j]), "f"(b[2 * j + 1]));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    unsigned long long aa;
    asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a[i]));
#pragma unroll
    for (int j = 0; j < 4; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(p[4 * i + j]) : "l"(aa), "l"(bb[j]));
  }
}
__device__ __forceinline__ void outer(double* acc, const double* a, const double* b) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[8 * i + j] += a[i] * b[j];
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kThreads) k_gemm(const __grid_constant__ Gemm<T> g) {
  constexpr bool TN = MODE == kWeights, NT = MODE == kBackward;
  constexpr int KS = BK<T>, QA = BM * KS / 4 / kThreads, QB = BN * KS / 4 / kThreads;
  int grp = 0;
  while (grp + 1 < g.ng && (int)blockIdx.x >= g.first[grp + 1]) ++grp;
  int local = blockIdx.x - g.first[grp];
  const int ntile = (g.N + BN - 1) / BN;
  const int n0 = local % ntile * BN;
  local /= ntile;
  const int M = TN ? g.M : g.rows2[grp];
  const int mtile = (M + BM - 1) / BM;
  const int m0 = local % mtile * BM;
  const int split = local / mtile;
  const int kb = TN ? split * g.kper : 0;
  const int ke = TN ? min(g.rows2[grp], kb + g.kper) : g.K;
  const T* __restrict__ a0 = g.a0[grp];
  const T* __restrict__ a1 = g.a1[grp];
  const T* __restrict__ b0 = g.b0[grp];
  const T* __restrict__ b1 = g.b1[grp];
  __shared__ __align__(16) T As[2][KS][BM + 4];
  __shared__ __align__(16) T Bs[2][KS][BN + 4];
  const int tid = threadIdx.x, tx = tid & 7, ty = tid >> 3;
  Four<T> ra[QA], rb[QB];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int e = tid + kThreads * q;
      if (TN) {
        const int m = m0 + (e % (BM / 4)) * 4, k = k0 + e / (BM / 4);
        const T* row = ((k & 1) ? a1 : a0) + (size_t)(k >> 1) * g.lda;
        ra[q] = load4(row + m, k < ke ? M - m : 0, g.vec);
      } else {
        const int k = k0 + (e % (KS / 4)) * 4, m = m0 + e / (KS / 4);
        const T* row = ((m & 1) ? a1 : a0) + (size_t)(m >> 1) * g.lda;
        ra[q] = load4(row + k, m < M ? ke - k : 0, g.vec);
      }
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int e = tid + kThreads * q;
      if (NT) {
        const int k = k0 + (e % (KS / 4)) * 4, n = n0 + e / (KS / 4);
        rb[q] = load4(b0 + (size_t)n * g.ldb + k, n < g.N ? ke - k : 0, g.vec);
      } else {
        const int n = n0 + (e % (BN / 4)) * 4, k = k0 + e / (BN / 4);
        const T* row = TN ? ((k & 1) ? b1 : b0) + (size_t)(k >> 1) * g.ldb : b0 + (size_t)k * g.ldb;
        rb[q] = load4(row + n, k < ke ? g.N - n : 0, g.vec);
      }
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int q = 0; q < QA; ++q) {
      const int e = tid + kThreads * q;
      if (TN) {
        store4(&As[buf][e / (BM / 4)][(e % (BM / 4)) * 4], ra[q].v, 4, true);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) As[buf][(e % (KS / 4)) * 4 + u][e / (KS / 4)] = ra[q].v[u];
      }
    }
#pragma unroll
    for (int q = 0; q < QB; ++q) {
      const int e = tid + kThreads * q;
      if (NT) {
#pragma unroll
        for (int u = 0; u < 4; ++u) Bs[buf][(e % (KS / 4)) * 4 + u][e / (KS / 4)] = rb[q].v[u];
      } else {
        store4(&Bs[buf][e / (BN / 4)][(e % (BN / 4)) * 4], rb[q].v, 4, true);
      }
    }
  };
  __align__(16) T acc[64];
#pragma unroll
  for (int i = 0; i < 64; ++i) acc[i] = T(0);
  int buf = 0;
  fetch(kb);
  put(0);
  __syncthreads();
  for (int k0 = kb; k0 < ke; k0 += KS) {
    const bool more = k0 + KS < ke;
    if (more) fetch(k0 + KS);
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      T a[8], b[8];
      lds4(&As[buf][kk][ty * 4], a);
      lds4(&As[buf][kk][64 + ty * 4], a + 4);
      lds4(&Bs[buf][kk][tx * 4], b);
      lds4(&Bs[buf][kk][32 + tx * 4], b + 4);
      outer(acc, a, b);
    }
    if (more) put(buf ^ 1);
    __syncthreads();
    buf ^= 1;
  }
  const int N = g.N;
#pragma unroll
  for (int h = 0; h < 2; ++h) {  // columns n .. n + 3
    const int n = n0 + 32 * h + tx * 4;
    if (n >= N) continue;
    Four<T> bias{}, w4{};
    if (MODE == kForward || MODE == kHead) bias = load4(g.aux[grp] + n, N - n, false);
    if (MODE == kHead) w4 = load4(g.w4[grp] + n, N - n, false);
#pragma unroll
    for (int i = 0; i < 8; i += 2) {  // rows m (z) and m + 1 (its tangent)
      const int m = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
      const T *u = acc + 8 * i + 4 * h, *v = acc + 8 * (i + 1) + 4 * h;
      if (MODE == kWeights) {
        T* out = g.c[grp] + (size_t)split * M * N;
        if (m < M) store4(out + (size_t)m * N + n, u, N - n, g.vec);
        if (m + 1 < M) store4(out + (size_t)(m + 1) * N + n, v, N - n, g.vec);
        continue;
      }
      if (m >= M) continue;
      const size_t at = (size_t)m * N + n;
      T p[4], q[4], r[4], s[4];
      if (MODE == kBackward) {
        const Four<T> z = load4(g.aux[grp] + at, N - n, g.vec), zd = load4(g.aux[grp] + at + N, N - n, g.vec);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          T hh, d1, d2;
          celu3(z.v[j], g.alpha, hh, d1, d2);
          p[j] = d1 * u[j] + d2 * zd.v[j] * v[j];
          q[j] = d1 * v[j];
        }
        store4(g.h[grp] + at, p, N - n, g.vec);
        store4(g.h[grp] + at + N, q, N - n, g.vec);
        continue;
      }
      const T ce = MODE == kHead ? g.c_row[grp][m >> 1] : T(0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const T z = u[j] + bias.v[j], zd = v[j];
        T d1, d2;
        celu3(z, g.alpha, p[j], d1, d2);
        q[j] = d1 * zd;
        if (MODE == kHead) {  // seeds hbar = c_e w4, hdbar = -w4 through the CELU
          r[j] = d1 * (ce * w4.v[j]) + d2 * zd * -w4.v[j];
          s[j] = d1 * -w4.v[j];
        } else {
          r[j] = z;
          s[j] = zd;
        }
      }
      T* other = MODE == kHead ? g.zb[grp] : g.c[grp];
      store4(g.h[grp] + at, p, N - n, g.vec);
      store4(g.h[grp] + at + N, q, N - n, g.vec);
      store4(other + at, r, N - n, g.vec);
      store4(other + at + N, s, N - n, g.vec);
    }
  }
}

// Weight gradients from their partial products, in split order.
template <typename T>
struct SplitSum {
  const T* part[kMaxG];
  T* out[kMaxG];
  int splits[kMaxG];
  int mn, vec;
};
template <typename T>
__global__ void __launch_bounds__(256) k_split_sum(const SplitSum<T> s) {
  const int grp = blockIdx.y, i = (blockIdx.x * 256 + threadIdx.x) * 4;
  const int valid = s.mn - i;
  if (valid <= 0 || s.splits[grp] == 1) return;
  T v[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 4
  for (int k = 0; k < s.splits[grp]; ++k) {
    const Four<T> t = load4(s.part[grp] + (size_t)k * s.mn + i, valid, s.vec);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] += t.v[j];
  }
  store4(s.out[grp] + i, v, valid, s.vec);
}

// Column sums over the rows of a species, in a fixed order: every bias gradient
// and the last layer's kernel, each (species, output) one job.  A block sums 32
// columns with 32 threads a column; bound by latency (R / 32 loads a thread,
// eight in flight: 256 molecules 53 -> 25 us against a loop that had fewer).
constexpr int kMaxJobs = 5 * kMaxG;
constexpr int kColBatch = 8;  // rows of a slice in flight
template <typename T>
struct ColSums {
  const T* in[kMaxJobs];   // [2 rows][d]: rows 2r are summed
  const T* c[kMaxJobs];    // not NULL: sum of c[r] in[2r][j] - in[2r + 1][j] instead
  T* out[kMaxJobs];
  int rows[kMaxJobs], d[kMaxJobs], step[kMaxJobs];  // step: elements between rows 2r
};
template <typename T>
__global__ void __launch_bounds__(1024) k_colsum(const __grid_constant__ ColSums<T> s) {
  const int job = blockIdx.y, d = s.d[job], R = s.rows[job];
  const int col = threadIdx.x & 31, j = blockIdx.x * 32 + col, slice = threadIdx.x >> 5;
  if (blockIdx.x * 32 >= d) return;
  const T* in = s.in[job];
  const T* c = s.c[job];
  const size_t step = s.step[job];
  __shared__ T part[32][33];
  T sum = T(0);
  if (j < d) {
    for (int r0 = slice; r0 < R; r0 += 32 * kColBatch) {
      T v[kColBatch], w[kColBatch], f[kColBatch];
#pragma unroll
      for (int u = 0; u < kColBatch; ++u) {
        const int r = r0 + 32 * u;
        v[u] = r < R ? in[r * step + j] : T(0);
        w[u] = c && r < R ? in[r * step + d + j] : T(0);
        f[u] = c && r < R ? c[r] : T(1);
      }
#pragma unroll
      for (int u = 0; u < kColBatch; ++u) sum += f[u] * v[u] - w[u];
    }
  }
  part[slice][col] = sum;
  __syncthreads();
  // warp w adds the slices of column w
  T v = part[col][slice];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int out = blockIdx.x * 32 + slice;
  if (col == 0 && out < d) s.out[job][out] = v;
}

// Loss seeds: per atom u = dL/dF (as the displacement field of the AEV tangent)
// and c_row = dL/dE of its system, per block partial sums of the squared errors.
template <typename T>
__global__ void __launch_bounds__(256) k_loss_seed(const double* __restrict__ energy, const double* __restrict__ e_ref,
                                                   int nsys, const float* __restrict__ forces,
                                                   const double* __restrict__ f_ref, int n,
                                                   const int* __restrict__ atom_sys, const int* __restrict__ atom_row,
                                                   double w_e, double w_f, float4* __restrict__ du,
                                                   T* __restrict__ c_row, double* __restrict__ part) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  double se = 0.0, sf = 0.0;
  if (i < n) {
    double d[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      d[k] = (double)forces[3 * (size_t)i + k] - f_ref[3 * (size_t)i + k];
      sf += d[k] * d[k];
    }
    const double s = 2.0 * w_f / (3.0 * n);
    du[i] = make_float4((float)(s * d[0]), (float)(s * d[1]), (float)(s * d[2]), 0.f);
    const int b = atom_sys[i];
    c_row[atom_row[i]] = (T)(2.0 * w_e / nsys * (energy[b] - e_ref[b]));
  }
  for (int b = i; b < nsys; b += gridDim.x * 256) {
    const double d = energy[b] - e_ref[b];
    se += d * d;
  }
  __shared__ double pe[256], pf[256];
  pe[threadIdx.x] = se;
  pf[threadIdx.x] = sf;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      pe[threadIdx.x] += pe[threadIdx.x + o];
      pf[threadIdx.x] += pf[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = pe[0];
    part[2 * blockIdx.x + 1] = pf[0];
  }
}
// The two loss terms, behind the status words as float64.
__global__ void __launch_bounds__(256) k_loss_terms(const double* __restrict__ part, int blocks, int nsys, int n,
                                                    double w_e, double w_f, const int* __restrict__ status,
                                                    double* __restrict__ out) {
  __shared__ double p[2][256];
  double s[2] = {0.0, 0.0};
  for (int b = threadIdx.x; b < blocks; b += 256) {
    s[0] += part[2 * b];
    s[1] += part[2 * b + 1];
  }
  p[0][threadIdx.x] = s[0];
  p[1][threadIdx.x] = s[1];
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o)
      for (int k = 0; k < 2; ++k) p[k][threadIdx.x] += p[k][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < FENNOL_STATUS_WORDS) out[threadIdx.x] = (double)status[threadIdx.x];
  if (threadIdx.x == 0) {
    out[FENNOL_STATUS_WORDS] = w_e * p[0][0] / nsys;
    out[FENNOL_STATUS_WORDS + 1] = w_f * p[1][0] / (3.0 * n);
  }
}

// Rows of a species' K slice of a weight gradient: about 1,100 blocks over the
// species (2.5 waves of three blocks per SM; 600 ran as two waves of longer
// blocks, 18 % slower), but 256 rows at least: shorter slices of the small
// layers' few tiles only move more partial products (128 rows: 25 us more in
// the sum over the slices).
int rows_per_split(int m, int n, long long rows2) {
  const long long tiles = (long long)((m + BM - 1) / BM) * ((n + BN - 1) / BN);
  const long long per = (rows2 * tiles + 1099) / 1100;
  return (int)std::max<long long>(256, (per + 15) / 16 * 16);
}

// workspace carve-up of one species with R rows (elements of T)
struct Carve {
  size_t z[3], h[4], zb[4], total;
};

Carve carve(const int* dims, int R) {
  Carve c{};
  size_t o = 0;
  auto take = [&](size_t n) {
    size_t p = o;
    o += (n + 31) / 32 * 32;  // 256-byte alignment for doubles
    return p;
  };
  const size_t R2 = 2 * (size_t)R;
  for (int l = 1; l <= 3; ++l) {
    if (l < 3) c.z[l] = take(R2 * dims[l]);
    c.h[l] = take(R2 * dims[l]);
    c.zb[l] = take(R2 * dims[l]);
  }
  c.total = o;
  return c;
}

// elements of the partial products of the weight gradients (one layer at a time)
size_t part_elems(const fennol_net_train* net, const int* host_rows) {
  long long rows2 = 0;
  for (int s = 0; s < net->n_species; ++s) rows2 += 2ll * std::max(host_rows[s], 0);
  size_t most = 0;
  for (int l = 0; l < 3; ++l) {
    const int kper = rows_per_split(net->dims[l], net->dims[l + 1], rows2);
    size_t n = 0;
    for (int s = 0; s < net->n_species; ++s)
      if (host_rows[s] > 0) n += (size_t)((2ll * host_rows[s] + kper - 1) / kper);
    most = std::max(most, n * net->dims[l] * net->dims[l + 1]);
  }
  return (most + 31) / 32 * 32;
}

template <typename T>
int run(const fennol_net_train* net, const int* host_row0, const int* host_rows, const void* x_, const void* t_,
        int ld, const void* c_row_, void* ws, cudaStream_t st) {
  const int* d = net->dims;
  const T* x = (const T*)x_;
  const T* t = (const T*)t_;
  const T* c_row = (const T*)c_row_;
  // the species with rows, in order
  int sp[kMaxG], ng = 0;
  Carve cv[kMaxG];
  T* base[kMaxG];
  size_t off = 0;
  long long rows2 = 0;
  for (int s = 0; s < net->n_species; ++s) {
    if (host_rows[s] <= 0) continue;
    sp[ng] = s;
    cv[ng] = carve(d, host_rows[s]);
    base[ng] = (T*)ws + off;
    off += cv[ng].total;
    rows2 += 2ll * host_rows[s];
    ++ng;
  }
  if (ng == 0) return FENNOL_OK;
  T* part = (T*)ws + off;
  auto blocks_of = [&](Gemm<T>& g, int mode) -> int {
    int n = 0;
    for (int gi = 0; gi < ng; ++gi) {
      g.first[gi] = n;
      const int M = mode == kWeights ? g.M : g.rows2[gi];
      n += (M + BM - 1) / BM * ((g.N + BN - 1) / BN) * (mode == kWeights ? g.splits[gi] : 1);
    }
    g.first[ng] = n;
    return n;
  };
  // operands of layer l (1..3): paired rows of the layer before it
  auto paired = [&](int l, int gi, const T*& p0, const T*& p1, int& lda) {
    if (l == 0) {
      p0 = x + (size_t)host_row0[sp[gi]] * ld;
      p1 = t + (size_t)host_row0[sp[gi]] * ld;
      lda = ld;
    } else {
      p0 = base[gi] + cv[gi].h[l];
      p1 = p0 + d[l];
      lda = 2 * d[l];
    }
  };
  // 16-byte accesses: every array aligned, every row a multiple of four values
  auto aligned = [&](std::initializer_list<int> widths, const Gemm<T>& g) -> int {
    for (int w : widths)
      if (w % 4 != 0) return 0;
    uintptr_t bits = 0;
    for (int gi = 0; gi < ng; ++gi)
      bits |= (uintptr_t)g.a0[gi] | (uintptr_t)g.a1[gi] | (uintptr_t)g.b0[gi] | (uintptr_t)g.b1[gi] |
              (uintptr_t)g.c[gi] | (uintptr_t)g.h[gi] | (uintptr_t)g.zb[gi];
    return (bits & 15) == 0;
  };
  auto start = [&](int N, int K) {
    Gemm<T> g{};
    g.ng = ng;
    g.N = N;
    g.K = K;
    g.alpha = (T)net->celu_alpha;
    for (int gi = 0; gi < ng; ++gi) g.rows2[gi] = 2 * host_rows[sp[gi]];
    return g;
  };
  // forward through the three hidden layers, the seeds with the last one
  for (int l = 1; l <= 3; ++l) {
    Gemm<T> g = start(d[l], d[l - 1]);
    for (int gi = 0; gi < ng; ++gi) {
      paired(l - 1, gi, g.a0[gi], g.a1[gi], g.lda);
      g.b0[gi] = (const T*)net->w[l - 1][sp[gi]];
      g.aux[gi] = (const T*)net->b[l - 1][sp[gi]];
      g.h[gi] = base[gi] + cv[gi].h[l];
      if (l < 3) {
        g.c[gi] = base[gi] + cv[gi].z[l];
      } else {
        g.zb[gi] = base[gi] + cv[gi].zb[3];
        g.w4[gi] = (const T*)net->w[3][sp[gi]];
        g.c_row[gi] = c_row + host_row0[sp[gi]];
      }
    }
    g.ldb = d[l];
    g.vec = aligned({g.lda, g.ldb, g.N, g.K}, g);
    if (l < 3)
      k_gemm<T, kForward><<<blocks_of(g, kForward), kThreads, 0, st>>>(g);
    else
      k_gemm<T, kHead><<<blocks_of(g, kHead), kThreads, 0, st>>>(g);
  }
  // backward through the hidden layers
  for (int l = 3; l >= 1; --l) {
    // grad W_{l-1} = [h; hd]_{l-1}^T [zbar; zdbar]_l
    Gemm<T> g = start(d[l], 0);
    SplitSum<T> s{};
    g.M = d[l - 1];
    g.kper = rows_per_split(d[l - 1], d[l], rows2);
    s.mn = d[l - 1] * d[l];
    size_t at = 0;
    int most = 1;
    for (int gi = 0; gi < ng; ++gi) {
      paired(l - 1, gi, g.a0[gi], g.a1[gi], g.lda);
      g.b0[gi] = base[gi] + cv[gi].zb[l];
      g.b1[gi] = g.b0[gi] + d[l];
      g.splits[gi] = s.splits[gi] = (g.rows2[gi] + g.kper - 1) / g.kper;
      s.part[gi] = part + at;
      s.out[gi] = (T*)net->gw[l - 1][sp[gi]];
      g.c[gi] = g.splits[gi] == 1 ? s.out[gi] : part + at;
      at += (size_t)g.splits[gi] * s.mn;
      most = std::max(most, g.splits[gi]);
    }
    g.ldb = 2 * d[l];
    g.vec = aligned({g.lda, g.ldb, g.N, g.M, d[l]}, g);
    k_gemm<T, kWeights><<<blocks_of(g, kWeights), kThreads, 0, st>>>(g);
    if (most > 1) {
      uintptr_t bits = 0;
      for (int gi = 0; gi < ng; ++gi) bits |= (uintptr_t)s.part[gi] | (uintptr_t)s.out[gi];
      s.vec = s.mn % 4 == 0 && (bits & 15) == 0;
      k_split_sum<T><<<dim3((s.mn + 1023) / 1024, ng), 256, 0, st>>>(s);
    }
    if (l == 1) break;
    // [hbar; hdbar]_{l-1} = [zbar; zdbar]_l W_{l-1}^T, through the CELU to [zbar; zdbar]_{l-1}
    Gemm<T> h = start(d[l - 1], d[l]);
    for (int gi = 0; gi < ng; ++gi) {
      h.a0[gi] = base[gi] + cv[gi].zb[l];
      h.a1[gi] = h.a0[gi] + d[l];
      h.b0[gi] = (const T*)net->w[l - 1][sp[gi]];
      h.aux[gi] = base[gi] + cv[gi].z[l - 1];
      h.h[gi] = base[gi] + cv[gi].zb[l - 1];
    }
    h.lda = 2 * d[l];
    h.ldb = d[l];
    h.vec = aligned({h.lda, h.ldb, h.N, h.K}, h);
    k_gemm<T, kBackward><<<blocks_of(h, kBackward), kThreads, 0, st>>>(h);
  }
  // bias gradients and the last layer
  ColSums<T> cs{};
  int jobs = 0, widest = 1;
  auto job = [&](const T* in, const T* c, void* out, int rows, int width, int step) {
    cs.in[jobs] = in;
    cs.c[jobs] = c;
    cs.out[jobs] = (T*)out;
    cs.rows[jobs] = rows;
    cs.d[jobs] = width;
    cs.step[jobs] = step;
    widest = std::max(widest, width);
    ++jobs;
  };
  for (int gi = 0; gi < ng; ++gi) {
    const int R = host_rows[sp[gi]];
    const T* c = c_row + host_row0[sp[gi]];
    for (int l = 1; l <= 3; ++l) job(base[gi] + cv[gi].zb[l], nullptr, net->gb[l - 1][sp[gi]], R, d[l], 2 * d[l]);
    job(base[gi] + cv[gi].h[3], c, net->gw[3][sp[gi]], R, d[3], 2 * d[3]);
    job(c, nullptr, net->gb[3][sp[gi]], R, 1, 1);
  }
  k_colsum<T><<<dim3((widest + 31) / 32, jobs), 1024, 0, st>>>(cs);
  return cudaGetLastError() == cudaSuccess ? FENNOL_OK : FENNOL_ERR_CUDA;
}

bool net_ok(const fennol_net_train* net) {
  if (!net || net->n_species < 1 || net->n_species > kMaxG || net->dims[4] != 1) return false;
  for (int l = 0; l < 4; ++l)
    if (net->dims[l] <= 0) return false;
  return true;
}

size_t elem_size(const fennol_net_train* net) { return net->is_double ? sizeof(double) : sizeof(float); }

}  // namespace

extern "C" size_t fennol_net_loss_grad_workspace_bytes(const fennol_net_train* net, const int* host_rows) {
  if (!net_ok(net) || !host_rows) return 0;
  size_t n = part_elems(net, host_rows);
  for (int s = 0; s < net->n_species; ++s)
    if (host_rows[s] > 0) n += carve(net->dims, host_rows[s]).total;
  return n * elem_size(net) + 256;
}

extern "C" int fennol_net_loss_grad(const fennol_net_train* net, const int* host_row0, const int* host_rows,
                                    const void* x, const void* t, int ld, const void* c_row, void* workspace,
                                    size_t workspace_bytes, void* stream) {
  if (!net_ok(net) || !host_row0 || !host_rows) return FENNOL_ERR_INVALID;
  if (ld < net->dims[0]) return FENNOL_ERR_INVALID;
  bool any = false;
  for (int s = 0; s < net->n_species; ++s) {
    if (host_rows[s] < 0 || host_row0[s] < 0) return FENNOL_ERR_INVALID;
    if (host_rows[s] == 0) continue;
    any = true;
    for (int l = 0; l < 4; ++l)
      if (!net->w[l][s] || !net->b[l][s] || !net->gw[l][s] || !net->gb[l][s]) return FENNOL_ERR_INVALID;
  }
  if (!any) return FENNOL_OK;
  if (!x || !t || !c_row || !workspace) return FENNOL_ERR_INVALID;
  if (((uintptr_t)workspace & 255) != 0) return FENNOL_ERR_INVALID;
  if (workspace_bytes < fennol_net_loss_grad_workspace_bytes(net, host_rows)) return FENNOL_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  return net->is_double ? run<double>(net, host_row0, host_rows, x, t, ld, c_row, workspace, st)
                        : run<float>(net, host_row0, host_rows, x, t, ld, c_row, workspace, st);
}

extern "C" size_t fennol_loss_seed_workspace_bytes(int natoms) {
  return natoms <= 0 ? 16 : ((size_t)natoms + 255) / 256 * 2 * sizeof(double);
}

extern "C" int fennol_loss_seed(const double* energy, const double* e_ref, int nsys, const float* forces,
                                const double* f_ref, int natoms, const int* atom_sys, const int* atom_row, double w_e,
                                double w_f, const int* status, float* du4, void* c_row, int is_double,
                                double* terms, void* workspace, size_t workspace_bytes, void* stream) {
  if (natoms <= 0 || nsys <= 0) return FENNOL_ERR_INVALID;
  if (!energy || !e_ref || !forces || !f_ref || !atom_sys || !atom_row || !status || !du4 || !c_row || !terms ||
      !workspace)
    return FENNOL_ERR_INVALID;
  if (((uintptr_t)du4 & 15) != 0 || ((uintptr_t)workspace & 7) != 0) return FENNOL_ERR_INVALID;
  if (workspace_bytes < fennol_loss_seed_workspace_bytes(natoms)) return FENNOL_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  const int blocks = (natoms + 255) / 256;
  double* part = (double*)workspace;
  if (is_double)
    k_loss_seed<double><<<blocks, 256, 0, st>>>(energy, e_ref, nsys, forces, f_ref, natoms, atom_sys, atom_row, w_e, w_f,
                                                (float4*)du4, (double*)c_row, part);
  else
    k_loss_seed<float><<<blocks, 256, 0, st>>>(energy, e_ref, nsys, forces, f_ref, natoms, atom_sys, atom_row, w_e, w_f,
                                               (float4*)du4, (float*)c_row, part);
  k_loss_terms<<<1, 256, 0, st>>>(part, blocks, nsys, natoms, w_e, w_f, status, terms);
  return cudaGetLastError() == cudaSuccess ? FENNOL_OK : FENNOL_ERR_CUDA;
}
