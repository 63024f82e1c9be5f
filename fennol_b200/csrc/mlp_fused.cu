// Fused, persistent species MLP on tcgen05 (sm_100a): forward + input gradient
// of FullyConnectedNet (src/fennol/models/misc/nets.py:13-102) inside
// SpeciesIndexNet (:301-426), with the ensemble mean, in one launch.
//
// One CTA per SM takes an even share of the (128-row tile of one species,
// model) items and runs, for each, the six GEMMs of the layer chain
//     L1 X.W1  L2 H1.W2  L3 H2.W3 (+ energy head)  B3 G3.W3^T  B2 G2.W2^T  B1 G1.W1^T
// (energies only: the first three) keeping the activations on chip:
//   * warp 0 (one thread) streams the AEV tile and W1^T through an L1 ring laid
//     over the activation buffer and the weight slots, then all other weights
//     through the weight slots;
//   * warp 1 owns the 512 TMEM columns (two 256-column FP32 accumulators used
//     alternately) and one thread issues tcgen05.mma / tcgen05.commit;
//   * warps 2-17 are the epilogue: they read an accumulator (tcgen05.ld, one
//     row per thread, four warps per lane quarter), apply bias + CELU, the
//     energy head, or CELU' masks, and write the next A operand as 16-bit hi
//     (+ lo) pairs straight into shared memory in the 128-byte-swizzled K-major
//     layout the MMA descriptors expect (fence.proxy.async before the MMA
//     reads it).
// What bounds it: the chain of GEMM -> epilogue -> GEMM of one item, which
// nothing else fills.  So the epilogue is short (packed FP32 instructions, no
// selects, biases in shared memory, no spills: with 16 warps a spilled register
// is an L2 round trip, 62k cycles per water item against 47k), its warps finish
// one 64-column K-atom after the other so that the next GEMM starts early, and
// dX is summed over the models in scratch instead of by bulk adds, which held
// up the loads of the next item.  98,304 atoms x 8 models (f16x3x1, water):
// 1.53 ms with 8 epilogue warps, 64-column chunks and whole tiles per CTA,
// 0.97 ms now; 192 atoms x 8 models 0.25 ms to 0.035 ms.
// Operand forms: BF16 (A hi, optionally A lo; weights BF16) and FP16 (the
// kernel template's F16 flag).  The FP16 forms split the activations and the
// power-of-two-scaled float32 weights into float16 hi + lo: the forward GEMMs
// run A_hi W_hi + A_lo W_hi + A_hi W_lo, the input-gradient GEMMs G_hi W_hi
// (+ G_hi W_lo).  Each epilogue divides its accumulator by the layer's weight
// scale; the backward chain carries the power-of-two scale of the last layer's
// kernel until dX.
// Active columns: the caller names the 16-column groups (one MMA K step each)
// of the input that may be non-zero; L1 leaves the K steps of the others out
// (their products are zero: the sums do not change) and streams only units of
// 64 or 32 columns that hold one.  B1 computes dX for the groups asked for, in
// runs of up to 16, whatever lies between them.
// CELU' of layers 1-2 (needed by the backward) goes to a per-CTA scratch in
// global memory that stays L2 resident.  The models of a tile are summed in
// model order, those of a tile shared by CTAs part by part, so the per-row
// energy and dE/dAEV sums are deterministic.  Every wait is bounded (2 s); a timeout sets the error word,
// raises a shared abort flag that ends all roles, and the CTA frees its TMEM.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "mlp_common.cuh"
#include "umma.cuh"

using namespace fnl;
using namespace fnl::umma;

namespace {

constexpr int kEpiWarps = 16;                     // four per TMEM lane quadrant
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int BM = 128, BK = 64;
constexpr int kGroup = 16;                        // columns of one active-column group: one MMA K step
constexpr uint32_t kAtom = BM * BK * 2;           // one 128 x 64 16-bit K-atom: 16 KB
constexpr uint32_t kActHalf = 4 * kAtom;          // up to K = 256 per hi (or lo) operand
constexpr uint32_t kActBytes = 2 * kActHalf;      // 128 KB
constexpr uint32_t kWStage = 256 * BK * 2;        // 32 KB
// Operand memory: activations hi [0, 64 K), activations lo [64 K, 128 K),
// weight slots 0 and 1 [128 K, 192 K).  Weight slots 2 and 3 are the lo half
// of the activations: the input-gradient GEMMs of forms without gradient lo
// parts leave it free once L3 has run.
constexpr int kWSlots = 4;
constexpr uint32_t kRing = kActBytes + 2 * kWStage;  // 192 KB
// L1 ring: stages of one column unit (64 columns with 128-byte swizzle, or 32
// with 64-byte swizzle), A hi | A lo | B hi (| B lo), laid through the operand
// memory from 64 K on and round to its start, so that the first stages avoid
// the activations hi, which the last GEMM of the previous item still reads.
constexpr int kXStages = 6;
constexpr uint32_t kXBase = kActHalf;
constexpr int kMaxUnits = 4096 / 32, kMaxGroups = 4096 / kGroup;
constexpr uint32_t kXpose = kEpiWarps * 32 * kGroup * 4;  // per-epilogue-warp 32 x 16 dX staging tiles: 32 KB
constexpr uint32_t kSmemMain = kRing + kXpose;            // 224 KB
// The same 32 KB hold an item's biases and last kernel (b1 | b2 | b3 | w4, 256
// floats each) until its dX leaves.
constexpr int kBias = 256;
// bounded waits: default limit, and the settings of fennol_mlp_wait_limit /
// fennol_mlp_inject_stall (host side)
constexpr uint64_t kTimeoutNs = 2000000000ull;
uint64_t g_wait_limit_ns = kTimeoutNs;
int g_stall_launches = 0;

struct FusedParams {
  int ntiles, n_models, n_species;
  const int* tile_species;
  const int* tile_row;
  int d0, d1, d2, d3;
  int a_lo;   // forward A operands (X, H1, H2) carry a lo part
  int g_lo;   // input-gradient A operands (G3, G2, G1) carry a lo part
  int wf_lo;  // forward GEMMs add A_hi x W_lo
  int wb_lo;  // input-gradient GEMMs add G_hi x W_lo
  int bslots;       // weight slots of the input-gradient GEMMs (4, or 2 with gradient lo parts)
  int unit;         // columns of an L1 unit: 64 or 32
  int nunits;       // active L1 units
  int xstages;
  uint32_t xstage;  // bytes of an L1 stage
  uint32_t slot_stages[2];        // L1 stages that overlap weight slots 0, 1 (bit per stage)
  uint32_t stage_slots[kXStages]; // weight slots that overlap an L1 stage (bits 0-3); bit 4: activations
  float alpha, inv_models;
  unsigned long long timeout_ns;  // limit of every bounded wait
  int stall;                      // the load producer issues no copies (timeout tests)
  const float4* scales;  // F16 forms: per group (s_W1, s_W2, s_W3, s_w4) powers of two
  const float* b1;
  const float* b2;
  const float* b3;
  const float* w4;
  const float* b4;
  float* e_rows;
  float* dx;
  float* dc;  // [gridDim.x][(d1 + d2) / 4][128][4]
  // ensembles: dX summed over the models so far, [gridDim.x][2][d0 / 4][128][4]
  // (first and other tiles of a CTA), and the energies of the models of tiles
  // shared by CTAs, [ntiles][n_models][128]
  float* xs;
  float* e_part;
  int* err;
  int ndx;                        // dX column groups (0: energies only)
  unsigned char xunit[kMaxUnits];   // L1 units and the K steps of each that are active (bit per 16 columns)
  unsigned char xbits[kMaxUnits];
  unsigned char dgroup[kMaxGroups]; // dX column groups, ascending
};

struct Maps {
  CUtensorMap x, xlo, w1t, w2t, w3t, w3, w2, w1, w1g;
  CUtensorMap w1t_lo, w2t_lo, w3t_lo, w3_lo, w2_lo, w1_lo, w1g_lo;  // low parts (unused maps alias the high ones)
  CUtensorMap dx;  // FP32 [rows][d0], 32-row x 16-column boxes, 64-byte swizzle
};

// The (tile, model) items of one CTA.  All items are numbered tile by tile and
// cut into `blocks` contiguous ranges of (nearly) equal length, so a range may
// begin and end inside a tile: those parts of a tile leave their sums in the
// CTA's scratch and k_mlp_join adds the parts up in model order.  (Whole tiles
// per CTA left 98,304 atoms x 8 models 6 tiles on some CTAs and 5 on others,
// 12,288 atoms 52 of 148 SMs idle, and ran a small box's 8 models one after
// the other.)
__host__ __device__ __forceinline__ int first_item(int ntiles, int M, int block, int blocks) {
  return (int)((long long)ntiles * M * block / blocks);
}
struct Items {
  int M, lo, count;
  __device__ void cut(int ntiles, int M_, int block, int blocks) {
    M = M_;
    lo = first_item(ntiles, M, block, blocks);
    count = first_item(ntiles, M, block + 1, blocks) - lo;
  }
  __device__ void at(int k, int& tile, int& model) const {
    tile = (lo + k) / M;
    model = lo + k - tile * M;
  }
};

struct Bars {
  uint64_t x_full[kXStages], x_empty[kXStages], w_full[kWSlots], w_empty[kWSlots];
  uint64_t acc_full[2], acc_free[2], act_ready[4], act_free, lo_free, done, ex_ready, ex_free, bias_full, bias_free;
  uint32_t tmem_slot;
  int abort_flag;
  Items items;
  float ex[BM];
};

// Drop the 128-byte L2 line at a (128-byte aligned) without writing it back;
// its contents become undefined.
__device__ __forceinline__ void discard_l2(const void* a) {
  asm volatile("discard.global.L2 [%0], 128;" ::"l"(a) : "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Two FP32 values in one 64-bit register, and the packed FP32 instructions
// (each half is rounded as the scalar instruction rounds it).
struct F2 {
  uint64_t v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// CELU and its derivative of two values from one exponential each:
// e = 2^(min(z, 0) k2), k2 = log2(e) / alpha, is celu' (exactly 1 for z > 0),
// and max(z, 0) + (alpha e - alpha) is celu (the bracket is exactly 0 for z > 0).
__device__ __forceinline__ void celu_pair2(F2 z, F2 alpha, F2 neg_alpha, F2 k2, F2& h, F2& dh) {
  float a, b;
  unpack2(z, a, b);
  float ea, eb;
  unpack2(mul2(pack2(fminf(a, 0.f), fminf(b, 0.f)), k2), ea, eb);
  dh = pack2(ex2(ea), ex2(eb));
  h = add2(pack2(fmaxf(a, 0.f), fmaxf(b, 0.f)), fma2(alpha, dh, neg_alpha));
}
__device__ __forceinline__ F2 dcelu2(F2 z, F2 k2) {
  float a, b;
  unpack2(z, a, b);
  float ea, eb;
  unpack2(mul2(pack2(fminf(a, 0.f), fminf(b, 0.f)), k2), ea, eb);
  return pack2(ex2(ea), ex2(eb));
}

// Bounded wait that also gives up when another role has aborted.
// Threads sleep in mbarrier.try_wait (woken when the phase completes) instead
// of polling, so waiting epilogue warps do not take issue slots from the MMA
// and TMA threads.
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err,
                                         uint64_t p_timeout_ns) {
  if (mbar_try(bar, parity, 20000u)) return true;
  const uint64_t deadline = globaltimer() + p_timeout_ns;
  while (true) {
    if (mbar_try(bar, parity, 20000u)) return true;
    if (*abort_flag) return false;
    if (globaltimer() > deadline) {
      *abort_flag = 1;
      atomicExch(err, 1);
      return false;
    }
  }
}

// Write 8 consecutive columns [n, n + 8) of row r as 16-bit hi (+ lo) into
// the swizzled K-major activation buffer (BF16, or FP16 when F16); one paired
// conversion per two columns for the high parts and one for the residuals.
template <bool F16>
__device__ __forceinline__ void act_store(uint8_t* act, int r, int n, const F2* v, bool with_lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float a, b;
    unpack2(v[k], a, b);
    if constexpr (F16) {
      const __half2 hb = __floats2half2_rn(a, b);
      h[k] = *reinterpret_cast<const uint32_t*>(&hb);
    } else {
      const __nv_bfloat162 hb = __floats2bfloat162_rn(a, b);
      h[k] = *reinterpret_cast<const uint32_t*>(&hb);
    }
  }
  uint8_t* dst = act + (n >> 6) * kAtom + (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u +
                 ((((n & 63) >> 3) ^ (r & 7)) << 4);
  *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
  if (!with_lo) return;
  const F2 minus = pack2(-1.f, -1.f);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float a, b;
    if constexpr (F16) {
      const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&h[k]));
      unpack2(fma2(pack2(hf.x, hf.y), minus, v[k]), a, b);  // v - hi, rounded once
      const __half2 lb = __floats2half2_rn(a, b);
      l[k] = *reinterpret_cast<const uint32_t*>(&lb);
    } else {
      const float2 hf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&h[k]));
      unpack2(fma2(pack2(hf.x, hf.y), minus, v[k]), a, b);
      const __nv_bfloat162 lb = __floats2bfloat162_rn(a, b);
      l[k] = *reinterpret_cast<const uint32_t*>(&lb);
    }
  }
  *reinterpret_cast<uint4*>(dst + kActHalf) = make_uint4(l[0], l[1], l[2], l[3]);
}

template <bool F16>
__global__ void __launch_bounds__(kThreads, 1)
k_mlp_fused(const __grid_constant__ Maps maps, const __grid_constant__ FusedParams p) {
  extern __shared__ uint8_t smem_raw[];
  // rounded up to 1024 bytes by an offset, so that accesses stay in the shared window
  uint8_t* smem = smem_raw + (0u - smem_u32(smem_raw) & 1023u);
  uint8_t* act = smem;
  float* xpose = reinterpret_cast<float*>(smem + kRing);
  Bars* bars = reinterpret_cast<Bars*>(smem + kSmemMain);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int M = p.n_models;
  const int XS = p.xstages;
  const bool grad = p.ndx > 0;
  // weight slot s: 0, 1 behind the activations, 2, 3 in the activations' lo half
  auto slot_at = [&](int s) -> uint8_t* { return act + (s < 2 ? kActBytes + s * kWStage : kActHalf + (s - 2) * kWStage); };
  // component at byte `off` of L1 stage s
  auto stage_at = [&](int s, uint32_t off) -> uint8_t* {
    uint32_t o = kXBase + s * p.xstage + off;
    return act + (o >= kRing ? o - kRing : o);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kXStages; ++s) {
      mbar_init(&bars->x_full[s], 1);
      mbar_init(&bars->x_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->acc_full[s], 1);
      mbar_init(&bars->acc_free[s], kEpiWarps);
    }
    for (int s = 0; s < kWSlots; ++s) {
      mbar_init(&bars->w_full[s], 1);
      mbar_init(&bars->w_empty[s], 1);
    }
    for (int a = 0; a < 4; ++a) mbar_init(&bars->act_ready[a], kEpiWarps);
    mbar_init(&bars->act_free, 1);
    mbar_init(&bars->lo_free, 1);
    mbar_init(&bars->done, 1);
    mbar_init(&bars->ex_ready, BM);
    mbar_init(&bars->ex_free, BM);
    mbar_init(&bars->bias_full, 1);
    mbar_init(&bars->bias_free, kEpiWarps);
    bars->abort_flag = 0;
    fence_barrier_init();
  }
  if (threadIdx.x == 32) bars->items.cut(p.ntiles, M, blockIdx.x, gridDim.x);
  if (warp == 1) tmem_alloc(&bars->tmem_slot, 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = bars->tmem_slot;
  const Items& items = bars->items;
  // Launched as a programmatic dependent of the AEV forward: the set-up above
  // (barriers, TMEM) touches no global memory and overlaps that kernel's last
  // wave; every role reads or writes global memory only after this wait.
  pdl_wait();

  // L1 stage layout: A hi | A lo | B hi | B lo, each `unit` columns wide
  const uint32_t xa = BM * p.unit * 2, xb = (uint32_t)p.d1 * p.unit * 2, xb_slot = 256u * p.unit * 2;
  const uint32_t x_tx = xa * (1 + p.a_lo) + xb * (1 + p.wf_lo);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // (with p.stall it issues nothing: the other roles' waits run out)
    if (lane == 0 && !p.stall) {
      const uint64_t keep = l2_evict_last();
      uint32_t x_used = 0, x_par = 0;  // per L1 stage: used before; parity of its next use
      uint32_t w_used = 0, w_par = 0;  // the same per weight slot
      int bias_loaded = 0;
      bool ok = true;
      // the latest copy into slot s has been multiplied
      auto slot_free = [&](int s) -> bool {
        return !((w_used >> s) & 1) ||
               wait_bar(&bars->w_empty[s], ((w_par >> s) & 1) ^ 1, abort_flag, p.err, p.timeout_ns);
      };
      auto stage_free = [&](int s) -> bool {
        return !((x_used >> s) & 1) ||
               wait_bar(&bars->x_empty[s], ((x_par >> s) & 1) ^ 1, abort_flag, p.err, p.timeout_ns);
      };
      auto take_slot = [&](int s, uint32_t bytes) -> bool {
        if (!slot_free(s)) return false;
        w_used |= 1u << s;
        w_par ^= 1u << s;
        mbar_expect_tx(&bars->w_full[s], bytes);
        return true;
      };
      for (int it = 0; it < items.count && ok; ++it) {
        int tile, m;
        items.at(it, tile, m);
        const int row0 = p.tile_row[tile];
        const int g = m * p.n_species + p.tile_species[tile];
        bool act_ok = it == 0;  // the previous item's last GEMM has read the activations
        for (int u = 0; u < p.nunits; ++u) {
          const int s = u % XS;
          if (u < XS) {
            // first use in this item: what the previous item kept there must have been read
            if (!act_ok && (p.stage_slots[s] & 16u)) {
              if (!(ok = wait_bar(&bars->act_free, (it - 1) & 1, abort_flag, p.err, p.timeout_ns))) break;
              act_ok = true;
            }
            if (!act_ok)
              for (int q = 0; q < kWSlots && ok; ++q)
                if ((p.stage_slots[s] >> q) & 1) ok = slot_free(q);
            if (!ok) break;
          }
          if (!(ok = stage_free(s))) break;
          x_used |= 1u << s;
          x_par ^= 1u << s;
          const int c = p.xunit[u] * p.unit;
          mbar_expect_tx(&bars->x_full[s], x_tx);
          // the AEV tile is read once per model: kept in L2 ahead of other lines
          tma_load_2d_hint(&maps.x, &bars->x_full[s], stage_at(s, 0), c, row0, keep);
          if (p.a_lo) tma_load_2d_hint(&maps.xlo, &bars->x_full[s], stage_at(s, xa), c, row0, keep);
          tma_load_2d(&maps.w1t, &bars->x_full[s], stage_at(s, 2 * xa), c, g * p.d1);
          if (p.wf_lo) tma_load_2d(&maps.w1t_lo, &bars->x_full[s], stage_at(s, 2 * xa + xb_slot), c, g * p.d1);
        }
        if (!ok) break;
        // the item's biases and last kernel
        if (it > 0 && !(ok = wait_bar(&bars->bias_free, (it - 1) & 1, abort_flag, p.err, p.timeout_ns))) break;
        mbar_expect_tx(&bars->bias_full, (uint32_t)(p.d1 + p.d2 + 2 * p.d3) * 4);
        bulk_load(&bars->bias_full, xpose, p.b1 + (size_t)g * p.d1, p.d1 * 4);
        bulk_load(&bars->bias_full, xpose + kBias, p.b2 + (size_t)g * p.d2, p.d2 * 4);
        bulk_load(&bars->bias_full, xpose + 2 * kBias, p.b3 + (size_t)g * p.d3, p.d3 * 4);
        bulk_load(&bars->bias_full, xpose + 3 * kBias, p.w4 + (size_t)g * p.d3, p.d3 * 4);
        bias_loaded = it + 1;
        // weight chunks of the remaining GEMMs, in MMA order
        // (a GEMM with weight low parts takes the hi and lo chunks of each K step)
        const CUtensorMap* wm[4] = {&maps.w2t, &maps.w3t, &maps.w3, &maps.w2};
        const CUtensorMap* wml[4] = {&maps.w2t_lo, &maps.w3t_lo, &maps.w3_lo, &maps.w2_lo};
        const int rows_g[4] = {p.d2, p.d3, p.d2, p.d1};
        const int nk[4] = {p.d1 / BK, p.d2 / BK, p.d3 / BK, p.d2 / BK};
        int q = 0;
        bool lo_ok = false;  // L3 has read the activations' lo half
        // slots 2 and 3 may be filled once L3 has run
        auto back_slot = [&](uint32_t bytes) -> int {
          const int s = q++ & (p.bslots - 1);
          if (s >= 2 && !lo_ok) {
            if (!wait_bar(&bars->lo_free, it & 1, abort_flag, p.err, p.timeout_ns)) return -1;
            lo_ok = true;
          }
          return take_slot(s, bytes) ? s : -1;
        };
        for (int jb = 0; jb < (grad ? 4 : 2) && ok; ++jb) {
          if (jb == 2) q = 0;
          for (int kc = 0; kc < nk[jb] && ok; ++kc) {
            for (int t = 0; t < 1 + (jb < 2 ? p.wf_lo : p.wb_lo); ++t) {
              const uint32_t bytes = (uint32_t)rows_g[jb] * BK * 2;
              int s;
              if (jb < 2) {
                s = q & 1;
                if (q < 2)  // the L1 stages that overlap the slot have been read
                  for (int xs = 0; xs < XS && ok; ++xs)
                    if ((p.slot_stages[s] >> xs) & 1) ok = stage_free(xs);
                ++q;
                if (!ok || !(ok = take_slot(s, bytes))) break;
              } else {
                s = back_slot(bytes);
                if (!(ok = s >= 0)) break;
              }
              tma_load_2d(t ? wml[jb] : wm[jb], &bars->w_full[s], slot_at(s), kc * BK, g * rows_g[jb]);
            }
          }
        }
        // B1: the W1 rows of up to 16 dX column groups per run, stacked in the
        // slot; four groups of an aligned 64-column chunk take one box
        for (int r0 = 0; r0 < p.ndx && ok; r0 += 16) {
          const int ng = min(16, p.ndx - r0);
          for (int kc = 0; kc < p.d1 / BK && ok; ++kc) {
            for (int t = 0; t < 1 + p.wb_lo; ++t) {
              const int s = back_slot((uint32_t)ng * kGroup * BK * 2);
              if (!(ok = s >= 0)) break;
              for (int i = 0; i < ng;) {
                const int gr = p.dgroup[r0 + i];
                const bool four = (gr & 3) == 0 && i + 4 <= ng && p.dgroup[r0 + i + 3] == gr + 3;
                const CUtensorMap* mp = four ? (t ? &maps.w1_lo : &maps.w1) : (t ? &maps.w1g_lo : &maps.w1g);
                tma_load_2d(mp, &bars->w_full[s], slot_at(s) + i * kGroup * BK * 2, kc * BK, g * p.d0 + gr * kGroup);
                i += four ? 4 : 1;
              }
            }
          }
        }
      }
      // Before the CTA can exit, every issued TMA load must have landed (on an
      // abort some stages may never be consumed).  Bounded, ignores the abort flag.
      int dummy = 0;
      for (int s = 0; s < XS; ++s)
        if ((x_used >> s) & 1) wait_bar(&bars->x_full[s], ((x_par >> s) & 1) ^ 1, &dummy, p.err, p.timeout_ns);
      for (int s = 0; s < kWSlots; ++s)
        if ((w_used >> s) & 1) wait_bar(&bars->w_full[s], ((w_par >> s) & 1) ^ 1, &dummy, p.err, p.timeout_ns);
      if (bias_loaded) wait_bar(&bars->bias_full, (bias_loaded - 1) & 1, &dummy, p.err, p.timeout_ns);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      uint32_t x_par = 0, w_par = 0, act_par = 0;  // parities of the next full phase (bit per stage, slot, atom)
      uint32_t job = 0;
      bool ok = true;
      const uint32_t act_hi = smem_u32(act), act_lo = smem_u32(act + kActHalf);
      auto acquire_acc = [&](uint32_t b) -> bool {
        return job < 2 || wait_bar(&bars->acc_free[b], ((job >> 1) - 1) & 1, abort_flag, p.err, p.timeout_ns);
      };
      auto wait_slot = [&](int s) -> bool {
        if (!wait_bar(&bars->w_full[s], (w_par >> s) & 1, abort_flag, p.err, p.timeout_ns)) return false;
        w_par ^= 1u << s;
        fence_after_sync();
        return true;
      };
      int q = 0;  // weight chunks taken since the slots were restarted
      // one GEMM whose A operand is the activation buffer (K/64 atoms) and B the
      // weight slots.  With wait_act, each K-atom is used as soon as the epilogue
      // has published it, so the GEMM overlaps the epilogue that feeds it.
      // alo: A carries a lo part; wlo: each K step also has a W lo chunk.
      auto gemm_act = [&](int n, int k, uint32_t b, int slots, bool wait_act, bool alo, bool wlo) -> bool {
        const uint32_t idesc = F16 ? idesc_f16_f32(n) : idesc_bf16_f32(n);
        const uint32_t d = tmem + b * 256;
        for (int kc = 0; kc < k / BK; ++kc) {
          if (wait_act) {
            if (!wait_bar(&bars->act_ready[kc], (act_par >> kc) & 1, abort_flag, p.err, p.timeout_ns)) return false;
            act_par ^= 1u << kc;
          }
          int s = q++ & (slots - 1);
          if (!wait_slot(s)) return false;
          uint32_t bs = smem_u32(slot_at(s));
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            const uint64_t bd = sdesc_sw128(bs + kk * 32);
            mma_bf16(d, sdesc_sw128(act_hi + kc * kAtom + kk * 32), bd, idesc, (kc | kk) != 0);
            if (alo) mma_bf16(d, sdesc_sw128(act_lo + kc * kAtom + kk * 32), bd, idesc, 1u);
          }
          mma_commit(&bars->w_empty[s]);
          if (wlo) {
            s = q++ & (slots - 1);
            if (!wait_slot(s)) return false;
            bs = smem_u32(slot_at(s));
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              mma_bf16(d, sdesc_sw128(act_hi + kc * kAtom + kk * 32), sdesc_sw128(bs + kk * 32), idesc, 1u);
            mma_commit(&bars->w_empty[s]);
          }
        }
        return true;
      };
      for (int it = 0; it < items.count && ok; ++it) {
        // L1: A and B from the X ring; K steps of columns that are zero in every row are left out
        {
          const uint32_t b = job & 1;
          if (!(ok = acquire_acc(b))) break;
          const uint32_t idesc = F16 ? idesc_f16_f32(p.d1) : idesc_bf16_f32(p.d1);
          const uint32_t d = tmem + b * 256;
          uint32_t started = 0;
          for (int u = 0; u < p.nunits; ++u) {
            const int s = u % XS;
            if (!(ok = wait_bar(&bars->x_full[s], (x_par >> s) & 1, abort_flag, p.err, p.timeout_ns))) break;
            x_par ^= 1u << s;
            fence_after_sync();
            const uint32_t ah = smem_u32(stage_at(s, 0)), al = smem_u32(stage_at(s, xa));
            const uint32_t bh = smem_u32(stage_at(s, 2 * xa)), bl = smem_u32(stage_at(s, 2 * xa + xb_slot));
            const uint32_t bits = p.xbits[u];
            for (int kk = 0; kk < p.unit / 16; ++kk) {
              if (!((bits >> kk) & 1)) continue;
              const uint64_t ad = p.unit == 64 ? sdesc_sw128(ah + kk * 32) : sdesc_sw64(ah + kk * 32);
              const uint64_t bd = p.unit == 64 ? sdesc_sw128(bh + kk * 32) : sdesc_sw64(bh + kk * 32);
              mma_bf16(d, ad, bd, idesc, started);
              started = 1;
              if (p.a_lo) mma_bf16(d, p.unit == 64 ? sdesc_sw128(al + kk * 32) : sdesc_sw64(al + kk * 32), bd, idesc, 1u);
              if (p.wf_lo) mma_bf16(d, ad, p.unit == 64 ? sdesc_sw128(bl + kk * 32) : sdesc_sw64(bl + kk * 32), idesc, 1u);
            }
            mma_commit(&bars->x_empty[s]);
          }
          if (!ok) break;
          mma_commit(&bars->acc_full[b]);
          ++job;
        }
        // L2, L3, B3, B2: A from the activation buffer written by the epilogue
        const int ns[4] = {p.d2, p.d3, p.d2, p.d1};
        const int ks[4] = {p.d1, p.d2, p.d3, p.d2};
        q = 0;
        for (int jb = 0; jb < (grad ? 4 : 2) && ok; ++jb) {
          const uint32_t b = job & 1;
          const bool fwd = jb < 2;
          if (jb == 2) q = 0;
          if (!(ok = acquire_acc(b))) break;
          if (!(ok = gemm_act(ns[jb], ks[jb], b, fwd ? 2 : p.bslots, true, fwd ? p.a_lo : p.g_lo,
                              fwd ? p.wf_lo : p.wb_lo)))
            break;
          mma_commit(&bars->acc_full[b]);
          if (jb == 1 && grad) mma_commit(&bars->lo_free);
          ++job;
        }
        if (!ok) break;
        // B1: dX on runs of up to 16 column groups (<= 256 columns), A = G1
        // (published atom by atom for the first run)
        for (int r0 = 0; r0 < p.ndx && ok; r0 += 16) {
          const uint32_t b = job & 1;
          if (!(ok = acquire_acc(b))) break;
          if (!(ok = gemm_act(kGroup * min(16, p.ndx - r0), p.d1, b, p.bslots, r0 == 0, p.g_lo, p.wb_lo))) break;
          mma_commit(&bars->acc_full[b]);
          ++job;
        }
        if (!ok) break;
        mma_commit(&bars->act_free);
      }
      // all issued MMAs complete before TMEM is released
      mma_commit(&bars->done);
      wait_bar(&bars->done, 0, abort_flag, p.err, p.timeout_ns);
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    // Warp (q, part) owns rows [32 q, 32 q + 32) and, of every 64-column
    // K-atom, the columns [16 part, 16 part + 16): the 16 warps finish the
    // atoms one after the other, and the next GEMM starts on the first.
    const int q = warp & 3;
    const int part = (warp - 2) >> 2;
    const int r = 32 * q + lane;
    const uint32_t lane_base = (uint32_t)(32 * q) << 16;
    uint32_t job = 0;  // accumulators taken; they alternate between the two buffers
    bool ok = true;
    // per-CTA CELU' scratch [(d1 + d2) / 4][128 rows][4]: 16 bytes of a thread, 512 of a warp
    float4* dc = reinterpret_cast<float4*>(p.dc + (size_t)blockIdx.x * BM * (p.d1 + p.d2)) + r;
    float4* xs = reinterpret_cast<float4*>(p.xs + (size_t)blockIdx.x * 2 * BM * p.d0) + r;  // the dX sums, laid out alike
    const float* dc_lines = p.dc + (size_t)blockIdx.x * BM * (p.d1 + p.d2) + 128 * q;
    const float k2 = 1.4426950408889634f / p.alpha;  // log2(e) / alpha
    const F2 k2p = pack2(k2, k2), alp = pack2(p.alpha, p.alpha), nalp = pack2(-p.alpha, -p.alpha);
    const bool with_lo = p.a_lo != 0;    // forward activations
    const bool grad_lo = p.g_lo != 0;    // input-gradient operands
    auto take_acc = [&](uint32_t b) -> bool {
      bool ready = __all_sync(0xffffffffu, wait_bar(&bars->acc_full[b], (job >> 1) & 1, abort_flag, p.err, p.timeout_ns));
      if (ready) fence_after_sync();
      return ready;
    };
    auto release_acc = [&](uint32_t b) {
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_free[b]);
      ++job;
    };
    // the 16 columns of K-atom a written by this warp are visible to the MMA
    // (async proxy); the atom is complete when all epilogue warps arrived
    auto publish_atom = [&](int a) {
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->act_ready[a]);
    };
    // four FP32 values (two pairs) of a uniform shared address
    auto load4 = [&](const float* a, F2& lo, F2& hi) {
      const float4 t = *reinterpret_cast<const float4*>(a);
      lo = pack2(t.x, t.y);
      hi = pack2(t.z, t.w);
    };
    // H = celu(Z / s_W + bias) -> act for columns [0, n); celu'(z) / s_W' -> dc
    // columns [dc0, dc0 + n), where s_W' is the scale of the weights the
    // input gradient of this layer is taken through (a power of two, so the
    // product is exact).  inv_s = 1 / s_W, dscale = 1 / s_W' (1 for the BF16
    // forms).
    auto celu_layer = [&](const float* bias /* shared */, int n, int dc0, float inv_s, float dscale) -> bool {
      const uint32_t b = job & 1;
      const F2 isp = pack2(inv_s, inv_s), dsp = pack2(dscale, dscale);
      if (!take_acc(b)) return false;
#pragma unroll 1
      for (int a = 0; a < n / 64; ++a) {
        const int c = 64 * a + 16 * part;
        float v[16];
        tmem_ld16(tmem + b * 256 + lane_base + c, v);
        float4* dst = dc + (size_t)((dc0 + c) / 4) * BM;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          F2 bb[4], h[4], dh[4];
          load4(bias + c + 8 * hf, bb[0], bb[1]);
          load4(bias + c + 8 * hf + 4, bb[2], bb[3]);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            celu_pair2(fma2(pack2(v[8 * hf + 2 * k], v[8 * hf + 2 * k + 1]), isp, bb[k]), alp, nalp, k2p, h[k], dh[k]);
          act_store<F16>(act, r, c + 8 * hf, h, with_lo);
          if (grad) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              float4 t;
              unpack2(mul2(dh[2 * k], dsp), t.x, t.y);
              unpack2(mul2(dh[2 * k + 1], dsp), t.z, t.w);
              dst[(2 * hf + k) * BM] = t;
            }
          }
        }
        publish_atom(a);
      }
      release_acc(b);
      return true;
    };
    // G = D / s_W * celu'(z) -> act for columns [0, n), celu'(z) / s_W read
    // back from dc columns [dc0, dc0 + n) (written by this thread) an atom
    // ahead, the first before the accumulator is waited for.
    auto mask_layer = [&](int n, int dc0) -> bool {
      const uint32_t b = job & 1;
      const int na = n / 64;
      const float4* src = dc + (size_t)((dc0 + 16 * part) / 4) * BM;
      float4 dd[4];
      auto fetch = [&](int a) {
#pragma unroll
        for (int k = 0; k < 4; ++k) dd[k] = src[(16 * a + k) * BM];
      };
      fetch(0);
      if (!take_acc(b)) return false;
#pragma unroll 1
      for (int a = 0; a < na; ++a) {
        const int c = 64 * a + 16 * part;
        float v[16];
        tmem_ld16(tmem + b * 256 + lane_base + c, v);
        F2 gg[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          gg[2 * k] = mul2(pack2(v[4 * k], v[4 * k + 1]), pack2(dd[k].x, dd[k].y));
          gg[2 * k + 1] = mul2(pack2(v[4 * k + 2], v[4 * k + 3]), pack2(dd[k].z, dd[k].w));
        }
        if (a + 1 < na) fetch(a + 1);
        act_store<F16>(act, r, c, gg, grad_lo);
        act_store<F16>(act, r, c + 8, gg + 4, grad_lo);
        publish_atom(a);
        // the warp has read these 16 columns of its 32 rows for the last time
        // (16 lines): they are dropped from L2 without a write-back (the next
        // item rewrites them before reading)
        if (lane < 16)
          discard_l2(dc_lines + (size_t)((dc0 + c) / 4 + (lane >> 2)) * BM * 4 + 32 * (lane & 3));
      }
      release_acc(b);
      return true;
    };
    float e_row = 0.f;  // ensemble-mean row energy, accumulated model by model in registers
    for (int it = 0; it < items.count && ok; ++it) {
      int tile, m;
      items.at(it, tile, m);
      // this CTA's models of the tile: [m_first, m_end)
      const int m_first = max(0, items.lo - tile * M);
      const int m_end = min(M, items.lo + items.count - tile * M);
      const bool whole = m_first == 0 && m_end == M;
      const bool last_here = m + 1 == m_end;
      if (m == 0) e_row = 0.f;
      const int tile_row = p.tile_row[tile];
      const int g = m * p.n_species + p.tile_species[tile];
      // weight scales of this group (powers of two: the reciprocals are exact)
      float inv_s1 = 1.f, inv_s2 = 1.f, inv_s3 = 1.f, s_g = 1.f;
      if constexpr (F16) {
        const float4 sc = __ldg(p.scales + g);
        inv_s1 = 1.f / sc.x;
        inv_s2 = 1.f / sc.y;
        inv_s3 = 1.f / sc.z;
        s_g = sc.w;
      }
      ok = __all_sync(0xffffffffu, wait_bar(&bars->bias_full, it & 1, abort_flag, p.err, p.timeout_ns));
      if (!ok) break;
      // E1: H1 = celu(Z1 + b1) -> act; celu'(z1) -> dc[0:d1]
      if (!(ok = celu_layer(xpose, p.d1, 0, inv_s1, inv_s2))) break;
      // E2: H2 = celu(Z2 + b2) -> act; celu'(z2) -> dc[d1:d1+d2]
      if (!(ok = celu_layer(xpose + kBias, p.d2, p.d1, inv_s2, inv_s3))) break;
      // E3: G3 = s_g w4 * celu'(z3) -> act, then, while B3 runs, the energy head:
      // the part 0 and part 1 warps sum the 32-column chunks 0, 2, .. and
      // 1, 3, .. of a row in column order (the accumulator still holds Z3), and
      // the part 1 sum reaches the part 0 thread through shared memory guarded
      // by two mbarriers (bounded waits, no CTA barrier).
      float e = 0.f;
      {
        const uint32_t b = job & 1;
        const float *bias = xpose + 2 * kBias, *w4 = xpose + 3 * kBias;
        const F2 isp = pack2(inv_s3, inv_s3), sgp = pack2(s_g, s_g);
        if (!(ok = take_acc(b))) break;
        if (grad) {
#pragma unroll 1
          for (int a = 0; a < p.d3 / 64; ++a) {
            const int c = 64 * a + 16 * part;
            float v[16];
            tmem_ld16(tmem + b * 256 + lane_base + c, v);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
              F2 bb[4], ww[4];
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                load4(bias + c + 8 * hf + 4 * k, bb[2 * k], bb[2 * k + 1]);
                load4(w4 + c + 8 * hf + 4 * k, ww[2 * k], ww[2 * k + 1]);
              }
#pragma unroll
              for (int k = 0; k < 4; ++k)
                ww[k] = mul2(mul2(sgp, ww[k]),
                             dcelu2(fma2(pack2(v[8 * hf + 2 * k], v[8 * hf + 2 * k + 1]), isp, bb[k]), k2p));
              act_store<F16>(act, r, c + 8 * hf, ww, grad_lo);
            }
            publish_atom(a);
          }
        }
        if (part < 2) {
#pragma unroll 1
          for (int c = 32 * part; c < p.d3; c += 64) {
#pragma unroll 1
            for (int hh = 0; hh < 2; ++hh) {
              float v[16];
              tmem_ld16(tmem + b * 256 + lane_base + c + 16 * hh, v);
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                F2 bb[2], ww[2];
                load4(bias + c + 16 * hh + 4 * k, bb[0], bb[1]);
                load4(w4 + c + 16 * hh + 4 * k, ww[0], ww[1]);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  F2 h, dh;
                  celu_pair2(fma2(pack2(v[4 * k + 2 * u], v[4 * k + 2 * u + 1]), isp, bb[u]), alp, nalp, k2p, h, dh);
                  float h0, h1, w0, w1;
                  unpack2(h, h0, h1);
                  unpack2(ww[u], w0, w1);
                  e = fmaf(h0, w0, e);
                  e = fmaf(h1, w1, e);
                }
              }
            }
          }
        }
        release_acc(b);
        if (part == 1) {
          // the previous row energies must have been read before they are overwritten
          if (it > 0) {
            ok = __all_sync(0xffffffffu, wait_bar(&bars->ex_free, (it - 1) & 1, abort_flag, p.err, p.timeout_ns));
            if (!ok) break;
          }
          bars->ex[r] = e;
          mbar_arrive(&bars->ex_ready);
        }
      }
      if (grad) {
        // E4: G2 = D2 * celu'(z2) -> act
        if (!(ok = mask_layer(p.d2, p.d1))) break;
        // E5: G1 = D1 * celu'(z1) -> act
        if (!(ok = mask_layer(p.d1, 0))) break;
      }
      // the row's energy
      if (part == 0) {
        ok = __all_sync(0xffffffffu, wait_bar(&bars->ex_ready, it & 1, abort_flag, p.err, p.timeout_ns));
        if (!ok) break;
        e += bars->ex[r] + __ldg(p.b4 + g);
        mbar_arrive(&bars->ex_free);
      }
      if (part == 0) {
        if (whole) {
          e_row = fmaf(e, p.inv_models, e_row);
          if (last_here) p.e_rows[tile_row + r] = e_row;
        } else {
          p.e_part[((size_t)tile * M + m) * BM + r] = e;
        }
      }
      // E6: dX groups.  A thread adds its 16 columns of a group to the models
      // before (in model order, kept in the CTA's scratch).  With the last
      // model of a whole tile each warp stages its 32 x 16 block in its own
      // shared-memory tile, in the 64-byte-swizzled layout of the dX tensor
      // map, and the TMA engine writes it out.
      uint8_t* stage = reinterpret_cast<uint8_t*>(xpose + (warp - 2) * 32 * kGroup);
      uint8_t* trow = stage + lane * 64;
      const float dx_scale = p.inv_models * (inv_s1 / s_g);
      const F2 dxs = pack2(dx_scale, dx_scale);
      const bool out = whole && last_here;
      float4* sums = xs + (tile == items.lo / M ? 0 : (size_t)BM * p.d0 / 4);
      for (int r0 = 0; r0 < p.ndx && ok; r0 += 16) {
        const uint32_t b = job & 1;
        const int ng = min(16, p.ndx - r0);
#pragma unroll 1
        for (int i = part; i < ng || i == part; i += 4) {
          float4 sum[4];
          float4* scratch = sums + (size_t)(r0 + i) * 4 * BM;
          if (m > m_first && i < ng) {
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j] = __ldcg(scratch + j * BM);
          }
          if (i == part && !(ok = take_acc(b))) break;
          if (i >= ng) break;
          float v[16];
          tmem_ld16(tmem + b * 256 + lane_base + i * kGroup, v);
          if (out) {
            if (lane == 0) bulk_wait_read();  // the tile's previous copy has read it
            __syncwarp();
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            F2 a = mul2(pack2(v[4 * j], v[4 * j + 1]), dxs), c = mul2(pack2(v[4 * j + 2], v[4 * j + 3]), dxs);
            if (m > m_first) {
              a = add2(pack2(sum[j].x, sum[j].y), a);
              c = add2(pack2(sum[j].z, sum[j].w), c);
            }
            float4 t;
            unpack2(a, t.x, t.y);
            unpack2(c, t.z, t.w);
            if (out)
              *reinterpret_cast<float4*>(trow + ((j ^ ((lane >> 1) & 3)) << 4)) = t;
            else
              __stcg(scratch + j * BM, t);
          }
          if (out) {
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d_hint(&maps.dx, stage, p.dgroup[r0 + i] * kGroup, tile_row + 32 * q, l2_evict_last());
              bulk_commit();
            }
          }
        }
        if (!ok) break;
        release_acc(b);
      }
      if (!ok) break;
      // the biases' place is free again
      if (lane == 0) {
        bulk_wait_read();
        mbar_arrive(&bars->bias_free);
      }
    }
    // the dX copies have completed (and no longer read shared memory) before
    // the CTA exits
    if (lane == 0) bulk_wait_all();
    __syncwarp();
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// Tiles whose models several CTAs of k_mlp_fused shared: dX and the energies of
// the parts, added in model order.  Block (b, y): the tile that range b + 1
// starts inside of, if no earlier range does; y: a dX column group, a thread
// four columns of a row (four consecutive threads hold a row's 16).  It is
// bound by latency (one round of loads per four parts): a block per group keeps
// it to a few microseconds where one block per eight groups, a part after the
// other, took 104 us on 192 atoms x 8 models.
constexpr int kJoinThreads = BM * 4;
__global__ void __launch_bounds__(kJoinThreads) k_mlp_join(const __grid_constant__ FusedParams p, int blocks) {
  pdl_wait();
  const int M = p.n_models, b = blockIdx.x + 1;
  const int start = first_item(p.ntiles, M, b, blocks);
  const int tile = start / M, t0 = tile * M;
  if (start == t0 || first_item(p.ntiles, M, b - 1, blocks) > t0) return;  // no tile is cut here, or not first
  const int row0 = p.tile_row[tile];
  if (blockIdx.y == 0 && threadIdx.x < BM) {
    float e = 0.f;
    const float* part = p.e_part + (size_t)tile * M * BM + threadIdx.x;
#pragma unroll 4
    for (int m = 0; m < M; ++m) e = fmaf(__ldcg(part + (size_t)m * BM), p.inv_models, e);
    p.e_rows[row0 + threadIdx.x] = e;
  }
  const int i = blockIdx.y, r = threadIdx.x >> 2, j = threadIdx.x & 3;
  if (i >= p.ndx) return;
  // part c of the tile lies in range c's first (slot 0) or another (slot 1) tile
  const float4* xs = reinterpret_cast<const float4*>(p.xs) + (size_t)(i * 4 + j) * BM + r;
  const size_t per = (size_t)BM * p.d0 / 4;
  float4 v;
  for (int c0 = b - 1; c0 < blocks; c0 += 4) {
    float4 t[4];
    int n = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int lo = first_item(p.ntiles, M, c0 + k, blocks);
      if (c0 + k < blocks && lo < t0 + M) {
        t[k] = __ldcg(xs + ((size_t)(c0 + k) * 2 + (lo / M == tile ? 0 : 1)) * per);
        n = k + 1;
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k >= n) break;
      if (c0 + k == b - 1) {
        v = t[k];
      } else {
        v.x += t[k].x;
        v.y += t[k].y;
        v.z += t[k].z;
        v.w += t[k].w;
      }
    }
    if (n < 4) break;
  }
  *reinterpret_cast<float4*>(p.dx + (size_t)(row0 + r) * p.d0 + p.dgroup[i] * kGroup + 4 * j) = v;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }
  return fn;
}

// 16-bit [rows][cols] operand (BF16, or FP16 when f16) in boxes of box_rows
// rows x box_cols columns (64: 128-byte swizzle; 32: 64-byte swizzle)
bool map2d(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, bool f16,
           uint32_t box_cols = BK) {
  auto fn = encode_fn();
  if (!fn || !base) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
            dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE,
            box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// dX as FP32 [rows][cols] in boxes of 32 rows x 16 columns (64-byte rows, 64-byte swizzle)
bool map_dx(CUtensorMap* m, void* base, uint64_t rows, uint64_t cols) {
  auto fn = encode_fn();
  if (!fn || !base) return false;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * 4};
  cuuint32_t box[2] = {(cuuint32_t)kGroup, 32};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  }
  return n;
}

bool is_f16_form(int precision) {
  return precision == FENNOL_MLP_F16X3X1 || precision == FENNOL_MLP_F16X3X2;
}

}  // namespace

// Shape check: the fused kernel needs every hidden width <= 256 (activation
// buffer), the input width a multiple of 256 and a BF16, BF16x2 or FP16 form.
bool fnl_mlp_fused_supported(int precision, const fennol_mlp_weights* w) {
  const int* d = w->dims;
  if (precision != FENNOL_MLP_BF16 && precision != FENNOL_MLP_BF16X2 && !is_f16_form(precision)) return false;
  if (is_f16_form(precision) && !w->f16_scale) return false;
  if (d[0] % 256 != 0 || d[0] > 4096) return false;
  for (int l = 1; l < 4; ++l)
    if (d[l] > 256 || d[l] % 64 != 0) return false;
  return true;
}

namespace {

// CTAs of a launch: one per SM, or per (tile, model) item where there are fewer
int fused_grid(int tiles, int n_models) {
  const long long items = (long long)tiles * n_models;
  return items < sm_count() ? (int)items : sm_count();
}
size_t dc_bytes(int grid, const fennol_mlp_weights* w) {
  return (size_t)grid * BM * (w->dims[1] + w->dims[2]) * sizeof(float);
}
size_t xs_bytes(int grid, const fennol_mlp_weights* w) {
  return w->n_models > 1 ? (size_t)grid * 2 * BM * w->dims[0] * sizeof(float) : 0;
}
size_t e_part_bytes(int tiles, const fennol_mlp_weights* w) {
  return w->n_models > 1 ? (size_t)tiles * w->n_models * BM * sizeof(float) : 0;
}

}  // namespace

// error word, CELU' scratch on a 128-byte boundary (its L2 lines are discarded
// whole), dX sums and energies of ensembles
size_t fnl_mlp_fused_workspace(int rows, const fennol_mlp_weights* w) {
  const int grid = fused_grid(rows / BM, w->n_models);
  return 256 + 128 + dc_bytes(grid, w) + xs_bytes(grid, w) + e_part_bytes(rows / BM, w);
}

int fnl_mlp_fused(int precision, int rows, int ntiles, const int* tile_species, const int* tile_row,
                  const fennol_mlp_weights* w, const void* x, const void* x_lo, ColumnGroups xg, ColumnGroups dg,
                  float* e_rows, float* dx, void* ws, size_t ws_bytes, cudaStream_t st) {
  if (!encode_fn()) return FENNOL_ERR_UNSUPPORTED;
  if (ws_bytes < fnl_mlp_fused_workspace(rows, w)) return FENNOL_ERR_WORKSPACE;
  const int* d = w->dims;
  const int G = w->n_models * w->n_species;
  const bool f16 = is_f16_form(precision);
  const bool alo = precision == FENNOL_MLP_BF16X2 || f16;
  const bool glo = precision == FENNOL_MLP_BF16X2;
  const bool wflo = f16;
  const bool wblo = precision == FENNOL_MLP_F16X3X2;
  if (f16 && (!w->wt_lo[0] || !w->wt_lo[1] || !w->wt_lo[2])) return FENNOL_ERR_INVALID;
  if (wblo && (!w->w_lo[0] || !w->w_lo[1] || !w->w_lo[2])) return FENNOL_ERR_INVALID;
  if (f16 && ((uintptr_t)w->f16_scale & 15) != 0) return FENNOL_ERR_INVALID;
  FusedParams p{};
  // Column lists.  L1 streams units of 64 columns, or of 32 where that leaves
  // out enough zero columns (a 32-column unit is half a 128-byte swizzle row:
  // the same bytes in twice the copies).
  const int ngroups = d[0] / kGroup;
  int n64 = 0, n32 = 0;
  for (int c = 0; c < d[0] / 64; ++c) {
    const bool h0 = xg.has(4 * c) || xg.has(4 * c + 1), h1 = xg.has(4 * c + 2) || xg.has(4 * c + 3);
    n64 += h0 || h1;
    n32 += (int)h0 + (int)h1;
  }
  if (n64 == 0) return FENNOL_ERR_INVALID;
  p.unit = n32 * 5 <= n64 * 8 ? 32 : 64;
  const int per = p.unit / kGroup;
  for (int u = 0; u < ngroups / per; ++u) {
    int bits = 0;
    for (int k = 0; k < per; ++k) bits |= xg.has(u * per + k) ? 1 << k : 0;
    if (!bits) continue;
    p.xunit[p.nunits] = (unsigned char)u;
    p.xbits[p.nunits] = (unsigned char)bits;
    ++p.nunits;
  }
  if (dx)
    for (int g = 0; g < ngroups; ++g)
      if (dg.has(g)) p.dgroup[p.ndx++] = (unsigned char)g;
  // maps of absent low parts alias the high parts (never loaded)
  const void* wtl[3] = {wflo ? w->wt_lo[0] : w->wt_hi[0], wflo ? w->wt_lo[1] : w->wt_hi[1],
                        wflo ? w->wt_lo[2] : w->wt_hi[2]};
  const void* wl[3] = {wblo ? w->w_lo[0] : w->w_hi[0], wblo ? w->w_lo[1] : w->w_hi[1],
                       wblo ? w->w_lo[2] : w->w_hi[2]};
  Maps maps;
  const uint32_t un = (uint32_t)p.unit;
  bool ok = map2d(&maps.x, x, rows, d[0], BM, f16, un) && map2d(&maps.xlo, alo ? x_lo : x, rows, d[0], BM, f16, un) &&
            map2d(&maps.w1t, w->wt_hi[0], (uint64_t)G * d[1], d[0], d[1], f16, un) &&
            map2d(&maps.w1t_lo, wtl[0], (uint64_t)G * d[1], d[0], d[1], f16, un) &&
            map2d(&maps.w2t, w->wt_hi[1], (uint64_t)G * d[2], d[1], d[2], f16) &&
            map2d(&maps.w3t, w->wt_hi[2], (uint64_t)G * d[3], d[2], d[3], f16) &&
            map2d(&maps.w3, w->w_hi[2], (uint64_t)G * d[2], d[3], d[2], f16) &&
            map2d(&maps.w2, w->w_hi[1], (uint64_t)G * d[1], d[2], d[1], f16) &&
            map2d(&maps.w1, w->w_hi[0], (uint64_t)G * d[0], d[1], 64, f16) &&
            map2d(&maps.w1g, w->w_hi[0], (uint64_t)G * d[0], d[1], kGroup, f16) &&
            map2d(&maps.w2t_lo, wtl[1], (uint64_t)G * d[2], d[1], d[2], f16) &&
            map2d(&maps.w3t_lo, wtl[2], (uint64_t)G * d[3], d[2], d[3], f16) &&
            map2d(&maps.w3_lo, wl[2], (uint64_t)G * d[2], d[3], d[2], f16) &&
            map2d(&maps.w2_lo, wl[1], (uint64_t)G * d[1], d[2], d[1], f16) &&
            map2d(&maps.w1_lo, wl[0], (uint64_t)G * d[0], d[1], 64, f16) &&
            map2d(&maps.w1g_lo, wl[0], (uint64_t)G * d[0], d[1], kGroup, f16);
  if (ok && dx) ok = map_dx(&maps.dx, dx, rows, d[0]);
  if (!dx) maps.dx = maps.x;  // never used
  if (!ok) return FENNOL_ERR_CUDA;
  p.ntiles = ntiles;
  p.n_models = w->n_models;
  p.n_species = w->n_species;
  p.tile_species = tile_species;
  p.tile_row = tile_row;
  p.d0 = d[0];
  p.d1 = d[1];
  p.d2 = d[2];
  p.d3 = d[3];
  p.a_lo = alo ? 1 : 0;
  p.g_lo = glo ? 1 : 0;
  p.wf_lo = wflo ? 1 : 0;
  p.wb_lo = wblo ? 1 : 0;
  p.bslots = glo ? 2 : kWSlots;
  p.xstage = (uint32_t)p.unit * 2 * (2 * BM + 256 * (1 + p.wf_lo));
  p.xstages = (int)(kRing / p.xstage);
  // what each L1 stage lies on: per component (start, bytes), round the ring
  for (int s = 0; s < p.xstages; ++s)
    for (uint32_t off = 0; off < p.xstage; off += 8192) {  // every component is a multiple of 8 KB
      const uint32_t a = (kXBase + s * p.xstage + off) % kRing;
      if (a >= kActBytes) {
        const int q = (int)((a - kActBytes) / kWStage);
        p.stage_slots[s] |= 1u << q;
        p.slot_stages[q] |= 1u << s;
      } else if (a >= kActHalf && p.ndx > 0 && p.bslots == kWSlots) {
        p.stage_slots[s] |= 4u << ((a - kActHalf) / kWStage);
      } else {
        p.stage_slots[s] |= 16u;
      }
    }
  p.scales = reinterpret_cast<const float4*>(w->f16_scale);
  p.alpha = w->celu_alpha;
  p.inv_models = 1.0f / (float)w->n_models;
  p.b1 = w->b32[0];
  p.b2 = w->b32[1];
  p.b3 = w->b32[2];
  p.w4 = w->w32[3];
  p.b4 = w->b32[3];
  p.e_rows = e_rows;
  p.dx = dx;
  p.err = (int*)ws;
  p.timeout_ns = g_wait_limit_ns;
  p.stall = 0;
  if (g_stall_launches > 0) {
    p.stall = 1;
    --g_stall_launches;
  }
  p.dc = (float*)(((uintptr_t)ws + 256 + 127) & ~(uintptr_t)127);
  const size_t smem = kSmemMain + sizeof(Bars) + 1024;
  static bool attr[2] = {false, false};
  auto kern = f16 ? k_mlp_fused<true> : k_mlp_fused<false>;
  if (!attr[f16]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return FENNOL_ERR_CUDA;
    attr[f16] = true;
  }
  if (ntiles <= 0) return FENNOL_OK;
  // one item per (tile, model); the CTAs share the items out evenly
  const int grid = fused_grid(ntiles, w->n_models);
  p.xs = (float*)((char*)p.dc + dc_bytes(grid, w));
  p.e_part = (float*)((char*)p.xs + xs_bytes(grid, w));
  FNL_LAUNCH_PDL(kern, dim3(grid), dim3(kThreads), smem, st, maps, p);
  FNL_CHECK_LAUNCH();
  if (w->n_models > 1 && ntiles % grid != 0) {  // ranges that begin inside a tile
    FNL_LAUNCH_PDL(k_mlp_join, dim3(grid - 1, p.ndx > 0 ? p.ndx : 1), dim3(kJoinThreads), 0, st, p, grid);
    FNL_CHECK_LAUNCH();
  }
  return FENNOL_OK;
}

extern "C" int fennol_mlp_wait_limit(double seconds) {
  if (!(seconds > 0.0) || seconds > 60.0) return FENNOL_ERR_INVALID;
  g_wait_limit_ns = (uint64_t)(seconds * 1e9);
  return FENNOL_OK;
}

extern "C" int fennol_mlp_inject_stall(int launches) {
  if (launches < 0) return FENNOL_ERR_INVALID;
  g_stall_launches = launches;
  return FENNOL_OK;
}
