// Fused, persistent species MLP on tcgen05 (sm_100a): forward + input gradient
// of FullyConnectedNet (src/fennol/models/misc/nets.py:13-102) inside
// SpeciesIndexNet (:301-426), with the ensemble mean, in one launch.
//
// One CTA per SM takes an even share of the (128-row tile of one species,
// model) items and runs, for each, the six GEMMs of the layer chain
//     L1 X.W1  L2 H1.W2  L3 H2.W3 (+ energy head)  B3 G3.W3^T  B2 G2.W2^T  B1 G1.W1^T
// (energies only: the first three) keeping the activations on chip:
//   * warp 0 streams the AEV tile and all weights through one TMA ring in shared
//     memory, in the order the GEMMs take them, as far ahead as the ring holds;
//   * warp 1 owns the 512 TMEM columns (two regions of 256, accumulators and
//     activations in turn) and issues tcgen05.mma / tcgen05.commit;
//   * warps 2-17 are the epilogue: they read an accumulator (tcgen05.ld, one
//     row per thread, four warps per lane quarter), apply bias + CELU, the
//     energy head, or CELU' masks, and put the next A operand, 16-bit hi (+ lo)
//     pairs, over it in tensor memory (tcgen05.st).
// What bounds it: the chain of GEMM -> epilogue -> GEMM of one item, about 36k
// cycles for a water tile, of which the MMAs are 15k and the streaming of 0.96
// MB of operands at 50 bytes per cycle 19k; neither is full, each waits for the
// other at the ends of a GEMM.  So the epilogue is short (packed FP32
// instructions, no selects, biases in shared memory, no spills: with 16 warps a
// spilled register is an L2 round trip), its warps finish one 64-column K-atom
// after the other so that the next GEMM starts early, dX is summed over the
// models in scratch (bulk adds held up the loads of the next item), and the
// activations stay in tensor memory: through shared memory, the A operand's
// reads and writes and the W chunks took its whole bandwidth in L2 and L3, and
// the ring was too small to prefetch the next item.  98,304 atoms x 8 models
// (f16x3x1, water): 1.53 ms at first (62k cycles an item, whole tiles per CTA),
// 0.97 ms with the activations in shared memory (47k), 0.85 ms now; 192 atoms x 8
// models 0.25 ms at first, 0.03 ms now.
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
// 32 columns that hold one.  B1 computes dX for the groups asked for, in runs of
// up to 8, whatever lies between them.
// CELU' of layers 1-2 (needed by the backward) goes to a per-CTA scratch in
// global memory that stays L2 resident.  Row energies are summed in model order,
// and so is dE/dAEV, except in shared tiles where more than 16 column groups are
// wanted and the CTAs have more than one item each: there part by part, always in
// the same way for the same batch, but with a rounding that depends on how many
// tiles it has.  Every wait is bounded (2 s); a timeout sets the error word, raises
// a shared abort flag that ends all roles, and the CTA frees its TMEM.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "mlp_common.cuh"
#include "umma.cuh"

using namespace fnl;
using namespace fnl::umma;

namespace {

constexpr int kEpiWarps = 16;                     // four per TMEM lane quadrant
constexpr int kThreads = (2 + kEpiWarps) * 32;
constexpr int BM = 128, BK = 64;
constexpr int kGroup = 16;                        // columns of one active-column group: one MMA K step
// Shared memory: a ring that every operand from global memory streams through
// (activations live in tensor memory), an item's biases and last kernel (b1 | b2
// | b3 | w4, 256 floats each), and per-epilogue-warp 32 x 16 dX staging tiles.
// Ring components (an A or B tile of a chunk) start on 2 KB, the size of a dX
// column group's weights; the swizzles repeat every 1 KB and 512 bytes.
constexpr uint32_t kRing = 46 * 4096;
constexpr int kBias = 256;
constexpr uint32_t kXpose = kEpiWarps * 32 * kGroup * 4;
constexpr uint32_t kSmemMain = kRing + 4 * kBias * 4 + kXpose;
constexpr int kChunks = 16;      // chunks in flight at most
// L1 streams units of 32 columns (64-byte swizzle): half of a 64-column unit
// would often be zero columns, and with all columns active two of those (96 KB
// each with the W1 low parts) do not fit the ring.  Compared when the AEV kernels
// were slower than now: the whole call on 256 molecules x 8 models took 7 % less
// than with 64 columns, 8 MD steps of 98,304 atoms x 8 models 3 % less.
constexpr int kUnit = 32;
constexpr int kMaxUnits = 4096 / kUnit, kMaxGroups = 4096 / kGroup;
constexpr int kRunGroups = 8;    // dX column groups of one B1 run (128 columns)
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
  int wb_lo;  // input-gradient GEMMs add G_hi x W_lo
  int nunits;  // active L1 units
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
  // ensembles: dX summed over the models so far and dX of shared tiles,
  // [gridDim.x][slots][ndx * 4][128][4], and the energies of the models of
  // shared tiles, [tiles][n_models][128]
  float* xs;
  float* e_part;
  int xs_slots;
  int apart;  // the models of shared tiles have a slot each (else the parts of tiles)
  int* err;
  int ndx;                        // dX column groups (0: energies only)
  unsigned char xunit[kMaxUnits];   // L1 units and the K steps of each that are active (bit per 16 columns)
  unsigned char xbits[kMaxUnits];
  unsigned char dgroup[kMaxGroups]; // dX column groups, ascending
  // the boxes that W1 rows of the groups are loaded in, run by run: first group, groups
  unsigned char box_g[kMaxGroups], box_n[kMaxGroups];
};

struct Maps {
  CUtensorMap x, xlo, w1t, w2t, w3t, w3, w2, w1, w1p, w1g;
  CUtensorMap w1t_lo, w2t_lo, w3t_lo, w3_lo, w2_lo, w1_lo, w1p_lo, w1g_lo;  // low parts (unused maps alias the high ones)
  CUtensorMap dx;  // FP32 [rows][d0], 32-row x 16-column boxes, 64-byte swizzle
};

// The (tile, model) items of one CTA: `whole` tiles with all their models, then
// a contiguous range (nearly equal ones) of the items of the tiles left over,
// which CTAs share: they leave their dX in scratch and k_mlp_join adds the
// models up.  (Whole tiles only gave 98,304 atoms x 8 models 6 tiles on some
// CTAs and 5 on others, left 52 of 148 SMs idle at 12,288 atoms, and ran a small
// box's 8 models one after the other.)
struct Share {
  int M, blocks, whole, left;  // whole tiles per CTA; tiles left over
  // a 64-bit division is some hundred instructions, which was a third of k_mlp_join
  __host__ __device__ static int quotient(long long a, long long b) {
    return (a | b) >> 32 ? (int)(a / b) : (int)((unsigned)a / (unsigned)b);
  }
  __host__ __device__ Share(int ntiles, int M_, int blocks_)
      : M(M_), blocks(blocks_), whole(ntiles / blocks_), left(ntiles - whole * blocks_) {}
  // first item (of the tiles left over) of a CTA, and the CTA that has an item
  __host__ __device__ int first(int block) const { return quotient((long long)left * M * block, blocks); }
  __host__ __device__ int owner(int item) const {
    const long long n = (long long)left * M;
    return quotient((long long)(item + 1) * blocks + n - 1, n) - 1;
  }
  __host__ __device__ int most() const { return (int)(((long long)left * M + blocks - 1) / blocks); }  // items of a CTA
};
struct Items {
  int M, tile0, nwhole, shared0, lo, count;  // items of whole tiles; first tile left over
  __device__ void cut(int ntiles, int M_, int block, int blocks) {
    const Share s(ntiles, M_, blocks);
    M = M_;
    tile0 = block * s.whole;
    nwhole = s.whole * M;
    shared0 = s.whole * blocks;
    lo = s.first(block);
    count = nwhole + s.first(block + 1) - lo;
  }
  __device__ void at(int k, int& tile, int& model) const {
    const int i = k < nwhole ? k : lo + k - nwhole;
    tile = i / M;
    model = i - tile * M;
    tile += k < nwhole ? tile0 : shared0;
  }
};

struct Bars {
  uint64_t full[kChunks], empty[kChunks];
  uint64_t acc_full[2], act_ready[4], dx_free[2], r0_free, done, bias_full, bias_free;
  uint64_t e_fwd[8], e_back[8], e_half[4];  // row energies handed from warp to warp
  uint32_t tmem_slot;
  int abort_flag;
  Items items;
  float e_row[3][2][BM];
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

// Two columns of a row as packed 16-bit values: the high parts and, with_lo, the
// residuals (BF16, or FP16 when F16), each by one paired conversion.
template <bool F16>
__device__ __forceinline__ void split_pair(F2 v, bool with_lo, uint32_t& hi, uint32_t& lo) {
  float a, b;
  unpack2(v, a, b);
  const F2 minus = pack2(-1.f, -1.f);
  if constexpr (F16) {
    const __half2 hb = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&hb);
    if (!with_lo) return;
    const float2 hf = __half22float2(hb);
    unpack2(fma2(pack2(hf.x, hf.y), minus, v), a, b);  // v - hi, rounded once
    const __half2 lb = __floats2half2_rn(a, b);
    lo = *reinterpret_cast<const uint32_t*>(&lb);
  } else {
    const __nv_bfloat162 hb = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&hb);
    if (!with_lo) return;
    const float2 hf = __bfloat1622float2(hb);
    unpack2(fma2(pack2(hf.x, hf.y), minus, v), a, b);
    const __nv_bfloat162 lb = __floats2bfloat162_rn(a, b);
    lo = *reinterpret_cast<const uint32_t*>(&lb);
  }
}

// Operand forms: which lo parts there are.
enum Form { kBf16 = 0, kBf16x2 = 1, kF16 = 2 };
template <int FORM>
__global__ void __launch_bounds__(kThreads, 1)
k_mlp_fused(const __grid_constant__ Maps maps, const __grid_constant__ FusedParams p) {
  constexpr bool F16 = FORM == kF16;
  constexpr bool a_lo = FORM != kBf16;     // forward A operands (X, H1, H2)
  constexpr bool g_lo = FORM == kBf16x2;   // input-gradient A operands (G3, G2, G1)
  constexpr bool wf_lo = FORM == kF16;     // forward GEMMs add A_hi x W_lo
  extern __shared__ uint8_t smem_raw[];
  // rounded up to 1024 bytes by an offset, so that accesses stay in the shared window
  uint8_t* smem = smem_raw + (0u - smem_u32(smem_raw) & 1023u);
  float* biases = reinterpret_cast<float*>(smem + kRing);
  float* xpose = biases + 4 * kBias;
  Bars* bars = reinterpret_cast<Bars*>(smem + kSmemMain);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int M = p.n_models;
  const bool grad = p.ndx > 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kChunks; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int s = 0; s < 8; ++s) {
      mbar_init(&bars->e_fwd[s], 1);
      mbar_init(&bars->e_back[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->acc_full[s], 1);
      mbar_init(&bars->dx_free[s], kEpiWarps);
    }
    for (int a = 0; a < 4; ++a) {
      mbar_init(&bars->act_ready[a], kEpiWarps);
      mbar_init(&bars->e_half[a], 1);
    }
    mbar_init(&bars->r0_free, kEpiWarps);
    mbar_init(&bars->done, 1);
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

  // The producer and the MMA issuer run warp-wide, one elected lane issuing the
  // copies, MMAs and commits: their operands are then warp-uniform, where a
  // single thread's would be moved to uniform registers one by one.  (With one
  // thread and a table of ring places in shared memory the issue itself was the
  // bound: 1.2k cycles for the four copies of an L1 chunk, 620 for the four MMAs
  // of a B1 chunk.)
  auto wait_all = [&](uint64_t* bar, uint32_t parity) -> bool {
    return __all_sync(0xffffffffu, wait_bar(bar, parity, abort_flag, p.err, p.timeout_ns));
  };
  // Ring places: components one after the other, none across the end.  The
  // producer and the issuer work them out alike.
  auto place = [](uint32_t& pos, uint32_t bytes) -> uint32_t {
    const uint32_t at = pos + bytes > kRing ? 0 : pos;
    pos = at + bytes;
    return at;
  };
  const uint32_t xa = BM * kUnit * 2, xb = (uint32_t)p.d1 * kUnit * 2;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // Every chunk in the order the GEMMs take them, as far ahead as the ring
    // holds: the next item's L1 streams in while this one's gradient runs.
    // (with p.stall it issues nothing: the other roles' waits run out)
    if (!p.stall) {
      const bool leader = elect_one();
      const uint64_t keep = l2_evict_last();
      uint32_t seq = 0, oldest = 0;  // next chunk, oldest chunk not known to be consumed
      uint32_t pos = 0;
      int room = kRing, taken = 0, size = 0;  // bytes free; of this chunk; of the chunk in slot `lane`
      int biases_loaded = 0;
      bool ok = true;
      auto retire = [&]() -> bool {
        const uint32_t s = oldest % kChunks;
        if (!wait_all(&bars->empty[s], (oldest / kChunks) & 1)) return false;
        room += __shfl_sync(0xffffffffu, size, s);
        ++oldest;
        return true;
      };
      // starts a chunk of `bytes` in all: its barrier, and what it takes of the ring
      auto open = [&](uint32_t bytes) -> bool {
        while (seq - oldest >= kChunks)
          if (!retire()) return false;
        if (leader) mbar_expect_tx(&bars->full[seq % kChunks], bytes);
        taken = 0;
        return true;
      };
      // place of a component, once it is free
      auto room_for = [&](uint32_t bytes, uint32_t& at) -> bool {
        const uint32_t before = pos;
        at = place(pos, bytes);
        const int used = (int)bytes + (at == 0 && before != 0 ? (int)(kRing - before) : 0);
        room -= used;
        taken += used;
        while (room < 0)
          if (!retire()) return false;
        return true;
      };
      auto load = [&](const CUtensorMap* map, int x, int y, uint32_t bytes) -> bool {
        uint32_t at;
        if (!room_for(bytes, at)) return false;
        if (leader) tma_load_2d(map, &bars->full[seq % kChunks], smem + at, x, y);
        return true;
      };
      // the AEV tile is read once per model: kept in L2 ahead of other lines
      auto load_keep = [&](const CUtensorMap* map, int x, int y, uint32_t bytes) -> bool {
        uint32_t at;
        if (!room_for(bytes, at)) return false;
        if (leader) tma_load_2d_hint(map, &bars->full[seq % kChunks], smem + at, x, y, keep);
        return true;
      };
      auto close = [&]() {
        if (lane == (int)(seq % kChunks)) size = taken;
        ++seq;
      };
      for (int it = 0; it < items.count && ok; ++it) {
        int tile, m;
        items.at(it, tile, m);
        const int row0 = p.tile_row[tile];
        const int g = m * p.n_species + p.tile_species[tile];
        for (int u = 0; u < p.nunits && ok; ++u) {
          const int c = p.xunit[u] * kUnit;
          ok = open(xa * (1 + a_lo) + xb * (1 + wf_lo)) && load_keep(&maps.x, c, row0, xa) &&
               (!a_lo || load_keep(&maps.xlo, c, row0, xa)) && load(&maps.w1t, c, g * p.d1, xb) &&
               (!wf_lo || load(&maps.w1t_lo, c, g * p.d1, xb));
          if (ok) close();
        }
        if (!ok) break;
        // the item's biases and last kernel
        if (it > 0 && !(ok = wait_all(&bars->bias_free, (it - 1) & 1))) break;
        if (leader) {
          mbar_expect_tx(&bars->bias_full, (uint32_t)(p.d1 + p.d2 + 2 * p.d3) * 4);
          bulk_load(&bars->bias_full, biases, p.b1 + (size_t)g * p.d1, p.d1 * 4);
          bulk_load(&bars->bias_full, biases + kBias, p.b2 + (size_t)g * p.d2, p.d2 * 4);
          bulk_load(&bars->bias_full, biases + 2 * kBias, p.b3 + (size_t)g * p.d3, p.d3 * 4);
          bulk_load(&bars->bias_full, biases + 3 * kBias, p.w4 + (size_t)g * p.d3, p.d3 * 4);
        }
        biases_loaded = it + 1;
        // weight chunks of the remaining GEMMs, in MMA order: a K step of 64 each
        auto weights = [&](const CUtensorMap* hi, const CUtensorMap* lo, int rows, int k, bool with_lo) -> bool {
          const uint32_t bytes = (uint32_t)rows * BK * 2;
          for (int kc = 0; kc < k; kc += BK) {
            if (!open(bytes * (1 + with_lo)) || !load(hi, kc, g * rows, bytes) ||
                (with_lo && !load(lo, kc, g * rows, bytes)))
              return false;
            close();
          }
          return true;
        };
        ok = weights(&maps.w2t, &maps.w2t_lo, p.d2, p.d1, wf_lo) && weights(&maps.w3t, &maps.w3t_lo, p.d3, p.d2, wf_lo);
        if (!ok) break;
        if (!grad) continue;
        ok = weights(&maps.w3, &maps.w3_lo, p.d2, p.d3, p.wb_lo) && weights(&maps.w2, &maps.w2_lo, p.d1, p.d2, p.wb_lo);
        // B1: the W1 rows of the run's dX column groups, stacked: boxes of 4, 2
        // or 1 neighbouring groups
        int b0 = 0;
        for (int r0 = 0; r0 < p.ndx && ok; r0 += kRunGroups) {
          const uint32_t bytes = (uint32_t)min(kRunGroups, p.ndx - r0) * kGroup * BK * 2;
          int b = b0;
          for (int kc = 0; kc < p.d1 && ok; kc += BK) {
            ok = open(bytes * (1 + p.wb_lo));
            for (int t = 0; t < 1 + p.wb_lo && ok; ++t) {
              uint32_t at;
              if (!(ok = room_for(bytes, at))) break;
              b = b0;
              for (uint32_t off = 0; off < bytes; ++b) {
                const uint32_t n = p.box_n[b];
                const CUtensorMap* mp = n == 4 ? (t ? &maps.w1_lo : &maps.w1)
                                               : (n == 2 ? (t ? &maps.w1p_lo : &maps.w1p) : (t ? &maps.w1g_lo : &maps.w1g));
                if (leader)
                  tma_load_2d(mp, &bars->full[seq % kChunks], smem + at + off, kc, g * p.d0 + p.box_g[b] * kGroup);
                off += n * kGroup * BK * 2;
              }
            }
            if (ok) close();
          }
          b0 = b;
        }
      }
      // Before the CTA can exit, every issued TMA load must have landed (on an
      // abort some chunks may never be consumed, the last one not be complete).
      // Bounded, ignores the abort flag.
      if (leader) {
        int dummy = 0;
        const uint32_t end = seq + (ok ? 0 : 1);
        for (uint32_t k = end > kChunks ? end - kChunks : 0; k < end; ++k)
          wait_bar(&bars->full[k % kChunks], (k / kChunks) & 1, &dummy, p.err, p.timeout_ns);
        if (biases_loaded) wait_bar(&bars->bias_full, (biases_loaded - 1) & 1, &dummy, p.err, p.timeout_ns);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // Tensor memory: two regions of 256 columns.  L1 -> R0, L2 -> R1, L3 -> R0,
    // B3 -> R1, B2 -> R0, B1 runs -> the halves of R1 in turn; the A operand of
    // each GEMM but L1 is the other region, where the epilogue has put it over
    // the accumulator it came from.  So a region is overwritten only by a GEMM
    // whose own A operand was made from the result of the last reader; what that
    // leaves open (the next item's L1 and L2, B1 halves) is waited for, and so is
    // what it leaves open about the barriers (the next item's L1).
    const bool leader = elect_one();
    uint32_t seq = 0, pos = 0;      // next chunk and its place in the ring
    uint32_t act_par = 0;           // parity of the atoms' next phases
    uint32_t job = 0, runs = 0;     // accumulators committed; B1 runs issued
    bool ok = true;
    auto take = [&]() -> bool {
      if (!wait_all(&bars->full[seq % kChunks], (seq / kChunks) & 1)) return false;
      fence_after_sync();
      return true;
    };
    auto give = [&]() {
      if (leader) mma_commit(&bars->empty[seq % kChunks]);
      ++seq;
    };
    auto finish = [&]() {
      if (leader) mma_commit(&bars->acc_full[job & 1]);
      ++job;
    };
    // shared-memory descriptors: constant high word, start address in the low one
    const uint32_t base = smem_u32(smem);
    auto desc = [&](uint32_t at, uint32_t hi) -> uint64_t { return sdesc_of((base + at) >> 4, hi); };
    const uint32_t hi128 = sdesc_hi128(), hi64 = sdesc_hi64();
    // D (n columns at d) = A (k columns, in tensor memory at a) x the weight chunks.
    // With wait_act, each K-atom is used as soon as the epilogue has published
    // it, so the GEMM overlaps the epilogue that feeds it.
    // alo: A carries a lo part; wlo: each chunk also has the W lo part.
    auto gemm_act = [&](int n, int k, uint32_t d, uint32_t a, bool wait_act, bool alo, bool wlo) -> bool {
      const uint32_t idesc = F16 ? idesc_f16_f32(n) : idesc_bf16_f32(n);
      const uint32_t bytes = (uint32_t)n * BK * 2;
      for (int kc = 0; kc < k / BK; ++kc) {
        if (wait_act) {
          if (!wait_all(&bars->act_ready[kc], (act_par >> kc) & 1)) return false;
          act_par ^= 1u << kc;
        }
        if (!take()) return false;
        const uint64_t bh = desc(place(pos, bytes), hi128);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            mma_ts(d, a + 64 * kc + 16 * kk, bh + 2 * kk, idesc, (kc | kk) != 0);
            if (alo) mma_ts(d, a + 64 * kc + 16 * kk + 8, bh + 2 * kk, idesc, 1u);
          }
        }
        if (wlo) {
          const uint64_t bl = desc(place(pos, bytes), hi128);
          if (leader) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk) mma_ts(d, a + 64 * kc + 16 * kk, bl + 2 * kk, idesc, 1u);
          }
        }
        give();
      }
      return true;
    };
    // the halves of R1 that hold dX have been read
    auto dx_read = [&](uint32_t half) -> bool {
      const uint32_t uses = (runs + 1 - half) >> 1;
      return uses == 0 || wait_all(&bars->dx_free[half], (uses - 1) & 1);
    };
    const uint32_t R0 = tmem, R1 = tmem + 256;
    for (int it = 0; it < items.count && ok; ++it) {
      // L1: A and B from the ring; K steps of columns that are zero in every row are left out
      if (it > 0) {
        // B1 has read R0 (energies only: the epilogue has)
        ok = grad ? wait_all(&bars->acc_full[(job - 1) & 1], ((job - 1) >> 1) & 1) : wait_all(&bars->r0_free, (it - 1) & 1);
        if (!ok) break;
        fence_after_sync();
      }
      {
        const uint32_t idesc = F16 ? idesc_f16_f32(p.d1) : idesc_bf16_f32(p.d1);
        uint32_t started = 0;
        for (int u = 0; u < p.nunits; ++u) {
          if (!(ok = take())) break;
          const uint64_t ah = desc(place(pos, xa), hi64), al = a_lo ? desc(place(pos, xa), hi64) : 0ull;
          const uint64_t bh = desc(place(pos, xb), hi64), bl = wf_lo ? desc(place(pos, xb), hi64) : 0ull;
          const uint32_t bits = p.xbits[u];
#pragma unroll
          for (int kk = 0; kk < kUnit / 16; ++kk) {
            if (!((bits >> kk) & 1)) continue;
            if (leader) {
              mma_bf16(R0, ah + 2 * kk, bh + 2 * kk, idesc, started);
              if (a_lo) mma_bf16(R0, al + 2 * kk, bh + 2 * kk, idesc, 1u);
              if (wf_lo) mma_bf16(R0, ah + 2 * kk, bl + 2 * kk, idesc, 1u);
            }
            started = 1;
          }
          give();
        }
        if (!ok) break;
        // The two accumulator barriers take turns, and a phase must not complete
        // while a warp still waits for the one before it.  L1's was last used by
        // the item before: by B2 after one run, else by its run before the last,
        // which every warp has taken once it has read it.
        if (p.ndx > kRunGroups && !(ok = dx_read(runs & 1))) break;
        finish();
      }
      // L2, L3, B3, B2
      if (!(ok = dx_read(0) && dx_read(1))) break;
      fence_after_sync();
      ok = gemm_act(p.d2, p.d1, R1, R0, true, a_lo, wf_lo);
      if (!ok) break;
      finish();
      ok = gemm_act(p.d3, p.d2, R0, R1, true, a_lo, wf_lo);
      if (!ok) break;
      finish();
      if (!grad) continue;
      ok = gemm_act(p.d2, p.d3, R1, R0, true, g_lo, p.wb_lo);
      if (!ok) break;
      finish();
      ok = gemm_act(p.d1, p.d2, R0, R1, true, g_lo, p.wb_lo);
      if (!ok) break;
      finish();
      // B1: dX on runs of up to 8 column groups (<= 128 columns), A = G1
      // (published atom by atom for the first run)
      for (int r0 = 0; r0 < p.ndx && ok; r0 += kRunGroups) {
        const uint32_t half = runs & 1;
        if (!(ok = dx_read(half))) break;
        fence_after_sync();
        if (!(ok = gemm_act(kGroup * min(kRunGroups, p.ndx - r0), p.d1, R1 + 128 * half, R0, r0 == 0, g_lo, p.wb_lo))) break;
        finish();
        ++runs;
      }
    }
    // all issued MMAs complete before TMEM is released
    if (leader) mma_commit(&bars->done);
    wait_bar(&bars->done, 0, abort_flag, p.err, p.timeout_ns);
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue
    // Warp (q, part) owns rows [32 q, 32 q + 32) and, of every 64-column
    // K-atom, the columns [16 part, 16 part + 16) (one MMA K step): it turns
    // the accumulator's 16 columns into the 8 + 8 columns of packed 16-bit hi
    // and lo parts that the next GEMM reads as its A operand, in place.  The
    // 16 warps finish the atoms one after the other, and the next GEMM starts
    // on the first.
    const int q = warp & 3;
    const int part = (warp - 2) >> 2;
    const int r = 32 * q + lane;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
    uint32_t job = 0, runs = 0;
    bool ok = true;
    // per-CTA CELU' scratch [(d1 + d2) / 4][128 rows][4]: 16 bytes of a thread, 512 of a warp
    float4* dc = reinterpret_cast<float4*>(p.dc + (size_t)blockIdx.x * BM * (p.d1 + p.d2)) + r;
    const float k2 = 1.4426950408889634f / p.alpha;  // log2(e) / alpha
    const F2 k2p = pack2(k2, k2), alp = pack2(p.alpha, p.alpha), nalp = pack2(-p.alpha, -p.alpha);
    auto take_acc = [&]() -> bool {
      const bool ready = wait_all(&bars->acc_full[job & 1], (job >> 1) & 1);
      ++job;
      if (ready) fence_after_sync();
      return ready;
    };
    auto arrive = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // this warp's 16 columns of K-atom a are in tensor memory
    auto publish_atom = [&](int a) {
      tmem_wait_st();
      fence_before_sync();
      arrive(&bars->act_ready[a]);
    };
    // four FP32 values (two pairs) of a uniform shared address
    auto load4 = [&](const float* a, F2& lo, F2& hi) {
      const float4 t = *reinterpret_cast<const float4*>(a);
      lo = pack2(t.x, t.y);
      hi = pack2(t.z, t.w);
    };
    // H = celu(Z / s_W + bias) over columns [0, n) of the accumulator at `at`;
    // celu'(z) / s_W' -> dc columns [dc0, dc0 + n), where s_W' is the scale of
    // the weights the input gradient of this layer is taken through (a power of
    // two, so the product is exact).  inv_s = 1 / s_W, dscale = 1 / s_W' (1 for
    // the BF16 forms).
    auto celu_layer = [&](uint32_t at, const float* bias /* shared */, int n, int dc0, float inv_s, float dscale) -> bool {
      const F2 isp = pack2(inv_s, inv_s), dsp = pack2(dscale, dscale);
      if (!take_acc()) return false;
#pragma unroll 1
      for (int a = 0; a < n / 64; ++a) {
        const int c = 64 * a + 16 * part;
        float v[16];
        tmem_ld16(at + c, v);
        uint32_t w[16];
        float4* dst = dc + (size_t)((dc0 + c) / 4) * BM;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          F2 bb[2], h[2], dh[2];
          load4(bias + c + 4 * k, bb[0], bb[1]);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            celu_pair2(fma2(pack2(v[4 * k + 2 * u], v[4 * k + 2 * u + 1]), isp, bb[u]), alp, nalp, k2p, h[u], dh[u]);
            split_pair<F16>(h[u], a_lo, w[2 * k + u], w[8 + 2 * k + u]);
          }
          if (grad) {
            float4 t;
            unpack2(mul2(dh[0], dsp), t.x, t.y);
            unpack2(mul2(dh[1], dsp), t.z, t.w);
            dst[k * BM] = t;
          }
        }
        if constexpr (a_lo)
          tmem_st16(at + c, w);
        else
          tmem_st8(at + c, w);
        publish_atom(a);
      }
      return true;
    };
    // G = D / s_W * celu'(z) over columns [0, n) of the accumulator at `at`,
    // celu'(z) / s_W read back from dc columns [dc0, dc0 + n) (written by this
    // thread) an atom ahead, the first before the accumulator is waited for.
    auto mask_layer = [&](uint32_t at, int n, int dc0) -> bool {
      const int na = n / 64;
      const float4* src = dc + (size_t)((dc0 + 16 * part) / 4) * BM;
      float4 dd[4];
      auto fetch = [&](int a) {
#pragma unroll
        for (int k = 0; k < 4; ++k) dd[k] = src[(16 * a + k) * BM];
      };
      fetch(0);
      if (!take_acc()) return false;
#pragma unroll 1
      for (int a = 0; a < na; ++a) {
        const int c = 64 * a + 16 * part;
        float v[16];
        tmem_ld16(at + c, v);
        uint32_t w[16];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          split_pair<F16>(mul2(pack2(v[4 * k], v[4 * k + 1]), pack2(dd[k].x, dd[k].y)), g_lo, w[2 * k], w[8 + 2 * k]);
          split_pair<F16>(mul2(pack2(v[4 * k + 2], v[4 * k + 3]), pack2(dd[k].z, dd[k].w)), g_lo, w[2 * k + 1],
                          w[9 + 2 * k]);
        }
        if (a + 1 < na) fetch(a + 1);
        if constexpr (g_lo)
          tmem_st16(at + c, w);
        else
          tmem_st8(at + c, w);
        publish_atom(a);
        // the warp has read these 16 columns of its 32 rows for the last time
        // (16 lines): they are dropped from L2 without a write-back (the next
        // item rewrites them before reading)
        if (lane < 16)
          discard_l2(dc - lane + ((dc0 + c) / 4 + (lane >> 2)) * BM + 8 * (lane & 3));
      }
      return true;
    };
    // Row energies: a row's terms are summed in the order of 32-column chunks
    // 0, 2, .. and 1, 3, .. of its atoms (two sums), each chunk's columns in
    // order.  A chunk lies with two warps (parts 0, 1 or 2, 3), so the running
    // sum goes to and fro between them through shared memory, off the path of
    // the GEMMs (the atom has been published), guarded by barriers.
    const int pair = 4 * (part >> 1) + q;
    uint32_t handed = 0;  // sums passed on by the even part so far
    float e_row = 0.f;  // ensemble-mean row energy, accumulated model by model in registers
    for (int it = 0; it < items.count && ok; ++it) {
      // what the item is (worked out again for its last part, to hold fewer
      // registers in between)
      int tile, m;
      items.at(it, tile, m);
      int g = m * p.n_species + p.tile_species[tile];
      // weight scales of this group (powers of two: the reciprocals are exact)
      float inv_s1 = 1.f, inv_s2 = 1.f, inv_s3 = 1.f, s_g = 1.f;
      if constexpr (F16) {
        const float4 sc = __ldg(p.scales + g);
        inv_s1 = 1.f / sc.x;
        inv_s2 = 1.f / sc.y;
        inv_s3 = 1.f / sc.z;
        s_g = sc.w;
      }
      const float dx_scale = p.inv_models * (inv_s1 / s_g);
      const uint32_t R0 = lane_base, R1 = lane_base + 256;
      if (!(ok = wait_all(&bars->bias_full, it & 1))) break;
      // E1: H1 = celu(Z1 + b1); celu'(z1) -> dc[0:d1]
      if (!(ok = celu_layer(R0, biases, p.d1, 0, inv_s1, inv_s2))) break;
      // E2: H2 = celu(Z2 + b2); celu'(z2) -> dc[d1:d1+d2]
      if (!(ok = celu_layer(R1, biases + kBias, p.d2, p.d1, inv_s2, inv_s3))) break;
      // E3: G3 = s_g w4 * celu'(z3), and the energy head
      float e = 0.f;
      {
        const float *bias = biases + 2 * kBias, *w4 = biases + 3 * kBias;
        const F2 isp = pack2(inv_s3, inv_s3), sgp = pack2(s_g, s_g);
        if (!(ok = take_acc())) break;
        const int na = p.d3 / 64;
        // the warp's staging tile holds H3 until the sum gets to it
        float4* h3 = reinterpret_cast<float4*>(xpose + (warp - 2) * 32 * kGroup) + lane;
        if (lane == 0) bulk_wait_read();
        __syncwarp();
#pragma unroll 1
        for (int a = 0; a < na && ok; ++a) {
          const int c = 64 * a + 16 * part;
          float v[16];
          tmem_ld16(R0 + c, v);
          uint32_t w[16];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            F2 bb[2], ww[2], h[2];
            load4(bias + c + 4 * k, bb[0], bb[1]);
            load4(w4 + c + 4 * k, ww[0], ww[1]);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              F2 dh;
              celu_pair2(fma2(pack2(v[4 * k + 2 * u], v[4 * k + 2 * u + 1]), isp, bb[u]), alp, nalp, k2p, h[u], dh);
              split_pair<F16>(mul2(mul2(sgp, ww[u]), dh), g_lo, w[2 * k + u], w[8 + 2 * k + u]);
            }
            float4 t;
            unpack2(h[0], t.x, t.y);
            unpack2(h[1], t.z, t.w);
            h3[32 * k] = t;
          }
          if (grad) {
            if constexpr (g_lo)
              tmem_st16(R0 + c, w);
            else
              tmem_st8(R0 + c, w);
            publish_atom(a);
          }
          // the running sum of this warp's rows, on from the other warp's
          if (part & 1) {
            if (!(ok = wait_all(&bars->e_fwd[pair], handed & 1))) break;
            e = bars->e_row[0][part >> 1][r];
          } else if (a > 0) {
            if (!(ok = wait_all(&bars->e_back[pair], (handed - 1) & 1))) break;
            e = bars->e_row[1][part >> 1][r];
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 t = *reinterpret_cast<const float4*>(w4 + c + 4 * k), h = h3[32 * k];
            e = fmaf(h.x, t.x, e);
            e = fmaf(h.y, t.y, e);
            e = fmaf(h.z, t.z, e);
            e = fmaf(h.w, t.w, e);
          }
          if (!(part & 1)) {
            bars->e_row[0][part >> 1][r] = e;
            arrive(&bars->e_fwd[pair]);
          } else {
            // after the last atom nobody waits: the phase only keeps step
            bars->e_row[1][part >> 1][r] = e;
            arrive(&bars->e_back[pair]);
          }
          ++handed;
        }
        if (!ok) break;
        if (!grad) {
          fence_before_sync();
          arrive(&bars->r0_free);
        }
        // the biases' place is free again
        arrive(&bars->bias_free);
        if (part == 3) {
          bars->e_row[2][0][r] = e;
          arrive(&bars->e_half[q]);
        }
      }
      if (grad) {
        // E4: G2 = D2 * celu'(z2)
        if (!(ok = mask_layer(R1, p.d2, p.d1))) break;
        // E5: G1 = D1 * celu'(z1)
        if (!(ok = mask_layer(R0, p.d1, 0))) break;
      }
      items.at(it, tile, m);
      g = m * p.n_species + p.tile_species[tile];
      const int tile_row = p.tile_row[tile];
      const bool whole = it < items.nwhole || M == 1;
      const int k = it - items.nwhole;  // among the CTA's items of shared tiles
      // first model of the sum this one belongs to, and the sum's slot
      const int first_shared = max(0, items.lo - (tile - items.shared0) * M);
      const int m_first = whole ? 0 : (p.apart ? m : first_shared);
      const int slot = whole ? 0 : (p.apart ? k : (tile == items.shared0 + items.lo / M ? 0 : 1));
      const bool last_here = m + 1 == M;
      // the row's energy (part 1 holds the first sum, part 3 the second)
      if (part == 1) {
        if (!(ok = wait_all(&bars->e_half[q], it & 1))) break;
        e += bars->e_row[2][0][r] + __ldg(p.b4 + g);
        if (whole) {
          e_row = fmaf(e, p.inv_models, m == 0 ? 0.f : e_row);
          if (last_here) p.e_rows[tile_row + r] = e_row;
        } else {
          p.e_part[(size_t)(items.lo + k) * BM + r] = e;
        }
      }
      // E6: dX groups.  A thread adds its 16 columns of a group to the models
      // before (in model order, kept in the CTA's scratch).  With the last
      // model of a whole tile each warp stages its 32 x 16 block in its own
      // shared-memory tile, in the 64-byte-swizzled layout of the dX tensor
      // map, and the TMA engine writes it out.
      uint8_t* stage = reinterpret_cast<uint8_t*>(xpose + (warp - 2) * 32 * kGroup);
      uint8_t* trow = stage + lane * 64;
      const F2 dxs = pack2(dx_scale, dx_scale);
      const bool out = whole && last_here;
      // laid out as the CELU' scratch
      float4* sums = reinterpret_cast<float4*>(p.xs) +
                     ((size_t)blockIdx.x * p.xs_slots + slot) * ((size_t)p.ndx * 4 * BM) + r;
      for (int r0 = 0; r0 < p.ndx && ok; r0 += kRunGroups) {
        const int ng = min(kRunGroups, p.ndx - r0);
        const uint32_t at = R1 + 128 * (runs & 1);
#pragma unroll 1
        for (int i = part; i < ng || i == part; i += 4) {
          float4 sum[4];
          float4* scratch = sums + (size_t)(r0 + i) * 4 * BM;
          if (m > m_first && i < ng) {
#pragma unroll
            for (int j = 0; j < 4; ++j) sum[j] = __ldcg(scratch + j * BM);
          }
          if (i == part && !(ok = take_acc())) break;
          if (i >= ng) break;
          float v[16];
          tmem_ld16(at + i * kGroup, v);
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
        fence_before_sync();
        arrive(&bars->dx_free[runs & 1]);
        ++runs;
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

// The tiles left over: dX and the energies of their models, which several CTAs
// of k_mlp_fused had, added in model order (or part by part, see apart).  Block
// (t, y): a tile and a dX column group, a thread four columns of a row (four
// consecutive threads hold a row's 16).  Bound by latency (a round of loads per
// eight models): a block per group keeps it to a few microseconds where one
// block per eight groups, a part after the other, took 104 us on 192 atoms x 8
// models; with every column wanted by its memory traffic (256 molecules x 8
// models, 130 MB: 59 us -> 36 with 32-bit quotients in Share).
constexpr int kJoinThreads = BM * 4;
__global__ void __launch_bounds__(kJoinThreads) k_mlp_join(const __grid_constant__ FusedParams p, int blocks) {
  pdl_wait();
  const int M = p.n_models, t0 = blockIdx.x * M;
  const Share share(p.ntiles, M, blocks);
  const int row0 = p.tile_row[share.whole * blocks + blockIdx.x];
  if (blockIdx.y == 0 && threadIdx.x < BM) {
    float e = 0.f;
    const float* part = p.e_part + (size_t)t0 * BM + threadIdx.x;
#pragma unroll 4
    for (int m = 0; m < M; ++m) e = fmaf(__ldcg(part + (size_t)m * BM), p.inv_models, e);
    p.e_rows[row0 + threadIdx.x] = e;
  }
  const int i = blockIdx.y, r = threadIdx.x >> 2, j = threadIdx.x & 3;
  if (i >= p.ndx) return;
  const float4* xs = reinterpret_cast<const float4*>(p.xs) + (size_t)(i * 4 + j) * BM + r;
  const size_t per = (size_t)p.ndx * 4 * BM;
  // slot of the k-th summand: model k, or part k (the CTAs from the tile's first on,
  // each of which has items then)
  const int c0 = share.owner(t0);
  const int n = p.apart ? M : share.owner(t0 + M - 1) - c0 + 1;
  __shared__ int slots[kJoinThreads];
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < n; k0 += kJoinThreads) {
    const int k = k0 + threadIdx.x;
    __syncthreads();
    if (k < n) {
      const int c = p.apart ? share.owner(t0 + k) : c0 + k;
      slots[threadIdx.x] = c * p.xs_slots + (p.apart ? t0 + k - share.first(c) : (share.first(c) / M == (int)blockIdx.x ? 0 : 1));
    }
    __syncthreads();
    for (int u0 = 0; u0 < min(n - k0, kJoinThreads); u0 += 8) {
      float4 t[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (k0 + u0 + u < n) t[u] = __ldcg(xs + (size_t)slots[u0 + u] * per);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (k0 + u0 + u >= n) break;
        if (k0 + u0 + u == 0) {
          v = t[0];
        } else {
          v.x += t[u].x;
          v.y += t[u].y;
          v.z += t[u].z;
          v.w += t[u].w;
        }
      }
    }
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
// Up to 16 dX column groups the models of a shared tile are kept apart, so that
// its sum does not depend on how it was shared; wider rows are summed part by
// part (kept apart, 256 molecules x 8 models would move 0.23 GB more).  Parts need
// an item for every CTA: with fewer items than CTAs those without one lie among
// the owners of a tile's items, and their slots hold something else.  There a CTA
// has one item at most, so that keeping the models apart takes no more slots.
constexpr int kApartGroups = 16;
bool models_apart(const Share& share, int ndx) { return ndx <= kApartGroups || share.most() <= 1; }
int xs_slots(const Share& share, int ndx, int n_models) {
  if (n_models == 1) return 0;
  return std::max(1, models_apart(share, ndx) ? share.most() : std::min(share.most(), 2));
}
// for any number of tiles up to `tiles`
size_t xs_bytes(int tiles, int grid, const fennol_mlp_weights* w) {
  const int M = w->n_models;
  if (M == 1 || grid == 0) return 0;
  const size_t most = tiles < sm_count() ? ((size_t)tiles * M + grid - 1) / grid : M;
  const size_t all = w->dims[0] / kGroup;
  const size_t slots = std::max(std::min(most, (size_t)2) * all, most * std::min(all, (size_t)kApartGroups));
  return (size_t)grid * slots * kGroup * BM * sizeof(float);
}
size_t e_part_bytes(int tiles, const fennol_mlp_weights* w) {
  return w->n_models > 1 ? (size_t)tiles * w->n_models * BM * sizeof(float) : 0;
}

}  // namespace

// error word, CELU' scratch on a 128-byte boundary (its L2 lines are discarded
// whole), dX sums and energies of ensembles
size_t fnl_mlp_fused_workspace(int rows, const fennol_mlp_weights* w) {
  const int grid = fused_grid(rows / BM, w->n_models);
  return 256 + 128 + dc_bytes(grid, w) + xs_bytes(rows / BM, grid, w) + e_part_bytes(rows / BM, w);
}

// The kernel, and the join of the tiles that CTAs share.
int fnl_mlp_fused_launches(int ntiles, const fennol_mlp_weights* w) {
  const Share share(ntiles, w->n_models, fused_grid(ntiles, w->n_models));
  return w->n_models > 1 && share.left > 0 ? 2 : 1;
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
  const bool wflo = f16;
  const bool wblo = precision == FENNOL_MLP_F16X3X2;
  if (f16 && (!w->wt_lo[0] || !w->wt_lo[1] || !w->wt_lo[2])) return FENNOL_ERR_INVALID;
  if (wblo && (!w->w_lo[0] || !w->w_lo[1] || !w->w_lo[2])) return FENNOL_ERR_INVALID;
  if (f16 && ((uintptr_t)w->f16_scale & 15) != 0) return FENNOL_ERR_INVALID;
  // bulk copies bring them to shared memory; a group's start is aligned where the
  // array is (widths are multiples of 64)
  if ((((uintptr_t)w->b32[0] | (uintptr_t)w->b32[1] | (uintptr_t)w->b32[2] | (uintptr_t)w->w32[3]) & 15) != 0)
    return FENNOL_ERR_INVALID;
  FusedParams p{};
  // Column lists: the L1 units with a column that may be non-zero, and which of
  // their K steps have one
  const int ngroups = d[0] / kGroup;
  for (int u = 0; u < ngroups / 2; ++u) {
    const int bits = (xg.has(2 * u) ? 1 : 0) | (xg.has(2 * u + 1) ? 2 : 0);
    if (!bits) continue;
    p.xunit[p.nunits] = (unsigned char)u;
    p.xbits[p.nunits] = (unsigned char)bits;
    ++p.nunits;
  }
  if (p.nunits == 0) return FENNOL_ERR_INVALID;
  if (dx)
    for (int g = 0; g < ngroups; ++g)
      if (dg.has(g)) p.dgroup[p.ndx++] = (unsigned char)g;
  for (int i = 0, b = 0; i < p.ndx; ++b) {
    const int left = std::min(kRunGroups - i % kRunGroups, p.ndx - i);
    int n = 1;
    while (n < left && n < 4 && p.dgroup[i + n] == p.dgroup[i] + n) ++n;
    if (n == 3) n = 2;
    p.box_g[b] = p.dgroup[i];
    p.box_n[b] = (unsigned char)n;
    i += n;
  }
  // maps of absent low parts alias the high parts (never loaded)
  const void* wtl[3] = {wflo ? w->wt_lo[0] : w->wt_hi[0], wflo ? w->wt_lo[1] : w->wt_hi[1],
                        wflo ? w->wt_lo[2] : w->wt_hi[2]};
  const void* wl[3] = {wblo ? w->w_lo[0] : w->w_hi[0], wblo ? w->w_lo[1] : w->w_hi[1],
                       wblo ? w->w_lo[2] : w->w_hi[2]};
  Maps maps;
  bool ok = map2d(&maps.x, x, rows, d[0], BM, f16, kUnit) && map2d(&maps.xlo, alo ? x_lo : x, rows, d[0], BM, f16, kUnit) &&
            map2d(&maps.w1t, w->wt_hi[0], (uint64_t)G * d[1], d[0], d[1], f16, kUnit) &&
            map2d(&maps.w1t_lo, wtl[0], (uint64_t)G * d[1], d[0], d[1], f16, kUnit) &&
            map2d(&maps.w2t, w->wt_hi[1], (uint64_t)G * d[2], d[1], d[2], f16) &&
            map2d(&maps.w3t, w->wt_hi[2], (uint64_t)G * d[3], d[2], d[3], f16) &&
            map2d(&maps.w3, w->w_hi[2], (uint64_t)G * d[2], d[3], d[2], f16) &&
            map2d(&maps.w2, w->w_hi[1], (uint64_t)G * d[1], d[2], d[1], f16) &&
            map2d(&maps.w1, w->w_hi[0], (uint64_t)G * d[0], d[1], 64, f16) &&
            map2d(&maps.w1p, w->w_hi[0], (uint64_t)G * d[0], d[1], 2 * kGroup, f16) &&
            map2d(&maps.w1g, w->w_hi[0], (uint64_t)G * d[0], d[1], kGroup, f16) &&
            map2d(&maps.w2t_lo, wtl[1], (uint64_t)G * d[2], d[1], d[2], f16) &&
            map2d(&maps.w3t_lo, wtl[2], (uint64_t)G * d[3], d[2], d[3], f16) &&
            map2d(&maps.w3_lo, wl[2], (uint64_t)G * d[2], d[3], d[2], f16) &&
            map2d(&maps.w2_lo, wl[1], (uint64_t)G * d[1], d[2], d[1], f16) &&
            map2d(&maps.w1_lo, wl[0], (uint64_t)G * d[0], d[1], 64, f16) &&
            map2d(&maps.w1p_lo, wl[0], (uint64_t)G * d[0], d[1], 2 * kGroup, f16) &&
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
  p.wb_lo = wblo ? 1 : 0;
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
  static bool attr[3] = {false, false, false};
  const int form = f16 ? kF16 : (alo ? kBf16x2 : kBf16);
  auto kern = form == kF16 ? k_mlp_fused<kF16> : (form == kBf16x2 ? k_mlp_fused<kBf16x2> : k_mlp_fused<kBf16>);
  if (!attr[form]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return FENNOL_ERR_CUDA;
    attr[form] = true;
  }
  if (ntiles <= 0) return FENNOL_OK;
  // one item per (tile, model); the CTAs share the items out evenly
  const int grid = fused_grid(ntiles, w->n_models);
  p.xs = (float*)((char*)p.dc + dc_bytes(grid, w));
  p.e_part = (float*)((char*)p.xs + xs_bytes(ntiles, grid, w));
  const Share share(ntiles, w->n_models, grid);
  p.xs_slots = xs_slots(share, p.ndx, w->n_models);
  p.apart = models_apart(share, p.ndx);
  FNL_LAUNCH_PDL(kern, dim3(grid), dim3(kThreads), smem, st, maps, p);
  FNL_CHECK_LAUNCH();
  if (w->n_models > 1 && share.left > 0) {
    FNL_LAUNCH_PDL(k_mlp_join, dim3(share.left, p.ndx > 0 ? p.ndx : 1), dim3(kJoinThreads), 0, st, p, grid);
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
