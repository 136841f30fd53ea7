// Products of a mixture of experts for many rows, bf16, 32-bit accumulators: the sums of k_rows_moe_tc.cu, with two SMs on one tile.
//
// There a CTA multiplies 128 pairs by 256 columns, and shared memory carries 96 cycles of operand reads and 96 of fills for each product of 128 tensor
// cycles.  Here a cluster of two CTAs issues one product (cta_group::2): 256 weight rows, 128 in each CTA, by up to 256 pairs of an expert, half of
// their rows in each CTA, so that a CTA's reads and fills take 64 cycles each.  Tiles hold up to 256 pairs, an expert's pairs
// cut evenly (k_rows_moe.cu's plan), and a product is as wide as its tile, in steps of 64 pairs, so that little is done for padding.
//
//   gated   act(x Wg^T, x Wu^T): 128 columns, 64 gate rows beside their 64 up rows in each CTA; the up half passes its sums through shared memory
//   single  act(x W^T), 256 columns
//   down    256 columns; every result row goes to its [row][choice]
//
// Persistent: one cluster per two SMs takes every 74th of the tiles x column blocks.  Warp 0 copies (K in steps of 64 through a ring of six stages; both
// CTAs' copies report to the first one's barriers), warp 1 of the first CTA issues the products, warps 2-5 take each CTA's 128 weight rows out of tensor
// memory, 32 pairs at a time by way of shared memory, so that results leave as whole 16-byte words of a row, under the next tile's products; of a
// gated product the gate and the up warps give each other half of their sums.  Every wait is bounded and reports through the status word; no copy is
// delivered to several CTAs.
// 32 experts, 4 per row, 4,096 wide, 2,048 (shared 4,096) inside, 4,096 rows: gated 676 -> 650 us, down 439 -> 337 (1.25 PFLOP/s); 2,000 rows 395 -> 342 and 201 -> 170.
// Ungated 2,048 / 2,304, 3,000 rows: 111 -> 96 and 113 -> 96.  Where it is taken: ops/rows.py moe_duo_takes.
#include "k_rows_tc.cuh"

namespace sfb {
namespace rmoeduo {
using namespace tc;

constexpr int THREADS = 192, COLS = 128, PAIRS = 256, STEP = 64, KS = 64, ST = 6, SLAB = 128 * 128, BOX = 32;
constexpr int DOWN = 0, GATED = 1, SINGLE = 2;

struct Args {
  const int *order, *tiles, *count;
  __nv_bfloat16 *out, *sout; // first product: [pairs, M], the shared expert's [n, SM]; down: [n, slots, M]
  int M, K, SM, SK, top, slots, act, cblocks, sblocks;     // cblocks, sblocks: blocks of 128 (gated) or 256 columns
  int stotal, stile, n;      // tiles x column blocks of the shared expert (0: none), rows of its tiles, rows
  float alpha, limit, slimit;
  Status* status;
};

struct Job {
  int4 t;                    // expert, first place (shared: row), pairs, -
  int c0, M, K, shared, N;   // N: pairs of the product
};
template <int KIND>
__device__ __forceinline__ Job job(const Args& a, int b) {
  Job j;
  j.shared = b < a.stotal;
  const int x = j.shared ? b : b - a.stotal, blocks = j.shared ? a.sblocks : a.cblocks, ti = x / blocks;
  j.t = j.shared ? make_int4(0, ti * a.stile, min(a.stile, a.n - ti * a.stile), 0) : reinterpret_cast<const int4*>(a.tiles)[ti];
  j.c0 = (x % blocks) * (KIND == GATED ? 128 : 256);
  j.M = j.shared ? a.SM : a.M;
  j.K = j.shared ? a.SK : a.K;
  j.N = (j.t.z + STEP - 1) / STEP * STEP;
  return j;
}

struct Smem {
  alignas(1024) uint8_t w[ST * SLAB];
  alignas(1024) uint8_t x[ST * SLAB];
  union {                    // two of each, in turn: 32 pairs on their way out
    alignas(16) __nv_bfloat16 res[2][32][COLS];
    struct { float half[2][2][16][64]; __nv_bfloat16 res[2][32][64]; } g;
  };
  int64_t row[2][32];
  alignas(8) uint64_t full[ST], empty[ST], acc_full[2], acc_empty[2];
  uint32_t tmem;
  int dead;
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a copy into this CTA that reports to the barrier at the same place of the pair's first CTA
__device__ __forceinline__ void load(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar) & 0xfeffffffu) : "memory");
}
__device__ __forceinline__ void mma2(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// an arrival on both CTAs' barriers when the products issued so far are done
__device__ __forceinline__ void commit2(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(b)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void arrive_first(uint64_t* b) {
  asm volatile("{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %0, 0;\n\tmbarrier.arrive.release.cluster.shared::cluster.b64 _, [r];\n\t}" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void epilogue_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
moe_duo_kernel(const __grid_constant__ CUtensorMap mx, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap msx,
               const __grid_constant__ CUtensorMap msw, Args a) {
  extern __shared__ uint8_t raw[];
  Smem& S = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int rank = (int)cluster_rank(), step = gridDim.x / 2;
  volatile int* dead = &S.dead;
  if (tid == 0) {
    S.dead = 0;
    for (int i = 0; i < ST; ++i) { mbar_init(&S.full[i], 1); mbar_init(&S.empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&S.acc_full[i], 1); mbar_init(&S.acc_empty[i], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&S.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_launch_dependents();
  fence_before();
  cluster_sync();            // both CTAs' barriers stand before the first copy
  fence_after();
  pdl_wait();
  const uint32_t tmem = S.tmem;
  const int total = a.stotal + *a.count * a.cblocks;

  if (warp == 0) {
    if (elect_one()) {
      int it = 0;            // stages filled so far
      for (int b = blockIdx.x / 2; b < total && !*dead; b += step) {
        const Job j = job<KIND>(a, b);
        const int steps = (j.K + KS - 1) / KS, half = j.N / 2;
        const int wrow = KIND == GATED ? j.t.x * 2 * j.M + j.c0 + rank * 64 : j.t.x * j.M + j.c0 + rank * 128, wrow2 = wrow + (KIND == GATED ? j.M : 64);
        const CUtensorMap *x = j.shared ? &msx : &mx, *w = j.shared ? &msw : &mw;
        int k = 0;
        for (; k < steps; ++k, ++it) {
          const int st = it % ST;
          if (!mbar_wait(&S.empty[st], ((it / ST) & 1) ^ 1, dead)) break;
          if (rank == 0) mbar_expect(&S.full[st], 2 * (SLAB + half * 128));
          load(S.w + st * SLAB, w, k * KS, wrow, &S.full[st]);
          load(S.w + st * SLAB + SLAB / 2, w, k * KS, wrow2, &S.full[st]);
          for (int r = 0; r < half; r += BOX) load(S.x + st * SLAB + r * 128, x, k * KS, j.t.y + rank * half + r, &S.full[st]);
        }
        if (k < steps) break;
      }
      if (*dead && rank == 0) {       // copies still in flight must land before the CTAs end
        for (int k = max(0, it - ST); k < it; ++k)
          for (int i = 0; i < 100000 && !mbar_try(&S.full[k % ST], (k / ST) & 1); ++i) __nanosleep(64);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t dw = desc(smem_u32(S.w), 16), dx = desc(smem_u32(S.x), 16);
      int it = 0, n = 0;
      bool ok = true;
      for (int b = blockIdx.x / 2; ok && b < total; b += step, ++n) {
        const Job j = job<KIND>(a, b);
        const int acc = n & 1, steps = (j.K + KS - 1) / KS;
        if (rank) { it += steps; continue; }
        const uint32_t id = idesc(j.N, 0, 0, 256);
        if (!(ok = mbar_wait(&S.acc_empty[acc], ((n >> 1) & 1) ^ 1, dead))) break;
        fence_after();
        for (int k = 0; k < steps; ++k, ++it) {
          const int st = it % ST;
          if (!(ok = mbar_wait(&S.full[st], (it / ST) & 1, dead))) break;
          fence_after();
          const uint64_t w = dw + (uint64_t)st * (SLAB >> 4), x = dx + (uint64_t)st * (SLAB >> 4);
#pragma unroll
          for (int q = 0; q < KS / 16; ++q) mma2(tmem + acc * PAIRS, w + q * 2, x + q * 2, id, (k | q) ? 1u : 0u);
          commit2(&S.empty[st]);
        }
        if (ok) commit2(&S.acc_full[acc]);
      }
      // no arrival may be under way when a CTA ends
      for (int k = max(0, it - ST); ok && k < it; ++k) ok = mbar_wait(&S.empty[k % ST], (k / ST) & 1, dead);
    }
  } else {
    const int w4 = warp & 3, t = (warp - 2) * 32 + lane;
    const uint32_t lanes = (uint32_t)(w4 * 32) << 16;      // tensor memory lanes of this warp: weight rows
    int n = 0, turn = 0;
    for (int b = blockIdx.x / 2; b < total; b += step, ++n) {
      const Job j = job<KIND>(a, b);
      const int acc = n & 1;
      constexpr int WORDS = KIND == GATED ? 8 : 16;        // of 16 bytes in a result row of this CTA
      const int col = j.c0 + rank * (KIND == GATED ? 64 : 128);
      __nv_bfloat16* out = KIND != DOWN && j.shared ? a.sout : a.out;
      const float limit = j.shared ? a.slimit : a.limit;
      const bool ok = mbar_wait(&S.acc_full[acc], (n >> 1) & 1, dead);
      if (!__all_sync(0xffffffffu, ok)) break;
      fence_after();
      const uint32_t ta = tmem + acc * PAIRS + lanes;
      float f[32], next[32];
      ld32(ta, next);
      for (int c = 0; c < j.t.z; c += 32, turn ^= 1) {
        if (w4 == 0) {
          int64_t row = -1;
          const int p = j.t.y + c + lane;
          if (c + lane < j.t.z) {
            if (KIND != DOWN) row = p;
            else if (j.shared) row = (int64_t)p * a.slots + a.top;
            else { const int pair = a.order[p]; row = (int64_t)(pair / a.top) * a.slots + pair % a.top; }
          }
          S.row[turn][lane] = row;
        }
        wait_ld();
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = next[i];
        if (c + 32 < j.t.z) {
          ld32(ta + c + 32, next);                            // under this one's way out
        } else {                                              // the accumulator is read
          fence_before();
          if (lane == 0) arrive_first(&S.acc_empty[acc]);
        }
        if constexpr (KIND == GATED) {
          // gate rows in warps with w4 < 2, up rows in the others: each gives the other its sums of sixteen pairs and makes the rest
          const int r = (w4 & 1) * 32 + lane;
          float(*mine)[64] = S.g.half[turn][w4 >> 1], (*other)[64] = S.g.half[turn][(w4 >> 1) ^ 1];
          if (w4 < 2) {
#pragma unroll
            for (int i = 0; i < 16; ++i) mine[i][r] = f[16 + i];
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) mine[i][r] = f[i];
          }
          epilogue_sync();
          if (w4 < 2) {
#pragma unroll
            for (int i = 0; i < 16; ++i) S.g.res[turn][i][r] = __float2bfloat16_rn(rows::gate_clamp<__nv_bfloat16>(f[i], other[i][r], a.alpha, limit));
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) S.g.res[turn][16 + i][r] = __float2bfloat16_rn(rows::gate_clamp<__nv_bfloat16>(other[i][r], f[16 + i], a.alpha, limit));
          }
        } else {
          if constexpr (KIND == SINGLE) {
            if (a.act == rows::ACT_RELU2) {
#pragma unroll
              for (int k = 0; k < 32; ++k) { const float p = fmaxf(f[k], 0.f); f[k] = p * p; }
            } else {
#pragma unroll
              for (int k = 0; k < 32; ++k) f[k] = rows::act_single<__nv_bfloat16>(f[k], rows::ACT_XIELU, a.alpha, limit);
            }
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) S.res[turn][i][w4 * 32 + lane] = __float2bfloat16_rn(f[i]);
        }
        epilogue_sync();       // (what the next 32 pairs write lies in the other half, and they meet at a barrier before the ones after them)
#pragma unroll
        for (int k = 0; k < 32 * WORDS / 128; ++k) {
          const int i = (t + k * 128) / WORDS, word = (t + k * 128) % WORDS;
          const int64_t row = S.row[turn][i];
          const __nv_bfloat16* res = KIND == GATED ? S.g.res[turn][i] : S.res[turn][i];
          if (row >= 0 && col + word * 8 < j.M)               // M is a multiple of eight
            *reinterpret_cast<uint4*>(out + row * j.M + col + word * 8) = *reinterpret_cast<const uint4*>(res + word * 8);
        }
      }
    }
  }
  __syncwarp();
  fence_before();
  cluster_sync();            // nothing of a CTA may be under way in the other when it ends
  if (tid == 0 && *dead) status_set(a.status, ST_TIMEOUT, 79, blockIdx.x, KIND);
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

template <int KIND>
static int launch(const CUtensorMap* mx, const CUtensorMap* mw, const CUtensorMap* msx, const CUtensorMap* msw, const Args& a, int most, cudaStream_t st) {
  const size_t smem = sizeof(Smem) + 1024;
  static bool done = false;
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(moe_duo_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long jobs = (long long)most * a.cblocks + a.stotal;
  return (int)sfb_launch(moe_duo_kernel<KIND>, dim3(2 * (unsigned)(jobs < sms / 2 ? jobs : sms / 2)), dim3(THREADS), smem, st, *mx, *mw, *msx, *msw, a);
}

}  // namespace rmoeduo
}  // namespace sfb

using namespace sfb;
using namespace sfb::rmoeduo;

extern "C" {

// mx: rows [pairs, K] in plan order (tiles of up to 256 pairs), box 32 rows; mw: weights [E (2) M, K], box 64 rows.  msx, msw: the same of the shared
// expert (rows in order), or null.  The rest as sfb_rows_moe_gemm.
int sfb_rows_moe_duo(const void* mx, const void* mw, const void* msx, const void* msw, const void* order, const void* tiles, const void* count, void* out, void* sout,
                     int most, int n, int M, int K, int SM, int SK, int top, int slots, int act, float alpha, float limit, float slimit, void* status,
                     cudaStream_t stream) {
  if (most < 1 || n < 1 || M < 8 || M % 8 || K < 8 || K % 8 || top < 1 || (act && act != rows::ACT_CLAMP && act != rows::ACT_RELU2 && act != rows::ACT_XIELU) ||
      (msx && (SM < 8 || SM % 8 || SK < 8 || SK % 8 || slots <= top)) || (uintptr_t)out % 16 || (uintptr_t)sout % 16)
    return (int)cudaErrorInvalidValue;
  const int per = act == rows::ACT_CLAMP ? 128 : 256, stiles = (n + PAIRS - 1) / PAIRS;
  Args a{(const int*)order, (const int*)tiles, (const int*)count, (__nv_bfloat16*)out, (__nv_bfloat16*)sout, M, K, SM, SK, top, slots, act, (M + per - 1) / per,
         (SM + per - 1) / per, 0, ((n + stiles - 1) / stiles + STEP - 1) / STEP * STEP, n, alpha, limit, slimit, (Status*)status};
  if (msx) a.stotal = (n + a.stile - 1) / a.stile * a.sblocks;
  const CUtensorMap *x = (const CUtensorMap*)mx, *w = (const CUtensorMap*)mw, *sx = msx ? (const CUtensorMap*)msx : x, *sw = msw ? (const CUtensorMap*)msw : w;
  if (act == rows::ACT_CLAMP) return launch<GATED>(x, w, sx, sw, a, most, stream);
  if (act) return launch<SINGLE>(x, w, sx, sw, a, most, stream);
  return launch<DOWN>(x, w, sx, sw, a, most, stream);
}

}  // extern "C"
