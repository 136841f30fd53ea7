// CSA2 sparse-MLA attention for the rows step: every (row, head) attends the causal window
// (FP8 ring, one UE8M0 scale per 32) followed by the selected compressed entries (FP4 with an E4M3
// scale per 16) of the layer that owns the compressed cache.  One latent KV row serves as key and
// value for all heads.  Online softmax; the per-head sink enters the denominator only; the query
// RoPE is applied on load and the inverse RoPE on the output's rope slice.
//
// Reference behaviour: kernels/opt_attn_sm121.cu:96 (opt_flash_mla_csa2_seq), kernels/opt_rows_sm121.cu
// attn:1097, kernels/flash_mla_csa2_common_sm121.cuh; docs/architecture/01-csa2-attention.md:98-104,212-229.
#include <cooperative_groups.h>

#include "k_cache_bf16.cuh"

namespace cg = cooperative_groups;

namespace sfb {

struct AttnArgs {
  const __nv_bfloat16* q;   // [n, q_stride]; head h at h*hd
  int64_t q_stride;
  const float2* rope;       // [n, rope_stride]: (cos, sin) of the row's position
  int rope_stride;
  const int* row_lane;
  const int* row_pos;
  const uint8_t* win_q;     // [lanes, ring, hd]
  const uint8_t* win_s;     // [lanes, ring, hd/32]
  int64_t win_lane_q, win_lane_s;
  const uint8_t* ckv_q;     // [lanes, max_entries, hd/2] (null when the layer has no compressed path)
  const uint8_t* ckv_s;     // [lanes, max_entries, hd/16]
  int64_t ckv_lane_q, ckv_lane_s;
  const int* sel;           // [n, K] ascending ids, -1 padded
  const int* sel_count;     // [n]
  int K;
  const float* sink;        // [heads]
  __nv_bfloat16* out;       // [n, heads*hd]
  uint8_t* out_q;           // optional two-term FP8 copy for the tensor-core arm: rows [0,n) hi, [n,2n) lo
  uint8_t* out_atom;        // its scale atoms (rows = hi rows then lo rows)
  int n, heads, rd, window, ring;
  float scale;
  // optional explicit window per row: positions [win_lo[row], win_hi[row]] of the ring instead of the causal window that
  // ends at the row's own position (draft blocks attend their whole block: no causal mask inside it)
  const int* win_lo;
  const int* win_hi;
  int wide_q, wide_out;     // query rows start on 16-byte boundaries; output rows on 4-byte (bf16) and 2-byte (FP8) ones
};

constexpr int AT_HPB = 8;       // heads per block
constexpr int AT_SPLITS = 8;    // CTAs of one cluster share a (row, head group); each takes 1/8 of the entries
constexpr int AT_EC = 80;       // entries staged at once: an eighth of a 128-entry window and 512 selected entries
constexpr int AT_THREADS = 4 * AT_EC;
template <int HD> __host__ __device__ constexpr int at_row() { return HD * 2 + (HD == 512 ? 64 : 0); }      // bytes of a staged entry
// Byte of 16-byte piece `c` of a staged entry.  With HD = 512 a lane's share of a dot product is two pieces: the even and the odd ones lie apart,
// so that neighbouring lanes read neighbouring banks, and 64 bytes more, so that neighbouring pieces also lie in different ones.
template <int HD> __device__ __forceinline__ int at_piece(int c) {
  if constexpr (HD == 512) return (c & 1) * (HD + 64) + (c >> 1) * 16;
  else return c * 16;
}
template <int HD> __host__ __device__ constexpr int at_qlane() { return HD / 32 * AT_HPB * 4 + 16; }   // bytes of one lane's query elements, eight heads each
template <int HD> __host__ __device__ constexpr size_t at_smem() {
  return (size_t)AT_EC * at_row<HD>() + 32 * at_qlane<HD>() + (2 * AT_EC * AT_HPB + AT_EC / 4 * AT_HPB + 2 * AT_HPB) * sizeof(float);
}

// two floats in one 64-bit register; every operation rounds each of them as the scalar instruction does
__device__ __forceinline__ uint64_t pack2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

// grid (AT_SPLITS, head groups of 8, n) in clusters of AT_SPLITS.  A CTA requests its share of the row's KV entries at once - up to 80, every load in
// flight before the first is used - and keeps them in shared memory as bf16, which holds them exactly (k_cache_bf16.cuh).  Everything after
// that is 32-bit in one fixed order - a dot product is 32 shares of HD / 32 elements, added as a butterfly over the shares; the softmax runs
// over groups of four entries - but each part is spread as it suits the machine:
//   scores   lane = share, a warp per four entries: sixteen sums of two heads each in packed instructions, one pass over the queries in shared
//            memory; at each level of the butterfly a lane gives half of its sums away, so that 31 shuffles leave one sum in each lane
//   softmax  a warp per head, a lane per group: the running maximum is a scan, and only the denominator is a chain
//   values   thread = four dims of four heads
// The partial (max, sum, accumulator) of every head stays in shared memory, and after a cluster barrier CTA rank h merges head h across the eight
// CTAs in rank order through distributed shared memory - no global scratch, no atomics.  The split is a function of the row alone, so a
// row's bits do not depend on the batch.
// One row is bound by latency (ids, then codes; barriers; the merge), sixteen by the issue of the products.  640 entries, 64 heads, rows 4 / 16 / 64:
// 25 / 93 / 334 us.  A rank with fewer heads has fewer CTAs and is no worse off than with four heads in each: L2 flushed, 1 / 16 / 64 rows, eight heads 23 / 31 / 57 us
// against 47 / 49 / 107, sixteen 23 / 33 / 104 against 45 / 55 / 199, four 23 / 31 / 56 against 45 / 49 / 59.
template <int HD>
__global__ void __cluster_dims__(AT_SPLITS, 1, 1) __launch_bounds__(AT_THREADS, 2) attn_rows_kernel(AttnArgs a) {
  constexpr int EPL = HD / 32;          // elements per share
  constexpr int TPE = HD / 32;          // threads that decode one entry (32 elements each)
  constexpr int NI = (AT_EC * TPE + AT_THREADS - 1) / AT_THREADS;
  constexpr int KB = at_row<HD>(), QB = at_qlane<HD>();
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) uint8_t smem[];
  uint8_t* kv = smem;                                                      // [EC] rows of bf16
  uint8_t* qs = kv + AT_EC * KB;                                           // [32 shares][EPL][8 heads] fp32
  float* sc = reinterpret_cast<float*>(qs + 32 * QB);                      // [8][EC] dot products
  float* ps = sc + AT_HPB * AT_EC;                                         // [EC][8] probabilities
  float* cs = ps + AT_HPB * AT_EC;                                         // [EC / 4][8] rescale before the group
  float* part_m = cs + AT_EC / 4 * AT_HPB;                                 // [8] maxima, [8] sums of this CTA's entries
  float* part_l = part_m + AT_HPB;
  float* part = reinterpret_cast<float*>(kv);                              // [8][HD] accumulators, once the entries are used up
  const int sp = blockIdx.x, hg = blockIdx.y, row = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch_dependents();
  pdl_wait();
  const int pos = a.row_pos[row], L = a.row_lane[row];
  const int r0 = HD - a.rd;
  const int w_first = a.win_lo ? a.win_lo[row] : (pos - a.window + 1 > 0 ? pos - a.window + 1 : 0);
  const int n_win = (a.win_hi ? a.win_hi[row] : pos) - w_first + 1;
  const int n_sel = a.ckv_q ? a.sel_count[row] : 0;
  const int total = n_win + n_sel;
  const int e_lo = (int)((int64_t)total * sp / AT_SPLITS), e_hi = (int)((int64_t)total * (sp + 1) / AT_SPLITS);
  float m_run = -1e30f, l_run = 0.f;                             // of head `warp`
  constexpr int DG = HD / 4;
  const int dg = tid % DG, hh4 = tid / DG;                       // values: dims 4 dg.., heads 4 hh4..
  uint64_t acc[4][2];                                            // dims, pairs of heads
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0;

#pragma unroll 1
  for (int base = e_lo; base < e_hi; base += AT_EC) {
    const int cnt = e_hi - base < AT_EC ? e_hi - base : AT_EC, groups = (cnt + 3) >> 2;
    // ---- every load of the chunk ----
    int id[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int el = (tid + i * AT_THREADS) / TPE, e = base + el;
      id[i] = el < cnt ? (e < n_win ? (w_first + e) % a.ring : a.sel[(size_t)row * a.K + (e - n_win)]) : 0;
    }
    uint4 raw0[NI], raw1[NI];
    uint32_t scl[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int el = (tid + i * AT_THREADS) / TPE, prt = (tid + i * AT_THREADS) % TPE;
      if (el >= cnt) continue;
      if (base + el < n_win) {
        const uint8_t* kq = a.win_q + (size_t)L * a.win_lane_q + (size_t)id[i] * HD + prt * 32;
        raw0[i] = *reinterpret_cast<const uint4*>(kq);
        raw1[i] = *reinterpret_cast<const uint4*>(kq + 16);
        scl[i] = a.win_s[(size_t)L * a.win_lane_s + (size_t)id[i] * (HD / 32) + prt];
      } else {
        raw0[i] = *reinterpret_cast<const uint4*>(a.ckv_q + (size_t)L * a.ckv_lane_q + (size_t)id[i] * (HD / 2) + prt * 16);
        const uint8_t* ks = a.ckv_s + (size_t)L * a.ckv_lane_s + (size_t)id[i] * (HD / 16) + prt * 2;
        scl[i] = (uint32_t)ks[0] | ((uint32_t)ks[1] << 8);
      }
    }
    if (base == e_lo) {
      // ---- queries of the group's heads, rope on the last rd dims; heads past the last one are zero ----
      for (int i = tid; i < AT_HPB * HD / 8; i += AT_THREADS) {
        const int hh = i / (HD / 8), c = i % (HD / 8), head = hg * AT_HPB + hh;
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        const bool head_ok = head < a.heads;
        if (head_ok) {
          const __nv_bfloat16* src = a.q + (size_t)row * a.q_stride + (size_t)head * HD + c * 8;
          if (a.wide_q) {
            const uint4 v = *reinterpret_cast<const uint4*>(src);
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = (uint32_t)__bfloat16_as_ushort(src[2 * j]) | ((uint32_t)__bfloat16_as_ushort(src[2 * j + 1]) << 16);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x = __uint_as_float(w[j] << 16), y = __uint_as_float(w[j] & 0xffff0000u);
          const int dim = c * 8 + 2 * j;
          if (dim >= r0 && head_ok) {
            const float2 c2 = a.rope[(size_t)row * a.rope_stride + ((dim - r0) >> 1)];
            const float x0 = x, y0 = y;
            x = bfr(__fmaf_rn(x0, c2.x, -__fmul_rn(y0, c2.y)));      // which product is rounded first decides ties: spelled out
            y = bfr(__fmaf_rn(x0, c2.y, __fmul_rn(y0, c2.x)));
          }
          float* d = reinterpret_cast<float*>(qs + dim / EPL * QB) + dim % EPL * AT_HPB + hh;
          d[0] = x;
          d[AT_HPB] = y;      // EPL is even: the pair lies in one share
        }
      }
    }
    // ---- entries to bf16; zeros up to the end of the last group ----
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int el = (tid + i * AT_THREADS) / TPE, prt = (tid + i * AT_THREADS) % TPE;
      if (el >= groups * 4) continue;
      uint4 o[4];
      if (el >= cnt) {
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = make_uint4(0u, 0u, 0u, 0u);
      } else if (base + el < n_win) {
        const uint32_t m = ue8m0_splat((uint8_t)scl[i]);
        fp8x16_to_bf16(raw0[i], m, o[0], o[1]);
        fp8x16_to_bf16(raw1[i], m, o[2], o[3]);
      } else {
        uint32_t s0, s1;
        e4m3x2_splat((uint16_t)scl[i], s0, s1);
        o[0] = fp4x8_to_bf16(raw0[i].x, s0); o[1] = fp4x8_to_bf16(raw0[i].y, s0);
        o[2] = fp4x8_to_bf16(raw0[i].z, s1); o[3] = fp4x8_to_bf16(raw0[i].w, s1);
      }
      const bool turn = HD == 512 && (prt & 4);      // of eight neighbouring threads the second four store their later pieces first: eight different bank groups
      uint8_t* dst = kv + el * KB;
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(dst + at_piece<HD>(prt * 4 + (turn ? j ^ 2 : j))) = turn ? o[j ^ 2] : o[j];
    }
    __syncthreads();
    // ---- scores: lane = share, four entries at a time ----
#pragma unroll 1
    for (int g = warp; g < groups; g += AT_THREADS / 32) {
      uint64_t s[4][4];      // entry, pair of heads
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) s[u][i] = 0;
      const uint8_t* kp = kv + g * 4 * KB;
      const uint8_t* qp = qs + lane * QB;
#pragma unroll 1
      for (int j0 = 0; j0 < EPL; j0 += 8) {
        constexpr int W = EPL < 8 ? EPL / 2 : 4;
        uint32_t w[4][W];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if constexpr (EPL == 16) {
            const uint4 x = *reinterpret_cast<const uint4*>(kp + u * KB + at_piece<HD>(2 * lane + j0 / 8));
            w[u][0] = x.x; w[u][1] = x.y; w[u][2] = x.z; w[u][3] = x.w;
          } else {
#pragma unroll
            for (int i = 0; i < W; ++i) w[u][i] = reinterpret_cast<const uint32_t*>(kp + u * KB + lane * EPL * 2)[i];
          }
        }
#pragma unroll
        for (int j = 0; j < 2 * W; ++j) {
          const ulonglong2 qa = *reinterpret_cast<const ulonglong2*>(qp + (j0 + j) * 32), qb = *reinterpret_cast<const ulonglong2*>(qp + (j0 + j) * 32 + 16);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float x = __uint_as_float(j & 1 ? w[u][j / 2] & 0xffff0000u : w[u][j / 2] << 16);
            const uint64_t xx = pack2(x, x);
            s[u][0] = fma2(qa.x, xx, s[u][0]); s[u][1] = fma2(qa.y, xx, s[u][1]); s[u][2] = fma2(qb.x, xx, s[u][2]); s[u][3] = fma2(qb.y, xx, s[u][3]);
          }
        }
      }
      float d[32];           // entry * 8 + head
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < 4; ++i) unpack2(s[u][i], d[u * 8 + 2 * i], d[u * 8 + 2 * i + 1]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;      // keeps the upper half of its sums
#pragma unroll
        for (int i = 0; i < o; ++i) {
          const float mine = up ? d[i + o] : d[i], other = up ? d[i] : d[i + o];
          d[i] = mine + __shfl_xor_sync(0xffffffffu, other, o);
        }
      }
      sc[(lane & 7) * AT_EC + g * 4 + (lane >> 3)] = d[0];
    }
    __syncthreads();
    // ---- softmax: warp = head, lane = group of four entries ----
    if (warp < AT_HPB) {
      float d[4], x = m_run;
      const bool any = lane < groups;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        d[u] = any && lane * 4 + u < cnt ? __fmul_rn(sc[warp * AT_EC + lane * 4 + u], a.scale) : -INFINITY;
        x = fmaxf(x, d[u]);
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const float y = __shfl_up_sync(0xffffffffu, x, o); if (lane >= o) x = fmaxf(x, y); }
      float before = __shfl_up_sync(0xffffffffu, x, 1);
      if (lane == 0) before = m_run;
      const float corr = __expf(before - x);
#pragma unroll
      for (int u = 0; u < 4; ++u) d[u] = __expf(d[u] - x);
      const float sum = (d[0] + d[1]) + (d[2] + d[3]);
      if (any) {
#pragma unroll
        for (int u = 0; u < 4; ++u) ps[(lane * 4 + u) * AT_HPB + warp] = d[u];
        cs[lane * AT_HPB + warp] = corr;
      }
#pragma unroll 4
      for (int g = 0; g < groups; ++g) l_run = fmaf(l_run, __shfl_sync(0xffffffffu, corr, g), __shfl_sync(0xffffffffu, sum, g));
      m_run = __shfl_sync(0xffffffffu, x, groups - 1);
    }
    __syncthreads();
    // ---- values: thread = four dims of four heads ----
    if (tid < 2 * DG) {
      const uint8_t* kp = kv + at_piece<HD>(dg >> 1) + (dg & 1) * 8;
#pragma unroll 1
      for (int g = 0; g < groups; ++g) {
        uint64_t p[4][2];
        uint2 w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          w[u] = *reinterpret_cast<const uint2*>(kp + (g * 4 + u) * KB);
          const ulonglong2 pa = *reinterpret_cast<const ulonglong2*>(ps + (g * 4 + u) * AT_HPB + hh4 * 4);
          p[u][0] = pa.x; p[u][1] = pa.y;
        }
        const ulonglong2 ca = *reinterpret_cast<const ulonglong2*>(cs + g * AT_HPB + hh4 * 4);
        const uint64_t corr[2] = {ca.x, ca.y};
#pragma unroll
        for (int dd = 0; dd < 4; ++dd) {
          uint64_t k2[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint32_t v = dd < 2 ? w[u].x : w[u].y;
            const float x = __uint_as_float(dd & 1 ? v & 0xffff0000u : v << 16);
            k2[u] = pack2(x, x);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            acc[dd][i] = fma2(acc[dd][i], corr[i], add2(fma2(p[0][i], k2[0], mul2(p[1][i], k2[1])), fma2(p[2][i], k2[2], mul2(p[3][i], k2[3]))));
        }
      }
    }
    __syncthreads();                     // the entries are used up
  }
  // ---- partial of this CTA, visible to the cluster ----
  if (tid < 2 * DG) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float x[4], y[4];
#pragma unroll
      for (int dd = 0; dd < 4; ++dd) unpack2(acc[dd][i], x[dd], y[dd]);
      float* d = part + (hh4 * 4 + 2 * i) * HD + dg * 4;
      *reinterpret_cast<float4*>(d) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(d + HD) = make_float4(y[0], y[1], y[2], y[3]);
    }
  }
  if (lane == 0 && warp < AT_HPB) { part_m[warp] = m_run; part_l[warp] = l_run; }
  cluster.sync();
  // ---- CTA rank h merges head h over the eight CTAs in rank order, two dims per thread ----
  const int mh = sp, ghead = hg * AT_HPB + mh;
  if (ghead < a.heads && tid < HD / 2) {
    const int e = tid * 2;
    float ms[AT_SPLITS], ls[AT_SPLITS], mt = -1e30f;
    float2 av[AT_SPLITS];
#pragma unroll
    for (int r = 0; r < AT_SPLITS; ++r) {
      ms[r] = cluster.map_shared_rank(part_m, r)[mh];
      ls[r] = cluster.map_shared_rank(part_l, r)[mh];
      av[r] = *reinterpret_cast<const float2*>(cluster.map_shared_rank(part, r) + mh * HD + e);
    }
#pragma unroll
    for (int r = 0; r < AT_SPLITS; ++r) mt = fmaxf(mt, ms[r]);
    float den = __expf(a.sink[ghead] - mt);
    float o[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < AT_SPLITS; ++r) {
      const float wgt = __expf(ms[r] - mt);
      den += ls[r] * wgt;
      o[0] += av[r].x * wgt;
      o[1] += av[r].y * wgt;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) o[j] = bfr(o[j] / den);
    if (e >= r0) {      // inverse rope
      const float2 c2 = a.rope[(size_t)row * a.rope_stride + ((e - r0) >> 1)];
      const float x = o[0], y = o[1];
      o[0] = bfr(__fmaf_rn(x, c2.x, __fmul_rn(y, c2.y)));
      o[1] = bfr(__fmaf_rn(y, c2.x, -__fmul_rn(x, c2.y)));
    }
    const size_t Wd = (size_t)a.heads * HD, c = (size_t)ghead * HD + e;
    __nv_bfloat16* op = a.out + (size_t)row * Wd + c;
    if (a.wide_out) *reinterpret_cast<__nv_bfloat162*>(op) = __floats2bfloat162_rn(o[0], o[1]);
    else { op[0] = __float2bfloat16_rn(o[0]); op[1] = __float2bfloat16_rn(o[1]); }
    if (a.out_q) {
      float amax = fmaxf(fabsf(o[0]), fabsf(o[1]));
#pragma unroll
      for (int ofs = 1; ofs < 16; ofs <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, ofs));      // sixteen lanes hold a 32-group
      const uint8_t scode = act_scale_code_fp8(amax);
      const float inv = bits_f32(((uint32_t)(254 - scode)) << 23);
      const uint16_t hi = enc_e4m3x2(o[0] * inv, o[1] * inv);
      const float2 dq = cvt_e4m3x2(hi);
      const uint16_t lo = enc_e4m3x2((o[0] * inv - dq.x) * 16.f, (o[1] * inv - dq.y) * 16.f);
      uint8_t *qh = a.out_q + (size_t)row * Wd + c, *ql8 = a.out_q + (size_t)(a.n + row) * Wd + c;
      if (a.wide_out) {
        *reinterpret_cast<uint16_t*>(qh) = hi;
        *reinterpret_cast<uint16_t*>(ql8) = lo;
      } else {
        qh[0] = (uint8_t)hi; qh[1] = (uint8_t)(hi >> 8);
        ql8[0] = (uint8_t)lo; ql8[1] = (uint8_t)(lo >> 8);
      }
      if ((tid & 15) == 0) {
        const int KB = a.heads * HD / 32, kb = ghead * (HD / 32) + e / 32;
        a.out_atom[sf_offset(row, kb, KB)] = scode;
        a.out_atom[sf_offset(a.n + row, kb, KB)] = scode >= 4 ? (uint8_t)(scode - 4) : (uint8_t)0;
      }
    }
  }
  cluster.sync();  // nobody leaves while its shared memory may still be read
}

}  // namespace sfb

using namespace sfb;

extern "C" {

int sfb_attn_rows_range(const void* q, int64_t q_stride, const void* rope, int rope_stride, const int* row_lane,
                        const int* row_pos, const void* win_q, const void* win_s, int64_t win_lane_q,
                        int64_t win_lane_s, const void* ckv_q, const void* ckv_s, int64_t ckv_lane_q,
                        int64_t ckv_lane_s, const int* sel, const int* sel_count, int K, const float* sink,
                        void* out, void* out_q, void* out_atom, int n, int heads, int hd, int rd, int window, int ring,
                        float scale, const int* win_lo, const int* win_hi, cudaStream_t stream);

int sfb_attn_rows(const void* q, int64_t q_stride, const void* rope, int rope_stride, const int* row_lane,
                  const int* row_pos, const void* win_q, const void* win_s, int64_t win_lane_q,
                  int64_t win_lane_s, const void* ckv_q, const void* ckv_s, int64_t ckv_lane_q,
                  int64_t ckv_lane_s, const int* sel, const int* sel_count, int K, const float* sink,
                  void* out, void* out_q, void* out_atom, int n, int heads, int hd, int rd, int window, int ring,
                  float scale, cudaStream_t stream) {
  return sfb_attn_rows_range(q, q_stride, rope, rope_stride, row_lane, row_pos, win_q, win_s, win_lane_q, win_lane_s, ckv_q, ckv_s,
                             ckv_lane_q, ckv_lane_s, sel, sel_count, K, sink, out, out_q, out_atom, n, heads, hd, rd, window, ring,
                             scale, nullptr, nullptr, stream);
}

int sfb_attn_rows_range(const void* q, int64_t q_stride, const void* rope, int rope_stride, const int* row_lane,
                        const int* row_pos, const void* win_q, const void* win_s, int64_t win_lane_q,
                        int64_t win_lane_s, const void* ckv_q, const void* ckv_s, int64_t ckv_lane_q,
                        int64_t ckv_lane_s, const int* sel, const int* sel_count, int K, const float* sink,
                        void* out, void* out_q, void* out_atom, int n, int heads, int hd, int rd, int window, int ring,
                        float scale, const int* win_lo, const int* win_hi, cudaStream_t stream) {
  if ((hd / 32) % 2) return (int)cudaErrorInvalidValue;
  const int wide_q = ((uintptr_t)q % 16 == 0 && q_stride % 8 == 0) ? 1 : 0;
  const int wide_out = ((uintptr_t)out % 4 == 0 && (uintptr_t)out_q % 2 == 0) ? 1 : 0;
  AttnArgs a{(const __nv_bfloat16*)q, q_stride, (const float2*)rope, rope_stride, row_lane, row_pos, (const uint8_t*)win_q,
             (const uint8_t*)win_s, win_lane_q, win_lane_s, (const uint8_t*)ckv_q, (const uint8_t*)ckv_s,
             ckv_lane_q, ckv_lane_s, sel, sel_count, K, sink, (__nv_bfloat16*)out, (uint8_t*)out_q, (uint8_t*)out_atom,
             n, heads, rd, window, ring, scale, win_lo, win_hi, wide_q, wide_out};
  dim3 grid(AT_SPLITS, (heads + AT_HPB - 1) / AT_HPB, n);
  cudaError_t launch_rc = cudaSuccess;
#define SFB_AT(HDV)                                                                                         \
  {                                                                                                         \
    static bool done = false;                                                                               \
    if (!done) {                                                                                            \
      cudaFuncSetAttribute(attn_rows_kernel<HDV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)at_smem<HDV>());  \
      done = true;                                                                                          \
    }                                                                                                       \
    launch_rc = sfb_launch(attn_rows_kernel<HDV>, grid, dim3(AT_THREADS), at_smem<HDV>(), stream, a);                \
  }
  if (hd == 512) SFB_AT(512) else if (hd == 64) SFB_AT(64) else if (hd == 128) SFB_AT(128)
  else return (int)cudaErrorInvalidValue;
#undef SFB_AT
  return (int)launch_rc;
}

}  // extern "C"
