// Seam of the layered decoders for many rows, bf16 activations: the sums of k_rows.cu's seam_kernel, bit for bit, with the rows moved through shared memory.
//
// Bound by memory.  A block per row loads, reduces and stores one after the other, and its loads stand still meanwhile.  Here one persistent CTA per
// SM walks over its rows: warp 0 brings them into a ring of stages by bulk copies (residual, output or its parts), groups of warps take a row each -
// every weight once in shared memory, requested before the previous kernel has finished - and write the new residual and h over what they read,
// and warp 1 sends these out and frees the stage.  A stage is on its way in, in work or on its way out, so copies do not wait for sums; three groups of
// 256 threads (d = 4,096; more and smaller ones below) keep up with them, one or two do not (78 and 51 us for 44).  Every wait is bounded
// and reports through the status word.
// Alone, caches emptied, us (floor at the copy rate): 4,096 x 4,096 layer norms 56 -> 44 (31), RMS norm after a scale 49 -> 37 (31), merged branches 82 -> 66 (36), five
// parts 93 -> 75 (51; three stages fit); 4,096 x 2,048 34 -> 27 (15), 47 -> 34 (18) and 52 -> 34 (26); 600 x 4,096 20 -> 16, 300 x 2,048 14 -> 11.  Narrow rows
// have too little to move for the way through shared memory: 4,096 x 1,024 29 -> 25, 600 x 1,024 11 -> 12, 4,096 x 264 17 -> 24.
#include "k_rows_seam.cuh"
#include "k_rows_tc.cuh"

namespace sfb {
namespace rows {

constexpr int MANY_MAX_STAGES = 12, MANY_MAX_GROUPS = 12, MANY_NV = 4, MANY_SMEM = 224 * 1024;

struct SeamMany {
  SeamArgs a;
  int n, stages, groups, threads;          // threads: of a group
  uint32_t load, stage, weights;           // bytes of a row's loads, of a stage, of all weights
};

struct ManyBars {
  alignas(8) uint64_t full[MANY_MAX_STAGES], done[MANY_MAX_STAGES], empty[MANY_MAX_STAGES], weights;
  alignas(16) float sums[MANY_MAX_GROUPS][2][3 * 8];
  int dead;
};

__device__ __forceinline__ void bulk_in(uint8_t* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_out(void* dst, const uint8_t* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(tc::smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void group_sync(int group, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(threads) : "memory"); }

// Eight numbers that the warps left (zeros where there are fewer), read at once and added up in the order of the warps.
__device__ __forceinline__ float sum8(const float* s) {
  const float4 a = *reinterpret_cast<const float4*>(s), b = *reinterpret_cast<const float4*>(s + 4);
  return (((((((0.f + a.x) + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
}
// The moments of row_moments (k_rows.cu) over a group of warps; s: two halves, successive calls take turns.
template <int NV>
__device__ __forceinline__ void group_moments(const float (&x)[NV][4], int c0, int step, int d, float wcnt, float winv, float inv_d, float* s, int warps, int w, int lane, int group,
                                              float& mu, float& m2) {
  float t = 0.f, q = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (c0 + i * step < d) {
#pragma unroll
      for (int k = 0; k < 4; ++k) t += x[i][k];
    }
  const float wm = warp_sum(t) * winv;
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (c0 + i * step < d) {
#pragma unroll
      for (int k = 0; k < 4; ++k) { const float e = x[i][k] - wm; q += e * e; }
    }
  q = warp_sum(q);
  if (lane == 0) { s[w] = wm; s[8 + w] = q; s[16 + w] = wcnt; }
  group_sync(group, warps * 32);
  const float4 m0 = *reinterpret_cast<const float4*>(s), m1 = *reinterpret_cast<const float4*>(s + 4);
  const float4 k0 = *reinterpret_cast<const float4*>(s + 16), k1 = *reinterpret_cast<const float4*>(s + 20);
  const float mi = s[lane & 7], vi = s[8 + (lane & 7)], ci = s[16 + (lane & 7)];
  mu = 0.f;
  mu += m0.x * k0.x; mu += m0.y * k0.y; mu += m0.z * k0.z; mu += m0.w * k0.w;
  mu += m1.x * k1.x; mu += m1.y * k1.y; mu += m1.z * k1.z; mu += m1.w * k1.w;
  mu *= inv_d;
  const float e = mi - mu, part = vi + ci * e * e;       // a lane per warp, then in order
  m2 = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) m2 += __shfl_sync(0xffffffffu, part, i);
}

template <int NV>
__global__ void __launch_bounds__(64 + 768, 1) seam_many_kernel(SeamMany m) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ ManyBars B;
  const SeamArgs& a = m.a;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, d = a.d;
  volatile int* dead = &B.dead;
  uint8_t* ring = smem + m.weights;
  if (tid == 0) {
    B.dead = 0;
    for (int i = 0; i < m.stages; ++i) { tc::mbar_init(&B.full[i], 1); tc::mbar_init(&B.done[i], m.threads / 32); tc::mbar_init(&B.empty[i], 1); }
    tc::mbar_init(&B.weights, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < MANY_MAX_GROUPS * 48; i += blockDim.x) (&B.sums[0][0][0])[i] = 0.f;
  pdl_launch_dependents();
  __syncthreads();
  if (warp == 0) {
    if (elect_one()) {
      if (m.weights) {
        tc::mbar_expect(&B.weights, m.weights);
        uint8_t* p = smem;
        const float* w[6] = {a.y2 ? a.mw : nullptr, a.y2 ? a.mw2 : nullptr, a.y ? a.pw : nullptr, a.y ? a.pb : nullptr, a.nw, a.nw ? a.nb : nullptr};
        for (int i = 0; i < 6; ++i)
          if (w[i]) { bulk_in(p, w[i], d * 4, &B.weights); p += d * 4; }
      }
      pdl_wait();
      int k = 0;
      for (int r = blockIdx.x; r < m.n; r += gridDim.x, ++k) {
        const int st = k % m.stages;
        if (k >= m.stages && !tc::mbar_wait(&B.empty[st], (k / m.stages - 1) & 1, dead)) break;
        tc::mbar_expect(&B.full[st], m.load);
        uint8_t* p = ring + (size_t)st * m.stage;
        bulk_in(p, a.x + (size_t)r * d, d * 4, &B.full[st]);
        p += d * 4;
        if (a.y) {
          const int parts = a.parts_w ? a.parts : 1;
          bulk_in(p, (const T*)a.y + (size_t)r * parts * d, parts * d * 2, &B.full[st]);
          if (a.y2) bulk_in(p + d * 2, (const T*)a.y2 + (size_t)r * d, d * 2, &B.full[st]);
        }
      }
      if (*dead)                 // copies still in flight must land before the CTA ends
        for (int j = max(0, k - m.stages); j < k; ++j)
          for (int i = 0; i < 100000 && !tc::mbar_try(&B.full[j % m.stages], (j / m.stages) & 1); ++i) __nanosleep(64);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      pdl_wait();
      int k = 0;
      for (int r = blockIdx.x; r < m.n; r += gridDim.x, ++k) {
        const int st = k % m.stages;
        if (!tc::mbar_wait(&B.done[st], (k / m.stages) & 1, dead)) break;
        const uint8_t* p = ring + (size_t)st * m.stage;
        if (a.y) bulk_out(a.x + (size_t)r * d, p, d * 4);
        if (a.h) bulk_out((T*)a.h + (size_t)r * d, p + d * 4, d * 2);
        tc::bulk_commit();
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        if (k > 0) tc::mbar_arrive(&B.empty[(k - 1) % m.stages]);
      }
      tc::bulk_wait_read();
    }
  } else {
    const int g = (tid - 64) / m.threads, t = (tid - 64) % m.threads, w = t >> 5, warps = m.threads >> 5;
    const int step = m.threads * 4, c0 = t * 4;
    const float inv_d = 1.f / (float)d;
    int mine = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) mine += max(0, min(4, d - (c0 + i * step)));
    const float wcnt = warp_sum((float)mine), winv = wcnt > 0.f ? 1.f / wcnt : 0.f;
    const float* next = reinterpret_cast<const float*>(smem);
    auto take = [&](bool there) { const float* p = there ? next : nullptr; if (there) next += d; return p; };
    const float *mw = take(a.y2), *mw2 = take(a.y2), *pw = take(a.y), *pb = take(a.y && a.pb), *nw = take(a.nw), *nb = take(a.nw && a.nb);
    bool ok = m.weights == 0 || tc::mbar_wait(&B.weights, 0, dead);
    pdl_wait();
    int k = g, phase = 0;
    for (int r = blockIdx.x + g * gridDim.x; ok && r < m.n; r += m.groups * gridDim.x, k += m.groups) {
      const int st = k % m.stages;
      float wj[8];
      if (a.parts_w) {
#pragma unroll
        for (int j = 0; j < 8; ++j) wj[j] = j < a.parts ? a.parts_w[(size_t)r * a.parts + j] : 0.f;
      }
      if (lane == 0) ok = tc::mbar_wait(&B.full[st], (k / m.stages) & 1, dead);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      float* xs = reinterpret_cast<float*>(ring + (size_t)st * m.stage);
      T* ys = reinterpret_cast<T*>(xs + d);
      float x[NV][4];
      if (a.y) {
        float y[NV][4];
        if (a.y2) {
          float s0 = 0.f, s1 = 0.f;
#pragma unroll
          for (int i = 0; i < NV; ++i)
            if (c0 + i * step < d) {
              float z[4];
              load_v<T, 4>(ys + c0 + i * step, y[i]);
              load_v<T, 4>(ys + d + c0 + i * step, z);
#pragma unroll
              for (int q = 0; q < 4; ++q) { s0 += y[i][q] * y[i][q]; s1 += z[q] * z[q]; }
            }
          s0 = warp_sum(s0); s1 = warp_sum(s1);
          float* s = B.sums[g][phase & 1];
          ++phase;
          if (lane == 0) { s[w] = s0; s[8 + w] = s1; }
          group_sync(g, m.threads);
          s0 = sum8(s);
          s1 = sum8(s + 8);
          const float r0 = 0.5f / sqrtf(s0 * inv_d + a.eps), r1 = 0.5f / sqrtf(s1 * inv_d + a.eps);
#pragma unroll
          for (int i = 0; i < NV; ++i)
            if (c0 + i * step < d) {
              float w0[4], w1[4], z[4];
              load_v<T, 4>(ys + d + c0 + i * step, z);
              load_v<float, 4>(mw + c0 + i * step, w0);
              load_v<float, 4>(mw2 + c0 + i * step, w1);
#pragma unroll
              for (int q = 0; q < 4; ++q) y[i][q] = y[i][q] * r0 * w0[q] + z[q] * r1 * w1[q];
            }
        } else if (a.parts_w) {
#pragma unroll
          for (int i = 0; i < NV; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) y[i][q] = 0.f;
          for (int j = 0; j < a.parts; ++j) {
            float f = j < 8 ? 0.f : a.parts_w[(size_t)r * a.parts + j];
#pragma unroll
            for (int q = 0; q < 8; ++q) if (j == q) f = wj[q];
#pragma unroll
            for (int i = 0; i < NV; ++i)
              if (c0 + i * step < d) {
                float z[4];
                load_v<T, 4>(ys + (size_t)j * d + c0 + i * step, z);
#pragma unroll
                for (int q = 0; q < 4; ++q) y[i][q] = fmaf(f, z[q], y[i][q]);
              }
          }
        } else {
#pragma unroll
          for (int i = 0; i < NV; ++i)
            if (c0 + i * step < d) load_v<T, 4>(ys + c0 + i * step, y[i]);
        }
        float mu = 0.f, rs = 1.f;
        if (a.post != POST_SCALE) {
          float m2;
          group_moments<NV>(y, c0, step, d, wcnt, winv, inv_d, B.sums[g][phase++ & 1], warps, w, lane, g, mu, m2);
          rs = 1.f / sqrtf((a.post == POST_RMS ? fmaf(mu, mu, m2 * inv_d) : m2 * inv_d) + a.eps);
          if (a.post == POST_RMS) mu = 0.f;
        }
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (c0 + i * step < d) {
            float f[4], b[4] = {0.f, 0.f, 0.f, 0.f};
            load_v<float, 4>(xs + c0 + i * step, x[i]);
            load_v<float, 4>(pw + c0 + i * step, f);
            if (pb) load_v<float, 4>(pb + c0 + i * step, b);
#pragma unroll
            for (int q = 0; q < 4; ++q) x[i][q] += (y[i][q] - mu) * rs * f[q] + b[q];
            store_v<float, 4>(xs + c0 + i * step, x[i]);
          }
      } else {
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (c0 + i * step < d) load_v<float, 4>(xs + c0 + i * step, x[i]);
      }
      if (a.h) {
        float mu = 0.f, rs = 1.f;
        if (a.nw) {
          float m2;
          group_moments<NV>(x, c0, step, d, wcnt, winv, inv_d, B.sums[g][phase++ & 1], warps, w, lane, g, mu, m2);
          rs = 1.f / sqrtf((a.rms ? fmaf(mu, mu, m2 * inv_d) : m2 * inv_d) + a.eps);
          if (a.rms) mu = 0.f;
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int c = c0 + i * step;
          if (c >= d) continue;
          float f[4], b[4] = {0.f, 0.f, 0.f, 0.f}, o[4];
          if (a.nw) {
            load_v<float, 4>(nw + c, f);
            if (nb) load_v<float, 4>(nb + c, b);
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q] = (x[i][q] - mu) * rs * f[q] + b[q];
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q] = x[i][q];
          }
          store_v<T, 4>(ys + c, o);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&B.done[st]);
    }
  }
  __syncthreads();
  if (tid == 0 && *dead) status_set(a.status, ST_TIMEOUT, 78, blockIdx.x, 0);
}

// The same for S streams: k_rows_streams.cu's sums, a row of all streams a stage.  Four streams, us (floor): 3,000 x 2,048 47 -> 35 (34), with four parts 73 -> 41 (39); 600 x 2,048
// 16 -> 14 and 23 -> 16; 3,000 x 3,000 67 -> 52 (49) and 149 -> 66 (58); 3,000 x 1,024 23 -> 21 and 35 -> 23; 300 x 1,024 9 -> 10 and 11 -> 10.  Four streams of 4,096
// do not fit three stages and keep the block per row.
struct StreamsMany {
  StreamArgs a;
  int n, stages, groups, threads;
  uint32_t load, stage, weights;
};

template <int S, int NV>
__global__ void __launch_bounds__(64 + 512, 1) streams_many_kernel(StreamsMany m) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ ManyBars B;
  const StreamArgs& a = m.a;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, d = a.d, parts = a.parts_w ? a.parts : 1;
  volatile int* dead = &B.dead;
  uint8_t* ring = smem + m.weights;
  if (tid == 0) {
    B.dead = 0;
    for (int i = 0; i < m.stages; ++i) { tc::mbar_init(&B.full[i], 1); tc::mbar_init(&B.done[i], m.threads / 32); tc::mbar_init(&B.empty[i], 1); }
    tc::mbar_init(&B.weights, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < MANY_MAX_GROUPS * 48; i += blockDim.x) (&B.sums[0][0][0])[i] = 0.f;
  pdl_launch_dependents();
  __syncthreads();
  if (warp == 0) {
    if (elect_one()) {
      tc::mbar_expect(&B.weights, m.weights);
      bulk_in(smem, a.nw, d * 4, &B.weights);
      pdl_wait();
      int k = 0;
      for (int r = blockIdx.x; r < m.n; r += gridDim.x, ++k) {
        const int st = k % m.stages;
        if (k >= m.stages && !tc::mbar_wait(&B.empty[st], (k / m.stages - 1) & 1, dead)) break;
        tc::mbar_expect(&B.full[st], m.load);
        uint8_t* p = ring + (size_t)st * m.stage;
        bulk_in(p, a.x + (size_t)r * S * d, S * d * 4, &B.full[st]);
        bulk_in(p + S * d * 4, (const T*)a.y + (size_t)r * parts * d, parts * d * 2, &B.full[st]);
      }
      if (*dead)                 // copies still in flight must land before the CTA ends
        for (int j = max(0, k - m.stages); j < k; ++j)
          for (int i = 0; i < 100000 && !tc::mbar_try(&B.full[j % m.stages], (j / m.stages) & 1); ++i) __nanosleep(64);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      pdl_wait();
      int k = 0;
      for (int r = blockIdx.x; r < m.n; r += gridDim.x, ++k) {
        const int st = k % m.stages;
        if (!tc::mbar_wait(&B.done[st], (k / m.stages) & 1, dead)) break;
        const uint8_t* p = ring + (size_t)st * m.stage;
        if (a.keep) bulk_out(a.x + (size_t)r * S * d, p, S * d * 4);
        bulk_out((T*)a.h + (size_t)r * d, p + S * d * 4, d * 2);
        tc::bulk_commit();
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        if (k > 0) tc::mbar_arrive(&B.empty[(k - 1) % m.stages]);
      }
      tc::bulk_wait_read();
    }
  } else {
    const int g = (tid - 64) / m.threads, t0 = (tid - 64) % m.threads, w = t0 >> 5;
    const int step = m.threads * 4, c0 = t0 * 4;
    float mix[S][S], out[S], in[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      in[s] = a.in ? a.in[s] : 1.f;
      out[s] = a.out[s];
#pragma unroll
      for (int t = 0; t < S; ++t) mix[s][t] = a.mix[s * S + t];
    }
    const float* nw = reinterpret_cast<const float*>(smem);
    bool ok = tc::mbar_wait(&B.weights, 0, dead);
    pdl_wait();
    int k = g, phase = 0;
    for (int r = blockIdx.x + g * gridDim.x; ok && r < m.n; r += m.groups * gridDim.x, k += m.groups) {
      const int st = k % m.stages;
      float wj[8];
      if (a.parts_w) {
#pragma unroll
        for (int j = 0; j < 8; ++j) wj[j] = j < a.parts ? a.parts_w[(size_t)r * a.parts + j] : 0.f;
      }
      if (lane == 0) ok = tc::mbar_wait(&B.full[st], (k / m.stages) & 1, dead);
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      float* xs = reinterpret_cast<float*>(ring + (size_t)st * m.stage);
      T* ys = reinterpret_cast<T*>(xs + S * d);
      float u[NV][4], ss = 0.f;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = c0 + i * step;
        if (c >= d) continue;
        float y[4], x[S][4];
        if (a.parts_w) {
#pragma unroll
          for (int q = 0; q < 4; ++q) y[q] = 0.f;
          for (int j = 0; j < a.parts; ++j) {
            float f = j < 8 ? 0.f : a.parts_w[(size_t)r * a.parts + j], z[4];
#pragma unroll
            for (int q = 0; q < 8; ++q) if (j == q) f = wj[q];
            load_v<T, 4>(ys + (size_t)j * d + c, z);
#pragma unroll
            for (int q = 0; q < 4; ++q) y[q] = fmaf(f, z[q], y[q]);
          }
        } else {
          load_v<T, 4>(ys + c, y);
        }
#pragma unroll
        for (int s = 0; s < S; ++s) load_v<float, 4>(xs + s * d + c, x[s]);
#pragma unroll
        for (int q = 0; q < 4; ++q) u[i][q] = 0.f;
#pragma unroll
        for (int t = 0; t < S; ++t) {
          float n[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            n[q] = out[t] * y[q];
#pragma unroll
            for (int s = 0; s < S; ++s) n[q] = fmaf(mix[s][t], x[s][q], n[q]);
            u[i][q] = fmaf(in[t], n[q], u[i][q]);
          }
          if (a.keep) store_v<float, 4>(xs + t * d + c, n);
        }
      }
#pragma unroll
      for (int i = 0; i < NV; ++i)
        if (c0 + i * step < d) {
#pragma unroll
          for (int q = 0; q < 4; ++q) ss = fmaf(u[i][q], u[i][q], ss);
        }
      float* s = B.sums[g][phase++ & 1];
      ss = warp_sum(ss);
      if (lane == 0) s[w] = ss;
      group_sync(g, m.threads);
      ss = sum8(s);
      const float rs = 1.f / sqrtf(ss / (float)d + a.eps);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = c0 + i * step;
        if (c >= d) continue;
        float o[4], f[4];
        load_v<float, 4>(nw + c, f);
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = u[i][q] * rs * f[q];
        store_v<T, 4>(ys + c, o);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&B.done[st]);
    }
  }
  __syncthreads();
  if (tid == 0 && *dead) status_set(a.status, ST_TIMEOUT, 80, blockIdx.x, 0);
}

static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}
template <int S, int NV>
static int launch_streams_many(const StreamsMany& m, cudaStream_t stream) {
  static bool done = false;
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(streams_many_kernel<S, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, MANY_SMEM);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const int sms = sm_count();
  return (int)sfb_launch(streams_many_kernel<S, NV>, dim3(m.n < sms ? m.n : sms), dim3(64 + m.groups * m.threads), m.weights + m.stages * m.stage, stream, m);
}

int streams_many(const StreamArgs& a, int n, cudaStream_t stream) {
  const int d = a.d;
  if (n < SEAM_MANY_ROWS || !a.y || a.tap || a.row_map || a.cw || a.S < 2 || a.S > 4 || d % 8 || d > 4096 || d < 1024) return -1;
  if (((uintptr_t)a.x | (uintptr_t)a.y | (uintptr_t)a.nw | (uintptr_t)a.h) % 16) return -1;
  StreamsMany m{};
  m.a = a; m.n = n;
  const int parts = a.parts_w ? a.parts : 1;
  m.weights = d * 4;
  m.load = a.S * d * 4 + parts * d * 2;
  m.stage = (m.load + 127) & ~127u;
  if ((long long)m.weights + 3ll * m.stage > MANY_SMEM) return -1;
  m.stages = (int)((MANY_SMEM - m.weights) / m.stage);
  if (m.stages > MANY_MAX_STAGES) m.stages = MANY_MAX_STAGES;
  int nv = 1;              // as launch_streams spreads a row
  while (nv < 4 && (d / 4 + nv - 1) / nv > (nv >= 2 ? 256 : 128)) nv *= 2;
  m.threads = ((d / 4 + nv - 1) / nv + 31) / 32 * 32;
  m.groups = 512 / m.threads;
  if (m.groups > m.stages - 1) m.groups = m.stages - 1;
  if (nv <= 2) return a.S == 2 ? launch_streams_many<2, 2>(m, stream) : a.S == 3 ? launch_streams_many<3, 2>(m, stream) : launch_streams_many<4, 2>(m, stream);
  return a.S == 2 ? launch_streams_many<2, 4>(m, stream) : a.S == 3 ? launch_streams_many<3, 4>(m, stream) : launch_streams_many<4, 4>(m, stream);
}

// Not: fewer rows, the ends of a forward (embedding, chosen rows), convolutions of single rows, rows that are not whole 16-byte words or do not fit.
int seam_many(const SeamArgs& a, int n, cudaStream_t stream) {
  const int d = a.d;
  if (n < SEAM_MANY_ROWS || a.from_embed || a.add_embed || a.step_vec || a.tap || a.row_map || a.cw || (!a.y && !a.h) || d % 8 || d > 4096 || d < (n < 2048 ? 2048 : 1024))
    return -1;
  const uintptr_t bits = (uintptr_t)a.x | (uintptr_t)a.y | (uintptr_t)a.y2 | (uintptr_t)a.mw | (uintptr_t)a.mw2 | (uintptr_t)a.pw | (uintptr_t)a.pb | (uintptr_t)a.nw |
                         (uintptr_t)a.nb | (uintptr_t)a.h;
  if (bits % 16) return -1;
  SeamMany m{};
  m.a = a; m.n = n;
  const int pieces = a.y2 ? 2 : a.parts_w ? a.parts : 1;
  m.weights = d * 4 * ((a.y2 ? 2 : 0) + (a.y ? 1 : 0) + (a.y && a.pb ? 1 : 0) + (a.nw ? 1 : 0) + (a.nw && a.nb ? 1 : 0));
  m.stage = ((uint32_t)d * 4 + (uint32_t)d * 2 * pieces + 127) & ~127u;
  m.load = d * 4 + (a.y ? d * 2 * pieces : 0);
  if ((long long)m.weights + 3ll * m.stage > MANY_SMEM) return -1;
  m.stages = (int)((MANY_SMEM - m.weights) / m.stage);
  if (m.stages > MANY_MAX_STAGES) m.stages = MANY_MAX_STAGES;
  int nv = 1;              // as launch_seam spreads a row, so that the sums are its sums
  while (nv < 4 && (d / 4 + nv - 1) / nv > 128) nv *= 2;
  m.threads = ((d / 4 + nv - 1) / nv + 31) / 32 * 32;
  m.groups = 768 / m.threads;
  if (m.groups > MANY_MAX_GROUPS) m.groups = MANY_MAX_GROUPS;
  if (m.groups > m.stages - 1) m.groups = m.stages - 1;
  static bool done = false;
  if (!done) {
    const cudaError_t e = cudaFuncSetAttribute(seam_many_kernel<MANY_NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, MANY_SMEM);
    if (e != cudaSuccess) return (int)e;
    done = true;
  }
  const int sms = sm_count();
  return (int)sfb_launch(seam_many_kernel<MANY_NV>, dim3(n < sms ? n : sms), dim3(64 + m.groups * m.threads), m.weights + m.stages * m.stage, stream, m);
}

}  // namespace rows
}  // namespace sfb
