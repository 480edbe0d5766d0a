// Per-row state and the 32-token chunk step shared by the scalar forward kernels.
#pragma once
#include "psa_common.cuh"

namespace psa {

// Four threads share a row.  Thread g of the four owns channels {16 i + 4 g .. 16 i + 4 g + 3}, so that it reads a key or value
// row from shared memory 16 bytes at a time (the four read 64 consecutive bytes, the other rows of the warp the same ones):
// one shared-memory load feeds four multiply-adds.  With every fourth channel (one load per multiply-add) the loads were the
// bound.  2 heads x 4096 tokens x 64, default ratios, with the rows of a block dealt to four CTAs: 238 -> 207 us,
// 166 us with eight staging loads in flight, 130 us with the chunks of a row dealt to four sets of threads.
template <typename T, int D>
struct FwdCore {
  static constexpr int DPT = D / 4;
  static __device__ __forceinline__ int channel(int d, int g) { return (d >> 2) * 16 + g * 4 + (d & 3); }
  float q[DPT], acc[DPT];
  float m, l;

  static __device__ __forceinline__ void sync(int bar, int nt) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nt) : "memory"); }

  __device__ __forceinline__ void init(const T* qrow, bool valid, int g) {
#pragma unroll
    for (int d = 0; d < DPT; ++d) { q[d] = valid ? Elem<T>::to_f(qrow[channel(d, g)]) : 0.f; acc[d] = 0.f; }
    m = -INFINITY; l = 0.f;
  }

  // Attend to C (<= 32) consecutive pooled tokens [t0, t0+C) of one level; only the first nv exist.
  // causal_level > 0: pooled token j is visible iff (j+1)*causal_level - 1 <= qpos.
  // Called by nt threads (this one is number tid) that share Ks, Vs and the hardware barrier `bar`.
  __device__ __forceinline__ void chunk(const T* __restrict__ Kl, const T* __restrict__ Vl, int64_t t0, int C, int nv,
                                        float bias, float scale, float (*Ks)[D], float (*Vs)[D], int g,
                                        int causal_level, int64_t qpos, int tid, int nt, int bar) {
    sync(bar, nt);
    // eight elements of each operand in flight per thread (a block of 128 threads stages 16 to 32 of each)
    constexpr int kUnroll = 8;
    for (int e0 = tid; e0 < C * D; e0 += kUnroll * nt) {
      float kx[kUnroll], vx[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int e = e0 + u * nt;
        const bool ok = e < C * D && e / D < nv;
        kx[u] = ok ? Elem<T>::to_f(Kl[t0 * D + e]) : 0.f;
        vx[u] = ok ? Elem<T>::to_f(Vl[t0 * D + e]) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int e = e0 + u * nt;
        if (e < C * D) { Ks[e / D][e % D] = kx[u]; Vs[e / D][e % D] = vx[u]; }
      }
    }
    sync(bar, nt);
    // 8 tokens per softmax step keeps the scores in registers without unrolling the whole chunk
    for (int c0 = 0; c0 < C; c0 += 8) {
      float s[8];
      float mx = -INFINITY;
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) {
        const int c = c0 + cc;
        float part = 0.f;
        if (c < C) {
#pragma unroll
          for (int d = 0; d < DPT; d += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(&Ks[c][channel(d, g)]);
            part = fmaf(q[d], k4.x, part);
            part = fmaf(q[d + 1], k4.y, part);
            part = fmaf(q[d + 2], k4.z, part);
            part = fmaf(q[d + 3], k4.w, part);
          }
        }
        part += __shfl_xor_sync(0xffffffffu, part, 1);
        part += __shfl_xor_sync(0xffffffffu, part, 2);
        bool vis = c < nv && (causal_level == 0 || ((t0 + c + 1) * causal_level - 1 <= qpos));
        s[cc] = vis ? part * scale + bias : -INFINITY;
        mx = fmaxf(mx, s[cc]);
      }
      const float m_new = fmaxf(m, mx);
      if (m_new == -INFINITY) continue;   // nothing visible yet for this row
      const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
      float lsum = 0.f;
#pragma unroll
      for (int d = 0; d < DPT; ++d) acc[d] *= alpha;
#pragma unroll
      for (int cc = 0; cc < 8; ++cc) {
        const int c = c0 + cc;
        if (c < C) {
          float p = s[cc] == -INFINITY ? 0.f : expf(s[cc] - m_new);
          lsum += p;
          float pr = Elem<T>::round(p);
#pragma unroll
          for (int d = 0; d < DPT; d += 4) {
            const float4 v4 = *reinterpret_cast<const float4*>(&Vs[c][channel(d, g)]);
            acc[d] = fmaf(pr, v4.x, acc[d]);
            acc[d + 1] = fmaf(pr, v4.y, acc[d + 1]);
            acc[d + 2] = fmaf(pr, v4.z, acc[d + 2]);
            acc[d + 3] = fmaf(pr, v4.w, acc[d + 3]);
          }
        }
      }
      l = l * alpha + lsum;
      m = m_new;
    }
  }
};

struct LevelPtrs {
  const void* k[4];
  const void* v[4];
  int64_t n[4];  // tokens per head at levels 1,2,4,8
};

}  // namespace psa
