// All-reduce + residual + RMSNorm when every rank's tensors are in one GPU's address space (a world of one, an emulated
// world): nothing is exchanged.  A cluster of `parts` CTAs owns a row for ALL ranks: it reads the row of every rank's x
// once, adds in rank order in fp32, adds each rank's residual, rounds, and normalises; the rows stay in registers between
// the statistic and the scaling, and the CTAs of a row hand each other their sums of squares through distributed shared
// memory.  Bound by launch and memory latency at decode sizes (8 ranks, 16 rows of 8192: 9.2 us cold, the flag-in-data
// kernel 20.4), above by memory, mostly its writes, and by how many CTAs' loads are in flight beside the arithmetic: on pairs of fp32
// values (each rounded as by itself) 8 ranks, 512 rows of 8192 48.5 -> 46.7 us for 209 MB (bf16 60.6 -> 60.3: its registers leave room
// for two CTAs an SM, not three; capped, 52 there and 6 - 18 % more at fewer rows), 300 x 5120 21.9 -> 19.8, 16 x 8192 5.2 -> 4.8.
#pragma once

#include "../coll/bulk_kernels.cuh"
#include "../common/pdl.h"

namespace b200ipc {

constexpr int kDirectNormThreads = 512;
constexpr int kDirectNormMaxParts = 8;

struct DirectNormArgs {
  const void* x[kMaxRanks];
  const void* residual[kMaxRanks];
  const void* gamma[kMaxRanks];
  void* out[kMaxRanks];
  void* res_out[kMaxRanks];
  int row_vecs;   // hidden / 8
  int part_vecs;  // vectors of a row that one CTA takes: at most U x blockDim
  float hidden, eps;
};

// N ranks, U vectors per thread (one with 8 ranks: more do not fit the registers); cluster (parts, 1, 1), blockIdx.x = row * parts + part.
template <typename T, int N, int U>
__global__ void __launch_bounds__(kDirectNormThreads) direct_norm_kernel(const __grid_constant__ DirectNormArgs args) {
  __shared__ float s_warp[kDirectNormThreads / 32][N];
  __shared__ float s_part[kDirectNormMaxParts][N];  // every CTA of the row writes its sums into every CTA
  uint32_t part, parts;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(part));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(parts));
  const int tid = int(threadIdx.x), step = int(blockDim.x);
  const int first = int(part) * args.part_vecs;
  const int last = min(first + args.part_vecs, args.row_vecs);
  const size_t row0 = size_t(blockIdx.x / parts) * size_t(args.row_vecs);
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // this CTA runs: its shared memory may be written
  pdl_wait();
  pdl_launch_dependents();

  uint4 keep[N][U];
  float2 ss2[N];
#pragma unroll
  for (int q = 0; q < N; ++q) ss2[q] = make_float2(0.f, 0.f);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int v = first + tid + u * step;
    if (v >= last) continue;
    uint4 x[N];
#pragma unroll
    for (int q = 0; q < N; ++q) {
      x[q] = static_cast<const uint4*>(args.x[q])[row0 + v];
      keep[q][u] = static_cast<const uint4*>(args.residual[q])[row0 + v];
    }
    float2 a[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) a[e] = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const uint32_t xs[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = add_f32x2(a[e], Cvt<T>::up(xs[e]));
    }
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const uint4 res = keep[q][u];
      const uint32_t rs[4] = {res.x, res.y, res.z, res.w};
      uint32_t ys[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 b = add_f32x2(a[e], Cvt<T>::up(rs[e]));
        ys[e] = Cvt<T>::down(b.x, b.y);
        const float2 r = Cvt<T>::up(ys[e]);
        ss2[q] = fma_f32x2(r, r, ss2[q]);
      }
      keep[q][u] = make_uint4(ys[0], ys[1], ys[2], ys[3]);
    }
  }
  float ss[N];
#pragma unroll
  for (int q = 0; q < N; ++q) ss[q] = ss2[q].x + ss2[q].y;
  // The row statistic, from the rounded sums; the order depends on nothing but thread and part numbers, so ranks with the
  // same residual get the same bits.
#pragma unroll
  for (int q = 0; q < N; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss[q] += __shfl_xor_sync(0xffffffffu, ss[q], o);
    if ((tid & 31) == 0) s_warp[tid >> 5][q] = ss[q];
  }
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // every CTA of the row runs
  for (int i = tid; i < N * int(parts); i += step) {
    const int q = i % N, to = i / N;
    float s = 0.f;
    for (int w = 0; w < (step >> 5); ++w) s += s_warp[w][q];
    uint32_t dst;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(uint32_t(__cvta_generic_to_shared(&s_part[part][q]))), "r"(to));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(s) : "memory");
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  float inv[N];
#pragma unroll
  for (int q = 0; q < N; ++q) {
    float s = 0.f;
    for (uint32_t p = 0; p < parts; ++p) s += s_part[p][q];
    inv[q] = rsqrtf(s / args.hidden + args.eps);
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int v = first + tid + u * step;
    if (v >= last) continue;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const uint4 g = static_cast<const uint4*>(args.gamma[q])[v];
      const uint32_t xs[4] = {keep[q][u].x, keep[q][u].y, keep[q][u].z, keep[q][u].w}, gs[4] = {g.x, g.y, g.z, g.w};
      uint32_t ys[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 y = mul_f32x2(mul_f32x2(Cvt<T>::up(xs[e]), make_float2(inv[q], inv[q])), Cvt<T>::up(gs[e]));
        ys[e] = Cvt<T>::down(y.x, y.y);
      }
      static_cast<uint4*>(args.res_out[q])[row0 + v] = keep[q][u];
      static_cast<uint4*>(args.out[q])[row0 + v] = make_uint4(ys[0], ys[1], ys[2], ys[3]);
    }
  }
}

}  // namespace b200ipc
