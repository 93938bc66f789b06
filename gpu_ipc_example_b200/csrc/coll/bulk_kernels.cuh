// Large-message collectives over the symmetric heap: all-reduce, reduce-scatter
// and all-gather, each in two flavours selected by a template flag:
//   P2P   the owner of a shard loads it from every peer (16 B vectors over NVLink),
//         adds in rank order in fp32 and stores the result into every peer;
//   NVLS  multimem.ld_reduce lets the NVSwitch add the copies, multimem.st lets it
//         replicate the result: one load and one store per 16 B whatever the world.
// 100 % of the bytes on the wire are payload; ranks meet at per-CTA flag barriers
// (CTA b of every rank only ever depends on CTA b of the others), every wait is
// bounded.  These have no counterpart in the reference, whose kernels are all
// flag-in-data; they exist because at tens of megabytes the 6-50 % flag overhead
// and the register-resident messages stop paying.
#pragma once

#include "../common/pdl.h"
#include "../proto/dev_backend.cuh"
#include "kernel_table.h"

namespace b200ipc {

constexpr int kBulkThreads = 512;

enum class BulkMode : int { AllReduce = 0, ReduceScatter = 1, AllGather = 2 };

// aux[1] bits
constexpr uint64_t kBulkCopyIn = 1;   // stage `in` into the symmetric buffer first
constexpr uint64_t kBulkCopyOut = 2;  // copy the result from the symmetric buffer to `out`

// Where the ranks' data lives.  Heap: at one offset of every rank's symmetric heap.  Direct: in the callers' own
// buffers, which every rank of an emulated world can address (the launch arguments hold all of them), so that
// nothing is staged and the ranks do not meet: they are block rows of one launch, which starts when every input is in place
// and whose end is the point that whoever comes after it waits for.  `auto` takes it there; "bulk" by name is Heap.
enum class BulkPlace : int { Heap = 0, Direct = 1 };

__device__ __forceinline__ void st_release_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_sys_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <typename T>
__device__ __forceinline__ uint4 multimem_ld_reduce_add(const void* mc_addr);
template <>
__device__ __forceinline__ uint4 multimem_ld_reduce_add<__half>(const void* mc_addr) {
  uint4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.f16x2 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(mc_addr)
               : "memory");
  return v;
}
template <>
__device__ __forceinline__ uint4 multimem_ld_reduce_add<__nv_bfloat16>(const void* mc_addr) {
  uint4 v;
  asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v4.bf16x2 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(mc_addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void multimem_st_v4(void* mc_addr, uint4 v) {
  asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(mc_addr), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

__device__ __forceinline__ void st_relaxed_sys_u32(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed_sys_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_volatile_u4(const void* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

// Barrier between CTA `blockIdx.x` of every rank.  All threads call it; returns
// false (to all threads) if the wait ran out or the collective was aborted.
// `publish` = this CTA has written something the other ranks are about to read (its
// signal must then be a release); an arrival that only says "my kernel has started" is a
// plain store.  The polls are relaxed loads, and what the other ranks published is read
// afterwards with loads that go around L1 (ld.volatile / multimem), issued after the poll
// has returned: no acquire fence is paid for.
__device__ __forceinline__ bool cta_rank_barrier(const RankView& me, const HeapLayout& lay, uint32_t value,
                                                 int site, bool publish) {
  __shared__ int s_fail;
  const int tid = int(threadIdx.x);
  if (tid == 0) s_fail = 0;
  __syncthreads();  // also orders every thread's earlier writes before the signal below
  const size_t pad_off = lay.ctrl_off + kCtrlBarrierOff + size_t(blockIdx.x) * kMaxRanks * sizeof(uint32_t);
  if (tid < me.world && tid != me.rank) {
    uint32_t* abort_word = reinterpret_cast<uint32_t*>(me.heap + lay.ctrl_off + kCtrlAbortOff);
    if (!(me.flags & kMuteSends)) {
      uint32_t* dst = reinterpret_cast<uint32_t*>(me.peer[tid] + pad_off) + me.rank;
      // st.release.sys orders the CTA's earlier accesses (made visible to this thread by the
      // barrier above) before the signal
      if (publish) st_release_sys_u32(dst, value);
      else st_relaxed_sys_u32(dst, value);
    }
    const uint32_t* mine = reinterpret_cast<const uint32_t*>(me.heap + pad_off) + tid;
    uint32_t spins = 0;
    uint64_t t0 = 0;
    for (;;) {
      uint32_t seen = ld_relaxed_sys_u32(mine);
      if (int32_t(seen - value) >= 0) break;
      if ((++spins & 0x3fu) == 0) {
        if (ld_volatile_u32(abort_word) != 0) {
          note_aborted_by_peer(abort_word, me.status, me.rank, site);
          s_fail = 1;
          break;
        }
        const uint64_t now = globaltimer_ns();
        if (t0 == 0) {
          t0 = now;
        } else if (now - t0 > me.timeout_ns) {
          if (claim_status(abort_word, kTimeout)) {
            StatusBlock* s = me.status;
            s->rank = uint32_t(me.rank);
            s->peer = uint32_t(tid);
            s->wire = blockIdx.x;
            s->step = 0;
            s->expected = value;
            s->seen = seen;
            s->where = uint32_t(site);
            __threadfence_system();
            s->code = kTimeout;
            __threadfence_system();
          }
          for (int q = 0; q < me.world; ++q)  // own abort word included
            st_volatile_u32(reinterpret_cast<uint32_t*>(me.peer[q] + lay.ctrl_off + kCtrlAbortOff), 1u);
          s_fail = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
  return s_fail == 0;
}

template <typename T>
__device__ __forceinline__ void acc8_add(float (&a)[8], uint4 v) {
  float2 x;
  x = Cvt<T>::up(v.x); a[0] += x.x; a[1] += x.y;
  x = Cvt<T>::up(v.y); a[2] += x.x; a[3] += x.y;
  x = Cvt<T>::up(v.z); a[4] += x.x; a[5] += x.y;
  x = Cvt<T>::up(v.w); a[6] += x.x; a[7] += x.y;
}
template <typename T>
__device__ __forceinline__ uint4 acc8_pack(const float (&a)[8]) {
  return make_uint4(Cvt<T>::down(a[0], a[1]), Cvt<T>::down(a[2], a[3]), Cvt<T>::down(a[4], a[5]),
                    Cvt<T>::down(a[6], a[7]));
}

// Of a row norm: the squares of eight elements, and the eight scaled.
template <typename T>
__device__ __forceinline__ void row_norm_squares(float2& ss, uint4 x) {
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 f = Cvt<T>::up(xs[e]);
    ss = fma_f32x2(f, f, ss);
  }
}
template <typename T>
__device__ __forceinline__ uint4 row_norm_scale(uint4 x, uint4 g, float inv) {
  const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, gs[4] = {g.x, g.y, g.z, g.w};
  uint32_t ys[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 y = mul_f32x2(mul_f32x2(Cvt<T>::up(xs[e]), make_float2(inv, inv)), Cvt<T>::up(gs[e]));
    ys[e] = Cvt<T>::down(y.x, y.y);
  }
  return make_uint4(ys[0], ys[1], ys[2], ys[3]);
}

// Elements [0, nelems) of a 16-bit buffer as 16 B vectors, guarded at the tail.
__device__ __forceinline__ uint4 ld_vec_guarded(const uint16_t* src, int64_t vec, int64_t nelems) {
  const int64_t e0 = vec * 8;
  if (e0 + 8 <= nelems && ((reinterpret_cast<uintptr_t>(src) & 15) == 0)) {
    return *reinterpret_cast<const uint4*>(src + e0);
  }
  uint16_t t[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) t[k] = (e0 + k < nelems) ? src[e0 + k] : uint16_t(0);
  return make_uint4(uint32_t(t[0]) | (uint32_t(t[1]) << 16), uint32_t(t[2]) | (uint32_t(t[3]) << 16),
                    uint32_t(t[4]) | (uint32_t(t[5]) << 16), uint32_t(t[6]) | (uint32_t(t[7]) << 16));
}
__device__ __forceinline__ void st_vec_guarded(uint16_t* dst, int64_t vec, int64_t nelems, uint4 v) {
  const int64_t e0 = vec * 8;
  if (e0 + 8 <= nelems && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
    *reinterpret_cast<uint4*>(dst + e0) = v;
    return;
  }
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 8; ++k)
    if (e0 + k < nelems) dst[e0 + k] = uint16_t(w[k >> 1] >> ((k & 1) * 16));
}

// Eight elements starting h (1..7) elements into the 16-byte aligned vector at src: two aligned vectors and a shift.  The
// second vector is the first one of the next thread, so it comes out of L1.  h is the same for every thread.
__device__ __forceinline__ uint4 ld_vec_shifted(const uint16_t* src, int h) {
  const uint4 x = *reinterpret_cast<const uint4*>(src);
  const uint4 y = *reinterpret_cast<const uint4*>(src + 8);
  uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  if (h & 4) { w[0] = w[2]; w[1] = w[3]; w[2] = w[4]; w[3] = w[5]; w[4] = w[6]; w[5] = w[7]; }
  if (h & 2) { w[0] = w[1]; w[1] = w[2]; w[2] = w[3]; w[3] = w[4]; w[4] = w[5]; }
  if (h & 1) {
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(w[k], w[k + 1], 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Streaming store: nothing of this launch reads the results again.
__device__ __forceinline__ void st_stream_u4(void* p, uint4 v) { __stcs(reinterpret_cast<uint4*>(p), v); }

// The collective over the callers' own buffers: owner r reads shard r of every rank's `in` and writes it where it
// belongs in every rank's `out`.  All buffers are 16-byte aligned (the host sees to it); the shards of a reduce-scatter or
// an all-gather need not be: their unaligned side is read through ld_vec_shifted, what does not fill a vector goes
// element by element.  Bound by memory: every input is read once, every output written once, in 16-byte vectors with
// world x kU loads of a thread in flight.  One B200, 8 ranks: all-reduce of 16 MiB 50 us = 5.4 TB/s (flag-in-data rings
// 282 us), reduce-scatter of 16 MiB 26 us (staged form 110), all-gather of 1 MiB per rank 13.4 us (direct push 59).
// Streaming stores: 22.9 -> 19.2 us at 8 MiB x 8, level elsewhere; streaming loads lose where the producer left the
// inputs in L2 (reduce-scatter of 8 MiB 9.0 -> 12.0 us).  Programmatic launch, back to back: reduce-scatter of 16 MiB 27.0 ->
// 25.8 us, all-reduce of 2 KiB 6.3 -> 5.4.  Other splits (128 - 1024 threads, 1 - 4 vectors, 1 - 16 CTAs per SM, streaming loads)
// are within 3 % of this one; a device-to-device memcpy of the same 197 MB takes 35 us, the all-reduce of 4 x 24.7 MB 38.
template <typename T, int N, BulkMode M>
__device__ __forceinline__ void bulk_direct_body(const KArgs& args, int r, int64_t shard_elems, int64_t valid) {
  constexpr int kU = M == BulkMode::AllGather ? 4 : bulk_unroll(N, false);
  const int tid = int(threadIdx.x);
  const int nthreads = int(blockDim.x);
  const int G = int(gridDim.x);
  const int64_t e0 = int64_t(r) * shard_elems;  // where shard r starts in a whole buffer
  auto in16 = [&](int q) { return static_cast<const uint16_t*>(args.v[q].in); };
  auto out16 = [&](int q) { return static_cast<uint16_t*>(args.v[q].out); };
  if (M == BulkMode::AllGather) {
    const uint16_t* src = in16(r);
    int64_t head = (8 - (e0 & 7)) & 7;  // elements in front of the first vector that is aligned in the destination
    if (head > valid) head = valid;
    const int h = int(head);
    // vectors whose source can be read as whole aligned vectors
    int64_t body = (valid - head) / 8;
    if (h != 0 && body > 0 && body * 8 + 8 > valid) --body;
    for (int64_t tile = int64_t(blockIdx.x); tile * nthreads < body; tile += int64_t(G) * kU) {
      uint4 v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i < body) v[u] = h == 0 ? *reinterpret_cast<const uint4*>(src + i * 8) : ld_vec_shifted(src + i * 8, h);
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i >= body) continue;
#pragma unroll
        for (int q = 0; q < N; ++q) st_stream_u4(out16(q) + e0 + head + i * 8, v[u]);
      }
    }
    if (int(blockIdx.x) == G - 1) {
      const int64_t rest = valid - body * 8;  // head and tail together: fewer than 24 elements
      for (int64_t k = tid; k < rest * N; k += nthreads) {
        const int64_t j = k / N;
        const int64_t e = j < head ? j : body * 8 + j;
        out16(int(k % N))[e0 + e] = src[e];
      }
    }
    return;
  }
  // AllReduce: shards start on vectors.  ReduceScatter: shard r may start anywhere, the output starts on a vector.
  const int h = M == BulkMode::ReduceScatter ? int(e0 & 7) : 0;
  const int64_t o0 = M == BulkMode::ReduceScatter ? 0 : e0;
  int64_t body = valid / 8;
  if (h == 0) {
    for (int64_t tile = int64_t(blockIdx.x); tile * nthreads < body; tile += int64_t(G) * kU) {
      uint4 v[kU][N];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i < body) {
#pragma unroll
          for (int q = 0; q < N; ++q) v[u][q] = *reinterpret_cast<const uint4*>(in16(q) + e0 + i * 8);
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i >= body) continue;
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < N; ++q) acc8_add<T>(a, v[u][q]);
        const uint4 res = acc8_pack<T>(a);
        if (M == BulkMode::ReduceScatter) {
          st_stream_u4(out16(r) + i * 8, res);
        } else {
#pragma unroll
          for (int q = 0; q < N; ++q) st_stream_u4(out16(q) + e0 + i * 8, res);
        }
      }
    }
  } else {
    // the vector behind the last one read must still be inside the buffer (it is, except in the last shard)
    const int64_t whole = (int64_t(N) * shard_elems - (e0 - h)) / 8 - 1;
    if (body > whole) body = whole < 0 ? 0 : whole;
    for (int64_t i = int64_t(blockIdx.x) * nthreads + tid; i < body; i += int64_t(G) * nthreads) {
      uint4 v[N];
#pragma unroll
      for (int q = 0; q < N; ++q) v[q] = ld_vec_shifted(in16(q) + e0 - h + i * 8, h);
      float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < N; ++q) acc8_add<T>(a, v[q]);
      *reinterpret_cast<uint4*>(out16(r) + i * 8) = acc8_pack<T>(a);
    }
  }
  if (int(blockIdx.x) == G - 1) {  // fewer than 24 elements
    for (int64_t e = body * 8 + tid; e < valid; e += nthreads) {
      float a = 0.f;
#pragma unroll
      for (int q = 0; q < N; ++q) a += float(reinterpret_cast<const T*>(in16(q))[e0 + e]);
      const T res = T(a);
      if (M == BulkMode::ReduceScatter) {
        reinterpret_cast<T*>(out16(r))[e] = res;
      } else {
#pragma unroll
        for (int q = 0; q < N; ++q) reinterpret_cast<T*>(out16(q))[o0 + e] = res;
      }
    }
  }
}

// Work split: the buffer is `parts` shards of shard_vec vectors; inside a shard,
// tile j (kU * blockDim vectors) belongs to CTA j % gridDim.x on every rank.
template <typename T, int N, bool NVLS, BulkMode M, BulkPlace P = BulkPlace::Heap>
__global__ void __launch_bounds__(kBulkThreads) bulk_kernel(const __grid_constant__ KArgs args) {
  const RankView& me = args.v[blockIdx.y];
  const HeapLayout& lay = args.lay;
  constexpr int kU = bulk_unroll(N, NVLS);
  const int tid = int(threadIdx.x);
  const int nthreads = int(blockDim.x);
  const int G = int(gridDim.x);
  const int b = int(blockIdx.x);
  const int r = me.rank;
  const size_t sym_off = size_t(me.aux[0]);
  const bool copy_in = (me.aux[1] & kBulkCopyIn) != 0;
  const bool copy_out = (me.aux[1] & kBulkCopyOut) != 0;

  // Shards.  In the caller's buffer shard s holds shard_elems elements starting at
  // s * shard_elems (AllReduce: a vector-aligned cut of the whole buffer;
  // ReduceScatter: nelems / N; AllGather: nelems = one rank's contribution).  In the
  // symmetric buffer shard s starts at vector s * shard_vec.
  const int64_t nelems = int64_t(me.nelems);
  int64_t shard_elems, shard_vec;
  if (M == BulkMode::AllReduce) {
    const int64_t total_vec = (nelems + 7) / 8;
    shard_vec = (total_vec + N - 1) / N;
    shard_elems = shard_vec * 8;
  } else if (M == BulkMode::ReduceScatter) {
    shard_elems = nelems / N;
    shard_vec = (shard_elems + 7) / 8;
  } else {
    shard_elems = nelems;
    shard_vec = (shard_elems + 7) / 8;
  }
  auto valid = [&](int s) -> int64_t {
    if (M != BulkMode::AllReduce) return shard_elems;
    int64_t v = nelems - int64_t(s) * shard_elems;
    return v < 0 ? 0 : (v > shard_elems ? shard_elems : v);
  };
  if constexpr (P == BulkPlace::Direct) {
    // launched while the kernel before may still run: nothing is touched before the wait, and the next launch is let in at once
    pdl_launch_dependents();
    pdl_wait();
    bulk_direct_body<T, N, M>(args, r, shard_elems, valid(r));
    return;
  }
  uint32_t bar = me.bar_seq;
  if (me.seq_dev) bar += ld_volatile_u32(me.seq_dev + 2);
  // A slab is blockDim consecutive vectors; slab j belongs to CTA j % gridDim.x on every rank
  // and a CTA keeps kU of its slabs in flight.
  const int64_t ntiles = (shard_vec + nthreads - 1) / nthreads;

  char* my_buf = me.heap + sym_off;
  const uint16_t* in16 = static_cast<const uint16_t*>(me.in);
  uint16_t* out16 = static_cast<uint16_t*>(me.out);

  // ---- phase 0: stage the input ------------------------------------------------
  if (M != BulkMode::AllGather && copy_in) {
    for (int s = 0; s < N; ++s) {
      const int64_t nv = valid(s);
      for (int64_t tile = b; tile < ntiles; tile += int64_t(G) * kU)
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
          if (i < shard_vec && i * 8 < nv)
            *reinterpret_cast<uint4*>(my_buf + (int64_t(s) * shard_vec + i) * 16) =
                ld_vec_guarded(in16 + int64_t(s) * shard_elems, i, nv);
        }
    }
  }
  // Every rank has arrived (so it has left the previous collective and, for the
  // reducing modes, its input is in place) before any remote access.
  if (!cta_rank_barrier(me, lay, bar + 1, 10, /*publish=*/copy_in)) return;

  // ---- phase 1: the collective ---------------------------------------------------
  if (M == BulkMode::AllGather) {
    const uint16_t* src16 = copy_in ? in16 : reinterpret_cast<const uint16_t*>(my_buf + int64_t(r) * shard_vec * 16);
    for (int64_t tile = b; tile < ntiles; tile += int64_t(G) * kU) {
      uint4 v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i < shard_vec) v[u] = ld_vec_guarded(src16, i, shard_elems);
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i >= shard_vec) continue;
        const size_t off = sym_off + size_t(int64_t(r) * shard_vec + i) * 16;
        if (me.flags & kMuteSends) continue;
        if (NVLS) {
          multimem_st_v4(me.mc + off, v[u]);
        } else {
#pragma unroll
          for (int k = 0; k < N; ++k) {
            const int q = (r + k) % N;
            if (q == r && !copy_in) continue;
            *reinterpret_cast<uint4*>(me.peer[q] + off) = v[u];
          }
        }
      }
    }
  } else {
    for (int64_t tile = b; tile < ntiles; tile += int64_t(G) * kU) {
      uint4 res[kU];
      if (NVLS) {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
          if (i < shard_vec)
            res[u] = multimem_ld_reduce_add<T>(me.mc + sym_off + size_t(int64_t(r) * shard_vec + i) * 16);
        }
      } else {
        uint4 v[kU][N];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
          if (i < shard_vec) {
            const size_t off = sym_off + size_t(int64_t(r) * shard_vec + i) * 16;
#pragma unroll
            for (int q = 0; q < N; ++q) v[u][q] = ld_volatile_u4(me.peer[q] + off);
          }
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int q = 0; q < N; ++q) acc8_add<T>(a, v[u][q]);
          res[u] = acc8_pack<T>(a);
        }
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
        if (i >= shard_vec) continue;
        if (M == BulkMode::ReduceScatter) {
          st_vec_guarded(out16, i, shard_elems, res[u]);  // my shard only, straight to the caller
        } else if (!(me.flags & kMuteSends)) {
          const size_t off = sym_off + size_t(int64_t(r) * shard_vec + i) * 16;
          if (NVLS) {
            multimem_st_v4(me.mc + off, res[u]);
          } else {
#pragma unroll
            for (int k = 0; k < N; ++k) {
              const int q = (r + k) % N;
              *reinterpret_cast<uint4*>(me.peer[q] + off) = res[u];
            }
          }
        }
      }
    }
  }

  // ---- phase 2: everyone's loads and stores are done ---------------------------------
  if (!cta_rank_barrier(me, lay, bar + 2, 11, /*publish=*/true)) return;

  // ---- phase 3: hand the result to the caller ----------------------------------------
  if (M != BulkMode::ReduceScatter && copy_out) {
    for (int s = 0; s < N; ++s) {
      const int64_t nv = valid(s);
      for (int64_t tile = b; tile < ntiles; tile += int64_t(G) * kU)
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const int64_t i = (tile + int64_t(u) * G) * nthreads + tid;
          if (i < shard_vec && i * 8 < nv)
            st_vec_guarded(out16 + int64_t(s) * shard_elems, i, nv, ld_volatile_u4(my_buf + (int64_t(s) * shard_vec + i) * 16));
        }
    }
  }

  // ---- device-side sequence counter (graph-captured launches) ---------------------------
  if (me.seq_dev) {
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(me.seq_dev + 1, 1u) == gridDim.x - 1) {
        me.seq_dev[1] = 0;
        me.seq_dev[2] += 4;
        __threadfence();
      }
    }
  }
}

using BulkKernelFn = void (*)(const KArgs);
BulkKernelFn bulk_lookup(DType t, int world, bool nvls, BulkMode m);
BulkKernelFn bulk_direct_lookup(DType t, int world, BulkMode m);

}  // namespace b200ipc
