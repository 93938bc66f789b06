// The linear layers of gemm_local.cuh for the few rows of a decode step: at most 64 rows of X, so that what counts is the
// stream of W from memory.  As there, every rank's operands are in one address space and nothing is exchanged.
//
// One tile per CTA (cluster): 128 rows of W (the tensor core's M side) and all rows of X, padded to 16, 32 or 64 (its N side).  K is
// split over the CTAs of a cluster until tiles x splits fill the places; every CTA hands its fp32 partial sums for a share of the
// rows of X to the CTA that owns them (st.async, counted on the receiver's barrier), and the owner adds them in a fixed order.
//
// What bounds it is the chain around the stream: launch and first loads 4.5 us, split sum, epilogue and exit 4, norm 2.6 of the
// 17.2 us that 16 rows x 3584 x 8192 with norm took in the kernel of gemm_local.cuh, one launch after the other.  So this one is
// cut to let the next launch in: 106 KB of shared memory, 72 or 80 registers x 320 threads and 64 columns of tensor memory leave
// room for a second CTA on the SM, and dependents are let go at once.  The next kernel's CTAs set up and bring the first 24 MB of
// W to L2 as soon as there is room for them, while this kernel's stragglers or its norm are at work.  Now 13.5 us (one row 17.0 ->
// 12.6, 32 rows 17.9 -> 14.5, 2048 x 6016 12.0 -> 9.2, 8192 x 7168 26.0 -> 23.3, back to back; 0.3 of it the norm).  0.2 - 0.5 of that came with the
// cluster's barrier in two halves: a warp arrives when it has sent its sums and has the others', and its stores pass while the rest
// of the cluster gets there.  With less of W fetched ahead the memory idles between the launches (16 MB: +0.5), more takes from the
// stream of the kernel in front (40 MB: +1.6).
#pragma once

#include "gemm_local.cuh"

namespace b200ipc {

constexpr int kStrThreads = 320;  // warp 0: TMA, warp 1: MMA, warps 2-5 and 6-9: two epilogue groups
constexpr int kStrWRows = 128;
constexpr int kStrMaxRows = 64;   // rows of X
constexpr int kStrTmemCols = 64;  // accumulator columns
constexpr int kStrMaxStages = 8;
constexpr int kStrSmemBudget = 106 * 1024;
constexpr int kStrTileBytes = kStrWRows * kGemmBK * 2;  // a stage's block of W
constexpr int64_t kStrWarmBytes = int64_t(24) << 20;    // of W that a launch brings to L2 before its wait

struct StreamGemmArgs {
  alignas(64) CUtensorMap tma_x[kMaxRanks];  // X of rank r [rows, K], box 64 x BN
  alignas(64) CUtensorMap tma_w[kMaxRanks];  // W of rank r [N, K], box 64 x 128
  const void* w[kMaxRanks];
  const void* residual[kMaxRanks];           // [rows, N] or nullptr (linear only)
  void* sum[kMaxRanks];                      // [rows, N]: the result before the norm
  void* copy[kMaxRanks];                     // [rows, N] or nullptr: a second copy of it
  StatusBlock* status;
  uint32_t* abort_word;
  uint64_t timeout_ns;
  int rank;
  int rows;         // rows of X per shard
  int N, K;
  int segs;         // ranks whose K slices follow one another (linear: world, else 1)
  int merged;       // X is the rows of this many shards, merged_rows columns of the tile each; else 0
  int merged_rows;
  int groups;       // products with a W and an output of their own (linear: 1, else world)
  int n_tiles;
  int splits;       // K splits = CTAs per cluster
  int stages;
  int mute;         // the partial sums stay unsent (failure injection)
  int warm;         // k blocks of W that a CTA brings to L2 before the wait for the previous kernel
};

// 2, 4 or 8 accumulator columns of the warp's 32 lanes
template <int O>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[O]) {
  if constexpr (O == 2)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr) : "memory");
  else if constexpr (O == 4)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
  else
    tmem_ld_8cols(taddr, r);
}

// BN: columns of the accumulator: 16, 32 or 64.
template <typename T, int BN>
__global__ void __launch_bounds__(kStrThreads, 2) gemm_stream_kernel(const __grid_constant__ StreamGemmArgs args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t full[kStrMaxStages], empty[kStrMaxStages], acc_full, slab_full, mma_done;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = int(threadIdx.x & 31);
  const int splits = args.splits, split = int(cluster_rank());
  const int tile = int(blockIdx.x) / splits;
  const int group = tile / args.n_tiles, n0 = (tile - group * args.n_tiles) * kStrWRows;
  const int N = args.N, rows = args.rows, stages = args.stages;
  const uint32_t w_bytes = kStrTileBytes, x_bytes = uint32_t(BN) * kGemmBK * 2, stage_bytes = w_bytes + x_bytes;
  const int kb_seg = (args.K + kGemmBK - 1) / kGemmBK;  // columns past K read as zeros
  const int kb_total = kb_seg * args.segs;
  const int kb0 = int(int64_t(kb_total) * split / splits), kb1 = int(int64_t(kb_total) * (split + 1) / splits);
  const int own = BN / splits;  // rows of X whose sums this CTA finishes: a multiple of 4
  const uint64_t timeout_ns = args.timeout_ns;
  volatile int* abort_flag = &s_abort;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&slab_full, 1);
    mbar_init(&mma_done, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  struct KPos {
    const CUtensorMap *w, *x;
    int col;
  };
  auto first_k = [&]() {
    const int seg = kb0 / kb_seg;
    return KPos{&args.tma_w[args.groups > 1 ? group : seg], &args.tma_x[args.groups > 1 ? 0 : seg], (kb0 - seg * kb_seg) * kGemmBK};
  };
  auto next_k = [&](KPos& k) {
    k.col += kGemmBK;
    if (k.col >= args.K) {  // the next rank's slice (with one slice per product this is past the last block)
      k.col = 0;
      ++k.w;
      ++k.x;
    }
  };
  // Nothing is loaded before the wait, W included: the kernel before this one may write it.  The epilogue's threads bring the
  // first blocks of this CTA's share to L2, a row's 128 bytes each (TMA prefetches would stand in front of the first loads).
  if (warp >= 2) {
    const int rows_w = min(kStrWRows, N - n0), blocks = min(kb1 - kb0, args.warm);
    const int r = (int(threadIdx.x) - 64) & (kStrWRows - 1), part = (int(threadIdx.x) - 64) / kStrWRows;  // a row, every other block
    if (r < rows_w) {
      for (int b = part; b < blocks; b += 2) {
        const int seg = (kb0 + b) / kb_seg, block = kb0 + b - seg * kb_seg;
        const char* p = static_cast<const char*>(args.w[args.groups > 1 ? group : seg]) + (size_t(n0 + r) * size_t(args.K) + size_t(block * kGemmBK)) * 2;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
      }
    }
  }
  if (warp == 1) {
    tmem_alloc(&s_tmem, kStrTmemCols);
    tmem_relinquish();
  }
  __syncwarp();
  tc_fence_before_sync();
  cluster_sync_all();  // peers store into this CTA's shared memory and count on its barrier
  tc_fence_after_sync();
  const uint32_t tmem_base = s_tmem;
  const uint32_t ring_addr = smem_u32(ring);
  pdl_wait();

  if (warp == 0) {
    if (elect_one()) {
      uint32_t st = 0, ph = 1;
      int it = 0;
      KPos k = first_k();
      const uint64_t policy = evict_first_policy();
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb, ++it, next_k(k)) {
        if (!mbar_wait_long(&empty[st], ph, abort_flag, timeout_ns)) break;
        mbar_expect_tx(&full[st], stage_bytes);
        unsigned char* dst = ring + st * stage_bytes;
        tma_stream_2d(dst, k.w, &full[st], k.col, n0, policy);
        if (args.merged == 0) {
          tma_load_2d(dst + w_bytes, k.x, &full[st], k.col, 0);
        } else {
          for (int i = 0; i < args.merged; ++i)
            tma_load_2d(dst + w_bytes + uint32_t(i * args.merged_rows) * 128u, k.x + i, &full[st], k.col, 0);
        }
        if (++st == uint32_t(stages)) {
          st = 0;
          ph ^= 1u;
        }
      }
      // copies in flight land before the CTA leaves
      const uint64_t t0 = globaltimer_ns();
      for (int back = 1; back <= min(it, stages); ++back)
        mbar_drain(&full[(it - back) % stages], uint32_t((it - back) / stages) & 1u, t0);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc<T>(kStrWRows, BN);
      uint32_t st = 0, ph = 0;
      bool ok = true;
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_long(&full[st], ph, abort_flag, timeout_ns)) { ok = false; break; }
        tc_fence_after_sync();
        const uint64_t da = make_sw128_kmajor_desc(ring_addr + st * stage_bytes);
        const uint64_t db = make_sw128_kmajor_desc(ring_addr + st * stage_bytes + w_bytes);
#pragma unroll
        for (int k = 0; k < kGemmBK / 16; ++k)
          umma_f16(tmem_base, da + uint64_t(2 * k), db + uint64_t(2 * k), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        umma_commit(&empty[st]);
        if (++st == uint32_t(stages)) {
          st = 0;
          ph ^= 1u;
        }
      }
      if (ok) umma_commit(&acc_full);
      umma_commit(&mma_done);
      mbar_drain(&mma_done, 0, globaltimer_ns());
    }
  } else {
    // ---- epilogue: lane = a row of W (an output column), accumulator columns = rows of X, one half of them per group.  A warp's
    // store of one X row is 64 contiguous bytes. ----
    const int half = warp >= 6 ? 1 : 0;
    const int my_n = (warp & 3) * 32 + lane;
    const uint32_t tmem_lane = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const bool col_ok = n0 + my_n < N;
    const size_t col = size_t(n0 + my_n);
    const int valid = args.merged ? BN : rows;  // accumulator columns that mean something
    // [splits - 1][own][128] fp32 behind the ring, in split order
    float* slab = reinterpret_cast<float*>(ring + size_t(stages) * stage_bytes);
    if (splits > 1 && threadIdx.x == 64)
      mbar_expect_tx(&slab_full, uint32_t(splits - 1) * uint32_t(max(0, min(own, (valid - split * own + 3) / 4 * 4))) * 512u);
    constexpr int kChunk = 8;
    const int q0 = args.groups > 1 ? group : 0, q1 = args.groups > 1 ? group + 1 : args.segs;
    const int width = own / 2, first = split * own + half * width;  // the rows that this group finishes
    const int mine = col_ok ? min(width, valid - first) : 0;        // ... and this lane stores
    const size_t at0 = size_t(first) * size_t(N) + col;
    T rv[kChunk];  // the first chunk's residual is on its way before the accumulator is complete
    const T* res0 = static_cast<const T*>(args.residual[0]);
    auto load_residual = [&](const T* res, int c) {
      const T* p = res + at0 + size_t(c) * size_t(N);
#pragma unroll
      for (int j = 0; j < kChunk; ++j)
        if (c + j < mine) rv[j] = p[size_t(j) * size_t(N)];
    };
    if (res0) load_residual(res0, 0);
    bool ok = !__any_sync(0xffffffffu, !mbar_wait_long(&acc_full, 0, abort_flag, timeout_ns));
    if (ok) {
      tc_fence_after_sync();
      if (splits > 1) {  // the others' shares to them, straight from the registers
        constexpr int H = BN / 2;
        const int sent = args.mute ? 0 : (valid + 3) / 4 * 4;
        uint32_t acc[H];
#pragma unroll
        for (int c = 0; c < H; c += 8) tmem_ld_8cols(tmem_lane + uint32_t(half * H + c), acc + c);
        tmem_ld_wait();
        uint32_t dst = 0, bar = 0;
        int o = 0;
#pragma unroll
        for (int j = 0; j < H; ++j) {
          const int c = half * H + j;
          if (j == 0 || (j % 4 == 0 && (c & (own - 1)) == 0)) {
            o = c / own;
            dst = map_to_cta(smem_u32(slab + (size_t(split < o ? split : split - 1) * own + size_t(c - o * own)) * 128 + my_n), uint32_t(o)) - uint32_t(j) * 512u;
            bar = map_to_cta(smem_u32(&slab_full), uint32_t(o));
          }
          if (o != split && c < sent) st_async(dst + uint32_t(j) * 512u, acc[j], bar);
        }
        ok = !__any_sync(0xffffffffu, !mbar_wait_long(&slab_full, 0, abort_flag, timeout_ns));
        asm volatile("fence.acq_rel.cluster;" ::: "memory");
      }
    }
    __syncwarp();
    if (splits > 1) cluster_arrive();  // this warp has sent its sums and has all of the others'
    // Rows c .. c + O of this group's share.
    auto finish = [&](auto count, int c) {
      constexpr int O = decltype(count)::value;
      uint32_t acc[O];
      tmem_ld_cols<O>(tmem_lane + uint32_t(first + c), acc);
      tmem_ld_wait();
      float v[O];
#pragma unroll
      for (int j = 0; j < O; ++j) v[j] = __uint_as_float(acc[j]);
      const float* sp = slab + size_t(half * width + c) * 128 + my_n;
#pragma unroll 1
      for (int s = 0; s < splits - 1; ++s, sp += size_t(own) * 128) {
#pragma unroll
        for (int j = 0; j < O; ++j) v[j] += sp[size_t(j) * 128];
      }
      if (args.merged) {  // the tile's columns are the rows of several shards, with padding between them
        T* sum = static_cast<T*>(args.sum[q0]) + col;
        int shard = (first + c) / args.merged_rows, m = first + c - shard * args.merged_rows;
#pragma unroll
        for (int j = 0; j < O; ++j) {
          if (c + j < mine && m < rows) sum[(size_t(shard) * size_t(rows) + size_t(m)) * size_t(N)] = T(v[j]);
          if (++m == args.merged_rows) {
            m = 0;
            ++shard;
          }
        }
        return;
      }
      const size_t at = at0 + size_t(c) * size_t(N);
#pragma unroll 1
      for (int q = q0; q < q1; ++q) {
        T* sum = static_cast<T*>(args.sum[q]) + at;
        const T* res = static_cast<const T*>(args.residual[q]);
        if (res && (q > q0 || c > 0)) load_residual(res, c);
        T* copy = args.copy[q] ? static_cast<T*>(args.copy[q]) + at : nullptr;
#pragma unroll
        for (int j = 0; j < O; ++j) {
          if (c + j >= mine) continue;
          const T y = T(res ? v[j] + float(rv[j]) : v[j]);
          sum[size_t(j) * size_t(N)] = y;
          if (copy) copy[size_t(j) * size_t(N)] = y;
        }
      }
    };
    if (ok) {
      if (width == 2) {
        finish(std::integral_constant<int, 2>(), 0);
      } else if (width == 4) {
        finish(std::integral_constant<int, 4>(), 0);
      } else {
#pragma unroll 1
        for (int c = 0; c < width && first + c < valid; c += kChunk) finish(std::integral_constant<int, kChunk>(), c);
      }
    }
  }

  // ---- a CTA leaves when nobody will store into it any more; tensor memory goes back -------------------------------------
  __syncwarp();
  if (splits > 1 && warp < 2) cluster_arrive();
  tc_fence_before_sync();
  __syncthreads();
  if (splits > 1) cluster_wait();
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc(tmem_base, kStrTmemCols);
  if (*abort_flag && threadIdx.x == 0) {
    if (splits > 1) mbar_drain(&slab_full, 0, globaltimer_ns());  // what the others had sent before they got here
    st_volatile_u32(args.abort_word, 1u);
    if (claim_status(args.abort_word, kTimeout)) {
      StatusBlock* sb = args.status;
      sb->rank = uint32_t(args.rank);
      sb->peer = uint32_t(args.rank);
      sb->wire = blockIdx.x;
      sb->where = 41;  // a pipeline wait of the weight-streaming kernel gave up
      __threadfence_system();
      sb->code = kTimeout;
      __threadfence_system();
    }
  }
}

}  // namespace b200ipc
