// The row-parallel linear layer + all-reduce (+ residual + RMSNorm) and the all-gather + column-parallel linear
// layer when every rank's data is in ONE GPU's address space: a world of one, and emulated worlds.  Nothing has to be
// exchanged there, so there is no landing zone, no flag and no wait on another CTA's work:
//
//   linear         Y = sum over r of X_r W_r^T is ONE contraction over the ranks' concatenated K: the ranks' slices
//                  follow one another into the same accumulator, and the epilogue writes every rank's output
//                  (+ its residual).  The sum is rounded once.  RMSNorm is a second, tiny kernel over rows that are
//                  still in L2 (programmatic dependent launch).
//   gather linear  Y_r = concat_q(X_q) W_r^T reads the shards where they are; no tile straddles two shards.
//
// Both are the same kernel.  The operands are swapped (the tensor core's M side is a tile of 256 rows of W, its N side
// is BN rows of X, BN any multiple of 32 up to 256), so that a ragged or small number of rows wastes no tensor time
// and one tile shape serves decode and prefill.  Two SMs share a tile (cta_group::2): each holds 128 rows of W and half
// of the X rows, which halves what a tile reads through shared memory per FLOP.  Warp 0 issues the TMA loads (no
// multicast), warp 1 of the even CTA the tcgen05.mma, warps 2-9 read the accumulator (double-buffered in tensor memory),
// round and store.
//
// Many tiles: those behind the last full wave are cut in two or four along X, so that the wave which fills a fraction of the GPU
// is a shorter one (2048 rows x 3584 x 8192 with norm, 256 tiles for 74 pairs: 127 -> 121 us at the power cap).
//
// Few tiles (decode, narrow layers): K is split over the pairs of a cluster of 2, 4 or 8 CTAs; after the last MMA every
// pair hands its fp32 partial sums for a share of the rows to the pair that owns them through distributed shared
// memory (st.async, counted on the receiver's barrier), and the owners add them in a fixed order (the result does not depend on
// timing) and run the epilogue.
// What bounds it, one B200: a large product the tensor pipe (98 % of active cycles at 2 x 4096 x 8192 x 7168, 657 us at the
// power cap, the kernel with the exchange 950); one row of tiles per SM pair or less, the chain of launch, first loads (2.5 us)
// and epilogue (0.9 + 0.013 BN us); up to 64 rows the weight stream, where gemm_stream.cuh is ahead (16 x 3584 x 8192 with norm 17.2 us here, 13.5).
// The issuing threads had bounded it before: a lane picked by its number made every MMA and TMA copy cost ~90 ns (elect.sync:
// 393 -> 302 ns per 256 x 256 x 64 block), and integer divisions of the ring position another 160 ns of the loads' loop.
// Epilogue: 2-byte stores, 64 contiguous bytes of a row per warp, 3.3 us per 256 x 256 tile; transposed through shared memory
// with 16-byte stores 4.1, with TMA stores 5.4, with 4 x 4 shuffles and 8-byte stores 5.9.
#pragma once

#include "gemm_ar.cuh"

namespace b200ipc {

constexpr int kLocThreads = 320;      // warp 0: TMA, warp 1: MMA, warps 2-5 and 6-9: two epilogue groups
constexpr int kLocWRows = 256;        // rows of W per tile (128 per CTA of the pair)
constexpr int kLocMaxBN = 256;        // rows of X per tile
constexpr int kLocMaxStages = 10;
constexpr int kLocChunk = 16;         // rows of X an epilogue warp takes at a time
constexpr int kLocSmemBudget = 226 * 1024;

struct LocalGemmArgs {
  alignas(64) CUtensorMap tma_x[kMaxRanks];  // X of rank r [rows, K], box 64 x BN / 2
  alignas(64) CUtensorMap tma_w[kMaxRanks];  // W of rank r [N, K], box 64 x 128
  alignas(64) CUtensorMap tma_x_cut[kMaxRanks];  // X of rank r, box 64 x BN / cut / 2
  const void* residual[kMaxRanks];           // [M, N] or nullptr (linear only)
  void* sum[kMaxRanks];                      // [M, N]: the result before the norm
  void* copy[kMaxRanks];                     // [M, N] or nullptr: a second copy of it
  StatusBlock* status;
  uint32_t* abort_word;
  uint64_t timeout_ns;
  int rank;
  int rows;      // rows of X per shard
  int N, K;
  int segs;      // ranks whose K slices follow one another (linear: world, gather: 1)
  int shards;    // row shards of X that a tile lies in one of (linear: 1, gather: world)
  int merged;    // gather of few rows: the tile holds the rows of this many shards, merged_rows each; else 0
  int merged_rows;  // rows a shard takes in such a tile: `rows` rounded up to whole swizzle blocks
  int groups;    // products with a W and an output of their own (linear: 1, gather: world)
  int bn;        // X rows per tile
  int cut, cut_from;  // BN > 128: tiles from number cut_from on are taken in `cut` parts of BN / cut rows
  int m_tiles;   // per shard
  int n_tiles;
  int band;      // m-tiles visited before the next W tile
  int splits;    // K splits = pairs per cluster
  int mute;      // the partial sums stay unsent (failure injection)
  int stages;
  int warm_w;    // the first stages' W boxes are brought to L2 before the wait for the previous kernel
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The two halves apart: every thread of the cluster's CTAs arrives once, and waits for all of them later.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr), "r"(rank));
  return a;
}
// Store into another CTA's shared memory whose bytes are counted on a barrier of that CTA.
__device__ __forceinline__ void st_async(uint32_t cluster_addr, uint32_t v, uint32_t bar_cluster) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(cluster_addr), "r"(v), "r"(bar_cluster)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// The tile lands in this CTA; the bytes are counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar_cluster, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair once the MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(mask)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_8cols(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_16cols(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr)
               : "memory");
}

// Where tile t lies: (group, first X row inside the shard, shard, first W row).
struct LocTile {
  int group, shard, m0, n0, bn;
};
template <bool CUT>
__device__ __forceinline__ LocTile loc_tile(const LocalGemmArgs& a, int t) {
  const int mt_all = a.shards * a.m_tiles;
  const int per_group = mt_all * a.n_tiles;
  LocTile o;
  o.bn = a.bn;
  int part = 0;
  if (CUT && t >= a.cut_from) {
    o.bn = a.bn / a.cut;
    part = (t - a.cut_from) % a.cut;
    t = a.cut_from + (t - a.cut_from) / a.cut;
  }
  o.group = t / per_group;
  int u = t % per_group;
  const int per_band = a.band * a.n_tiles;
  const int band = u / per_band;
  u %= per_band;
  int width = mt_all - band * a.band;
  if (width > a.band) width = a.band;
  const int m = band * a.band + u % width;
  o.n0 = (u / width) * kLocWRows;
  o.shard = m / a.m_tiles;
  o.m0 = (m % a.m_tiles) * a.bn + part * o.bn;
  return o;
}

// KSUB: 64-column k blocks per stage.
template <typename T, int KSUB>
__global__ void __launch_bounds__(kLocThreads, 1) gemm_local_kernel(const __grid_constant__ LocalGemmArgs args) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t full[kLocMaxStages], empty[kLocMaxStages], acc_full[2], acc_empty[2], slab_full, mma_done;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = int(threadIdx.x & 31);
  const uint32_t crank = cluster_rank();
  const int splits = args.splits;
  const int side = int(crank & 1);       // which CTA of the pair
  const int split = int(crank >> 1);     // which pair of the cluster = which share of K
  const int cluster = int(blockIdx.x) / (2 * splits);
  const int nclusters = int(gridDim.x) / (2 * splits);
  const int bn = args.bn, N = args.N, rows = args.rows;
  const int stages = args.stages;
  const uint32_t a_bytes = 128 * kGemmBK * 2;
  const uint32_t blk_bytes = a_bytes + uint32_t(bn / 2) * kGemmBK * 2;  // a k block of this CTA: W rows, then X rows
  const uint32_t stage_bytes = blk_bytes * KSUB;
  const int kb_seg = (args.K + kGemmBK - 1) / kGemmBK;  // columns past K read as zeros
  const int kb_total = kb_seg * args.segs;
  const int kb0 = int(int64_t(kb_total) * split / splits), kb1 = int(int64_t(kb_total) * (split + 1) / splits);
  const int tiles = args.groups * args.shards * args.m_tiles * args.n_tiles;
  const int total = KSUB > 1 ? tiles : args.cut_from + (tiles - args.cut_from) * args.cut;
  const uint64_t timeout_ns = args.timeout_ns;
  volatile int* abort_flag = &s_abort;

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 16);  // eight epilogue warps of both CTAs
    }
    mbar_init(&slab_full, 1);
    mbar_init(&mma_done, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  __syncwarp();
  tc_fence_before_sync();
  cluster_sync_all();  // the peer signals these barriers
  tc_fence_after_sync();
  const uint32_t tmem_base = s_tmem;

  // One k block of a tile is a stage: this CTA's 128 rows of W and its half of the X rows, counted on the even CTA's
  // barrier.  The loops below run in one thread each and what they spend per k block bounds the kernel, so stage, phase,
  // column and rank are counted and not divided out.
  const uint32_t ring_addr = smem_u32(ring);
  const uint32_t full_pair = map_to_cta(smem_u32(&full[0]), crank & ~1u);
  struct KPos {
    const CUtensorMap *w, *x;
    int col;
  };
  auto first_k = [&](const LocTile& t) {
    const int seg = kb0 / kb_seg;
    return KPos{&args.tma_w[args.groups > 1 ? t.group : seg], &(KSUB > 1 || t.bn == bn ? args.tma_x : args.tma_x_cut)[args.shards > 1 ? t.shard : seg], (kb0 - seg * kb_seg) * kGemmBK};
  };
  auto next_k = [&](KPos& k) {
    k.col += kGemmBK;
    if (k.col >= args.K) {  // the next rank's slice (with one slice per product this is past the last block)
      k.col = 0;
      ++k.w;
      ++k.x;
    }
  };
  auto load_w = [&](uint32_t st, int sub, const KPos& k, const LocTile& t) {
    tma_load_2d_pair(ring_addr + st * stage_bytes + uint32_t(sub) * blk_bytes, k.w, full_pair + st * 8, k.col, t.n0 + side * 128);
  };
  auto load_x = [&](uint32_t st, int sub, const KPos& k, const LocTile& t) {
    const uint32_t dst = ring_addr + st * stage_bytes + uint32_t(sub) * blk_bytes + a_bytes;
    if (args.merged == 0) {
      tma_load_2d_pair(dst, k.x, full_pair + st * 8, k.col, t.m0 + side * (t.bn / 2));
    } else {
      const int per_side = args.merged / 2;
      for (int i = 0; i < per_side; ++i)
        tma_load_2d_pair(dst + uint32_t(i * args.merged_rows) * 128u, k.x + side * per_side + i, full_pair + st * 8, k.col, 0);
    }
  };
  // No load before the wait: W may be what the kernel before this one writes (the entry points themselves copy a strided one).
  if (args.warm_w && warp == 0 && cluster < total && elect_one()) {
    const LocTile t = loc_tile<KSUB == 1>(args, cluster);
    KPos k = first_k(t);
    if (t.n0 + side * 128 < N)
      for (int kb = kb0; kb < min(kb1, kb0 + stages * KSUB); ++kb, next_k(k)) tma_prefetch_2d(k.w, k.col, t.n0 + side * 128);
  }
  pdl_wait();
  pdl_launch_dependents();  // after the wait: whoever starts early finds everything before this kernel complete

  if (warp == 0) {
    if (elect_one()) {
      uint32_t it = 0, st = 0, ph = 1;
      for (int tt = cluster; tt < total && !*abort_flag; tt += nclusters) {
        const LocTile t = loc_tile<KSUB == 1>(args, tt);
        KPos k = first_k(t);
        const uint32_t tile_bytes = 2 * (a_bytes + uint32_t(t.bn / 2) * kGemmBK * 2);  // a k block of both CTAs
#pragma unroll 1
        for (int kb = kb0; kb < kb1; kb += KSUB, ++it) {
          const int nsub = KSUB == 1 ? 1 : min(KSUB, kb1 - kb);
          if (!mbar_wait_long(&empty[st], ph, abort_flag, timeout_ns)) break;
          if (side == 0) mbar_expect_tx(&full[st], tile_bytes * uint32_t(nsub));
#pragma unroll
          for (int sub = 0; sub < KSUB; ++sub) {
            if (sub >= nsub) break;
            load_w(st, sub, k, t);
            load_x(st, sub, k, t);
            next_k(k);
          }
          if (++st == uint32_t(stages)) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
      // copies in flight land in the pair's shared memory: the even CTA sees them all arrive
      const uint64_t t0 = globaltimer_ns();
      if (side == 0)
        for (uint32_t back = 0; back < uint32_t(stages) && back < it; ++back) {
          const uint32_t j = it - 1 - back;
          mbar_drain(&full[j % uint32_t(stages)], (j / uint32_t(stages)) & 1u, t0);
        }
    }
  } else if (warp == 1) {
    if (side == 0 && elect_one()) {
      const uint16_t mask = uint16_t(3u << (crank & ~1u));
      uint32_t st = 0, ph = 0, i = 0;
      for (int tt = cluster; tt < total && !*abort_flag; tt += nclusters, ++i) {
        const uint32_t buf = i & 1u;
        const uint32_t idesc = make_idesc<T>(kLocWRows, KSUB > 1 || tt < args.cut_from ? bn : bn / args.cut);
        if (!mbar_wait_long(&acc_empty[buf], ((i >> 1) & 1u) ^ 1u, abort_flag, timeout_ns)) break;
        tc_fence_after_sync();
        bool ok = true;
#pragma unroll 1
        for (int kb = kb0; kb < kb1; kb += KSUB) {
          if (!mbar_wait_long(&full[st], ph, abort_flag, timeout_ns)) { ok = false; break; }
          tc_fence_after_sync();
          const int nsub = KSUB == 1 ? 1 : min(KSUB, kb1 - kb);
#pragma unroll
          for (int sub = 0; sub < KSUB; ++sub) {
            if (sub >= nsub) break;
            const uint64_t da = make_sw128_kmajor_desc(ring_addr + st * stage_bytes + uint32_t(sub) * blk_bytes);
            const uint64_t db = make_sw128_kmajor_desc(ring_addr + st * stage_bytes + uint32_t(sub) * blk_bytes + a_bytes);
#pragma unroll
            for (int k = 0; k < kGemmBK / 16; ++k)
              umma_f16_pair(tmem_base + buf * kLocMaxBN, da + uint64_t(2 * k), db + uint64_t(2 * k), idesc,
                            (kb > kb0 || sub > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty[st], mask);
          if (++st == uint32_t(stages)) {
            st = 0;
            ph ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit_pair(&acc_full[buf], mask);
      }
    }
  }

  // ---- epilogue: lane = a row of W (an output column), accumulator columns = rows of X.  A warp's store of one X row is
  // 64 contiguous bytes; nothing is staged and the warps never meet.  The two groups take turns with the chunks. ----
  const int group = warp >= 6 ? 1 : 0;
  const int my_n = (warp & 3) * 32 + lane;  // within this CTA's 128 columns
  const uint32_t tmem_lane = uint32_t((warp & 3) * 32) << 16;
  const int col_left = N - side * 128 - my_n;  // the lane's column of a tile at n0 exists if n0 < col_left
  // Row c of a tile and this lane's column in an output, and how many of the cw rows from there exist.
  auto out_off = [&](const LocTile& t, int c) {
    return (size_t(t.shard) * rows + size_t(t.m0 + c)) * size_t(N) + size_t(t.n0 + side * 128 + my_n);
  };
  auto tile_rows = [&](const LocTile& t) { return args.merged ? bn : min(t.bn, rows - t.m0); };
  auto rows_left = [&](const LocTile& t, int c, int cw) { return t.n0 < col_left ? min(cw, rows - t.m0 - c) : 0; };
  auto load_residual = [&](const T* res, size_t off, int left, T (&rv)[kLocChunk]) {
    if (left >= kLocChunk) {
#pragma unroll
      for (int j = 0; j < kLocChunk; ++j) rv[j] = res[off + size_t(j) * size_t(N)];
    } else {
#pragma unroll
      for (int j = 0; j < kLocChunk; ++j)
        if (j < left) rv[j] = res[off + size_t(j) * size_t(N)];
    }
  };
  auto store_rows = [&](T* dst, size_t off, int left, auto value) {
    if (left >= kLocChunk) {
#pragma unroll
      for (int j = 0; j < kLocChunk; ++j) dst[off + size_t(j) * size_t(N)] = T(value(j));
    } else {
#pragma unroll
      for (int j = 0; j < kLocChunk; ++j)
        if (j < left) dst[off + size_t(j) * size_t(N)] = T(value(j));
    }
  };
  // Rounds and stores cw (at most kLocChunk) rows of sums from row c of the tile to every rank's output; rv = the residual of the
  // first one (overwritten by the others').
  auto finish_rows = [&](const LocTile& t, int c, int cw, const uint32_t (&acc)[kLocChunk], T (&rv)[kLocChunk]) {
    const int q0 = args.groups > 1 ? t.group : 0, q1 = args.groups > 1 ? t.group + 1 : args.segs;
    const size_t off = out_off(t, c);
    const int left = rows_left(t, c, cw);
    if (args.merged) {
      if (t.n0 >= col_left) return;
      T* dst = static_cast<T*>(args.sum[q0]) + size_t(t.n0 + side * 128 + my_n);
      int shard = c / args.merged_rows, m = c - shard * args.merged_rows;
#pragma unroll
      for (int j = 0; j < kLocChunk; ++j) {
        if (j < cw && m < rows) dst[(size_t(shard) * rows + size_t(m)) * size_t(N)] = T(__uint_as_float(acc[j]));
        if (++m == args.merged_rows) {
          m = 0;
          ++shard;
        }
      }
      return;
    }
    for (int q = q0; q < q1; ++q) {
      T* sum = static_cast<T*>(args.sum[q]);
      const T* res = static_cast<const T*>(args.residual[q]);
      if (res == nullptr) {
        store_rows(sum, off, left, [&](int j) { return __uint_as_float(acc[j]); });
        continue;
      }
      if (q > 0) load_residual(res, off, left, rv);
      auto value = [&](int j) { return __uint_as_float(acc[j]) + float(rv[j]); };
      store_rows(sum, off, left, value);
      if (args.copy[q]) store_rows(static_cast<T*>(args.copy[q]), off, left, value);
    }
  };

  if (splits == 1) {
    if (warp >= 2) {
      const T* res0 = static_cast<const T*>(args.residual[0]);
      uint32_t i = 0;
      for (int tt = cluster; tt < total; tt += nclusters, ++i) {
        const LocTile t = loc_tile<KSUB == 1>(args, tt);
        const uint32_t buf = i & 1u;
        const int valid = tile_rows(t);
        T rv[kLocChunk];
        // the residual is on its way before the accumulator is complete
        const int c0 = group * kLocChunk;
        if (res0) {
          // the tile's residual comes to L2 while the MMAs run: a lane per row, two 128-byte lines
          const int row = int(threadIdx.x) - 64, n = t.n0 + side * 128;
          for (int q = 0; q < args.segs; ++q) {
            const T* r = static_cast<const T*>(args.residual[q]) + (size_t(t.m0) + size_t(row)) * size_t(N) + size_t(n);
            if (row < valid && n < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(r));
            if (row < valid && n + 64 < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(r + 64));
          }
          if (c0 < valid) load_residual(res0, out_off(t, c0), rows_left(t, c0, kLocChunk), rv);
        }
        if (__any_sync(0xffffffffu, !mbar_wait_long(&acc_full[buf], (i >> 1) & 1u, abort_flag, timeout_ns))) break;
        tc_fence_after_sync();
        for (int c = c0; c < valid; c += 2 * kLocChunk) {
          uint32_t acc[kLocChunk];
          tmem_ld_16cols(tmem_base + tmem_lane + buf * kLocMaxBN + uint32_t(c), acc);
          tmem_ld_wait();
          T next[kLocChunk];
          const int cn = c + 2 * kLocChunk;
          if (res0 && cn < valid) load_residual(res0, out_off(t, cn), rows_left(t, cn, kLocChunk), next);
          finish_rows(t, c, kLocChunk, acc, rv);
#pragma unroll
          for (int j = 0; j < kLocChunk; ++j) rv[j] = next[j];
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&acc_empty[buf]), crank & ~1u));
      }
    }
  } else {
    // one tile per cluster
    const LocTile t = loc_tile<KSUB == 1>(args, cluster);
    const int own = bn / splits;  // rows of X whose sums this pair finishes: a multiple of 8
    const int c_own = split * own, valid = tile_rows(t);
    const T* res0 = static_cast<const T*>(args.residual[0]);
    T rv[kLocChunk];
    // What the pairs hand over lies behind the ring: nobody has to wait until the others' MMAs have read theirs.  A piece is
    // 16 rows (8 at the end of a share that is not a multiple of 16); pieces without rows of X are not sent.
    float* slab = reinterpret_cast<float*>(ring + size_t(stages) * stage_bytes);  // [splits - 1][own][128] fp32, in split order
    auto sent_rows = [&](int o) { return o * own >= valid ? 0 : min(own, (valid - o * own + 15) / 16 * 16); };
    if (threadIdx.x == 64) mbar_expect_tx(&slab_full, uint32_t(splits - 1) * uint32_t(sent_rows(split)) * 512u);
    if (warp >= 2) {
      const int c0 = group * kLocChunk;
      if (res0) load_residual(res0, out_off(t, c_own + c0), rows_left(t, c_own + c0, min(own - c0, kLocChunk)), rv);
    }
    const bool bad = warp < 2 || __any_sync(0xffffffffu, !mbar_wait_long(&acc_full[0], 0, abort_flag, timeout_ns));
    if (!bad) {
      tc_fence_after_sync();
      for (int d = 1; d < splits && !args.mute; ++d) {
        const int o = (split + d) % splits;
        const int slot = split < o ? split : split - 1;
        const uint32_t dst = map_to_cta(smem_u32(slab + size_t(slot) * own * 128 + my_n), uint32_t(2 * o + side));
        const uint32_t bar = map_to_cta(smem_u32(&slab_full), uint32_t(2 * o + side));
        for (int c = 16 * group; c < sent_rows(o); c += 32) {
          uint32_t acc[16];
          tmem_ld_8cols(tmem_base + tmem_lane + uint32_t(o * own + c), acc);
          if (c + 8 < own) tmem_ld_8cols(tmem_base + tmem_lane + uint32_t(o * own + c + 8), acc + 8);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < 8 || c + 8 < own) st_async(dst + uint32_t(c + j) * 512u, acc[j], bar);
        }
      }
    }
    if (!bad && !__any_sync(0xffffffffu, !mbar_wait_long(&slab_full, 0, abort_flag, timeout_ns))) {
      asm volatile("fence.acq_rel.cluster;" ::: "memory");
      for (int c = group * kLocChunk; c < own && c_own + c < valid; c += 2 * kLocChunk) {
        const int cw = min(own - c, kLocChunk);
        if (res0 && c >= 2 * kLocChunk) load_residual(res0, out_off(t, c_own + c), rows_left(t, c_own + c, cw), rv);
        uint32_t acc[kLocChunk];
        tmem_ld_8cols(tmem_base + tmem_lane + uint32_t(c_own + c), acc);
        if (cw > 8) tmem_ld_8cols(tmem_base + tmem_lane + uint32_t(c_own + c + 8), acc + 8);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kLocChunk; ++j) {
          if (j >= 8 && cw <= 8) continue;
          const float* sp = slab + size_t(c + j) * 128 + my_n;
          float v = __uint_as_float(acc[j]) + sp[0];
          if (splits > 2) v = (v + sp[size_t(own) * 128]) + sp[size_t(own) * 256];
          acc[j] = __float_as_uint(v);
        }
        finish_rows(t, c_own + c, cw, acc, rv);
      }
    }
  }

  // ---- the pair leaves together; tensor memory goes back ------------------------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1 && side == 0 && *abort_flag) {  // elsewhere the epilogue has seen every accumulator complete
    if (elect_one()) {  // (the lane that issued the MMAs: the same one is elected every time)
      umma_commit_pair(&mma_done, uint16_t(1u << crank));
      mbar_drain(&mma_done, 0, globaltimer_ns());
    }
  }
  __syncwarp();
  cluster_sync_all();
  tc_fence_after_sync();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  if (*abort_flag && threadIdx.x == 0) {
    // What the others had sent before they got here lands first, and copies of an odd CTA that was a stage ahead when the even one,
    // whose barriers count them, gave up.
    const uint64_t t0 = globaltimer_ns();
    if (splits > 1) mbar_drain(&slab_full, 0, t0);
    while (side == 1 && globaltimer_ns() - t0 < kMbarDrainNs) __nanosleep(1000);
    st_volatile_u32(args.abort_word, 1u);
    if (claim_status(args.abort_word, kTimeout)) {
      StatusBlock* sb = args.status;
      sb->rank = uint32_t(args.rank);
      sb->peer = uint32_t(args.rank);
      sb->wire = blockIdx.x;
      sb->where = 40;  // a pipeline wait (TMA / MMA / epilogue hand-over) gave up
      __threadfence_system();
      sb->code = kTimeout;
      __threadfence_system();
    }
  }
}

// out = RMSNorm(sum) * gamma for the rows of every rank (blockIdx.y); `out` may be `sum` itself.  One CTA per row; rows of up to
// 4 x 8 x blockDim elements stay in registers between the statistic and the scaling.  Behind few rows it is bound by its launch;
// behind 2048 rows of 8192 it was by instructions: 18 per element (loads chosen by a flag beside the registers, additions of
// zero, single fp32 operations), 72 % of the issue slots, 16.2 us cold where memory takes 8.  In a body of its own for rows in
// registers, on pairs of fp32: 11 instructions, 13.4 - 14.6 us; 16 rows x 3584 x 8192 with its GEMM 13.7 -> 13.2 us a call.
struct RowNormArgs {
  const void* sum[kMaxRanks];
  const void* gamma[kMaxRanks];
  void* out[kMaxRanks];
  int N;
  float eps;
};
template <typename T>
__global__ void __launch_bounds__(512) row_norm_kernel(const __grid_constant__ RowNormArgs args) {
  constexpr int U = 4;
  __shared__ float s_part[16];
  const int q = int(blockIdx.y), N = args.N, nvec = N / 8, tid = int(threadIdx.x);
  const uint4* gamma = static_cast<const uint4*>(args.gamma[q]);
  const int step = int(blockDim.x);
  const bool in_regs = nvec <= U * step;
  pdl_launch_dependents();
  pdl_wait();
  const uint4* src = static_cast<const uint4*>(args.sum[q]) + size_t(blockIdx.x) * nvec;
  uint4* dst = static_cast<uint4*>(args.out[q]) + size_t(blockIdx.x) * nvec;
  uint4 x[U], g[U];
  float2 ss = make_float2(0.f, 0.f);
  if (in_regs) {
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = tid + u * step < nvec ? src[tid + u * step] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (tid + u * step < nvec) g[u] = gamma[tid + u * step];
#pragma unroll
    for (int u = 0; u < U; ++u) row_norm_squares<T>(ss, x[u]);
  } else {
    for (int v = tid; v < nvec; v += step) row_norm_squares<T>(ss, src[v]);
  }
  float sum = ss.x + ss.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((tid & 31) == 0) s_part[tid >> 5] = sum;
  __syncthreads();
  // at most 16 warps: their sums by shuffles, not one shared-memory load after another
  float tot = (tid & 15) < (step >> 5) ? s_part[tid & 15] : 0.f;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  const float inv = rsqrtf(tot / float(N) + args.eps);
  if (in_regs) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (tid + u * step < nvec) dst[tid + u * step] = row_norm_scale<T>(x[u], g[u], inv);
  } else {
    for (int v = tid; v < nvec; v += step) dst[v] = row_norm_scale<T>(src[v], gamma[v], inv);
  }
}

}  // namespace b200ipc
