// One decode step of the Llama-shaped tensor-parallel decoder as ONE persistent kernel, for a process that drives every rank
// (a world of one, an emulated world): QKV projection, rotary embedding + cache append + attention, output projection,
// residual + RMSNorm, gate/up projection, SiLU * up, down projection, residual + RMSNorm, layer after layer, then the
// vocabulary head and the arg-max.
//
// A step is bound by what it reads once: the weights and the cache.  As a chain of kernels (eight per layer) every one of them
// pays its launch, its first loads and its drain while the memory idles: batch 32 at 2048 tokens, hidden 8192, FFN 3584, eight
// query heads on one KV head, 85 us per layer for 247 MB (38 us at the copy rate).  Here one CTA per SM stays for the whole step
// and one thread streams everything the CTA will need, in order, through one ring of 16 KB stages (128 x 64 tiles of W, 64
// positions of K or V): the stream does not wait for the math, so while the CTAs meet between two phases the ring fills with the
// weights of the next.
//
//   warp 0       stream: W tiles, K and V tiles (TMA, never waits for another CTA)
//   warp 1       X tiles: waits until the phase's input is complete, then loads it beside the W tiles
//   warp 2       tcgen05.mma: 128 rows of W (M) x the batch padded to 16, 32 or 64 (N)
//   warps 4-11   accumulators to memory, attention, norms, SiLU, arg-max
//
// Work split: a GEMM is tiles of 128 W rows x blocks of 64 columns, attention (rank, sequence, KV head) x 64 positions; both
// are cut into grid-size equal runs in that order, whatever the shape, so no SM idles.  A run's partial sums of a tile go to
// memory in fp32, in a slot of their own (tile + CTA number), and whoever needs the result adds a tile's slots in order: the
// result does not depend on timing.
//
// CTAs wait on one another: the launch is cooperative.  Every wait is bounded; a CTA whose wait runs out stops arriving, also at its
// own barriers (an arrival that stands for a wait that failed could complete a phase early), which ends the others' waits the same way.
//
// Measured, four layers and the head of that shape as one step: 423 us as a chain of kernels, 317 here (floor 194: 1.25 GB).
// Two thirds of a layer are bound by the stream (gate/up and down: 6 - 7 TB/s), the rest by the chain of meetings: about 1.5 us
// from the last CTA's store to everybody's next load, eight times a layer, attention 9 us, each norm 2.7 us.  What mattered: one
// body of code for all phases (with one per phase, 320 KB of instructions, every phase ran into cold instruction caches: 528
// us); streamed lines first to leave L2, where the partial sums and X live (348 -> 324 us); several CTAs per row of a norm.
// Bringing tiles to L2 ahead of the ring, by TMA or by plain prefetches of a warp of its own, 14 stages: gate/up 16.8 -> 12.7 us, but
// every meeting slower by as much (64 sequences x 4096: 3 - 5 % behind).
#pragma once

#include "../fused/gemm_ar.cuh"
#include "decode_math.cuh"

namespace b200ipc {

constexpr int kStepThreads = 384;
constexpr int kStepComputeWarps = 8;
constexpr int kStepCompute = kStepComputeWarps * 32;
constexpr int kStepMaxStages = 12;
constexpr int kStepMaxBatch = 64;
constexpr int kStepMapsPerRank = 6;  // per layer: wqkv, wo, wgu, wdown, K, V
constexpr int kStepMaps = 48;        // tensor maps of layers per launch
constexpr int kStepMaxLayers = kStepMaps / kStepMapsPerRank;
constexpr int kStepTileRows = 128;
constexpr int kStepTileBytes = kStepTileRows * kGemmBK * 2;
constexpr int kStepPos = 64;         // positions per K / V tile
constexpr int kStepSyncs = 8;        // meeting points per layer
constexpr int kStepSyncStride = 8;   // words between their counters
constexpr int kStepMaxParts = 8;     // CTAs that share a row of a norm or of the arg-max
constexpr int kStepMaxG = 8;
constexpr int kStepSmemBudget = 226 * 1024;
constexpr int kStepMaxHidden = 16384;
constexpr int kMergeRow = kAttnD + 4;  // rows of partial outputs (fp32) and of q, padded: a warp's accesses hit 32 banks
constexpr int kQRow = kAttnD + 8;

// What the compute warps keep behind the ring: the warps' partial attention outputs for G heads, or a row of a norm; maxima and
// sums, the table of the rotation, q, the new k and v.
B200_HD constexpr int step_shared_row(int G, int hidden) {
  return (kStepComputeWarps * G * kMergeRow * 4 > hidden * 2 ? kStepComputeWarps * G * kMergeRow * 4 : hidden * 2) + 127 & ~127;
}
B200_HD constexpr int step_scratch_bytes(int G, int hidden) {
  return step_shared_row(G, hidden) + (2 * kStepComputeWarps + 1) * kStepMaxG * 4 + kAttnD / 2 * 8 +
         kStepMaxG * kQRow * 2 + 2 * kAttnD * 2;
}

// The GEMMs of a layer and the head.  Each has two meeting points (counters 2 g and 2 g + 1 of the layer; the head counts as a
// layer of its own): the partial sums of all CTAs are there; what is made of them (attention, norm, SiLU * up, norm) is.
enum StepGemm { kGemmQkv, kGemmO, kGemmGateUp, kGemmDown, kGemmHead };

struct DecodeStepArgs {
  alignas(64) CUtensorMap maps[kStepMaps];  // [layer][rank][kStepMapsPerRank]
  alignas(64) CUtensorMap head[kMaxRanks];
  alignas(64) CUtensorMap x_norm;
  alignas(64) CUtensorMap x_attn[kMaxRanks];
  alignas(64) CUtensorMap x_act[kMaxRanks];
  void* kcache[kStepMaxLayers];  // [layer][rank]
  void* vcache[kStepMaxLayers];
  const void* gamma_mlp[kStepMaxLayers];
  const void* gamma_attn[kStepMaxLayers];  // the one behind the layer: the next layer's, or the final one
  void* hidden_out[kMaxRanks];             // with the head: the final norm's output, a copy per rank
  int64_t* ids;                            // with the head: [batch]
  void* h;        // [batch, hidden] residual stream
  void* xnorm;    // [batch, hidden]
  void* attn;     // [world][batch, hq * 128]
  void* act;      // [world][batch, ffn]
  float* part;    // partial sums: [tile + CTA][batch][128]
  float* apart;   // attention: [(rank, sequence, KV head) + CTA][G][4 + 128]
  uint32_t* squares;   // sums of squares of a row's parts, two norms by turns: [2][batch][kStepMaxParts]; 0 = not there yet
  uint32_t* sync;
  uint32_t* arrivals;  // [rank, sequence, KV head], then for the arg-max [sequence]: CTAs that are through
  StatusBlock* status;
  uint32_t* abort_word;
  uint64_t timeout_ns;
  int rank;
  int layers, first_layer;  // of this launch; number of the first one in the model
  int with_head;
  int world, batch, bn, stages;
  int hidden, hq, hkv, ffn, vocab;  // per rank
  int max_ctx, pos;
  int mute;  // CTA 0 arrives at no meeting point (failure injection)
  float eps, scale_log2, log2_theta;
};

__device__ __forceinline__ uint32_t ld_acquire_gpu_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(uint32_t* p, uint32_t v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t atom_acq_rel_gpu_add(uint32_t* p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ uint32_t ld_relaxed_gpu_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_relaxed_gpu_or(uint32_t* p, uint32_t v) {
  asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Generic stores before it are seen by asynchronous (TMA) reads after it, and the other way round.
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void tma_stream_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "l"(policy)
      : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void step_tmem_ld_8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// Barrier among the compute warps; `bad` of any of them is returned to all.
__device__ __forceinline__ bool compute_sync(bool bad = false) {
  uint32_t any;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.aligned.pred q, 1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"(uint32_t(bad)), "n"(kStepCompute)
      : "memory");
  return any != 0;
}
// A GEMM of the step, and the run of it that a CTA takes: units [u0, u1), unit = tile * kb + block of columns.
struct StepShape {
  const CUtensorMap *w, *x;  // of rank 0
  int w_step, x_step;        // maps from one rank to the next
  int tiles, per_rank;  // per_rank: tiles of one rank where the ranks' products follow one another, 0 where they are summed
  int kb, kb_seg;       // column blocks of a tile, of one rank's share of them
  int up_row;           // gate/up: first row of `up`; even tiles are gate rows, odd ones the up rows beside them
  int u0, u1;
};
__device__ __forceinline__ int ceil_div_dev(int a, int b) { return (a + b - 1) / b; }
// Runs are of equal length and none is empty: with fewer units than CTAs the last CTAs take none.  32 bits: the host keeps
// units * CTAs below 2^31.
__device__ __forceinline__ int runs_of(int units) { return min(units, int(gridDim.x)); }
__device__ __forceinline__ int run_start(int units, int cta) {
  const int runs = runs_of(units);
  return int(uint32_t(units) * uint32_t(min(cta, runs)) / uint32_t(runs));
}
// The CTA whose run holds a unit.
__device__ __forceinline__ int run_of(int unit, int units) {
  return int((uint32_t(unit + 1) * uint32_t(runs_of(units)) - 1u) / uint32_t(units));
}

__device__ __noinline__ StepShape step_shape(const DecodeStepArgs& a, int l, int which) {
  StepShape g;
  const CUtensorMap* m = a.maps + size_t(l) * a.world * kStepMapsPerRank;
  const int kb_hidden = ceil_div_dev(a.hidden, kGemmBK);
  g.up_row = 0;
  g.w_step = kStepMapsPerRank;
  g.x_step = 0;
  if (which == kGemmO || which == kGemmDown) {
    g.w = m + (which == kGemmO ? 1 : 3);
    g.x = which == kGemmO ? a.x_attn : a.x_act;
    g.x_step = 1;
    g.tiles = ceil_div_dev(a.hidden, kStepTileRows);
    g.per_rank = 0;
    g.kb_seg = which == kGemmO ? a.hq * (kAttnD / kGemmBK) : ceil_div_dev(a.ffn, kGemmBK);
    g.kb = g.kb_seg * a.world;
  } else {
    g.w = which == kGemmHead ? a.head : m + (which == kGemmQkv ? 0 : 2);
    g.x = &a.x_norm;
    g.per_rank = which == kGemmQkv ? a.hq + 2 * a.hkv : which == kGemmGateUp ? 2 * ceil_div_dev(a.ffn, kStepTileRows) : ceil_div_dev(a.vocab, kStepTileRows);
    if (which == kGemmGateUp) g.up_row = a.ffn;
    if (which == kGemmHead) g.w_step = 1;
    g.tiles = g.per_rank * a.world;
    g.kb = g.kb_seg = kb_hidden;
  }
  const int units = g.tiles * g.kb;
  g.u0 = run_start(units, int(blockIdx.x));
  g.u1 = run_start(units, int(blockIdx.x) + 1);
  return g;
}

// Walks the units of a run: which rank's box of W, which box of X they are.
struct StepWalk {
  const StepShape* g;
  int tile, seg, col_block, rank, row;
  __device__ __forceinline__ StepWalk(const StepShape& shape) : g(&shape) {
    tile = shape.u0 / shape.kb;
    const int k = shape.u0 - tile * shape.kb;
    seg = k / shape.kb_seg;
    col_block = k - seg * shape.kb_seg;
    place();
  }
  __device__ __forceinline__ void place() {
    if (g->per_rank) {
      rank = tile / g->per_rank;
      const int t = tile - rank * g->per_rank;
      row = g->up_row ? (t & 1) * g->up_row + (t >> 1) * kStepTileRows : t * kStepTileRows;
    } else {
      rank = seg;
      row = tile * kStepTileRows;
    }
  }
  __device__ __forceinline__ void next() {
    if (++col_block < g->kb_seg) return;
    col_block = 0;
    if (++seg * g->kb_seg == g->kb) {
      seg = 0;
      ++tile;
    }
    place();
  }
  __device__ __forceinline__ int col() const { return col_block * kGemmBK; }
};

// The attention's work: sequences (rank, sequence, KV head) of `per_seq` tiles of positions.  A run that holds parts of two
// sequences pays q, the merge of the warps and the hand-over twice (about as long as eight tiles take), so where it costs no
// more than that, a CTA takes parts of one sequence only (`parts` CTAs share it), or whole ones; else the tiles are cut into
// equal runs.  Batch 32, 2048 positions, one KV head on 148 SMs: 8 tiles a CTA 11 us, runs of 6.9 tiles 17.
struct StepAttn {
  int sequences, per_seq, parts, u0, u1;
  bool whole;
  __device__ __forceinline__ StepAttn(const DecodeStepArgs& a) {
    const int ctas = int(gridDim.x);
    sequences = a.world * a.batch * a.hkv;
    per_seq = ceil_div_dev(a.pos, kStepPos);
    const int most = sequences * per_seq / ctas + 8;
    parts = sequences <= ctas ? min(ctas / sequences, per_seq) : 0;
    if (parts && ceil_div_dev(per_seq, parts) > most) parts = 0;
    whole = parts == 0 && ceil_div_dev(sequences, ctas) * per_seq <= most;
    u0 = start(int(blockIdx.x));
    u1 = start(int(blockIdx.x) + 1);
  }
  __device__ __forceinline__ int start(int cta) const {
    if (parts) {
      const int seq = min(cta / parts, sequences), part = seq < sequences ? cta - seq * parts : 0;
      return seq * per_seq + per_seq * part / parts;
    }
    return whole ? run_start(sequences, cta) * per_seq : run_start(sequences * per_seq, cta);
  }
  __device__ __forceinline__ int first_cta(int seq) const {
    return parts ? seq * parts : whole ? run_of(seq, sequences) : run_of(seq * per_seq, sequences * per_seq);
  }
  __device__ __forceinline__ int last_cta(int seq) const {
    return parts ? seq * parts + parts - 1 : whole ? run_of(seq, sequences) : run_of(seq * per_seq + per_seq - 1, sequences * per_seq);
  }
};

// Everything a CTA streams, in order: box(layer, shape, walk, which) for a tile of W, pair(layer, rank, sequence of the rank,
// first position) for a K tile and the V tile of the same positions; either returns false to stop.
template <typename Box, typename Pair>
__device__ __forceinline__ void step_stream(const DecodeStepArgs& a, const StepAttn& at, Box box, Pair pair) {
#pragma unroll 1
  for (int phase = 0; phase < 4 * a.layers + (a.with_head ? 1 : 0); ++phase) {
    const int l = phase >> 2, which = l < a.layers ? phase & 3 : int(kGemmHead);
    const StepShape g = step_shape(a, l, which);
    StepWalk w(g);
#pragma unroll 1
    for (int u = g.u0; u < g.u1; ++u, w.next())
      if (!box(l, g, w, which)) return;
    if (which != kGemmQkv) continue;
#pragma unroll 1
    for (int u = at.u0; u < at.u1; ++u) {
      const int seq = u / at.per_seq, per_rank = a.batch * a.hkv, rank = seq / per_rank;
      if (!pair(l, rank, seq - rank * per_rank, (u - seq * at.per_seq) * kStepPos)) return;
    }
  }
}

__device__ __forceinline__ Best warp_best(Best best) {
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1)
    best = better(best, Best{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
  return best;
}

template <typename T>
__global__ void __launch_bounds__(kStepThreads, 1) decode_step_kernel(const __grid_constant__ DecodeStepArgs args) {
  using T2 = typename Num<T>::T2;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t full_w[kStepMaxStages], full_x[kStepMaxStages], empty[kStepMaxStages], acc_full[2], acc_empty[2], attn_done, mma_done;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort, s_flag;
  __shared__ float s_red[kStepComputeWarps], s_inv;
  __shared__ Best s_best[kStepComputeWarps];
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = int(threadIdx.x & 31);
  const int cta = int(blockIdx.x), ctas = int(gridDim.x);
  const int B = args.batch, bn = args.bn, W = args.world;
  const uint32_t stages = uint32_t(args.stages);
  const uint32_t x_bytes = uint32_t(bn) * kGemmBK * 2, stage_bytes = kStepTileBytes + x_bytes;
  const uint32_t ring_addr = smem_u32(ring);
  const uint64_t timeout_ns = args.timeout_ns;
  volatile int* abort_flag = &s_abort;
  const StepAttn at(args);
  const int a0 = at.u0, a1 = at.u1;
  const int parts = min(max(ctas / B, 1), kStepMaxParts);  // CTAs that share a row of a norm or of the arg-max
  auto counter = [&](int l, int s) { return args.sync + (size_t(args.first_layer + l) * kStepSyncs + size_t(s)) * kStepSyncStride; };
  // Bounded: false where `there` did not become true in time or this CTA has given up.
  auto wait_for = [&](auto there) {
    uint64_t t0 = 0;
    for (uint32_t n = 0;; ++n) {
      if (there()) return true;
      if ((n & 63u) == 63u) {
        if (*abort_flag) return false;
        const uint64_t now = globaltimer_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > timeout_ns) break;
      }
    }
    *abort_flag = 1;
    return false;
  };
  auto wait_count = [&](const uint32_t* p, uint32_t target) { return wait_for([&]() { return ld_acquire_gpu_u32(p) >= target; }); };

  if (threadIdx.x == 0) {
#pragma unroll 1
    for (uint32_t i = 0; i < stages; ++i) {
      mbar_init(&full_w[i], 1);
      mbar_init(&full_x[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], kStepComputeWarps);
    }
    mbar_init(&attn_done, 1);
    mbar_init(&mma_done, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    tmem_alloc(&s_tmem, 2 * kStepMaxBatch);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = s_tmem;

  if (warp == 0) {
    // ---- the stream -------------------------------------------------------------------------------------------------------
    if (elect_one()) {
      uint32_t st = 0, ph = 1;
      int it = 0;
      const uint64_t policy = evict_first_policy();
      auto ready = [&]() {
        if (!mbar_wait_long(&empty[st], ph, abort_flag, timeout_ns)) return false;
        mbar_expect_tx(&full_w[st], kStepTileBytes);
        return true;
      };
      auto advance = [&]() {
        if (++st == stages) {
          st = 0;
          ph ^= 1u;
        }
        ++it;
      };
      step_stream(
          args, at,
          [&](int, const StepShape& g, const StepWalk& w, int) {
            if (!ready()) return false;
            tma_stream_2d(ring + st * stage_bytes, g.w + w.rank * g.w_step, &full_w[st], w.col(), w.row, policy);
            advance();
            return true;
          },
          [&](int l, int rank, int seq, int first) {
            const CUtensorMap* m = args.maps + (size_t(l) * W + rank) * kStepMapsPerRank + 4;
#pragma unroll 1
            for (int kv = 0; kv < 2; ++kv) {
              if (!ready()) return false;
              tma_stream_3d(ring + st * stage_bytes, m + kv, &full_w[st], 0, first, seq, policy);
              tma_stream_3d(ring + st * stage_bytes + kStepPos * 128, m + kv, &full_w[st], kGemmBK, first, seq, policy);
              advance();
            }
            return true;
          });
      // copies in flight land before the CTA leaves
      const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
      for (int back = 1; back <= min(it, int(stages)); ++back)
        mbar_drain(&full_w[uint32_t(it - back) % stages], (uint32_t(it - back) / stages) & 1u, t0);
    }
  } else if (warp == 1) {
    // ---- X tiles ----------------------------------------------------------------------------------------------------------
    if (elect_one()) {
      uint32_t st = 0, ph = 1;
      int it = 0;
      bool ok = true;
      auto advance = [&]() {
        if (++st == stages) {
          st = 0;
          ph ^= 1u;
        }
        ++it;
      };
#pragma unroll 1
      for (int phase = 0; ok && phase < 4 * args.layers + (args.with_head ? 1 : 0); ++phase) {
        const int l = phase >> 2, which = l < args.layers ? phase & 3 : int(kGemmHead);
        const StepShape g = step_shape(args, l, which);
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(g.x)) : "memory");
        // what the GEMM before this one was made into
        if (which == kGemmO) ok = wait_count(counter(l, 2 * kGemmQkv + 1), uint32_t(ctas));
        else if (which == kGemmGateUp) ok = wait_count(counter(l, 2 * kGemmO + 1), uint32_t(B * parts));
        else if (which == kGemmDown) ok = wait_count(counter(l, 2 * kGemmGateUp + 1), uint32_t(ctas));
        else if (l > 0) ok = wait_count(counter(l - 1, 2 * kGemmDown + 1), uint32_t(B * parts));
        fence_proxy_async_global();  // the generic stores that were waited for, before TMA reads
        StepWalk w(g);
#pragma unroll 1
        for (int u = g.u0; ok && u < g.u1; ++u, w.next()) {
          ok = mbar_wait_long(&empty[st], ph, abort_flag, timeout_ns);
          if (!ok) break;
          mbar_expect_tx(&full_x[st], x_bytes);
          tma_load_2d(ring + st * stage_bytes + kStepTileBytes, g.x + w.rank * g.x_step, &full_x[st], w.col(), 0);
          advance();
        }
        if (which != kGemmQkv) continue;
#pragma unroll 1
        for (int u = 2 * a0; ok && u < 2 * a1; ++u) {  // K and V tiles have no X beside them
          ok = mbar_wait_long(&empty[st], ph, abort_flag, timeout_ns);
          if (!ok) break;
          mbar_arrive(&full_x[st]);
          advance();
        }
      }
      const uint64_t t0 = globaltimer_ns();
#pragma unroll 1
      for (int back = 1; back <= min(it, int(stages)); ++back)
        mbar_drain(&full_x[uint32_t(it - back) % stages], (uint32_t(it - back) / stages) & 1u, t0);
    }
  } else if (warp == 2) {
    // ---- tcgen05.mma ------------------------------------------------------------------------------------------------------
    if (elect_one()) {
      const uint32_t idesc = make_idesc<T>(kStepTileRows, bn);
      uint32_t st = 0, ph = 0, seg = 0;
      bool ok = true;
#pragma unroll 1
      for (int phase = 0; ok && phase < 4 * args.layers + (args.with_head ? 1 : 0); ++phase) {
        const int l = phase >> 2, which = l < args.layers ? phase & 3 : int(kGemmHead);
        const StepShape g = step_shape(args, l, which);
        for (int u = g.u0; ok && u < g.u1; ++seg) {
          const int end = min(g.u1, (u / g.kb + 1) * g.kb);
          const uint32_t buf = seg & 1u;
          ok = mbar_wait_long(&acc_empty[buf], ((seg >> 1) & 1u) ^ 1u, abort_flag, timeout_ns);
          if (!ok) break;
          tc_fence_after_sync();
          uint32_t accumulate = 0;
#pragma unroll 1
          for (; u < end; ++u) {
            ok = mbar_wait_long(&full_w[st], ph, abort_flag, timeout_ns) && mbar_wait_long(&full_x[st], ph, abort_flag, timeout_ns);
            if (!ok) break;
            tc_fence_after_sync();
            const uint64_t da = make_sw128_kmajor_desc(ring_addr + st * stage_bytes);
            const uint64_t db = make_sw128_kmajor_desc(ring_addr + st * stage_bytes + kStepTileBytes);
#pragma unroll
            for (int k = 0; k < kGemmBK / 16; ++k) {
              umma_f16(tmem_base + buf * kStepMaxBatch, da + uint64_t(2 * k), db + uint64_t(2 * k), idesc, accumulate);
              accumulate = 1;
            }
            umma_commit(&empty[st]);
            if (++st == stages) {
              st = 0;
              ph ^= 1u;
            }
          }
          if (ok) umma_commit(&acc_full[buf]);
        }
        if (which == kGemmQkv) {
          // The attention's stages go by.  A wait for the parity of a later round would pass before they have: not until
          // the compute warps are through with them.
          ok = ok && mbar_wait_long(&attn_done, uint32_t(l) & 1u, abort_flag, timeout_ns);
          const uint32_t n = st + 2u * uint32_t(a1 - a0);
          ph ^= (n / stages) & 1u;
          st = n % stages;
        }
      }
      umma_commit(&mma_done);
      mbar_drain(&mma_done, 0, globaltimer_ns());
    }
  } else if (warp >= 4) {
    // ---- compute ----------------------------------------------------------------------------------------------------------
    const int tid = int(threadIdx.x) - 128, cw = warp - 4;
    const int G = args.hq / args.hkv;
    // Scratch behind the ring.  The attention's part and a row of a norm take turns on the first bytes.
    float* s_o = reinterpret_cast<float*>(ring + stages * stage_bytes);                                     // [warp][G][kMergeRow]
    uint2* s_row = reinterpret_cast<uint2*>(s_o);                                                           // [hidden]
    float* s_ml = s_o + step_shared_row(G, args.hidden) / 4;                                                // [2][warp][kStepMaxG]
    float* s_new = s_ml + 2 * kStepComputeWarps * kStepMaxG;                                                // [kStepMaxG]
    float2* s_rot = reinterpret_cast<float2*>(s_new + kStepMaxG);                                           // [64] (sin, cos)
    T* s_q = reinterpret_cast<T*>(s_rot + kAttnD / 2);                                                      // [G][kQRow]
    T* s_k = s_q + kStepMaxG * kQRow;                                                                       // the new k and v of the sequence in work
    T* s_v = s_k + kAttnD;
    if (tid < kAttnD / 2) {
      // angle = pos * theta^(-i / half)
      float sn, cs;
      sincosf(float(args.pos) * exp2f(-args.log2_theta * float(tid) / float(kAttnD / 2)), &sn, &cs);
      s_rot[tid] = make_float2(sn, cs);
    }
    bool bad = false;
    uint32_t seg_no = 0;
    uint32_t st = 0, ph = 0;  // the stage and the round of the ring that the compute warps are at
    auto skip = [&](uint32_t n) {
      n += st;
      ph ^= (n / stages) & 1u;
      st = n % stages;
    };

    // Everything the compute warps have stored so far is complete: adds one to a meeting point's counter.
    auto arrive = [&](uint32_t* p) {
      bad = compute_sync(bad);
      if (tid == 0 && !bad && !(args.mute && cta == 0)) red_release_gpu_add(p, 1u);
    };
    auto wait = [&](const uint32_t* p, uint32_t target) {
      if (tid == 0 && !bad) bad = !wait_count(p, target);
      bad = compute_sync(bad);
    };
    auto pack4 = [&](float4 v) {
      return make_uint2(pack2<T>(v.x, v.y), pack2<T>(v.z, v.w));
    };
    auto unpack4 = [&](uint2 v) {
      const float2 a = Num<T>::up(*reinterpret_cast<const T2*>(&v.x)), b = Num<T>::up(*reinterpret_cast<const T2*>(&v.y));
      return make_float4(a.x, a.y, b.x, b.y);
    };
    auto add4 = [](float4& a, const float4& x) { a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w; };
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t slot_floats = size_t(B) * kStepTileRows;
    // The slots that hold a tile's partial sums.
    auto slots_of = [&](const StepShape& g, int units, int t) {
      const int first = run_of(t * g.kb, units);
      return make_int2(t + first, run_of(t * g.kb + g.kb - 1, units) - first + 1);
    };
    // Their sums in order for two tiles: row b, four columns from off0 and off1 on; all loads of up to eight slots in flight.
    auto tile_sums = [&](const int2 (&sl)[2], float4 (&v)[2], int b, int off0, int off1) {
      const float* p0 = args.part + size_t(sl[0].x) * slot_floats + size_t(b) * kStepTileRows + off0;
      const float* p1 = args.part + size_t(sl[1].x) * slot_floats + size_t(b) * kStepTileRows + off1;
      v[0] = v[1] = zero4;
#pragma unroll 1
      for (int s = 0; s < max(sl[0].y, sl[1].y); s += 8, p0 += 8 * slot_floats, p1 += 8 * slot_floats) {
        float4 x[2][8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x[0][j] = s + j < sl[0].y ? __ldcg(reinterpret_cast<const float4*>(p0 + size_t(j) * slot_floats)) : zero4;
          x[1][j] = s + j < sl[1].y ? __ldcg(reinterpret_cast<const float4*>(p1 + size_t(j) * slot_floats)) : zero4;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          add4(v[0], x[0][j]);
          add4(v[1], x[1][j]);
        }
      }
    };

    // One body for every GEMM of the step: the kernel has to stay small enough for the instruction caches.
#pragma unroll 1
    for (int phase = 0; phase < 4 * args.layers + (args.with_head ? 1 : 0) && !bad; ++phase) {
      const int l = phase >> 2, which = l < args.layers ? phase & 3 : int(kGemmHead);
      const StepShape g = step_shape(args, l, which);
      const int units = g.tiles * g.kb;
      uint32_t* sums = counter(l, 2 * (which & 3));
      uint32_t* done = sums + kStepSyncStride;

      // ---- the run's accumulators to their slots ------------------------------------------------------------------------
      const int half = bn / 2, c0 = (cw >> 2) * half;
#pragma unroll 1
      for (int u = g.u0; u < g.u1; ++seg_no) {
        const int t = u / g.kb;
        u = min(g.u1, (t + 1) * g.kb);
        const uint32_t buf = seg_no & 1u;
        bad = __any_sync(0xffffffffu, !mbar_wait_long(&acc_full[buf], (seg_no >> 1) & 1u, abort_flag, timeout_ns));
        if (bad) break;
        tc_fence_after_sync();
        float* slot = args.part + size_t(t + cta) * slot_floats + (warp & 3) * 32 + lane;
#pragma unroll 1
        for (int c = c0; c < c0 + half && c < B; c += 8) {
          uint32_t v[8];
          step_tmem_ld_8(tmem_base + buf * kStepMaxBatch + (uint32_t((warp & 3) * 32) << 16) + uint32_t(c), v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (c + j < B) slot[size_t(c + j) * kStepTileRows] = __uint_as_float(v[j]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      skip(uint32_t(g.u1 - g.u0));
      arrive(sums);

      if (which == kGemmQkv) {
        // ---- attention over the cache, positions [0, pos), and the new position -------------------------------------------
        wait(sums, uint32_t(ctas));
#pragma unroll 1
        for (int u = a0; u < a1 && !bad;) {
          const int seq = u / at.per_seq, rank = seq / (B * args.hkv), local = seq - rank * (B * args.hkv), b = local / args.hkv, kvh = local - b * args.hkv;
          const int end = min(a1, (seq + 1) * at.per_seq);
          const bool owns_new = end == (seq + 1) * at.per_seq;
          // q of the G heads, rounded, turned and rounded; where this run ends with the sequence, the new k and v too.  A warp
          // per head, four dimensions per lane; the other element of a pair is 16 lanes away.
#pragma unroll 1
          for (int head = cw; head < G + (owns_new ? 2 : 0); head += kStepComputeWarps) {
            const int t = rank * g.per_rank + (head < G ? kvh * G + head : head == G ? args.hq + kvh : args.hq + args.hkv + kvh);
            const int2 slots = slots_of(g, units, t);
            const float* p = args.part + size_t(slots.x) * slot_floats + size_t(b) * kStepTileRows + lane * 4;
            float4 v = zero4;
#pragma unroll 1
            for (int s = 0; s < slots.y; s += 16, p += 16 * slot_floats) {
              float4 x[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) x[j] = s + j < slots.y ? __ldcg(reinterpret_cast<const float4*>(p + size_t(j) * slot_floats)) : zero4;
#pragma unroll
              for (int j = 0; j < 16; ++j) add4(v, x[j]);
            }
            uint2 y = pack4(v);
            if (head <= G) {
              v = unpack4(y);
              const float mine[4] = {v.x, v.y, v.z, v.w};
              float turned[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float other = __shfl_xor_sync(0xffffffffu, mine[e], 16);
                const float2 r = s_rot[(lane & 15) * 4 + e];
                const float2 pair = lane < 16 ? rope_pair(mine[e], other, r.x, r.y) : rope_pair(other, mine[e], r.x, r.y);
                turned[e] = lane < 16 ? pair.x : pair.y;
              }
              y = pack4(make_float4(turned[0], turned[1], turned[2], turned[3]));
            }
            *reinterpret_cast<uint2*>((head < G ? s_q + head * kQRow : head == G ? s_k : s_v) + lane * 4) = y;
            if (head >= G)
              *reinterpret_cast<uint2*>(static_cast<T*>((head == G ? args.kcache : args.vcache)[l * W + rank]) +
                                        (size_t(local) * args.max_ctx + args.pos) * kAttnD + lane * 4) = y;
          }
          bad = compute_sync(bad);
          // Tiles go in pairs: four warps take one of them, 16 positions each, and four the other.
          const int r = lane >> 2, c = lane & 3, group = cw >> 2;
          float m = -INFINITY, lsum = 0.f;  // running state of head r
          float acc[8][4];                  // O^T: dims 16 t + r, + 8 of heads 2c, 2c + 1
#pragma unroll
          for (int t = 0; t < 8; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
          uint32_t qa[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) qa[i] = r < G ? reinterpret_cast<const uint32_t*>(s_q + r * kQRow)[4 * i + c] : 0u;
          // this lane's row of the 16 x 16 blocks that ldmatrix reads: position, and which 16-byte chunk of the pair
          const int lrow = (cw & 3) * 16 + ((lane >> 4) & 1) * 8 + (lane & 7), lchunk = (lane >> 3) & 1;
          // A pair's stages: K and V of its first tile, of its second.
          auto stage = [&](uint32_t n, uint32_t* parity) {
            n += st;
            *parity = n >= stages ? ph ^ 1u : ph;
            return n >= stages ? n - stages : n;
          };
          for (int pair = u; pair < end; pair += 2) {
            const int v = pair + group;
            if (v < end) {
              uint32_t pk, pv;
              const uint32_t sk = stage(2u * uint32_t(group), &pk), sv = stage(2u * uint32_t(group) + 1u, &pv);
              if (!mbar_wait_long(&full_w[sk], pk, abort_flag, timeout_ns)) bad = true;
              if (!mbar_wait_long(&full_w[sv], pv, abort_flag, timeout_ns)) bad = true;
              // (the arrival that stands for the missing X tile, so that this round of the barrier is over as well)
              if (!mbar_wait_long(&full_x[sk], pk, abort_flag, timeout_ns)) bad = true;
              if (!mbar_wait_long(&full_x[sv], pv, abort_flag, timeout_ns)) bad = true;
              __syncwarp();
              const uint32_t kt = ring_addr + sk * stage_bytes, vt = ring_addr + sv * stage_bytes;
              auto chunk_addr = [&](uint32_t tile, int chunk) {  // 16-byte chunk 0..15 of this lane's position, 128-byte swizzle
                return tile + uint32_t(chunk >> 3) * (kStepPos * 128) + uint32_t(lrow) * 128u + uint32_t(((chunk & 7) ^ (lrow & 7)) << 4);
              };
              float s[2][4];
#pragma unroll
              for (int j = 0; j < 2; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                uint32_t kf[4];
                ldmatrix_x4(kf, chunk_addr(kt, 2 * k + lchunk));
                mma_16816<T>(s[0], qa[2 * k], 0u, qa[2 * k + 1], 0u, kf[0], kf[1]);
                mma_16816<T>(s[1], qa[2 * k], 0u, qa[2 * k + 1], 0u, kf[2], kf[3]);
              }
              const int base = (v - seq * at.per_seq) * kStepPos + (cw & 3) * 16;
              float sc[4];
#pragma unroll
              for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) sc[2 * j + e] = (base + 8 * j + 2 * c + e < args.pos) ? s[j][e] * args.scale_log2 : -INFINITY;
              float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
              const float mnew = fmaxf(m, mx);
              const float mref = mnew == -INFINITY ? 0.f : mnew;  // no position of this warp exists yet
              const float corr = exp2f(m - mref);
              m = mnew;
              float pr[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) pr[e] = exp2f(sc[e] - mref);
              lsum = lsum * corr + (pr[0] + pr[1]) + (pr[2] + pr[3]);
              const uint32_t pb0 = pack2<T>(pr[0], pr[1]), pb1 = pack2<T>(pr[2], pr[3]);
              const float corr0 = __shfl_sync(0xffffffffu, corr, 8 * c), corr1 = __shfl_sync(0xffffffffu, corr, 8 * c + 4);
#pragma unroll
              for (int t = 0; t < 8; ++t) {
                uint32_t vf[4];
                ldmatrix_x4_trans(vf, chunk_addr(vt, 2 * t + lchunk));
                acc[t][0] *= corr0; acc[t][1] *= corr1; acc[t][2] *= corr0; acc[t][3] *= corr1;
                mma_16816<T>(acc[t], vf[0], vf[1], vf[2], vf[3], pb0, pb1);
              }
            }
            bad = compute_sync(bad);  // nobody is more than a pair ahead, so a stage's parity is never taken for the round before
            if (bad) break;
            const uint32_t used = 2u * uint32_t(min(2, end - pair));
            uint32_t unused;
            if (uint32_t(tid) < used) mbar_arrive(&empty[stage(uint32_t(tid), &unused)]);
            st += used;
            if (st >= stages) {
              st -= stages;
              ph ^= 1u;
            }
          }
          if (bad) break;
          lsum += __shfl_xor_sync(0xffffffffu, lsum, 1);
          lsum += __shfl_xor_sync(0xffffffffu, lsum, 2);
          if (c == 0) {
            s_ml[cw * kStepMaxG + r] = m;
            s_ml[(kStepComputeWarps + cw) * kStepMaxG + r] = lsum;
          }
          {
            float* so = s_o + cw * G * kMergeRow;
#pragma unroll
            for (int t = 0; t < 8; ++t) {
              if (2 * c < G) {
                so[(2 * c) * kMergeRow + 16 * t + r] = acc[t][0];
                so[(2 * c) * kMergeRow + 16 * t + 8 + r] = acc[t][2];
              }
              if (2 * c + 1 < G) {
                so[(2 * c + 1) * kMergeRow + 16 * t + r] = acc[t][1];
                so[(2 * c + 1) * kMergeRow + 16 * t + 8 + r] = acc[t][3];
              }
            }
          }
          if (owns_new && cw < G) {  // the new position's score for head cw
            const float4 x = unpack4(*reinterpret_cast<const uint2*>(s_q + cw * kQRow + lane * 4));
            const float4 y = unpack4(*reinterpret_cast<const uint2*>(s_k + lane * 4));
            float d = x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if (lane == 0) s_new[cw] = d * args.scale_log2;
          }
          bad = compute_sync(bad);
          // merge: thread (head g, four dims)
          const int first = at.first_cta(seq), last = at.last_cta(seq);
          T* out = static_cast<T*>(args.attn) + (size_t(rank) * B + b) * (size_t(args.hq) * kAttnD) + size_t(kvh) * G * kAttnD;
          const size_t part_stride = size_t(G) * kMergeRow;
          const int hd = tid >> 5, ln = tid & 31;
          if (hd < G) {
            float mm = owns_new ? s_new[hd] : -INFINITY;
#pragma unroll
            for (int w = 0; w < kStepComputeWarps; ++w) mm = fmaxf(mm, s_ml[w * kStepMaxG + hd]);
            float ll = 0.f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            if (owns_new) {
              const float p = exp2f(s_new[hd] - mm);
              const float4 y = unpack4(*reinterpret_cast<const uint2*>(s_v + ln * 4));
              ll = p;
              o = make_float4(p * y.x, p * y.y, p * y.z, p * y.w);
            }
#pragma unroll
            for (int w = 0; w < kStepComputeWarps; ++w) {
              const float wm = s_ml[w * kStepMaxG + hd];
              const float p = wm == -INFINITY ? 0.f : exp2f(wm - mm);
              const float4 x = *reinterpret_cast<const float4*>(s_o + (w * G + hd) * kMergeRow + ln * 4);
              ll += s_ml[(kStepComputeWarps + w) * kStepMaxG + hd] * p;
              o.x += x.x * p; o.y += x.y * p; o.z += x.z * p; o.w += x.w * p;
            }
            if (first == last) {
              const float inv = 1.f / ll;
              *reinterpret_cast<uint2*>(out + hd * kAttnD + ln * 4) = pack4(make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
            } else {
              float* dst = args.apart + size_t(seq + cta) * part_stride + size_t(hd) * kMergeRow;
              if (ln == 0) *reinterpret_cast<float2*>(dst) = make_float2(mm, ll);
              *reinterpret_cast<float4*>(dst + 4 + ln * 4) = o;
            }
          }
          bool finish = true;
          if (first != last) {  // the last CTA of the sequence to arrive adds them up
            bad = compute_sync(bad);
            if (tid == 0) s_flag = atom_acq_rel_gpu_add(args.arrivals + seq, 1u) == uint32_t(last - first);
            bad = compute_sync(bad);
            finish = s_flag != 0;
            if (finish && hd < G) {
              const float* src = args.apart + size_t(seq + first) * part_stride + size_t(hd) * kMergeRow;
              float mm = -INFINITY, ll = 0.f;
              float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
              for (int s = first; s <= last; s += 8, src += 8 * part_stride) {  // eight at a time in flight
                float2 ml[8];
                float4 x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const float* from = src + (s + j <= last ? size_t(j) * part_stride : 0);
                  ml[j] = __ldcg(reinterpret_cast<const float2*>(from));
                  x[j] = __ldcg(reinterpret_cast<const float4*>(from + 4 + ln * 4));
                  if (s + j > last) ml[j].x = -INFINITY;
                }
                float mn = mm;
#pragma unroll
                for (int j = 0; j < 8; ++j) mn = fmaxf(mn, ml[j].x);  // finite: a run has at least one position
                const float p0 = exp2f(mm - mn);
                ll *= p0;
                o.x *= p0; o.y *= p0; o.z *= p0; o.w *= p0;
                mm = mn;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const float p = exp2f(ml[j].x - mm);
                  ll += ml[j].y * p;
                  o.x += x[j].x * p; o.y += x[j].y * p; o.z += x[j].z * p; o.w += x[j].w * p;
                }
              }
              const float inv = 1.f / ll;
              *reinterpret_cast<uint2*>(out + hd * kAttnD + ln * 4) = pack4(make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
            }
            if (finish && tid == 0) args.arrivals[seq] = 0;
          }
          bad = compute_sync(bad);  // the scratch is written again
          u = end;
        }
        if (tid == 0 && !bad) mbar_arrive(&attn_done);
        arrive(done);
      } else if (which == kGemmGateUp) {
        // ---- SiLU(gate) * up -----------------------------------------------------------------------------------------------
        wait(sums, uint32_t(ctas));
        const int row = args.ffn / 4;
#pragma unroll 1
        for (int i = cta * kStepCompute + tid; i < W * B * row; i += ctas * kStepCompute) {
          const int rb = i / row, f = (i - rb * row) * 4, rank = rb / B, b = rb - rank * B;
          const int t = rank * g.per_rank + 2 * (f >> 7);
          const int2 sl[2] = {slots_of(g, units, t), slots_of(g, units, t + 1)};
          float4 xy[2];
          tile_sums(sl, xy, b, f & 127, f & 127);
          const float4 x = xy[0], y = xy[1];
          const float4 o = make_float4(x.x / (1.f + __expf(-x.x)) * y.x, x.y / (1.f + __expf(-x.y)) * y.y, x.z / (1.f + __expf(-x.z)) * y.z,
                                       x.w / (1.f + __expf(-x.w)) * y.w);
          *reinterpret_cast<uint2*>(static_cast<T*>(args.act) + size_t(rb) * args.ffn + f) = pack4(o);
        }
        arrive(done);
      } else {
        // ---- h += product; normed h (with the head: the arg-max of the product).  `parts` CTAs share a row. ----------------
        const bool head = which == kGemmHead;
        const void* gamma = which == kGemmO ? args.gamma_mlp[l] : args.gamma_attn[head ? 0 : l];
        const bool last = args.with_head && phase == 4 * args.layers - 1;
        if (cta >= B * parts) continue;
        const int part0 = cta % parts;
        const int all = g.tiles * 32;  // chunks of four columns
        const int i0 = all / 32 * part0 / parts * 32, i1 = all / 32 * (part0 + 1) / parts * 32;
        if (!head)
          for (int i = i0 + tid * 16; i < i1; i += kStepCompute * 16)
            if (i * 4 < args.hidden) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const T*>(gamma) + i * 4));
        wait(sums, uint32_t(ctas));
#pragma unroll 1
        for (int item = cta; item < B * parts; item += ctas / parts * parts) {  // the same part of further rows
          const int b = item / parts;
          uint2* h = reinterpret_cast<uint2*>(static_cast<T*>(args.h) + size_t(b) * args.hidden);
          float ss = 0.f;
          Best best{-INFINITY, 0x7fffffff};
#pragma unroll 1
          for (int c = i0 + tid; c < i1; c += 2 * kStepCompute) {
            const int c2 = c + kStepCompute;
            const int2 sl[2] = {slots_of(g, units, c >> 5), c2 < i1 ? slots_of(g, units, c2 >> 5) : make_int2(0, 0)};
            uint2 r[2] = {make_uint2(0, 0), make_uint2(0, 0)};
            if (!head && c * 4 < args.hidden) r[0] = h[c];
            if (!head && c2 < i1 && c2 * 4 < args.hidden) r[1] = h[c2];
            float4 sums2[2];
            tile_sums(sl, sums2, b, (c & 31) * 4, (c2 & 31) * 4);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int i = c + q * kStepCompute;
              float4 v = sums2[q];
              add4(v, unpack4(r[q]));
              const uint2 y = pack4(v);
              v = unpack4(y);
              if (i >= i1) continue;
              if (head) {
                const int rank = (i >> 5) / g.per_rank, n = i * 4 - rank * g.per_rank * kStepTileRows;
                const float e4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                  if (n + e < args.vocab) best = better(best, Best{e4[e], rank * args.vocab + n + e});
              } else if (i * 4 < args.hidden) {
                h[i] = y;
                s_row[i - i0] = y;
                ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
              }
            }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          if (head) best = warp_best(best);
          if (lane == 0) {
            s_red[cw] = ss;
            s_best[cw] = best;
          }
          bad = compute_sync(bad);
          if (head) {  // the last CTA of the row compares what they found
            if (cw == 0 && !bad) {
              best = warp_best(s_best[lane % kStepComputeWarps]);
              float2* found = reinterpret_cast<float2*>(args.apart) + size_t(b) * kStepMaxParts;
              int is_last = 0;
              if (lane == 0) {
                found[part0] = make_float2(best.v, __int_as_float(best.i));
                is_last = atom_acq_rel_gpu_add(args.arrivals + at.sequences + b, 1u) == uint32_t(parts - 1);
              }
              is_last = __shfl_sync(0xffffffffu, is_last, 0);
              __syncwarp();  // a shuffle orders no memory: lane 0's acquire comes before the other lanes' loads through this
              if (is_last) {
                const float2 f = __ldcg(found + lane % parts);
                best = warp_best(Best{f.x, __float_as_int(f.y)});
                if (lane == 0) args.ids[b] = best.i;
              }
            }
            bad = compute_sync(bad);
            continue;
          }
          // The parts' sums of squares.  A word is its own signal (sign bit set, never zero): nothing else is handed over, so there
          // is nothing to release, and no second load behind the wait: 1.0 us, not 1.8 (with a counter and a release).  As a
          // reduction: plain stores came up to 2 us later while the ring fills.  The other norm's words were read by all before
          // anybody got here: cleared for the next one.
          if (cw == 0) {
            const int turn = phase >> 1 & 1;
            uint32_t* sq = args.squares + (size_t(turn) * B + b) * kStepMaxParts;
            if (lane == 0 && !bad) {
              float mine = 0.f;
#pragma unroll
              for (int w = 0; w < kStepComputeWarps; ++w) mine += s_red[w];
              red_relaxed_gpu_or(sq + part0, __float_as_uint(mine) | 0x80000000u);
              args.squares[(size_t(turn ^ 1) * B + b) * kStepMaxParts + part0] = 0u;
            }
            uint32_t word = 0;
            if (lane < parts && !bad) bad = !wait_for([&]() { return (word = ld_relaxed_gpu_u32(sq + lane)) != 0u; });
            __syncwarp();
            float tot = __uint_as_float(word & 0x7fffffffu);
#pragma unroll
            for (int o = kStepMaxParts / 2; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
            if (lane == 0) s_inv = rsqrtf(tot / float(args.hidden) + args.eps);
          }
          bad = compute_sync(bad);
          const float inv = s_inv;
#pragma unroll 2
          for (int i = i0 + tid; i < min(i1, args.hidden / 4); i += kStepCompute) {
            const float4 v = unpack4(s_row[i - i0]), ga = unpack4(static_cast<const uint2*>(gamma)[i]);
            const uint2 y = pack4(make_float4(v.x * inv * ga.x, v.y * inv * ga.y, v.z * inv * ga.z, v.w * inv * ga.w));
            reinterpret_cast<uint2*>(static_cast<T*>(args.xnorm) + size_t(b) * args.hidden)[i] = y;
            if (last)
              for (int q = 0; q < W; ++q) reinterpret_cast<uint2*>(static_cast<T*>(args.hidden_out[q]) + size_t(b) * args.hidden)[i] = y;
          }
          arrive(done);
        }
      }
    }
  }

  // ---- everyone leaves; tensor memory goes back -----------------------------------------------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 2) tmem_dealloc(tmem_base, 2 * kStepMaxBatch);
  if (*abort_flag && threadIdx.x == 0) {
    st_volatile_u32(args.abort_word, 1u);
    if (claim_status(args.abort_word, kTimeout)) {
      StatusBlock* sb = args.status;
      sb->rank = uint32_t(args.rank);
      sb->peer = uint32_t(args.rank);
      sb->wire = blockIdx.x;
      sb->where = 50;  // a wait of the decode step gave up
      __threadfence_system();
      sb->code = kTimeout;
      __threadfence_system();
    }
  }
}

// What the step needs before its first phase: the meeting points' counters at zero, and the first norm's output.  All loads of a row are
// in flight at once and it stays in registers: 6.0 -> 3.6 us cold for 32 rows of 8192, the whole step 0.6 % faster.
template <typename T>
__global__ void __launch_bounds__(512) decode_step_begin_kernel(const T* h, const T* gamma, T* xnorm, uint32_t* counters, int words, int hidden,
                                                                float eps) {
  constexpr int U = kStepMaxHidden / 8 / 512;
  __shared__ float s_part[16];
  const int tid = int(threadIdx.x), nvec = hidden / 8;
  pdl_launch_dependents();
  pdl_wait();
  const uint4* src = reinterpret_cast<const uint4*>(h + size_t(blockIdx.x) * hidden);
  uint4* dst = reinterpret_cast<uint4*>(xnorm + size_t(blockIdx.x) * hidden);
  uint4 x[U], g[U];
#pragma unroll
  for (int u = 0; u < U; ++u) x[u] = tid + u * 512 < nvec ? src[tid + u * 512] : make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (tid + u * 512 < nvec) g[u] = reinterpret_cast<const uint4*>(gamma)[tid + u * 512];
  for (int i = int(blockIdx.x) * 512 + tid; i < words; i += int(gridDim.x) * 512) counters[i] = 0;
  float2 ss = make_float2(0.f, 0.f);
#pragma unroll
  for (int u = 0; u < U; ++u) row_norm_squares<T>(ss, x[u]);
  float sum = ss.x + ss.y;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((tid & 31) == 0) s_part[tid >> 5] = sum;
  __syncthreads();
  float tot = s_part[tid & 15];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  const float inv = rsqrtf(tot / float(hidden) + eps);
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (tid + u * 512 < nvec) dst[tid + u * 512] = row_norm_scale<T>(x[u], g[u], inv);
}

}  // namespace b200ipc
