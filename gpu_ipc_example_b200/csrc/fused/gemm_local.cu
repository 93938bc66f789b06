#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>

#include "../common/check.h"
#include "fused_ops.h"
#include "gemm_local.cuh"
#include "gemm_stream.cuh"
#include "tensor_map.h"

namespace b200ipc {
namespace {

struct LocalPlan {
  int bn = 32, m_tiles = 1, splits = 1;
  int cut = 1;  // parts that the tiles behind the last full wave are taken in
};

// k blocks per stage: two where a block holds too little work for what its barriers and its commit cost
int local_ksub(int bn) { return bn <= 128 ? 2 : 1; }

int local_stages(int bn, int splits) {
  const int stage = (128 + bn / 2) * kGemmBK * 2 * local_ksub(bn);
  const int slab = (splits - 1) * (bn / splits) * 128 * 4;  // what the other pairs of a cluster hand over
  return std::min(kLocMaxStages, (kLocSmemBudget - 1024 - slab) / stage);
}

const void* local_kernel(DType t, int bn) {
  const bool two = local_ksub(bn) == 2;
  if (t == DType::F16)
    return two ? reinterpret_cast<const void*>(&gemm_local_kernel<__half, 2>) : reinterpret_cast<const void*>(&gemm_local_kernel<__half, 1>);
  return two ? reinterpret_cast<const void*>(&gemm_local_kernel<__nv_bfloat16, 2>)
             : reinterpret_cast<const void*>(&gemm_local_kernel<__nv_bfloat16, 1>);
}

// Pairs (clusters of 2, 4, 8 CTAs) that can run at once on a device.
int resident_clusters(const void* fn, int device, int splits) {
  static std::mutex mu;
  static std::map<std::pair<const void*, std::pair<int, int>>, int> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(fn, std::make_pair(device, splits));
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  B200_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kLocSmemBudget));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(2 * splits));
  cfg.blockDim = dim3(kLocThreads);
  cfg.dynamicSmemBytes = kLocSmemBudget;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(2 * splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  B200_CUDA_CHECK(cudaOccupancyMaxActiveClusters(&n, fn, &cfg));
  known[key] = n;
  return n;
}

// Microseconds that a plan takes apart from what all plans share (launch, first loads).  Fitted to one B200: a k block of a
// pair 0.08 + 0.0012 BN (K = 8192, M = 2048, N = 7168: BN = 160 166 us, 224 170, 256 197, 128 197); the epilogue of a
// tile 0.5 + 0.0133 BN, hidden behind the next tile's MMAs where there is one; handing partial sums between the pairs of a
// cluster 1.4 + 0.006 BN (K = 1024, M = 16, N = 8192: one split 15.4 us, two 17.4; K = 3584: 18.6 and 14.5 back to back; both
// taken with the first W loads ahead of the wait for the kernel in front, 15.5 with a prefetch to L2 there).
double plan_cost(int64_t tiles, int64_t room, int64_t kb_total, int bn, int splits, int cut) {
  auto wave = [&](int rows) { return std::max(double(ceil_div64(kb_total, splits)) * (0.08 + 0.0012 * rows), 0.5 + 0.0133 * rows / splits); };
  const int64_t left = tiles % room;
  return double(tiles / room) * wave(bn) + (left ? wave(bn / cut) : 0) + 0.5 + 0.0133 * (left ? bn / cut : bn) / splits +
         (splits > 1 ? 1.4 + 0.006 * bn : 0);
}

// The tile height and the K split of a problem.  bn_only: the tile's height is given (merged shards).
LocalPlan plan_local(DType t, int device, int64_t rows, int64_t shards, int64_t groups, int64_t N, int64_t kb_total, int bn_only) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int64_t, int64_t, int64_t, int64_t, int64_t, int>, LocalPlan> plans;
  const auto key = std::make_tuple(int(t), device, rows, shards, groups, N, kb_total, bn_only);
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = plans.find(key);
    if (it != plans.end()) return it->second;
  }
  LocalPlan best;
  double best_cost = 0;
  const int64_t n_tiles = ceil_div64(N, kLocWRows);
  for (int bn = bn_only ? bn_only : 32; bn <= (bn_only ? bn_only : kLocMaxBN); bn += 32) {
    const int64_t m_tiles = bn_only ? 1 : ceil_div64(rows, bn);
    if (!bn_only && bn > 32 && ceil_div64(rows, bn - 32) == m_tiles) continue;  // the lower tile covers the rows in as many
    const int64_t tiles = m_tiles * shards * groups * n_tiles;
    for (int splits = 1; splits <= 4; splits *= 2) {
      const int64_t room = resident_clusters(local_kernel(t, bn), device, splits);
      if (room < 1) continue;
      if (splits > 1 && (tiles > room || kb_total < 4 * splits)) break;  // one tile per cluster, every split with work
      // The last wave of tiles often fills a fraction of the GPU: cut in two or four it is over sooner (2048 rows x 3584 x 8192: 256
      // tiles of 256 rows for 74 pairs, the last 34 in two parts each).  Tall tiles and a long K only, and for what the model gives
      // as 4 % or more: with K = 1000 and tiles of 128 rows it measured behind.
      for (int cut = 1; cut <= 4; cut *= 2) {
        if (cut > 1 && (bn_only || splits > 1 || bn <= 128 || kb_total < 32 || bn % (16 * cut) || tiles <= room || tiles % room * cut > room)) continue;
        const double cost = plan_cost(tiles, room, kb_total, bn, splits, cut) * (cut > 1 ? 1.04 : 1.0);
        if (best_cost == 0 || cost < best_cost) {
          best_cost = cost;
          best.bn = bn;
          best.m_tiles = int(m_tiles);
          best.splits = splits;
          best.cut = cut;
        }
      }
    }
  }
  std::lock_guard<std::mutex> lk(mu);
  if (plans.size() >= 1024) plans.clear();  // a plan depends on nothing but its key and costs microseconds
  plans[key] = best;
  return best;
}

void launch_local(Comm& comm, LocalGemmArgs& args, DType t, const LocalPlan& p, const void* const* xs,
                  const void* const* ws, cudaStream_t stream, CollInfo* info) {
  const int W = comm.world();
  const void* fn = local_kernel(t, p.bn);
  args.bn = p.bn;
  args.m_tiles = p.m_tiles;
  args.n_tiles = int(ceil_div64(args.N, kLocWRows));
  args.splits = p.splits;
  args.stages = local_stages(p.bn, p.splits);
  args.warm_w = p.bn == 32 ? 1 : 0;
  const int64_t mt_all = int64_t(args.shards) * p.m_tiles;
  // as many m-tiles side by side as keep their X rows in a quarter of L2 while the W tiles pass by
  const int64_t x_bytes = int64_t(p.bn) * args.K * 2 * args.segs;
  args.band = int(std::min<int64_t>(mt_all, std::max<int64_t>(1, (int64_t(32) << 20) / x_bytes)));
  const int64_t total = mt_all * args.n_tiles * args.groups;
  const int64_t clusters = std::min<int64_t>(total, resident_clusters(fn, comm.device(), p.splits));
  B200_REQUIRE(clusters >= 1 && (p.splits == 1 || clusters == total), "GEMM kernel does not fit on the device");
  args.cut = p.cut;
  args.cut_from = int(p.cut > 1 ? total - total % clusters : total);
  for (int r = 0; r < W; ++r) {
    encode_tile_map(&args.tma_x[r], t, xs[r], uint64_t(args.rows), uint64_t(args.K), uint32_t(args.merged ? args.merged_rows : p.bn / 2));
    if (p.cut > 1) encode_tile_map(&args.tma_x_cut[r], t, xs[r], uint64_t(args.rows), uint64_t(args.K), uint32_t(p.bn / p.cut / 2));
    encode_tile_map(&args.tma_w[r], t, ws[r], uint64_t(args.N), uint64_t(args.K), 128);
  }
  KArgs views;
  comm.fill_views(&views, nullptr, nullptr, 0, 0);
  args.status = views.v[0].status;
  args.abort_word = reinterpret_cast<uint32_t*>(views.v[0].heap + views.lay.ctrl_off + kCtrlAbortOff);
  args.timeout_ns = views.v[0].timeout_ns;
  args.rank = views.v[0].rank;

  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(clusters * 2 * p.splits));
  cfg.blockDim = dim3(kLocThreads);
  cfg.dynamicSmemBytes = kLocSmemBudget;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(2 * p.splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2u : 1u;
  void* params[] = {&args};
  B200_CUDA_CHECK(cudaLaunchKernelExC(&cfg, fn, params));
  comm.note_launch();
  info->sched = SchedKind::Bulk;
  info->proto = ProtoKind::LL512;
  info->ctas = int(cfg.gridDim.x);
  info->warps = kLocThreads / 32;
  info->nwires = info->ctas * info->warps;
  info->steps = args.cut_from + (total - args.cut_from) * p.cut;  // tiles and parts of tiles that the pairs take
  info->launches = 1;
}

template <typename T>
const void* stream_kernel_of(int bn) {
  return bn == 16 ? reinterpret_cast<const void*>(&gemm_stream_kernel<T, 16>)
         : bn == 32 ? reinterpret_cast<const void*>(&gemm_stream_kernel<T, 32>) : reinterpret_cast<const void*>(&gemm_stream_kernel<T, 64>);
}
const void* stream_kernel(DType t, int bn) { return t == DType::F16 ? stream_kernel_of<__half>(bn) : stream_kernel_of<__nv_bfloat16>(bn); }

// Accumulator columns and K split of the weight-streaming kernel; bn = 0 where the tiles of gemm_local.cuh are taken.
struct StreamPlan {
  int bn = 0, splits = 1;
};

// `columns`: the rows of X, with their padding between shards; `exact`: the accumulator has just these.  As many splits as there
// are places for CTAs (two on an SM), with at least eight blocks of K and four rows to finish for each; a narrow layer pads its rows
// to 32 for an eighth split (8 rows x 8192 x 1280: four splits 13.1 us, eight 9.6, the other kernel 11.4).  That one keeps what
// it measured ahead or level in (with norm, this kernel / that one): more than 16 rows for a CTA to finish (24 rows x 448 x 4864
// 8.2 us / 7.8), more than 32 rows where that leaves places empty (fewer than 200 of the 296 that 148 SMs have: 48 x 3584 x 8192, 256
// CTAs 17.0 / 18.7; 48 x 3000 x 5120, 160 CTAs 15.2 / 14.0), weights of which the part fetched ahead is next to nothing (470 MB: 81 / 80).
StreamPlan plan_stream(const Comm& comm, int64_t columns, bool exact, int64_t tiles, int64_t kb_total) {
  StreamPlan p;
  if (columns > kStrMaxRows || (exact && columns != 16 && columns != 32 && columns != 64)) return p;
  if (tiles * kb_total * kStrTileBytes > (int64_t(192) << 20)) return p;
  int bn = columns <= 16 ? 16 : columns <= 32 ? 32 : 64;
  auto room = [&](int splits) { return tiles * splits <= 2 * comm.sm_count() && kb_total >= 8 * splits; };
  while (p.splits < 8 && bn / (2 * p.splits) >= 4 && room(2 * p.splits)) p.splits *= 2;
  if (bn == 16 && p.splits == 4 && !exact && room(8)) {
    bn = 32;
    p.splits = 8;
  }
  if (std::min<int64_t>(bn / p.splits, columns) <= 16 && (bn < 64 || tiles * p.splits >= 200)) p.bn = bn;
  return p;
}

void launch_stream(Comm& comm, StreamGemmArgs& args, DType t, const StreamPlan& p, const void* const* xs, const void* const* ws,
                   cudaStream_t stream, CollInfo* info) {
  const int W = comm.world();
  const void* fn = stream_kernel(t, p.bn);
  args.n_tiles = int(ceil_div64(args.N, kStrWRows));
  args.splits = p.splits;
  const int64_t ctas = int64_t(args.n_tiles) * args.groups * p.splits;
  const int slab = (p.splits - 1) * (p.bn / p.splits) * 128 * 4;
  args.stages = std::min(kStrMaxStages, (kStrSmemBudget - 1024 - slab) / (kStrTileBytes + p.bn * kGemmBK * 2));
  args.warm = int(kStrWarmBytes / (ctas * kStrTileBytes));
  for (int r = 0; r < W; ++r) {
    encode_tile_map(&args.tma_x[r], t, xs[r], uint64_t(args.rows), uint64_t(args.K), uint32_t(args.merged ? args.merged_rows : p.bn));
    encode_tile_map(&args.tma_w[r], t, ws[r], uint64_t(args.N), uint64_t(args.K), kStrWRows);
    args.w[r] = ws[r];
  }
  KArgs views;
  comm.fill_views(&views, nullptr, nullptr, 0, 0);
  args.status = views.v[0].status;
  args.abort_word = reinterpret_cast<uint32_t*>(views.v[0].heap + views.lay.ctrl_off + kCtrlAbortOff);
  args.timeout_ns = views.v[0].timeout_ns;
  args.rank = views.v[0].rank;
  B200_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kStrSmemBudget));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(ctas));
  cfg.blockDim = dim3(kStrThreads);
  cfg.dynamicSmemBytes = kStrSmemBudget;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(p.splits);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2u : 1u;
  void* params[] = {&args};
  B200_CUDA_CHECK(cudaLaunchKernelExC(&cfg, fn, params));
  comm.note_launch();
  info->sched = SchedKind::Bulk;
  info->proto = ProtoKind::LL512;
  info->ctas = int(ctas);
  info->warps = kStrThreads / 32;
  info->nwires = info->ctas * info->warps;
  info->steps = 1;
  info->launches = 1;
}

void check_local(Comm& comm, int64_t M, int64_t N, int64_t K) {
  B200_REQUIRE(comm.nlocal() == comm.world(), "every rank must be driven by this process");
  const int W = comm.world();
  B200_REQUIRE(W == 1 || W == 2 || W == 4 || W == 8, "world size must be 1, 2, 4 or 8");  // a tile of merged shards is cut in powers of two
  B200_REQUIRE(M > 0 && N > 0 && K > 0, "empty GEMM");
  B200_REQUIRE(N % 64 == 0, "N must be a multiple of 64");
  B200_REQUIRE(K % 8 == 0, "K must be a multiple of 8");
  B200_CUDA_CHECK(cudaSetDevice(comm.device()));
}

}  // namespace

CollInfo local_gemm_allreduce(Comm& comm, DType t, const GemmArPtrs* ptrs, int64_t M, int64_t N, int64_t K, float eps,
                              bool with_norm, cudaStream_t stream, uint32_t flags) {
  check_local(comm, M, N, K);
  const int W = comm.world();
  const int64_t kb = ceil_div64(K, kGemmBK) * W;
  const StreamPlan stream_plan = plan_stream(comm, M, false, ceil_div64(N, kStrWRows), kb);
  LocalGemmArgs args;
  StreamGemmArgs sargs;
  if (stream_plan.bn) {
    std::memset(&sargs, 0, sizeof(sargs));
    sargs.rows = int(M);
    sargs.N = int(N);
    sargs.K = int(K);
    sargs.segs = W;
    sargs.groups = 1;
    sargs.mute = (flags & kMuteSends) != 0;
  } else {
    std::memset(&args, 0, sizeof(args));
    args.rows = int(M);
    args.N = int(N);
    args.K = int(K);
    args.segs = W;
    args.shards = args.groups = 1;
    args.mute = (flags & kMuteSends) != 0;
  }
  RowNormArgs norm;
  std::memset(&norm, 0, sizeof(norm));
  norm.N = int(N);
  norm.eps = eps;
  const void* xs[kMaxRanks];
  const void* ws[kMaxRanks];
  for (int i = 0; i < W; ++i) {
    const GemmArPtrs& p = ptrs[i];
    for (const void* q : {p.residual, p.gamma, static_cast<const void*>(p.out), static_cast<const void*>(p.res_out)})
      B200_REQUIRE((reinterpret_cast<uintptr_t>(q) & 15) == 0, "linear + all-reduce needs 16-byte aligned tensors");
    if (with_norm) B200_REQUIRE(p.gamma != nullptr, "RMSNorm needs gamma");
    xs[i] = p.x;
    ws[i] = p.w;
    void* sum = p.res_out ? p.res_out : p.out;
    void* copy = (p.res_out && !with_norm) ? p.out : nullptr;
    (stream_plan.bn ? sargs.residual : args.residual)[i] = p.residual;
    (stream_plan.bn ? sargs.sum : args.sum)[i] = sum;
    (stream_plan.bn ? sargs.copy : args.copy)[i] = copy;
    norm.sum[i] = sum;
    norm.gamma[i] = p.gamma;
    norm.out[i] = p.out;
  }
  CollInfo info;
  if (stream_plan.bn)
    launch_stream(comm, sargs, t, stream_plan, xs, ws, stream, &info);
  else
    launch_local(comm, args, t, plan_local(t, comm.device(), M, 1, 1, N, kb, 0), xs, ws, stream, &info);
  if (with_norm) {
    // two vectors a thread where there are too few rows to fill the GPU otherwise
    const int threads = M * W <= 2 * comm.sm_count() ? 512 : 256;
    const void* nf = t == DType::F16 ? reinterpret_cast<const void*>(&row_norm_kernel<__half>)
                                     : reinterpret_cast<const void*>(&row_norm_kernel<__nv_bfloat16>);
    void* params[] = {&norm};
    B200_CUDA_CHECK(launch_maybe_pdl(nf, dim3(unsigned(M), unsigned(W)), dim3(unsigned(threads)), params, 0, stream, true));
    comm.note_launch();
    info.launches = 2;
  }
  return info;
}

CollInfo local_allgather_gemm(Comm& comm, DType t, const AgGemmPtrs* ptrs, int64_t M, int64_t N, int64_t K, cudaStream_t stream) {
  check_local(comm, M, N, K);
  const int W = comm.world();
  B200_REQUIRE(M % W == 0, "the rows of X must divide evenly over the ranks");
  LocalGemmArgs args;
  std::memset(&args, 0, sizeof(args));
  args.rows = int(M / W);
  args.N = int(N);
  args.K = int(K);
  args.segs = 1;
  args.shards = args.groups = W;
  // Few rows: one tile takes the rows of all shards, so that W is read once and not once per shard (4 ranks, 16 rows each,
  // K = 8192, N = 7168: 133 us, one shard per tile 180).
  int bn_only = 0;
  if (W > 1) {
    const int64_t unit = W == 2 ? 16 : 8;  // whole swizzle blocks, and a tile of a multiple of 32 rows
    const int64_t per_shard = ceil_div64(M / W, unit) * unit;
    if (per_shard * W <= kLocMaxBN) {
      args.merged = W;
      args.merged_rows = int(per_shard);
      args.shards = 1;
      bn_only = int(per_shard * W);
    }
  }
  // the weight-streaming kernel's tile: all shards side by side, in whole swizzle blocks of eight rows
  const int64_t stream_rows = W > 1 ? ceil_div64(M / W, 8) * 8 : M;
  const StreamPlan stream_plan = plan_stream(comm, stream_rows * W, W > 1, ceil_div64(N, kStrWRows) * W, ceil_div64(K, kGemmBK));
  const void* xs[kMaxRanks];
  const void* ws[kMaxRanks];
  for (int i = 0; i < W; ++i) {
    B200_REQUIRE((reinterpret_cast<uintptr_t>(ptrs[i].out) & 15) == 0, "x and out must be 16-byte aligned");
    xs[i] = ptrs[i].x_shard;
    ws[i] = ptrs[i].w;
    args.sum[i] = ptrs[i].out;
  }
  CollInfo info;
  if (stream_plan.bn) {
    StreamGemmArgs sargs;
    std::memset(&sargs, 0, sizeof(sargs));
    sargs.rows = args.rows;
    sargs.N = args.N;
    sargs.K = args.K;
    sargs.segs = 1;
    sargs.groups = W;
    if (W > 1) {
      sargs.merged = W;
      sargs.merged_rows = int(stream_rows);
    }
    for (int i = 0; i < W; ++i) sargs.sum[i] = ptrs[i].out;
    launch_stream(comm, sargs, t, stream_plan, xs, ws, stream, &info);
    return info;
  }
  launch_local(comm, args, t, plan_local(t, comm.device(), M / W, args.shards, W, N, ceil_div64(K, kGemmBK), bn_only), xs, ws, stream, &info);
  return info;
}

}  // namespace b200ipc
