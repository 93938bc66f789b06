#include "fused_ops.h"

#include <algorithm>
#include <cstring>

#include "../common/check.h"
#include "norm_direct.cuh"
#include "oneshot_fused.cuh"

namespace b200ipc {
namespace {

template <typename T, typename Tout, int EPI>
KernelFn pick_world(int world) {
  auto cast = [](auto f) { return reinterpret_cast<KernelFn>(f); };
  switch (world) {
    case 1: return cast(&oneshot_fused_kernel<T, Tout, 1, EPI>);
    case 2: return cast(&oneshot_fused_kernel<T, Tout, 2, EPI>);
    case 4: return cast(&oneshot_fused_kernel<T, Tout, 4, EPI>);
    case 8: return cast(&oneshot_fused_kernel<T, Tout, 8, EPI>);
    default: return nullptr;
  }
}

// Vectors of a row that one CTA of the direct kernel can hold.
int64_t direct_norm_cta_vecs(int world) { return (world == 8 ? 1 : 2) * kDirectNormThreads; }
template <typename T, int N>
const void* direct_norm_fn(int u) {
  if constexpr (N < 8) {
    if (u == 2) return reinterpret_cast<const void*>(&direct_norm_kernel<T, N, 2>);
  }
  return reinterpret_cast<const void*>(&direct_norm_kernel<T, N, 1>);
}
template <typename T>
const void* direct_norm_lookup(int world, int u) {
  switch (world) {
    case 1: return direct_norm_fn<T, 1>(u);
    case 2: return direct_norm_fn<T, 2>(u);
    case 4: return direct_norm_fn<T, 4>(u);
    case 8: return direct_norm_fn<T, 8>(u);
    default: return nullptr;
  }
}

uint32_t float_bits(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return u;
}

// One launch, clusters of `parts` CTAs per row.
CollInfo direct_norm(Comm& comm, DType t, const FusedNormPtrs* ptrs, int64_t rows, int64_t hidden, float eps, cudaStream_t stream) {
  const int N = comm.world();
  const int64_t vecs = hidden / 8;
  // As many CTAs per row as it takes to have a CTA on every SM, each with a warp's worth of vectors at least; and no more than
  // 256 vectors a CTA, so that several CTAs share an SM's registers (512 rows of 8192 on 8 ranks 65 -> 53 us, on 4 ranks 37 -> 29).
  int64_t parts = 1;
  while (parts < kDirectNormMaxParts &&
         (ceil_div64(vecs, parts) > 256 || (rows * parts * 2 <= comm.sm_count() && ceil_div64(vecs, parts * 2) >= 32)))
    parts *= 2;
  const int64_t part_vecs = ceil_div64(vecs, parts);
  const int u = part_vecs > kDirectNormThreads ? 2 : 1;
  const int threads = int(round_up64(ceil_div64(part_vecs, u), 32));
  B200_REQUIRE(part_vecs <= int64_t(u) * threads && threads <= kDirectNormThreads && rows * parts <= INT32_MAX, "row too long or too many rows");
  DirectNormArgs args;
  std::memset(&args, 0, sizeof(args));
  for (int i = 0; i < N; ++i) {
    args.x[i] = ptrs[i].x;
    args.residual[i] = ptrs[i].residual;
    args.gamma[i] = ptrs[i].gamma;
    args.out[i] = ptrs[i].out;
    args.res_out[i] = ptrs[i].residual_out;
  }
  args.row_vecs = int(vecs);
  args.part_vecs = int(part_vecs);
  args.hidden = float(hidden);
  args.eps = eps;
  const void* fn = t == DType::F16 ? direct_norm_lookup<__half>(N, u) : direct_norm_lookup<__nv_bfloat16>(N, u);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(rows * parts));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(parts);
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2u : 1u;
  void* params[] = {&args};
  B200_CUDA_CHECK(cudaLaunchKernelExC(&cfg, fn, params));
  comm.note_launch();
  CollInfo info;
  info.sched = SchedKind::Bulk;
  info.proto = ProtoKind::LL512;
  info.ctas = int(cfg.gridDim.x);
  info.warps = threads / 32;
  info.nwires = info.ctas * info.warps;
  info.steps = u;
  info.launches = 1;
  return info;
}

}  // namespace

bool direct_norm_takes(const Comm& comm, int64_t hidden) {
  return comm.nlocal() == comm.world() && comm.max_ctas() == 0 && hidden > 0 && hidden % 8 == 0 && direct_norm_lookup<__half>(comm.world(), 1) != nullptr &&
         hidden / 8 <= kDirectNormMaxParts * direct_norm_cta_vecs(comm.world());
}

CollInfo fused_allreduce_residual_rmsnorm(Comm& comm, DType t, const FusedNormPtrs* ptrs, int64_t rows, int64_t hidden,
                                          float eps, int ctas_req, cudaStream_t stream) {
  B200_REQUIRE(rows > 0 && hidden > 0 && hidden % 8 == 0, "hidden must be a positive multiple of 8");
  const int N = comm.world();
  for (int i = 0; i < comm.nlocal(); ++i)
    for (const void* p : {ptrs[i].x, ptrs[i].residual, ptrs[i].gamma, static_cast<const void*>(ptrs[i].out),
                          static_cast<const void*>(ptrs[i].residual_out)})
      B200_REQUIRE((reinterpret_cast<uintptr_t>(p) & 15) == 0, "fused all-reduce + RMSNorm needs 16-byte aligned tensors");
  // Every rank is driven by this process: no exchange (an explicit CTA count, or a limit on them, asks for the kernel with it).  8 ranks, 16 rows
  // of 8192: 9.2 us against 20.4 (device time, cold cache).
  if (ctas_req == 0 && direct_norm_takes(comm, hidden)) return direct_norm(comm, t, ptrs, rows, hidden, eps, stream);
  KernelFn fn = t == DType::F16 ? pick_world<__half, __half, kEpiNorm>(N) : pick_world<__nv_bfloat16, __nv_bfloat16, kEpiNorm>(N);
  B200_REQUIRE(fn != nullptr, "no fused kernel for world size " << N);
  B200_CUDA_CHECK(cudaSetDevice(comm.device()));

  // Geometry: a CTA owns whole rows; its warps share the row's transactions.
  const int64_t row_dw = hidden / 2;
  const int64_t row_tx = ceil_div64(row_dw, 120);
  const int64_t want_warps = kFusedMaxThreads / 32;
  int warps = int(std::max<int64_t>(4, round_up64(std::min<int64_t>(row_tx, want_warps), 4)));
  int threads = warps * 32;
  int cap = std::min(comm.resident_ctas(fn, threads, 0), kMaxOneShotWires / warps);
  B200_REQUIRE(cap >= 1, "fused kernel does not fit");
  int ctas = ctas_req > 0 ? ctas_req : int(std::min<int64_t>(rows, cap));
  B200_REQUIRE(ctas <= cap, "requested " << ctas << " CTAs, only " << cap << " can run at once");
  const int64_t rows_per_cta = ceil_div64(rows, ctas);
  B200_REQUIRE(rows_per_cta <= kFusedMaxRowsPerCta,
               "too many rows (" << rows << ") for the one-shot fused kernel: at most " << int64_t(cap) * kFusedMaxRowsPerCta);
  const int64_t steps = ceil_div64(ceil_div64(rows_per_cta * row_dw, 120), warps);

  std::vector<const void*> ins(size_t(comm.nlocal()));
  std::vector<void*> outs(size_t(comm.nlocal()));
  for (int i = 0; i < comm.nlocal(); ++i) {
    ins[size_t(i)] = ptrs[i].x;
    outs[size_t(i)] = ptrs[i].out;
  }
  KArgs args;
  comm.fill_views(&args, ins.data(), outs.data(), size_t(rows * hidden), 0);
  const uint32_t adv = uint32_t(steps + 1);
  const uint32_t first = comm.take_seq(adv);
  for (int i = 0; i < comm.nlocal(); ++i) {
    args.v[i].seq = first;
    args.v[i].seq_step = adv;
    args.v[i].aux[0] = reinterpret_cast<uint64_t>(ptrs[i].residual);
    args.v[i].aux[1] = reinterpret_cast<uint64_t>(ptrs[i].gamma);
    args.v[i].aux[2] = reinterpret_cast<uint64_t>(ptrs[i].residual_out);
    args.v[i].aux[3] = uint64_t(uint32_t(hidden)) | (uint64_t(float_bits(eps)) << 32);
  }
  comm.launch(fn, ctas, threads, &args, 0, stream, true);
  CollInfo info;
  info.sched = SchedKind::OneShot;
  info.proto = ProtoKind::LL512;
  info.ctas = ctas;
  info.warps = warps;
  info.nwires = ctas * warps;
  info.steps = steps;
  info.first_flag = first;
  info.launches = 1;
  return info;
}

CollInfo fused_allreduce_scale_cast(Comm& comm, DType tin, DType tout, const void* const* ins, void* const* outs,
                                    size_t nelems, float scale, int ctas_req, cudaStream_t stream) {
  B200_REQUIRE(nelems > 0 && nelems % 2 == 0, "element count must be even");
  const int N = comm.world();
  KernelFn fn;
  if (tin == DType::F16)
    fn = tout == DType::F16 ? pick_world<__half, __half, kEpiScale>(N) : pick_world<__half, __nv_bfloat16, kEpiScale>(N);
  else
    fn = tout == DType::F16 ? pick_world<__nv_bfloat16, __half, kEpiScale>(N)
                            : pick_world<__nv_bfloat16, __nv_bfloat16, kEpiScale>(N);
  B200_REQUIRE(fn != nullptr, "no fused kernel for world size " << N);
  B200_CUDA_CHECK(cudaSetDevice(comm.device()));
  const int64_t total_dw = int64_t(nelems / 2);
  const int64_t ntx = ceil_div64(total_dw, 120);
  int warps = int(std::min<int64_t>(16, std::max<int64_t>(1, ntx)));
  int threads = warps * 32;
  int cap = std::min(comm.resident_ctas(fn, threads, 0), kMaxOneShotWires / warps);
  B200_REQUIRE(cap >= 1, "fused kernel does not fit");
  int ctas = ctas_req > 0 ? ctas_req : int(std::min<int64_t>(cap, ceil_div64(ntx, warps)));
  B200_REQUIRE(ctas <= cap, "requested " << ctas << " CTAs, only " << cap << " can run at once");
  const int64_t per = round_up64(ceil_div64(total_dw, ctas), 4);
  const int64_t steps = ceil_div64(ceil_div64(per, 120), warps);

  KArgs args;
  comm.fill_views(&args, ins, outs, nelems, 0);
  const uint32_t adv = uint32_t(steps + 1);
  const uint32_t first = comm.take_seq(adv);
  for (int i = 0; i < comm.nlocal(); ++i) {
    args.v[i].seq = first;
    args.v[i].seq_step = adv;
    args.v[i].aux[3] = uint64_t(float_bits(scale)) << 32;
    B200_REQUIRE((reinterpret_cast<uintptr_t>(ins[i]) & 3) == 0 && (reinterpret_cast<uintptr_t>(outs[i]) & 3) == 0,
                 "buffers must be 4-byte aligned");
  }
  comm.launch(fn, ctas, threads, &args, 0, stream, true);
  CollInfo info;
  info.sched = SchedKind::OneShot;
  info.proto = ProtoKind::LL512;
  info.ctas = ctas;
  info.warps = warps;
  info.nwires = ctas * warps;
  info.steps = steps;
  info.first_flag = first;
  info.launches = 1;
  return info;
}

}  // namespace b200ipc
