#include "decode_step.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "../common/check.h"
#include "../common/cu_driver.h"
#include "../common/pdl.h"
#include "../fused/tensor_map.h"
#include "decode_step.cuh"

namespace b200ipc {
namespace {

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
size_t round_up(size_t v) { return (v + 255) / 256 * 256; }

// Units of the longest GEMM and of the attention, and the tiles behind the former.
struct StepSizes {
  int64_t tiles, units, sequences, attn_units;
};
StepSizes step_sizes(int W, const DecodeStepShape& s, int pos) {
  const int64_t kb_hidden = ceil_div(s.hidden, kGemmBK), t_hidden = ceil_div(s.hidden, kStepTileRows);
  const int64_t tiles[5] = {int64_t(W) * (s.hq + 2 * s.hkv), t_hidden, 2 * W * ceil_div(s.ffn, kStepTileRows), t_hidden, W * ceil_div(s.vocab, kStepTileRows)};
  const int64_t kb[5] = {kb_hidden, int64_t(W) * s.hq * (kAttnD / kGemmBK), kb_hidden, W * ceil_div(s.ffn, kGemmBK), kb_hidden};
  StepSizes z{0, 0, int64_t(W) * s.batch * s.hkv, 0};
  for (int i = 0; i < 5; ++i) {
    z.tiles = std::max(z.tiles, tiles[i]);
    z.units = std::max(z.units, tiles[i] * kb[i]);
  }
  z.attn_units = z.sequences * ceil_div(pos, kStepPos);
  return z;
}

struct StepLayout {
  size_t sync, arrivals, squares, xnorm, attn, act, part, apart, total;
  int counter_words;
};
StepLayout step_layout(const Comm& comm, const DecodeStepShape& s) {
  const int W = comm.world(), ctas = comm.sm_count();
  const StepSizes z = step_sizes(W, s, s.max_ctx);
  const int G = s.hq / s.hkv;
  StepLayout l;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += round_up(bytes);
    return here;
  };
  l.sync = take(size_t(s.layers + 1) * kStepSyncs * kStepSyncStride * 4);
  l.arrivals = take(size_t(z.sequences + s.batch) * 4);
  l.squares = take(size_t(2 * s.batch) * kStepMaxParts * 4);
  l.counter_words = int(at / 4);
  l.xnorm = take(size_t(s.batch) * s.hidden * 2);
  l.attn = take(size_t(W) * s.batch * s.hq * kAttnD * 2);
  l.act = take(size_t(W) * s.batch * s.ffn * 2);
  l.part = take(size_t(z.tiles + ctas) * s.batch * kStepTileRows * 4);
  l.apart = take(std::max(size_t(z.sequences + ctas) * G * kMergeRow * 4, size_t(s.batch) * kStepMaxParts * sizeof(Best)));
  l.total = at;
  return l;
}

const void* step_kernel(DType t) {
  return t == DType::F16 ? reinterpret_cast<const void*>(&decode_step_kernel<__half>) : reinterpret_cast<const void*>(&decode_step_kernel<__nv_bfloat16>);
}

// Positions [0, pos) of a cache [sequences, max_ctx, 128], in boxes of 64 positions x 64 dimensions; a box that reaches past
// the last of them is filled with zeros.
void encode_cache_map(CUtensorMap* map, DType t, void* base, int sequences, int max_ctx, int pos) {
  cuuint64_t dims[3] = {cuuint64_t(kAttnD), cuuint64_t(pos), cuuint64_t(sequences)};
  cuuint64_t strides[2] = {cuuint64_t(kAttnD) * 2, cuuint64_t(max_ctx) * kAttnD * 2};
  cuuint32_t box[3] = {cuuint32_t(kGemmBK), cuuint32_t(kStepPos), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  B200_CU_CHECK(cu().TensorMapEncodeTiled(map, t == DType::F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base,
                                          dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
}

}  // namespace

bool decode_step_takes(const Comm& comm, const DecodeStepShape& s, int pos) {
  const int W = comm.world();
  if (comm.nlocal() != W || !(W == 1 || W == 2 || W == 4 || W == 8)) return false;
  if (s.batch < 1 || s.batch > kStepMaxBatch || s.layers < 1 || pos < 1 || pos >= s.max_ctx) return false;
  if (s.hkv < 1 || s.hq % s.hkv || s.hidden % 64 || s.hidden > kStepMaxHidden || s.ffn % 8 || s.ffn < 1 || s.vocab < 1) return false;
  const int G = s.hq / s.hkv;
  if (!(G == 1 || G == 2 || G == 4 || G == 8)) return false;
  const StepSizes z = step_sizes(W, s, s.max_ctx);
  // run_of() multiplies a unit with the number of CTAs in 32 bits
  return std::max(z.units, z.attn_units) * comm.sm_count() < (int64_t(1) << 31) && int64_t(W) * s.vocab < (int64_t(1) << 31);
}

// Eight heads per KV head and an accumulator for 64 sequences leave room for seven stages, three K and V pairs: too few in flight where
// the attention is most of the step.  One rank, FFN 3584, graphs, this kernel / the chain: 64 sequences, 4 KV heads, hidden 4096, 166
// tiles per SM 219 / 214 us, 221 263 / 250, 110 175 / 173; hidden 8192, 8 KV heads, 443 tiles 497 / 457; 56 sequences there 454 / 443,
// 52 432 / 441, 48 412 / 443 (the chain splits the context less evenly below 56).  Four heads per KV head, 886 tiles 719 / 733; two ranks,
// 443 tiles 450 / 463.
bool decode_step_pays(const Comm& comm, const DecodeStepShape& s, int pos) {
  return !(comm.world() == 1 && s.hq == 8 * s.hkv && s.batch >= 56 &&
           step_sizes(1, s, pos).attn_units >= int64_t(160) * comm.sm_count());
}

size_t decode_step_workspace_bytes(const Comm& comm, const DecodeStepShape& s) { return step_layout(comm, s).total; }

void decode_step(Comm& comm, DType t, const DecodeStepShape& s, const DecodeStepPtrs& p, int pos, float eps, float theta, cudaStream_t stream,
                 uint32_t flags) {
  B200_REQUIRE(decode_step_takes(comm, s, pos) && theta > 0.f, "decode step: shape not supported");
  B200_CUDA_CHECK(cudaSetDevice(comm.device()));
  const int W = comm.world(), G = s.hq / s.hkv, ctas = comm.sm_count();
  const StepLayout lay = step_layout(comm, s);
  char* ws = static_cast<char*>(p.workspace);
  DecodeStepArgs a;
  std::memset(&a, 0, sizeof(a));
  a.h = p.h;
  a.xnorm = ws + lay.xnorm;
  a.attn = ws + lay.attn;
  a.act = ws + lay.act;
  a.part = reinterpret_cast<float*>(ws + lay.part);
  a.apart = reinterpret_cast<float*>(ws + lay.apart);
  a.squares = reinterpret_cast<uint32_t*>(ws + lay.squares);
  a.sync = reinterpret_cast<uint32_t*>(ws + lay.sync);
  a.arrivals = reinterpret_cast<uint32_t*>(ws + lay.arrivals);
  KArgs views;
  comm.fill_views(&views, nullptr, nullptr, 0, 0);
  a.status = views.v[0].status;
  a.abort_word = reinterpret_cast<uint32_t*>(views.v[0].heap + views.lay.ctrl_off + kCtrlAbortOff);
  a.timeout_ns = views.v[0].timeout_ns;
  a.rank = views.v[0].rank;
  a.world = W;
  a.batch = s.batch;
  a.bn = s.batch <= 16 ? 16 : s.batch <= 32 ? 32 : 64;
  a.hidden = s.hidden;
  a.hq = s.hq;
  a.hkv = s.hkv;
  a.ffn = s.ffn;
  a.vocab = s.vocab;
  a.max_ctx = s.max_ctx;
  a.pos = pos;
  a.mute = (flags & kMuteSends) != 0;
  a.eps = eps;
  a.scale_log2 = 1.4426950408889634f / sqrtf(float(kAttnD));
  a.log2_theta = log2f(theta);
  const int stage_bytes = kStepTileBytes + a.bn * kGemmBK * 2;
  a.stages = std::min(kStepMaxStages, (kStepSmemBudget - 1024 - step_scratch_bytes(G, s.hidden)) / stage_bytes);
  const uint32_t bn = uint32_t(a.bn), B = uint32_t(s.batch);
  encode_tile_map(&a.x_norm, t, a.xnorm, B, uint64_t(s.hidden), bn);
  for (int r = 0; r < W; ++r) {
    encode_tile_map(&a.x_attn[r], t, static_cast<char*>(a.attn) + size_t(r) * B * s.hq * kAttnD * 2, B, uint64_t(s.hq) * kAttnD, bn);
    encode_tile_map(&a.x_act[r], t, static_cast<char*>(a.act) + size_t(r) * B * s.ffn * 2, B, uint64_t(s.ffn), bn);
    a.hidden_out[r] = p.hidden_out[size_t(r)];
    encode_tile_map(&a.head[r], t, p.head[size_t(r)], uint64_t(s.vocab), uint64_t(s.hidden), kStepTileRows);
  }
  a.ids = p.ids;

  {
    const void* fn = t == DType::F16 ? reinterpret_cast<const void*>(&decode_step_begin_kernel<__half>)
                                     : reinterpret_cast<const void*>(&decode_step_begin_kernel<__nv_bfloat16>);
    const void* gamma = p.gamma_attn[0];
    int words = lay.counter_words, hidden = s.hidden;
    float e = eps;
    void* params[] = {&a.h, &gamma, &a.xnorm, &a.sync, &words, &hidden, &e};
    B200_CUDA_CHECK(launch_maybe_pdl(fn, dim3(B), dim3(512), params, 0, stream, true));
    comm.note_launch();
  }
  const void* fn = step_kernel(t);
  B200_CUDA_CHECK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmemBudget));
  const int per_launch = kStepMaps / (kStepMapsPerRank * W);
  for (int l0 = 0; l0 < s.layers; l0 += per_launch) {
    a.first_layer = l0;
    a.layers = std::min(per_launch, s.layers - l0);
    a.with_head = l0 + a.layers == s.layers;
    for (int l = 0; l < a.layers; ++l) {
      a.gamma_mlp[l] = p.gamma_mlp[size_t(l0 + l)];
      a.gamma_attn[l] = l0 + l + 1 < s.layers ? p.gamma_attn[size_t(l0 + l + 1)] : p.gamma_final;
      for (int r = 0; r < W; ++r) {
        const size_t i = size_t(l0 + l) * W + size_t(r), to = size_t(l) * W + size_t(r);
        CUtensorMap* m = a.maps + to * kStepMapsPerRank;
        encode_tile_map(m + 0, t, p.wqkv[i], uint64_t(s.hq + 2 * s.hkv) * kAttnD, uint64_t(s.hidden), kStepTileRows);
        encode_tile_map(m + 1, t, p.wo[i], uint64_t(s.hidden), uint64_t(s.hq) * kAttnD, kStepTileRows);
        encode_tile_map(m + 2, t, p.wgu[i], uint64_t(s.ffn) * 2, uint64_t(s.hidden), kStepTileRows);
        encode_tile_map(m + 3, t, p.wdown[i], uint64_t(s.hidden), uint64_t(s.ffn), kStepTileRows);
        encode_cache_map(m + 4, t, p.kcache[i], s.batch * s.hkv, s.max_ctx, pos);
        encode_cache_map(m + 5, t, p.vcache[i], s.batch * s.hkv, s.max_ctx, pos);
        a.kcache[to] = p.kcache[i];
        a.vcache[to] = p.vcache[i];
      }
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(ctas));
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = kStepSmemBudget;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;  // CTAs wait on one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* params[] = {&a};
    B200_CUDA_CHECK(cudaLaunchKernelExC(&cfg, fn, params));
    comm.note_launch();
  }
}

}  // namespace b200ipc
