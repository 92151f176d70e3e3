// The whole MoE block in one call: the chain of kernels that mini_qwen/model/layers/moe.py:49-68 of the reference
// stands for (router, renormalise, permute, experts, unpermute), optionally with the decoder layer's norm in front and
// residual behind (mini_qwen/model/qwen3_moe.py:63-66).
//
// What bounds it at decode sizes is the host: a layer is four to eight launches of a few microseconds each, and issuing
// them one by one from Python, with an allocation and a dozen tensor queries around each, took 100 us a call.  Here
// every launch, tensor map and workspace offset is computed natively from one description of the layer; the caller
// passes one workspace.
#include "common.cuh"
#include "tc5.cuh"

namespace mq {

bool tc5_covers(int64_t S, int64_t E, int64_t N, int64_t Kd, bool swiglu);
bool generic_small_groups(int64_t S, int64_t E, int64_t N, bool swiglu);
int grouped_gemm_generic_dispatch(const void* a, const void* w, const int32_t* offsets, int64_t S, int64_t E,
                                  int64_t period, int64_t N, int64_t Kd, int dtype, bool swiglu, void* out,
                                  cudaStream_t st, const int32_t* perm, int64_t top_k);
bool w4a16_stream_covers(int64_t S, int64_t E, int64_t period, int64_t N, int64_t Kd, int64_t group);

namespace {

// How a call runs.
struct BlockPlan {
  bool w4, small, prepared, tile, stream, tc5, gather_in_kernel;
};

BlockPlan plan_of(const mq_moe_layer& L, int64_t T) {
  const int64_t H = L.hidden, I = L.inter, E = L.experts, K = L.top_k, S = T * K;
  BlockPlan p = {};
  p.w4 = L.group_size > 0;
  // decode batches: logits, top-k, plan (and the W4A16 activation preparation) in one launch
  p.small = T <= 64 && E <= 256 && K <= 32 && S <= 2048;
  if (p.w4) {
    const bool streams = H <= 4096 && w4a16_stream_covers(S, E, E, I, H, L.group_size);
    const bool prepared = streams && p.small && T <= E;         // by the routing launch
    // The tile kernel by the rule of the W4A16 dispatch.  Its bulk copies want the zero points 16-byte aligned; the other
    // kernels read them word by word.
    p.tile = mq_w4a16_tile_pays(S, E, I, H, L.group_size, 1, !prepared) && T * (H / 8) < ((int64_t)1 << 32) &&
             aligned16(L.gate[2]) && aligned16(L.up[2]);
    p.stream = !p.tile && streams;
    p.prepared = !p.tile && prepared;
    p.gather_in_kernel = p.tile || p.stream;
  } else {
    p.tc5 = L.dtype == MQ_BF16 && tc5_covers(S, E, I, H, true) && T * H < ((int64_t)1 << 32);
    p.gather_in_kernel = p.tc5 || generic_small_groups(S, E, I, true);
  }
  return p;
}

// Workspace of a call, carved in this order; every piece starts at a multiple of 256 bytes.
struct BlockSpace {
  uint8_t* base;
  size_t used;
  void* take(size_t bytes) {
    void* p = base + used;
    used += (bytes + 255) & ~(size_t)255;
    return p;
  }
};
struct BlockBuffers {
  void *xn, *rows, *h, *y, *xp;
  float *xs, *weights, *logits;
  int32_t *ids32, *perm, *inv, *offsets;
  void* plan_ws;
  size_t logits_bytes, plan_bytes;
};

size_t carve(const mq_moe_layer& L, int64_t T, const BlockPlan& p, bool norm, uint8_t* base, BlockBuffers& b) {
  BlockSpace s{base, 0};
  const int64_t H = L.hidden, I = L.inter, E = L.experts, S = T * L.top_k;
  const size_t el = dtype_size(L.dtype);
  b = {};
  if (norm) b.xn = s.take((size_t)(T * H) * el);
  b.ids32 = (int32_t*)s.take((size_t)S * 4);
  b.weights = (float*)s.take((size_t)S * 4);
  b.perm = (int32_t*)s.take((size_t)S * 4);
  b.inv = (int32_t*)s.take((size_t)S * 4);
  b.offsets = (int32_t*)s.take((size_t)(E + 1) * 4);
  if (!p.small) {
    b.logits_bytes = mq_router_workspace_bytes(T, H, E);
    b.logits = (float*)s.take(b.logits_bytes);
    b.plan_bytes = mq_permute_workspace_bytes(S, E);
    b.plan_ws = s.take(b.plan_bytes);
  }
  if (p.stream) {
    const int64_t n = p.prepared ? T : S;
    b.xp = s.take((size_t)(n * H) * 2);
    b.xs = (float*)s.take((size_t)n * 32 * 4);
  }
  if (!p.gather_in_kernel) b.rows = s.take((size_t)(S * H) * el);
  b.h = s.take((size_t)(S * I) * el);
  b.y = s.take((size_t)(S * H) * el);
  return s.used;
}

bool layer_ok(const mq_moe_layer* L) {
  return L != nullptr && L->hidden > 0 && L->inter > 0 && L->experts > 0 && L->top_k > 0 && L->group_size >= 0 &&
         valid_dtype(L->dtype) && valid_dtype(L->router_dtype) && (L->group_size == 0 || L->dtype == MQ_BF16);
}

}  // namespace
}  // namespace mq

extern "C" size_t mq_moe_forward_workspace_bytes(const mq_moe_layer* h_layer, int64_t T) {
  if (!mq::layer_ok(h_layer) || T <= 0) return 256;
  mq::BlockBuffers b;
  return mq::carve(*h_layer, T, mq::plan_of(*h_layer, T), true, nullptr, b);
}

#define MQ_BLOCK_STEP(call)        \
  do {                             \
    const int rc_ = (call);        \
    if (rc_ != MQ_OK) return rc_;  \
  } while (0)

extern "C" int mq_moe_forward(const mq_moe_layer* h_layer, const void* x, const void* norm_weight, float norm_eps,
                              const void* residual, int64_t T, void* route_workspace, size_t route_workspace_bytes,
                              void* workspace, size_t workspace_bytes, void* out, int32_t* d_status,
                              int32_t* h_launches, void* stream) {
  using namespace mq;
  if (!layer_ok(h_layer) || T < 0) return MQ_ERR_INVALID_ARGUMENT;
  if (h_launches) *h_launches = 0;
  if (T == 0) return MQ_OK;
  if (!x || !out || !workspace || !aligned16(workspace)) return MQ_ERR_INVALID_ARGUMENT;
  const mq_moe_layer& L = *h_layer;
  const BlockPlan p = plan_of(L, T);
  BlockBuffers b;
  if (carve(L, T, p, norm_weight != nullptr, reinterpret_cast<uint8_t*>(workspace), b) > workspace_bytes)
    return MQ_ERR_WORKSPACE_TOO_SMALL;
  const int64_t H = L.hidden, I = L.inter, E = L.experts, K = L.top_k, S = T * K;
  int n = 0;
  if (norm_weight != nullptr) {
    MQ_BLOCK_STEP(mq_rms_norm(x, L.dtype, norm_weight, norm_eps, T, H, b.xn, stream));
    x = b.xn;
    ++n;
  }
  if (p.small) {
    if (!route_workspace) return MQ_ERR_INVALID_ARGUMENT;
    MQ_BLOCK_STEP(mq_route_small(x, L.dtype, L.router, L.router_dtype, L.router_bias, T, H, E, K, L.renormalize,
                                 route_workspace, route_workspace_bytes, nullptr, b.ids32, b.weights, b.perm, b.inv, nullptr,
                                 b.offsets, p.prepared ? b.xp : nullptr, p.prepared ? b.xs : nullptr, p.prepared ? 1 : 0,
                                 stream));
    ++n;
  } else {
    MQ_BLOCK_STEP(mq_router_topk(x, L.dtype, L.router, L.router_dtype, L.router_bias, T, H, E, K, L.renormalize, b.logits,
                                 b.logits_bytes, nullptr, b.ids32, b.weights, stream));
    MQ_BLOCK_STEP(mq_permute_plan(b.ids32, 0, T, K, E, b.perm, b.inv, nullptr, b.offsets, b.plan_ws, b.plan_bytes, stream));
    n += 2 + (S <= 2048 ? 1 : 3);
  }
  auto i32 = [](const void* q) { return reinterpret_cast<const int32_t*>(q); };
  if (!p.gather_in_kernel) {
    MQ_BLOCK_STEP(mq_gather_rows(x, L.dtype, b.perm, S, K, H, b.rows, stream));
    ++n;
  }
  if (!p.w4) {
    if (p.tc5)
      MQ_BLOCK_STEP(mq_grouped_swiglu_gather(x, b.perm, L.gate[0], b.offsets, T, K, E, E, I, H, L.dtype, b.h, d_status, stream));
    else if (p.gather_in_kernel)
      MQ_BLOCK_STEP(grouped_gemm_generic_dispatch(x, L.gate[0], b.offsets, S, E, E, I, H, L.dtype, true, b.h,
                                                  reinterpret_cast<cudaStream_t>(stream), b.perm, K));
    else
      MQ_BLOCK_STEP(mq_grouped_swiglu(b.rows, L.gate[0], b.offsets, S, E, E, I, H, L.dtype, b.h, d_status, stream));
    MQ_BLOCK_STEP(mq_grouped_gemm(b.h, L.down[0], b.offsets, S, E, E, H, I, L.dtype, b.y, d_status, stream));
  } else {
    if (p.tile) {
      MQ_BLOCK_STEP(mq_w4a16_grouped_swiglu_gather(x, b.perm, i32(L.gate[0]), L.gate[1], i32(L.gate[2]), i32(L.up[0]), L.up[1],
                                                   i32(L.up[2]), b.offsets, T, K, E, E, I, H, L.group_size, b.h, d_status,
                                                   stream));
    } else if (p.stream) {
      if (!p.prepared) {
        MQ_BLOCK_STEP(mq_w4a16_tc_prep(x, b.perm, K, S, H, 1, b.xp, b.xs, stream));
        ++n;
      }
      MQ_BLOCK_STEP(mq_w4a16_stream_swiglu(b.xp, b.xs, 1, p.prepared ? b.perm : nullptr, K, i32(L.gate[0]), L.gate[1],
                                           i32(L.gate[2]), i32(L.up[0]), L.up[1], i32(L.up[2]), b.offsets, S, E, E, I, H,
                                           L.group_size, 0, b.h, d_status, stream));
    } else {
      MQ_BLOCK_STEP(mq_w4a16_grouped_swiglu_ex(b.rows, i32(L.gate[0]), L.gate[1], i32(L.gate[2]), i32(L.up[0]), L.up[1],
                                               i32(L.up[2]), b.offsets, S, 0, E, E, I, H, L.group_size, b.h, d_status,
                                               stream));
    }
    MQ_BLOCK_STEP(mq_w4a16_grouped_gemm_ex(b.h, i32(L.down[0]), L.down[1], i32(L.down[2]), b.offsets, S, 0, E, E, H, I,
                                           L.group_size, b.y, d_status, stream));
  }
  MQ_BLOCK_STEP(mq_unpermute_combine_residual(b.y, L.dtype, b.weights, b.inv, residual, T, K, H, out, stream));
  if (h_launches) *h_launches = n + 3;
  return MQ_OK;
}
