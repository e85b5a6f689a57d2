// Routing bookkeeping of a quantized mixture-of-experts layer, on the device:
//   pe_moe_plan    (token, slot) pairs -> rows grouped by expert + the problem list of
//                  pe_gemv_grouped, in one launch and without a host round trip;
//   pe_moe_route_plan routing and plan of a decode-size batch;
//   pe_moe_combine weighted sum of the experts' outputs back into token order.
// The reference's layer does this with a Python loop over the selected experts
// (nemotron_offload.py:190-226).
#include "pe_common.cuh"

namespace pe {

constexpr int kPlanThreads = 1024;
constexpr int kPlanMaxExperts = 1024;
constexpr int kRouteMaxPerLane = 32;   // up to 1024 experts
constexpr int kRoutePlanPairs = 1024;  // (token, slot) pairs that the joint routing-and-plan block keeps in shared memory

// ---- routing: one token by one warp -------------------------------------------------------------------------------
// fp32 softmax over the experts, the top_k largest (ties go to the lower expert id, as a stable descending sort would
// have them).  Lane l holds experts l, l + 32, ... (PER_LANE of them: most layers have 128 or fewer, and registers
// for 1024 made every step of the selection eight times as long).  Returns the slot's weight and id in lanes < top_k.
template <int PER_LANE>
__device__ __forceinline__ void route_token(const void* logits, int dtype, int64_t row, int n_experts, int top_k, int renormalize, int lane,
                                            float& my_w, int& my_id) {
  float v[PER_LANE];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int e = lane + 32 * i;
    v[i] = e < n_experts ? load_as_float(logits, dtype, row + e) : -INFINITY;
  }
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) mx = fmaxf(mx, v[i]);
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    if (lane + 32 * i < n_experts) { v[i] = expf(v[i] - mx); sum += v[i]; }
    else v[i] = -1.f;  // never picked: probabilities are >= 0
  }
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
  const float inv = 1.f / sum;
  float kept = 0.f;
  my_w = 0.f;
  my_id = 0;
  for (int k = 0; k < top_k; ++k) {
    float best = -1.f;
    int best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (v[i] > best) { best = v[i]; best_e = lane + 32 * i; }  // lowest slot of this lane first
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, m);
      const int oe = __shfl_xor_sync(0xffffffffu, best_e, m);
      if (ob > best || (ob == best && oe < best_e)) { best = ob; best_e = oe; }
    }
    if ((best_e & 31) == lane) {
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i)
        if (i == (best_e >> 5)) v[i] = -1.f;
    }
    const float w = best * inv;
    kept += w;
    if (lane == k) { my_w = w; my_id = best_e; }  // top_k <= 32
  }
  if (renormalize) my_w /= kept;
}

template <int PER_LANE>
__global__ void __launch_bounds__(256) moe_route_kernel(const void* logits, int dtype, int64_t ld, int n_tokens, int n_experts, int top_k,
                                                        int renormalize, float* weights, int64_t* ids) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int tok = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (tok >= n_tokens) return;
  float w;
  int id;
  route_token<PER_LANE>(logits, dtype, (int64_t)tok * ld, n_experts, top_k, renormalize, lane, w, id);
  if (lane < top_k) {
    weights[(int64_t)tok * top_k + lane] = w;
    ids[(int64_t)tok * top_k + lane] = id;
  }
}

// ---- plan ----------------------------------------------------------------------------------------------------------
struct PlanArgs {
  const int64_t* expert_map; int n_global, n_pairs, top_k, n_local, rows_per_problem, max_problems;
  int32_t *row_token, *pos; int4* problems; int32_t* expert_rows;
};

// inclusive sum over the block's threads of two counts at once
__device__ __forceinline__ int2 block_scan2(int2 v, int2* warp_tot) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, v.x, o), y = __shfl_up_sync(0xffffffffu, v.y, o);
    if (lane >= o) { v.x += x; v.y += y; }
  }
  if (lane == 31) warp_tot[w] = v;
  __syncthreads();
  if (w == 0) {
    int2 t = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, t.x, o), y = __shfl_up_sync(0xffffffffu, t.y, o);
      if (lane >= o) { t.x += x; t.y += y; }
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  if (w > 0) { v.x += warp_tot[w - 1].x; v.y += warp_tot[w - 1].y; }
  return v;
}

// One block of kPlanThreads.  Pairs are bucketed by local expert with shared-memory counters; the order of
// the rows inside an expert depends on the arrival order of the atomics, which is harmless:
// every row of a grouped problem is computed independently of its neighbours, and the
// combine step finds a pair's row through `pos`.  expert_of(i): expert id of pair i as routed.
template <typename ExpertOf>
__device__ __forceinline__ void plan_body(const PlanArgs& p, ExpertOf expert_of) {
  __shared__ int cnt[kPlanMaxExperts];    // pairs per expert, then a running cursor
  __shared__ int first[kPlanMaxExperts];  // first row of the expert in the grouped order
  __shared__ int2 warp_tot[kPlanThreads / 32];
  const int tid = threadIdx.x;
  auto local_of = [&](int i) {
    int64_t e = expert_of(i);
    if (p.expert_map) e = (e >= 0 && e < p.n_global) ? p.expert_map[e] : -1;  // ids outside the map belong to nobody
    return e >= 0 && e < p.n_local ? (int)e : -1;
  };
  cnt[tid] = 0;
  __syncthreads();
  for (int i = tid; i < p.n_pairs; i += kPlanThreads) {
    const int e = local_of(i);
    if (e >= 0) atomicAdd(&cnt[e], 1);
  }
  __syncthreads();
  const int c = cnt[tid], probs = (c + p.rows_per_problem - 1) / p.rows_per_problem;
  const int2 upto = block_scan2(make_int2(c, probs), warp_tot);
  const int first_row = upto.x - c, first_prob = upto.y - probs, total_problems = warp_tot[kPlanThreads / 32 - 1].y;
  first[tid] = first_row;
  cnt[tid] = 0;  // now the cursor inside the expert
  // problem list: the expert of this thread owns problems first_prob ..; unused slots get zero rows
  if (tid < p.n_local) {
    if (p.expert_rows) { p.expert_rows[2 * tid] = first_row; p.expert_rows[2 * tid + 1] = c; }
    for (int j = 0; j < probs && first_prob + j < p.max_problems; ++j) {
      const int rows = c - j * p.rows_per_problem;
      p.problems[first_prob + j] = make_int4(tid, first_row + j * p.rows_per_problem, rows < p.rows_per_problem ? rows : p.rows_per_problem, 0);
    }
  }
  for (int i = total_problems + tid; i < p.max_problems; i += kPlanThreads) p.problems[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  for (int i = tid; i < p.n_pairs; i += kPlanThreads) {
    const int e = local_of(i);
    if (e >= 0) {
      const int r = first[e] + atomicAdd(&cnt[e], 1);
      p.row_token[r] = i / p.top_k;
      p.pos[i] = r;
    } else {
      p.pos[i] = -1;  // routed to an expert of another rank
    }
  }
}

__global__ void __launch_bounds__(kPlanThreads) moe_plan_kernel(const int64_t* ids, const PlanArgs p) {
  pdl_enter();
  plan_body(p, [&](int i) { return ids[i]; });
}

// Routing and plan of a decode-size batch in one block: a launch and a memory round trip less (one token of 128
// experts: 17 us for the two, 6 us now).
template <int PER_LANE>
__global__ void __launch_bounds__(kPlanThreads) moe_route_plan_kernel(const void* logits, int dtype, int64_t ld, int n_tokens, int n_experts, int renormalize,
                                                                      float* weights, int64_t* ids, const PlanArgs p) {
  __shared__ int picked[kRoutePlanPairs];
  pdl_enter();
  const int lane = threadIdx.x & 31;
  for (int tok = threadIdx.x >> 5; tok < n_tokens; tok += kPlanThreads / 32) {
    float w;
    int id;
    route_token<PER_LANE>(logits, dtype, (int64_t)tok * ld, n_experts, p.top_k, renormalize, lane, w, id);
    if (lane < p.top_k) {
      weights[(int64_t)tok * p.top_k + lane] = w;
      ids[(int64_t)tok * p.top_k + lane] = id;
      picked[tok * p.top_k + lane] = id;
    }
  }
  __syncthreads();
  plan_body(p, [&](int i) { return (int64_t)picked[i]; });
}

// out[t, :] = sum_j w[t, j] * y[pos[t * top_k + j], :] over the slots with pos >= 0, in slot
// order (bit-reproducible); 4 columns per thread.
__global__ void __launch_bounds__(256) moe_combine_kernel(const float* y, int64_t ld_y, const int32_t* pos, const float* w, int top_k,
                                                          void* out, int out_dtype, int64_t ld_out, int hidden, int64_t n_vec) {
  pdl_enter();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= n_vec) return;
  const int per_row = hidden >> 2;
  const int64_t t = idx / per_row;
  const int col = (int)(idx - t * per_row) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int U = 8;  // rows, weights and values of eight slots requested together
  for (int j0 = 0; j0 < top_k; j0 += U) {
    int r[U];
    float wt[U];
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool on = j0 + u < top_k;
      r[u] = on ? pos[t * top_k + j0 + u] : -1;
      wt[u] = on ? w[t * top_k + j0 + u] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = r[u] >= 0 ? *reinterpret_cast<const float4*>(y + (int64_t)r[u] * ld_y + col) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (r[u] >= 0) { acc.x += wt[u] * v[u].x; acc.y += wt[u] * v[u].y; acc.z += wt[u] * v[u].z; acc.w += wt[u] * v[u].w; }
  }
  if (out_dtype == PE_F16 && ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
    *reinterpret_cast<uint2*>(static_cast<__half*>(out) + t * ld_out + col) = make_uint2(pack_half2(acc.x, acc.y), pack_half2(acc.z, acc.w));
  } else {
    store_from_float(out, out_dtype, t * ld_out + col, acc.x);
    store_from_float(out, out_dtype, t * ld_out + col + 1, acc.y);
    store_from_float(out, out_dtype, t * ld_out + col + 2, acc.z);
    store_from_float(out, out_dtype, t * ld_out + col + 3, acc.w);
  }
}

}  // namespace pe

using namespace pe;

static int plan_args(PlanArgs& p, const int64_t* expert_map, int n_global_experts, int n_pairs, int top_k, int n_local_experts, int rows_per_problem,
                     int max_problems, int32_t* row_token, int32_t* pos, int32_t* problems, int32_t* expert_rows) {
  if (!row_token || !pos || !problems || n_pairs < 1 || top_k < 1 || max_problems < 1) return PE_ERR_ARG;
  if (rows_per_problem < 1 || rows_per_problem > 16) return PE_ERR_ARG;
  if (expert_map && n_global_experts < 1) return PE_ERR_ARG;
  if (n_local_experts < 1 || n_local_experts > kPlanMaxExperts) return PE_ERR_LIMIT;
  if (reinterpret_cast<uintptr_t>(problems) & 15) return PE_ERR_ALIGN;
  // every possible routing must fit: at most min(experts, pairs) partial problems plus pairs / rows full ones
  const int worst = (n_local_experts < n_pairs ? n_local_experts : n_pairs) + n_pairs / rows_per_problem;
  if (max_problems < worst) return PE_ERR_WORKSPACE;
  p = {expert_map, n_global_experts, n_pairs, top_k, n_local_experts, rows_per_problem, max_problems, row_token, pos,
       reinterpret_cast<int4*>(problems), expert_rows};
  return PE_OK;
}

extern "C" int pe_moe_plan(const int64_t* topk_ids, const int64_t* expert_map, int n_global_experts, int n_pairs, int top_k,
                           int n_local_experts,
                           int rows_per_problem, int max_problems, int32_t* row_token, int32_t* pos, int32_t* problems,
                           int32_t* expert_rows, void* stream) {
  if (!topk_ids) return PE_ERR_ARG;
  PlanArgs p;
  const int c = plan_args(p, expert_map, n_global_experts, n_pairs, top_k, n_local_experts, rows_per_problem, max_problems, row_token, pos, problems,
                          expert_rows);
  if (c != PE_OK) return c;
  PE_CUDA_TRY(launch_pdl(moe_plan_kernel, dim3(1), dim3(kPlanThreads), 0, static_cast<cudaStream_t>(stream), topk_ids, p));
  return PE_OK;
}

static int route_check(const void* logits, int dtype, int64_t ld_logits, int n_tokens, int n_experts, int top_k, const float* weights, const int64_t* ids) {
  if (!logits || !weights || !ids || n_tokens < 1) return PE_ERR_ARG;
  if (dtype < PE_F32 || dtype > PE_BF16 || ld_logits < n_experts) return PE_ERR_ARG;
  if (n_experts < 1 || n_experts > 32 * kRouteMaxPerLane || top_k < 1 || top_k > 32 || top_k > n_experts) return PE_ERR_LIMIT;
  return PE_OK;
}

extern "C" int pe_moe_route_plan(const void* logits, int dtype, int64_t ld_logits, int n_tokens, int n_experts, int top_k, int renormalize,
                                 float* weights, int64_t* ids, const int64_t* expert_map, int n_global_experts, int n_local_experts,
                                 int rows_per_problem, int max_problems, int32_t* row_token, int32_t* pos, int32_t* problems,
                                 int32_t* expert_rows, void* stream) {
  int c = route_check(logits, dtype, ld_logits, n_tokens, n_experts, top_k, weights, ids);
  if (c != PE_OK) return c;
  if ((int64_t)n_tokens * top_k > kRoutePlanPairs) return PE_ERR_LIMIT;
  PlanArgs p;
  c = plan_args(p, expert_map, n_global_experts, n_tokens * top_k, top_k, n_local_experts, rows_per_problem, max_problems, row_token, pos, problems,
                expert_rows);
  if (c != PE_OK) return c;
  auto kfn = n_experts <= 128 ? moe_route_plan_kernel<4> : n_experts <= 256 ? moe_route_plan_kernel<8> : moe_route_plan_kernel<32>;
  PE_CUDA_TRY(launch_pdl(kfn, dim3(1), dim3(kPlanThreads), 0, static_cast<cudaStream_t>(stream), logits, dtype, ld_logits, n_tokens, n_experts,
                         renormalize, weights, ids, p));
  return PE_OK;
}

extern "C" int pe_moe_combine(const float* y, int64_t ld_y, const int32_t* pos, const float* topk_weights, int tokens, int top_k,
                              void* out, int out_dtype, int64_t ld_out, int hidden, void* stream) {
  if (!y || !pos || !topk_weights || !out || tokens < 1 || top_k < 1 || hidden < 4) return PE_ERR_ARG;
  if (out_dtype < PE_F32 || out_dtype > PE_BF16) return PE_ERR_ARG;
  if (hidden % 4 || ld_y % 4 || ld_y < hidden || ld_out < hidden) return PE_ERR_SHAPE;
  if (reinterpret_cast<uintptr_t>(y) & 15) return PE_ERR_ALIGN;
  const int64_t n_vec = (int64_t)tokens * (hidden / 4);
  const int64_t blocks = (n_vec + 255) / 256;
  if (blocks > 0x7fffffff) return PE_ERR_LIMIT;
  PE_CUDA_TRY(launch_pdl(moe_combine_kernel, dim3((unsigned)blocks), dim3(256), 0, static_cast<cudaStream_t>(stream), y, ld_y, pos, topk_weights,
                         top_k, out, out_dtype, ld_out, hidden, n_vec));
  return PE_OK;
}

extern "C" int pe_moe_route(const void* logits, int dtype, int64_t ld_logits, int n_tokens, int n_experts, int top_k, int renormalize,
                            float* weights, int64_t* ids, void* stream) {
  const int c = route_check(logits, dtype, ld_logits, n_tokens, n_experts, top_k, weights, ids);
  if (c != PE_OK) return c;
  auto kfn = n_experts <= 128 ? moe_route_kernel<4> : n_experts <= 256 ? moe_route_kernel<8> : moe_route_kernel<32>;
  PE_CUDA_TRY(launch_pdl(kfn, dim3((unsigned)((n_tokens + 7) / 8)), dim3(256), 0, static_cast<cudaStream_t>(stream), logits, dtype, ld_logits,
                         n_tokens, n_experts, top_k, renormalize, weights, ids));
  return PE_OK;
}
