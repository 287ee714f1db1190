// Routed mixture of experts over a packed token batch:
//   moe_route_kernel    fp32 router logits (+ bias) -> the `top` largest per token and the softmax over those alone   (per token)
//   moe_route_scores_kernel  scores = sigmoid(logits), or their softmax over all experts; experts picked by score (+ correction)
//                       inside the best expert groups, a group counting as its best expert or as the sum of its two best; weights =
//                       the picked experts' scores over their sum, times a scale, or the scores as they are              (per token)
//   moe_plan_kernel     tokens counted per expert, segment offsets, a slot for every (token, choice)                 (one CTA)
//   moe_gather_kernel   activation rows copied into slot order, so that an expert's rows are contiguous              (per slot)
//   moe_combine_kernel  y[t] = gate[t] shared[t] + sum_k weight[t, k] * expert_out[slot(t, k)], in the order of the choices   (per token)
// The experts themselves are two grouped GEMMs (b200p_gemm_grouped) over the segments.  Every launch has the same shape whatever
// the routing, so a decode step with experts sits in a captured graph.
#include "common.cuh"

namespace b200p {

bool pdl_enabled_gemm();
// Programmatic launches for decode batches of up to 64 tokens, where the gaps between these kernels are a tenth of the call (32 tokens, 16
// experts of 2048 x 2048: 129 -> 102 us with the shared expert's products beside the routed ones').  Prompts launch plainly (the gaps are a
// hundredth there), and moe_combine, which ends every mixture, always does: a stream that held nothing but programmatic launches of these kernels
// and the products did not come to its end under CUPTI's kernel tracing, for a reason that the kernels do not show (each waits for its predecessor,
// allows its successor only once it holds its TMEM, and every other wait is bounded), so no chain of mixtures or of
// plain dense products is one.
static bool moe_pdl(int64_t tokens) { return pdl_enabled_gemm() && tokens <= 64; }

constexpr int MOE_MAX_PER_LANE = 32;    // experts <= 1024
constexpr int MOE_MAX_TOP = 32;

// Choices that found nothing above -inf (logits that are NaN or -inf) hold E: they get the first experts that the token has not chosen, so that it
// never gives an expert two rows and no group grows beyond the batch.  Whole warps; lane k holds choice k.
__device__ __forceinline__ void moe_fill_choices(int lane, int E, int top, int& my_id) {
  if (!__any_sync(0xffffffffu, lane < top && my_id >= E)) return;
  for (int k = 0; k < top; ++k) {
    if (__shfl_sync(0xffffffffu, my_id, k) < E) continue;
    int e = 0;
    while (__any_sync(0xffffffffu, lane < top && my_id == e)) ++e;
    if (lane == k) my_id = e;
  }
}

// One warp's token: the choice k goes to lane k.  PER_LANE * 32 experts at most.
template <int PER_LANE>
__device__ __forceinline__ void moe_route_token(const float* __restrict__ logits, int64_t ldl, const float* __restrict__ bias, int64_t t, int E,
                                                int top, int lane, int& my_id, float& my_wt) {
  float z[PER_LANE];
#pragma unroll
  for (int i = 0; i < PER_LANE; ++i) {
    const int e = i * 32 + lane;
    z[i] = e < E ? logits[t * ldl + e] + (bias ? bias[e] : 0.f) : -INFINITY;
  }
  float first = 0.f, den = 0.f, mine = 0.f;
  my_id = 0;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int be = E;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (z[i] > best) { best = z[i]; be = i * 32 + lane; }          // ascending e within a lane: ties keep the smallest index
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ob > best || (ob == best && oe < be)) { best = ob; be = oe; }
    }
    if (k == 0) first = best;
    const float p = expf(best - first);                              // the first pick is the largest: exponents <= 0
    den += p;
    if (lane == k) { mine = p; my_id = be; }
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i)
      if (i * 32 + lane == be) z[i] = -INFINITY;
  }
  my_wt = mine / den;                                                // (a filled choice: 0, or NaN where no logit is a number)
  moe_fill_choices(lane, E, top, my_id);
}

template <int PER_LANE>
__global__ void moe_route_kernel(const float* logits, int64_t ldl, const float* bias,
                                 int32_t* __restrict__ ids, float* __restrict__ wts, int64_t M, int E, int top) {
  const int lane = threadIdx.x & 31;
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_launch_dependents();
  pdl_wait();
  if (t >= M) return;
  int id;
  float wt;
  moe_route_token<PER_LANE>(logits, ldl, bias, t, E, top, lane, id, wt);
  if (lane < top) {
    ids[t * top + lane] = id;
    wts[t * top + lane] = wt;
  }
}

// One warp per token.  s_e = sigmoid(z_e); picking score c_e = s_e + correction_e.  The experts form `count` groups of
// neighbours; a group's score is the sum of its two largest picking scores (its only one for groups of one expert), or (group_best)
// its largest; only the experts of the `keep` best groups can be picked (the others count as -inf, since picking scores may be
// negative).  The `top` largest picking scores win, ties to the smaller index; weights w_k = s_k / (sum of the picked s + 1e-20) *
// scale.  softmax: s = softmax(z) over ALL experts, picked (and groups compared) by z, which orders the experts as s does.
__global__ void moe_route_scores_kernel(const float* logits, int64_t ldl, const float* correction,
                                         int32_t* __restrict__ ids, float* __restrict__ wts, int64_t M, int E, int top, int count,
                                         int keep, float scale, int renorm, int softmax, int group_best) {
  extern __shared__ float mr_sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  pdl_launch_dependents();
  pdl_wait();
  if (t >= M) return;
  float* sc = mr_sm + (size_t)warp * (2 * E + count);     // scores
  float* pick = sc + E;                                    // picking scores, -inf once masked or taken
  float* gs = pick + E;                                    // group scores
  if (softmax) {                                           // scores = softmax over ALL experts; picked by the logits themselves
    float top1 = -INFINITY, sum = 0.f;
    for (int e = lane; e < E; e += 32) top1 = fmaxf(top1, logits[t * ldl + e]);
    top1 = warp_max(top1);
    for (int e = lane; e < E; e += 32) {
      const float z = logits[t * ldl + e], p = expf(z - top1);
      sum += p;
      sc[e] = p;
      pick[e] = z;
    }
    sum = warp_sum(sum);
    for (int e = lane; e < E; e += 32) sc[e] /= sum;
  } else {
    for (int e = lane; e < E; e += 32) {
      const float s = 1.f / (1.f + expf(-logits[t * ldl + e]));
      sc[e] = s;
      pick[e] = s + (correction ? correction[e] : 0.f);
    }
  }
  __syncwarp();
  if (count > 1 && keep < count) {
    const int per = E / count;
    for (int g = lane; g < count; g += 32) {
      float a = -INFINITY, b = -INFINITY;                  // the two largest of the group
      for (int i = 0; i < per; ++i) {
        const float v = pick[g * per + i];
        if (v > a) { b = a; a = v; }
        else if (v > b) b = v;
      }
      gs[g] = per > 1 && !group_best ? a + b : a;
    }
    __syncwarp();
    // drop the count - keep worst groups: repeatedly the smallest score, ties dropping the larger index first
    for (int r = 0; r < count - keep; ++r) {
      float worst = INFINITY;
      int wg = -1;
      for (int g = lane; g < count; g += 32) {
        const float v = gs[g];
        if (v == v && (v < worst || (v == worst && g > wg))) { worst = v; wg = g; }      // NaN marks a dropped group
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ow = __shfl_xor_sync(0xffffffffu, worst, o);
        const int og = __shfl_xor_sync(0xffffffffu, wg, o);
        if (og >= 0 && (wg < 0 || ow < worst || (ow == worst && og > wg))) { worst = ow; wg = og; }
      }
      if (lane == 0) gs[wg] = __int_as_float(0x7fc00000);
      for (int i = lane; i < per; i += 32) pick[wg * per + i] = -INFINITY;
      __syncwarp();
    }
  }
  float den = 0.f, mine = 0.f;
  int my_id = 0;
  for (int k = 0; k < top; ++k) {
    float best = -INFINITY;
    int be = E;
    for (int e = lane; e < E; e += 32)
      if (pick[e] > best) { best = pick[e]; be = e; }                  // ascending e within a lane: ties keep the smallest index
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ob > best || (ob == best && oe < be)) { best = ob; be = oe; }
    }
    const float s = be < E ? sc[be] : sc[0];                            // (E: scores that are NaN; otherwise keep * per >= top)
    den += s;
    if (lane == k) { mine = s; my_id = be; }
    __syncwarp();
    if (lane == 0 && be < E) pick[be] = -INFINITY;
    __syncwarp();
  }
  moe_fill_choices(lane, E, top, my_id);
  if (lane < top) {
    ids[t * top + lane] = my_id;
    wts[t * top + lane] = renorm ? mine / (den + 1e-20f) * scale : mine * scale;       // renorm 0: the scores as they are
  }
}

// Segments and slots of n chosen experts, one block.  id_of(i): the expert of (token, choice) i; cnt: [2 E] in shared memory.
template <typename F>
__device__ __forceinline__ void moe_plan(F id_of, int32_t* cnt, int32_t* __restrict__ seg, int32_t* __restrict__ slot_of,
                                         int32_t* __restrict__ token_of, int64_t n, int E, int top) {
  constexpr int B = 8;                           // reads in flight per thread
  int32_t* cur = cnt + E;
  for (int e = threadIdx.x; e < E; e += blockDim.x) cnt[e] = 0;
  __syncthreads();
  for (int64_t i0 = threadIdx.x; i0 < n; i0 += (int64_t)B * blockDim.x) {
    int id[B];
#pragma unroll
    for (int r = 0; r < B; ++r) id[r] = i0 + r * (int64_t)blockDim.x < n ? id_of(i0 + r * (int64_t)blockDim.x) : -1;
#pragma unroll
    for (int r = 0; r < B; ++r)
      if (id[r] >= 0) atomicAdd(&cnt[id[r]], 1);
  }
  __syncthreads();
  if (threadIdx.x < 32) {                        // running sum of the counts
    int32_t run = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + (int)threadIdx.x, mine = e < E ? cnt[e] : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if ((int)threadIdx.x >= o) sum += v;
      }
      if (e < E) seg[e] = cur[e] = run + sum - mine;
      run += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (threadIdx.x == 0) seg[E] = run;
  }
  __syncthreads();
  // the order of an expert's rows is whatever the atomics give: every row is computed on its own, so the values do not depend on it
  for (int64_t i0 = threadIdx.x; i0 < n; i0 += (int64_t)B * blockDim.x) {
    int id[B];
#pragma unroll
    for (int r = 0; r < B; ++r) id[r] = i0 + r * (int64_t)blockDim.x < n ? id_of(i0 + r * (int64_t)blockDim.x) : -1;
#pragma unroll
    for (int r = 0; r < B; ++r) {
      if (id[r] < 0) continue;
      const int64_t i = i0 + r * (int64_t)blockDim.x;
      const int32_t s = atomicAdd(&cur[id[r]], 1);
      slot_of[i] = s;
      token_of[s] = (int32_t)(i / top);
    }
  }
}

__global__ void moe_plan_kernel(const int32_t* ids, int32_t* __restrict__ seg, int32_t* __restrict__ slot_of,
                                int32_t* __restrict__ token_of, int64_t n, int E, int top) {
  extern __shared__ int32_t cnt[];               // [E] counts, then [E] cursors
  pdl_launch_dependents();
  pdl_wait();
  moe_plan([&](int64_t i) { return ids[i]; }, cnt, seg, slot_of, token_of, n, E, top);
}

// Decode batches: choice and plan in one block (a launch less; 32 tokens, 16 experts, 2 of them each).
constexpr int MOE_ONE_BLOCK = 64;                // (token, choice) pairs
template <int PER_LANE>
__global__ void __launch_bounds__(1024)
moe_route_plan_kernel(const float* logits, int64_t ldl, const float* bias, int32_t* __restrict__ ids,
                      float* __restrict__ wts, int32_t* __restrict__ seg, int32_t* __restrict__ slot_of, int32_t* __restrict__ token_of,
                      int64_t M, int E, int top) {
  extern __shared__ int32_t cnt[];               // [E] counts, then [E] cursors
  __shared__ int32_t chosen[MOE_ONE_BLOCK];
  const int lane = threadIdx.x & 31;
  pdl_launch_dependents();
  pdl_wait();
  for (int64_t t = threadIdx.x >> 5; t < M; t += blockDim.x >> 5) {
    int id;
    float wt;
    moe_route_token<PER_LANE>(logits, ldl, bias, t, E, top, lane, id, wt);
    if (lane < top) {
      ids[t * top + lane] = chosen[t * top + lane] = id;
      wts[t * top + lane] = wt;
    }
  }
  moe_plan([&](int64_t i) { return chosen[i]; }, cnt, seg, slot_of, token_of, M * top, E, top);      // (its first barrier covers `chosen`)
}

template <typename T>
__global__ void moe_gather_kernel(const T* x, const int32_t* token_of, T* __restrict__ xs, int64_t W) {
  const int64_t s = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const T* src = x + (int64_t)token_of[s] * W;
  T* dst = xs + s * W;
  if (W % 8 == 0 && sizeof(T) == 2) {
    const int64_t step = blockDim.x * 8;
    for (int64_t c = threadIdx.x * 8; c < W; c += 4 * step) {          // (four pieces in flight)
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c + k * step < W) v[k] = *reinterpret_cast<const uint4*>(src + c + k * step);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c + k * step < W) *reinterpret_cast<uint4*>(dst + c + k * step) = v[k];
    }
  } else {
    for (int64_t c = threadIdx.x; c < W; c += blockDim.x) dst[c] = src[c];
  }
}

// xs[slot_of[t, k], :] = wts[t, k] * x[t, :]: designs whose routing weight multiplies the expert's INPUT (the product is
// formed in fp32 and rounded once to the storage type)
template <typename T>
__global__ void moe_scatter_scaled_kernel(const T* x, const int32_t* slot_of, const float* wts,
                                          T* __restrict__ xs, int64_t W) {
  const int64_t i = blockIdx.x;                        // (token, choice)
  const int top = gridDim.y;
  pdl_launch_dependents();
  pdl_wait();
  const int64_t tk = i * top + blockIdx.y;
  const float w = wts[tk];
  const T* src = x + i * W;
  T* dst = xs + (int64_t)slot_of[tk] * W;
  if (sizeof(T) == 2 && W % 8 == 0) {                  // 16-byte pieces of eight 16-bit values (rows start on 16-byte boundaries)
    for (int64_t c = threadIdx.x * 8; c < W; c += blockDim.x * 8) {
      uint4 raw = *reinterpret_cast<const uint4*>(src + c);
      T* v = reinterpret_cast<T*>(&raw);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = Tr<T>::from_f(w * Tr<T>::to_f(v[i]));
      *reinterpret_cast<uint4*>(dst + c) = raw;
    }
    return;
  }
  for (int64_t c = threadIdx.x; c < W; c += blockDim.x) dst[c] = Tr<T>::from_f(w * Tr<T>::to_f(src[c]));
}

// V neighbouring channels per access (4: rows of whole 16-byte pieces)
template <int V>
__global__ void moe_combine_kernel(const float* __restrict__ ye, const int32_t* __restrict__ slot_of, const float* __restrict__ wts,
                                   const float* __restrict__ shared_y, const float* __restrict__ shared_gate, int64_t ldg,
                                   float* __restrict__ y, int64_t W, int top) {
  const int64_t t = blockIdx.x;
  const float sg = shared_gate ? 1.f / (1.f + expf(-shared_gate[t * ldg])) : 1.f;
  __shared__ int32_t sl[MOE_MAX_TOP];
  __shared__ float wt[MOE_MAX_TOP];
  if (threadIdx.x < top) {
    sl[threadIdx.x] = slot_of[t * top + threadIdx.x];
    wt[threadIdx.x] = wts ? wts[t * top + threadIdx.x] : 1.f;
  }
  __syncthreads();
  for (int64_t c = (int64_t)threadIdx.x * V; c < W; c += (int64_t)blockDim.x * V) {
    float a[V];
#pragma unroll
    for (int i = 0; i < V; ++i) a[i] = 0.f;
    auto add = [&](float w, const float* p) {
      if constexpr (V == 4) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        a[0] = fmaf(w, q.x, a[0]); a[1] = fmaf(w, q.y, a[1]); a[2] = fmaf(w, q.z, a[2]); a[3] = fmaf(w, q.w, a[3]);
      } else {
        a[0] = fmaf(w, p[0], a[0]);
      }
    };
#pragma unroll 4
    for (int k = 0; k < top; ++k) add(wt[k], ye + (int64_t)sl[k] * W + c);
    if (shared_y) add(sg, shared_y + t * W + c);
    if constexpr (V == 4) *reinterpret_cast<float4*>(y + t * W + c) = make_float4(a[0], a[1], a[2], a[3]);
    else y[t * W + c] = a[0];
  }
}

}  // namespace b200p

using namespace b200p;

// One block for as few choices as its 32 warps make beside each other.  us, one block / two launches: 16 experts, 2 choices, 16 and 32 tokens 3.0 /
// 3.65, 3.6 / 3.65, 4 choices of 32 tokens 4.4 / 3.9, 8 of 64 10 / 4.6; 128 experts, 4 choices of 16 tokens 4.2 / 4.3, of 32 5.3 / 4.3; above 128
// a lane has up to 32 logits: 129 experts, 6 choices of 4 tokens 6.4 / 6.8, 2 of 8 and 16 5.2 / 5.4, 6.1 / 5.4, 160 experts, 16 choices of 64 tokens
// 71 / 12.
static bool moe_one_block(int64_t M, int E, int top) {
  return E <= 128 ? M <= 32 && M * top <= MOE_ONE_BLOCK : M * top <= (M <= 4 ? 32 : 16);
}

static int moe_plan_launch(const int32_t* ids, int32_t* seg, int32_t* slot_of, int32_t* token_of, int64_t M, int E, int top, cudaStream_t st) {
  cudaError_t e = launch_pdl_opt(moe_pdl(M), moe_plan_kernel, dim3(1), dim3(1024), 2 * E * sizeof(int32_t), st, ids, seg, slot_of, token_of,
                                 M * top, E, top);
  if (e != cudaSuccess) return cuda_fail(e, "moe_plan_kernel launch");
  return B200P_OK;
}

extern "C" int b200p_moe_route(const float* logits, int64_t ldl, const float* bias, int32_t* ids, float* wts, int32_t* seg,
                               int32_t* slot_of, int32_t* token_of, int64_t M, int E, int top, void* stream) {
  B200P_REQUIRE(logits && ids && wts && seg && slot_of && token_of, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(E > 0 && E <= 32 * MOE_MAX_PER_LANE && top > 0 && top <= E && top <= MOE_MAX_TOP, B200P_ERR_ARG,
                "experts in [1, %d] and top in [1, min(experts, %d)]", 32 * MOE_MAX_PER_LANE, MOE_MAX_TOP);
  if (M == 0) return B200P_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const bool pdl = moe_pdl(M);
  cudaError_t e;
  if (moe_one_block(M, E, top)) {
    auto kern = E <= 32 ? moe_route_plan_kernel<1> : E <= 128 ? moe_route_plan_kernel<4> : moe_route_plan_kernel<MOE_MAX_PER_LANE>;
    e = launch_pdl_opt(pdl, kern, dim3(1), dim3(1024), 2 * E * sizeof(int32_t), st, logits, ldl, bias, ids, wts, seg, slot_of, token_of, M, E, top);
    if (e != cudaSuccess) return cuda_fail(e, "moe_route_plan_kernel launch");
    return B200P_OK;
  }
  auto kern = E <= 32 ? moe_route_kernel<1> : E <= 128 ? moe_route_kernel<4> : moe_route_kernel<MOE_MAX_PER_LANE>;
  e = launch_pdl_opt(pdl, kern, dim3((unsigned)((M + 3) / 4)), dim3(128), 0, st, logits, ldl, bias, ids, wts, M, E, top);
  if (e != cudaSuccess) return cuda_fail(e, "moe_route_kernel launch");
  return moe_plan_launch(ids, seg, slot_of, token_of, M, E, top, st);
}

extern "C" int b200p_moe_route_sigmoid(const float* logits, int64_t ldl, const float* correction, int32_t* ids, float* wts,
                                       int32_t* seg, int32_t* slot_of, int32_t* token_of, int64_t M, int E, int top, int count,
                                       int keep, float scale, void* stream) {
  B200P_REQUIRE(logits && ids && wts && seg && slot_of && token_of, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(E > 0 && E <= 32 * MOE_MAX_PER_LANE && top > 0 && top <= E && top <= MOE_MAX_TOP, B200P_ERR_ARG,
                "experts in [1, %d] and top in [1, min(experts, %d)]", 32 * MOE_MAX_PER_LANE, MOE_MAX_TOP);
  B200P_REQUIRE(count >= 1 && E % count == 0 && keep >= 1 && keep <= count && (int64_t)keep * (E / count) >= top, B200P_ERR_ARG,
                "expert groups: equal groups, 1 <= keep <= count, and the kept groups hold at least `top` experts");
  if (M == 0) return B200P_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int warps = 4;
  const size_t smem = (size_t)warps * (2 * E + count) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(moe_route_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(moe_route_scores_kernel)");
  }
  cudaError_t e = launch_pdl_opt(moe_pdl(M), moe_route_scores_kernel, dim3((unsigned)((M + warps - 1) / warps)), dim3(warps * 32), smem, st, logits,
                                 ldl, correction, ids, wts, M, E, top, count, keep, scale, 1, 0, 0);
  if (e != cudaSuccess) return cuda_fail(e, "moe_route_scores_kernel launch");
  return moe_plan_launch(ids, seg, slot_of, token_of, M, E, top, st);
}

extern "C" int b200p_moe_route_scores(const float* logits, int64_t ldl, int32_t* ids, float* wts, int32_t* seg, int32_t* slot_of,
                                      int32_t* token_of, int64_t M, int E, int top, int softmax, int count, int keep, int renorm,
                                      void* stream) {
  B200P_REQUIRE(logits && ids && wts && seg && slot_of && token_of, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(E > 0 && E <= 32 * MOE_MAX_PER_LANE && top > 0 && top <= E && top <= MOE_MAX_TOP, B200P_ERR_ARG,
                "experts in [1, %d] and top in [1, min(experts, %d)]", 32 * MOE_MAX_PER_LANE, MOE_MAX_TOP);
  B200P_REQUIRE(count >= 1 && E % count == 0 && keep >= 1 && keep <= count && (int64_t)keep * (E / count) >= top, B200P_ERR_ARG,
                "expert groups: equal groups, 1 <= keep <= count, and the kept groups hold at least `top` experts");
  if (M == 0) return B200P_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int warps = 4;
  const size_t smem = (size_t)warps * (2 * E + count) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(moe_route_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(moe_route_scores_kernel)");
  }
  cudaError_t e = launch_pdl_opt(moe_pdl(M), moe_route_scores_kernel, dim3((unsigned)((M + warps - 1) / warps)), dim3(warps * 32), smem, st, logits,
                                 ldl, nullptr, ids, wts, M, E, top, count, keep, 1.f, renorm, softmax, 1);
  if (e != cudaSuccess) return cuda_fail(e, "moe_route_scores_kernel launch");
  return moe_plan_launch(ids, seg, slot_of, token_of, M, E, top, st);
}

extern "C" int b200p_moe_scatter_scaled(const void* x, const int32_t* slot_of, const float* wts, void* xs, int64_t M, int64_t W, int top,
                                        int dtype, void* stream) {
  B200P_REQUIRE(x && slot_of && wts && xs && W > 0 && top > 0 && top <= MOE_MAX_TOP, B200P_ERR_ARG, "null pointer or bad top");
  B200P_REQUIRE(dtype == B200P_F32 || W % 8 != 0 || (aligned(x, 16) && aligned(xs, 16)), B200P_ERR_ALIGN, "x and xs must be 16-byte aligned");
  if (M == 0) return B200P_OK;
  cudaError_t e = cudaSuccess;
  B200P_DISPATCH_DTYPE(dtype, T, (e = launch_pdl_opt(moe_pdl(M), moe_scatter_scaled_kernel<T>, dim3((unsigned)M, (unsigned)top), dim3(128), 0,
                                                     (cudaStream_t)stream, (const T*)x, slot_of, wts, (T*)xs, W)));
  if (e != cudaSuccess) return cuda_fail(e, "moe_scatter_scaled_kernel launch");
  return B200P_OK;
}

static int moe_gather_call(const void* x, const int32_t* token_of, void* xs, int64_t slots, bool pdl, int64_t W, int dtype, void* stream) {
  B200P_REQUIRE(x && token_of && xs && W > 0, B200P_ERR_ARG, "null pointer");
  if (slots == 0) return B200P_OK;
  cudaError_t e = cudaSuccess;
  B200P_DISPATCH_DTYPE(dtype, T, (e = launch_pdl_opt(pdl, moe_gather_kernel<T>, dim3((unsigned)slots), dim3(128), 0, (cudaStream_t)stream,
                                                     (const T*)x, token_of, (T*)xs, W)));
  if (e != cudaSuccess) return cuda_fail(e, "moe_gather_kernel launch");
  return B200P_OK;
}

extern "C" int b200p_moe_gather(const void* x, const int32_t* token_of, void* xs, int64_t slots, int64_t W, int dtype, void* stream) {
  return moe_gather_call(x, token_of, xs, slots, false, W, dtype, stream);
}

extern "C" int b200p_moe_gather_tokens(const void* x, const int32_t* token_of, void* xs, int64_t M, int top, int64_t W, int dtype, void* stream) {
  B200P_REQUIRE(M >= 0 && top > 0 && top <= MOE_MAX_TOP, B200P_ERR_ARG, "bad token count or top");
  return moe_gather_call(x, token_of, xs, M * top, moe_pdl(M), W, dtype, stream);
}

extern "C" int b200p_moe_combine(const float* ye, const int32_t* slot_of, const float* wts, const float* shared_y,
                                 const float* shared_gate, int64_t ldg, float* y, int64_t M, int64_t W, int top, void* stream) {
  B200P_REQUIRE(ye && slot_of && y && W > 0 && top > 0 && top <= MOE_MAX_TOP, B200P_ERR_ARG, "null pointer or bad top");
  if (M == 0) return B200P_OK;
  const unsigned threads = W >= 1024 ? 256 : 128;
  auto kern = W % 4 == 0 && aligned(ye, 16) && aligned(shared_y, 16) && aligned(y, 16) ? moe_combine_kernel<4> : moe_combine_kernel<1>;
  kern<<<(unsigned)M, threads, 0, (cudaStream_t)stream>>>(ye, slot_of, wts, shared_y, shared_gate, ldg, y, W, top);
  B200P_LAUNCH_CHECK("moe_combine_kernel");
  return B200P_OK;
}
