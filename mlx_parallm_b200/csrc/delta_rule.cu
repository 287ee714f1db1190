// Gated delta rule (a linear-attention layer with a per-head matrix state S [dk, dv] that is decayed, corrected towards the
// current value along the current key and read with the current query), as four kernels over a ragged batch:
//   delta_prep_kernel         short causal convolution + silu of q, k, v; unit q / k per head; beta and decay   (per token)
//   delta_conv_commit_kernel  the convolution's carried inputs                                                   (per entry)
//   delta_scan_kernel         the recurrence, fp32, token by token; decode steps: delta_step_kernel, long entries: delta_chunk_kernel  (per entry, head)
//   delta_out_kernel          per-head rms norm * weight * silu(gate)                                            (per token)
// The same kernels carry the variants other designs use: a decay per head AND key channel (a row of S each), a gate that is a
// sigmoid of a separate tensor, and the plain decayed accumulation S <- g S + k v^T (linear attention with a constant decay,
// fed by linear_attn_prep_kernel).
// Single tokens and entries of less than 32 run in one summation order, whatever kernel takes them; entries of 32 tokens and more (keys of 65 to 128
// channels, delta rule) 16 tokens at a time (delta_chunk_kernel), which differs in the last places, so a prompt and its portions agree to rounding.
// An entry's bits depend on its own tokens alone, with one exception: beside at least as many empty entries as it has tokens, in a call that
// does not say how long its longest entry is, it goes token by token (delta_step_kernel).
#include <type_traits>

#include "common.cuh"

namespace b200p {

int sm_count();
bool pdl_enabled_gemm();

// (a true quotient: __fdividef is 0 where the divisor is above 2^126, and float32 models round nothing away behind it)
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + __expf(-z)); }
// The same bits without the division's branch to its special cases (of all 2^32 arguments two differ by a unit, and some below 2^-100 in magnitude
// by a few subnormal ones): approximate reciprocal, then one step on the residual (Markstein, IBM J. Res. Dev. 34, 1990).  Both sides of the quotient
// carry a factor of 1/4, so that the reciprocal of the largest divisor is a normal number.  An infinite divisor or z has no residual (NaN); the
// first product is the result then: -0, infinity or NaN, as for the division.
__device__ __forceinline__ float silu_straight_f(float z) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
  const float d = fmaf(0.25f, e, 0.25f), n = 0.25f * z;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = n * r, rest = fmaf(-d, q, n);
  return rest == rest ? fmaf(rest, r, q) : q;
}
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

constexpr int DELTA_MAX_TAPS = 16;

template <int NT>
__global__ void __launch_bounds__(NT)
delta_prep_kernel(const float* __restrict__ proj, int64_t ldp, int64_t col_b, const float* __restrict__ a, int64_t lda, int dper,
                  const float* __restrict__ conv_w,
                  const float* __restrict__ conv_state, const float* __restrict__ A_log, const float* __restrict__ dt_bias,
                  const int32_t* __restrict__ t_row, const int32_t* __restrict__ t_pos, const int32_t* __restrict__ t_off,
                  float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vout, float* __restrict__ beta,
                  float* __restrict__ decay, int H, int KH, int dk, int dv, int taps) {
  extern __shared__ float qk[];                      // conv + silu of the q and k channels of this token
  const int64_t t = blockIdx.x;
  const int Cqk = 2 * KH * dk, C = Cqk + H * dv;
  const int row = t_row[t], pos = t_pos[t], off = t_off[t];
  const float* pt = proj + t * ldp;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < taps; ++j) {                 // tap j multiplies the input d = taps-1-j tokens back
      const int d = taps - 1 - j;
      float in;
      if (d > pos) in = 0.f;                         // before the sequence
      else if (d <= off) in = pt[c - (int64_t)d * ldp];
      else in = conv_state[((int64_t)row * (taps - 1) + (taps - 1 + off - d)) * C + c];
      acc = fmaf(conv_w[(int64_t)c * taps + j], in, acc);
    }
    const float a = silu_f(acc);
    if (c < Cqk) qk[c] = a;
    else vout[t * (int64_t)(H * dv) + (c - Cqk)] = a;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int hd = warp; hd < 2 * KH; hd += nw) {       // heads 0..KH-1 of q, then of k
    const float* src = qk + hd * dk;
    float ss = 0.f;
    for (int i = lane; i < dk; i += 32) ss = fmaf(src[i], src[i], ss);
    ss = warp_sum(ss);
    float inv = 1.f / sqrtf(ss + 1e-6f);
    float* dst;
    if (hd < KH) { inv *= 1.f / sqrtf((float)dk); dst = qn + t * (int64_t)(KH * dk) + hd * dk; }
    else dst = kn + t * (int64_t)(KH * dk) + (hd - KH) * dk;
    for (int i = lane; i < dk; i += 32) dst[i] = src[i] * inv;
  }
  for (int h = threadIdx.x; h < H; h += blockDim.x) beta[t * H + h] = 1.f / (1.f + expf(-pt[col_b + h]));
  // dper decays per head (1: the whole state of a head; dk: one per key channel), each with its own step input and bias
  const int nd = H * dper;
  const float* at = a + t * lda;
  for (int i = threadIdx.x; i < nd; i += blockDim.x)
    decay[t * (int64_t)nd + i] = expf(-expf(A_log[i / dper]) * softplus_f(at[i] + dt_bias[i]));
}

// The same for heads that are runs of 128 channels: a warp takes 128 channels (one q or k head, a piece of v, of the decays or
// of beta) through TT consecutive tokens, lane l the channels l, l + 32, l + 64, l + 96, and keeps the last TAPS - 1 inputs in
// registers, so the fp32 projection is read once instead of TAPS times.  Same operations in the same order per value as above: the
// results are bit for bit those of delta_prep_kernel.  Bound: instructions (two exponentials and a logarithm per decay, an exponential and a
// quotient per channel) and the latency of a warp's reads, which are asked for together; longer runs of tokens read the inputs before the first
// fewer times, shorter ones give a small call more warps.  16 + 16 heads of 128, us, decays per head / per channel, 1 (up to 128 tokens), 4 (to
// 512), 8 tokens at a time: 64 tokens 2.9 / 4.0, 496 8.3 / 13.0, 1664 22.7 / 40.5 (a block per token 10.5 / 11.1, the loop before, one token ahead,
// 9.7 / 15.2 and 26.6 / 50.1; with the quotient's special cases, four at a time, 29.7 / 44.3).
template <int TAPS, int TT>
__global__ void __launch_bounds__(128)
delta_prep_rows_kernel(const float* __restrict__ proj, int64_t ldp, int64_t col_b, const float* __restrict__ a, int64_t lda, int dper,
                       const float* __restrict__ conv_w, const float* __restrict__ conv_state, const float* __restrict__ A_log,
                       const float* __restrict__ dt_bias, const int32_t* __restrict__ t_row, const int32_t* __restrict__ t_pos,
                       const int32_t* __restrict__ t_off, float* __restrict__ qn, float* __restrict__ kn, float* __restrict__ vout,
                       float* __restrict__ beta, float* __restrict__ decay, int M, int H, int KH, int dv) {
  constexpr int DK = 128;
  const int lane = threadIdx.x & 31, unit = blockIdx.y * 4 + (threadIdx.x >> 5);
  const int t0 = blockIdx.x * TT, nt = min(TT, M - t0);
  const int nv = H * dv / 128, nd = H * dper, u_conv = 2 * KH + nv, u_dec = (nd + 127) / 128, u_beta = (H + 127) / 128;
  if (unit >= u_conv + u_dec + u_beta) return;
  if (unit >= u_conv) {                                       // decays, then betas: one value per token and entry
    const bool dec = unit < u_conv + u_dec;
    const int base = (dec ? unit - u_conv : unit - u_conv - u_dec) * 128 + lane, n = dec ? nd : H;
    const float* src = dec ? a : proj + col_b;
    const int64_t ld = dec ? lda : ldp;
#pragma unroll 1
    for (int c = base; c < n && c < base + 128; c += 32) {
      float x[TT];
#pragma unroll
      for (int i = 0; i < TT; ++i) x[i] = i < nt ? src[(int64_t)(t0 + i) * ld + c] : 0.f;
      const float ea = dec ? -expf(A_log[c / dper]) : 0.f, bias = dec ? dt_bias[c] : 0.f;
#pragma unroll
      for (int i = 0; i < TT; ++i) {
        if (i >= nt) break;
        if (dec) decay[(int64_t)(t0 + i) * nd + c] = expf(ea * softplus_f(x[i] + bias));
        else beta[(int64_t)(t0 + i) * H + c] = 1.f / (1.f + expf(-x[i]));
      }
    }
    return;
  }
  float in[TT][4];
  const int C = 2 * KH * DK + H * dv, c0 = unit * 128 + lane;
  int off[TT];
  const int row0 = t_row[t0], pos0 = t_pos[t0];
#pragma unroll
  for (int i = 0; i < TT; ++i) {
    off[i] = i < nt ? t_off[t0 + i] : 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) in[i][r] = i < nt ? proj[(int64_t)(t0 + i) * ldp + c0 + 32 * r] : 0.f;
  }
  float w[4][TAPS], win[4][TAPS];                             // win[r][j]: input of tap j
  const bool w16 = TAPS == 4 && (reinterpret_cast<uintptr_t>(conv_w) & 15) == 0;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (w16) {
      const float4 q = *reinterpret_cast<const float4*>(conv_w + (int64_t)(c0 + 32 * r) * TAPS);
      w[r][0] = q.x, w[r][1] = q.y, w[r][2] = q.z, w[r][3] = q.w;
    } else {
#pragma unroll
      for (int j = 0; j < TAPS; ++j) w[r][j] = conv_w[(int64_t)(c0 + 32 * r) * TAPS + j];
    }
  }
#pragma unroll
  for (int i = 0; i < TT; ++i) {
    if (i >= nt) break;
    const int t = t0 + i;
    if (i == 0 || off[i] == 0) {                              // the inputs before this token: of the portion, carried, or none
      const int row = i == 0 ? row0 : t_row[t], pos = i == 0 ? pos0 : t_pos[t];
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) {
        const int d = TAPS - 1 - j;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int c = c0 + 32 * r;
          float x = 0.f;
          if (d <= pos) x = d <= off[i] ? proj[(int64_t)(t - d) * ldp + c] : conv_state[((int64_t)row * (TAPS - 1) + (TAPS - 1 + off[i] - d)) * C + c];
          win[r][j] = x;
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int j = 0; j + 1 < TAPS; ++j) win[r][j] = win[r][j + 1];
    }
    float act[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      win[r][TAPS - 1] = in[i][r];
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < TAPS; ++j) acc = fmaf(w[r][j], win[r][j], acc);
      act[r] = silu_straight_f(acc);
    }
    if (unit >= 2 * KH) {
#pragma unroll
      for (int r = 0; r < 4; ++r) vout[(int64_t)t * (H * dv) + c0 + 32 * r - 2 * KH * DK] = act[r];
      continue;
    }
    float ss = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) ss = fmaf(act[r], act[r], ss);
    ss = warp_sum(ss);
    float inv = 1.f / sqrtf(ss + 1e-6f);
    float* dst;
    if (unit < KH) { inv *= 1.f / sqrtf((float)DK); dst = qn + (int64_t)t * (KH * DK) + c0; }
    else dst = kn + (int64_t)t * (KH * DK) + c0 - KH * DK;
#pragma unroll
    for (int r = 0; r < 4; ++r) dst[32 * r] = act[r] * inv;
  }
}

// Inputs of the plain decayed accumulation: q, k, v = silu of their projections (columns [0, Cqk), [Cqk, 2 Cqk), [2 Cqk, ..) of
// proj), and the constant per-head decay repeated for every token so that the scan reads it like a computed one.
__global__ void linear_attn_prep_kernel(const float* __restrict__ proj, int64_t ldp, const float* __restrict__ head_decay,
                                        float* __restrict__ q, float* __restrict__ k, float* __restrict__ v,
                                        float* __restrict__ decay, int H, int Cqk, int Cv) {
  const int64_t t = blockIdx.x;
  const float* pt = proj + t * ldp;
  for (int c = threadIdx.x; c < 2 * Cqk + Cv; c += blockDim.x) {
    const float a = silu_f(pt[c]);
    if (c < Cqk) q[t * Cqk + c] = a;
    else if (c < 2 * Cqk) k[t * Cqk + (c - Cqk)] = a;
    else v[t * (int64_t)Cv + (c - 2 * Cqk)] = a;
  }
  for (int h = threadIdx.x; h < H; h += blockDim.x) decay[t * H + h] = head_decay[h];
}

__global__ void delta_conv_commit_kernel(const float* __restrict__ proj, int64_t ldp, float* __restrict__ conv_state,
                                         const int32_t* __restrict__ cu, const int32_t* __restrict__ rows, int64_t C, int taps) {
  const int e = blockIdx.y;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int n = cu[e + 1] - cu[e];
  if (c >= C || n <= 0) return;
  float* st = conv_state + (int64_t)rows[e] * (taps - 1) * C + c;
  float keep[DELTA_MAX_TAPS];
#pragma unroll
  for (int i = 0; i < DELTA_MAX_TAPS; ++i) {
    if (i < taps - 1) {
      const int rel = n - (taps - 1) + i;            // input i of the new state, counted from the portion's first token
      keep[i] = rel >= 0 ? proj[((int64_t)cu[e] + rel) * ldp + c] : st[(int64_t)(i + n) * C];
    }
  }
#pragma unroll
  for (int i = 0; i < DELTA_MAX_TAPS; ++i)
    if (i < taps - 1) st[(int64_t)i * C] = keep[i];
}

// Rows of a state column are summed in segments: four interleaved partial sums each (rows i mod 4), combined in a fixed order, then the
// segments pairwise.  The kernels that go token by token, however many lanes they give to a column, add in this one order, so a token's numbers do
// not depend on whether it arrives in a short prompt or alone or on the size of the batch.
constexpr int ds_segs(int dkp) { return dkp <= 64 ? 4 : dkp <= 128 ? 8 : dkp / 32; }

// Sums of x and of y over the LANES lanes of a slot: even lanes get the sum of x, odd lanes that of y.
template <int LANES>
__device__ __forceinline__ float ds_reduce(float x, float y, bool odd) {
  const float give = odd ? x : y;
  float r = (odd ? y : x) + __shfl_xor_sync(0xffffffffu, give, 1);
#pragma unroll
  for (int m = 2; m < LANES; m <<= 1) r += __shfl_xor_sync(0xffffffffu, r, m);
  return r;
}

// the same for two pairs at once (two chains of exchanges that cover each other)
template <int LANES>
__device__ __forceinline__ float2 ds_reduce2(float x0, float y0, float x1, float y1, bool odd) {
  const float g0 = odd ? x0 : y0, g1 = odd ? x1 : y1;
  float r0 = __shfl_xor_sync(0xffffffffu, g0, 1), r1 = __shfl_xor_sync(0xffffffffu, g1, 1);
  r0 += odd ? y0 : x0;
  r1 += odd ? y1 : x1;
#pragma unroll
  for (int m = 2; m < LANES; m <<= 1) {
    const float a = __shfl_xor_sync(0xffffffffu, r0, m), b = __shfl_xor_sync(0xffffffffu, r1, m);
    r0 += a;
    r1 += b;
  }
  return make_float2(r0, r1);
}

// A thread's SUB segments of SEG rows of two state columns, rows 2 i (.x) and 2 i + 1 (.y) packed: the packed fp32 instructions of sm_100
// (FMUL2 / FFMA2: both halves rounded like the scalar operation) take two ROWS of a column at once, so that keys, queries and decays are
// operands as they are read (pairs of columns would need every one of them twice in a register pair).
// MODE 0: delta rule, one decay per head and token; 1: delta rule, one decay per head, key channel and token (decay
// [M, H, dk]); 2: no correction, S <- g S + k v^T (one decay per head and token; beta unused).
template <int SEG, int SUB> struct DsCols { float2 c0[SUB][SEG / 2], c1[SUB][SEG / 2]; };

// scale by the decays and, for the delta rule, dot with the key: the thread's share of both sums
template <int SEG, int SUB, int MODE>
__device__ __forceinline__ float2 ds_decay_dot(DsCols<SEG, SUB>& S, const float* kp, const float* gp, float g, float2 (&kr)[SUB][SEG / 2]) {
  float x[SUB], y[SUB];
#pragma unroll
  for (int u = 0; u < SUB; ++u) {
    float2 d0[2], d1[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) d0[a] = d1[a] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < SEG / 2; i += 2) {
      const float4 k4 = *reinterpret_cast<const float4*>(kp + u * (SEG + 4) + 2 * i);
      kr[u][i] = make_float2(k4.x, k4.y);
      kr[u][i + 1] = make_float2(k4.z, k4.w);
      float2 gg[2] = {make_float2(g, g), make_float2(g, g)};
      if constexpr (MODE == 1) {
        const float4 g4 = *reinterpret_cast<const float4*>(gp + u * (SEG + 4) + 2 * i);
        gg[0] = make_float2(g4.x, g4.y), gg[1] = make_float2(g4.z, g4.w);
      }
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        S.c0[u][i + a] = __fmul2_rn(S.c0[u][i + a], gg[a]);
        S.c1[u][i + a] = __fmul2_rn(S.c1[u][i + a], gg[a]);
        if constexpr (MODE != 2) {
          d0[a] = __ffma2_rn(S.c0[u][i + a], kr[u][i + a], d0[a]);
          d1[a] = __ffma2_rn(S.c1[u][i + a], kr[u][i + a], d1[a]);
        }
      }
    }
    x[u] = (d0[0].x + d0[0].y) + (d0[1].x + d0[1].y);
    y[u] = (d1[0].x + d1[0].y) + (d1[1].x + d1[1].y);
  }
  if constexpr (SUB == 2) return make_float2(x[0] + x[1], y[0] + y[1]);
  return make_float2(x[0], y[0]);
}

// add key times (ux, uy) and dot with the query: the thread's share of both outputs
template <int SEG, int SUB>
__device__ __forceinline__ float2 ds_update_dot(DsCols<SEG, SUB>& S, const float* qp, const float2 (&kr)[SUB][SEG / 2], float ux, float uy) {
  const float2 ux2 = make_float2(ux, ux), uy2 = make_float2(uy, uy);
  float x[SUB], y[SUB];
#pragma unroll
  for (int u = 0; u < SUB; ++u) {
    float2 p0[2], p1[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) p0[a] = p1[a] = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < SEG / 2; i += 2) {
      const float4 q4 = *reinterpret_cast<const float4*>(qp + u * (SEG + 4) + 2 * i);
      const float2 qq[2] = {make_float2(q4.x, q4.y), make_float2(q4.z, q4.w)};
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        S.c0[u][i + a] = __ffma2_rn(kr[u][i + a], ux2, S.c0[u][i + a]);
        S.c1[u][i + a] = __ffma2_rn(kr[u][i + a], uy2, S.c1[u][i + a]);
        p0[a] = __ffma2_rn(S.c0[u][i + a], qq[a], p0[a]);
        p1[a] = __ffma2_rn(S.c1[u][i + a], qq[a], p1[a]);
      }
    }
    x[u] = (p0[0].x + p0[0].y) + (p0[1].x + p0[1].y);
    y[u] = (p1[0].x + p1[0].y) + (p1[1].x + p1[1].y);
  }
  if constexpr (SUB == 2) return make_float2(x[0] + x[1], y[0] + y[1]);
  return make_float2(x[0], y[0]);
}

// Prompts, dk padded to DKP = 32 ... 512.  LANES lanes share a column slot of two state columns: every q / k element read from shared
// memory serves two columns.  The chain of a token (scale and dot with k, reduce over the lanes, update) is what bounds one CTA per SM, so
// each link is kept short: 16 rows per lane at 128-row states (eight lanes) and two warps per scheduler that cover each other's latencies;
// a reduction in which the two lanes of a pair first swap, so that one carries column j0 and the other j1 (1 + log2(lanes) exchanges for
// two sums instead of 2 log2(lanes)); outputs whose exchanges run beside those of the next token; whole chunks as straight-line code.
// 4 sequences of 512 tokens, 16 heads of 128 x 128, decays per channel: 0.42 us per token.  Where there are more CTAs than SMs the
// instructions and the state traffic bound it instead, and four lanes of 32 rows, which exchange and read half as often, are faster
// (delta_scan_launch).  q and k of CHUNK tokens are staged in shared memory with every segment padded by 16 bytes, so the lanes' 128-bit
// reads fall into different banks.
constexpr int ds_slots(int dkp) { return dkp <= 128 ? 32 : 4096 / dkp; }       // column slots per CTA, of two state columns each
template <int DKP, int MODE, int LANES, int PER_SM>
__global__ void __launch_bounds__(LANES * ds_slots(DKP), PER_SM)
delta_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ v,
                  const float* __restrict__ beta, const float* __restrict__ decay, float* __restrict__ state,
                  const int32_t* __restrict__ cu, const int32_t* __restrict__ rows, const int32_t* __restrict__ lengths,
                  float* __restrict__ o, int H, int KH, int dk, int dv, int most) {
  constexpr int SEGS = ds_segs(DKP), SUB = SEGS / LANES, SEG = DKP / SEGS;
  constexpr int DS_SLOTS = ds_slots(DKP), DS_COLS = 2 * DS_SLOTS, DS_THREADS = LANES * DS_SLOTS;
  constexpr int CHUNK = DKP <= 128 ? 8 : 1024 / DKP;             // tokens staged at a time
  // a thread's columns: half a CTA's width apart, or neighbours in one 8-byte access (few slots per warp: 4 x 64 tokens, 8 heads of
  // 256 x 256: 54 -> 50 us; at 128 rows the same change costs 10 % of a short scan)
  constexpr int NEXT = DKP <= 128 ? DS_SLOTS : 1, MUL = DKP <= 128 ? 1 : 2;
  constexpr int LDK = DKP + 4 * SEGS;                            // padded row of the staging buffers
  constexpr int PF = CHUNK * DKP / DS_THREADS;                   // q / k elements each thread stages per chunk
  constexpr int PV = (CHUNK * DS_COLS + DS_THREADS - 1) / DS_THREADS;
  __shared__ __align__(16) float ks[2][CHUNK][LDK], qs[2][CHUNK][LDK];
  __shared__ __align__(16) float gc[MODE == 1 ? 2 : 1][MODE == 1 ? CHUNK : 1][MODE == 1 ? LDK : 4];     // per-channel decays
  __shared__ float vs[2][CHUNK][DS_COLS], gs[2][CHUNK], bs[2][CHUNK];
  const int e = blockIdx.x, h = blockIdx.y;
  const int l = threadIdx.x & (LANES - 1), slot = threadIdx.x / LANES;
  const int c0 = MUL * slot, j0 = blockIdx.z * DS_COLS + c0, j1 = j0 + NEXT;     // this thread's two state columns
  const bool pairs = NEXT == 1 && (dv & 1) == 0 && (reinterpret_cast<uintptr_t>(state) & 7) == 0;
  const bool live0 = j0 < dv, live1 = j1 < dv, odd = (l & 1) != 0;
  const int t0 = cu[e], t1 = cu[e + 1];
  const bool waits = (blockIdx.x | blockIdx.y | blockIdx.z) == 0;        // (see delta_scan_launch: the grid ends no earlier than the launch before)
  if (t1 <= t0 || t1 - t0 > most) {                              // (longer entries: delta_chunk_kernel)
    if (waits) pdl_wait();
    return;
  }
  const int row = rows[e];
  const int kh = h / (H / KH);
  const int r0 = l * SUB * SEG, l0 = l * SUB * (SEG + 4);        // first row of the lane, and where it lies in the staging buffers
  DsCols<SEG, SUB> S;
  float* sp = state + (((int64_t)row * H + h) * dk + r0) * dv;
  const bool fresh = lengths[row] == 0;                          // first token of a sequence: the state starts at zero
#pragma unroll
  for (int u = 0; u < SUB; ++u)
#pragma unroll
    for (int i = 0; i < SEG / 2; ++i) {
      const int r = u * SEG + 2 * i;
      const bool in0 = !fresh && r0 + r < dk, in1 = !fresh && r0 + r + 1 < dk;
      const float* s0 = sp + (int64_t)r * dv;
      if (NEXT == 1 && pairs) {
        float2 a = make_float2(0.f, 0.f), b = a;
        if (in0 && live0) a = *reinterpret_cast<const float2*>(s0 + j0);
        if (in1 && live0) b = *reinterpret_cast<const float2*>(s0 + dv + j0);
        S.c0[u][i] = make_float2(a.x, b.x);
        S.c1[u][i] = make_float2(a.y, b.y);
        continue;
      }
      S.c0[u][i] = make_float2(in0 && live0 ? s0[j0] : 0.f, in1 && live0 ? s0[dv + j0] : 0.f);
      S.c1[u][i] = make_float2(in0 && live1 ? s0[j1] : 0.f, in1 && live1 ? s0[dv + j1] : 0.f);
    }
  // The next chunk's inputs are fetched into registers while the current chunk runs out of shared memory, then parked in the
  // other buffer: the recurrence never waits for global memory.
  float pk[PF], pq[PF], pv[PV], pg = 0.f, pb = 0.f;
  float pgc[MODE == 1 ? PF : 1];
  auto fetch = [&](int tc) {
    const int nt = min(CHUNK, t1 - tc);
#pragma unroll
    for (int r = 0; r < PF; ++r) {
      const int idx = threadIdx.x + r * DS_THREADS, tt = idx / DKP, i = idx % DKP;
      const bool ok = tt < nt && i < dk;
      const int64_t src = ((int64_t)(tc + tt) * KH + kh) * dk + i;
      pk[r] = ok ? kn[src] : 0.f;
      pq[r] = ok ? qn[src] : 0.f;
      if constexpr (MODE == 1) pgc[r] = ok ? decay[((int64_t)(tc + tt) * H + h) * dk + i] : 1.f;
    }
#pragma unroll
    for (int r = 0; r < PV; ++r) {
      const int idx = threadIdx.x + r * DS_THREADS, tt = idx / DS_COLS, c = blockIdx.z * DS_COLS + idx % DS_COLS;
      pv[r] = (tt < nt && c < dv) ? v[((int64_t)(tc + tt) * H + h) * dv + c] : 0.f;
    }
    if (threadIdx.x < nt) {
      if constexpr (MODE != 1) pg = decay[(int64_t)(tc + threadIdx.x) * H + h];
      if constexpr (MODE != 2) pb = beta[(int64_t)(tc + threadIdx.x) * H + h];
    }
  };
  auto park = [&](int buf) {
#pragma unroll
    for (int r = 0; r < PF; ++r) {
      const int idx = threadIdx.x + r * DS_THREADS, tt = idx / DKP, i = idx % DKP;
      ks[buf][tt][i + (i / SEG) * 4] = pk[r];
      qs[buf][tt][i + (i / SEG) * 4] = pq[r];
      if constexpr (MODE == 1) gc[buf][tt][i + (i / SEG) * 4] = pgc[r];
    }
#pragma unroll
    for (int r = 0; r < PV; ++r) {
      const int idx = threadIdx.x + r * DS_THREADS;
      if (idx < CHUNK * DS_COLS) vs[buf][idx / DS_COLS][idx % DS_COLS] = pv[r];
    }
    if (threadIdx.x < CHUNK) { gs[buf][threadIdx.x] = pg; bs[buf][threadIdx.x] = pb; }
  };
  // a token's output leaves one token later: its exchanges run beside those of the next token's dot product
  float2 out = make_float2(0.f, 0.f);
  auto put = [&](int tok, float val) {
    if (l < 2 && tok >= t0 && (odd ? live1 : live0)) o[((int64_t)tok * H + h) * dv + (odd ? j1 : j0)] = val;
  };
  fetch(t0);
  park(0);
  __syncthreads();
  int buf = 0;
  for (int tc = t0; tc < t1; tc += CHUNK, buf ^= 1) {
    const int nt = min(CHUNK, t1 - tc);
    const bool more = tc + CHUNK < t1;
    if (more) fetch(tc + CHUNK);
    auto step = [&](int tt) {
      const float v1 = vs[buf][tt][c0 + (odd ? NEXT : 0)];      // of the column this lane sums up
      float2 kr[SUB][SEG / 2];                                   // the keys stay in registers for the update
      const float2 d = ds_decay_dot<SEG, SUB, MODE>(S, &ks[buf][tt][l0], MODE == 1 ? &gc[buf][tt][l0] : nullptr, gs[buf][tt], kr);
      float u1 = v1;
      if constexpr (MODE != 2) {
        const float2 r = ds_reduce2<LANES>(d.x, d.y, out.x, out.y, odd);
        u1 = bs[buf][tt] * (v1 - r.x);
        put(tc + tt - 1, r.y);
      } else {
        put(tc + tt - 1, ds_reduce<LANES>(out.x, out.y, odd));
      }
      const float u_other = __shfl_xor_sync(0xffffffffu, u1, 1);
      out = ds_update_dot<SEG, SUB>(S, &qs[buf][tt][l0], kr, odd ? u_other : u1, odd ? u1 : u_other);
    };
    if (nt == CHUNK) {                // straight-line: the next token's operands are read while this one's sums are exchanged
#pragma unroll
      for (int tt = 0; tt < CHUNK; ++tt) step(tt);
    } else {
      for (int tt = 0; tt < nt; ++tt) step(tt);
    }
    if (more) park(buf ^ 1);          // the other buffer was last read in the previous iteration, before its closing barrier
    __syncthreads();
  }
  put(t1 - 1, ds_reduce<LANES>(out.x, out.y, odd));
#pragma unroll
  for (int u = 0; u < SUB; ++u)
#pragma unroll
    for (int i = 0; i < SEG / 2; ++i) {
      const int r = u * SEG + 2 * i;
      float* s0 = sp + (int64_t)r * dv;
      if (NEXT == 1 && pairs) {
        if (r0 + r < dk && live0) *reinterpret_cast<float2*>(s0 + j0) = make_float2(S.c0[u][i].x, S.c1[u][i].x);
        if (r0 + r + 1 < dk && live0) *reinterpret_cast<float2*>(s0 + dv + j0) = make_float2(S.c0[u][i].y, S.c1[u][i].y);
        continue;
      }
      if (r0 + r < dk) {
        if (live0) s0[j0] = S.c0[u][i].x;
        if (live1) s0[j1] = S.c1[u][i].x;
      }
      if (r0 + r + 1 < dk) {
        if (live0) s0[dv + j0] = S.c0[u][i].y;
        if (live1) s0[dv + j1] = S.c1[u][i].y;
      }
    }
  if (waits) pdl_wait();
}

// Prompts of keys of 65 to 128 channels, 16 tokens (a chunk) at a time, the products on the tensor cores.  With G_t the product of the decays of the
// chunk's tokens up to t and S the state before it,
//     X_t = v_t - S^T (G_t k_t)          A_tj = k_t . (G_t / G_j) k_j  (j < t)       P_tj = q_t . (G_t / G_j) k_j  (j <= t)
//     U = T X,  T = (I + diag(b) A)^-1 diag(b)       O = S^T (G_t q_t) + P U         S <- G S + sum_j (G / G_j) k_j u_j
// so the chain from state to state is two products per 16 tokens instead of two dot products per token, and T and P, which need no state, are made
// beforehand for all chunks at once (delta_triangle_kernel).  Every quotient of decays is a product of the decays in between: never above one, no
// division.
//
// All of it keeps fp32's accuracy.  An operand is the sum of three bf16 numbers, which hold all of its 24 bits, a product six MMAs (what is left out is below
// 2^-25 of it); the MMAs cut their sums off instead of rounding them, so the leading products of 16 channels, which hardly lose a bit, meet the others in
// rounding additions.  What a token's output hangs on most, its own value and its own key and query, passes no MMA: the diagonals of both triangles
// (b_t of U = X + (T - I) X with X = diag(b) (...), and P_tt) are fp32 FMAs.  Relative error of o / the state against 64 bits, 128 x 128, decays per
// channel, two tokens at a time in fp32 (the kernel before) -> so: decays as a layer has them, 512 tokens 7.9e-8 / 7.8e-8 -> 7.9e-8 / 7.7e-8, 600 tokens 7.9e-8 /
// 8.3e-8 -> 7.9e-8 / 7.4e-8, 33 to 100 tokens 8.7e-8 / 8.5e-8 -> 8.4e-8 / 7.6e-8; of 0.98 to 1, 512 tokens 1.6e-7 / 2.2e-7 -> 1.2e-7 / 1.4e-7; of 0.9996 to 1
// 3.5e-7 / 5.2e-7 -> 2.0e-7 / 2.7e-7.  Two tf32 numbers an operand and three MMAs a product take 12 % less time and have twice the error with a layer's
// decays (1.6e-7 / 1.5e-7): an operand then loses the last of its bits.
constexpr int DC_MIN = 32, DC_CHUNK = 16, DC_COLS = 64, DC_TEAM = 128;
constexpr int DC_MIN_DV = DC_CHUNK + 1;                        // a chunk of m tokens keeps T and P, m (m + 1) numbers, in its m rows of o until o is written

// k = 16: A [16, 16], B [16, 8]; k = 8: the first halves of both
__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], uint2 b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}
__device__ __forceinline__ void dc_mma0(float (&d)[4], const uint32_t (&a)[4], uint2 b) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y), "f"(0.f));
}
__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(b));
}
__device__ __forceinline__ void dc_mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(b), "f"(0.f));
}
// x and y (low and high halves of a word) as sums of three bf16 numbers: the nearest one, then the leading 8 bits of what is left, then the rest, which
// has 8 bits: nothing is lost
__device__ __forceinline__ void dc_split(float x, float y, uint32_t& w0, uint32_t& w1, uint32_t& w2) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w0) : "f"(y), "f"(x));
  const float rx = x - __uint_as_float(w0 << 16), ry = y - __uint_as_float(w0 & 0xffff0000u);
  w1 = __byte_perm(__float_as_uint(rx), __float_as_uint(ry), 0x7632);
  const float sx = rx - __uint_as_float(__float_as_uint(rx) & 0xffff0000u), sy = ry - __uint_as_float(__float_as_uint(ry) & 0xffff0000u);
  w2 = __byte_perm(__float_as_uint(sx), __float_as_uint(sy), 0x7632);
}
// two accumulators side by side (16 rows, 8 + 8 columns) as an A operand: their layouts are the same
__device__ __forceinline__ void dc_operand(const float (&c)[4], const float (&d)[4], uint32_t (&a)[3][4]) {
  dc_split(c[0], c[1], a[0][0], a[1][0], a[2][0]);
  dc_split(c[2], c[3], a[0][1], a[1][1], a[2][1]);
  dc_split(d[0], d[1], a[0][2], a[1][2], a[2][2]);
  dc_split(d[2], d[3], a[0][3], a[1][3], a[2][3]);
}
// the five products below the leading one: 2^-16 of it, then 2^-8
template <typename B, typename F>
__device__ __forceinline__ void dc_low_terms(const uint32_t (&a)[3][4], const B (&b)[3], F&& mma) {
  mma(a[2], b[0]);
  mma(a[0], b[2]);
  mma(a[1], b[1]);
  mma(a[1], b[0]);
  mma(a[0], b[1]);
}

// Columns of a head are dealt to the slices evenly, the first ones one more: never above DC_COLS (slices = columns / DC_COLS, rounded up), and two slices
// or more have at least DC_COLS / 2 each.  (A remainder of its own in the last slice could be narrower than DC_MIN_DV: 3088 columns in 49 slices of 63, 64.)
struct DcSlice { int z0, n; };
__device__ __forceinline__ DcSlice dc_slice(int dv, int slices, int z) {
  const int base = dv / slices, more = dv % slices;
  return {z * base + min(z, more), base + (z < more ? 1 : 0)};
}

// channel d of a chunk's keys, queries and decays; tokens past the end are ones that change nothing
template <int MODE>
__device__ __forceinline__ void dc_fetch(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ decay, int tc, int t1, int h, int kh,
                                         int d, int H, int KH, int dk, float (&k)[DC_CHUNK], float (&q)[DC_CHUNK], float (&gg)[DC_CHUNK]) {
  const float* ks = kn + ((int64_t)tc * KH + kh) * dk + d;
  const float* qs = qn + ((int64_t)tc * KH + kh) * dk + d;
  const float* gs = MODE == 1 ? decay + ((int64_t)tc * H + h) * dk + d : decay + (int64_t)tc * H + h;
  const int64_t k_step = (int64_t)KH * dk, g_step = MODE == 1 ? (int64_t)H * dk : H;
  if (tc + DC_CHUNK <= t1 && dk == 128) {
#pragma unroll
    for (int i = 0; i < DC_CHUNK; ++i) k[i] = ks[i * k_step], q[i] = qs[i * k_step], gg[i] = gs[i * g_step];
  } else {
#pragma unroll
    for (int i = 0; i < DC_CHUNK; ++i) {
      const bool in = tc + i < t1, ok = in && d < dk;
      k[i] = ok ? ks[i * k_step] : 0.f;
      q[i] = ok ? qs[i * k_step] : 0.f;
      gg[i] = (MODE == 1 ? ok : in) ? gs[i * g_step] : 1.f;
    }
  }
}

// T and P of every chunk of the entries of DC_MIN tokens and more, a CTA each, a thread per key channel: left in the chunk's rows of o, one copy per
// slice of columns, row by row (T's part, then P's).  A and P of two tokens in different halves of the chunk, or different quarters of a half, are a
// product of rows scaled from the border on and of rows scaled up to it (12 MMAs per warp); those of one quarter are summed over the channels directly.
// Bound: instructions (5500 per chunk and head, issue slots half used) and the latency of a CTA's reads: 104 chunks x 16 heads 15 us, six CTAs per SM; four 18 us.
template <int MODE>
__global__ void __launch_bounds__(DC_TEAM, 6)
delta_triangle_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ beta, const float* __restrict__ decay,
                      const int32_t* __restrict__ cu, float* __restrict__ o, int H, int KH, int dk, int dv, int slices) {
  constexpr int LDR = 40, LDP = 17;                            // padded rows: a half warp's 8-byte reads fall into different banks
  __shared__ __align__(16) float scratch_all[4][24 * LDR], part[4][2][16 * LDP], tri[16 * 20];
  __shared__ float out[16 * 17];
  const int h = blockIdx.y, d = threadIdx.x, w = d >> 5, lane = d & 31, g = lane >> 2, t = lane & 3;
  pdl_launch_dependents();
  const int t0 = cu[blockIdx.x], t1 = cu[blockIdx.x + 1];
  if (t1 - t0 < DC_MIN) return;
  const int kh = h / (H / KH), tok = lane & 15, wide = dc_slice(dv, slices, 0).n, narrow = dc_slice(dv, slices, slices - 1).n;
  const int per_wide = 65535 / wide + 1, per_narrow = 65535 / narrow + 1;      // i / w = (i * per) >> 16 for i < 272, w <= 64
  float* scratch = scratch_all[w];
  // where this lane's two sums of tokens of one quarter go: lane = 16 * (quarter of two) + (0 .. 5: A of pairs, 6 .. 11: P of them, 12 .. 15: P of the diagonal)
  const int idx = lane & 15, pair = idx < 6 ? idx : idx - 6;
  const int pt = idx < 12 ? (0x332321 >> (4 * pair)) & 15 : idx - 12, pj = idx < 12 ? (0x211000 >> (4 * pair)) & 15 : idx - 12;
  const int sum_at = ((lane >> 4) * 4 + pt) * LDP + (lane >> 4) * 4 + pj;
  for (int tc = t0 + (int)blockIdx.z * DC_CHUNK; tc < t1; tc += (int)gridDim.z * DC_CHUNK) {
    float k[DC_CHUNK], q[DC_CHUNK], gg[DC_CHUNK];              // tokens past the end are ones that change nothing
    dc_fetch<MODE>(qn, kn, decay, tc, t1, h, kh, d, H, KH, dk, k, q, gg);
    const float b = w == 0 && tc + tok < t1 ? beta[(int64_t)(tc + tok) * H + h] : 0.f;
    // ---- quarters: 32 sums over 32 lanes at a time (halve the values with every exchange)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float s[32];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int a = 8 * half + 4 * u;
        const float w01 = k[a] * gg[a + 1], w02 = w01 * gg[a + 2], w03 = w02 * gg[a + 3], w12 = k[a + 1] * gg[a + 2], w13 = w12 * gg[a + 3],
                    w23 = k[a + 2] * gg[a + 3];
        const float ws[6] = {w01, w02, w03, w12, w13, w23};
        const int to[6] = {1, 2, 3, 2, 3, 3};
#pragma unroll
        for (int i = 0; i < 6; ++i) s[16 * u + i] = k[a + to[i]] * ws[i], s[16 * u + 6 + i] = q[a + to[i]] * ws[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[16 * u + 12 + i] = q[a + i] * k[a + i];
      }
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (i >= m) continue;
          const float give = up ? s[i] : s[m + i], keep = up ? s[m + i] : s[i];
          s[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
        }
      }
      part[w][idx < 6 ? 0 : 1][sum_at + half * (8 * LDP + 8)] = s[0];
    }
    // ---- halves of the chunk, then the quarters of both halves: rows of k and q from the border on, rows of k up to it
#pragma unroll
    for (int level = 0; level < 2; ++level) {
#pragma unroll
      for (int u = 0; u < (level ? 2 : 1); ++u) {
        const int len = level ? 4 : 8, at = level ? 8 * u + 4 : 8, r0 = level ? 4 * u : 0;
        float c = 1.f;
#pragma unroll
        for (int i = 0; i < len; ++i) {
          c *= gg[at + i];
          scratch[(r0 + i) * LDR + lane] = k[at + i] * c;
          scratch[(8 + r0 + i) * LDR + lane] = q[at + i] * c;
        }
        c = 1.f;
#pragma unroll
        for (int i = len - 1; i >= 0; --i) {
          scratch[(16 + r0 + i) * LDR + lane] = k[at - len + i] * c;
          c *= gg[at - len + i];
        }
      }
      __syncwarp();
      float acc[4] = {0.f, 0.f, 0.f, 0.f}, rest[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {                         // rows of A: keys, queries
        auto at = [&](int row, int k) { return *reinterpret_cast<const float2*>(scratch + (row + g) * LDR + 16 * ks + k + 2 * t); };
        const float2 k0 = at(0, 0), q0 = at(8, 0), k1 = at(0, 8), q1 = at(8, 8), b0 = at(16, 0), b1 = at(16, 8);
        const float lo8[4] = {k0.x, k0.y, q0.x, q0.y}, hi8[4] = {k1.x, k1.y, q1.x, q1.y};
        uint32_t a[3][4];
        uint2 b[3];
        dc_operand(lo8, hi8, a);
        dc_split(b0.x, b0.y, b[0].x, b[1].x, b[2].x);
        dc_split(b1.x, b1.y, b[0].y, b[1].y, b[2].y);
        dc_low_terms(a, b, [&](const uint32_t (&x)[4], uint2 y) { dc_mma(rest, x, y); });
        float x[4];
        dc_mma0(x, a[0], b[0]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] += x[i];
      }
      const int i0 = g, j0 = 2 * t;                            // row of both kinds, columns j0, j0 + 1
      if (level == 0 || (i0 >> 2) == (j0 >> 2)) {
        const int at = level ? ((i0 >> 2) * 8 + 4 + (i0 & 3)) * LDP + (j0 >> 2) * 8 + (j0 & 3) : (8 + i0) * LDP + j0;
        part[w][0][at] = acc[0] + rest[0];
        part[w][0][at + 1] = acc[1] + rest[1];
        part[w][1][at] = acc[2] + rest[2];
        part[w][1][at + 1] = acc[3] + rest[3];
      }
      __syncwarp();
    }
    __syncthreads();
    if (w == 0) {                                              // lane: row of A (0 .. 15) or of P (16 .. 31), then column of the inverse
      float r[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int at = tok * LDP + j, kind = lane >> 4;
        r[j] = (part[0][kind][at] + part[1][kind][at]) + (part[2][kind][at] + part[3][kind][at]);
      }
      if (lane >= 16) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (j <= tok) out[(tok + 1) * (tok + 1) + j] = r[j];
      } else {
#pragma unroll
        for (int j = 0; j < 16; j += 4)
          *reinterpret_cast<float4*>(tri + tok * 20 + j) = make_float4(j < tok ? b * r[j] : 0.f, j + 1 < tok ? b * r[j + 1] : 0.f,
                                                                       j + 2 < tok ? b * r[j + 2] : 0.f, j + 3 < tok ? b * r[j + 3] : 0.f);
      }
      __syncwarp();
      float x[16];                                             // column tok of (I + diag(b) A)^-1, by rows
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float s[4] = {i == tok ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < i; j += 4) {
          const float4 l = *reinterpret_cast<const float4*>(tri + i * 20 + j);
          s[0] = fmaf(-l.x, x[j], s[0]);
          if (j + 1 < i) s[1] = fmaf(-l.y, x[j + 1], s[1]);
          if (j + 2 < i) s[2] = fmaf(-l.z, x[j + 2], s[2]);
          if (j + 3 < i) s[3] = fmaf(-l.w, x[j + 3], s[3]);
        }
        x[i] = (s[0] + s[1]) + (s[2] + s[3]);
        if (lane <= i) out[i * (i + 1) + lane] = lane < i ? x[i] : b;          // (lane 16 .. 31: not below 16)
      }
    }
    __syncthreads();
    const int m = min(DC_CHUNK, t1 - tc), numbers = m * (m + 1);
    for (int z = 0; z < slices; ++z) {
      const DcSlice sl = dc_slice(dv, slices, z);
      float* dst = o + ((int64_t)tc * H + h) * dv + sl.z0;
      for (int i = d; i < numbers; i += DC_TEAM) {
        const int r = (i * (sl.n == wide ? per_wide : per_narrow)) >> 16;
        dst[(int64_t)r * H * dv + (i - r * sl.n)] = out[i];
      }
    }
    __syncthreads();
  }
}

// The chain.  A CTA has up to 64 columns of a head.  Two warps keep S^T of 16 columns, half of the channels each, in the accumulators of m16n8k8 (rows: columns of
// the state), which are the A operand of the next products as they are; nothing of the state passes through shared memory, the two exchange
// their shares of the products with it.  Four more warps, a thread per key channel, scale the next chunks' vectors, split them and store them in the
// order in which the MMAs read them; three buffers, named barriers, so that pairs of warps may drift apart and cover each other's latencies.
// Bound: the state's warps, by their MMAs (324 per chunk and scheduler, 8 cycles each: 2600 of about 5600) and the fp32 instructions, which sm_100 does not
// issue beside them: a warp of mma.sync and one of FFMA on the same scheduler take the sum of their times (measured; integer instructions, three quarters
// of the sum).  Without any of the vectors' work a chunk takes 12 % less, without half of the first products' MMAs 15 % less.  All channels in one warp
// (nothing beside its MMAs) and making T and P here too, in both CTAs of a head, were slower (3.1 instead of 2.6 us and 4.4 us per chunk, with tf32 numbers).
// us, two tokens at a time in fp32 (the kernel before) -> now with the triangles, heads of 128 x 128, decays per channel / per head: 4 x 320 to 512 tokens, 16
// heads 155 -> 108 / 153 -> 108, 32 heads 266 -> 207 / 261 -> 205; 16 x 250, 32 heads 464 -> 413 / 456 -> 410; 1 x 1000, 16 heads 290 -> 187; 1 x 32 16 -> 14;
// but 8 x 33, 16 heads 26 -> 32 (three chunks for two and a bit).
// An entry takes this path if it has at least DC_MIN tokens, whatever the others have (the exception: top of the file); a prompt whose portions are
// shorter has the bits of single tokens, which differ in the last places.
// One buffer, in words of two bf16 numbers, three times each (the terms): K~ and Q~ as [8 blocks of 16 channels][4 tiles of 8 tokens][8 tokens][channels 2 t,
// 2 t + 1, then 8 more, t = 0 .. 3], tiles and blocks padded; K- as [16 tiles of 8 channels][8 channels][tokens 2 t, 2 t + 1, then 8 more] (halves of four words
// swapped in the upper four channels); T and P as [2 tiles of 8 tokens][8 tokens][columns 2 t, 2 t + 1, then 8 more]; and, in fp32, the decays over the whole chunk
constexpr int DC_STATE_WARPS = 8, DC_THREADS = 32 * DC_STATE_WARPS + DC_TEAM, DC_NBUF = 3;
constexpr int DC_TILE = 72, DC_BLOCK = 4 * DC_TILE + 16, DC_KQ = 8 * DC_BLOCK, DC_KM = 16 * 64, DC_TRI = 4 * 64;
constexpr int DC_KM_AT = 3 * DC_KQ, DC_TRI_AT = DC_KM_AT + 3 * DC_KM, DC_G = DC_TRI_AT + 3 * DC_TRI, DC_DIAG = DC_G + 128, DC_BUF = DC_DIAG + 32;
constexpr int DC_SWAP = DC_NBUF * DC_BUF;                      // [2][8 warps][3 pieces][32 lanes][4]
constexpr int DC_SMEM = (DC_SWAP + 2 * DC_STATE_WARPS * 3 * 128) * 4;
enum { DC_BAR_FULL = 1, DC_BAR_FREE = DC_BAR_FULL + DC_NBUF, DC_BAR_PAIR = DC_BAR_FREE + DC_NBUF };       // + buffer, + pair of warps

__device__ __forceinline__ void dc_sync(int bar, int n) { asm volatile("barrier.cta.sync %0, %1;" ::"r"(bar), "r"(n) : "memory"); }
__device__ __forceinline__ void dc_arrive(int bar, int n) { asm volatile("barrier.cta.arrive %0, %1;" ::"r"(bar), "r"(n) : "memory"); }
__device__ __forceinline__ int dc_tri_half(int tok, int j) { return 2 * ((tok >> 3) * 64 + (tok & 7) * 8 + ((j & 7) >> 1) * 2 + (j >> 3)) + (j & 1); }
struct DcTile { float x[2][4]; };                              // 16 columns of the state x 16 tokens, accumulator layout
__device__ __forceinline__ float dc_nonfinite(const DcTile& a) {             // 0, or NaN if an element is not finite
  float s[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) s[n] = fmaf(a.x[n][i], 0.f, s[n]);
  return s[0] + s[1];
}
// columns 8 N .. 8 N + 7 of in . M^T, added to out, with the lower triangle M [16, 16] (m: its words)
template <int N>
__device__ __forceinline__ void dc_triangle(float (&out)[4], const uint32_t (&a)[3][4], const uint32_t* m, int lane) {
  using B = std::conditional_t<N == 0, uint32_t, uint2>;       // (columns 8 .. 15 of the first eight rows are zero)
  B b[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) b[i] = *reinterpret_cast<const B*>(m + i * DC_TRI + 64 * N + 2 * lane);
  float r[4], s[4], u[4];                                      // (short chains)
  dc_mma0(r, a[0], b[0]);
  dc_mma0(s, a[2], b[0]);
  dc_mma0(u, a[0], b[2]);
  dc_mma(s, a[1], b[1]);
  dc_mma(u, a[0], b[1]);
  dc_mma(s, a[1], b[0]);
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] += (s[i] + u[i]) + r[i];
}
// The same for inputs that are not all finite: no product with the zeros above the diagonal, so a token's NaN or infinity reaches none before it.
__device__ __noinline__ DcTile dc_triangle_masked(DcTile in, const uint32_t* m, int lane) {
  const int t = lane & 3;
  const unsigned short* mh = reinterpret_cast<const unsigned short*>(m);
  DcTile out = {};
  for (int j = 0; j < 16; ++j) {
    const int from = (lane & ~3) | ((j & 7) >> 1);
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = __shfl_sync(0xffffffffu, j < 8 ? in.x[0][i] : in.x[1][i], from);
    const float xr[2] = {j & 1 ? x[1] : x[0], j & 1 ? x[3] : x[2]};
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int tok = 8 * n + 2 * t + c;
        if (tok <= j) continue;
        float w = 0.f;
#pragma unroll
        for (int i = 0; i < 3; ++i) w += __uint_as_float((uint32_t)mh[2 * i * DC_TRI + dc_tri_half(tok, j)] << 16);
        out.x[n][c] = fmaf(w, xr[0], out.x[n][c]);
        out.x[n][c + 2] = fmaf(w, xr[1], out.x[n][c + 2]);
      }
  }
  return out;
}

template <int MODE>
__global__ void __launch_bounds__(DC_THREADS, 1)
delta_chunk_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ v, const float* __restrict__ decay,
                   float* __restrict__ state, const int32_t* __restrict__ cu, const int32_t* __restrict__ rows, const int32_t* __restrict__ lengths,
                   float* o, int H, int KH, int dk, int dv) {
  extern __shared__ __align__(16) float dc_smem[];
  const int e = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  pdl_launch_dependents();
  const int t0 = cu[e], t1 = cu[e + 1];
  if (t1 - t0 < DC_MIN) {
    if ((blockIdx.x | blockIdx.y | blockIdx.z) == 0) pdl_wait();       // (this grid ends no earlier than the launch before, also where no entry is long)
    return;
  }
  const int row = rows[e], kh = h / (H / KH), chunks = (t1 - t0 + DC_CHUNK - 1) / DC_CHUNK;
  const DcSlice sl = dc_slice(dv, (int)gridDim.z, (int)blockIdx.z);
  const int z0 = sl.z0, z1 = z0 + sl.n;
  if (warp >= DC_STATE_WARPS) {
    // ===================================== vectors =====================================
    const int d = threadIdx.x - 32 * DC_STATE_WARPS;           // key channel
    float k[DC_CHUNK], q[DC_CHUNK], gg[DC_CHUNK], tp[3];
    // T and P: this thread's numbers d, d + 128, d + 256 of the packed rows
    const float* tp_src[3];
    int tp_dst[3], tp_tok[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const int i = d + r * DC_TEAM, wz = z1 - z0;
      int tt = 0;
      while ((tt + 1) * (tt + 2) <= i) ++tt;                   // rows below tt have tt (tt + 1) numbers
      const int in = i - tt * (tt + 1), p = in > tt ? 1 : 0, j = in - p * (tt + 1);
      tp_tok[r] = i < DC_CHUNK * (DC_CHUNK + 1) ? tt : 1 << 30;
      tp_dst[r] = j == tt ? -(DC_DIAG + p * 16 + tt) : 2 * (DC_TRI_AT + p * 128) + dc_tri_half(tt & 15, j);
      tp_src[r] = o + ((int64_t)(t0 + i / wz) * H + h) * dv + z0 + i % wz;
    }
    auto fetch = [&](int tc) {
      dc_fetch<MODE>(qn, kn, decay, tc, t1, h, kh, d, H, KH, dk, k, q, gg);
#pragma unroll
      for (int r = 0; r < 3; ++r) tp[r] = tc + tp_tok[r] < t1 ? tp_src[r][(int64_t)(tc - t0) * H * dv] : 0.f;
    };
    for (int i = d; i < DC_NBUF * 3 * DC_TRI; i += DC_TEAM) dc_smem[(i / (3 * DC_TRI)) * DC_BUF + DC_TRI_AT + i % (3 * DC_TRI)] = 0.f;       // (above the diagonal it stays so)
    pdl_wait();                                                // T and P
    fetch(t0);
    dc_sync(DC_BAR_FREE, DC_TEAM);                             // (the zeros before the numbers)
    for (int n = 0; n < chunks; ++n) {
      const int buf = n % DC_NBUF;
      float* b = dc_smem + buf * DC_BUF;
      uint32_t* bw = reinterpret_cast<uint32_t*>(b);
      if (n >= DC_NBUF) dc_sync(DC_BAR_FREE + buf, DC_THREADS);
      {                                                        // K~ = -G_t k_t and Q~ = G_t q_t: words of two channels, tokens 0 .. 7 in even lanes
        float c = 1.f, x[DC_CHUNK], y[DC_CHUNK];
#pragma unroll
        for (int i = 0; i < DC_CHUNK; ++i) c *= gg[i], x[i] = -k[i] * c, y[i] = q[i] * c;
        b[DC_G + d] = c;
        const bool odd = (d & 1) != 0;
        uint32_t* dst = bw + (d >> 4) * DC_BLOCK + (odd ? DC_TILE : 0) + ((d & 7) >> 1) * 2 + ((d >> 3) & 1);
        auto put = [&](const float (&v)[DC_CHUNK], uint32_t* to) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float other = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[8 + i], 1), own = odd ? v[8 + i] : v[i];
            uint32_t w0, w1, w2;
            dc_split(odd ? other : own, odd ? own : other, w0, w1, w2);
            to[i * 8] = w0, to[DC_KQ + i * 8] = w1, to[2 * DC_KQ + i * 8] = w2;
          }
        };
        put(x, dst);
        put(y, dst + 2 * DC_TILE);
      }
      {                                                        // K- = (G / G_j) k_j: words of two tokens
        float c = 1.f, x[DC_CHUNK];
#pragma unroll
        for (int i = DC_CHUNK - 1; i >= 0; --i) x[i] = k[i] * c, c *= gg[i];
        uint32_t* dst = bw + DC_KM_AT + (d >> 3) * 64 + (d & 7) * 8;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                          // t = 2 h, 2 h + 1
          uint32_t w[3][4];
          dc_split(x[4 * h], x[4 * h + 1], w[0][0], w[1][0], w[2][0]);
          dc_split(x[4 * h + 8], x[4 * h + 9], w[0][1], w[1][1], w[2][1]);
          dc_split(x[4 * h + 2], x[4 * h + 3], w[0][2], w[1][2], w[2][2]);
          dc_split(x[4 * h + 10], x[4 * h + 11], w[0][3], w[1][3], w[2][3]);
          uint32_t* at = dst + 4 * (h ^ ((d >> 2) & 1));
#pragma unroll
          for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(at + i * DC_KM) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
        }
      }
#pragma unroll
      for (int r = 0; r < 3; ++r)
        if (tp_dst[r] < 0 && tp_tok[r] < DC_CHUNK) {
          b[-tp_dst[r]] = tp[r];
        } else if (tp_tok[r] < DC_CHUNK) {
          uint32_t w0, w1, w2;
          dc_split(tp[r], 0.f, w0, w1, w2);
          unsigned short* at = reinterpret_cast<unsigned short*>(bw) + tp_dst[r];
          at[0] = (unsigned short)w0, at[2 * DC_TRI] = (unsigned short)w1, at[4 * DC_TRI] = (unsigned short)w2;
        }
      dc_arrive(DC_BAR_FULL + buf, DC_THREADS);
      if (n + 1 < chunks) fetch(t0 + (n + 1) * DC_CHUNK);
    }
    return;
  }
  // ===================================== state =======================================
  const int half = warp & 1, pair = warp >> 1;                 // 64 of the channels, 16 of the columns
  const int ja = z0 + 16 * pair + g, jb = ja + 8;              // this lane's columns of the state (rows of the fragments)
  const bool la = ja < z1, lb = jb < z1;
  float* sp = state + (((int64_t)row * H + h) * dk + 64 * half) * dv;
  const bool fresh = lengths[row] == 0;                        // first token of a sequence: the state starts at zero
  float S[8][4];                                               // [8 channels][(column a, channels 2 t, 2 t + 1), (column b, the same)]
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int r = 8 * n + 2 * t + c;
      const bool in = !fresh && 64 * half + r < dk;
      S[n][c] = in && la ? sp[(int64_t)r * dv + ja] : 0.f;
      S[n][2 + c] = in && lb ? sp[(int64_t)r * dv + jb] : 0.f;
    }
  DcTile vn;                                                   // the next chunk's values
  auto fetch_v = [&](int tc) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int tok = tc + 8 * n + 2 * t + c;
        const float* src = v + ((int64_t)tok * H + h) * dv;
        vn.x[n][c] = tok < t1 && la ? src[ja] : 0.f;
        vn.x[n][2 + c] = tok < t1 && lb ? src[jb] : 0.f;
      }
  };
  fetch_v(t0);
  for (int n = 0; n < chunks; ++n) {
    const int buf = n % DC_NBUF, tc = t0 + n * DC_CHUNK;
    const float* b = dc_smem + buf * DC_BUF;
    const uint32_t* bw = reinterpret_cast<const uint32_t*>(b);
    float4* swap = reinterpret_cast<float4*>(dc_smem + DC_SWAP) + (n & 1) * (DC_STATE_WARPS * 3 * 32) + lane;
    float sum[4][4], rest[4][4];                               // -S^T K~ of tokens 0 .. 7, 8 .. 15, S^T Q~ of both
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[m][i] = rest[m][i] = 0.f;
    dc_sync(DC_BAR_FULL + buf, DC_THREADS);
#pragma unroll
    for (int kb = 0; kb < 4; ++kb) {                           // (a block's leading products hardly lose a bit in one MMA; the blocks meet in rounding additions)
      float acc[4][4];
      uint32_t a[3][4];
      uint2 bv[4][3];
      dc_operand(S[2 * kb], S[2 * kb + 1], a);
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int j = 0; j < 3; ++j) bv[m][j] = *reinterpret_cast<const uint2*>(bw + j * DC_KQ + (4 * half + kb) * DC_BLOCK + m * DC_TILE + 2 * lane);
#pragma unroll
      for (int m = 0; m < 4; ++m) dc_mma0(acc[m], a[0], bv[m][0]);
#pragma unroll
      for (int m = 0; m < 4; ++m) dc_mma(rest[m], a[2], bv[m][0]);
#pragma unroll
      for (int m = 0; m < 4; ++m) dc_mma(rest[m], a[0], bv[m][2]);
#pragma unroll
      for (int m = 0; m < 4; ++m) dc_mma(rest[m], a[1], bv[m][1]);
#pragma unroll
      for (int m = 0; m < 4; ++m) dc_mma(rest[m], a[1], bv[m][0]);
#pragma unroll
      for (int m = 0; m < 4; ++m) dc_mma(rest[m], a[0], bv[m][1]);
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[m][i] += acc[m][i];
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int i = 0; i < 4; ++i) sum[m][i] += rest[m][i];
    // ---- the other half of the channels; this warp writes the outputs of tokens 8 half .. 8 half + 7
    float4* mine = swap + warp * 96;
    const float4* theirs = swap + (warp ^ 1) * 96;
    const float (&give)[4] = half ? sum[2] : sum[3];
    mine[0] = make_float4(sum[0][0], sum[0][1], sum[0][2], sum[0][3]);
    mine[32] = make_float4(sum[1][0], sum[1][1], sum[1][2], sum[1][3]);
    mine[64] = make_float4(give[0], give[1], give[2], give[3]);
    dc_sync(DC_BAR_PAIR + pair, 64);
    DcTile X;
    float2 bt[2];
    float out[4];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const float4 x = theirs[32 * m];
      X.x[m][0] = vn.x[m][0] + (sum[m][0] + x.x), X.x[m][1] = vn.x[m][1] + (sum[m][1] + x.y);
      X.x[m][2] = vn.x[m][2] + (sum[m][2] + x.z), X.x[m][3] = vn.x[m][3] + (sum[m][3] + x.w);
      bt[m] = *reinterpret_cast<const float2*>(b + DC_DIAG + 8 * m + 2 * t);
    }
    {
      const float4 x = theirs[64];
      out[0] = (half ? sum[3][0] : sum[2][0]) + x.x, out[1] = (half ? sum[3][1] : sum[2][1]) + x.y;
      out[2] = (half ? sum[3][2] : sum[2][2]) + x.z, out[3] = (half ? sum[3][3] : sum[2][3]) + x.w;
    }
    if (n + 1 < chunks) fetch_v(tc + DC_CHUNK);
    // ---- U = b X + (T - I) b X, O += P U: diagonals in fp32 FMAs, the last roundings but those of the large terms beside them
    DcTile Y, U = {};
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      Y.x[m][0] = X.x[m][0] * bt[m].x, Y.x[m][1] = X.x[m][1] * bt[m].y;
      Y.x[m][2] = X.x[m][2] * bt[m].x, Y.x[m][3] = X.x[m][3] * bt[m].y;
    }
    uint32_t a[3][4];
    if (__any_sync(0xffffffffu, dc_nonfinite(Y) != 0.f)) {
      U = dc_triangle_masked(Y, bw + DC_TRI_AT, lane);
    } else {
      dc_operand(Y.x[0], Y.x[1], a);
      dc_triangle<0>(U.x[0], a, bw + DC_TRI_AT, lane);
      dc_triangle<1>(U.x[1], a, bw + DC_TRI_AT, lane);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      U.x[m][0] = fmaf(X.x[m][0], bt[m].x, U.x[m][0]), U.x[m][1] = fmaf(X.x[m][1], bt[m].y, U.x[m][1]);
      U.x[m][2] = fmaf(X.x[m][2], bt[m].x, U.x[m][2]), U.x[m][3] = fmaf(X.x[m][3], bt[m].y, U.x[m][3]);
    }
    dc_operand(U.x[0], U.x[1], a);
    if (__any_sync(0xffffffffu, dc_nonfinite(U) != 0.f)) {
      const DcTile m = dc_triangle_masked(U, bw + DC_TRI_AT + 128, lane);
#pragma unroll
      for (int i = 0; i < 4; ++i) out[i] += half ? m.x[1][i] : m.x[0][i];
    } else if (half) {
      dc_triangle<1>(out, a, bw + DC_TRI_AT + 128, lane);
    } else {
      dc_triangle<0>(out, a, bw + DC_TRI_AT + 128, lane);
    }
    {
      const float2 pt = *reinterpret_cast<const float2*>(b + DC_DIAG + 16 + 8 * half + 2 * t);
      const float (&u)[4] = half ? U.x[1] : U.x[0];
      out[0] = fmaf(pt.x, u[0], out[0]), out[1] = fmaf(pt.y, u[1], out[1]), out[2] = fmaf(pt.x, u[2], out[2]), out[3] = fmaf(pt.y, u[3], out[3]);
    }
    // ---- S <- G S + K- U
    const uint32_t* kb = bw + DC_KM_AT + half * (8 * 64) + g * 8 + 4 * ((t >> 1) ^ (g >> 2)) + 2 * (t & 1);
#pragma unroll
    for (int m0 = 0; m0 < 8; m0 += 4) {                        // (four sums at a time cover each other's latencies)
      float acc[4][4], big[4][4];
      uint2 bv[4][3];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) bv[i][j] = *reinterpret_cast<const uint2*>(kb + j * DC_KM + (m0 + i) * 64);
#pragma unroll
      for (int i = 0; i < 4; ++i) dc_mma0(acc[i], a[2], bv[i][0]);
#pragma unroll
      for (int i = 0; i < 4; ++i) dc_mma(acc[i], a[0], bv[i][2]);
#pragma unroll
      for (int i = 0; i < 4; ++i) dc_mma(acc[i], a[1], bv[i][1]);
#pragma unroll
      for (int i = 0; i < 4; ++i) dc_mma(acc[i], a[1], bv[i][0]);
#pragma unroll
      for (int i = 0; i < 4; ++i) dc_mma(acc[i], a[0], bv[i][1]);
#pragma unroll
      for (int i = 0; i < 4; ++i) dc_mma0(big[i], a[0], bv[i][0]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 c = *reinterpret_cast<const float2*>(b + DC_G + 64 * half + 8 * (m0 + i) + 2 * t);
        float (&x)[4] = S[m0 + i];
        const float2 p = __ffma2_rn(make_float2(x[0], x[1]), c, make_float2(acc[i][0], acc[i][1]));
        const float2 r = __ffma2_rn(make_float2(x[2], x[3]), c, make_float2(acc[i][2], acc[i][3]));
        x[0] = p.x + big[i][0], x[1] = p.y + big[i][1], x[2] = r.x + big[i][2], x[3] = r.y + big[i][3];
      }
    }
    if (n + DC_NBUF < chunks) dc_arrive(DC_BAR_FREE + buf, DC_THREADS);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int tok = tc + 8 * half + 2 * t + c;
      float* dst = o + ((int64_t)tok * H + h) * dv;
      if (tok < t1 && la) dst[ja] = out[c];
      if (tok < t1 && lb) dst[jb] = out[2 + c];
    }
  }
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int r = 8 * n + 2 * t + c;
      if (64 * half + r >= dk) continue;
      if (la) sp[(int64_t)r * dv + ja] = S[n][c];
      if (lb) sp[(int64_t)r * dv + jb] = S[n][2 + c];
    }
}

// Decode steps (few tokens per entry).  Reading and writing the state is nearly all of it, so: small CTAs (16 KB of state at 128 rows,
// in the registers of four warps), as many per SM as fit, so that some load while others compute and store; the token's inputs are asked
// for first, so that they are staged while the state is on its way; neighbouring columns per thread, one 8-byte access where the
// alignment allows.  64 entries of one token, us, beside the kernel above: 32 heads of 128 x 128 78 / 80 (3.4 TB/s), of 64 x 64 15 / 24, 8 heads
// of 256 x 256 79 / 132.
constexpr int DT_THREADS = 128;
constexpr int dt_cols(int dkp) { return 2 * DT_THREADS / ds_segs(dkp); }
template <int DKP, int MODE>
__global__ void __launch_bounds__(DT_THREADS)
delta_step_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ v,
                  const float* __restrict__ beta, const float* __restrict__ decay, float* __restrict__ state,
                  const int32_t* __restrict__ cu, const int32_t* __restrict__ rows, const int32_t* __restrict__ lengths,
                  float* __restrict__ o, int H, int KH, int dk, int dv) {
  constexpr int LANES = ds_segs(DKP), SEG = DKP / LANES, LDK = DKP + 4 * LANES;
  constexpr int PF = (DKP + DT_THREADS - 1) / DT_THREADS;
  __shared__ __align__(16) float ks[LDK], qs[LDK], gc[MODE == 1 ? LDK : 4];
  const int e = blockIdx.x, h = blockIdx.y;
  const int l = threadIdx.x & (LANES - 1), slot = threadIdx.x / LANES;
  const int j0 = blockIdx.z * dt_cols(DKP) + 2 * slot, j1 = j0 + 1;
  const bool live0 = j0 < dv, live1 = j1 < dv, odd = (l & 1) != 0;
  const bool pairs = (dv & 1) == 0 && (reinterpret_cast<uintptr_t>(state) & 7) == 0;
  const int t0 = cu[e], t1 = cu[e + 1], row = rows[e];
  if (t1 <= t0) return;
  const int kh = h / (H / KH);
  float pk[PF], pq[PF], pg[MODE == 1 ? PF : 1], pv, g = 1.f, b = 0.f;
  auto fetch = [&](int t) {
#pragma unroll
    for (int r = 0; r < PF; ++r) {
      const int i = threadIdx.x + r * DT_THREADS;
      const bool ok = i < dk;
      pk[r] = ok ? kn[((int64_t)t * KH + kh) * dk + i] : 0.f;
      pq[r] = ok ? qn[((int64_t)t * KH + kh) * dk + i] : 0.f;
      if constexpr (MODE == 1) pg[r] = ok ? decay[((int64_t)t * H + h) * dk + i] : 1.f;
    }
    const int j = odd ? j1 : j0;
    pv = j < dv ? v[((int64_t)t * H + h) * dv + j] : 0.f;
    if constexpr (MODE != 1) g = decay[(int64_t)t * H + h];
    if constexpr (MODE != 2) b = beta[(int64_t)t * H + h];
  };
  fetch(t0);
  const bool fresh = lengths[row] == 0;                          // first token of a sequence: the state starts at zero
  float* sp = state + (((int64_t)row * H + h) * dk + l * SEG) * dv + j0;
  DsCols<SEG, 1> S;
#pragma unroll
  for (int i = 0; i < SEG / 2; ++i) {
    const bool in0 = l * SEG + 2 * i < dk, in1 = l * SEG + 2 * i + 1 < dk;
    const float* s0 = sp + (int64_t)(2 * i) * dv;
    float2 a = make_float2(0.f, 0.f), c = a;
    if (pairs) {
      if (in0 && live0) a = *reinterpret_cast<const float2*>(s0);
      if (in1 && live0) c = *reinterpret_cast<const float2*>(s0 + dv);
    } else {
      if (in0 && live0) a.x = s0[0];
      if (in0 && live1) a.y = s0[1];
      if (in1 && live0) c.x = s0[dv];
      if (in1 && live1) c.y = s0[dv + 1];
    }
    S.c0[0][i] = make_float2(a.x, c.x);
    S.c1[0][i] = make_float2(a.y, c.y);
  }
  for (int t = t0; t < t1; ++t) {
    if (t > t0) __syncthreads();                                 // the previous token's rows have been read
#pragma unroll
    for (int r = 0; r < PF; ++r) {
      const int i = threadIdx.x + r * DT_THREADS;
      if (i < DKP) {
        ks[i + (i / SEG) * 4] = pk[r];
        qs[i + (i / SEG) * 4] = pq[r];
        if constexpr (MODE == 1) gc[i + (i / SEG) * 4] = pg[r];
      }
    }
    const float v1 = pv, b1 = b, g1 = g;
    __syncthreads();
    if (t + 1 < t1) fetch(t + 1);
    if (t == t0 && fresh) {
#pragma unroll
      for (int i = 0; i < SEG / 2; ++i) S.c0[0][i] = S.c1[0][i] = make_float2(0.f, 0.f);
    }
    float2 kr[1][SEG / 2];
    const float2 d = ds_decay_dot<SEG, 1, MODE>(S, &ks[l * (SEG + 4)], &gc[MODE == 1 ? l * (SEG + 4) : 0], g1, kr);
    float u1 = v1;
    if constexpr (MODE != 2) u1 = b1 * (v1 - ds_reduce<LANES>(d.x, d.y, odd));
    const float u_other = __shfl_xor_sync(0xffffffffu, u1, 1);
    const float2 p = ds_update_dot<SEG, 1>(S, &qs[l * (SEG + 4)], kr, odd ? u_other : u1, odd ? u1 : u_other);
    const float out = ds_reduce<LANES>(p.x, p.y, odd);
    if (l < 2 && (odd ? live1 : live0)) o[((int64_t)t * H + h) * dv + (odd ? j1 : j0)] = out;
  }
#pragma unroll
  for (int i = 0; i < SEG / 2; ++i) {
    const bool in0 = l * SEG + 2 * i < dk, in1 = l * SEG + 2 * i + 1 < dk;
    float* s0 = sp + (int64_t)(2 * i) * dv;
    if (pairs) {
      if (in0 && live0) *reinterpret_cast<float2*>(s0) = make_float2(S.c0[0][i].x, S.c1[0][i].x);
      if (in1 && live0) *reinterpret_cast<float2*>(s0 + dv) = make_float2(S.c0[0][i].y, S.c1[0][i].y);
    } else {
      if (in0 && live0) s0[0] = S.c0[0][i].x;
      if (in0 && live1) s0[1] = S.c1[0][i].x;
      if (in1 && live0) s0[dv] = S.c0[0][i].y;
      if (in1 && live1) s0[dv + 1] = S.c1[0][i].y;
    }
  }
}

__device__ __forceinline__ float gate_act_f(float z, int act) { return act == 0 ? silu_f(z) : 1.f / (1.f + expf(-z)); }

// groups of dv values (a head each, or all heads as one group when H == 1) are rms-normed, weighted by norm_w [dv], gated by
// act(gate) (0 silu, 1 sigmoid) and scaled; out rows have stride ld_out
template <typename T>
__global__ void delta_out_kernel(const float* __restrict__ o, const float* __restrict__ gate, int64_t ldg,
                                 const float* __restrict__ norm_w, T* __restrict__ out, int64_t ld_out, int H, int dv, float eps,
                                 int act, float out_scale) {
  const int64_t t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (H == 1) {                                   // one wide group: the whole block sums it, in an order fixed by the block size
    __shared__ float red[32];
    const float* src = o + t * dv;
    const float* g = gate + t * ldg;
    float ss = 0.f;
    for (int i = threadIdx.x; i < dv; i += blockDim.x) ss = fmaf(src[i], src[i], ss);
    ss = warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float tot = 0.f;
    for (int i = 0; i < nw; ++i) tot += red[i];
    const float inv = out_scale / sqrtf(tot / (float)dv + eps);
    for (int i = threadIdx.x; i < dv; i += blockDim.x)
      out[t * ld_out + i] = Tr<T>::from_f(src[i] * inv * norm_w[i] * gate_act_f(g[i], act));
    return;
  }
  for (int h = warp; h < H; h += nw) {
    const float* src = o + (t * H + h) * dv;
    const float* g = gate + t * ldg + (int64_t)h * dv;
    float ss = 0.f;
    for (int i = lane; i < dv; i += 32) ss = fmaf(src[i], src[i], ss);
    ss = warp_sum(ss);
    const float inv = out_scale / sqrtf(ss / (float)dv + eps);
    for (int i = lane; i < dv; i += 32)
      out[t * ld_out + (int64_t)h * dv + i] = Tr<T>::from_f(src[i] * inv * norm_w[i] * gate_act_f(g[i], act));
  }
}

// The same for groups of 128 * NV values in 16-byte pieces: a warp per (token, head), its values in registers between the sum and the
// output.  1664 tokens, 16 heads of 128, bf16, us: 15.2 -> 8.4.
template <typename T, int NV>
__global__ void __launch_bounds__(256)
delta_out_rows_kernel(const float* __restrict__ o, const float* __restrict__ gate, int64_t ldg, const float* __restrict__ norm_w,
                      T* __restrict__ out, int64_t ld_out, int64_t pairs, int H, float eps, int act, float out_scale) {
  constexpr int DV = 128 * NV;
  const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= pairs) return;
  const int64_t t = i / H;
  const int h = (int)(i - t * H);
  float4 x[NV], g[NV], w[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const int c = 128 * k + 4 * lane;
    x[k] = *reinterpret_cast<const float4*>(o + i * DV + c);
    g[k] = *reinterpret_cast<const float4*>(gate + t * ldg + (int64_t)h * DV + c);
    w[k] = *reinterpret_cast<const float4*>(norm_w + c);
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k) ss = fmaf(x[k].x, x[k].x, fmaf(x[k].y, x[k].y, fmaf(x[k].z, x[k].z, fmaf(x[k].w, x[k].w, ss))));
  const float inv = out_scale / sqrtf(warp_sum(ss) / (float)DV + eps);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    __align__(16) T r[4] = {Tr<T>::from_f(x[k].x * inv * w[k].x * gate_act_f(g[k].x, act)), Tr<T>::from_f(x[k].y * inv * w[k].y * gate_act_f(g[k].y, act)),
                            Tr<T>::from_f(x[k].z * inv * w[k].z * gate_act_f(g[k].z, act)), Tr<T>::from_f(x[k].w * inv * w[k].w * gate_act_f(g[k].w, act))};
    T* dst = out + t * ld_out + (int64_t)h * DV + 128 * k + 4 * lane;
    if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(r);
    else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(r);
  }
}

}  // namespace b200p

using namespace b200p;

extern "C" int b200p_delta_prep(const float* proj, int64_t ldp, int64_t col_b, const float* a, int64_t lda, int decay_per_head,
                                const float* conv_w, const float* conv_state, const float* A_log, const float* dt_bias, const int32_t* t_row,
                                const int32_t* t_pos, const int32_t* t_off, float* qn, float* kn, float* v, float* beta,
                                float* decay, int64_t M, int H, int KH, int dk, int dv, int taps, void* stream) {
  B200P_REQUIRE(a && (decay_per_head == 1 || decay_per_head == dk), B200P_ERR_ARG, "one decay per head, or one per key channel");
  B200P_REQUIRE(proj && conv_w && conv_state && A_log && dt_bias && t_row && t_pos && t_off && qn && kn && v && beta && decay,
                B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(H > 0 && KH > 0 && H % KH == 0 && dk > 0 && dv > 0, B200P_ERR_ARG, "bad head geometry");
  B200P_REQUIRE(taps >= 1 && taps <= DELTA_MAX_TAPS, B200P_ERR_ARG, "convolution taps must be in [1, %d]", DELTA_MAX_TAPS);
  if (M == 0) return B200P_OK;
  const size_t smem = (size_t)2 * KH * dk * sizeof(float);
  B200P_REQUIRE(smem <= 48 * 1024, B200P_ERR_ARG, "q and k of one token must fit 48 KB of shared memory");
  if (M < (1ll << 30) && dk == 128 && dv % 128 == 0 && taps == 4) {             // heads of 128 channels; fewer tokens, shorter runs of them per warp
    const int tt = M > 512 ? 8 : M > 128 ? 4 : 1, nd = H * decay_per_head;
    const int units = 2 * KH + H * dv / 128 + (nd + 127) / 128 + (H + 127) / 128;
    const auto kern = tt == 8 ? delta_prep_rows_kernel<4, 8> : tt == 4 ? delta_prep_rows_kernel<4, 4> : delta_prep_rows_kernel<4, 1>;
    kern<<<dim3((unsigned)((M + tt - 1) / tt), (unsigned)((units + 3) / 4)), 128, 0, (cudaStream_t)stream>>>(
        proj, ldp, col_b, a, lda, decay_per_head, conv_w, conv_state, A_log, dt_bias, t_row, t_pos, t_off, qn, kn, v, beta, decay, (int)M, H, KH, dv);
    B200P_LAUNCH_CHECK("delta_prep_rows_kernel");
    return B200P_OK;
  }
  // a decode batch has few tokens and thousands of channels each: wider blocks shorten the per-thread channel loop
  if (M <= 256)
    delta_prep_kernel<1024><<<(unsigned)M, 1024, smem, (cudaStream_t)stream>>>(proj, ldp, col_b, a, lda, decay_per_head, conv_w, conv_state, A_log, dt_bias, t_row,
                                                                               t_pos, t_off, qn, kn, v, beta, decay, H, KH, dk, dv, taps);
  else
    delta_prep_kernel<256><<<(unsigned)M, 256, smem, (cudaStream_t)stream>>>(proj, ldp, col_b, a, lda, decay_per_head, conv_w, conv_state, A_log, dt_bias, t_row,
                                                                             t_pos, t_off, qn, kn, v, beta, decay, H, KH, dk, dv, taps);
  B200P_LAUNCH_CHECK("delta_prep_kernel");
  return B200P_OK;
}

extern "C" int b200p_delta_conv_commit(const float* proj, int64_t ldp, float* conv_state, const int32_t* cu, const int32_t* rows,
                                       int nb, int64_t C, int taps, void* stream) {
  B200P_REQUIRE(proj && conv_state && cu && rows && nb > 0 && nb < 65536, B200P_ERR_ARG, "null pointer or bad batch");
  B200P_REQUIRE(taps >= 1 && taps <= DELTA_MAX_TAPS, B200P_ERR_ARG, "convolution taps must be in [1, %d]", DELTA_MAX_TAPS);
  if (taps == 1) return B200P_OK;
  dim3 grid((unsigned)((C + 127) / 128), (unsigned)nb);
  delta_conv_commit_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(proj, ldp, conv_state, cu, rows, C, taps);
  B200P_LAUNCH_CHECK("delta_conv_commit_kernel");
  return B200P_OK;
}

// tokens: of all entries together, longest: of the longest; 0 if the caller does not say.
template <int MODE>
static cudaError_t delta_scan_launch(int64_t tokens, int64_t longest, int nb, cudaStream_t st, const float* qn, const float* kn, const float* v, const float* beta,
                              const float* decay, float* state, const int32_t* cu, const int32_t* rows, const int32_t* lengths,
                              float* o, int H, int KH, int dk, int dv) {
#define DELTA_STEP(DKP)                                                                                                          \
  delta_step_kernel<DKP, MODE><<<dim3((unsigned)nb, (unsigned)H, (unsigned)((dv + dt_cols(DKP) - 1) / dt_cols(DKP))), DT_THREADS, 0, st>>>( \
      qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv)
#define DELTA_SCAN(DKP, LANES, PER_SM)                                                                                           \
  launch_pdl_opt(chunks && pdl_enabled_gemm(), delta_scan_kernel<DKP, MODE, LANES, PER_SM>,                                        \
                 dim3((unsigned)nb, (unsigned)H, (unsigned)((dv + 2 * ds_slots(DKP) - 1) / (2 * ds_slots(DKP)))), dim3(LANES * ds_slots(DKP)), 0, st, \
                 qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv, chunks ? DC_MIN - 1 : INT32_MAX)
  // The step kernel for decode steps, and for as many tokens per entry as it keeps up with the scan (us, step / scan): 128 x 128, 16
  // entries of 1 / 2 / 4 tokens, 32 heads, 21.7 / 23.1, 27.1 / 25.3, 32.0 / 29.2; 64 x 64, 32 heads, of 2 / 4 / 8, 6.8 / 8.8, 7.9 / 9.6,
  // 10.2 / 11.4, but with 16 heads 4.3 / 4.6, 5.1 / 5.0, 7.3 / 6.4; 32 x 64, 16 heads, of 2 / 4, 3.4 / 3.5, 4.2 / 3.9; 256 x 256, 8 heads,
  // 4 entries of 16 / 64, 20 / 20, 58 / 50.
  // The plain accumulation of keys above 128 takes it at any length (16 x 250 tokens of 256 x 256: 407 / 678; 4 x 512: 315 / 309).
  const int most = dk > 128 ? 8 : dk > 64 ? 1 : dk > 32 ? 4 : 2;
  const bool by_chunks = MODE != 2 && dk > 64 && dk <= 128 && dv >= DC_MIN_DV && o != v;                   // entries of DC_MIN tokens and more
  const bool few = (tokens > 0 && tokens <= most * (int64_t)nb && !(by_chunks && longest >= DC_MIN)) || (MODE == 2 && dk > 128);
  // 128 rows: one CTA per SM takes eight lanes per column and the shortest chain (4 x 512 tokens, 16 heads, decays per channel / per
  // head: 220 / 193 us, the former four-lane kernel 280 / 206); more CTAs than SMs take four (32 heads 379 / 346 -> 356 / 317; 16 x 250
  // tokens 672 / 594 -> 637 / 544).
  const bool crowded = (int64_t)nb * H * ((dv + 63) / 64) > sm_count();
  // Entries of DC_MIN tokens and more in chunks (into values of more than 16 columns, other than v's own memory: o holds T and P), the shorter ones by the launch behind it, which needs nothing of it: it may start at
  // once (its inputs were complete when the first began), and one of its CTAs waits for the first launch, so that what follows waits for both.
  // (Only one: with every CTA waiting, those that do not fit beside the first launch started when it had ended: 15 entries of one token and one
  // of 40, 32 heads, decays per head / channel 43.7 / 45.7 -> 30 / 30.5 us, the scan alone 38 / 42.)  The long ones first: the short ones of such a
  // batch come with their tail.  A call that knows its longest entry to be short is spared the first launch: 16 entries of 4 tokens, 16 heads 14.4 ->
  // 13.3 us.
  const bool chunks = by_chunks && !few && (tokens == 0 || tokens >= DC_MIN) && (longest == 0 || longest >= DC_MIN);
  // An entry's own length alone decides, so that its bits do not depend on the others.  Beside the chunk kernel's CTAs, which take an SM's registers, the
  // token-by-token ones find little room: batches with entries on both sides of DC_MIN pay for that (us, the two-token kernel before / so / all entries of 16
  // and more in chunks: 40, 35, 30, 25 tokens, 32 heads 28 / 43 / 31; 60 to 34 tokens, eight entries of 16 heads 38 / 37 / 37; below 64 tokens only).
  if constexpr (MODE != 2) {
    if (chunks) {
      static const cudaError_t ready = cudaFuncSetAttribute(delta_chunk_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_SMEM);
      if (ready != cudaSuccess) return ready;
      const unsigned slices = (unsigned)((dv + DC_COLS - 1) / DC_COLS), most = (unsigned)(longest ? (longest + DC_CHUNK - 1) / DC_CHUNK : 16);
      delta_triangle_kernel<MODE><<<dim3((unsigned)nb, (unsigned)H, most < 1024 ? most : 1024), DC_TEAM, 0, st>>>(qn, kn, beta, decay, cu, o, H, KH, dk, dv, (int)slices);
      const cudaError_t e = launch_pdl_opt(pdl_enabled_gemm(), delta_chunk_kernel<MODE>, dim3((unsigned)nb, (unsigned)H, slices), dim3(DC_THREADS), DC_SMEM, st,
                                           qn, kn, v, decay, state, cu, rows, lengths, o, H, KH, dk, dv);
      if (e != cudaSuccess) return e;
    }
  }
  if (dk > 256) { if (few) DELTA_STEP(512); else DELTA_SCAN(512, 16, 1); }
  else if (dk > 128) { if (few) DELTA_STEP(256); else DELTA_SCAN(256, 8, 1); }
  else if (dk > 64) { if (few) DELTA_STEP(128); else if (crowded) DELTA_SCAN(128, 4, 2); else DELTA_SCAN(128, 8, 1); }
  else if (dk > 32) { if (few) DELTA_STEP(64); else DELTA_SCAN(64, 4, 1); }
  else { if (few) DELTA_STEP(32); else DELTA_SCAN(32, 4, 1); }
#undef DELTA_STEP
#undef DELTA_SCAN
  return cudaSuccess;
}

extern "C" int b200p_delta_scan_entries(const float* qn, const float* kn, const float* v, const float* beta, const float* decay,
                                       float* state, const int32_t* cu, const int32_t* rows, const int32_t* lengths, float* o, int64_t tokens,
                                       int64_t longest, int nb, int H, int KH, int dk, int dv, int mode, void* stream) {
  B200P_REQUIRE(qn && kn && v && decay && state && cu && rows && lengths && o, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(mode >= B200P_SCAN_DELTA && mode <= B200P_SCAN_ACCUMULATE, B200P_ERR_ARG, "unknown scan mode %d", mode);
  B200P_REQUIRE(beta || mode == B200P_SCAN_ACCUMULATE, B200P_ERR_ARG, "the delta rule needs beta");
  B200P_REQUIRE(nb > 0 && H > 0 && KH > 0 && H % KH == 0 && H < 65536 && dk > 0 && dv > 0, B200P_ERR_ARG, "bad head geometry");
  B200P_REQUIRE(tokens >= 0 && longest >= 0, B200P_ERR_ARG, "negative token count");
  B200P_REQUIRE(dk <= 512, B200P_ERR_ARG, "key size %d > 512 is not built", dk);
  cudaStream_t st = (cudaStream_t)stream;
  const auto launch = mode == B200P_SCAN_DELTA ? delta_scan_launch<0> : mode == B200P_SCAN_DELTA_CHANNEL ? delta_scan_launch<1> : delta_scan_launch<2>;
  if (const cudaError_t e = launch(tokens, longest, nb, st, qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv))
    return cuda_fail(e, "delta_chunk_kernel");
  B200P_LAUNCH_CHECK("delta_scan_kernel");
  return B200P_OK;
}

extern "C" int b200p_delta_scan_tokens(const float* qn, const float* kn, const float* v, const float* beta, const float* decay,
                                       float* state, const int32_t* cu, const int32_t* rows, const int32_t* lengths, float* o, int64_t tokens,
                                       int nb, int H, int KH, int dk, int dv, int mode, void* stream) {
  return b200p_delta_scan_entries(qn, kn, v, beta, decay, state, cu, rows, lengths, o, tokens < 0 ? 0 : tokens, 0, nb, H, KH, dk, dv, mode, stream);
}

extern "C" int b200p_delta_scan(const float* qn, const float* kn, const float* v, const float* beta, const float* decay,
                                float* state, const int32_t* cu, const int32_t* rows, const int32_t* lengths, float* o, int nb,
                                int H, int KH, int dk, int dv, int mode, void* stream) {
  return b200p_delta_scan_tokens(qn, kn, v, beta, decay, state, cu, rows, lengths, o, 0, nb, H, KH, dk, dv, mode, stream);
}

extern "C" int b200p_linear_attn_prep(const float* proj, int64_t ldp, const float* head_decay, float* q, float* k, float* v,
                                      float* decay, int64_t M, int H, int dk, int dv, void* stream) {
  B200P_REQUIRE(proj && head_decay && q && k && v && decay && H > 0 && dk > 0 && dv > 0, B200P_ERR_ARG, "null pointer");
  if (M == 0) return B200P_OK;
  linear_attn_prep_kernel<<<(unsigned)M, 256, 0, (cudaStream_t)stream>>>(proj, ldp, head_decay, q, k, v, decay, H, H * dk, H * dv);
  B200P_LAUNCH_CHECK("linear_attn_prep_kernel");
  return B200P_OK;
}

extern "C" int b200p_delta_out(const float* o, const float* gate, int64_t ldg, const float* norm_w, void* out, int64_t ld_out,
                               int64_t M, int H, int dv, float eps, int gate_act, float out_scale, int dtype, void* stream) {
  B200P_REQUIRE(o && gate && norm_w && out && H > 0 && dv > 0, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(gate_act == 0 || gate_act == 1, B200P_ERR_ARG, "gate activation: 0 silu, 1 sigmoid");
  B200P_REQUIRE(ld_out >= (int64_t)H * dv, B200P_ERR_ARG, "output rows are shorter than the heads");
  if (M == 0) return B200P_OK;
  const int nv = dv % 128 == 0 ? dv / 128 : 0, piece = dtype == B200P_F32 ? 16 : 8;
  if (H > 1 && (nv == 1 || nv == 2 || nv == 4) && aligned(o, 16) && aligned(gate, 16) && ldg % 4 == 0 && aligned(norm_w, 16) && aligned(out, piece) &&
      ld_out % 4 == 0) {
    const int64_t pairs = M * H;
    B200P_DISPATCH_DTYPE(dtype, T, {
      const auto kern = nv == 1 ? delta_out_rows_kernel<T, 1> : nv == 2 ? delta_out_rows_kernel<T, 2> : delta_out_rows_kernel<T, 4>;
      kern<<<(unsigned)((pairs + 7) / 8), 256, 0, (cudaStream_t)stream>>>(o, gate, ldg, norm_w, (T*)out, ld_out, pairs, H, eps, gate_act, out_scale);
    });
    B200P_LAUNCH_CHECK("delta_out_rows_kernel");
    return B200P_OK;
  }
  const unsigned threads = H == 1 ? (dv >= 1024 ? 256 : 128) : H >= 8 ? 256 : 32 * (unsigned)H;
  B200P_DISPATCH_DTYPE(dtype, T, (delta_out_kernel<T><<<(unsigned)M, threads, 0, (cudaStream_t)stream>>>(
      o, gate, ldg, norm_w, (T*)out, ld_out, H, dv, eps, gate_act, out_scale)));
  B200P_LAUNCH_CHECK("delta_out_kernel");
  return B200P_OK;
}
