// Gated delta rule (a linear-attention layer with a per-head matrix state S [dk, dv] that is decayed, corrected towards the
// current value along the current key and read with the current query), as four kernels over a ragged batch:
//   delta_prep_kernel         short causal convolution + silu of q, k, v; unit q / k per head; beta and decay   (per token)
//   delta_conv_commit_kernel  the convolution's carried inputs                                                   (per entry)
//   delta_scan_kernel         the recurrence, fp32, token by token; decode steps: delta_step_kernel, long entries: delta_pair_kernel  (per entry, head)
//   delta_out_kernel          per-head rms norm * weight * silu(gate)                                            (per token)
// The same kernels carry the variants other designs use: a decay per head AND key channel (a row of S each), a gate that is a
// sigmoid of a separate tensor, and the plain decayed accumulation S <- g S + k v^T (linear attention with a constant decay,
// fed by linear_attn_prep_kernel).
// Single tokens and entries of less than 32 run in one summation order, whatever kernel takes them; entries of 32 tokens and more (keys of 65 to 128
// channels, delta rule) two tokens at a time (delta_pair_kernel), which differs in the last places, so a prompt and its portions agree to rounding.
// An entry's bits depend on its own tokens alone, with one exception: beside at least as many empty entries as it has tokens, in a call that
// does not say how long its longest entry is, it goes token by token (delta_step_kernel).
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
  if (t1 <= t0 || t1 - t0 > most) {                              // (longer entries: delta_pair_kernel)
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

// Prompts of keys of 65 to 128 channels, two tokens at a time.  In the kernels above the chain of one token (dot, reduction over the lanes,
// update, dot) and the reads of shared memory for it are what bounds a CTA.  With g1, k1, q1, v1 and g2, k2, q2, v2 of two tokens and the
// state S before them,
//     u1 = b1 (v1 - S^T (g1 k1))                 o1 = S^T (g1 q1) + (q1 . k1) u1
//     u2 = b2 (v2 - S^T (g1 g2 k2) - (k2 . g2 k1) u1)      o2 = S^T (g1 g2 q2) + (q2 . g2 k1) u1 + (q2 . k2) u2
//     S <- g1 g2 S + (g2 k1) u1 + k2 u2
// so that four dot products with one state share a pass and a reduction, and 7 instead of 8 operations per element and pair are left.  The scaled
// vectors and the four scalars are the same for all columns: the threads that stage a token's row compute them.  All of it stays fp32.
// A thread holds 16 rows of FOUR columns: a 16-byte read of shared memory (four cycles of its port for a warp) serves 16 packed products; eight
// lanes share a column slot.  The exchanges for u run beside the products with the queries, those for o beside the update.
// An entry takes this path if it has at least DP_MIN tokens, whatever the others have (the exception: top of the file); a prompt whose portions are
// shorter has the bits of single tokens, which differ in the last places.
// Bound: FFMA2 with three distinct operands, one in about four cycles per scheduler (measured; scalar FFMA, two in 2.5, needs registers that are
// not there: 274 us).  us before -> now, heads of 128 x 128, decays per channel / per head: 4 x 512 tokens, 16 heads 221 -> 156 / 193 -> 152, 32
// heads 357 -> 266 / 315 -> 260 (two CTAs per SM; one: 304 / 298); 16 x 250, 32 heads 635 -> 449 / 542 -> 441; 1 x 32, 16 heads 18.6 -> 14.5.
constexpr int DP_MIN = 32, DP_CHUNK = 8, DP_COLS = 64, DP_LDK = 160;
// warps 0 .. 3 compute, 4 .. 7 stage; two CTAs per SM: registers at launch 256 x 128 = 128 x 168 + 128 x 88
constexpr int DP_TEAM = 128, DP_THREADS = 2 * DP_TEAM, DP_REGS_COMPUTE = 168, DP_REGS_STAGE = 88;
template <int MODE, int PER_SM>
__global__ void __launch_bounds__(DP_THREADS, PER_SM)
delta_pair_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ v, const float* __restrict__ beta,
                  const float* __restrict__ decay, float* __restrict__ state, const int32_t* __restrict__ cu, const int32_t* __restrict__ rows,
                  const int32_t* __restrict__ lengths, float* __restrict__ o, int H, int KH, int dk, int dv) {
  enum { K1, K2, Q1, Q2, GG, KD, KU, VECS };                   // g1 k1, g1 g2 k2, g1 q1, g1 g2 q2, g1 g2, g2 k1, k2
  constexpr int PAIRS = DP_CHUNK / 2;
  __shared__ __align__(16) float vec[2][PAIRS][VECS][DP_LDK];  // 16 rows per lane, padded by 16 bytes: the lanes' reads fall into different banks
  __shared__ __align__(16) float dots[2][PAIRS][4][4];         // k2 . kd, q1 . k1, q2 . kd, q2 . k2: a share per warp
  __shared__ __align__(16) float vs[2][DP_CHUNK][DP_COLS];
  __shared__ float bs[2][DP_CHUNK];
  const int e = blockIdx.x, h = blockIdx.y, tid = threadIdx.x & (DP_TEAM - 1), lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  const int t0 = cu[e], t1 = cu[e + 1];
  if (t1 - t0 < DP_MIN) return;
  const int row = rows[e], kh = h / (H / KH);
  if (threadIdx.x >= DP_TEAM) {
    if constexpr (PER_SM == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(DP_REGS_STAGE));
    // ===================================== staging =====================================
    // Inputs travel to registers a chunk ahead; tokens past the end are ones that change nothing.
    float pk[DP_CHUNK], pq[DP_CHUNK], pg[DP_CHUNK], pv[4], pb = 0.f;
    auto fetch = [&](int tc) {
#pragma unroll
      for (int t = 0; t < DP_CHUNK; ++t) {
        const bool ok = tc + t < t1 && tid < dk;
        const int64_t src = ((int64_t)(tc + t) * KH + kh) * dk + tid;
        pk[t] = ok ? kn[src] : 0.f;
        pq[t] = ok ? qn[src] : 0.f;
        if constexpr (MODE == 1) pg[t] = ok ? decay[((int64_t)(tc + t) * H + h) * dk + tid] : 1.f;
        else pg[t] = tc + t < t1 ? decay[(int64_t)(tc + t) * H + h] : 1.f;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int idx = tid + r * DP_TEAM, t = idx / DP_COLS, c = blockIdx.z * DP_COLS + idx % DP_COLS;
        pv[r] = tc + t < t1 && c < dv ? v[((int64_t)(tc + t) * H + h) * dv + c] : 0.f;
      }
      if (tid < DP_CHUNK) pb = tc + tid < t1 ? beta[(int64_t)(tc + tid) * H + h] : 0.f;
    };
    auto park = [&](int buf) {
      const int at = tid + (tid >> 4) * 4;
      float d[4 * PAIRS];
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) {
        const float g1 = pg[2 * p], g2 = pg[2 * p + 1], k1 = pk[2 * p], k2 = pk[2 * p + 1], q1 = pq[2 * p], q2 = pq[2 * p + 1];
        const float gg = g1 * g2, kd = g2 * k1;
        float (*w)[DP_LDK] = vec[buf][p];
        w[K1][at] = g1 * k1;
        w[K2][at] = gg * k2;
        w[Q1][at] = g1 * q1;
        w[Q2][at] = gg * q2;
        w[GG][at] = gg;
        w[KD][at] = kd;
        w[KU][at] = k2;
        d[4 * p] = k2 * kd;
        d[4 * p + 1] = q1 * k1;
        d[4 * p + 2] = q2 * kd;
        d[4 * p + 3] = q2 * k2;
      }
      // 16 sums over 32 lanes: halve the values with every exchange, lane l ends up with sum (l >> 1)
#pragma unroll
      for (int n = 8, m = 16; n >= 1; n >>= 1, m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i >= n) continue;
          const float give = up ? d[i] : d[n + i], keep = up ? d[n + i] : d[i];
          d[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
        }
      }
      d[0] += __shfl_xor_sync(0xffffffffu, d[0], 1);
      if (!(lane & 1)) dots[buf][lane >> 3][(lane >> 1) & 3][warp] = d[0];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int idx = tid + r * DP_TEAM;
        vs[buf][idx / DP_COLS][idx % DP_COLS] = pv[r];
      }
      if (tid < DP_CHUNK) bs[buf][tid] = pb;
    };
    fetch(t0);
    park(0);
    fetch(t0 + DP_CHUNK);
    __syncthreads();
    int buf = 0;
    for (int tc = t0; tc < t1; tc += DP_CHUNK, buf ^= 1) {      // (the other buffer was last read in the previous iteration)
      if (tc + DP_CHUNK < t1) park(buf ^ 1);
      if (tc + 2 * DP_CHUNK < t1) fetch(tc + 2 * DP_CHUNK);
      __syncthreads();
    }
    return;
  }
  if constexpr (PER_SM == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DP_REGS_COMPUTE));
  // ===================================== recurrence ==================================
  const int l = tid & 7, slot = tid >> 3, j0 = blockIdx.z * DP_COLS + 4 * slot;    // this thread's columns j0 .. j0 + 3, rows 16 l .. 16 l + 15
  const bool vec4 = (dv & 3) == 0 && (reinterpret_cast<uintptr_t>(state) & 15) == 0 && j0 + 3 < dv;
  float* sp = state + (((int64_t)row * H + h) * dk + 16 * l) * dv + j0;
  const bool fresh = lengths[row] == 0;
  float2 S[4][8];                                              // [column][row pair]
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int r = 2 * i + b;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!fresh && 16 * l + r < dk) {
        const float* s0 = sp + (int64_t)r * dv;
        if (vec4) x = *reinterpret_cast<const float4*>(s0);
        else {
          if (j0 < dv) x.x = s0[0];
          if (j0 + 1 < dv) x.y = s0[1];
          if (j0 + 2 < dv) x.z = s0[2];
          if (j0 + 3 < dv) x.w = s0[3];
        }
      }
      (b ? S[0][i].y : S[0][i].x) = x.x;
      (b ? S[1][i].y : S[1][i].x) = x.y;
      (b ? S[2][i].y : S[2][i].x) = x.z;
      (b ? S[3][i].y : S[3][i].x) = x.w;
    }
  const int jo = j0 + (l & 3);                                 // the column whose outputs this lane writes
  __syncthreads();
  int buf = 0;
  for (int tc = t0; tc < t1; tc += DP_CHUNK, buf ^= 1) {
    auto step = [&](int p) {
      const float* w = &vec[buf][p][0][20 * l];
      // this thread's rows of two dot products with the four columns
      auto dot2 = [&](int s0, float (&r1)[4], float (&r2)[4]) {
        float2 a[2][4];
#pragma unroll
        for (int c = 0; c < 4; ++c) a[0][c] = a[1][c] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const float4 x = *reinterpret_cast<const float4*>(w + (s0 + s) * DP_LDK + 4 * i);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              a[s][c] = __ffma2_rn(S[c][2 * i], make_float2(x.x, x.y), a[s][c]);
              a[s][c] = __ffma2_rn(S[c][2 * i + 1], make_float2(x.z, x.w), a[s][c]);
            }
          }
#pragma unroll
        for (int c = 0; c < 4; ++c) r1[c] = a[0][c].x + a[0][c].y, r2[c] = a[1][c].x + a[1][c].y;
      };
      // over the eight lanes: lane l < 4 gets the first product's sum of column l, lane l + 4 the second's
      auto reduce = [&](const float (&r1)[4], const float (&r2)[4]) {
        const bool b4 = (l & 4) != 0, b2 = (l & 2) != 0, b1 = (l & 1) != 0;
        float r[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) r[c] = (b4 ? r2[c] : r1[c]) + __shfl_xor_sync(0xffffffffu, b4 ? r1[c] : r2[c], 4);
#pragma unroll
        for (int c = 0; c < 2; ++c) r[c] = (b2 ? r[c + 2] : r[c]) + __shfl_xor_sync(0xffffffffu, b2 ? r[c] : r[c + 2], 2);
        return (b1 ? r[1] : r[0]) + __shfl_xor_sync(0xffffffffu, b1 ? r[0] : r[1], 1);
      };
      float r1[4], r2[4], y1[4], y2[4];
      dot2(K1, r1, r2);
      const float sk = reduce(r1, r2);
      dot2(Q1, y1, y2);                                        // (beside the exchanges of the sums for u)
      auto dot_of = [&](int d) {
        const float4 x = *reinterpret_cast<const float4*>(dots[buf][p][d]);
        return (x.x + x.y) + (x.z + x.w);
      };
      const float k2kd = dot_of(0), q1k1 = dot_of(1), q2kd = dot_of(2), q2k2 = dot_of(3), b1 = bs[buf][2 * p], b2 = bs[buf][2 * p + 1];
      const float4 v1 = *reinterpret_cast<const float4*>(&vs[buf][2 * p][4 * slot]), v2 = *reinterpret_cast<const float4*>(&vs[buf][2 * p + 1][4 * slot]);
      const float va[4] = {v1.x, v1.y, v1.z, v1.w}, vb[4] = {v2.x, v2.y, v2.z, v2.w};
      float u1[4], u2[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float s1 = __shfl_sync(0xffffffffu, sk, c, 8), s2 = __shfl_sync(0xffffffffu, sk, c + 4, 8);
        u1[c] = b1 * (va[c] - s1);
        u2[c] = b2 * (vb[c] - fmaf(k2kd, u1[c], s2));
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 g = *reinterpret_cast<const float4*>(w + GG * DP_LDK + 4 * i), kd = *reinterpret_cast<const float4*>(w + KD * DP_LDK + 4 * i);
        const float4 ku = *reinterpret_cast<const float4*>(w + KU * DP_LDK + 4 * i);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 ua = make_float2(u1[c], u1[c]), ub = make_float2(u2[c], u2[c]);
          S[c][2 * i] = __ffma2_rn(make_float2(ku.x, ku.y), ub, __ffma2_rn(make_float2(kd.x, kd.y), ua, __fmul2_rn(S[c][2 * i], make_float2(g.x, g.y))));
          S[c][2 * i + 1] = __ffma2_rn(make_float2(ku.z, ku.w), ub, __ffma2_rn(make_float2(kd.z, kd.w), ua, __fmul2_rn(S[c][2 * i + 1], make_float2(g.z, g.w))));
        }
      }
      const float sq = reduce(y1, y2);                         // (beside the update)
      const bool c2 = (l & 2) != 0, c1 = (l & 1) != 0;
      const float ua = c2 ? (c1 ? u1[3] : u1[2]) : (c1 ? u1[1] : u1[0]), ub = c2 ? (c1 ? u2[3] : u2[2]) : (c1 ? u2[1] : u2[0]);
      const float out = l < 4 ? fmaf(q1k1, ua, sq) : fmaf(q2k2, ub, fmaf(q2kd, ua, sq));
      const int t = tc + 2 * p + (l >> 2);
      if (jo < dv && t < t1) o[((int64_t)t * H + h) * dv + jo] = out;
    };
    if (t1 - tc >= DP_CHUNK) {
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) step(p);
    } else {
#pragma unroll 1
      for (int p = 0; tc + 2 * p < t1; ++p) step(p);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int r = 2 * i + b;
      if (16 * l + r >= dk) continue;
      const float4 x = b ? make_float4(S[0][i].y, S[1][i].y, S[2][i].y, S[3][i].y) : make_float4(S[0][i].x, S[1][i].x, S[2][i].x, S[3][i].x);
      float* s0 = sp + (int64_t)r * dv;
      if (vec4) *reinterpret_cast<float4*>(s0) = x;
      else {
        if (j0 < dv) s0[0] = x.x;
        if (j0 + 1 < dv) s0[1] = x.y;
        if (j0 + 2 < dv) s0[2] = x.z;
        if (j0 + 3 < dv) s0[3] = x.w;
      }
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
static void delta_scan_launch(int64_t tokens, int64_t longest, int nb, cudaStream_t st, const float* qn, const float* kn, const float* v, const float* beta,
                              const float* decay, float* state, const int32_t* cu, const int32_t* rows, const int32_t* lengths,
                              float* o, int H, int KH, int dk, int dv) {
#define DELTA_STEP(DKP)                                                                                                          \
  delta_step_kernel<DKP, MODE><<<dim3((unsigned)nb, (unsigned)H, (unsigned)((dv + dt_cols(DKP) - 1) / dt_cols(DKP))), DT_THREADS, 0, st>>>( \
      qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv)
#define DELTA_SCAN(DKP, LANES, PER_SM)                                                                                           \
  launch_pdl_opt(pairs && pdl_enabled_gemm(), delta_scan_kernel<DKP, MODE, LANES, PER_SM>,                                        \
                 dim3((unsigned)nb, (unsigned)H, (unsigned)((dv + 2 * ds_slots(DKP) - 1) / (2 * ds_slots(DKP)))), dim3(LANES * ds_slots(DKP)), 0, st, \
                 qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv, pairs ? DP_MIN - 1 : INT32_MAX)
  // The step kernel for decode steps, and for as many tokens per entry as it keeps up with the scan (us, step / scan): 128 x 128, 16
  // entries of 1 / 2 / 4 tokens, 32 heads, 21.7 / 23.1, 27.1 / 25.3, 32.0 / 29.2; 64 x 64, 32 heads, of 2 / 4 / 8, 6.8 / 8.8, 7.9 / 9.6,
  // 10.2 / 11.4, but with 16 heads 4.3 / 4.6, 5.1 / 5.0, 7.3 / 6.4; 32 x 64, 16 heads, of 2 / 4, 3.4 / 3.5, 4.2 / 3.9; 256 x 256, 8 heads,
  // 4 entries of 16 / 64, 20 / 20, 58 / 50.
  // The plain accumulation of keys above 128 takes it at any length (16 x 250 tokens of 256 x 256: 407 / 678; 4 x 512: 315 / 309).
  const int most = dk > 128 ? 8 : dk > 64 ? 1 : dk > 32 ? 4 : 2;
  const bool by_pairs = MODE != 2 && dk > 64 && dk <= 128;                   // entries of DP_MIN tokens and more
  const bool few = (tokens > 0 && tokens <= most * (int64_t)nb && !(by_pairs && longest >= DP_MIN)) || (MODE == 2 && dk > 128);
  // 128 rows: one CTA per SM takes eight lanes per column and the shortest chain (4 x 512 tokens, 16 heads, decays per channel / per
  // head: 220 / 193 us, the former four-lane kernel 280 / 206); more CTAs than SMs take four (32 heads 379 / 346 -> 356 / 317; 16 x 250
  // tokens 672 / 594 -> 637 / 544).
  const bool crowded = (int64_t)nb * H * ((dv + 63) / 64) > sm_count();
  // Entries of DP_MIN tokens and more two tokens at a time, the shorter ones by the launch behind it, which needs nothing of it: it may start at
  // once (its inputs were complete when the first began), and one of its CTAs waits for the first launch, so that what follows waits for both.
  // (Only one: with every CTA waiting, those that do not fit beside the first launch started when it had ended: 15 entries of one token and one
  // of 40, 32 heads, decays per head / channel 43.7 / 45.7 -> 30 / 30.5 us, the scan alone 38 / 42.)  The long ones first: the short ones of such a
  // batch come with their tail.  A call that knows its longest entry to be short is spared the first launch: 16 entries of 4 tokens, 16 heads 14.4 ->
  // 13.3 us.
  const bool pairs = by_pairs && !few && (tokens == 0 || tokens >= DP_MIN) && (longest == 0 || longest >= DP_MIN);
  if constexpr (MODE != 2) {
    const auto pair_kernel = crowded ? delta_pair_kernel<MODE, 2> : delta_pair_kernel<MODE, 1>;
    if (pairs)
      pair_kernel<<<dim3((unsigned)nb, (unsigned)H, (unsigned)((dv + DP_COLS - 1) / DP_COLS)), DP_THREADS, 0, st>>>(
          qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv);
  }
  if (dk > 256) { if (few) DELTA_STEP(512); else DELTA_SCAN(512, 16, 1); }
  else if (dk > 128) { if (few) DELTA_STEP(256); else DELTA_SCAN(256, 8, 1); }
  else if (dk > 64) { if (few) DELTA_STEP(128); else if (crowded) DELTA_SCAN(128, 4, 2); else DELTA_SCAN(128, 8, 1); }
  else if (dk > 32) { if (few) DELTA_STEP(64); else DELTA_SCAN(64, 4, 1); }
  else { if (few) DELTA_STEP(32); else DELTA_SCAN(32, 4, 1); }
#undef DELTA_STEP
#undef DELTA_SCAN
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
  launch(tokens, longest, nb, st, qn, kn, v, beta, decay, state, cu, rows, lengths, o, H, KH, dk, dv);
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
