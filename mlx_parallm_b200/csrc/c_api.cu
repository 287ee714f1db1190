// C-ABI glue: the path dispatchers of b200p_qmm / b200p_attn (error plumbing and device checks: runtime.cu).
#include <float.h>
#include <stdlib.h>

#include "common.cuh"

namespace b200p {

int sm_count();
// implemented in the kernel translation units
int qmv_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N,
               int64_t K, int64_t ldx, int64_t ldy, int gs, int bits, int dtype, int epi, int flags, cudaStream_t st);
bool qmm_tc_supported(int64_t M, int64_t N, int64_t K, int gs, int bits, int dtype, int epi);
int qmm_tc_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N,
                  int64_t K, int64_t ldx, int64_t ldy, int bits, int dtype, int epi, int flags, void* ws, size_t ws_bytes,
                  int64_t row0, cudaStream_t st);
size_t qmm_tc_workspace_bytes(int64_t M, int64_t N, int64_t K);
bool qmm_sk_supported(int64_t M, int64_t N, int64_t K, int bits, int epi, const void* y, int64_t ldy);
int qmm_sk_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N,
                  int64_t K, int64_t ldx, int64_t ldy, int bits, int dtype, int flags, cudaStream_t st);
void qmm_tc_set_min_m(int m);
bool qmv_mma_supported(int64_t M, int64_t N, int64_t K, int gs, int bits, int dtype, int epi);
bool qmm_mma_supported(int64_t M, int64_t N, int64_t K, int gs, int bits, int dtype, int epi, const void* y, int64_t ldy);
int qmm_mma_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K,
                   int64_t ldx, int64_t ldy, int dtype, int flags, cudaStream_t st);
bool qmm_wide_supported(int64_t M, int64_t N, int64_t K, int bits, int epi, const void* s, const void* b, const void* y, int64_t ldy);
int qmm_wide_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx,
                    int64_t ldy, int bits, int dtype, int epi, int flags, void* ws, size_t ws_bytes, cudaStream_t st);
bool qmv_ring_supported(int64_t M, int64_t N, int64_t K, int gs, int bits, int dtype, int epi);
int qmv_ring_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx,
                    int64_t ldy, int bits, int dtype, int epi, int flags, cudaStream_t st);
int qmv_mma_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K,
                   int64_t ldx, int64_t ldy, int dtype, int epi, int flags, cudaStream_t st);
int attn_generic_launch(const void* q, const void* kc, const void* vc, const int32_t* lengths, void* out,
                        int64_t B, int64_t L, int Hq, int Hkv, int D, int64_t Tcap, float scale, int dtype,
                        int out_perm, cudaStream_t st);
bool attn_decode_supported(int64_t L, int Hq, int Hkv, int D, int dtype);
int attn_decode_launch(const void* q, const void* kc, const void* vc, const int32_t* lengths, void* out,
                       int64_t B, int64_t L, int Hq, int Hkv, int D, int64_t Tcap, float scale, int dtype,
                       int out_perm, void* ws, size_t ws_bytes, cudaStream_t st);
size_t attn_decode_workspace_bytes(int64_t B, int64_t L, int Hq, int D);
bool attn_prefill_supported(int64_t L, int Hq, int Hkv, int D, int dtype);
bool attn_prefill_tc_supported(int64_t L, int Hq, int Hkv, int D, int dtype);
int attn_prefill_tc_launch(const void* q, const void* kc, const void* vc, const int32_t* lengths, void* out, int64_t B, int64_t L,
                           int Hq, int Hkv, int D, int64_t Tcap, float scale, int dtype, int out_perm, cudaStream_t st);
int attn_prefill_launch(const void* q, const void* kc, const void* vc, const int32_t* lengths, void* out, int64_t B, int64_t L,
                        int Hq, int Hkv, int D, int64_t Tcap, float scale, int dtype, int out_perm, cudaStream_t st);

static const bool g_use_sk = [] { const char* e = getenv("B200P_QMM_SK"); return !e || atoi(e) != 0; }();
static int g_qmm_path = 0;   // 0 auto, 1 CUDA-core gemv, 2 tcgen05 tiles, 3 mma.sync gemv, 4 mma.sync small-matrix GEMM
// pipeline-free mma.sync GEMM (qmm_mma.cu) for the accumulate epilogue above the GEMV's rows: matrices up to this many weights
// (q|k|v 25 M and o_proj 17 M of Llama-3-8B, every tensor-parallel shard; down_proj 59 M and gate|up stay on the tile kernels)
static long long g_mma_max_weights = [] { const char* e = getenv("B200P_MMA_MAX_WEIGHTS"); return e ? atoll(e) : (1ll << 25); }();
// ... and up to this many rows: measured against the tile kernels it wins at 8 and 16
// rows (q|k|v 6.2 vs 7.2 us, o_proj 4.3 vs 5.7, TP=8 shards 2.6-4.1 vs 3.8-5.3), ties at 32 and loses at 64, where it is bound
// by the mma.sync rate (q|k|v 14.6 vs 8.9 us)
static int g_gemv_silu_max_m = [] { const char* e = getenv("B200P_GEMV_SILU_MAX_M"); return e ? atoi(e) : 0; }();
static int g_mma_max_m = [] { const char* e = getenv("B200P_MMA_MAX_M"); return e ? atoi(e) : 16; }();
// Auto rule for the mma.sync GEMV, from the measured three-way sweep (us per
// launch in a CUDA graph): it wins where the tile kernel's fixed cost dominates -- M <= 4 and matrices up to ~32 M weights
// (q|k|v 6.4 vs 8.4 us, o_proj 5.2 vs 6.5 us at M = 1) -- and loses on the big streams (gate|up 23.9 vs 22.4 us) and as M
// grows (its activation loads are per 16-row warp, not shared through shared memory).  The CUDA-core GEMV loses everywhere.
static int g_gemv_max_m = [] { const char* e = getenv("B200P_GEMV_MAX_M"); return e ? atoi(e) : 4; }();
static long long g_gemv_max_weights = [] { const char* e = getenv("B200P_GEMV_MAX_WEIGHTS"); return e ? atoll(e) : (1ll << 25); }();
// The TMA-ring GEMV (qmv_ring.cu), measured against the kernels it replaces (us per launch in a CUDA graph over weight copies larger than
// L2): whole-tile epilogues gate|up 28672 x 4096 f16 16.2 against 21.7 at M = 1, 18.5 against 22.1 at M = 6 (bf16, direct dequantisation on both sides, 19.0 / 25.9, 21.3 /
// 26.1); 57344 x 8192 8-bit 82 against 92; accumulating o_proj 4096 x 4096 5.2 against 6.0 at M = 1, 5.8 against 6.9 at M = 4, down_proj
// 4096 x 14336 11.2 against 13.2 at M = 1, 12.2 against 13.9 at M = 2 but 13.2 against 12.1 at M = 3; in 8 bits it loses there (direct dequantisation: 62 against
// 53 us, 8192 x 28672 bf16).  Matrices under 8 M weights stay on the kernels without rings.
static bool qmv_ring_preferred(int64_t M, int64_t N, int64_t K, int bits, int epi) {
  if (N * K < (1ll << 23)) return false;
  if (epi != B200P_EPI_ADD_RESIDUAL) return M <= (bits == 4 ? 6 : 8);
  return bits == 4 && M <= 4 && N * K <= (M <= 2 ? 2 : 1) * g_gemv_max_weights;
}
static int g_attn_path = 0;  // 0 auto, 1 generic, 2 tensor, 3 tcgen05 prefill at any size, 4 mma.sync prefill at any size
}  // namespace b200p

using namespace b200p;

extern "C" int b200p_qmm_set_min_tensor_m(int m) {
  B200P_REQUIRE(m >= 1, B200P_ERR_ARG, "min tensor-path M must be >= 1");
  qmm_tc_set_min_m(m);
  return B200P_OK;
}

extern "C" int b200p_qmm_set_path(int path) {
  B200P_REQUIRE(path >= 0 && path <= 6 && path != 5, B200P_ERR_ARG, "path must be 0..4 or 6");
  g_qmm_path = path;
  return B200P_OK;
}

extern "C" int b200p_attn_set_path(int path) {
  B200P_REQUIRE(path >= 0 && path <= 4, B200P_ERR_ARG, "path must be 0..4");
  g_attn_path = path;
  return B200P_OK;
}

extern "C" size_t b200p_qmm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  return qmm_tc_workspace_bytes(M, N, K);
}

extern "C" int b200p_qmm_tensor_supported(int64_t M, int64_t N, int64_t K, int group_size, int bits, int dtype,
                                          int epilogue) {
  return qmm_tc_supported(M, N, K, group_size, bits, dtype, epilogue) ? 1 : 0;
}

extern "C" int b200p_qmm(const void* x, const uint32_t* w, const void* scales, const void* biases, void* y,
                         int64_t M, int64_t N, int64_t K, int64_t ldx, int64_t ldy, int group_size, int bits,
                         int dtype, int epilogue_flags, void* workspace, size_t workspace_bytes, void* stream) {
  const int epilogue = epilogue_flags & 0xff, flags = epilogue_flags & ~0xff;
  B200P_REQUIRE((flags & ~(B200P_X_PERM8 | B200P_Y_PERM8 | B200P_W_SMALLSCALE)) == 0, B200P_ERR_ARG, "unknown layout flags 0x%x", flags);
  B200P_REQUIRE(!(flags & B200P_X_PERM8) || (bits == 4 && dtype != B200P_F32), B200P_ERR_ARG,
                "B200P_X_PERM8 is the layout of 16-bit activations for 4-bit weights");
  B200P_REQUIRE(!(flags & B200P_Y_PERM8) || ((epilogue == B200P_EPI_STORE || epilogue == B200P_EPI_SILU_MUL) && dtype != B200P_F32),
                B200P_ERR_ARG, "B200P_Y_PERM8 applies to 16-bit outputs (STORE, SILU_MUL)");
  B200P_REQUIRE(x && w && scales && biases && y, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE(bits == 4 || bits == 8, B200P_ERR_ARG, "bits must be 4 or 8, got %d", bits);
  B200P_REQUIRE(M >= 0 && N > 0 && K > 0 && N % 2 == 0, B200P_ERR_ARG, "bad shape M=%lld N=%lld K=%lld (N must be even)",
                (long long)M, (long long)N, (long long)K);
  B200P_REQUIRE(group_size >= 32 && group_size % 32 == 0 && K % group_size == 0, B200P_ERR_ARG,
                "group_size %d must be a multiple of 32 dividing K=%lld", group_size, (long long)K);
  B200P_REQUIRE(epilogue >= 0 && epilogue <= 3, B200P_ERR_ARG, "bad epilogue %d", epilogue);
  B200P_REQUIRE(dtype >= 0 && dtype <= 2, B200P_ERR_ARG, "bad dtype %d", dtype);
  const size_t xs = dtype == B200P_F32 ? 4 : 2;
  B200P_REQUIRE(aligned(x, 16) && aligned(w, 16) && (ldx * xs) % 16 == 0 && ldx >= K, B200P_ERR_ALIGN,
                "x rows and w must be 16-byte aligned (ldx=%lld)", (long long)ldx);
  B200P_REQUIRE((K * bits / 8) % 16 == 0, B200P_ERR_ALIGN, "packed weight rows must be 16-byte multiples (K=%lld)",
                (long long)K);
  B200P_REQUIRE(ldy >= (epilogue == B200P_EPI_SILU_MUL ? N / 2 : N), B200P_ERR_ARG, "ldy too small");
  if (M == 0) return B200P_OK;
  PdlClass pdl_cls(64);
  cudaStream_t st = (cudaStream_t)stream;
  const bool ring_ok = qmv_ring_supported(M, N, K, group_size, bits, dtype, epilogue) && aligned(scales, 16) && aligned(biases, 16) &&
                       aligned(y, epilogue == B200P_EPI_STORE || epilogue == B200P_EPI_SILU_MUL ? 2 : 4);
  // The ring and the wide kernel need neither a workspace nor y rows of whole words (the wide one uses a workspace that it is given for a short last
  // round, whose rows are then summed in parts of K); a call that the kernels they stand in for would refuse goes on to those, and is refused there.
  const bool f32out = epilogue == B200P_EPI_STORE_F32 || epilogue == B200P_EPI_ADD_RESIDUAL;
  const bool tile_args = workspace && workspace_bytes >= qmm_tc_workspace_bytes(M, N, K) && aligned(workspace, 16) && aligned(y, 4) &&
                         (f32out || ldy % 2 == 0);
  const bool sk_args = g_use_sk && qmm_sk_supported(M, N, K, bits, epilogue, y, ldy);
  if (g_qmm_path == 6) B200P_REQUIRE(ring_ok, B200P_ERR_ARG, "ring GEMV forced but unsupported for this call");
  if (ring_ok && (g_qmm_path == 6 || (g_qmm_path == 0 && (tile_args || sk_args) && qmv_ring_preferred(M, N, K, bits, epilogue)))) {
    const int rc = qmv_ring_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, bits, dtype, epilogue, flags, st);
    if (rc <= 0) return rc;                      // 1: x does not fit beside the rings
    B200P_REQUIRE(g_qmm_path != 6, B200P_ERR_ARG, "ring GEMV forced but x does not fit");
  }
  // (SILU_MUL through the GEMV: 16-bit output, PERM8 allowed; the other GEMV epilogues write fp32 in the natural order)
  const bool mma_ok = qmv_mma_supported(M, N, K, group_size, bits, dtype, epilogue) && aligned(w, 32) &&
                      (epilogue == B200P_EPI_SILU_MUL ? aligned(y, 2) : (aligned(y, 4) && !(flags & B200P_Y_PERM8)));
  if (g_qmm_path == 3) B200P_REQUIRE(mma_ok, B200P_ERR_ARG, "mma.sync GEMV forced but unsupported for this call");
  // up to two rows the GEMV also wins on matrices of twice that size (down_proj 4096 x 14336: 12.8 vs 14.1 us at M = 1);
  // gate|up (117 M weights) stays on the tile kernel
  // gate|up with the fused silu(gate) * up epilogue through the GEMV (rows paired gate / up, no K split): up to
  // B200P_GEMV_SILU_MAX_M rows, any size; 0 = never (the default)
  if (mma_ok && epilogue == B200P_EPI_SILU_MUL && g_qmm_path == 0 && M <= g_gemv_silu_max_m)
    return qmv_mma_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, dtype, epilogue, flags, st);
  if (mma_ok && (g_qmm_path == 3 || (g_qmm_path == 0 && epilogue != B200P_EPI_SILU_MUL && M <= g_gemv_max_m &&
                                     N * K <= (M <= 2 ? 2 * g_gemv_max_weights : g_gemv_max_weights))))
    return qmv_mma_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, dtype, epilogue, flags, st);
  const bool gm_ok = qmm_mma_supported(M, N, K, group_size, bits, dtype, epilogue, y, ldy) && aligned(w, 32);
  if (g_qmm_path == 4) B200P_REQUIRE(gm_ok, B200P_ERR_ARG, "mma.sync small-matrix GEMM forced but unsupported for this call");
  if (gm_ok && (g_qmm_path == 4 || (g_qmm_path == 0 && M > g_gemv_max_m && M <= g_mma_max_m && N * K <= g_mma_max_weights)))
    return qmm_mma_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, dtype, flags, st);
  const bool tc_ok = qmm_tc_supported(M, N, K, group_size, bits, dtype, epilogue);
  if (g_qmm_path == 2) {
    B200P_REQUIRE(tc_ok, B200P_ERR_ARG, "tensor path forced but unsupported for this call");
  }
  // more than 128 tokens: one 128-row weight block against up to 256 tokens (the rule and its figures: qmm_wide.cu)
  if (tc_ok && g_qmm_path != 1 && (tile_args || sk_args) && qmm_wide_supported(M, N, K, bits, epilogue, scales, biases, y, ldy))
    return qmm_wide_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, bits, dtype, epilogue, flags, tile_args ? workspace : nullptr,
                           workspace_bytes, st);
  // fp32 accumulate epilogue: the stream-K kernel (partial tiles summed by TMA reduce-adds, no workspace, no tail);
  // B200P_QMM_SK=0 keeps everything on the whole-tile kernel (A/B measurements)
  if (tc_ok && g_qmm_path != 1 && sk_args)
    return qmm_sk_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, bits, dtype, flags, st);
  if (tc_ok && g_qmm_path != 1) {
    B200P_REQUIRE(workspace && workspace_bytes >= qmm_tc_workspace_bytes(M, N, K), B200P_ERR_ARG,
                  "tensor path needs a workspace of %zu bytes", qmm_tc_workspace_bytes(M, N, K));
    return qmm_tc_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, bits, dtype, epilogue, flags, workspace,
                         workspace_bytes, 0, st);
  }
  return qmv_launch(x, w, scales, biases, y, M, N, K, ldx, ldy, group_size, bits, dtype, epilogue, flags, st);
}

extern "C" size_t b200p_attn_workspace_bytes(int64_t B, int64_t L, int Hq, int D) {
  return attn_decode_workspace_bytes(B, L, Hq, D);
}

extern "C" int b200p_attn(const void* q, const void* kcache, const void* vcache, const int32_t* lengths, void* out,
                          int64_t B, int64_t L, int Hq, int Hkv, int D, int64_t Tcap, float scale, int dtype,
                          int flags, void* workspace, size_t workspace_bytes, void* stream) {
  B200P_REQUIRE(q && kcache && vcache && lengths && out, B200P_ERR_ARG, "null pointer");
  B200P_REQUIRE((flags & ~B200P_OUT_PERM8) == 0, B200P_ERR_ARG, "unknown flags 0x%x", flags);
  const int out_perm = (flags & B200P_OUT_PERM8) ? 1 : 0;
  B200P_REQUIRE(!out_perm || dtype != B200P_F32, B200P_ERR_ARG, "B200P_OUT_PERM8 is a 16-bit layout");
  B200P_REQUIRE(Hq > 0 && Hkv > 0 && Hq % Hkv == 0, B200P_ERR_ARG, "bad head counts %d/%d", Hq, Hkv);
  B200P_REQUIRE(B >= 0 && L >= 0 && Tcap > 0, B200P_ERR_ARG, "bad shape");
  B200P_REQUIRE(dtype >= 0 && dtype <= 2, B200P_ERR_ARG, "bad dtype %d", dtype);
  if (B * L == 0) return B200P_OK;
  PdlClass pdl_cls(8);
  cudaStream_t st = (cudaStream_t)stream;
  const bool tc_ok = attn_decode_supported(L, Hq, Hkv, D, dtype);
  const bool pf_ok = attn_prefill_supported(L, Hq, Hkv, D, dtype);
  if (g_attn_path == 2) B200P_REQUIRE(tc_ok || pf_ok, B200P_ERR_ARG, "tensor attention forced but unsupported for this call");
  // Prompts run on tcgen05 except the smallest: a call of at most 64 new tokens over a cache of at most 256 positions that fills
  // the SMs at most twice with mma.sync CTAs (64 queries of one head each) is shorter than the tcgen05 kernel's set-up (32 / 8
  // heads, B=1, empty cache, L=2 / 16 / 64: 4.1 / 4.4 / 4.9 against 6.9 / 6.9 / 9.0 us).  Beyond it tcgen05 wins at every size: 1000
  // cached positions 18.6 against 27.7 us (L=2, B=1), L=200 at B=8 19.6 against 33.5 us, L=777 at 8000 cached 125 against 568 us.
  // (Its softmax masks and takes the maximum before it scales, so a scale that is no normal positive number -- negative, zero, or so
  // small that a masked score's -inf would be lost -- stays on the mma.sync kernel, which scales first.)
  const float scale_log2e = scale * 1.4426950408889634f;
  const bool pf_scale = scale_log2e >= FLT_MIN && scale_log2e <= FLT_MAX;
  const bool pf_small = L <= 64 && Tcap <= 256 && B * Hq <= 2 * (int64_t)sm_count();
  // (What does not fit its 32-bit row numbers stays there too, to be run or refused as it is.)
  const bool pf_fits = L < (1ll << 30) && Tcap < (1ll << 31) - 128 && B < 65536 && Hq < 65536;
  if (g_attn_path != 1 && g_attn_path != 4 && pf_scale && pf_fits && (g_attn_path == 3 || !pf_small) && attn_prefill_tc_supported(L, Hq, Hkv, D, dtype))
    return attn_prefill_tc_launch(q, kcache, vcache, lengths, out, B, L, Hq, Hkv, D, Tcap, scale, dtype, out_perm, st);
  if (pf_ok && g_attn_path != 1)
    return attn_prefill_launch(q, kcache, vcache, lengths, out, B, L, Hq, Hkv, D, Tcap, scale, dtype, out_perm, st);
  if (tc_ok && g_attn_path != 1) {
    B200P_REQUIRE(workspace && workspace_bytes >= attn_decode_workspace_bytes(B, L, Hq, D), B200P_ERR_ARG,
                  "attention needs a workspace of %zu bytes", attn_decode_workspace_bytes(B, L, Hq, D));
    return attn_decode_launch(q, kcache, vcache, lengths, out, B, L, Hq, Hkv, D, Tcap, scale, dtype, out_perm, workspace,
                              workspace_bytes, st);
  }
  return attn_generic_launch(q, kcache, vcache, lengths, out, B, L, Hq, Hkv, D, Tcap, scale, dtype, out_perm, st);
}
