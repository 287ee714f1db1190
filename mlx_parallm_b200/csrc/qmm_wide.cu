// Tensor-core path of b200p_qmm for more than 128 tokens: W4A16 / W8A16 GEMM on tcgen05 with up to 256 tokens per tile.
//
//   Y[tok, n] (+)= sum_k X[tok, k] * (q[n,k] * s[n, k/64] + b[n, k/64])
//
// The manner is that of qmm_tc.cu (weights are the MMA's 128-row A operand, dequantised by 16 warps straight into TMEM; tokens are
// the N side, TMA-fed), the tile is not: ONE block of 128 weight rows against up to 256 tokens instead of two blocks against 128.
// Both are 512 tensor-core cycles per 64 k, but the wide tile dequantises half as many weights for them.  The dequantisers need 350 to
// 600 cycles per 256 rows x 64 k (more for 8-bit codes in bf16), which bounded the square tile at 0.6 of the tensor peak;
// here they have twice the time.
//
//   TMEM: D in columns 0..255 (tokens of half 0 at 0, of half 1 at 128), A ring of 8 k-blocks in columns 256..511
//   two MMA-issuing warps, one per half of the tokens: the next tile's first half starts while the second is still being stored
//   SILU_MUL: the 128 rows of a block are, per lane quarter, 16 gate rows and their 16 up rows: a warp holds both, one shuffle apart
//
// Draining a tile (TMEM -> registers -> y) stalls the tensor core, so all 20 warps that can do it share it: 5 per lane quarter, 3 or 4
// groups of 16 tokens each.  The dequantisers first prepare their next k-block of the FOLLOWING tile, so that the tensor core has four
// k-blocks waiting when the accumulators are free again.  (Draining with the four epilogue warps alone cost a third of the tile's time:
// gate|up at 4096 tokens 1017 us.)
//
// Schedule: epilogues that need whole sums take whole tiles round robin (CTAs running at one time share
// the larger operand through L2); the accumulating epilogue does the same as far as whole rounds go, cuts what is left into equal
// ranges of (tile, K stage) and adds its sums with cp.reduce.async.bulk.tensor (as qmm_sk.cu does).  Every mbarrier wait is bounded; one that runs out is reported.
//
// Measured (bf16 or f16, us, before / after): gate|up 28672 x 4096 4-bit 62 / 51 at 201 tokens, 64 / 57 at 256, 235 / 208 at 1000, 500 / 390 at
// 2048, 1261 / 780 at 4096 (1.2 PFLOP/s); 57344 x 8192 8-bit (bf16, with the fp32 dequantisation of dequant.cuh) 356 / 206 at 201, 1201 / 790 at 1000; down 4096 x 14336 405 / 359 at 4096.
//
// warp roles (768 threads): 0..15 dequantisers (group g = 4 warps takes k-blocks g, g + 4, ...; thread = weight row), 16..19 epilogue,
// 20 TMA producer of weights, scales and biases, 21 TMA producer of X, 22 / 23 MMA issuers.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "dequant.cuh"
#include "tc_ptx.cuh"

namespace b200p {

int sm_count();
bool pdl_enabled_gemm();
int qmm_tc_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx,
                  int64_t ldy, int bits, int dtype, int epi, int flags, void* ws, size_t ws_bytes, int64_t row0, cudaStream_t st);

namespace wide {

constexpr int DQ_WARPS = 16, EPI_WARPS = 4;       // (DQ_WARPS / 4 = groups of dequantisers)
constexpr int WARP_W = DQ_WARPS + EPI_WARPS, WARP_X = WARP_W + 1, WARP_MMA = WARP_X + 1;
constexpr int THREADS = (WARP_MMA + 2) * 32;
// registers at launch: 768 x 80 = 512 x 96 + 256 x 48
constexpr int REGS_DQ = 96, REGS_OTHER = 48;
constexpr int MAX_TN = 256;
constexpr int W_STAGE_BYTES = 128 * 128;          // 128 rows x 128 packed bytes
constexpr int SB_TILE_BYTES = 128 * 16;           // 128 rows x 8 k-blocks x 2 bytes
constexpr int NSB = 2, A_SLOTS = 8, X_SLOTS = 4, MAX_STAGES = 6;
constexpr uint32_t A_COL0 = 256;
constexpr int WORKERS = 1 + DQ_WARPS / 4;         // warps per lane quarter that drain a tile: the epilogue's and the four dequantisers
constexpr int ADD_TOK = 8, STAGE_OUT_BYTES = ADD_TOK * 128 * 4;      // staging of four warps' partial sums: 8 tokens x 128 rows
constexpr int SMEM_BUDGET = 227 * 1024;

struct Params {
  void* y;
  int M_tok, N, epi, y_perm;
  int TN, H0, H1;                                 // tokens per tile and of its two halves (multiples of 16)
  int64_t ldy;
  int num_st;                                     // stages along K
  int tiles_m, row_blocks, items, row_fast;       // token tiles, row blocks, all tiles and their order (tile_of)
  int w_stages;
  int* wait_word;                                 // where a wait that gives up reports
  // 0, which the compiler does not know.  A slot is handed back (and overwritten by the copy engine) only when what was read from it has arrived in
  // registers: the address of the arrival depends on it.  Reads that are merely issued before the arrival may still wait their turn behind another
  // kernel's memory instructions on the same SM, and rows 0 to 23 of a stage then came from the next one (5 to 8 columns in 3000 launches of
  // 18944 x 1024, 8 bits, 250 tokens, between elementwise kernels).
  uint32_t zero;
};
struct Shared {
  uint64_t full_w[MAX_STAGES], empty_w[MAX_STAGES], full_x[X_SLOTS], empty_x[X_SLOTS], full_a[A_SLOTS], empty_a[A_SLOTS];
  uint64_t sb_full[NSB], sb_empty[NSB], acc_full[2], acc_empty[2];
  uint32_t tmem;
  volatile int abort;
};

// The segments of a CTA: (tile, first stage, number of stages).  Whole tiles go round robin; of the accumulating epilogue only as many as
// fill every CTA alike, the rest is cut into equal contiguous ranges of stages.  (Ranges from the start would spread the CTAs over all
// of X and all of W at once: 4096 x 14336 at 4096 tokens 423 us, its 117 MB of X coming from HBM again and again.)
template <bool ADD> struct Segments {
  int next_tile, whole;          // round robin: tiles below `whole`
  int u, end;                    // then stages [u, end)
  int G;
  __device__ __forceinline__ Segments(const Params& p) {
    G = (int)gridDim.x;
    next_tile = blockIdx.x;
    whole = ADD ? p.items / G * G : p.items;
    const long long first = (long long)whole * p.num_st, U = (long long)(p.items - whole) * p.num_st;
    u = (int)(first + U * blockIdx.x / G);
    end = (int)(first + U * (blockIdx.x + 1) / G);
  }
  __device__ __forceinline__ bool next(const Params& p, int& tile, int& s0, int& ns) {
    if (next_tile < whole) {
      tile = next_tile;
      s0 = 0;
      ns = p.num_st;
      next_tile += G;
      return true;
    }
    if (!ADD || u >= end) return false;
    tile = u / p.num_st;
    s0 = u - tile * p.num_st;
    ns = min(p.num_st - s0, end - u);
    u += ns;
    return true;
  }
};
// Tiles that run at one time share weights (token tile fastest) or, where X is the larger operand, X (row block fastest).
__device__ __forceinline__ void tile_of(const Params& p, int tile, int& rb, int& tm) {
  if (p.row_fast) {
    tm = tile / p.row_blocks;
    rb = tile - tm * p.row_blocks;
  } else {
    rb = tile / p.tiles_m;
    tm = tile - rb * p.tiles_m;
  }
}

__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity, Shared* sh, const Params& p, int role) {
  return mbar_wait_warp(smem_u32(bar), parity, &sh->abort, p.wait_word, role);
}

// 16 tokens of one thread's output column
template <typename T>
__device__ __forceinline__ void emit(const Params& p, int rb, int q, int lane, int tok0, const float (&v)[16]) {
  if (p.epi == B200P_EPI_SILU_MUL) {
    // lanes 0..15 hold gate rows, lanes 16..31 the matching up rows: even tokens are finished by the former, odd ones by the latter
    const int n = rb * 64 + q * 16 + (lane & 15);
    const bool upper = lane >= 16;
    T* y = reinterpret_cast<T*>(p.y) + (p.y_perm ? perm8_pos(n) : n);
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const float give = upper ? v[j] : v[j + 1], other = __shfl_xor_sync(0xffffffffu, give, 16);
      const float gate = upper ? other : v[j], up = upper ? v[j + 1] : other;
      const int tok = tok0 + j + (upper ? 1 : 0);
      if (n < p.N / 2 && tok < p.M_tok) y[(int64_t)tok * p.ldy] = Tr<T>::from_f(__fdividef(gate, 1.0f + __expf(-gate)) * up);
    }
    return;
  }
  const int n = rb * 128 + q * 32 + lane;
  if (n >= p.N) return;
  if (p.epi == B200P_EPI_STORE_F32) {
    float* y = reinterpret_cast<float*>(p.y) + n;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (tok0 + j < p.M_tok) __stcg(y + (int64_t)(tok0 + j) * p.ldy, v[j]);
  } else {
    T* y = reinterpret_cast<T*>(p.y) + (p.y_perm ? perm8_pos(n) : n);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (tok0 + j < p.M_tok) y[(int64_t)(tok0 + j) * p.ldy] = Tr<T>::from_f(v[j]);
  }
}

// barrier over `threads` threads that tells all of them whether all of them said yes
__device__ __forceinline__ bool all_of(int id, int threads, bool v) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 p, %1, 0;\n"
      "barrier.cta.red.and.pred q, %2, %3, p;\n"
      "selp.b32 %0, 1, 0, q;\n"
      "}\n"
      : "=r"(r)
      : "r"(v ? 1u : 0u), "r"(id), "r"(threads)
      : "memory");
  return r != 0;
}

// One warp's share of a tile: token groups worker, worker + WORKERS, ... of lane quarter q.  ADD: the four warps of a worker fill one
// staging tile of 8 tokens x 128 rows and send it as one bulk reduction (one of 32 rows per warp was a third slower: the L2 adds lines
// of 512 bytes faster than four of 128).
template <typename T, bool FAST, bool ADD>
__device__ __forceinline__ bool drain(const Params& p, const CUtensorMap* tm_y, Shared* sh, uint32_t tmem, int tile, uint32_t parity, int worker,
                                      int q, int lane, uint32_t stage) {
  constexpr float DSCALE = FAST ? SmallScaleOut<T>::value : 1.f;
  constexpr int TOK = ADD ? ADD_TOK : 16;
  int rb, tm;
  tile_of(p, tile, rb, tm);
  const int tok0 = tm * p.TN;
  const uint32_t d = tmem + ((uint32_t)(q * 32) << 16);
  bool ok = wait(&sh->acc_full[0], parity, sh, p, 4) && wait(&sh->acc_full[1], parity, sh, p, 4);
  if (ADD) ok = all_of(1 + worker, 128, ok);                 // (the four warps meet at barriers below: one mind)
  if (!ok) return false;
  tc_fence_after();
  for (int t0 = worker * TOK; t0 < p.TN; t0 += WORKERS * TOK) {
    if (tok0 + t0 >= p.M_tok) break;                         // padding tokens of the last token tile
    const uint32_t src = d + (uint32_t)(t0 < p.H0 ? t0 : 128 + t0 - p.H0);
    float v[TOK];
    if constexpr (ADD) {
      tmem_ld8(src, v);
      if (q == 0 && lane == 0) bulk_wait_read<0>();          // the previous group has left the staging tile
      tmem_ld_wait();
      named_bar_sync(1 + worker, 128);
#pragma unroll
      for (int j = 0; j < TOK; ++j) sts32(stage + (uint32_t)(j * 128 + q * 32 + lane) * 4u, __float_as_uint(v[j] * DSCALE));
      fence_proxy_async_smem();
      named_bar_sync(1 + worker, 128);
      if (q == 0 && lane == 0) {                             // rows / tokens outside the tensor are clipped by the TMA unit
        tma_reduce_add_2d(tm_y, rb * 128, tok0 + t0, stage);
        bulk_commit();
      }
    } else {
      tmem_ld16(src, v);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < TOK; ++j) v[j] *= DSCALE;
      emit<T>(p, rb, q, lane, tok0 + t0, v);
    }
  }
  tc_fence_before();
  __syncwarp();
  if (lane == 0) {
    mbar_arrive(smem_u32(&sh->acc_empty[0]));
    mbar_arrive(smem_u32(&sh->acc_empty[1]));
  }
  return true;
}

// FAST: the small-scale dequant of dequant.cuh (caller promised B200P_W_SMALLSCALE): A and D are produced at 1 / SmallScaleOut<T>.
template <typename T, int BITS, bool XPERM, bool FAST, bool ADD>
__global__ void __launch_bounds__(THREADS, 1)
qmm_wide_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                const __grid_constant__ CUtensorMap tm_s, const __grid_constant__ CUtensorMap tm_b,
                const __grid_constant__ CUtensorMap tm_y, const Params p) {
  constexpr int PKB = 64 * BITS / 8;            // packed bytes per row per k-block
  constexpr int KPS = 128 / PKB;                // k-blocks per stage (4 / 2)
  constexpr int SPG = 8 / KPS;                  // stages per scale/bias group of 8 k-blocks
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t w_ring = (raw + 1023u) & ~1023u;
  const uint32_t x_bytes = (uint32_t)(p.TN * 128);
  const uint32_t x_ring = w_ring + (uint32_t)p.w_stages * W_STAGE_BYTES;
  const uint32_t sb_ring = x_ring + X_SLOTS * x_bytes;
  const uint32_t epi_ring = sb_ring + NSB * 2 * SB_TILE_BYTES;
  Shared* sh = reinterpret_cast<Shared*>(smem_raw + (epi_ring - raw) + (ADD ? WORKERS * STAGE_OUT_BYTES : 0));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool silu = !ADD && p.epi == B200P_EPI_SILU_MUL;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.w_stages; ++s) { mbar_init(smem_u32(&sh->full_w[s]), 1); mbar_init(smem_u32(&sh->empty_w[s]), KPS * 4); }
    for (int s = 0; s < X_SLOTS; ++s) { mbar_init(smem_u32(&sh->full_x[s]), 1); mbar_init(smem_u32(&sh->empty_x[s]), 2); }
    for (int s = 0; s < A_SLOTS; ++s) { mbar_init(smem_u32(&sh->full_a[s]), 4); mbar_init(smem_u32(&sh->empty_a[s]), 2); }
    for (int s = 0; s < NSB; ++s) { mbar_init(smem_u32(&sh->sb_full[s]), 1); mbar_init(smem_u32(&sh->sb_empty[s]), DQ_WARPS); }
    for (int h = 0; h < 2; ++h) { mbar_init(smem_u32(&sh->acc_full[h]), 1); mbar_init(smem_u32(&sh->acc_empty[h]), WORKERS * 4); }
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_s);
    tma_prefetch_desc(&tm_b);
  }
  if (warp == WARP_MMA) tmem_alloc(smem_u32(&sh->tmem), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;
  pdl_launch_dependents();
  Segments<ADD> segs(p);
  int tile, s0, ns;
  bool ok = true;

  if (warp >= DQ_WARPS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_OTHER));
  if (warp == WARP_W) {
    // weights, scales and biases depend on no previous kernel: no griddepcontrol.wait here
    int si = 0, sbi = 0;
    uint32_t ph = 0, sbph = 0;
    while (ok && segs.next(p, tile, s0, ns)) {
      int rb, tm;
      tile_of(p, tile, rb, tm);
      for (int st = s0; st < s0 + ns; ++st) {
        if (st == s0 || st % SPG == 0) {                    // a new group of 8 k-blocks
          if (!(ok = wait(&sh->sb_empty[sbi], sbph ^ 1u, sh, p, 0))) break;
          if (elect_one()) {
            const uint32_t dst = sb_ring + sbi * 2 * SB_TILE_BYTES, bar = smem_u32(&sh->sb_full[sbi]);
            const int kb0 = st / SPG * 8;
            mbar_arrive_expect_tx(bar, 2 * SB_TILE_BYTES);
            if (silu) {
              for (int i = 0; i < 8; ++i) {
                const int row = (i & 1 ? p.N / 2 : 0) + rb * 64 + (i >> 1) * 16;
                tma_load_2d(dst + i * 256, &tm_s, kb0, row, bar);
                tma_load_2d(dst + SB_TILE_BYTES + i * 256, &tm_b, kb0, row, bar);
              }
            } else {
              tma_load_2d(dst, &tm_s, kb0, rb * 128, bar);
              tma_load_2d(dst + SB_TILE_BYTES, &tm_b, kb0, rb * 128, bar);
            }
          }
          __syncwarp();
          if (++sbi == NSB) { sbi = 0; sbph ^= 1u; }
        }
        if (!(ok = wait(&sh->empty_w[si], ph ^ 1u, sh, p, 0))) break;
        if (elect_one()) {
          const uint32_t dst = w_ring + si * W_STAGE_BYTES, bar = smem_u32(&sh->full_w[si]);
          mbar_arrive_expect_tx(bar, W_STAGE_BYTES);
          if (silu) {
            for (int i = 0; i < 8; ++i)
              tma_load_2d(dst + i * 2048, &tm_w, st * 128, (i & 1 ? p.N / 2 : 0) + rb * 64 + (i >> 1) * 16, bar);
          } else {
            tma_load_2d(dst, &tm_w, st * 128, rb * 128, bar);
          }
        }
        __syncwarp();
        if (++si == p.w_stages) { si = 0; ph ^= 1u; }
      }
    }
  } else if (warp == WARP_X) {
    pdl_wait();                                             // X is the previous kernel's output
    int xs = 0;
    uint32_t ph = 0;
    while (ok && segs.next(p, tile, s0, ns)) {
      int rb, tm;
      tile_of(p, tile, rb, tm);
      const int tok0 = tm * p.TN;
      for (int kb = s0 * KPS; kb < (s0 + ns) * KPS; ++kb) {
        if (!(ok = wait(&sh->empty_x[xs], ph ^ 1u, sh, p, 1))) break;
        if (elect_one()) {
          const uint32_t bar = smem_u32(&sh->full_x[xs]);
          mbar_arrive_expect_tx(bar, x_bytes);
          tma_load_2d(x_ring + xs * x_bytes, &tm_x, kb * 64, tok0, bar);
        }
        __syncwarp();
        if (++xs == X_SLOTS) { xs = 0; ph ^= 1u; }
      }
    }
  } else if (warp >= WARP_MMA) {
    const int h = warp - WARP_MMA;
    {
      const uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)((h ? p.H1 : p.H0) >> 3) << 17) | ((128u >> 4) << 24);
      const uint32_t d = tmem + 128u * h;
      const uint64_t xdesc0 = make_desc_sw128(x_ring + (uint32_t)(h * p.H0) * 128u);
      int seg = 0, xs = 0;
      uint32_t slot = 0, aph = 0, xph = 0;
      for (; ok && segs.next(p, tile, s0, ns); ++seg) {
        if (seg > 0) {                                      // the epilogue has drained the previous segment's sums
          if (!(ok = wait(&sh->acc_empty[h], (uint32_t)((seg - 1) & 1), sh, p, 2))) break;
          tc_fence_after();
        }
        const int nkb = ns * KPS;
        for (int j = 0; j < nkb; ++j) {
          if (!(ok = wait(&sh->full_x[xs], xph, sh, p, 2) && wait(&sh->full_a[slot], aph, sh, p, 2))) break;
          tc_fence_after();
          if (elect_one()) {
            umma_half_kblock_f16_ts(d, tmem + A_COL0 + slot * 32, xdesc0 + (uint64_t)(xs * (x_bytes >> 4)), idesc, j > 0 ? 1u : 0u);
            umma_commit(smem_u32(&sh->empty_a[slot]));
            umma_commit(smem_u32(&sh->empty_x[xs]));
            if (j == nkb - 1) umma_commit(smem_u32(&sh->acc_full[h]));
          }
          __syncwarp();
          if (++slot == A_SLOTS) { slot = 0; aph ^= 1u; }
          if (++xs == X_SLOTS) { xs = 0; xph ^= 1u; }
        }
      }
    }
  } else if (warp < DQ_WARPS) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_DQ));
    // ===================================== dequantisers =====================================
    const int grp = warp >> 2, q = warp & 3, r = q * 32 + lane;
    const uint32_t a_dst = tmem + ((uint32_t)(q * 32) << 16) + A_COL0;
    const uint32_t w_row = (uint32_t)((r >> 3) * 1024 + (r & 7) * 128), w_xor = (uint32_t)(r & 7);
    int si = 0, sbi = 0;
    uint32_t ph = 0, sbph = 0, stage_no = 0;                // stage_no: stages of this CTA so far (k-block number = stage_no * KPS + j)
    uint4 s8 = make_uint4(0u, 0u, 0u, 0u), b8 = s8;
    const uint32_t out_stage = epi_ring + (uint32_t)((1 + grp) * STAGE_OUT_BYTES);
    int pending = -1;                                       // the previous segment's tile, still to be drained
    uint32_t drained = 0;                                   // segments drained so far
    bool voted = false;                                     // (ADD) left by the vote that drain() begins with
    auto drain_pending = [&]() {
      pdl_wait();                                           // y belongs to the previous kernels until here
      ok = drain<T, FAST, ADD>(p, &tm_y, sh, tmem, pending, drained & 1u, 1 + grp, q, lane, out_stage);
      voted = !ok;
      pending = -1;
      ++drained;
    };
    while (ok && segs.next(p, tile, s0, ns)) {
      for (int st = s0; st < s0 + ns; ++st, ++stage_no) {
        if (st == s0 || st % SPG == 0) {                    // scales / biases of this row for the next 8 k-blocks
          if (!(ok = wait(&sh->sb_full[sbi], sbph, sh, p, 3))) break;
          const uint32_t src = sb_ring + sbi * 2 * SB_TILE_BYTES + (uint32_t)(r * 16);
          s8 = lds128(src);
          b8 = lds128(src + SB_TILE_BYTES);
          const uint32_t done = smem_u32(&sh->sb_empty[sbi]) + ((s8.w | b8.w) & p.zero);
          __syncwarp();
          if (lane == 0) mbar_arrive(done);
          if (++sbi == NSB) { sbi = 0; sbph ^= 1u; }
        }
        // 4 bits: group g takes k-block g of every stage; 8 bits: k-block g & 1 of every second stage
        const bool mine = KPS == 4 || (int)(stage_no & 1u) == (grp >> 1);
        if (mine) {
          const int j = KPS == 4 ? grp : (grp & 1);
          if (!(ok = wait(&sh->full_w[si], ph, sh, p, 3))) break;
          constexpr int CPK = PKB / 16;
          uint4 pk[CPK];
          const uint32_t wsrc = w_ring + si * W_STAGE_BYTES + w_row;
#pragma unroll
          for (int c = 0; c < CPK; ++c) pk[c] = lds128(wsrc + ((((uint32_t)(j * CPK + c)) ^ w_xor) << 4));
          uint32_t all = 0;
#pragma unroll
          for (int c = 0; c < CPK; ++c) all |= pk[c].w;
          const uint32_t done = smem_u32(&sh->empty_w[si]) + (all & p.zero);          // (see Params::zero)
          __syncwarp();
          if (lane == 0) mbar_arrive(done);
          const int e = (st % SPG) * KPS + j;               // k-block within the group: half e & 1 of word e >> 1
          const int we = e >> 1;
          const uint32_t sw = we == 0 ? s8.x : we == 1 ? s8.y : we == 2 ? s8.z : s8.w;
          const uint32_t bw = we == 0 ? b8.x : we == 1 ? b8.y : we == 2 ? b8.z : b8.w;
          const uint32_t sel = e & 1 ? 0x3232u : 0x1010u;
          const uint32_t s2 = prmt(sw, 0u, sel), b2 = prmt(bw, 0u, sel);
          uint32_t o[32];
          const uint32_t* pw = reinterpret_cast<const uint32_t*>(pk);
          if constexpr (FAST) {
            const SmallScale sc = small_scale_prep<T>(s2, b2);
#pragma unroll
            for (int c = 0; c < 8; ++c) dequant8_small<T, BITS, XPERM>(pw + c * (BITS / 4), sc, o + 4 * c);
          } else {
#pragma unroll
            for (int c = 0; c < 8; ++c) dequant8<T, BITS, XPERM>(pw + c * (BITS / 4), s2, b2, o + 4 * c);
          }
          const uint32_t n = stage_no * KPS + (uint32_t)j, slot = n & (A_SLOTS - 1);
          if (!(ok = wait(&sh->empty_a[slot], ((n / A_SLOTS) & 1u) ^ 1u, sh, p, 3))) break;
          tc_fence_after();
          tmem_st32(a_dst + slot * 32, o);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh->full_a[slot]));
          if (pending >= 0) {                               // the first k-block of this segment is ready: now finish the previous tile
            drain_pending();
            if (!ok) break;
          }
        }
        if (++si == p.w_stages) { si = 0; ph ^= 1u; }
      }
      if (ok && pending >= 0) drain_pending();              // (a segment in which this group had no k-block)
      pending = tile;
    }
    if (ok && pending >= 0) drain_pending();
    // A warp that gave up outside a drain still owes its group one vote: the others come to it at their next drain, or here.
    if (ADD && !ok && !voted) all_of(2 + grp, 128, false);
    if (ADD && lane == 0) bulk_wait_all();                  // staging memory and outputs are settled before the CTA retires
  } else {
    // ===================================== epilogue =========================================
    const int q = warp & 3;
    uint32_t seg = 0;
    pdl_wait();                                             // y belongs to the previous kernels until here
    for (; ok && segs.next(p, tile, s0, ns); ++seg)
      ok = drain<T, FAST, ADD>(p, &tm_y, sh, tmem, tile, seg & 1u, 0, q, lane, epi_ring);
    if (ADD && lane == 0) bulk_wait_all();
  }
  if (sh->abort) wait_settle();
  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------ host
struct Plan { int tiles_m, TN, H0, H1, row_blocks, left, items, grid, w_stages, smem; };

// Row blocks of a short last round of whole tiles that are left to the kernel that splits K (qmm_tc.cu): row_blocks x tiles_m just above a multiple of the
// SMs is common (57344 gated rows are 448 blocks, three times 148 and four), and the few CTAs of the last round then take as long as all of one before.
// Behind the other launch the split one costs about 30000 cycles and its share of K; a round takes a k-block about 640 cycles with 8-bit codes.  So only
// long rounds are worth it (us, whole tiles / left, 8 bits: 57344 x 8192 at 129 / 201 / 300 / 600 tokens 190 / 174, 209 / 192, 319 / 303, 500 / 492, but
// 1349 / 1377 at 1300, 13 rounds; 19072 x 8192 at 201 / 600 / 1500 119 / 90, 209 / 196, 446 / 433; 22016 x 8192 at 201 115 / 105; 28672 x 8192 at 300
// 210 / 187), and never at 4 bits, whose rounds are shorter (28672 x 4096 96.3 / 97.5 at 300, 303 / 350 at 1500).
static int left_over(int row_blocks, int tiles_m, int tn, int64_t M, int64_t K, int bits) {
  if (bits != 8) return 0;
  const int sms = sm_count(), items = row_blocks * tiles_m, whole = items / sms * sms;
  if (whole == 0 || whole == items || whole > 9 * sms) return 0;
  const int left = row_blocks - whole / tiles_m;
  const int64_t tiles = (int64_t)(left + 1) / 2 * ((M + 127) / 128), splits = sms / tiles < 16 ? sms / tiles : 16;
  const double kb = (double)(K / 64), round = kb * std::max(2.0 * tn, 640.0);
  return splits >= 4 && 30000.0 + 700.0 * kb / (double)splits < 0.6 * round ? left : 0;
}

static Plan make_plan(int64_t M, int64_t N, int64_t K, int bits, int epi, bool may_leave) {
  Plan pl;
  const bool add = epi == B200P_EPI_ADD_RESIDUAL;
  const int rows = epi == B200P_EPI_SILU_MUL ? 64 : 128;
  pl.row_blocks = (int)(((epi == B200P_EPI_SILU_MUL ? N / 2 : N) + rows - 1) / rows);
  const int sms = sm_count(), t0 = (int)((M + MAX_TN - 1) / MAX_TN);
  // token tiles: as few as hold M, unless one or two more (smaller) ones fill the last wave of whole tiles better.  A k-block costs
  // 2 cycles per token on the tensor core and never less than the dequantisers' time for 128 rows.
  double best = 1e300;
  for (int tm = t0; tm <= t0 + 2; ++tm) {
    const int tn = (int)(((M + tm - 1) / tm + 15) / 16 * 16);
    const double kb = 2.0 * tn > 280.0 ? 2.0 * tn : 280.0;
    const int64_t items = (int64_t)pl.row_blocks * tm;
    const double waves = add ? (double)items / sms : (double)((items + sms - 1) / sms);
    const double cost = waves * (kb * (double)(K / 64) + 8.0 * tn);
    if (cost < best * 0.999) { best = cost; pl.tiles_m = tm; pl.TN = tn; }
  }
  pl.H0 = (pl.TN / 2 + 15) / 16 * 16;
  pl.H1 = pl.TN - pl.H0;
  pl.left = add || !may_leave ? 0 : left_over(pl.row_blocks, pl.tiles_m, pl.TN, M, K, bits);
  pl.row_blocks -= pl.left;
  pl.items = pl.row_blocks * pl.tiles_m;
  const int64_t units = add ? (int64_t)pl.items * (K * bits / 1024) / 2 : pl.items;      // at least two stages per CTA
  pl.grid = (int)(units < 1 ? 1 : units > sms ? sms : units);
  const int fixed = 1024 + NSB * 2 * SB_TILE_BYTES + (add ? WORKERS * STAGE_OUT_BYTES : 0) + (int)sizeof(Shared);
  int st = (SMEM_BUDGET - fixed - X_SLOTS * pl.TN * 128) / W_STAGE_BYTES;
  pl.w_stages = st > MAX_STAGES ? MAX_STAGES : st;
  // 8 bits: a group of dequantisers takes every second stage.  With an odd ring it would come to each slot every second time round, and
  // a wait for a slot's phase does not tell the fill before last from one that is still on its way.
  if (bits == 8) pl.w_stages &= ~1;
  pl.smem = fixed + X_SLOTS * pl.TN * 128 + pl.w_stages * W_STAGE_BYTES;
  return pl;
}

template <typename T, int BITS, bool XPERM, bool FAST, bool ADD>
static int run(const CUtensorMap* tm, const Params& p, const Plan& pl, cudaStream_t st) {
  auto kern = qmm_wide_kernel<T, BITS, XPERM, FAST, ADD>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BUDGET);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(qmm_wide_kernel)");
    attr_set = true;
  }
  cudaError_t e = launch_pdl_opt(pdl_enabled_gemm(), kern, pl.grid, THREADS, pl.smem, st, tm[0], tm[1], tm[2], tm[3], tm[4], p);
  if (e != cudaSuccess) return cuda_fail(e, "qmm_wide_kernel launch");
  return B200P_OK;
}

static int encode(TcEncodeFn enc, CUtensorMap* tm, CUtensorMapDataType dt, const void* base, uint64_t d0, uint64_t d1, uint64_t stride,
                  uint32_t b0, uint32_t b1, CUtensorMapSwizzle sw, const char* what) {
  cuuint64_t dims[2] = {d0, d1}, str[1] = {stride};
  cuuint32_t box[2] = {b0, b1}, es[2] = {1, 1};
  CUresult r = enc(tm, dt, 2, const_cast<void*>(base), dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B200P_REQUIRE(r == CUDA_SUCCESS, B200P_ERR_CUDA, "cuTensorMapEncodeTiled(%s) failed: %d", what, (int)r);
  return B200P_OK;
}

}  // namespace wide

constexpr int64_t MAX_TOKENS = wide::MAX_TN;

// the caller (c_api.cu) has already checked qmm_tc_supported()
bool qmm_wide_supported(int64_t M, int64_t N, int64_t K, int bits, int epi, const void* s, const void* b, const void* y, int64_t ldy) {
  if ((N / 64 + 2) * (M / 128 + 3) >= (1ll << 30) / (K / 64)) return false;      // (stages of all tiles are counted in 32 bits)
  if (M <= 128 || K % 512 != 0 || !aligned(s, 16) || !aligned(b, 16)) return false;
  if (epi == B200P_EPI_ADD_RESIDUAL) {
    if (N % 4 != 0 || !aligned(y, 16) || (ldy * 4) % 16 != 0) return false;
    // 4-bit sums of up to 1024 tokens: the stream-K kernel's 128-token tiles are as fast where they hold the tokens as tightly (4096 x
    // 14336, us, wide / stream-K: 26.3 / 27.4 at 201 tokens, 29.0 / 27.9 at 256, 43.1 / 44.0 at 400, 90.0 / 89.7 at 1000; 4096 x 4096: 14.1 /
    // 15.3, 16.2 / 15.6, 18.8 / 19.8, 30.8 / 29.5); above, 177 / 190 at 2048 and 359 / 405 at 4096.  8-bit codes: 94 / 127 at 201
    // tokens, 105 / 128 at 256, 400 / 510 at 1000 (8192 x 28672, bf16).
    const int64_t tm = (M + MAX_TOKENS - 1) / MAX_TOKENS, padded = tm * (((M + tm - 1) / tm + 15) / 16 * 16);
    return bits == 8 || M > 1024 || (M + 127) / 128 * 128 * 100 >= 108 * padded;
  }
  return aligned(y, epi == B200P_EPI_STORE_F32 ? 4 : 2);
}

int qmm_wide_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx,
                    int64_t ldy, int bits, int dtype, int epi, int flags, void* ws, size_t ws_bytes, cudaStream_t st) {
  using namespace wide;
  TcEncodeFn enc = tc_get_encode();
  B200P_REQUIRE(enc != nullptr, B200P_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  const bool x_perm = (flags & B200P_X_PERM8) != 0, add = epi == B200P_EPI_ADD_RESIDUAL;
  const bool fast = (flags & B200P_W_SMALLSCALE) != 0;
  const Plan pl = make_plan(M, N, K, bits, epi, ws != nullptr);
  B200P_REQUIRE(pl.w_stages >= 2, B200P_ERR_ARG, "shared memory too small for the tensor path");
  const CUtensorMapDataType dt16 = dtype == B200P_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const uint32_t box_rows = epi == B200P_EPI_SILU_MUL ? 16u : 128u;
  const uint64_t row_bytes = (uint64_t)K * bits / 8, ng = (uint64_t)K / 64;
  CUtensorMap tm[5];
  int rc = encode(enc, &tm[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, w, row_bytes, (uint64_t)N, row_bytes, 128u, box_rows, CU_TENSOR_MAP_SWIZZLE_128B, "weights");
  if (!rc) rc = encode(enc, &tm[1], dt16, x, (uint64_t)K, (uint64_t)M, (uint64_t)ldx * 2, 64u, (uint32_t)pl.TN, CU_TENSOR_MAP_SWIZZLE_128B, "x");
  if (!rc) rc = encode(enc, &tm[2], dt16, s, ng, (uint64_t)N, ng * 2, 8u, box_rows, CU_TENSOR_MAP_SWIZZLE_NONE, "scales");
  if (!rc) rc = encode(enc, &tm[3], dt16, b, ng, (uint64_t)N, ng * 2, 8u, box_rows, CU_TENSOR_MAP_SWIZZLE_NONE, "biases");
  tm[4] = tm[0];
  if (!rc && add)
    rc = encode(enc, &tm[4], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, y, (uint64_t)N, (uint64_t)M, (uint64_t)ldy * 4, 128u, (uint32_t)ADD_TOK,
                CU_TENSOR_MAP_SWIZZLE_NONE, "y");
  if (rc) return rc;
  Params p;
  p.zero = 0;
  if ((rc = wait_word(WAIT_QMM_WIDE, &p.wait_word))) return rc;
  p.y = y; p.M_tok = (int)M; p.N = (int)N; p.epi = epi; p.y_perm = (flags & B200P_Y_PERM8) ? 1 : 0;
  p.TN = pl.TN; p.H0 = pl.H0; p.H1 = pl.H1; p.ldy = ldy; p.num_st = (int)(row_bytes / 128);
  p.tiles_m = pl.tiles_m; p.row_blocks = pl.row_blocks; p.items = pl.items; p.w_stages = pl.w_stages;
  p.row_fast = M * K * 2 > N * K * bits / 8 ? 1 : 0;
#define GO(T_, B_, X_, F_) (add ? run<T_, B_, X_, F_, true>(tm, p, pl, st) : run<T_, B_, X_, F_, false>(tm, p, pl, st))
  const auto launch = [&]() -> int {
    if (dtype == B200P_F16) {
      if (bits == 8) return fast ? GO(__half, 8, false, true) : GO(__half, 8, false, false);
      if (fast) return x_perm ? GO(__half, 4, true, true) : GO(__half, 4, false, true);
      return x_perm ? GO(__half, 4, true, false) : GO(__half, 4, false, false);
    }
    if (bits == 8) return fast ? GO(__nv_bfloat16, 8, false, true) : GO(__nv_bfloat16, 8, false, false);
    if (fast) return x_perm ? GO(__nv_bfloat16, 4, true, true) : GO(__nv_bfloat16, 4, false, true);
    return x_perm ? GO(__nv_bfloat16, 4, true, false) : GO(__nv_bfloat16, 4, false, false);
  };
#undef GO
  rc = launch();
  if (rc || !pl.left) return rc;
  return qmm_tc_launch(x, w, s, b, y, M, N, K, ldx, ldy, bits, dtype, epi, flags, ws, ws_bytes,
                       (int64_t)pl.row_blocks * (epi == B200P_EPI_SILU_MUL ? 64 : 128), st);
}

}  // namespace b200p

// 0, or 1 + the role (0 weight loader, 1 X loader, 2 MMA issuer, 3 dequantiser, 4 epilogue) of the first wait of a wide quantised GEMM
// that ran out; reading clears it.  Synchronises the device.
extern "C" int b200p_qmm_wide_fault(void) { return b200p::wait_take(b200p::WAIT_QMM_WIDE); }
