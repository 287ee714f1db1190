// Dense 16-bit GEMM on tcgen05: y[M,N] = x[M,K] . w[N,K]^T (+ batch, or grouped), both operands in shared memory, accumulators in TMEM.
//
// Three kernels.  Two have the WEIGHTS on the MMA's M side and the tokens on the N side: the accumulator holds y transposed (lane = output
// column, TMEM column = token) and the epilogue stores it back transposed, a warp writing 32 consecutive outputs of one token.  All are
// persistent (CTA or pair c takes tiles c, c + grid, ...) with two accumulators, so that the epilogue of one tile overlaps the main
// loop of the next.
//
// gemm_tc_kernel, up to 64 tokens (decode batches): a CTA takes 128 weight rows against 32 or 64 tokens.  (With the tokens on the M side the
// MMA would read 128 rows of them from shared memory whatever they hold, and that read, not HBM, bounded the weight stream.)  Where
// the weight matrix has too few 128-row tiles to fill the GPU (narrow outputs with long K), K is split over several CTAs that
// add their partial sums into the zeroed fp32 output with red.global.add.
//   warp 0      TMA producer: w and x tiles of one 64-wide k-block per ring stage (3-d tensor maps: k, row, batch index), K-major, SWIZZLE_128B
//   warp 1      MMA issuer: four tcgen05.mma (M=128, N=BN, K=16) per stage, tcgen05.commit frees the stage; owns the TMEM allocation
//   warps 2..5  epilogue: tcgen05.ld (thread = output column, 32 tokens at a time) -> store / store fp32 / gated unit
//
// gemm_tc_pair_kernel, prompts: two CTAs on one tile; gemm_tc_rows_kernel, prompts with a short K or a narrow output: tokens on the M side.
//
// Rows, columns and k outside the tensors are zero-filled by the TMA unit and masked in the epilogue.  Every mbarrier wait is
// bounded: a wait that runs out raises a device flag (reported by the next launch) and the CTA leaves through the common exit,
// which frees its TMEM.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace b200p {

int sm_count();
bool pdl_chained();

constexpr int GT_BM = 128, GT_BK = 64, GT_THREADS = 192;
constexpr int GT_A_BYTES = GT_BM * GT_BK * 2;

struct GemmTcOut { void* y; int64_t R, ldy; };     // R: output columns (weight rows)
struct GemmTcParams {
  GemmTcOut out[2];              // of the product, and of the second one
  int64_t tokens, sy;            // tokens (of the largest group)
  int tiles_r, tiles_t, num_tiles, num_kb;
  int splits, kb_per_split;      // K split over `splits` CTAs per output tile (fp32 store only)
  int epi;
  float2 act;
  // grouped products: batch index z owns the rows [seg[z], seg[z+1]) of x and y; seg (device, groups + 1 offsets) is copied to shared
  // memory first, every CTA counts the groups' tiles there
  const int32_t* seg;
  int groups;
  // a plain product in the same launch (a mixture's shared expert beside the routed ones): its tiles come first, its K may be another
  struct Second {
    int64_t tokens;
    int tiles_r, tiles_t, num_tiles, num_kb, tn;
  } two;
  int* wait_word;                // where a wait that gives up reports
};
constexpr int GT_MAX_GROUPS = 1024;

// D[tmem] (+)= A[smem desc] * B[smem desc]^T, 16-bit inputs, fp32 accumulation
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accum)
      : "memory");
}

// This thread owns output column `n` (a weight row) and holds it for 32 consecutive tokens from `tok0`, of those below `tokens`.
// Gate / up pairs sit in neighbouring lanes.
template <typename T>
__device__ __forceinline__ void gemm_tc_store32(const GemmTcParams& p, const GemmTcOut& o, int64_t z_off, int64_t n, int64_t tok0, int64_t tokens,
                                                const float (&v)[32]) {
  if (gemm_epi_is_glu(p.epi)) {
    // the even lane of a pair holds the gate, the odd one the up row: the former finishes even tokens, the latter odd ones
    const bool odd = (threadIdx.x & 1) != 0;
    T* dst = reinterpret_cast<T*>(o.y) + z_off + (tok0 + odd) * o.ldy + (n >> 1);
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float other = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
      if ((n | 1) < o.R && tok0 + i + odd < tokens)
        dst[i * o.ldy] = Tr<T>::from_f(glu_unit16(odd ? other : v[i], odd ? v[i + 1] : other, p.epi, p.act));
    }
    return;
  }
  if (n >= o.R) return;
  if (p.epi == B200P_GEMM_STORE_F32) {
    float* dst = reinterpret_cast<float*>(o.y) + z_off + n;
    if (p.splits > 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (tok0 + i < tokens) atomicAdd(dst + (tok0 + i) * o.ldy, v[i]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (tok0 + i < tokens) dst[(tok0 + i) * o.ldy] = v[i];
    }
  } else if (p.epi == B200P_GEMM_CAP_F32) {
    float* dst = reinterpret_cast<float*>(o.y) + z_off + n;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (tok0 + i < tokens) dst[(tok0 + i) * o.ldy] = gemm_f32_act(v[i], p.epi, p.act);
  } else {
    T* dst = reinterpret_cast<T*>(o.y) + z_off + n;
    float a[32];                                   // one uniform branch for all elements
    if (p.epi == B200P_GEMM_XIELU) {
#pragma unroll
      for (int i = 0; i < 32; ++i) a[i] = xielu_unit(v[i], p.act);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) a[i] = p.epi == B200P_GEMM_RELU_SQ ? gemm_store_act(v[i], B200P_GEMM_RELU_SQ, p.act) : v[i];
    }
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (tok0 + i < tokens) dst[(tok0 + i) * o.ldy] = Tr<T>::from_f(a[i]);
  }
}

struct GemmTcShared {            // lives behind the ring stages (8-byte aligned)
  uint64_t full[10], empty[10], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
  int seg[GT_MAX_GROUPS + 1];
  int live[GT_MAX_GROUPS + 1];   // grouped products: row tiles of all groups before this one that hold rows
};

// Tile t of the launch: batch index (group) z, row tile rt; first token of the group in x / y and how many it has.  Grouped products
// number only the tiles of groups that hold tokens, so that the CTAs share them evenly whatever the routing.
struct GemmTcTile { int z, rt, first, len, kb0, kb1, second; };
__device__ __forceinline__ GemmTcTile gemm_tc_tile(const GemmTcParams& p, const GemmTcShared* sh, int t) {
  GemmTcTile r;
  r.second = t < p.two.num_tiles;
  r.kb0 = 0;
  if (r.second) {
    r.z = r.first = 0;
    r.rt = t;
    r.len = (int)p.two.tokens;
    r.kb1 = p.two.num_kb;
    return r;
  }
  t -= p.two.num_tiles;
  r.kb1 = p.num_kb;
  if (!p.seg) {
    const int ts = t / p.splits;
    r.kb0 = (t - ts * p.splits) * p.kb_per_split;
    r.kb1 = min(p.num_kb, r.kb0 + p.kb_per_split);
    r.z = ts / p.tiles_r;
    r.rt = ts - r.z * p.tiles_r;
    r.first = 0;
    r.len = (int)p.tokens;
    return r;
  }
  int lo = 0, hi = p.groups - 1;                  // last group z with live[z] <= t (groups without tiles share their start)
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (sh->live[mid] <= t) lo = mid; else hi = mid - 1;
  }
  r.z = lo;
  r.rt = t - sh->live[lo];
  r.first = sh->seg[lo];
  r.len = sh->seg[lo + 1] - r.first;
  return r;
}

template <typename T, int BN, int STAGES>
__global__ void __launch_bounds__(GT_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmw, const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw2,
               const __grid_constant__ CUtensorMap tmx2, const GemmTcParams p) {
  constexpr int B_BYTES = BN * GT_BK * 2, STAGE_BYTES = GT_A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN;           // 64 or 128: a power of two >= 32
  static_assert(STAGES <= 10 && (BN == 32 || BN == 64), "ring / tile shape");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;    // SWIZZLE_128B tiles start on 1024-byte boundaries
  GemmTcShared* sh = reinterpret_cast<GemmTcShared*>(smem_raw + (base - raw) + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&sh->acc_full[a]), 1);
      mbar_init(smem_u32(&sh->acc_empty[a]), 4);   // one arrival per epilogue warp
    }
    sh->abort = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmx);
    tma_prefetch_desc(&tmw);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh->tmem_base), TMEM_COLS);
    pdl_launch_dependents();                       // (behind the allocation: no successor's CTA can take the columns first and then wait for us)
  }
  pdl_wait();                                      // operands, seg and y belong to the previous kernels until here
  if (p.seg) {
    for (int i = threadIdx.x; i <= p.groups; i += blockDim.x) sh->seg[i] = p.seg[i];
    __syncthreads();
    if (warp == 2) {                               // running count of the groups' row tiles
      int run = 0;
      for (int z0 = 0; z0 < p.groups; z0 += 32) {
        const int z = z0 + lane, len = z < p.groups ? sh->seg[z + 1] - sh->seg[z] : 0;
        const int mine = len > 0 ? p.tiles_r : 0;
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += v;
        }
        if (z < p.groups) sh->live[z] = run + sum - mine;
        run += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) sh->live[p.groups] = run;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  const int num_tiles = p.two.num_tiles + (p.seg ? sh->live[p.groups] : p.num_tiles);

  // (whole warps walk the loops and one elected lane issues: operands of warp-uniform code need no uniformising)
  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const GemmTcTile tl = gemm_tc_tile(p, sh, t);
      const CUtensorMap *mw = tl.second ? &tmw2 : &tmw, *mx = tl.second ? &tmx2 : &tmx;
      for (int kb = tl.kb0; kb < tl.kb1; ++kb) {
        if (!(ok = mbar_wait_warp(smem_u32(&sh->empty[stage]), phase ^ 1u, &sh->abort, p.wait_word, 0))) break;
        if (elect_one()) {
          const uint32_t bar = smem_u32(&sh->full[stage]);
          const uint32_t dst = base + stage * STAGE_BYTES;
          mbar_arrive_expect_tx(bar, STAGE_BYTES);
          tma_load_3d(dst, mw, kb * GT_BK, tl.rt * GT_BM, tl.z, bar);
          tma_load_3d(dst + GT_A_BYTES, mx, kb * GT_BK, tl.first, p.seg ? 0 : tl.z, bar);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(GT_BM >> 4) << 24);
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      if (!(ok = mbar_wait_warp(smem_u32(&sh->acc_empty[acc]), acc_phase ^ 1u, &sh->abort, p.wait_word, 1))) break;
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)(acc * BN);
      const GemmTcTile tl = gemm_tc_tile(p, sh, t);
      for (int kb = tl.kb0; kb < tl.kb1; ++kb) {
        if (!(ok = mbar_wait_warp(smem_u32(&sh->full[stage]), phase, &sh->abort, p.wait_word, 1))) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t ad = make_desc_sw128(base + stage * STAGE_BYTES);
          const uint64_t bd = make_desc_sw128(base + stage * STAGE_BYTES + GT_A_BYTES);
#pragma unroll
          for (int k = 0; k < GT_BK / 16; ++k)       // 16 k = 32 bytes = 2 descriptor units inside the swizzle atom
            umma_f16_ss(d, ad + 2u * k, bd + 2u * k, idesc, ((kb - tl.kb0) | k) ? 1u : 0u);
          umma_commit(smem_u32(&sh->empty[stage]));
          if (kb == tl.kb1 - 1) umma_commit(smem_u32(&sh->acc_full[acc]));
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  } else {
    const int lg = warp & 3;                       // the TMEM lane quarter this warp may read
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const GemmTcTile tl = gemm_tc_tile(p, sh, t);
      if (!mbar_wait_warp(smem_u32(&sh->acc_full[acc]), acc_phase, &sh->abort, p.wait_word, 2)) break;
      tc_fence_after();
      const int64_t n = (int64_t)tl.rt * GT_BM + lg * 32 + lane;              // output column
      const GemmTcOut out = p.out[tl.second];
      const int64_t z_off = p.seg ? tl.first * out.ldy : (int64_t)tl.z * p.sy;       // (0 of the second product)
      const uint32_t tsrc = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(acc * BN);
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        if (c >= tl.len) break;                    // warp-uniform
        float v[32];
        tmem_ld16(tsrc + c, *reinterpret_cast<float(*)[16]>(&v[0]));
        tmem_ld16(tsrc + c + 16, *reinterpret_cast<float(*)[16]>(&v[16]));
        tmem_ld_wait();
        gemm_tc_store32<T>(p, out, z_off, n, c, tl.len, v);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->acc_empty[acc]));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }
  if (sh->abort) wait_settle();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------------- short K, narrow outputs
// More than 64 tokens where the pair kernel below has little to multiply: one CTA on a tile of 128 tokens (the M side) x BN weight rows.  The
// set-up is half of the pair's (no cluster, fewer TMEM columns), a narrow output pads no 256 rows, and a thread owns a token's row, so that its
// outputs leave as 16-byte pieces: at a short K the store is what bounds the call.  Bound: the output's way through L2 (64 x 1500 x 512 x 128 to
// bf16: L2 at 67 % of its peak, tensor pipe 16 %) or, in small calls, latency.  Where the line lies: gemm_tc_rows_better.
template <typename T> __device__ __forceinline__ uint32_t pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// outputs n0 .. n0 + 31 of one token's row (at element row_off of y); vec: whole pieces may leave as 16 bytes
template <typename T>
__device__ __forceinline__ void gemm_tc_store_row32(const GemmTcParams& p, int64_t row_off, int64_t n0, bool vec, const float (&v)[32]) {
  const int64_t R = p.out[0].R;
  if (p.epi == B200P_GEMM_STORE_F32) {
    float* dst = reinterpret_cast<float*>(p.out[0].y) + row_off + n0;
    if (vec && n0 + 32 <= R) {
#pragma unroll
      for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (n0 + i < R) dst[i] = v[i];
    }
    return;
  }
  float a[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) a[i] = p.epi == B200P_GEMM_RELU_SQ ? gemm_store_act(v[i], B200P_GEMM_RELU_SQ, p.act) : v[i];
  T* dst = reinterpret_cast<T*>(p.out[0].y) + row_off + n0;
  if (vec && n0 + 32 <= R) {
#pragma unroll
    for (int i = 0; i < 32; i += 8)
      *reinterpret_cast<uint4*>(dst + i) = make_uint4(pack2<T>(a[i], a[i + 1]), pack2<T>(a[i + 2], a[i + 3]), pack2<T>(a[i + 4], a[i + 5]), pack2<T>(a[i + 6], a[i + 7]));
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (n0 + i < R) dst[i] = Tr<T>::from_f(a[i]);
  }
}

template <typename T, int BN, int STAGES>
__global__ void __launch_bounds__(GT_THREADS, 1)
gemm_tc_rows_kernel(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw, const GemmTcParams p, const bool vec) {
  constexpr int B_BYTES = BN * GT_BK * 2, STAGE_BYTES = GT_A_BYTES + B_BYTES;
  constexpr uint32_t TMEM_COLS = 2 * BN;           // 128, 256 or 512
  static_assert(STAGES <= 10 && (BN == 64 || BN == 128 || BN == 256), "ring / tile shape");
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  GemmTcShared* sh = reinterpret_cast<GemmTcShared*>(smem_raw + (base - raw) + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&sh->acc_full[a]), 1);
      mbar_init(smem_u32(&sh->acc_empty[a]), 4);   // one arrival per epilogue warp
    }
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmx);
    tma_prefetch_desc(&tmw);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh->tmem_base), TMEM_COLS);
    pdl_launch_dependents();                       // (as above)
  }
  pdl_wait();                                      // operands and y belong to the previous kernels until here
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  const int per = p.tiles_t * p.tiles_r;           // tiles of a batch index, token tile fastest

  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.num_tiles && ok; t += gridDim.x) {
      const int z = t / per, rt = (t - z * per) / p.tiles_t, tt = (t - z * per) - rt * p.tiles_t;
      for (int kb = 0; kb < p.num_kb; ++kb) {
        if (!(ok = mbar_wait_warp(smem_u32(&sh->empty[stage]), phase ^ 1u, &sh->abort, p.wait_word, 0))) break;
        if (elect_one()) {
          const uint32_t bar = smem_u32(&sh->full[stage]), dst = base + stage * STAGE_BYTES;
          mbar_arrive_expect_tx(bar, STAGE_BYTES);
          tma_load_3d(dst, &tmx, kb * GT_BK, tt * GT_BM, z, bar);
          tma_load_3d(dst + GT_A_BYTES, &tmw, kb * GT_BK, rt * BN, z, bar);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(GT_BM >> 4) << 24);
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.num_tiles && ok; t += gridDim.x) {
      if (!(ok = mbar_wait_warp(smem_u32(&sh->acc_empty[acc]), acc_phase ^ 1u, &sh->abort, p.wait_word, 1))) break;
      tc_fence_after();
      const uint32_t d = tmem_base + (uint32_t)(acc * BN);
      for (int kb = 0; kb < p.num_kb; ++kb) {
        if (!(ok = mbar_wait_warp(smem_u32(&sh->full[stage]), phase, &sh->abort, p.wait_word, 1))) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t ad = make_desc_sw128(base + stage * STAGE_BYTES), bd = make_desc_sw128(base + stage * STAGE_BYTES + GT_A_BYTES);
#pragma unroll
          for (int k = 0; k < GT_BK / 16; ++k) umma_f16_ss(d, ad + 2u * k, bd + 2u * k, idesc, (kb | k) ? 1u : 0u);
          umma_commit(smem_u32(&sh->empty[stage]));
          if (kb == p.num_kb - 1) umma_commit(smem_u32(&sh->acc_full[acc]));
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  } else {
    const int lg = warp & 3;                       // the TMEM lane quarter this warp may read
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < p.num_tiles; t += gridDim.x) {
      const int z = t / per, rt = (t - z * per) / p.tiles_t, tt = (t - z * per) - rt * p.tiles_t;
      if (!mbar_wait_warp(smem_u32(&sh->acc_full[acc]), acc_phase, &sh->abort, p.wait_word, 2)) break;
      tc_fence_after();
      const int64_t row = (int64_t)tt * GT_BM + lg * 32 + lane, row_off = (int64_t)z * p.sy + row * p.out[0].ldy;
      const uint32_t tsrc = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(acc * BN);
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        const int64_t n0 = (int64_t)rt * BN + c;
        if (n0 >= p.out[0].R) break;               // warp-uniform
        float v[32];
        tmem_ld16(tsrc + c, *reinterpret_cast<float(*)[16]>(&v[0]));
        tmem_ld16(tsrc + c + 16, *reinterpret_cast<float(*)[16]>(&v[16]));
        tmem_ld_wait();
        if (row < p.tokens) gemm_tc_store_row32<T>(p, row_off, n0, vec, v);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->acc_empty[acc]));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }
  if (sh->abort) wait_settle();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------------------------------------------- two CTAs on one tile
// Prompts.  A pair of CTAs (a cluster of two, neighbouring SMs) computes 256 weight rows x up to 256 tokens with tcgen05.mma.cta_group::2:
//
//   A = w tile  [256 rows   x 64 k], CTA r stages rows [128 r, 128 r + 128)        (the M side; accumulator lane = output column)
//   B = x tile  [tn tokens  x 64 k], CTA r stages tokens [r tn / 2, (r + 1) tn / 2)  (the N side; accumulator column = token)
//   D = CTA r: its 128 rows x tn fp32 in its own TMEM, two buffers
//
// One CTA per tile is bounded by operand traffic: 128 x 256 x 64 k are 48 KB through L2 for 512 tensor cycles.  A CTA of a pair fetches 32 KB
// for the same cycles and each operand byte serves both (bf16, fp32 store, us, one CTA / pair: 6000 x 8192 x 2048 179 / 146, 1664 x 2048 x
// 2048 31 / 17, 1024 x 4096 x 3584 67 / 31, 200 x 7168 x 4096 37 / 22, 65 x 2048 x 4096 20.7 / 18.8; 16 groups of 375 rows, gated, 4096 x
// 2048, 77 / 74, of 125 rows 65 / 55; 1.3 to 1.4 PFLOP/s at the large end).  Weights are the M side because the N side may be any multiple of 32 tokens: row counts that fill no 128 or 256 rows (an
// expert's share of a prompt, a portion) are cut evenly, and the host narrows the tile where that fills the last wave.  The stores of a warp
// are then runs of 32 neighbouring outputs of one token.
//
// warp 0: TMA of its CTA's halves (completion counted on the leader's barriers); warp 1 of the leader: MMA issue, commits go to both
// CTAs; warps 2..9: epilogue, two per lane quarter, alternate pieces of 32 tokens.
namespace pair {

constexpr int EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS, STAGES = 6, MAX_TN = 256, TN_STEP = 32;
constexpr int A_BYTES = 128 * GT_BK * 2, B_BYTES = MAX_TN / 2 * GT_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;

struct Params {
  GemmTcParams g;
  int tn;                        // tokens per tile (plain products; a group's own are cut evenly)
  int box;                       // tokens per TMA box
};
struct Shared {
  uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  volatile int abort;
  int seg[GT_MAX_GROUPS + 1], live[GT_MAX_GROUPS + 1];       // group offsets; token tiles of all groups before this one
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_leader(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// this CTA's tile part, its bytes counted on a barrier of either CTA of the pair
__device__ __forceinline__ void load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar) {  // arrives at this offset in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3)
               : "memory");
}

// token tiles of a group of `len` tokens and their width
__device__ __forceinline__ int even_tn(int len) {
  const int nt = (len + MAX_TN - 1) / MAX_TN;
  return nt == 0 ? TN_STEP : ((len + nt - 1) / nt + TN_STEP - 1) / TN_STEP * TN_STEP;
}

struct Tile { int z, rt, tok0, first, len, tn, num_kb, second; };      // batch index (group), row tile, first token within it, ...
__device__ __forceinline__ Tile tile_of(const Params& p, const Shared* sh, int t) {
  Tile r;
  int in, nt;
  r.second = t < p.g.two.num_tiles;
  r.num_kb = r.second ? p.g.two.num_kb : p.g.num_kb;
  if (!r.second) t -= p.g.two.num_tiles;
  if (r.second) {
    nt = p.g.two.tiles_t;
    in = t;
    r.z = r.first = 0;
    r.len = (int)p.g.two.tokens;
    r.tn = p.g.two.tn;
  } else if (!p.g.seg) {
    nt = p.g.tiles_t;
    const int per = p.g.tiles_r * nt;
    r.z = t / per;
    in = t - r.z * per;
    r.first = 0;
    r.len = (int)p.g.tokens;
    r.tn = p.tn;
  } else {
    int lo = 0, hi = p.g.groups - 1;                         // last group with live * tiles_r <= t
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (sh->live[mid] * p.g.tiles_r <= t) lo = mid; else hi = mid - 1;
    }
    r.z = lo;
    nt = sh->live[lo + 1] - sh->live[lo];
    in = t - sh->live[lo] * p.g.tiles_r;
    r.first = sh->seg[lo];
    r.len = sh->seg[lo + 1] - r.first;
    r.tn = even_tn(r.len);
  }
  r.rt = in / nt;                                            // token tile fastest: pairs that run together share weights
  r.tok0 = (in - r.rt * nt) * r.tn;
  return r;
}

template <typename T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmw, const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw2,
                    const __grid_constant__ CUtensorMap tmx2, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;              // the same offset in both CTAs
  Shared* sh = reinterpret_cast<Shared*>(smem_raw + (base - raw) + STAGES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int pair0 = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
  int* word = p.g.wait_word;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&sh->full[s]), 1);                  // used in the leader
      mbar_init(smem_u32(&sh->empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&sh->acc_full[a]), 1);
      mbar_init(smem_u32(&sh->acc_empty[a]), 2 * EPI_WARPS); // used in the leader: the epilogue warps of both CTAs
    }
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmw);
    tma_prefetch_desc(&tmx);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    pdl_launch_dependents();                                 // (behind the allocation, as above)
  }
  pdl_wait();                                                // x, seg and y belong to the previous kernels until here
  if (p.g.seg) {
    for (int i = threadIdx.x; i <= p.g.groups; i += THREADS) sh->seg[i] = p.g.seg[i];
    __syncthreads();
    if (warp == 2) {                                         // running count of the groups' token tiles
      int run = 0;
      for (int z0 = 0; z0 < p.g.groups; z0 += 32) {
        const int z = z0 + lane, len = z < p.g.groups ? sh->seg[z + 1] - sh->seg[z] : 0, tn = even_tn(len);
        const int mine = (len + tn - 1) / tn;
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, sum, o);
          if (lane >= o) sum += v;
        }
        if (z < p.g.groups) sh->live[z] = run + sum - mine;
        run += __shfl_sync(0xffffffffu, sum, 31);
      }
      if (lane == 0) sh->live[p.g.groups] = run;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                            // both CTAs' barriers exist
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  const int num_tiles = p.g.two.num_tiles + (p.g.seg ? sh->live[p.g.groups] * p.g.tiles_r : p.g.num_tiles);

  // (whole warps walk the loops and one elected lane issues: operands of warp-uniform code need no uniformising)
  if (warp == 0) {
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = pair0; t < num_tiles && ok; t += pairs) {
      const Tile tl = tile_of(p, sh, t);
      const int box = tl.second ? tl.tn / 2 : p.box, half = tl.tn / 2, boxes = (half + box - 1) / box;
      const CUtensorMap *mw = tl.second ? &tmw2 : &tmw, *mx = tl.second ? &tmx2 : &tmx;
      const int row = tl.rt * 256 + (int)rank * 128, tok = tl.first + tl.tok0 + (int)rank * half, zx = p.g.seg ? 0 : tl.z;
      const uint32_t box_bytes = (uint32_t)box * GT_BK * 2, bytes = 2u * (uint32_t)(A_BYTES + boxes * box_bytes);
      for (int kb = 0; kb < tl.num_kb; ++kb) {
        if (!(ok = mbar_wait_warp(smem_u32(&sh->empty[stage]), phase ^ 1u, &sh->abort, word, 0))) break;
        if (elect_one()) {
          const uint32_t bar = map_to_leader(smem_u32(&sh->full[stage])), dst = base + stage * STAGE_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(smem_u32(&sh->full[stage]), bytes);
          load_3d(dst, mw, kb * GT_BK, row, tl.z, bar);
          for (int b = 0; b < boxes; ++b) load_3d(dst + A_BYTES + b * box_bytes, mx, kb * GT_BK, tok + b * box, zx, bar);
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
    // the pair's last commits have arrived here before this CTA may leave
    for (int s = 0; s < STAGES && ok; ++s) {
      ok = mbar_wait_warp(smem_u32(&sh->empty[stage]), phase ^ 1u, &sh->abort, word, 0);
      if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int t = pair0; t < num_tiles && ok; t += pairs) {
        const Tile tl = tile_of(p, sh, t);
        const int tn = tl.tn;
        const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(tn >> 3) << 17) | ((256u >> 4) << 24);
        if (!(ok = mbar_wait_warp(smem_u32(&sh->acc_empty[acc]), acc_phase ^ 1u, &sh->abort, word, 1))) break;
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)(acc * MAX_TN);
        for (int kb = 0; kb < tl.num_kb; ++kb) {
          if (!(ok = mbar_wait_warp(smem_u32(&sh->full[stage]), phase, &sh->abort, word, 1))) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t ad = make_desc_sw128(base + stage * STAGE_BYTES), bd = make_desc_sw128(base + stage * STAGE_BYTES + A_BYTES);
#pragma unroll
            for (int k = 0; k < GT_BK / 16; ++k) umma_pair(d, ad + 2u * k, bd + 2u * k, idesc, (kb | k) ? 1u : 0u);
            commit_pair(smem_u32(&sh->empty[stage]));
            if (kb == tl.num_kb - 1) commit_pair(smem_u32(&sh->acc_full[acc]));
          }
          __syncwarp();
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    const int lg = warp & 3, part = (warp - 2) >> 2;         // TMEM lane quarter; which pieces of 32 tokens
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = pair0; t < num_tiles; t += pairs) {
      const Tile tl = tile_of(p, sh, t);
      if (!mbar_wait_warp(smem_u32(&sh->acc_full[acc]), acc_phase, &sh->abort, word, 2)) break;
      tc_fence_after();
      const int64_t n = (int64_t)tl.rt * 256 + rank * 128 + lg * 32 + lane;
      const GemmTcOut out = p.g.out[tl.second];
      const int64_t z_off = p.g.seg ? (int64_t)tl.first * out.ldy : (int64_t)tl.z * p.g.sy;
      const uint32_t src = tmem_base + ((uint32_t)(lg * 32) << 16) + (uint32_t)(acc * MAX_TN);
      const int most = min(tl.tn, tl.len - tl.tok0);         // tokens of this tile
#pragma unroll 1
      for (int c = 32 * part; c < most; c += 64) {
        float v[32];
        tmem_ld16(src + c, *reinterpret_cast<float(*)[16]>(&v[0]));
        tmem_ld16(src + c + 16, *reinterpret_cast<float(*)[16]>(&v[16]));
        tmem_ld_wait();
        gemm_tc_store32<T>(p.g, out, z_off, n, tl.tok0 + c, tl.tok0 + most, v);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_cluster(map_to_leader(smem_u32(&sh->acc_empty[acc])));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }
  if (sh->abort) wait_settle();
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                            // neither CTA's memory is read or signalled any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

}  // namespace pair

// ------------------------------------------------------------------------------------------------ host
static TcEncodeFn gemm_tc_encode_fn() {
  static TcEncodeFn fn = nullptr;
  if (!fn) {
    void* q = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &q, cudaEnableDefault, &r) == cudaSuccess && r == cudaDriverEntryPointSuccess)
      fn = (TcEncodeFn)q;
  }
  return fn;
}

// [batch][rows][K] 16-bit tensor, box = 64 k x box_rows rows of one batch index, SWIZZLE_128B
static bool gemm_tc_map(TcEncodeFn enc, CUtensorMap* tm, CUtensorMapDataType dt, const void* base, int64_t K, int64_t rows,
                        int64_t batch, int64_t ld, int64_t stride, int box_rows) {
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)(batch > 1 ? stride : ld * rows) * 2};
  cuuint32_t box[3] = {(cuuint32_t)GT_BK, (cuuint32_t)box_rows, 1u};
  cuuint32_t estr[3] = {1u, 1u, 1u};
  return enc(tm, dt, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static void gemm_tc_set_second(GemmTcParams& p, const GemmTcPlain* two, int rows) {
  p.two = {};
  p.out[1] = p.out[0];
  if (!two) return;
  p.out[1] = {two->y, two->N, two->ldy};
  p.two.tokens = two->M;
  p.two.tiles_r = (int)((two->N + rows - 1) / rows);
  p.two.tiles_t = 1;
  p.two.num_tiles = p.two.tiles_r;
  p.two.num_kb = (int)((two->K + GT_BK - 1) / GT_BK);
}

// (pdl_chained: launched programmatically in a mixture and where the caller says that other kernels surround the product; a program may issue any
// number of other products in a row, and streams of nothing but programmatic launches are avoided, moe.cu)
template <typename T, int BN, int STAGES>
static int gemm_tc_run(const CUtensorMap* tm, GemmTcParams p, cudaStream_t st) {
  constexpr size_t smem = 1024 + (size_t)STAGES * (GT_A_BYTES + BN * GT_BK * 2) + sizeof(GemmTcShared);
  auto kern = gemm_tc_kernel<T, BN, STAGES>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(gemm_tc_kernel)");
    attr_set = true;
  }
  if (const int rc = wait_word(WAIT_GEMM_TC, &p.wait_word)) return rc;
  const int tiles = p.num_tiles + p.two.num_tiles, grid = tiles < sm_count() ? tiles : sm_count();
  cudaError_t e = launch_pdl_opt(pdl_chained(), kern, dim3((unsigned)grid), dim3(GT_THREADS), smem, st, tm[0], tm[1], tm[2], tm[3], p);
  if (e != cudaSuccess) return cuda_fail(e, "gemm_tc_kernel launch");
  return B200P_OK;
}

namespace pair {

template <typename T>
static int run(const CUtensorMap* tm, Params p, int64_t tiles, cudaStream_t st) {
  constexpr size_t smem = 1024 + (size_t)STAGES * STAGE_BYTES + sizeof(Shared);
  auto kern = gemm_tc_pair_kernel<T>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(gemm_tc_pair_kernel)");
    attr_set = true;
  }
  if (const int rc = wait_word(WAIT_GEMM_TC, &p.g.wait_word)) return rc;
  const int64_t pairs = sm_count() / 2;
  const unsigned grid = 2u * (unsigned)(tiles < pairs ? tiles : pairs);
  cudaError_t e = launch_pdl_opt(pdl_chained(), kern, dim3(grid), dim3(THREADS), smem, st, tm[0], tm[1], tm[2], tm[3], p);
  if (e != cudaSuccess) return cuda_fail(e, "gemm_tc_pair_kernel launch");
  return B200P_OK;
}

// Width and number of the token tiles: whole waves of pairs, each as long as the slower of tensor core (2 cycles per token and k-block) and
// operand fetch (16 KB of weights and half the tokens per CTA, at about 70 bytes per cycle).
static void plan(int64_t tokens, int64_t R, int64_t batch, int& tn, int64_t& tiles_t) {
  const int64_t pairs = sm_count() / 2, tiles_r = (R + 255) / 256 * batch, t0 = (tokens + MAX_TN - 1) / MAX_TN, one_wave = pairs / tiles_r;
  double best = 1e300;
  for (int64_t i = 0; i <= 9; ++i) {
    const int64_t n = i < 9 ? t0 + i : one_wave > t0 ? one_wave : t0;
    const int w = (int)(((tokens + n - 1) / n + TN_STEP - 1) / TN_STEP * TN_STEP);
    const int64_t nt = (tokens + w - 1) / w, waves = (tiles_r * nt + pairs - 1) / pairs;
    const double mma = 2.0 * w, fetch = (16384.0 + 64.0 * w) / 70.0, c = (double)waves * (mma > fetch ? mma : fetch);
    if (c < best * 0.999) { best = c; tn = w; tiles_t = nt; }
  }
}

template <typename T>
static int launch(TcEncodeFn enc, const T* x, const T* w, void* y, const int32_t* seg, int64_t x_rows, int64_t tokens, int tn, int64_t tiles_t, int64_t R,
                  int64_t K, int64_t ldx, int64_t ldw, int64_t ldy, int64_t batch, int64_t sx, int64_t sw, int64_t sy, int epi, float2 act,
                  const GemmTcPlain* two, cudaStream_t st) {
  const CUtensorMapDataType dt = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm[4];
  if (!gemm_tc_map(enc, &tm[0], dt, w, K, R, batch, ldw, sw, 128)) return 1;
  Params p;
  p.box = seg ? 64 : tn / 2;
  if (!gemm_tc_map(enc, &tm[1], dt, x, K, x_rows, seg ? 1 : batch, ldx, sx, p.box)) return 1;
  GemmTcParams& g = p.g;
  g.out[0] = {y, R, ldy};
  g.tokens = tokens; g.sy = seg ? 0 : sy;
  g.tiles_r = (int)((R + 255) / 256);
  g.tiles_t = (int)tiles_t;
  const int64_t tiles = (int64_t)g.tiles_r * tiles_t * batch;
  if (tiles >= (1ll << 30)) return 1;
  g.num_tiles = (int)tiles;
  g.num_kb = (int)((K + GT_BK - 1) / GT_BK);
  g.splits = 1; g.kb_per_split = g.num_kb;
  g.seg = seg;
  g.groups = seg ? (int)batch : 0;
  g.epi = epi;
  g.act = act;
  p.tn = tn;
  gemm_tc_set_second(g, two, 256);
  tm[2] = tm[0];
  tm[3] = tm[1];
  if (two) {
    int64_t tiles_t2 = 0;
    plan(two->M, two->N, 1, g.two.tn, tiles_t2);
    g.two.tiles_t = (int)tiles_t2;
    g.two.num_tiles *= (int)tiles_t2;
    if (!gemm_tc_map(enc, &tm[2], dt, two->w, two->K, two->N, 1, two->ldw, 0, 128)) return 1;
    if (!gemm_tc_map(enc, &tm[3], dt, two->x, two->K, two->M, 1, two->ldx, 0, g.two.tn / 2)) return 1;
  }
  return run<T>(tm, p, tiles + g.two.num_tiles, st);
}

}  // namespace pair

// Up to 64 tokens: weights on the M side, tokens on the N side, transposed store, K split where the output is narrow.
template <typename T>
static int gemm_tc_launch_decode(TcEncodeFn enc, const T* x, const T* w, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx, int64_t ldw,
                                 int64_t ldy, int64_t batch, int64_t sx, int64_t sw, int64_t sy, int epi, float2 act, cudaStream_t st) {
  const CUtensorMapDataType dt = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const int bn = M <= 32 ? 32 : 64;
  CUtensorMap tm[4];                               // A = weights (128-row boxes), B = tokens (bn-row boxes)
  if (!gemm_tc_map(enc, &tm[0], dt, w, K, N, batch, ldw, sw, GT_BM)) return 1;
  if (!gemm_tc_map(enc, &tm[1], dt, x, K, M, batch, ldx, sx, bn)) return 1;
  tm[2] = tm[0];
  tm[3] = tm[1];
  GemmTcParams p;
  p.out[0] = {y, N, ldy};
  p.tokens = M; p.sy = sy;
  p.tiles_r = (int)((N + GT_BM - 1) / GT_BM);
  p.tiles_t = 1;
  p.num_kb = (int)((K + GT_BK - 1) / GT_BK);
  const int64_t tiles = (int64_t)p.tiles_r * batch;
  if (tiles >= (1ll << 24)) return 1;
  // few weight tiles and a long K: split K so that about one CTA per SM streams weights, at least 4 k-blocks each
  int splits = 1;
  if (epi == B200P_GEMM_STORE_F32 && batch == 1 && ldy == N && tiles * 2 <= sm_count()) {
    splits = (int)min((int64_t)(sm_count() / tiles), (int64_t)(p.num_kb / 4));
    if (splits < 1) splits = 1;
  }
  p.kb_per_split = (p.num_kb + splits - 1) / splits;
  p.splits = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;          // no empty split
  p.num_tiles = (int)(tiles * p.splits);
  p.seg = nullptr;
  p.groups = 0;
  p.epi = epi;
  p.act = act;
  if (p.splits > 1) {
    cudaError_t e = cudaMemsetAsync(y, 0, (size_t)M * N * sizeof(float), st);
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync(split-K output)");
  }
  gemm_tc_set_second(p, nullptr, GT_BM);
  if (bn == 32) return gemm_tc_run<T, 32, 10>(tm, p, st);
  return gemm_tc_run<T, 64, 8>(tm, p, st);
}

// Which of the two kernels of more than 64 tokens (us, one CTA / pair, bf16).  tiles: of 128 tokens x 64 outputs.
//   16-bit stores: 2048 x 2048 x 128 8.1 / 11.0, x 512 13.4 / 12.9, 4096 x 2048 x 512 16.2 / 20.4, 64 x 1500 x 512 x 128 43 / 85; up to K = 1024 while
//     one wave holds the tiles (512 x 2048 x 1024 8.5 / 9.4; 1024 x 2048 x 1024 13.2 / 11.1);
//   fp32: up to K = 256 (512 x 2048 x 128 4.9 / 5.8, 64 x 512 x 512 x 128 28 / 31, 2048 x 8192 x 256 29.8 / 31.4) unless the output is large (4096 x 8192 x
//     256 59 / 52); up to K = 768 in one wave (512 x 2048 x 512 6.7 / 7.1; 1024 x 2048 x 512 9.2 / 8.5);
//   outputs that fill half of the pair's 256 rows: up to K = 512 (64 x 1500 x 128 x 512 33 / 44), and the narrowest of many tokens at any K
//     (4096 x 16 x 2048 12.1 / 14.4, x 64 12.3 / 11.9).
// Gated units and the activations with exponentials stay with the pair, whose epilogue has twice the warps (128 x 2048 x 128 gated 7.5 / 6.5).
static bool gemm_tc_rows_better(int64_t M, int64_t N, int64_t K, int64_t batch, int epi) {
  if (epi != B200P_GEMM_STORE && epi != B200P_GEMM_RELU_SQ && epi != B200P_GEMM_STORE_F32) return false;
  const int64_t sms = sm_count(), tiles = (M + GT_BM - 1) / GT_BM * ((N + 63) / 64) * batch;
  if ((N <= 128 && K <= 512) || (N <= 32 && M > 1024)) return true;
  if (epi != B200P_GEMM_STORE_F32) return K <= 512 || (K <= 1024 && tiles <= sms);
  return (K <= 256 && tiles <= 14 * sms) || (K <= 768 && tiles <= sms);
}

template <typename T, int BN, int STAGES>
static int gemm_tc_rows_run(const CUtensorMap& tmx, const CUtensorMap& tmw, GemmTcParams p, bool vec, cudaStream_t st) {
  constexpr size_t smem = 1024 + (size_t)STAGES * (GT_A_BYTES + BN * GT_BK * 2) + sizeof(GemmTcShared);
  auto kern = gemm_tc_rows_kernel<T, BN, STAGES>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(gemm_tc_rows_kernel)");
    attr_set = true;
  }
  if (const int rc = wait_word(WAIT_GEMM_TC, &p.wait_word)) return rc;
  const unsigned grid = (unsigned)(p.num_tiles < sm_count() ? p.num_tiles : sm_count());
  cudaError_t e = launch_pdl_opt(pdl_chained(), kern, dim3(grid), dim3(GT_THREADS), smem, st, tmx, tmw, p, vec);
  if (e != cudaSuccess) return cuda_fail(e, "gemm_tc_rows_kernel launch");
  return B200P_OK;
}

template <typename T>
static int gemm_tc_launch_rows(TcEncodeFn enc, const T* x, const T* w, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx, int64_t ldw,
                               int64_t ldy, int64_t batch, int64_t sx, int64_t sw, int64_t sy, int epi, float2 act, cudaStream_t st) {
  // widest weight tile that still gives every SM about two tiles
  const int64_t tiles_t = (M + GT_BM - 1) / GT_BM, want = 2ll * sm_count();
  int bn = 256;
  if (N <= 64 || tiles_t * ((N + 127) / 128) * batch < want) bn = 64;
  else if (N <= 128 || tiles_t * ((N + 255) / 256) * batch < want) bn = 128;
  const int64_t tiles_r = (N + bn - 1) / bn, tiles = tiles_t * tiles_r * batch;
  if (tiles >= (1ll << 30)) return 1;
  const CUtensorMapDataType dt = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tmx, tmw;
  if (!gemm_tc_map(enc, &tmx, dt, x, K, M, batch, ldx, sx, GT_BM)) return 1;
  if (!gemm_tc_map(enc, &tmw, dt, w, K, N, batch, ldw, sw, bn)) return 1;
  GemmTcParams p = {};
  p.out[0] = {y, N, ldy};
  p.tokens = M; p.sy = sy;
  p.tiles_r = (int)tiles_r;
  p.tiles_t = (int)tiles_t;
  p.num_tiles = (int)tiles;
  p.num_kb = (int)((K + GT_BK - 1) / GT_BK);
  p.epi = epi;
  p.act = act;
  const int64_t eb = epi == B200P_GEMM_STORE_F32 ? 4 : 2;
  const bool vec = aligned(y, 16) && (ldy * eb) % 16 == 0 && (batch == 1 || (sy * eb) % 16 == 0);
  if (bn == 256) return gemm_tc_rows_run<T, 256, 4>(tmx, tmw, p, vec, st);
  if (bn == 128) return gemm_tc_rows_run<T, 128, 6>(tmx, tmw, p, vec, st);
  return gemm_tc_rows_run<T, 64, 8>(tmx, tmw, p, vec, st);
}

// Returns B200P_OK, an error, or 1 when the shape is not one this kernel takes (the caller then runs the mma.sync kernel).
template <typename T>
int gemm_tc_launch(const T* x, const T* w, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx, int64_t ldw, int64_t ldy,
                   int64_t batch, int64_t sx, int64_t sw, int64_t sy, int epi, float2 act, cudaStream_t st) {
  if (K < GT_BK || M >= (1ll << 31) || N >= (1ll << 31) || K >= (1ll << 31)) return 1;
  TcEncodeFn enc = gemm_tc_encode_fn();
  if (!enc) return 1;
  if (M <= 64) return gemm_tc_launch_decode<T>(enc, x, w, y, M, N, K, ldx, ldw, ldy, batch, sx, sw, sy, epi, act, st);
  if (gemm_tc_rows_better(M, N, K, batch, epi)) return gemm_tc_launch_rows<T>(enc, x, w, y, M, N, K, ldx, ldw, ldy, batch, sx, sw, sy, epi, act, st);
  int tn = 0;
  int64_t tiles_t = 0;
  pair::plan(M, N, batch, tn, tiles_t);
  return pair::launch<T>(enc, x, w, y, nullptr, M, M, tn, tiles_t, N, K, ldx, ldw, ldy, batch, sx, sw, sy, epi, act, nullptr, st);
}

// Grouped product: x [total_rows, K] holds the groups' rows back to back (group z: rows [seg[z], seg[z+1]), at most max_rows of
// them), w [groups][N][K].  The grid is sized for the tiles that total_rows rows can make, the kernel numbers those that exist.  A tile's
// box may reach into the next group's rows (or past the tensor, which reads zeros): those accumulator columns are not stored.  Groups of at
// most 64 rows (decode steps) take the one-CTA tiles.  `two`: a plain product of max_rows tokens in the same
// launch.  Declined when the groups that can have rows are too few to occupy the SMs.
template <typename T>
int gemm_tc_launch_grouped(const T* x, const T* w, void* y, const int32_t* seg, int64_t total_rows, int64_t max_rows, int64_t N,
                           int64_t K, int64_t ldx, int64_t ldw, int64_t ldy, int64_t groups, int64_t sw, int epi, float2 act,
                           const GemmTcPlain* two, cudaStream_t st) {
  if (two && (two->K < GT_BK || two->M != max_rows || two->N >= (1ll << 31) || two->K >= (1ll << 31))) return 1;
  if (K < GT_BK || total_rows >= (1ll << 31) || N >= (1ll << 31) || K >= (1ll << 31) || groups > GT_MAX_GROUPS) return 1;
  TcEncodeFn enc = gemm_tc_encode_fn();
  if (!enc) return 1;
  if (max_rows > 64) {
    const int64_t tiles_t = min(groups, total_rows) + total_rows / pair::MAX_TN;
    return pair::launch<T>(enc, x, w, y, seg, total_rows, max_rows, 0, (tiles_t + groups - 1) / groups, N, K, ldx, ldw, ldy, groups, 0, sw, 0, epi, act, two, st);
  }
  if (min(groups, total_rows) * ((N + GT_BM - 1) / GT_BM) + (two ? (two->N + GT_BM - 1) / GT_BM : 0) < sm_count()) return 1;
  const int bn = max_rows <= 32 ? 32 : 64;
  const CUtensorMapDataType dt = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUtensorMap tm[4];
  if (!gemm_tc_map(enc, &tm[0], dt, w, K, N, groups, ldw, sw, GT_BM)) return 1;
  if (!gemm_tc_map(enc, &tm[1], dt, x, K, total_rows, 1, ldx, 0, bn)) return 1;
  tm[2] = tm[0];
  tm[3] = tm[1];
  if (two && !(gemm_tc_map(enc, &tm[2], dt, two->w, two->K, two->N, 1, two->ldw, 0, GT_BM) &&
               gemm_tc_map(enc, &tm[3], dt, two->x, two->K, two->M, 1, two->ldx, 0, bn)))
    return 1;
  GemmTcParams p;
  p.out[0] = {y, N, ldy};
  p.tokens = max_rows; p.sy = 0;
  p.tiles_r = (int)((N + GT_BM - 1) / GT_BM);
  p.tiles_t = 1;
  const int64_t nt = (int64_t)p.tiles_r * groups;
  if (nt >= (1ll << 31)) return 1;
  p.num_tiles = (int)nt;
  p.num_kb = (int)((K + GT_BK - 1) / GT_BK);
  p.splits = 1;
  p.kb_per_split = p.num_kb;
  p.seg = seg;
  p.groups = (int)groups;
  p.epi = epi;
  p.act = act;
  gemm_tc_set_second(p, two, GT_BM);
  return bn == 32 ? gemm_tc_run<T, 32, 10>(tm, p, st) : gemm_tc_run<T, 64, 8>(tm, p, st);
}
template int gemm_tc_launch_grouped<__half>(const __half*, const __half*, void*, const int32_t*, int64_t, int64_t, int64_t, int64_t, int64_t,
                                            int64_t, int64_t, int64_t, int64_t, int, float2, const GemmTcPlain*, cudaStream_t);
template int gemm_tc_launch_grouped<__nv_bfloat16>(const __nv_bfloat16*, const __nv_bfloat16*, void*, const int32_t*, int64_t, int64_t,
                                                   int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int, float2, const GemmTcPlain*,
                                                   cudaStream_t);

template int gemm_tc_launch<__half>(const __half*, const __half*, void*, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t,
                                    int64_t, int64_t, int64_t, int64_t, int, float2, cudaStream_t);
template int gemm_tc_launch<__nv_bfloat16>(const __nv_bfloat16*, const __nv_bfloat16*, void*, int64_t, int64_t, int64_t, int64_t,
                                           int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int, float2, cudaStream_t);

}  // namespace b200p

// 0, or 1 + the role (0 loader, 1 MMA issuer, 2 epilogue) of the first wait of a tcgen05 dense GEMM that ran out; reading
// clears it.  Synchronises the device.
extern "C" int b200p_gemm_tc_fault(void) { return b200p::wait_take(b200p::WAIT_GEMM_TC); }
