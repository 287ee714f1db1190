// Small-batch (M <= 16) fused-dequant GEMV of b200p_qmm: 4- and 8-bit group-64 weights, 16-bit activations, every epilogue.
//
//   y[m, n] (+)= sum_k x[m, k] * (q[n,k] * s[n, k/64] + b[n, k/64])
//
// A pure weight stream: at HBM speed an SM has 23 bytes, 41 4-bit weights, per cycle to take in, and about 1.9 lane operations per
// weight to spend on them (60 % of its issue slots, so it needs four warps per scheduler to cover their latencies).  What else
// bounds the stream is bytes in flight (a microsecond of latency times 44 KB per microsecond and SM) and the start: every kernel of a
// decode step begins with an empty pipe.  Hence
//   * every warp owns a ring of TMA stages (16 rows x 512 k: codes, scales, biases) that it refills itself, an elected lane issuing, as soon
//     as a stage sits in registers: no producer warp, no barrier between warps, no register spent on loads in flight;
//   * the rings are filled BEFORE griddepcontrol.wait (weights depend on no previous kernel), so under programmatic dependent launch
//     a matrix starts to stream in while its predecessor still computes;
//   * x is staged in shared memory once per CTA, every lane's 16-byte pieces in different banks, PERM8 applied on the way if the
//     caller's layout is the natural one.
// The products run on mma.sync.m16n8k16 straight from registers: lane (g, t) of a warp holds rows g and g + 8 of a tile and, per
// step of 128 packed bytes per row, the 32 bytes [32 t, 32 t + 32) of both (one quantisation group); the MMA's k index is a label,
// A and B use the same one.
//
// Schedule.  A unit is (16-row tile, 512 k).  Epilogues that need whole sums deal whole tiles to the CTAs; the accumulating epilogue
// deals units (panel of k, tile, chunk) evenly whatever N and K are, a panel being as much k as x fits shared memory.  Inside a
// CTA every warp takes an equal contiguous run of units; runs that end inside a tile meet in shared memory once, at the end, and are
// added in a fixed order.  The accumulating epilogue adds one piece of a tile per CTA and panel that holds units of it (a CTA's run is often shorter
// than a tile), in order of arrival: its results are reproducible up to the order of fp32 sums.  (The dispatch takes at most 8 tokens;
// 9 to 16 run when the path is forced.)
//
// Measured (CUDA graph over weight copies larger than L2, us; before: the tile kernel and the register GEMV): gate|up 28672 x 4096 4-bit
// f16 at M = 1 / 4: 16.0 / 17.2 (21.7 / 22.0; with the copies issued under lane == 0 16.5 / 17.9), = 4.1 TB/s at M = 1; 34816 x 5120 at M = 1: 21.4
// (26.8), = 4.7 TB/s; 57344 x 8192 8-bit: 78.5 (92), = 6.3 TB/s; down 4096 x 14336 at M = 1: 11.0 (13.2).  Two warps per scheduler instead of four: 19.1.
//
// Algorithmic HBM bytes per launch: N*K*bits/8 + 2*N*(K/64)*2.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "dequant.cuh"
#include "tc_ptx.cuh"

namespace b200p {

int sm_count();
bool pdl_enabled_gemm();

constexpr int QR_STAGES = 2;
constexpr int QR_UNIT_K = 512;

struct QrParams {
  const void* x;
  void* y;
  int M, N, K, epi, x_perm, y_perm;
  int64_t ldx, ldy;
  int tiles;             // 16-row tiles (SILU_MUL: 8 gate rows and their 8 up rows)
  int chunks;            // K / 512
  int panels;            // k panels of the accumulating epilogue (1: none)
  int* wait_word;        // where a wait that gives up reports
  uint32_t zero;         // 0, which the compiler does not know: a stage is refilled only when what was read from it has arrived in registers, the
                         // addresses of the copies depend on it (what happens otherwise: qmm_wide.cu)
};

// unit u of the linear order (panel, tile, chunk within the panel): panel p covers chunks [p * chunks / panels, (p + 1) * chunks / panels)
struct QrPos { int tile, ch, ch0, ch1; };    // chunk and the panel's chunk range
__device__ __forceinline__ QrPos qr_locate(const QrParams& p, int u) {
  QrPos r;
  int pn = 0;
  r.ch0 = 0;
  r.ch1 = p.chunks / p.panels;
  while (pn + 1 < p.panels && u >= p.tiles * r.ch1) {
    ++pn;
    r.ch0 = r.ch1;
    r.ch1 = (int)(((int64_t)(pn + 1) * p.chunks) / p.panels);
  }
  const int rel = u - p.tiles * r.ch0, n = r.ch1 - r.ch0;
  r.tile = rel / n;
  r.ch = r.ch0 + rel - r.tile * n;
  return r;
}
__device__ __forceinline__ void qr_next(const QrParams& p, QrPos& r) {
  if (++r.ch < r.ch1) return;
  if (++r.tile < p.tiles) { r.ch = r.ch0; return; }
  r.tile = 0;
  const int n = r.ch1;                        // next panel: its end from its index
  int pn = 0;
  while ((int)(((int64_t)(pn + 1) * p.chunks) / p.panels) <= n && pn + 1 < p.panels) ++pn;
  r.ch0 = n;
  r.ch1 = (int)(((int64_t)(pn + 1) * p.chunks) / p.panels);
  r.ch = r.ch0;
}

__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return (uint32_t)v;
}
// (not volatile: the scheduler may move the loads of later operands across it)
template <typename T>
__device__ __forceinline__ void qr_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __half>::value) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

template <typename T, int NT>
__device__ __forceinline__ void qr_emit(const QrParams& p, int tile, int g, int t, const float (&acc)[NT][4]) {
  const bool silu = p.epi == B200P_EPI_SILU_MUL;
  const int r0 = silu ? tile * 8 + g : tile * 16 + g, r1 = r0 + 8;
#pragma unroll
  for (int n = 0; n < NT; ++n) {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int tok = 8 * n + 2 * t + j;
      if (tok >= p.M) continue;
      const float a = acc[n][j], b = acc[n][2 + j];
      if (silu) {
        reinterpret_cast<T*>(p.y)[tok * p.ldy + (p.y_perm ? perm8_pos(r0) : r0)] = Tr<T>::from_f(silu_tc(a) * b);
      } else if (p.epi == B200P_EPI_STORE) {
        T* y = reinterpret_cast<T*>(p.y) + tok * p.ldy;
        y[p.y_perm ? perm8_pos(r0) : r0] = Tr<T>::from_f(a);
        y[p.y_perm ? perm8_pos(r1) : r1] = Tr<T>::from_f(b);
      } else {
        float* y = reinterpret_cast<float*>(p.y) + tok * p.ldy;
        if (p.epi == B200P_EPI_ADD_RESIDUAL) {
          atomicAdd(y + r0, a);
          atomicAdd(y + r1, b);
        } else {
          y[r0] = a;
          y[r1] = b;
        }
      }
    }
  }
}

// NW warps; FAST: the small-scale dequant of dequant.cuh (caller promised B200P_W_SMALLSCALE): A and the sums are produced at
// 1 / SmallScaleOut<T>; NT: n-tiles of 8 tokens.
template <typename T, int BITS, bool FAST, int NT, int NW>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
qmv_ring_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_s,
                const __grid_constant__ CUtensorMap tm_b, const QrParams p) {
  constexpr int STEP_K = 1024 / BITS;                      // k per step of 128 packed bytes per row
  constexpr int STEPS = QR_UNIT_K / STEP_K;                // 2 at 4 bits, 4 at 8
  constexpr int CODE_BYTES = 2 * STEPS * 1024;             // [rows g | rows g + 8][step][8 rows][128 bytes]
  constexpr int SCALE_BYTES = 512;                         // scales, biases of both row groups: 4 x [8 rows][8 groups]
  constexpr int PARK_BYTES = NT * 4 * 32 * 4;              // a warp's sums of one tile
  constexpr int PIECES = STEP_K / 32;                      // 16-byte pieces of x per lane and step (8 codes each): 8 / 4
  constexpr int SEG = PIECES * 16 + 16;                    // a lane's piece of x in shared memory, padded: the four t of a row differ in bank
  constexpr int X_STEP = 4 * SEG;                          // per token and step: a multiple of 64, not of 128: two tokens differ too
  constexpr uint32_t S = QR_STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring0 = (raw + 1023u) & ~1023u;
  const uint32_t sc_ring0 = ring0 + NW * S * CODE_BYTES;   // (code stages start on 1024-byte boundaries: SWIZZLE_128B)
  const uint32_t park0 = sc_ring0 + NW * S * SCALE_BYTES;
  const uint32_t x_base = park0 + NW * PARK_BYTES;
  __shared__ __align__(8) uint64_t bars[NW * QR_STAGES];
  __shared__ int seg_of[NW];                               // the tile, opened by an earlier warp, that a warp left a piece of
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bool silu = p.epi == B200P_EPI_SILU_MUL;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;
  int c0, c1;                                              // the CTA's units
  if (p.epi == B200P_EPI_ADD_RESIDUAL) {
    const int64_t U = (int64_t)p.tiles * p.chunks;
    c0 = (int)(U * cta / G);
    c1 = (int)(U * (cta + 1) / G);
  } else {
    c0 = (int)((int64_t)p.tiles * cta / G) * p.chunks;
    c1 = (int)((int64_t)p.tiles * (cta + 1) / G) * p.chunks;
  }
  const int nu = c1 - c0;
  const int u0 = c0 + (int)((int64_t)nu * warp / NW), u1 = c0 + (int)((int64_t)nu * (warp + 1) / NW);
  const uint32_t my_ring = ring0 + (uint32_t)warp * S * CODE_BYTES, my_scales = sc_ring0 + (uint32_t)warp * S * SCALE_BYTES;
  const uint32_t my_bar = smem_u32(&bars[warp * QR_STAGES]);
  if (lane == 0) {
    for (uint32_t s = 0; s < S; ++s) mbar_init(my_bar + 8 * s, 1);
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  __syncwarp();
  QrPos pr = qr_locate(p, u0 < u1 ? u0 : c0);              // position of the next unit to fetch
  int pu = u0;
  auto fetch = [&](uint32_t stage, uint32_t after) {        // (after: 0, known when the stage has been read: QrParams::zero)
    if (elect_one()) {                                       // (not `lane == 0`: operands of warp-uniform code need no uniformising)
      const uint32_t bar = my_bar + 8 * stage + after, dst = my_ring + stage * CODE_BYTES + after, sdst = my_scales + stage * SCALE_BYTES + after;
      const int ra = silu ? pr.tile * 8 : pr.tile * 16, rb = silu ? p.N / 2 + ra : ra + 8;
      mbar_arrive_expect_tx(bar, CODE_BYTES + SCALE_BYTES);
      tma_load_3d(dst, &tm_w, 0, ra, pr.ch * STEPS, bar);
      tma_load_3d(dst + CODE_BYTES / 2, &tm_w, 0, rb, pr.ch * STEPS, bar);
      tma_load_2d(sdst, &tm_s, pr.ch * 8, ra, bar);
      tma_load_2d(sdst + 128, &tm_b, pr.ch * 8, ra, bar);
      tma_load_2d(sdst + 256, &tm_s, pr.ch * 8, rb, bar);
      tma_load_2d(sdst + 384, &tm_b, pr.ch * 8, rb, bar);
    }
    __syncwarp();
    ++pu;
    qr_next(p, pr);
  };
  QrPos at = pr;                                           // position of the unit being computed
  for (uint32_t s = 0; s < S && pu < u1; ++s) fetch(s, 0);
  pdl_launch_dependents();
  pdl_wait();                                              // x is the previous kernel's output; y its accumulator

  // ---- x of the CTA's k range: [step][token][4 lanes][pieces]
  const QrPos first = qr_locate(p, c0), last = qr_locate(p, nu > 0 ? c1 - 1 : c0);
  const int k0 = first.ch0 * QR_UNIT_K, k1 = last.ch1 * QR_UNIT_K;
  {
    const int per_row = (k1 - k0) / 8;                     // 16-byte pieces per token
    const T* xs = reinterpret_cast<const T*>(p.x) + k0;
    for (int i = threadIdx.x; i < per_row * p.M; i += NW * 32) {
      const int m = i / per_row, c = i - m * per_row;
      uint4 v = *reinterpret_cast<const uint4*>(xs + (int64_t)m * p.ldx + 8 * c);
      if (BITS == 4 && !p.x_perm) {                        // natural order -> (x0,x4) (x1,x5) (x2,x6) (x3,x7)
        const uint4 u = v;
        v.x = prmt(u.x, u.z, 0x5410u);
        v.y = prmt(u.x, u.z, 0x7632u);
        v.z = prmt(u.y, u.w, 0x5410u);
        v.w = prmt(u.y, u.w, 0x7632u);
      }
      const int st = c / (4 * PIECES), in = c - st * 4 * PIECES;
      const uint32_t dst = x_base + (uint32_t)((st * p.M + m) * X_STEP + (in / PIECES) * SEG + (in % PIECES) * 16);
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    }
  }
  __syncthreads();

  float acc[NT][4], acc2[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[n][j] = acc2[n][j] = 0.f;
  uint32_t stage = 0, ph = 0;
  int parked0 = -1, parked1 = -1;                          // the tile whose piece this warp left in shared memory / still holds
  float* park = reinterpret_cast<float*>(smem_raw + (park0 - raw) + warp * PARK_BYTES);
  // columns of tokens past M are never stored: their lanes read the last token's x (a broadcast) instead of zeros
  const uint8_t* x_mine = smem_raw + (x_base - raw) + min(g, p.M - 1) * X_STEP + t * SEG;
  const int x_second = (min(8 + g, p.M - 1) - min(g, p.M - 1)) * X_STEP, x_step = p.M * X_STEP;
  int seg_start = u0;                                      // first unit of the current tile that this warp computed
  bool ok = true;
  for (int u = u0; u < u1; ++u) {
    if (!(ok = mbar_wait_warp(my_bar + 8 * stage, ph, nullptr, p.wait_word, 0))) break;      // (a warp's stages are its own: it gives up alone)
    const uint32_t sb = my_ring + stage * CODE_BYTES + g * 128, ss = my_scales + stage * SCALE_BYTES + g * 16;
    const uint8_t* xs = x_mine + ((at.ch * QR_UNIT_K - k0) / STEP_K) * x_step;
#pragma unroll
    for (int half = 0; half < STEPS / 2; ++half) {
      uint4 qa[2][2], qb[2][2];
      uint32_t sva[2], bva[2], svb[2], bvb[2];
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {
        const int c = 2 * half + c2;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t ch = (uint32_t)(((2 * t + h) ^ g) << 4);
          qa[c2][h] = lds128(sb + c * 1024 + ch);
          qb[c2][h] = lds128(sb + CODE_BYTES / 2 + c * 1024 + ch);
        }
        const int grp = BITS == 4 ? 4 * c + t : 2 * c + (t >> 1);
        sva[c2] = lds_u16(ss + 2 * grp);
        bva[c2] = lds_u16(ss + 128 + 2 * grp);
        svb[c2] = lds_u16(ss + 256 + 2 * grp);
        bvb[c2] = lds_u16(ss + 384 + 2 * grp);
      }
      if (half == STEPS / 2 - 1) {
        uint32_t all = 0;
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) all |= qa[c2][0].w | qa[c2][1].w | qb[c2][0].w | qb[c2][1].w | sva[c2] | bva[c2] | svb[c2] | bvb[c2];
        all &= p.zero;
        __syncwarp();                                      // the stage sits in registers: hand it back to the stream
        if (pu < u1) fetch(stage, all);
      }
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {
        const int c = 2 * half + c2;
        const uint32_t s2a = sva[c2] | (sva[c2] << 16), b2a = bva[c2] | (bva[c2] << 16);
        const uint32_t s2b = svb[c2] | (svb[c2] << 16), b2b = bvb[c2] | (bvb[c2] << 16);
        const uint32_t* pa = reinterpret_cast<const uint32_t*>(qa[c2]);
        const uint32_t* pb = reinterpret_cast<const uint32_t*>(qb[c2]);
        SmallScale ca, cb;
        if constexpr (FAST) { ca = small_scale_prep<T>(s2a, b2a); cb = small_scale_prep<T>(s2b, b2b); }
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
          uint32_t da[4], db[4];
          if constexpr (FAST) {
            dequant8_small<T, BITS, true>(pa + i * (BITS / 4), ca, da);
            dequant8_small<T, BITS, true>(pb + i * (BITS / 4), cb, db);
          } else {
            dequant8<T, BITS, true>(pa + i * (BITS / 4), s2a, b2a, da);
            dequant8<T, BITS, true>(pb + i * (BITS / 4), s2b, b2b, db);
          }
          const uint32_t a_lo[4] = {da[0], db[0], da[1], db[1]};
          const uint32_t a_hi[4] = {da[2], db[2], da[3], db[3]};
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const uint4 xv = *reinterpret_cast<const uint4*>((n == 0 ? xs : xs + x_second) + c * x_step + i * 16);
            qr_mma<T>(acc[n], a_lo, xv.x, xv.y);
            qr_mma<T>(acc2[n], a_hi, xv.z, xv.w);
          }
        }
      }
    }
    if (++stage == S) { stage = 0; ph ^= 1u; }
    // ---- end of the tile, of the panel or of this warp's run: the sums leave the accumulators
    const bool tile_ends = at.ch + 1 == at.ch1;
    if (tile_ends || u + 1 == u1) {
      constexpr float D = FAST ? SmallScaleOut<T>::value : 1.f;
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc[n][j] = (acc[n][j] + acc2[n][j]) * D; acc2[n][j] = 0.f; }
      const int ub = u - (at.ch - at.ch0);                 // the tile's first unit: names the (panel, tile)
      const bool opens = seg_start <= max(ub, c0);         // this warp holds the tile's first unit of the CTA ...
      const bool closes = tile_ends || u + 1 == c1;        // ... and its last
      if (opens && !closes) {
        parked1 = ub;                                      // the run ends here: the sums stay in the accumulators
      } else {
        if (opens) {
          qr_emit<T, NT>(p, at.tile, g, t, acc);
        } else {
          parked0 = ub;
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int j = 0; j < 4; ++j) park[(n * 4 + j) * 32 + lane] = acc[n][j];
        }
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
      }
      seg_start = u + 1;
    }
    if (u + 1 < u1) qr_next(p, at);
  }
  if (!ok) wait_settle();
  // ---- tiles shared by several warps of the CTA: the warp that opened a tile adds the others' pieces in warp order
  if (lane == 0) seg_of[warp] = parked0;
  __syncthreads();
  if (parked1 != -1 && ok) {
    for (int w = warp + 1; w < NW; ++w) {
      if (seg_of[w] != parked1) continue;                  // (warps without units lie in between)
      const float* q = park + (w - warp) * (PARK_BYTES / 4);
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] += q[(n * 4 + j) * 32 + lane];
    }
    qr_emit<T, NT>(p, at.tile, g, t, acc);
  }
}

// ------------------------------------------------------------------------------------------------ host
bool qmv_ring_supported(int64_t M, int64_t N, int64_t K, int gs, int bits, int dtype, int epi) {
  if (gs != 64 || (bits != 4 && bits != 8) || (dtype != B200P_F16 && dtype != B200P_BF16)) return false;
  if (M < 1 || M > 16 || K % QR_UNIT_K != 0 || N % 16 != 0) return false;
  if (epi < 0 || epi > 3 || N >= (1ll << 27) || K >= (1ll << 27) || (N / 16 + 1) * (K / QR_UNIT_K) >= (1ll << 30)) return false;
  return true;
}

constexpr int QR_SMEM_HALF = 112 * 1024, QR_SMEM_FULL = 224 * 1024;

struct QrPlan { int nw, grid, panels, smem; };
// Two CTAs of 8 warps per SM where x fits twice beside their rings, else one of 16 warps, else (8-bit stages are twice as large) one
// of 8; the fewest panels of k first, since every panel's sums are added to y on their own.
static bool qr_plan(int64_t M, int64_t tiles, int64_t chunks, int bits, int epi, QrPlan* pl) {
  const int stage = 2 * (QR_UNIT_K * bits / 8) * 8 + 512, x_per_k = bits == 4 ? 9 : 10;      // x bytes per token per 4 k, padding included
  const int park = M <= 8 ? 512 : 1024;
  const bool add = epi == B200P_EPI_ADD_RESIDUAL;
  const struct { int nw, per_sm, limit; } shapes[3] = {{8, 2, QR_SMEM_HALF}, {16, 1, QR_SMEM_FULL}, {8, 1, QR_SMEM_FULL}};
  for (int64_t pn = 1; pn <= (add ? (chunks < 16 ? chunks : 16) : 1); ++pn) {
    for (const auto& sh : shapes) {
      const int64_t work = add ? tiles * chunks : tiles, slots = (int64_t)sm_count() * sh.per_sm;
      const int64_t grid = work < slots ? work : slots, upc = (tiles * chunks + grid - 1) / grid;
      const int64_t fixed = 1024 + (int64_t)sh.nw * (QR_STAGES * stage + park);
      // a CTA's units reach over as many panels as its share of them is long, and one more boundary
      const int64_t panel = (chunks + pn - 1) / pn;
      int64_t span = pn == 1 ? chunks : ((upc + tiles * (chunks / pn) - 1) / (tiles * (chunks / pn)) + 1) * panel;
      if (span > chunks) span = chunks;
      const int64_t xb = M * span * QR_UNIT_K * x_per_k / 4;
      if (fixed + xb > sh.limit) continue;
      pl->nw = sh.nw; pl->grid = (int)grid; pl->panels = (int)pn; pl->smem = (int)(fixed + xb);
      return true;
    }
  }
  return false;
}

template <typename T, int BITS, bool FAST, int NT, int NW>
static int qr_run(const CUtensorMap* tm, const QrParams& p, const QrPlan& pl, cudaStream_t st) {
  auto kern = qmv_ring_kernel<T, BITS, FAST, NT, NW>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, QR_SMEM_FULL);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(qmv_ring_kernel)");
    attr_set = true;
  }
  cudaError_t e = launch_pdl_opt(pdl_enabled_gemm(), kern, pl.grid, NW * 32, pl.smem, st, tm[0], tm[1], tm[2], p);
  if (e != cudaSuccess) return cuda_fail(e, "qmv_ring_kernel launch");
  return B200P_OK;
}

// Returns B200P_OK, an error, or 1 when x does not fit beside the rings (the caller then takes another kernel).
int qmv_ring_launch(const void* x, const uint32_t* w, const void* s, const void* b, void* y, int64_t M, int64_t N, int64_t K, int64_t ldx,
                    int64_t ldy, int bits, int dtype, int epi, int flags, cudaStream_t st) {
  QrParams p;
  p.zero = 0;
  p.x = x; p.y = y; p.M = (int)M; p.N = (int)N; p.K = (int)K; p.epi = epi; p.ldx = ldx; p.ldy = ldy;
  p.x_perm = (flags & B200P_X_PERM8) ? 1 : 0;
  p.y_perm = (flags & B200P_Y_PERM8) ? 1 : 0;
  p.tiles = (int)(N / 16);
  p.chunks = (int)(K / QR_UNIT_K);
  QrPlan pl;
  if (!qr_plan(M, p.tiles, p.chunks, bits, epi, &pl)) return 1;
  p.panels = pl.panels;
  if (const int rc = wait_word(WAIT_QMV_RING, &p.wait_word)) return rc;
  TcEncodeFn enc = tc_get_encode();
  B200P_REQUIRE(enc != nullptr, B200P_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  const CUtensorMapDataType dt16 = dtype == B200P_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tm[3];
  const int64_t row_bytes = K * bits / 8;
  {
    const int steps = QR_UNIT_K * bits / 1024;
    cuuint64_t dims[3] = {128, (cuuint64_t)N, (cuuint64_t)(row_bytes / 128)}, str[2] = {(cuuint64_t)row_bytes, 128};
    cuuint32_t box[3] = {128, 8, (cuuint32_t)steps}, es[3] = {1, 1, 1};
    CUresult r = enc(&tm[0], CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint32_t*>(w), dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200P_REQUIRE(r == CUDA_SUCCESS, B200P_ERR_CUDA, "cuTensorMapEncodeTiled(weights) failed: %d", (int)r);
  }
  for (int i = 0; i < 2; ++i) {
    cuuint64_t dims[2] = {(cuuint64_t)(K / 64), (cuuint64_t)N}, str[1] = {(cuuint64_t)(K / 64) * 2};
    cuuint32_t box[2] = {8, 8}, es[2] = {1, 1};
    CUresult r = enc(&tm[1 + i], dt16, 2, const_cast<void*>(i ? b : s), dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200P_REQUIRE(r == CUDA_SUCCESS, B200P_ERR_CUDA, "cuTensorMapEncodeTiled(scales) failed: %d", (int)r);
  }
  const bool fast = (flags & B200P_W_SMALLSCALE) != 0;
#define GO2(T_, B_, F_, N_) (pl.nw == 8 ? qr_run<T_, B_, F_, N_, 8>(tm, p, pl, st) : qr_run<T_, B_, F_, N_, 16>(tm, p, pl, st))
#define GO(T_, B_, F_) (M <= 8 ? GO2(T_, B_, F_, 1) : GO2(T_, B_, F_, 2))
  if (dtype == B200P_F16) {
    if (bits == 4) return fast ? GO(__half, 4, true) : GO(__half, 4, false);
    return fast ? GO(__half, 8, true) : GO(__half, 8, false);
  }
  if (bits == 4) return fast ? GO(__nv_bfloat16, 4, true) : GO(__nv_bfloat16, 4, false);
  return fast ? GO(__nv_bfloat16, 8, true) : GO(__nv_bfloat16, 8, false);
#undef GO
#undef GO2
}

}  // namespace b200p

// 1 after a TMA stage of qmv_ring_kernel failed to arrive in about a second; reading clears it.  Synchronises the device.
extern "C" int b200p_qmv_fault(void) { return b200p::wait_take(b200p::WAIT_QMV_RING); }
