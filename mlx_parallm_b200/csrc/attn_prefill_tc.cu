// Causal flash-style attention for prefill chunks on tcgen05, 16-bit caches, head_dim 128:
//
//   out[b, l, h, :] = softmax_j( scale * q[b,l,h,:] . K[b, h/G, j, :] ) V[b, h/G, j, :]   for keys j < lengths[b] + l + 1
//
// (the rule of attn_prefill.cu).  The G query heads of a key/value head share its keys, so a tile's 128 rows are (query, head)
// pairs: floor(128 / G) consecutive queries times G heads.  A CTA owns TWO such tiles, consecutive in the sequence, and streams
// every key / value tile once for both: 256 rows per 64 KB of keys and values, which keeps the L2 -> shared-memory traffic at a
// quarter of what one tile per head would need.
//
// Per 128 keys and tile: S = Q K^T into TMEM (8 MMAs of M=128, N=128, K=16), one thread per row reads its 128 scores, keeps the
// running maximum and sum in registers, writes the probabilities as 16-bit A operand over the scores' own TMEM columns, and
// O += P V accumulates in TMEM with V read as it lies in the cache (N-major operand), no transpose anywhere.  The two tiles
// take turns: while one's softmax runs on the CUDA cores, the tensor core works for the other.
// O is rescaled whenever the maximum of one of a warp's rows grows, so a row's largest probability is exactly 1 and carries no
// rounding.  (A maximum that may lag by 2^8 spares most rescales, 455 instead of 510 us for 4096 tokens behind 4096, 40 / 8 heads, bf16, but
// the largest probability is then rounded like the others: 2 % to 14 % more error against 64 bits at scores of deviation 1 to 4, f16 16 %.)
// The sum is taken over the ROUNDED probabilities, so the weights of a row add up to one whatever their rounding.
//
// Bound: the tensor core needs 2048 cycles per 128 keys and CTA, the exponentials 2048 (32768 of them at 16 per cycle and SM).
//
// warp roles (384 threads): warps 0..3 / 4..7 softmax and output of tile 0 / 1 (thread = row), warp 8 MMA issuer (owns TMEM),
// warp 9 TMA producer, warps 10 and 11 only give their registers away.  Shared memory: Q 2 x 32 KB, a ring of five 32 KB slots that alternate K and V tiles.
// Every mbarrier wait is bounded; one that runs out is reported and every role leaves through the common exit.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace b200p {

int sm_count();

constexpr int FT_D = 128, FT_ROWS = 128, FT_KEYS = 128;
constexpr int FT_TILE_BYTES = 128 * FT_D * 2;              // 32 KB: a Q, K or V tile, two halves of [128 rows x 128 bytes]
constexpr int FT_HALF = FT_TILE_BYTES / 2;
constexpr int FT_RING = 5;
constexpr int FT_THREADS = 384;
// registers of 384 threads at launch: 384 x 168 = 64512 = 256 x 216 + 128 x 72, with several items per CTA 256 x 200 + 128 x 104
constexpr int ft_regs_softmax(bool many) { return many ? 200 : 216; }
constexpr int ft_regs_other(bool many) { return many ? 104 : 72; }
constexpr int FT_SMEM = 1024 + (2 + FT_RING) * FT_TILE_BYTES + 256;

struct AttnTcParams {
  const int32_t* lengths;
  void* out;
  int L, Hq, Hkv, G, qpt;       // qpt: queries per tile
  int pairs;                    // items (two tiles) per (row, key/value head)
  int bh, items;                // (row, key/value head)s, and items of the launch
  int64_t Tcap;
  float scale_log2e;
  int out_perm, out_vec;
  int* wait_word;               // where a wait that gives up reports
};

struct AttnTcShared {
  uint64_t q_full, q_empty, kv_full[FT_RING], kv_empty[FT_RING], s_full[2], p_full[2], o_full[2];
  uint32_t tmem_base;
  volatile int abort;
};

__device__ __forceinline__ bool ft_wait(uint32_t bar, uint32_t parity, AttnTcShared* sh, const AttnTcParams& p, int role) {
  return mbar_wait_warp(bar, parity, &sh->abort, p.wait_word, role);
}

__device__ __forceinline__ void ft_tma_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void ft_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
// N-major (rows of the tile = k, 64 n per 128-byte row) SWIZZLE_128B operand: 8-k groups 1024 bytes apart, the next 64 n one half
// tile further
__device__ __forceinline__ uint64_t ft_desc_n_major(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(FT_HALF >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,"
      "%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <typename T> __device__ __forceinline__ uint32_t ft_pack(float a, float b);
template <> __device__ __forceinline__ uint32_t ft_pack<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <> __device__ __forceinline__ uint32_t ft_pack<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <typename T> __device__ __forceinline__ float2 ft_unpack(uint32_t u);
template <> __device__ __forceinline__ float2 ft_unpack<__half>(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
template <> __device__ __forceinline__ float2 ft_unpack<__nv_bfloat16>(uint32_t u) {
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

// MANY: the launch has more items than CTAs
template <typename T, bool MANY>
__global__ void __launch_bounds__(FT_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmq, const __grid_constant__ CUtensorMap tmk,
                       const __grid_constant__ CUtensorMap tmv, const AttnTcParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t ring = base + 2 * FT_TILE_BYTES;
  AttnTcShared* sh = reinterpret_cast<AttnTcShared*>(smem_raw + (base - raw) + (2 + FT_RING) * FT_TILE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&sh->q_full), 1);
    mbar_init(smem_u32(&sh->q_empty), 1);
    for (int s = 0; s < FT_RING; ++s) { mbar_init(smem_u32(&sh->kv_full[s]), 1); mbar_init(smem_u32(&sh->kv_empty[s]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&sh->s_full[i]), 1); mbar_init(smem_u32(&sh->p_full[i]), 4); mbar_init(smem_u32(&sh->o_full[i]), 1); }
    sh->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmq);
    tma_prefetch_desc(&tmk);
    tma_prefetch_desc(&tmv);
  }
  if (warp == 8) tmem_alloc(smem_u32(&sh->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;                     // S of tile i at 128 i (P over its first 64), O of tile i at 256 + 128 i

  // Items are numbered from the longest key range (the last queries) down and dealt to the CTAs in rounds that run back and forth, so that every CTA gets
  // long and short ones.  Barriers, TMEM and ring are set up once per CTA, and the loads and first products of an item pass beside the output of the
  // one before.  us, a CTA per item / so: 4 x 777 tokens, 32 / 8 heads 41.9 / 37.5, 64 / 8 heads 86 / 72; 8 x 1000, 40 / 8 heads 147 / 122; 4096 tokens
  // behind 4096, 40 / 8 heads 360 / 342; 8 x 300 behind 500, 64 / 8 heads 84 / 75.
  struct Item { int b, kvh, l0, len_b, kend, n_tiles; };
  auto place = [&](int it, Item& w) {
    const int pair = p.pairs - 1 - it / p.bh, rest = it % p.bh;
    w.b = rest / p.Hkv, w.kvh = rest - w.b * p.Hkv, w.l0 = pair * 2 * p.qpt;
  };
  auto extent = [&](Item& w) {
    w.len_b = p.lengths[w.b];
    // keys any row of this item may see; at least one, so that rows that see none (negative lengths) come out as NaN from one masked tile
    // instead of waiting for a tile that nobody fetches
    w.kend = max(1, (int)min((int64_t)w.len_b + min(p.L, w.l0 + 2 * p.qpt), p.Tcap));
    w.n_tiles = (w.kend + FT_KEYS - 1) / FT_KEYS;
  };
  auto item_of = [&](int round, Item& w) {
    const int G = (int)gridDim.x, c = (int)blockIdx.x, it = round * G + ((round & 1) ? G - 1 - c : c);
    if (it >= p.items) return false;
    place(it, w);
    extent(w);
    return true;
  };
  Item w;
  if constexpr (!MANY) place((int)blockIdx.x, w);          // (before the wait: 0.5 to 0.8 us of a short call)
  pdl_wait();
  if constexpr (!MANY) extent(w);

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ft_regs_other(MANY)));
   if (warp == 9) {
    // ===================================== TMA producer =====================================
    if (lane == 0) {
      const uint32_t qb = smem_u32(&sh->q_full);
      int slot = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int round = 0; ok && (MANY ? item_of(round, w) : round == 0); ++round) {
        if (MANY && round > 0 && !mbar_wait_lane(smem_u32(&sh->q_empty), (uint32_t)((round - 1) & 1), &sh->abort, p.wait_word, 0)) break;
        mbar_arrive_expect_tx(qb, 4u * (uint32_t)(p.G * p.qpt * 128));
        for (int i = 0; i < 2; ++i)
          for (int hf = 0; hf < 2; ++hf)
            ft_tma_5d(base + i * FT_TILE_BYTES + hf * FT_HALF, &tmq, hf * 64, 0, w.kvh, w.l0 + i * p.qpt, w.b, qb);
        const int z = w.b * p.Hkv + w.kvh;
        for (int issued = 0; issued < 2 * w.n_tiles; ++issued) {                       // K0 V0 K1 V1 ...
          if (!(ok = mbar_wait_lane(smem_u32(&sh->kv_empty[slot]), ph ^ 1u, &sh->abort, p.wait_word, 0))) break;
          const uint32_t bar = smem_u32(&sh->kv_full[slot]), dst = ring + slot * FT_TILE_BYTES;
          mbar_arrive_expect_tx(bar, FT_TILE_BYTES);
          const CUtensorMap* m = (issued & 1) ? &tmv : &tmk;
          tma_load_3d(dst, m, 0, (issued >> 1) * FT_KEYS, z, bar);
          tma_load_3d(dst + FT_HALF, m, 64, (issued >> 1) * FT_KEYS, z, bar);
          if (++slot == FT_RING) { slot = 0; ph ^= 1u; }
        }
      }
    }
   } else if (warp == 8) {
    // ===================================== MMA issuer =======================================
    constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
    constexpr uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    constexpr uint32_t idesc_pv = idesc | (1u << 16);      // B is N-major
    auto qk = [&](int i, int slot) {
      const uint64_t ad = make_desc_sw128(base + i * FT_TILE_BYTES), bd = make_desc_sw128(ring + slot * FT_TILE_BYTES);
#pragma unroll
      for (int k = 0; k < 8; ++k) {                        // 16 k = 32 bytes of a 128-byte row; k 4..7 in the other half tile
        const uint64_t off = (uint64_t)((k & 3) * 2 + (k >> 2) * (FT_HALF >> 4));
        ft_mma_ss(tmem + 128 * i, ad + off, bd + off, idesc, k ? 1u : 0u);
      }
    };
    auto pv = [&](int i, int slot, uint32_t acc) {
      const uint64_t bd = ft_desc_n_major(ring + slot * FT_TILE_BYTES);
#pragma unroll
      for (int k = 0; k < 8; ++k)                          // 16 keys = 2048 bytes; P: 8 columns
        umma_f16_ts(tmem + 256 + 128 * i, tmem + 128 * i + 8 * k, bd + (uint64_t)(k * (2048 >> 4)), idesc_pv, (k || acc) ? 1u : 0u);
    };
    int slot = 0;
    uint32_t ph = 0, pph = 0;                              // phases of `slot` and of the probabilities' barriers
    bool ok = true;
    for (int round = 0; ok && (MANY ? item_of(round, w) : round == 0); ++round) {
      // (the scores' columns are free: their probabilities were multiplied by products issued before, which run in order)
      const int k0 = slot, n_tiles = w.n_tiles;
      if (!(ok = ft_wait(smem_u32(&sh->q_full), (uint32_t)(round & 1), sh, p, 1) && ft_wait(smem_u32(&sh->kv_full[k0]), ph, sh, p, 1))) break;
      if (++slot == FT_RING) { slot = 0; ph ^= 1u; }
      tc_fence_after();
      if (elect_one()) {
        qk(0, k0);
        umma_commit(smem_u32(&sh->s_full[0]));
        qk(1, k0);
        umma_commit(smem_u32(&sh->s_full[1]));
        umma_commit(smem_u32(&sh->kv_empty[k0]));
        if (MANY && n_tiles == 1) umma_commit(smem_u32(&sh->q_empty));
      }
      __syncwarp();
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int vslot = slot;
        if (!(ok = ft_wait(smem_u32(&sh->kv_full[vslot]), ph, sh, p, 1))) break;
        if (++slot == FT_RING) { slot = 0; ph ^= 1u; }
        if (j == n_tiles - 1 && w.kend < n_tiles * FT_KEYS) {
          // the probabilities of keys past kend are zero, but what the cache holds there may not be finite: zero those rows of V
          const int r0 = w.kend - j * FT_KEYS;
          for (int c = lane; c < (FT_KEYS - r0) * 16; c += 32) {
            const int row = r0 + (c >> 4), hf = (c >> 3) & 1, ch = c & 7;
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(ring + vslot * FT_TILE_BYTES + hf * FT_HALF + row * 128 + ch * 16), "r"(0) : "memory");
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
        const bool more = j + 1 < n_tiles;
        const int kslot = slot;
        if (more) {
          if (!(ok = ft_wait(smem_u32(&sh->kv_full[kslot]), ph, sh, p, 1))) break;
          if (++slot == FT_RING) { slot = 0; ph ^= 1u; }
        }
        for (int i = 0; i < 2; ++i) {
          if (!(ok = ft_wait(smem_u32(&sh->p_full[i]), pph, sh, p, 1))) break;
          tc_fence_after();
          if (elect_one()) {
            pv(i, vslot, j > 0 ? 1u : 0u);
            if (i == 1) umma_commit(smem_u32(&sh->kv_empty[vslot]));
            if (more) {
              qk(i, kslot);
              umma_commit(smem_u32(&sh->s_full[i]));
              if (i == 1) umma_commit(smem_u32(&sh->kv_empty[kslot]));
              if (MANY && i == 1 && j + 2 == n_tiles) umma_commit(smem_u32(&sh->q_empty));
            } else {
              umma_commit(smem_u32(&sh->o_full[i]));
            }
          }
          __syncwarp();
        }
        pph ^= 1u;
      }
    }
   }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ft_regs_softmax(MANY)));
    // ===================================== softmax and output ===============================
    const int i = warp >> 2, q = warp & 3;
    const int r = q * 32 + lane;                           // row of the tile = TMEM lane
    const uint32_t s_addr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(128 * i), o_addr = s_addr + 256;
    const int lq = r / p.G, g = r - lq * p.G;              // rows past qpt * G carry nothing and are not stored
    const float2 sc2 = make_float2(p.scale_log2e, p.scale_log2e);
    uint32_t sph = 0;
    bool ok = true;
   for (int round = 0; ok && (MANY ? item_of(round, w) : round == 0); ++round) {
    const int n_tiles = w.n_tiles;
    const int bound = (int)min((int64_t)w.len_b + min(w.l0 + i * p.qpt + lq, p.L - 1) + 1, p.Tcap);
    // tiles below `free_tiles` lie inside the bound of every row of this warp: no masking
    const int l_first = min(w.l0 + i * p.qpt + (q * 32) / p.G, p.L - 1);
    const int free_tiles = (int)min((int64_t)w.len_b + l_first + 1, p.Tcap) / FT_KEYS;
    float m = -INFINITY, sum = 0.f;
    for (int j = 0; j < n_tiles; ++j) {
      if (!(ok = ft_wait(smem_u32(&sh->s_full[i]), sph, sh, p, 2 + i))) break;
      sph ^= 1u;
      tc_fence_after();
      float s[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + 32 * c, s + 32 * c);
      tmem_ld_wait();
      if (j >= free_tiles) {
        const int n = bound - j * FT_KEYS;                 // keys of this tile the row may see
#pragma unroll
        for (int c = 0; c < 128; ++c) s[c] = c < n ? s[c] : -INFINITY;
      }
      float t0 = max3(s[0], s[1], s[2]), t1 = max3(s[3], s[4], s[5]), t2 = max3(s[6], s[7], s[8]), t3 = max3(s[9], s[10], s[11]);
#pragma unroll
      for (int c = 12; c + 8 <= 128; c += 8) {
        t0 = max3(t0, s[c], s[c + 1]);
        t1 = max3(t1, s[c + 2], s[c + 3]);
        t2 = max3(t2, s[c + 4], s[c + 5]);
        t3 = max3(t3, s[c + 6], s[c + 7]);
      }
      t0 = max3(t0, s[124], s[125]);
      t1 = max3(t1, s[126], s[127]);
      const float mt = fmaxf(fmaxf(t0, t1), fmaxf(t2, t3)) * p.scale_log2e;          // (the scale is normal and positive)
      // the first tile holds key 0, which every row sees: m is finite from then on.  O(j - 1) is complete: S(j) was issued behind it
      // Rows whose maximum stays have a factor of exactly one (the vote only skips the work where no row wants it): a row's bits depend
      // on its own scores, not on which tokens and heads share its warp.
      const float mn = fmaxf(m, mt), f = ex2(m - mn);      // (before the first tile f is 0 and nothing is scaled)
      const bool rescale = j > 0 && __any_sync(0xffffffffu, mn > m);
      m = mn;
      const float2 nm2 = make_float2(-m, -m);
      float2 a0 = make_float2(0.f, 0.f), a1 = a0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t u[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const float2 x = __ffma2_rn(make_float2(s[64 * h + 2 * c], s[64 * h + 2 * c + 1]), sc2, nm2);
          u[c] = ft_pack<T>(ex2(x.x), ex2(x.y));
          const float2 e = ft_unpack<T>(u[c]);             // the sum is that of the weights as the product uses them
          if (c & 1) a1 = __fadd2_rn(a1, e); else a0 = __fadd2_rn(a0, e);
        }
        tmem_st32(s_addr + 32 * h, u);
      }
      if (rescale) {                                       // here, where the scores have left their registers: two loads in flight
        const float2 f2 = make_float2(f, f);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float o[2][32];
          tmem_ld32(o_addr + 64 * h, o[0]);
          tmem_ld32(o_addr + 64 * h + 32, o[1]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t u[32];
#pragma unroll
            for (int k = 0; k < 32; k += 2) {
              const float2 w = __fmul2_rn(make_float2(o[c][k], o[c][k + 1]), f2);
              u[k] = __float_as_uint(w.x);
              u[k + 1] = __float_as_uint(w.y);
            }
            tmem_st32(o_addr + 64 * h + 32 * c, u);
          }
        }
      }
      tmem_st_wait();
      sum = sum * f + ((a0.x + a0.y) + (a1.x + a1.y));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->p_full[i]));
    }
    if (ok) ok = ft_wait(smem_u32(&sh->o_full[i]), (uint32_t)(round & 1), sh, p, 2 + i);
    if (!MANY || (round + 1) * (int)gridDim.x >= p.items) pdl_launch_dependents();                 // (the last round)
    if (ok) {
      tc_fence_after();
      const float inv = 1.f / sum;
      if constexpr (MANY) {                                // (where the row goes is worked out anew: the tiles' loop has no registers for it)
        int again = round;
        asm volatile("" : "+r"(again));
        item_of(again, w);
      }
      const int l = w.l0 + i * p.qpt + lq;
      T* dst = reinterpret_cast<T*>(p.out) + (((int64_t)w.b * p.L + min(l, p.L - 1)) * p.Hq + (w.kvh * p.G + g)) * FT_D;
      const bool live = lq < p.qpt && l < p.L;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float o[32];
        tmem_ld32(o_addr + 32 * c, o);
        tmem_ld_wait();
        if (!live) continue;
#pragma unroll
        for (int k = 0; k < 32; k += 8) {                  // PERM8: [0,4,1,5,2,6,3,7]
          float* v = o + k;
          uint32_t u[4];
          if (p.out_perm) {
            u[0] = ft_pack<T>(v[0] * inv, v[4] * inv); u[1] = ft_pack<T>(v[1] * inv, v[5] * inv);
            u[2] = ft_pack<T>(v[2] * inv, v[6] * inv); u[3] = ft_pack<T>(v[3] * inv, v[7] * inv);
          } else {
            u[0] = ft_pack<T>(v[0] * inv, v[1] * inv); u[1] = ft_pack<T>(v[2] * inv, v[3] * inv);
            u[2] = ft_pack<T>(v[4] * inv, v[5] * inv); u[3] = ft_pack<T>(v[6] * inv, v[7] * inv);
          }
          if (p.out_vec) {
            *reinterpret_cast<uint4*>(dst + 32 * c + k) = make_uint4(u[0], u[1], u[2], u[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) reinterpret_cast<uint32_t*>(dst + 32 * c + k)[e] = u[e];
          }
        }
      }
    }
   }
  }
  if (sh->abort) wait_settle();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------------ host
bool attn_prefill_tc_supported(int64_t L, int Hq, int Hkv, int D, int dtype) {
  return L > 1 && D == FT_D && (dtype == B200P_F16 || dtype == B200P_BF16) && Hq % Hkv == 0 && Hq / Hkv <= FT_ROWS;
}

template <typename T, bool MANY>
static int attn_prefill_tc_run(const CUtensorMap* tm, const AttnTcParams& p, unsigned grid, cudaStream_t st) {
  auto kern = attn_prefill_tc_kernel<T, MANY>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FT_SMEM);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(attn_prefill_tc_kernel)");
    attr_set = true;
  }
  launch_pdl(kern, grid, FT_THREADS, FT_SMEM, st, tm[0], tm[1], tm[2], p);
  B200P_LAUNCH_CHECK("attn_prefill_tc_kernel");
  return B200P_OK;
}

int attn_prefill_tc_launch(const void* q, const void* kc, const void* vc, const int32_t* lengths, void* out, int64_t B, int64_t L,
                           int Hq, int Hkv, int D, int64_t Tcap, float scale, int dtype, int out_perm, cudaStream_t st) {
  B200P_REQUIRE(attn_prefill_tc_supported(L, Hq, Hkv, D, dtype), B200P_ERR_ARG, "tensor prefill attention: unsupported shape");
  B200P_REQUIRE(L < (1ll << 30) && Tcap < (1ll << 31) - FT_KEYS && B * Hkv < (1ll << 31), B200P_ERR_ARG, "problem too large");
  B200P_REQUIRE(aligned(q, 16) && aligned(kc, 16) && aligned(vc, 16) && aligned(out, 4), B200P_ERR_ALIGN,
                "q / caches must be 16-byte aligned");
  TcEncodeFn enc = tc_get_encode();
  B200P_REQUIRE(enc != nullptr, B200P_ERR_CUDA, "cuTensorMapEncodeTiled entry point not available");
  AttnTcParams p;
  if (const int rc = wait_word(WAIT_ATTN_TC, &p.wait_word)) return rc;
  p.lengths = lengths; p.out = out; p.L = (int)L; p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv; p.qpt = FT_ROWS / p.G;
  p.pairs = (int)((L + 2 * p.qpt - 1) / (2 * p.qpt));
  p.Tcap = Tcap; p.scale_log2e = scale * 1.4426950408889634f; p.out_perm = out_perm; p.out_vec = aligned(out, 16) ? 1 : 0;
  const int64_t items = (int64_t)p.pairs * B * Hkv;
  B200P_REQUIRE(items < (1ll << 30), B200P_ERR_ARG, "grid too large");
  p.bh = (int)(B * Hkv); p.items = (int)items;
  const unsigned grid = (unsigned)(items < sm_count() ? items : sm_count());
  const CUtensorMapDataType dt = dtype == B200P_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  CUtensorMap tm[3];
  {
    cuuint64_t dims[5] = {FT_D, (cuuint64_t)p.G, (cuuint64_t)Hkv, (cuuint64_t)L, (cuuint64_t)B};
    cuuint64_t str[4] = {FT_D * 2, (cuuint64_t)p.G * FT_D * 2, (cuuint64_t)Hq * FT_D * 2, (cuuint64_t)L * Hq * FT_D * 2};
    cuuint32_t box[5] = {64, (cuuint32_t)p.G, 1, (cuuint32_t)p.qpt, 1}, es[5] = {1, 1, 1, 1, 1};
    CUresult r = enc(&tm[0], dt, 5, const_cast<void*>(q), dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200P_REQUIRE(r == CUDA_SUCCESS, B200P_ERR_CUDA, "cuTensorMapEncodeTiled(q) failed: %d", (int)r);
  }
  for (int i = 0; i < 2; ++i) {
    cuuint64_t dims[3] = {FT_D, (cuuint64_t)Tcap, (cuuint64_t)(B * Hkv)};
    cuuint64_t str[2] = {FT_D * 2, (cuuint64_t)Tcap * FT_D * 2};
    cuuint32_t box[3] = {64, FT_KEYS, 1}, es[3] = {1, 1, 1};
    CUresult r = enc(&tm[1 + i], dt, 3, const_cast<void*>(i ? vc : kc), dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200P_REQUIRE(r == CUDA_SUCCESS, B200P_ERR_CUDA, "cuTensorMapEncodeTiled(cache) failed: %d", (int)r);
  }
  const bool many = items > (int64_t)grid;       // (one item per CTA: the loop over them costs 2 to 5 % of a short call, 2 x 129 tokens 12.2 / 12.9 us)
  if (dtype == B200P_F16) return many ? attn_prefill_tc_run<__half, true>(tm, p, grid, st) : attn_prefill_tc_run<__half, false>(tm, p, grid, st);
  return many ? attn_prefill_tc_run<__nv_bfloat16, true>(tm, p, grid, st) : attn_prefill_tc_run<__nv_bfloat16, false>(tm, p, grid, st);
}

}  // namespace b200p

// 0, or 1 + the role (0 loader, 1 MMA issuer, 2 / 3 softmax) of the first wait of a tcgen05 prefill attention that ran out;
// reading clears it.  Synchronises the device.
extern "C" int b200p_attn_tc_fault(void) { return b200p::wait_take(b200p::WAIT_ATTN_TC); }
