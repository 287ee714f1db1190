"""Kernel-level parity: every C-ABI entry point against the oracle on the same seeded inputs."""
import os

import numpy as np
import pytest
import torch

from oracle import mlx_ops as ref
from helpers import rel_err

pytestmark = pytest.mark.gpu

TD = {"float32": torch.float32, "float16": torch.float16, "bfloat16": torch.bfloat16}


def t_(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(TD[dtype]).cuda()


def w_(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def bits_of(t, dtype):
    if dtype == "float32":
        return t.cpu().numpy().view(np.uint32)
    return t.cpu().view(torch.int16).numpy().view(np.uint16)


@pytest.fixture(scope="module")
def ops():
    from mlx_parallm_b200 import ops as o, _lib
    _lib.require_device()
    return o


# ---------------------------------------------------------------- dequantize: bit-exact, all modes
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_dequantize_bit_exact_golden(ops, golden_dir, bits, dtype, mode):
    g = np.load(os.path.join(golden_dir, "dequantize_bits.npz"))
    out = ops.dequantize(w_(g[f"w_{bits}"]), t_(g[f"s_{bits}_{dtype}"], dtype), t_(g[f"b_{bits}_{dtype}"], dtype), 64, bits, mode)
    assert np.array_equal(bits_of(out, dtype), g[f"out_{bits}_{dtype}_{mode}"])


@pytest.mark.parametrize("bits,dtype", [(4, "float16"), (8, "bfloat16"), (4, "float32")])
def test_dequantize_bit_exact_random_large(ops, bits, dtype):
    rng = np.random.default_rng(11)
    N, K = 257, 4096
    wq = rng.integers(0, 2 ** 32, (N, K * bits // 32), dtype=np.uint32)
    s = ref.round_to(rng.uniform(-0.02, 0.02, (N, K // 64)), dtype)
    b = ref.round_to(rng.uniform(-0.2, 0.2, (N, K // 64)), dtype)
    for mode in (0, 1, 2):
        out = ops.dequantize(w_(wq), t_(s, dtype), t_(b, dtype), 64, bits, mode)
        exp = ref.storage_bits(ref.dequantize(wq, s, b, 64, bits, dtype, mode), dtype)
        assert np.array_equal(bits_of(out, dtype), exp), mode


def test_dequantize_empty_and_embed_gather(ops):
    rng = np.random.default_rng(12)
    V, K = 300, 128
    wq = rng.integers(0, 2 ** 32, (V, K // 8), dtype=np.uint32)
    s = ref.round_to(rng.uniform(-0.02, 0.02, (V, 2)), "float16")
    b = ref.round_to(rng.uniform(-0.2, 0.2, (V, 2)), "float16")
    out = ops.dequantize(w_(wq[:0]), t_(s[:0], "float16"), t_(b[:0], "float16"))
    assert out.shape == (0, K)
    ids = np.array([5, 0, 299, 5, 17], np.int32)
    e = ops.embed(torch.from_numpy(ids).cuda(), w_(wq), t_(s, "float16"), t_(b, "float16"))
    exp = ref.dequantize(wq[ids], s[ids], b[ids], 64, 4, "float16")
    assert e.dtype == torch.float32 and np.array_equal(e.cpu().numpy(), exp)


# ---------------------------------------------------------------- quantize: bit-exact (codes, scales, biases)
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("gs", [32, 64, 128])
def test_quantize_bit_exact(ops, bits, dtype, gs):
    rng = np.random.default_rng(bits * 100 + gs)
    N, K = 37, 512
    w = rng.standard_normal((N, K)).astype(np.float32) * 0.05
    w[0] = 0.0                                     # all-zero groups: scale falls back to eps, codes 0
    if dtype != "float16":
        w[1] = 0.031                               # constant groups (in f16 edge / eps overflows: NaN codes in MLX and the oracle alike)
    w[2, :gs] = -np.abs(w[2, :gs])                 # min side dominates -> positive scale
    w[3, :gs] = np.abs(w[3, :gs])                  # max side dominates -> negative scale
    w[4, ::2] = 0.0                                # zeros must be exactly representable
    w = ref.round_to(w, dtype)
    eq, es, eb = ref.quantize(w, gs, bits, dtype)
    gq, gsx, gb = ops.quantize(t_(w, dtype), gs, bits)
    assert np.array_equal(gq.cpu().numpy().view(np.uint32), eq)
    assert np.array_equal(bits_of(gsx, dtype), ref.storage_bits(es, dtype))
    assert np.array_equal(bits_of(gb, dtype), ref.storage_bits(eb, dtype))


def test_quantize_dequantize_roundtrip_full_size(ops):
    """Size-independent property at a full-size shape (down_proj of Llama-3-8B): dequantize(quantize(w)) is within half a
    quantisation step (+ storage rounding) of w, group by group, and quantising the dequantised matrix again reproduces
    the codes (idempotence)."""
    g = torch.Generator(device="cuda").manual_seed(4)
    w = (torch.randn((4096, 14336), generator=g, device="cuda") * 0.02).to(torch.float16)
    wq, s, b = ops.quantize(w, 64, 4)
    d = ops.dequantize(wq, s, b, 64, 4)
    step = s.float().abs().repeat_interleave(64, 1)
    # the scale is snapped to edge / rint(edge / scale), so the far end of a group may clip by up to ~0.8 step
    assert bool(((d.float() - w.float()).abs() <= 1.0 * step + 4e-3 * w.float().abs() + 1e-5).all())
    assert float(((d.float() - w.float()).abs() / step).mean()) < 0.3
    wq2, s2, b2 = ops.quantize(d, 64, 4)
    d2 = ops.dequantize(wq2, s2, b2, 64, 4)
    assert float((d2.float() - d.float()).abs().max()) <= float(step.max()) * 1.01


# ---------------------------------------------------------------- quantized matmul
def qmm_case(ops, M, N, K, bits, dtype, epi, seed=0, path=0, ragged_ld=False, small_scale=False):
    from mlx_parallm_b200 import _lib
    rng = np.random.default_rng(seed)
    wq = rng.integers(0, 2 ** 32, (N, K * bits // 32), dtype=np.uint32)
    nb = (1 << bits) - 1
    s = ref.round_to(rng.uniform(0.5, 1.5, (N, K // 64)) * rng.choice([-1, 1], (N, K // 64)) * (2 / nb) / np.sqrt(K), dtype)
    b = ref.round_to(-s * nb / 2 + rng.normal(0, 0.01 / np.sqrt(K), (N, K // 64)), dtype)
    x = ref.round_to(rng.standard_normal((M, K)), dtype)
    acc = ref.quantized_matmul_grouped(x, wq, s, b, 64, bits) if M * N * K <= 2 ** 24 else \
        ref.quantized_matmul(x, wq, s, b, 64, bits).astype(np.float64)
    xt = t_(x, dtype)
    if ragged_ld:
        big = torch.zeros((M, K + 64), dtype=xt.dtype, device="cuda")
        big[:, :K] = xt
        xt = big[:, :K]
    ws = torch.zeros((max(ops.qmm_workspace_bytes(M, N, K), 16),), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().b200p_qmm_set_path(path))
    try:
        if epi == _lib.EPI_ADD_RESIDUAL:
            res = rng.standard_normal((M, N)).astype(np.float32)
            out = torch.from_numpy(res.copy()).cuda()
            ops.qmm(xt, w_(wq), t_(s, dtype), t_(b, dtype), 64, bits, epi, out=out, workspace=ws, small_scale=small_scale)
            exp = res + acc
        else:
            out = ops.qmm(xt, w_(wq), t_(s, dtype), t_(b, dtype), 64, bits, epi, workspace=ws, small_scale=small_scale)
            if epi == _lib.EPI_SILU_MUL:
                g, u = acc[:, :N // 2], acc[:, N // 2:]
                exp = g / (1 + np.exp(-g)) * u
            else:
                exp = acc
    finally:
        _lib.lib().b200p_qmm_set_path(0)
    return out.float().cpu().numpy(), exp


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("M", [1, 3, 8])
def test_qmv_store_matches_oracle(ops, dtype, bits, M):
    got, exp = qmm_case(ops, M, 96, 512, bits, dtype, 0, seed=M, path=1)
    tol = {"float32": 2e-5, "float16": 2e-3, "bfloat16": 1e-2}[dtype]     # output rounding of the storage type
    assert rel_err(got, exp) < tol


@pytest.mark.parametrize("epi", [1, 2, 3])
def test_qmv_epilogues(ops, epi):
    got, exp = qmm_case(ops, 5, 128, 256, 4, "float16", epi, seed=epi, path=1, ragged_ld=True)
    assert rel_err(got, exp) < (2e-3 if epi == 3 else 2e-5)


def test_qmv_tiny_model_shapes(ops):
    # K = 64 (one group per row, tiny hidden) and K = 128 (tiny down_proj), float32 like config 1
    for K in (64, 128):
        got, exp = qmm_case(ops, 8, 64, K, 4, "float32", 1, seed=K, path=1)
        assert rel_err(got, exp) < 2e-5


def test_qmm_rejects_bad_arguments(ops):
    from mlx_parallm_b200 import _lib
    x = torch.zeros((1, 96), dtype=torch.float16, device="cuda")
    w = torch.zeros((4, 12), dtype=torch.int32, device="cuda")
    s = torch.zeros((4, 1), dtype=torch.float16, device="cuda")
    with pytest.raises(_lib.B200PError):
        ops.qmm(x, w, s, s, 64, 4)                      # K=96 not a multiple of group 64


# ---------------------------------------------------------------- rmsnorm / rope+append / attention
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_rmsnorm(ops, dtype):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((7, 512)).astype(np.float32) * 3
    w = ref.round_to(1 + 0.1 * rng.standard_normal(512), dtype)
    y = ops.rmsnorm(torch.from_numpy(x).cuda(), t_(w, dtype), 1e-5)
    exp = ref.rms_norm(x, w, 1e-5, dtype)
    # identical up to 1 ulp of the storage type (fp32 reduction order differs)
    assert rel_err(y.float().cpu().numpy(), exp) < {"float32": 1e-6, "float16": 1.1e-3, "bfloat16": 8.1e-3}[dtype]


@pytest.mark.parametrize("dtype,M,H", [
    ("float16", 8, 4096),       # one pass (16-bit rows of up to 16384), two groups of 8 per thread
    ("float16", 1, 4096),
    ("bfloat16", 8, 5120),      # three
    ("float16", 64, 4096),      # (Llama-3-8B decode at B=64)
    ("bfloat16", 32, 8192),     # four (70B-class)
    ("float16", 16, 2048),      # one
    ("bfloat16", 64, 5120),     # (Qwen3-14B)
    ("float16", 100, 4096),
    ("bfloat16", 8, 16392),     # wider: two passes, below 16 rows 256 threads
    ("float16", 16, 16392),     # from 16 rows on the early kernel of 128
    ("bfloat16", 40, 20480),
])
@pytest.mark.parametrize("perm", [False, True])
def test_rmsnorm_variants_at_decode_sizes(ops, dtype, M, H, perm):
    """Every RMSNorm variant the dispatcher can pick (csrc/elementwise.cu), PERM8 and plain, against the oracle."""
    rng = np.random.default_rng(31)
    x = rng.standard_normal((M, H)).astype(np.float32) * 3
    x[M // 2] *= 50.0                               # rows of very different norms
    w = ref.round_to(1 + 0.1 * rng.standard_normal(H), dtype)
    y = ops.rmsnorm(torch.from_numpy(x).cuda(), t_(w, dtype), 1e-5, out_perm=perm).float().cpu().numpy()
    if perm:                                        # undo [0,4,1,5,2,6,3,7] inside every aligned group of 8
        y = y.reshape(M, H // 8, 8)[:, :, [0, 2, 4, 6, 1, 3, 5, 7]].reshape(M, H)
    exp = ref.rms_norm(x, w, 1e-5, dtype)
    for r in range(M):                              # per row: a row of small norm must not hide behind a large one
        assert rel_err(y[r], exp[r]) < {"float16": 1.1e-3, "bfloat16": 8.1e-3}[dtype], r


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("H", [8, 1016, 1024, 1032, 3584, 7176, 8192, 8200, 16384, 16392])   # groups per thread, partly filled ones, beyond
@pytest.mark.parametrize("M", [1, 17])
def test_rmsnorm_one_pass_at_every_width(ops, dtype, H, M):
    """16-bit rows of any number of whole groups of 8, plain and PERM8, against 64 bits; neighbours of the output stay as they were.

    Tolerance per element: half an ulp of the storage type (relative ``u``), plus the fp32 arithmetic before it: a thread's 64
    terms, 5 steps of the warp, 8 of the block, halved by the square root, and 5 more roundings, below 64 * 2^-24 together; plus
    half the smallest subnormal of fp16."""
    rng = np.random.default_rng(H + M)
    x = rng.standard_normal((M, H)).astype(np.float32) * 3
    x[M // 2] *= 50.0
    w = ref.round_to(1 + 0.1 * rng.standard_normal(H), dtype)
    want = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-5) * np.asarray(w, np.float64)
    u = {"float16": 2.0 ** -11, "bfloat16": 2.0 ** -8}[dtype]
    for perm in (False, True):
        buf = torch.full((M + 2, H), 7.0, dtype=TD[dtype], device="cuda")
        ops.rmsnorm(torch.from_numpy(x).cuda(), t_(w, dtype), 1e-5, out_perm=perm, out=buf[1:-1])
        got = buf.float().cpu().numpy()
        assert (got[0] == 7).all() and (got[-1] == 7).all()
        y = got[1:-1]
        if perm:
            y = y.reshape(M, H // 8, 8)[:, :, [0, 2, 4, 6, 1, 3, 5, 7]].reshape(M, H)
        assert (np.abs(y - want) <= np.abs(want) * (u + 64 * 2.0 ** -24) + 2.0 ** -25).all()


@pytest.mark.parametrize("H", [1024, 4096, 5120, 8192, 16384])
def test_rmsnorm_of_weights_that_the_kernel_before_writes(ops, H):
    """A norm that starts while the kernel before it still runs reads nothing of its, weights included: chains of two norms, the second's weights an output of the
    first, give the bits of the same calls one at a time."""
    g, n = torch.Generator(device="cuda").manual_seed(H), 24
    x = torch.randn(n, 150, H, generator=g, device="cuda")
    row, w0 = torch.randn(1, H, generator=g, device="cuda"), torch.randn(H, generator=g, device="cuda").bfloat16()

    def chain(apart):
        buf, outs = torch.full((150, H), 3.0, dtype=torch.bfloat16, device="cuda"), torch.empty(n, 1, H, dtype=torch.bfloat16, device="cuda")
        for i in range(n):
            ops.rmsnorm(x[i], w0, 1e-5, out=buf)
            if apart:
                torch.cuda.synchronize()
            ops.rmsnorm(row, buf[149], 1e-5, out=outs[i])
            if apart:
                torch.cuda.synchronize()
        return outs

    want = chain(True)
    assert torch.equal(chain(False), want)
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        got = chain(False)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype,D,qk_norm", [("float16", 128, False), ("bfloat16", 128, True), ("float32", 16, False), ("float16", 64, True)])
def test_rope_kv_append(ops, dtype, D, qk_norm):
    rng = np.random.default_rng(4)
    B, L, Hq, Hkv, Tcap = 3, 2, 4, 2, 40
    lengths = np.array([0, 7, 33], np.int32)
    qkv = ref.round_to(rng.standard_normal((B * L, (Hq + 2 * Hkv) * D)), dtype)
    qn = ref.round_to(1 + 0.1 * rng.standard_normal(D), dtype)
    kn = ref.round_to(1 + 0.1 * rng.standard_normal(D), dtype)
    q_out = torch.zeros((B, L, Hq, D), dtype=TD[dtype], device="cuda")
    kc = torch.zeros((B, Hkv, Tcap, D), dtype=TD[dtype], device="cuda")
    vc = torch.zeros_like(kc)
    ops.rope_kv_append(t_(qkv, dtype), q_out, kc, vc, torch.from_numpy(lengths).cuda(), B, L, Hq, Hkv, D, 10000.0, 1.0,
                       t_(qn, dtype) if qk_norm else None, t_(kn, dtype) if qk_norm else None, 1e-6)
    r = qkv.reshape(B, L, Hq + 2 * Hkv, D)
    q, k, v = r[:, :, :Hq], r[:, :, Hq:Hq + Hkv], r[:, :, Hq + Hkv:]
    if qk_norm:
        q = ref.rms_norm(q, qn, 1e-6, dtype)
        k = ref.rms_norm(k, kn, 1e-6, dtype)
    qe = ref.rope(q.transpose(0, 2, 1, 3), lengths, 10000.0, 1.0, dtype).transpose(0, 2, 1, 3)
    ke = ref.rope(k.transpose(0, 2, 1, 3), lengths, 10000.0, 1.0, dtype)
    tol = {"float32": 3e-6, "float16": 1.5e-3, "bfloat16": 1e-2}[dtype]
    assert rel_err(q_out.float().cpu().numpy(), qe) < tol
    kcn, vcn = kc.float().cpu().numpy(), vc.float().cpu().numpy()
    for b in range(B):
        s = lengths[b]
        assert rel_err(kcn[b, :, s:s + L], ke[b]) < tol
        assert np.array_equal(vcn[b, :, s:s + L], v[b].transpose(1, 0, 2))
        assert not kcn[b, :, s + L:].any() and not kcn[b, :, :s].any()      # nothing else touched


@pytest.mark.parametrize("D", [128, 64])          # the head_dim-128 warp kernel and the generic one
def test_rope_kv_append_counts_rows_beyond_capacity(ops, D):
    """A row whose position reached Tcap cannot be appended: the kernel drops it and bumps the per-device counter that
    b200p_kv_overflow_count reads (and the generation loop checks); rows with room are written as usual."""
    B, L, Hq, Hkv, Tcap = 3, 1, 4, 2, 8
    ops.kv_overflow_count(reset=True)
    lengths = torch.tensor([3, 8, 9], dtype=torch.int32, device="cuda")       # row 0 fits, rows 1 and 2 are full
    qkv = torch.randn((B * L, (Hq + 2 * Hkv) * D), device="cuda").to(torch.float16)
    q_out = torch.zeros((B, L, Hq, D), dtype=torch.float16, device="cuda")
    kc = torch.zeros((B, Hkv, Tcap, D), dtype=torch.float16, device="cuda")
    vc = torch.zeros_like(kc)
    ops.rope_kv_append(qkv, q_out, kc, vc, lengths, B, L, Hq, Hkv, D, 10000.0)
    assert ops.kv_overflow_count() == 2 * Hkv                 # one count per dropped (token, V head)
    assert ops.kv_overflow_count(reset=True) == 2 * Hkv       # reading does not clear; reset returns the old value
    assert ops.kv_overflow_count() == 0
    v_row0 = qkv[0].view(Hq + 2 * Hkv, D)[Hq + Hkv:]
    assert torch.equal(vc[0, :, 3], v_row0) and not vc[1:].any() and not kc[1:].any()
    ops.rope_kv_append(qkv[:1], q_out[:1], kc[:1], vc[:1], lengths[:1], 1, L, Hq, Hkv, D, 10000.0)
    assert ops.kv_overflow_count() == 0                       # nothing dropped: the counter stays clear


@pytest.mark.parametrize("dtype,B,L,Hq,Hkv,norm", [
    ("float16", 1, 256, 4, 2, False),             # the smallest call of the row kernel: one token per CTA
    ("bfloat16", 3, 211, 5, 1, True),             # 633 tokens: two per CTA, the last CTA half empty
    ("float16", 2, 601, 3, 3, True),              # 1202 tokens: four per CTA
    ("bfloat16", 1, 2371, 40, 8, True),           # eight per CTA, more heads than walkers
])
def test_rope_kv_append_prompt_rows(ops, dtype, B, L, Hq, Hkv, norm):
    """Calls of 256 tokens and more (16-byte accesses, angles shared by the heads) against the per-head kernel fed the same tokens in
    smaller portions.  Without norms bit for bit; with them the sum of squares runs in another order: one rounding of the result."""
    D, dt = 128, TD[dtype]
    g = torch.Generator(device="cuda").manual_seed(L)
    qkv = torch.randn((B, L, (Hq + 2 * Hkv) * D), generator=g, device="cuda").to(dt)
    wq, wk = ((1 + 0.1 * torch.randn(D, generator=g, device="cuda")).to(dt) if norm else None for _ in range(2))
    lengths = torch.tensor([3 * b for b in range(B)], dtype=torch.int32, device="cuda")
    cap = L + 3 * (B - 1) - 1                     # the last row's last token does not fit
    res = []
    for portion in (L, 200 // B):
        q = torch.zeros((B, L, Hq, D), dtype=dt, device="cuda")
        kc, vc = (torch.zeros((B, Hkv, cap, D), dtype=dt, device="cuda") for _ in range(2))
        ops.kv_overflow_count(reset=True)
        for l in range(0, L, portion):
            n = min(portion, L - l)
            qo = torch.zeros((B, n, Hq, D), dtype=dt, device="cuda")
            ops.rope_kv_append(qkv[:, l:l + n].contiguous(), qo, kc, vc, lengths + l, B, n, Hq, Hkv, D, 10000.0, 1.0, wq, wk, 1e-6)
            q[:, l:l + n] = qo
        res.append((q, kc, vc, ops.kv_overflow_count(reset=True)))
    (q, kc, vc, n), (q2, kc2, vc2, n2) = res
    assert n == n2 == Hkv and torch.equal(vc, vc2)
    for a, b in ((q, q2), (kc, kc2)):
        if not norm:
            assert torch.equal(a, b)
        else:
            ulp = 2.0 ** (-10 if dtype == "float16" else -7)
            assert (a.float() - b.float()).abs().max() <= 2 * ulp * b.float().abs().max() and (a != b).float().mean() < 1e-2


def attn_case(ops, B, L, Hq, Hkv, D, lengths, dtype, path, seed=5):
    from mlx_parallm_b200 import _lib
    rng = np.random.default_rng(seed)
    Tcap = int(max(lengths)) + L + 3
    q = ref.round_to(rng.standard_normal((B, L, Hq, D)), dtype)
    k = ref.round_to(rng.standard_normal((B, Hkv, Tcap, D)), dtype)
    v = ref.round_to(rng.standard_normal((B, Hkv, Tcap, D)), dtype)
    out = torch.zeros((B, L, Hq * D), dtype=TD[dtype], device="cuda")
    ws = torch.empty((max(ops.attn_workspace_bytes(B, L, Hq, D), 16),), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().b200p_attn_set_path(path))
    try:
        ops.attn(t_(q, dtype), t_(k, dtype), t_(v, dtype), torch.from_numpy(np.asarray(lengths, np.int32)).cuda(), out,
                 B, L, Hq, Hkv, D, D ** -0.5, workspace=ws)
    finally:
        _lib.lib().b200p_attn_set_path(0)
    exp = np.zeros((B, L, Hq * D), np.float32)
    for b in range(B):
        T = lengths[b] + L
        mask = ref.additive_causal_mask_variable(L, [lengths[b]], T)
        o = ref.sdpa(q[b:b + 1].transpose(0, 2, 1, 3), k[b:b + 1, :, :T], v[b:b + 1, :, :T], D ** -0.5, mask if L > 1 else None)
        exp[b] = o.transpose(0, 2, 1, 3).reshape(L, Hq * D)
    return out.float().cpu().numpy(), exp


@pytest.mark.parametrize("dtype,D,Hq,Hkv", [("float32", 16, 4, 4), ("float16", 128, 8, 2), ("bfloat16", 128, 5, 1), ("float16", 64, 4, 2)])
def test_attention_generic_decode_ragged_lengths(ops, dtype, D, Hq, Hkv):
    got, exp = attn_case(ops, 3, 1, Hq, Hkv, D, [0, 5, 130], dtype, path=1)
    assert rel_err(got, exp) < {"float32": 2e-5, "float16": 1.5e-3, "bfloat16": 1e-2}[dtype]


def test_attention_generic_prefill_causal(ops):
    got, exp = attn_case(ops, 2, 9, 4, 2, 64, [0, 4], "float16", path=1)
    assert rel_err(got, exp) < 1.5e-3


@pytest.mark.parametrize("dtype,B,L,Hq,Hkv,lengths", [
    ("float16", 2, 70, 8, 2, [0, 37]),            # two query tiles per row, ragged cache offsets
    ("bfloat16", 3, 9, 5, 1, [0, 4, 130]),        # fewer queries than a tile, G = 5
    ("float16", 1, 200, 4, 4, [64]),              # several key tiles, MHA
    ("float16", 2, 64, 8, 8, [0, 0]),             # exactly one query tile, pure causal
])
@pytest.mark.parametrize("path", [2, 4])
def test_attention_tensor_prefill_causal(ops, dtype, B, L, Hq, Hkv, lengths, path):
    """Tensor prefill against the oracle's SDPA with the additive causal mask: as dispatched (the second and the last case on mma.sync,
    attn_prefill.cu, the others on tcgen05) and all of it on mma.sync."""
    got, exp = attn_case(ops, B, L, Hq, Hkv, 128, lengths, dtype, path=path)
    assert rel_err(got, exp) < {"float16": 2e-3, "bfloat16": 1.2e-2}[dtype]
    gen, _ = attn_case(ops, B, L, Hq, Hkv, 128, lengths, dtype, path=1)
    assert rel_err(got, gen) < {"float16": 2e-3, "bfloat16": 1.2e-2}[dtype]


@pytest.mark.parametrize("dtype,B,L,Hq,Hkv,lengths", [
    ("float16", 1, 2, 4, 1, [0]),                 # the smallest call: two queries, one key tile
    ("float16", 2, 31, 8, 2, [97, 96]),           # keys end at / one short of a tile edge (128)
    ("bfloat16", 2, 33, 8, 2, [96, 230]),         # one key past a tile edge; a second, nearly empty query tile
    ("float16", 1, 129, 4, 4, [0]),               # one head per key head: 128 queries per tile, one in the second
    ("bfloat16", 1, 26, 10, 2, [127]),            # five heads per key head: 125 of 128 rows of a tile
    ("float16", 3, 70, 16, 1, [0, 300, 700]),     # sixteen heads per key head, more key tiles than ring slots
    ("bfloat16", 1, 300, 6, 2, [40]),             # three heads per key head, several query tiles
])
@pytest.mark.parametrize("perm", [False, True])
def test_attention_tcgen05_prefill(ops, dtype, B, L, Hq, Hkv, lengths, perm):
    """attn_prefill_tc.cu against the oracle's SDPA at the edges of its tiles.  The cache holds NaN behind the last key, scores reach
    far apart (rows dominated by one key).  Tolerances as for the mma.sync kernel: the same roundings (probabilities, output)."""
    from mlx_parallm_b200 import _lib
    D, dt, scale = 128, TD[dtype], 128 ** -0.5
    rng = np.random.default_rng(L)
    Tcap = max(lengths) + L + 3
    q = (rng.standard_normal((B, L, Hq, D)) * 3).astype(np.float32)
    k = rng.standard_normal((B, Hkv, Tcap, D)).astype(np.float32)
    v = rng.standard_normal((B, Hkv, Tcap, D)).astype(np.float32)
    qt, kt, vt = (torch.from_numpy(a).to(dt).cuda() for a in (q, k, v))
    exp = np.zeros((B, L, Hq * D))
    for b in range(B):
        n = lengths[b] + L
        kt[b, :, n:], vt[b, :, n:] = float("nan"), float("nan")
        kb, vb = (t[b, :, :n].double().cpu().repeat_interleave(Hq // Hkv, 0) for t in (kt, vt))
        s = torch.einsum("lhd,htd->hlt", qt[b].double().cpu(), kb) * scale
        s.masked_fill_(torch.arange(n)[None, None] > (lengths[b] + torch.arange(L))[None, :, None], -float("inf"))
        exp[b] = torch.einsum("hlt,htd->lhd", s.softmax(-1), vb).reshape(L, Hq * D).numpy()
    out = torch.full((B, L, Hq * D), 7.0, dtype=dt, device="cuda")
    ws = torch.empty((max(ops.attn_workspace_bytes(B, L, Hq, D), 16),), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().b200p_attn_set_path(3))
    try:
        ops.attn(qt, kt, vt, torch.tensor(lengths, dtype=torch.int32, device="cuda"), out, B, L, Hq, Hkv, D, scale, workspace=ws, out_perm=perm)
    finally:
        _lib.lib().b200p_attn_set_path(0)
    assert _lib.lib().b200p_attn_tc_fault() == 0
    got = out.float().cpu().numpy()
    if perm:                                              # undo [0,4,1,5,2,6,3,7] inside every group of 8
        got = got.reshape(B, L, -1, 8)[..., [0, 2, 4, 6, 1, 3, 5, 7]].reshape(B, L, Hq * D)
    assert rel_err(got, exp) < {"float16": 2e-3, "bfloat16": 1.2e-2}[dtype]


def prefill(ops, q, k, v, lengths, scale, path=0):
    """ops.attn over prompts: q [B, L, Hq, D], k / v [B, Hkv, Tcap, D] -> [B, L, Hq, D]."""
    from mlx_parallm_b200 import _lib
    B, L, Hq, D = q.shape
    out = torch.full((B, L, Hq * D), 7.0, dtype=q.dtype, device="cuda")
    ws = torch.empty((max(ops.attn_workspace_bytes(B, L, Hq, D), 16),), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().b200p_attn_set_path(path))
    try:
        ops.attn(q, k, v, torch.tensor(lengths, dtype=torch.int32, device="cuda"), out, B, L, Hq, k.shape[1], D, scale, workspace=ws)
    finally:
        _lib.lib().b200p_attn_set_path(0)
    assert _lib.lib().b200p_attn_tc_fault() == 0
    return out.view(B, L, Hq, D)


def prefill_exact(q, k, v, lengths, scale):
    """The same in 64 bits."""
    B, L, Hq, D = q.shape
    out = torch.empty((B, L, Hq, D), dtype=torch.float64, device="cuda")
    for b in range(B):
        n = lengths[b] + L
        kb, vb = (t[b, :, :n].double().repeat_interleave(Hq // k.shape[1], 0) for t in (k, v))
        s = torch.einsum("lhd,htd->hlt", q[b].double(), kb) * scale
        s.masked_fill_(torch.arange(n, device="cuda")[None, None] > (lengths[b] + torch.arange(L, device="cuda"))[None, :, None], -float("inf"))
        out[b] = torch.einsum("hlt,htd->lhd", s.softmax(-1), vb)
    return out


def prefill_inputs(dtype, B, L, Hq, Hkv, Tcap, seed, spread=1.0):
    """Queries, keys, values; scores q.k / sqrt(128) have standard deviation ``spread``."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda *shape: torch.randn(shape, generator=g, device="cuda")
    return (r(B, L, Hq, 128) * spread).to(TD[dtype]), r(B, Hkv, Tcap, 128).to(TD[dtype]), r(B, Hkv, Tcap, 128).to(TD[dtype])


@pytest.mark.parametrize("B,L,Hq,Hkv,T", [(20, 50, 32, 8, 0), (8, 300, 32, 8, 77), (3, 700, 40, 8, 300), (5, 513, 64, 8, 0), (40, 2, 8, 8, 130)])
def test_attention_tcgen05_prefill_of_more_items_than_sms(ops, B, L, Hq, Hkv, T):
    """CTAs that take several items in turn (items of one key tile, two to four rounds, the last one partly filled) give the bits of every sequence
    alone, whose items all have a CTA of their own; sequences of different lengths."""
    from mlx_parallm_b200 import _lib
    D, g, dt = 128, torch.Generator(device="cuda").manual_seed(B + L), torch.bfloat16
    cap = -(-(T + L) // 128) * 128 + 128
    q = torch.randn(B * L, Hq * D, generator=g, device="cuda").to(dt)
    kc, vc = (torch.randn(B, Hkv, cap, D, generator=g, device="cuda").to(dt) for _ in range(2))
    lengths = torch.tensor([T - (i * 7) % (T + 1) for i in range(B)], dtype=torch.int32, device="cuda")
    out, alone = torch.zeros_like(q), torch.zeros_like(q)
    _lib.lib().b200p_attn_set_path(3)
    try:
        ops.attn(q, kc, vc, lengths, out, B, L, Hq, Hkv, D, D ** -0.5)
        for b in range(B):
            rows = slice(b * L, (b + 1) * L)
            ops.attn(q[rows], kc[b:b + 1], vc[b:b + 1], lengths[b:b + 1], alone[rows], 1, L, Hq, Hkv, D, D ** -0.5)
    finally:
        _lib.lib().b200p_attn_set_path(0)
    assert _lib.lib().b200p_attn_tc_fault() == 0
    assert torch.equal(out, alone) and bool(out.isfinite().all())


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("scale", [0.0, 1e-44, 1e-39, -0.11, 2e-38])
@pytest.mark.parametrize("path", [0, 3])
def test_attention_prefill_of_scales_that_are_not_normal_positive_numbers(ops, dtype, scale, path):
    """Scale 0 is the mean of the visible values (masked scores stay masked), as are scales below the normal numbers; 2e-38 is the
    smallest kind that the tcgen05 kernel takes; negative scales prefer the least similar keys.  70 tokens over up to 370 positions: beyond the rule for
    the smallest calls.  Tolerances as for the other prefill tests."""
    q, k, v = prefill_inputs(dtype, 2, 70, 8, 2, 400, seed=3)
    got = prefill(ops, q, k, v, [0, 300], scale, path)
    exp = prefill_exact(q, k, v, [0, 300], scale)
    assert torch.isfinite(got).all()
    assert rel_err(got.float().cpu().numpy(), exp.cpu().numpy()) < {"float16": 2e-3, "bfloat16": 1.2e-2}[dtype]


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("path", [3, 4])
def test_attention_prefill_rows_do_not_depend_on_their_neighbours(ops, dtype, path):
    """A token's output is a function of its own query and the keys before it, bit for bit: other tokens' and heads' scores grow at other
    tiles, and a prompt cut into two portions puts a token into another tile row beside other tokens."""
    q, k, v = prefill_inputs(dtype, 1, 150, 8, 2, 1300, seed=11, spread=2.0)
    one = prefill(ops, q, k, v, [1100], 128 ** -0.5, path)
    other = q.clone()
    other[:, 1::2] *= 3
    other[:, :, ::4] = 0
    keep = torch.zeros((1, 150, 8, 1), dtype=torch.bool, device="cuda")
    keep[:, ::2] = True
    keep[:, :, ::4] = False
    two = prefill(ops, other, k, v, [1100], 128 ** -0.5, path)
    assert torch.equal(one.masked_fill(~keep, 0), two.masked_fill(~keep, 0))
    for cut in (37, 90):
        parts = [prefill(ops, q[:, a:b].contiguous(), k, v, [1100 + a], 128 ** -0.5, path) for a, b in ((0, cut), (cut, 150))]
        assert torch.equal(one, torch.cat(parts, 1))


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("spread", [1.0, 2.0, 4.0])
def test_attention_tcgen05_prefill_is_as_exact_as_the_mma_sync_kernel(ops, dtype, spread):
    """Error against 64 bits over 6000 keys, from flat rows to rows that one key dominates.  Both kernels round the probabilities and the
    output to 16 bits; over half a million outputs their errors agree to better than a percent if nothing else is rounded."""
    q, k, v = prefill_inputs(dtype, 1, 64, 64, 8, 6064, seed=int(spread), spread=spread)
    exp = prefill_exact(q, k, v, [6000], 128 ** -0.5)
    err = {path: float((prefill(ops, q, k, v, [6000], 128 ** -0.5, path).double() - exp).norm() / exp.norm()) for path in (3, 4)}
    assert err[3] < 1.01 * err[4], err


def test_attention_prefill_of_rows_that_see_no_key(ops):
    """Negative cache lengths: tokens without a visible key are NaN on both kernels, the others are as usual; no wait runs out."""
    q, k, v = prefill_inputs("float16", 3, 70, 8, 2, 400, seed=5)
    lengths = [-500, -30, 200]
    for path in (3, 4):
        got = prefill(ops, q, k, v, lengths, 128 ** -0.5, path)
        assert torch.isnan(got[0]).all() and torch.isnan(got[1, :30]).all()
        exp = prefill_exact(q[1:, 30:].contiguous(), k[1:], v[1:], [0, 230], 128 ** -0.5)
        assert rel_err(got[1:, 30:].float().cpu().numpy(), exp.cpu().numpy()) < 2e-3


# ---------------------------------------------------------------- samplers
def test_argmax_ties_and_probs(ops):
    rng = np.random.default_rng(6)
    lg = rng.standard_normal((5, 1000)).astype(np.float32)
    lg[0, 17] = lg[0, 900] = 9.0                       # tie -> lowest index
    lg[1, 999] = 12.0
    probs = torch.zeros(5, device="cuda")
    tok = ops.argmax(torch.from_numpy(lg).cuda(), probs_out=probs)
    assert tok.tolist() == ref.argmax_tokens(lg)[:, 0].tolist() and tok[0].item() == 17
    sm = ref.softmax(lg)
    assert np.allclose(probs.cpu().numpy(), sm[np.arange(5), tok.cpu().numpy()], rtol=1e-4)


def test_argmax_large_vocab_unaligned(ops):
    rng = np.random.default_rng(7)
    lg = rng.standard_normal((3, 151937)).astype(np.float32)
    t = torch.from_numpy(lg).cuda()
    assert ops.argmax(t).tolist() == lg.argmax(-1).tolist()


@pytest.mark.parametrize("B,V", [(1, 1), (2, 3), (1, 32), (3, 4101), (1, 32000), (5, 16384 * 8 + 4), (300, 70)])
def test_argmax_and_probability_at_segment_edges(ops, B, V):
    """Segments, loads and warps that are not full, rows that no 16-byte load reads, ties, NaN, rows of -inf and a row with +inf.

    Tolerance of the probability: __expf is right to 2 ulp of its argument's product, here at most 2^-22 * 16, for two of them and two
    roundings of each of the 20 sums in a chain: 1e-5 of the value."""
    rng = np.random.default_rng(V)
    for ld in (V, (V + 3) // 4 * 4, V + 1):
        lg = (rng.standard_normal((B, V)) * 3).astype(np.float32)
        lg[0, V // 2] = lg[0, V - 1] = 9.0                  # tie (the lower index wins)
        if B > 1:
            lg[1] = -np.inf
        if B > 2:
            lg[2, ::2] = np.nan
        buf = torch.full((B, ld), 50.0, device="cuda")
        buf[:, :V] = torch.from_numpy(lg)
        probs = torch.full((B,), -1.0, device="cuda")
        tok = ops.argmax(buf[:, :V], probs_out=probs).tolist()
        fin = np.where(np.isnan(lg), -np.inf, lg).astype(np.float64)
        assert tok == fin.argmax(-1).tolist()
        with np.errstate(invalid="ignore"):
            want = 1.0 / np.exp(fin - fin.max(-1, keepdims=True)).sum(-1)
        want[np.isnan(want)] = 0.0                          # nothing but -inf
        assert np.allclose(probs.cpu().numpy(), want, rtol=1e-5, atol=0)
        buf[0, V // 3] = float("inf")
        tok = ops.argmax(buf[:, :V], probs_out=probs)
        assert int(tok[0]) == V // 3 and float(probs[0]) == 0.0


@pytest.mark.parametrize("top_p,temp", [(0.9, 1.0), (0.5, 0.7), (1.0, 1.3)])
def test_top_p_sampling_distribution(ops, top_p, temp):
    """Distributional parity (A.7: MLX's threefry stream is not reproducible outside MLX): draws must stay in
    the oracle's nucleus and match its renormalised probabilities (chi-square style bound on the big bins)."""
    rng = np.random.default_rng(8)
    V, n = 200, 20000
    lg = (rng.standard_normal(V) * 2.0).astype(np.float32)
    dist = ref.top_p_distribution(lg[None], top_p, temp)[0]
    logits = torch.from_numpy(np.tile(lg, (n, 1))).cuda()
    tok = ops.sample_top_p(logits, temp, top_p, seed=123, offset=0).cpu().numpy()
    assert dist[tok].min() > 0, "sampled a token outside the nucleus"
    freq = np.bincount(tok, minlength=V) / n
    big = dist > 0.01
    assert np.abs(freq[big] - dist[big]).max() < 4 * np.sqrt(dist[big].max() / n) + 2e-3
    tok2 = ops.sample_top_p(logits, temp, top_p, seed=123, offset=0).cpu().numpy()
    assert np.array_equal(tok, tok2)                     # counter-based RNG: reproducible
    tok3 = ops.sample_top_p(logits, temp, top_p, seed=123, offset=1).cpu().numpy()
    assert not np.array_equal(tok, tok3)


@pytest.mark.parametrize("V,top_p,temp", [(128256, 0.9, 0.7), (151937, 0.6, 1.0), (32000, 0.95, 1.2)])
def test_top_p_large_vocab_stays_in_the_oracle_nucleus(ops, V, top_p, temp):
    """Full vocabulary sizes (151 937 = unaligned rows -> scalar loads): LM-like logits (a gaussian body, a few large values,
    a block of exactly equal logits as untrained vocab slots have), 1500 draws: every token inside the oracle's nucleus,
    frequencies of the heavy tokens as the oracle's renormalised distribution says."""
    rng = np.random.default_rng(V)
    n = 1500
    lg = (rng.standard_normal(V) * 2.0).astype(np.float32)
    lg[rng.choice(V, 40, replace=False)] = (8.0 + 1.5 * rng.random(40)).astype(np.float32)
    lg[1000:3000] = -3.25
    dist = ref.top_p_distribution(lg[None], top_p, temp)[0]
    assert 5 < (dist > 0).sum() < V
    logits = torch.from_numpy(lg).cuda().repeat(n, 1)
    probs = torch.zeros(n, device="cuda")
    tok = ops.sample_top_p(logits, temp, top_p, seed=5, offset=9, probs_out=probs).cpu().numpy()
    # the nucleus ends among thousands of tokens of ~1e-5 each: WHICH token is the last one kept depends on the summation
    # order of ~1e4 float32 terms (numpy's sequential cumsum vs the kernel's tree), so membership is checked against the
    # float64 cumulative mass with a 1e-4 band at the boundary, the frequencies against the oracle's table
    p64 = np.exp((lg.astype(np.float64) - lg.max()) / temp)
    p64 /= p64.sum()
    order = np.argsort(-p64, kind="stable")
    cum = np.empty(V)
    cum[order] = np.cumsum(p64[order])
    assert cum[tok].max() <= top_p + 1e-4, "sampled a token outside the nucleus"
    freq = np.bincount(tok, minlength=V) / n
    big = dist > 0.008
    assert big.sum() >= 3 and np.abs(freq[big] - dist[big]).max() < 4 * np.sqrt(dist[big].max() / n) + 5e-3
    sm = ref.softmax(lg[None])[0]
    assert np.allclose(probs.cpu().numpy(), sm[tok], rtol=2e-3)        # probs = softmax(logits)[token] (utils.py:363)
    # top_p = 1: plain categorical over the whole vocabulary
    tok1 = ops.sample_top_p(logits, temp, 1.0, seed=5, offset=9).cpu().numpy()
    d1 = ref.top_p_distribution(lg[None], 1.0, temp)[0]
    big1 = d1 > 0.008
    f1 = np.bincount(tok1, minlength=V) / n
    assert np.abs(f1[big1] - d1[big1]).max() < 4 * np.sqrt(d1[big1].max() / n) + 5e-3


@pytest.mark.parametrize("B", [1, 30, 70, 200])
def test_samplers_at_every_cluster_size(ops, B):
    """Rows are split over thread-block clusters of 8 / 4 / 2 / 1 CTAs depending on the batch (sampler.cu cluster_for): same
    argmax (ties -> lowest index, also across segment borders), same softmax prob, draws inside the nucleus at each size."""
    rng = np.random.default_rng(B)
    V = 40003                                            # unaligned rows: scalar loads, ragged last segment
    lg = (rng.standard_normal((B, V)) * 2.0).astype(np.float32)
    lg[:, 77] = lg[:, 39000] = 11.0                      # tie between the first and the last segment
    if B > 1:
        lg[1, 39000] = 12.0
    t = torch.from_numpy(lg).cuda()
    probs = torch.zeros(B, device="cuda")
    tok = ops.argmax(t, probs_out=probs).cpu().numpy()
    assert tok.tolist() == lg.argmax(-1).tolist() and tok[0] == 77
    sm = ref.softmax(lg)
    assert np.allclose(probs.cpu().numpy(), sm[np.arange(B), tok], rtol=1e-4)
    lg[:, rng.choice(V, 30, replace=False)] = (7.0 + 2.0 * rng.random(30)).astype(np.float32)
    t = torch.from_numpy(lg).cuda()
    for trial in range(3):
        tk = ops.sample_top_p(t, 0.8, 0.9, seed=11, offset=trial, probs_out=probs).cpu().numpy()
        p64 = np.exp((lg.astype(np.float64) - lg.max(-1, keepdims=True)) / 0.8)
        p64 /= p64.sum(-1, keepdims=True)
        for b in range(B):
            order = np.argsort(-p64[b], kind="stable")
            cum = np.cumsum(p64[b, order])
            rank = int(np.nonzero(order == tk[b])[0][0])
            assert cum[rank] <= 0.9 + 1e-4, (b, tk[b])
        assert np.allclose(probs.cpu().numpy(), ref.softmax(lg)[np.arange(B), tk], rtol=2e-3)


def test_top_p_exact_boundary_and_ties(ops):
    """cum <= top_p keeps exactly the prefix the reference keeps (sample_utils.py:25-31): p = .4 .3 .2 .1 with top_p .75 ->
    {0, 1}; top_p .95 -> {0, 1, 2}.  A nucleus that ends inside a run of EQUAL probabilities: the reference keeps as many of the run as fit, in
    whatever order its argsort leaves ties; this kernel selects by value and drops the run (documented in sampler.cu)."""
    p = np.array([0.4, 0.3, 0.2, 0.1], np.float32)
    lg = torch.from_numpy(np.tile(np.log(p), (4096, 1))).cuda()
    t = ops.sample_top_p(lg, 1.0, 0.75, 3, 0).cpu().numpy()
    assert set(t.tolist()) == {0, 1} and abs((t == 0).mean() - 4 / 7) < 0.04
    t = ops.sample_top_p(lg, 1.0, 0.95, 3, 1).cpu().numpy()
    assert set(t.tolist()) == {0, 1, 2}
    q = np.array([0.4, 0.2, 0.2, 0.2], np.float32)          # cum: .4 .6 .8 1.0, top_p .7 cuts inside the run of .2s
    lq = torch.from_numpy(np.tile(np.log(q), (1024, 1))).cuda()
    t = ops.sample_top_p(lq, 1.0, 0.7, 3, 2).cpu().numpy()
    assert set(t.tolist()) <= {0, 1, 2, 3} and (t == 0).mean() > 0.6


def test_top_p_empty_nucleus_returns_argmax(ops):
    lg = np.log(np.array([[0.6, 0.3, 0.1]], np.float32))
    tok = ops.sample_top_p(torch.from_numpy(np.tile(lg, (64, 1))).cuda(), 1.0, 0.5, 1, 0)
    assert (tok.cpu().numpy() == 0).all()


# ---------------------------------------------------------------- tcgen05 tile path of b200p_qmm
TC_CASES = [  # M, N, K, bits, dtype, epilogue
    (8, 256, 256, 4, "float16", 1), (16, 512, 1024, 4, "float16", 0), (64, 1024, 512, 4, "float16", 2),
    (64, 2048, 1024, 4, "float16", 3), (5, 1000, 192, 4, "float16", 1), (100, 1000, 448, 4, "bfloat16", 1),
    (300, 512, 512, 4, "float16", 0), (64, 512, 2048, 8, "float16", 1), (33, 768, 640, 4, "bfloat16", 3),
    (64, 256, 4096, 4, "float16", 2),          # deep K with few row blocks -> split-K + last-arriver fix-up
    # 8-bit bf16: the code goes through fp32 (128 + q is exact in bf16 only below 128), one rounding to bf16
    (64, 512, 2048, 8, "bfloat16", 1), (8, 1024, 1024, 8, "bfloat16", 2), (40, 768, 512, 8, "bfloat16", 3), (128, 512, 1024, 8, "bfloat16", 0),
]


@pytest.mark.parametrize("M,N,K,bits,dtype,epi", TC_CASES)
def test_qmm_tensor_path_matches_oracle(ops, M, N, K, bits, dtype, epi):
    got, exp = qmm_case(ops, M, N, K, bits, dtype, epi, seed=M + N, path=2)
    # A is the storage-rounded dequantised weight (round_T(q*s+b)), accumulation fp32 in TMEM
    tol = {"float16": 3e-3, "bfloat16": 2e-2}[dtype]
    assert rel_err(got, exp) < tol


def test_qmm_tensor_path_is_bit_reproducible_and_matches_gemv(ops):
    # whole-tile kernel (STORE / STORE_F32 / SILU_MUL): K splits are reduced from per-CTA partial tiles in CTA order (no
    # atomics): two runs agree bit for bit.  The fp32 accumulate epilogue runs on the stream-K kernel, whose partial tiles
    # are summed by the L2 atomic units in arrival order: equal up to fp32 summation order only.
    for epi in (1, 3, 0):
        a1, _ = qmm_case(ops, 64, 512, 4096, 4, "float16", epi, seed=3, path=2)
        a2, _ = qmm_case(ops, 64, 512, 4096, 4, "float16", epi, seed=3, path=2)
        assert np.array_equal(a1, a2), epi
    a1, _ = qmm_case(ops, 64, 512, 4096, 4, "float16", 2, seed=3, path=2)
    a2, _ = qmm_case(ops, 64, 512, 4096, 4, "float16", 2, seed=3, path=2)
    assert rel_err(a1, a2) < 1e-6
    g, _ = qmm_case(ops, 64, 512, 4096, 4, "float16", 1, seed=3, path=1)
    a1, _ = qmm_case(ops, 64, 512, 4096, 4, "float16", 1, seed=3, path=2)
    assert rel_err(a1, g) < 1e-3


SPLIT_CASES = [  # every CTA holds a head AND a tail partial tile, tiles shared by 2..8 CTAs, ragged token / row edges
    (64, 4096, 4096, 4, "float16", 2), (64, 6144, 4096, 4, "float16", 0), (64, 28672 // 4, 4096, 4, "float16", 3),
    (64, 4096, 14336 // 2, 4, "float16", 2), (37, 1000, 2048, 4, "bfloat16", 1), (128, 1024, 4096, 4, "float16", 3),
    (130, 520, 1536, 4, "float16", 0), (8, 4096, 4096, 8, "float16", 2), (1, 768, 8192, 4, "float16", 1),
]


@pytest.mark.parametrize("M,N,K,bits,dtype,epi", SPLIT_CASES)
def test_qmm_tensor_path_split_tiles(ops, M, N, K, bits, dtype, epi):
    """Layer-sized shapes where stream-K splits every tile: partial tiles through the workspace, shared final reduction,
    counters left re-armed (the second call reuses the same workspace inside qmm_case's fresh allocation, the third
    test below reuses one workspace across shapes)."""
    got, exp = qmm_case(ops, M, N, K, bits, dtype, epi, seed=M + N + K, path=2)
    tol = {"float16": 3e-3, "bfloat16": 2e-2}[dtype]
    assert rel_err(got, exp) < tol


def test_qmm_tensor_path_workspace_is_left_rearmed(ops):
    """One workspace, many launches of different shapes back to back (what a decode step does): the per-tile counters
    must be back at zero after every launch, stale partial tiles must never be read."""
    from mlx_parallm_b200 import _lib
    rng = np.random.default_rng(5)
    shapes = [(64, 4096, 4096, 2), (64, 6144, 4096, 0), (64, 2048, 1024, 3), (16, 512, 8192, 1), (64, 4096, 4096, 2)]
    ws = torch.zeros((max(ops.qmm_workspace_bytes(64, n, k) for _, n, k, _ in shapes),), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.lib().b200p_qmm_set_path(2))
    try:
        for rep in range(3):
            for M, N, K, epi in shapes:
                wq = rng.integers(0, 2 ** 32, (N, K // 8), dtype=np.uint32)
                s = ref.round_to(rng.uniform(0.5, 1.5, (N, K // 64)) * (2 / 15) / np.sqrt(K), "float16")
                b = ref.round_to(-s * 7.5, "float16")
                x = ref.round_to(rng.standard_normal((M, K)), "float16")
                acc = ref.quantized_matmul(x, wq, s, b, 64, 4).astype(np.float64)
                if epi == 2:
                    out = torch.zeros((M, N), dtype=torch.float32, device="cuda")
                    ops.qmm(t_(x, "float16"), w_(wq), t_(s, "float16"), t_(b, "float16"), 64, 4, epi, out=out, workspace=ws)
                    exp = acc
                else:
                    out = ops.qmm(t_(x, "float16"), w_(wq), t_(s, "float16"), t_(b, "float16"), 64, 4, epi, workspace=ws)
                    exp = acc if epi != 3 else acc[:, :N // 2] / (1 + np.exp(-acc[:, :N // 2])) * acc[:, N // 2:]
                assert rel_err(out.float().cpu().numpy(), exp) < 3e-3, (rep, M, N, K, epi)
        torch.cuda.synchronize()
        ncnt = 2 * ((4096 + 255) // 256 + 1)
        assert int(ws[:ncnt * 4].view(torch.int32).abs().sum()) == 0
    finally:
        _lib.lib().b200p_qmm_set_path(0)


@pytest.mark.parametrize("M,N,K,bits,epi", [(64, 2048, 1024, 4, 3), (64, 4096, 4096, 4, 2), (8, 256, 256, 4, 1), (16, 512, 1024, 4, 0),
                                            (64, 512, 2048, 8, 1), (5, 1000, 192, 4, 1), (200, 512, 512, 4, 0)])
def test_qmm_small_scale_dequant_is_bit_identical(ops, M, N, K, bits, epi):
    """B200P_W_SMALLSCALE (one half2 FMA per code pair on subnormal operands, accumulator rescaled by 16) rounds q*s+b at
    the same point as the 3-op dequant: identical outputs wherever the operand / 16 stays a normal half."""
    a, exp = qmm_case(ops, M, N, K, bits, "float16", epi, seed=11, path=2, small_scale=False)
    f, _ = qmm_case(ops, M, N, K, bits, "float16", epi, seed=11, path=2, small_scale=True)
    assert rel_err(f, exp) < 3e-3
    if bits == 4 and K <= 1024:
        assert np.array_equal(a, f)          # every |q*s+b| / 16 is a normal half here
    else:
        assert rel_err(a, f) < 2e-5          # operands below 2^-10 round as subnormals at 1/16: absolute error <= 2^-21


@pytest.mark.parametrize("M,N,K,bits,epi,path", [(1, 1024, 1024, 4, 3, 6), (2, 512, 2048, 8, 2, 6), (5, 1000, 192, 4, 1, 2), (64, 2048, 1024, 4, 3, 2),
                                                 (64, 4096, 1024, 4, 2, 2), (24, 512, 2048, 8, 1, 2), (60, 512, 320, 8, 2, 0), (200, 512, 512, 4, 0, 0),
                                                 (300, 264, 1536, 4, 2, 0), (201, 1000, 1024, 8, 3, 0)])
def test_qmm_small_scale_dequant_of_bf16(ops, M, N, K, bits, epi, path):
    """bf16: codes as integers times 2^-133, scales times 2^120, operands at 2^-13: every step but the one rounding of q*s+b is exact, so
    4-bit products equal the direct form's where the order of the sums is fixed (whole tiles, or one CTA per K range); 8-bit operands,
    which go through fp32 and a rounded constant otherwise, are no farther from the 64-bit result."""
    a, exp = qmm_case(ops, M, N, K, bits, "bfloat16", epi, seed=M, path=path, small_scale=False)
    f, _ = qmm_case(ops, M, N, K, bits, "bfloat16", epi, seed=M, path=path, small_scale=True)
    if bits == 4 and epi != 2:
        assert np.array_equal(a, f)
    elif bits == 4:
        assert rel_err(f, a) < 1e-6                              # fp32 sums in another order
    assert rel_err(f, exp) < rel_err(a, exp) * 1.05 + 1e-6


@pytest.mark.parametrize("M,N,K,bits,epi", [(2, 8192, 1024, 4, 3), (201, 512, 512, 4, 0), (300, 512, 1024, 8, 1)])
def test_qmm_arguments_of_the_tile_kernel_stay_required(ops, M, N, K, bits, epi):
    """The ring and wide kernels use no workspace, but a call without one, or with 16-bit rows of odd length, is refused as on any size."""
    from mlx_parallm_b200 import _lib
    wq, s = torch.zeros((N, K * bits // 32), dtype=torch.int32, device="cuda"), torch.zeros((N, K // 64), dtype=torch.float16, device="cuda")
    x, ws = torch.zeros((M, K), dtype=torch.float16, device="cuda"), torch.zeros(ops.qmm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    n = N // 2 if epi == 3 else N
    out = torch.empty((M, n + 1), dtype=torch.float32 if epi == 1 else torch.float16, device="cuda")

    def call(ld, work, nbytes):
        return _lib.lib().b200p_qmm(x.data_ptr(), wq.data_ptr(), s.data_ptr(), s.data_ptr(), out.data_ptr(), M, N, K, K, ld, 64, bits, _lib.F16, epi,
                                    work, nbytes, torch.cuda.current_stream().cuda_stream)
    assert call(n, ws.data_ptr(), ws.numel()) == 0
    assert call(n, None, 0) < 0 and call(n, ws.data_ptr(), ws.numel() - 1) < 0
    assert (call(n + 1, ws.data_ptr(), ws.numel()) == 0) == (epi == 1)
    torch.cuda.synchronize()


# ---------------------------------------------------------------- wide tiles of b200p_qmm (M > 128)
@pytest.mark.parametrize("M,N,K,bits,dtype,epi,small", [
    (129, 128, 512, 4, "float16", 1, True),       # one tile, the shortest K: two stages
    (201, 1000, 1024, 4, "bfloat16", 0, False),   # rows past N in the last block, tokens past M in the tile
    (256, 208, 1536, 4, "float16", 3, False),     # gated: a block whose last gate rows do not exist, a full token tile
    (257, 2000, 512, 4, "bfloat16", 3, False),    # two token tiles, one row of the second in use by one token less than half
    (300, 264, 4096, 4, "float16", 2, True),      # accumulate: K ranges of one tile on several CTAs
    (1100, 5120, 512, 4, "float16", 2, False),    # accumulate: a whole round of tiles, the rest cut along K
    (140, 512, 2048, 8, "float16", 1, True),      # 8 bits: two k-blocks per stage
    (333, 384, 1024, 8, "bfloat16", 3, False),
    (205, 260 * 4, 512, 8, "bfloat16", 2, False),
    (201, 264, 8192, 8, "bfloat16", 2, True),     # accumulate: token tiles of 208, beside which an odd number of weight stages would fit
    (256, 512, 8192, 8, "float16", 0, False),     # the same of 256
])
def test_qmm_wide_tiles(ops, M, N, K, bits, dtype, epi, small):
    """csrc/qmm_wide.cu against the oracle.  Tolerances as for the other 16-bit paths (A rounded to the storage type, fp32 sums)."""
    from mlx_parallm_b200 import _lib
    got, exp = qmm_case(ops, M, N, K, bits, dtype, epi, seed=M + N, path=2, ragged_ld=(M in (201, 300)), small_scale=small)
    assert _lib.lib().b200p_qmm_wide_fault() == 0
    assert rel_err(got, exp) < {"float16": 3e-3, "bfloat16": 2e-2}[dtype]


# 148 SMs: gated rows, 151 blocks of 64; 149 row blocks for two token tiles each; 2 x 148 blocks and one that is partly filled
@pytest.mark.parametrize("M,N,K,bits,epi", [(130, 19328, 8192, 8, 3), (300, 19072, 8192, 8, 0), (145, 38008, 8192, 8, 1)])
def test_qmm_wide_tiles_leave_a_short_last_round(ops, M, N, K, bits, epi):
    """Row blocks beyond whole rounds of tiles go to the kernel that splits K: every column against a float64 product (1.5e-2: one bf16 rounding of weights,
    activations and outputs each), twice with one workspace, whose counters are left as they were found and whose partial sums show that the split kernel
    had its share."""
    g = torch.Generator(device="cuda").manual_seed(N)
    w = torch.randint(-2 ** 31, 2 ** 31, (N, K // 4), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    s = ((torch.rand((N, K // 64), generator=g, device="cuda") + 0.5) * 2 / 255 / K ** 0.5).bfloat16()
    b = (-s.float() * 255 / 2).bfloat16()
    x = torch.randn((M, K), generator=g, device="cuda").bfloat16()
    ws = torch.zeros(ops.qmm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        got = ops.qmm(x, w, s, b, 64, bits, epi, workspace=ws, small_scale=True).double()
        full = torch.empty(M, N, dtype=torch.float64, device="cuda")
        for i in range(0, N, 4096):
            codes = ((w[i:i + 4096].unsqueeze(-1) >> torch.arange(0, 32, 8, device="cuda", dtype=torch.int32)) & 255).reshape(-1, K // 64, 64).double()
            full[:, i:i + 4096] = x.double() @ (codes * s[i:i + 4096].double().unsqueeze(-1) + b[i:i + 4096].double().unsqueeze(-1)).reshape(-1, K).t()
        want = torch.nn.functional.silu(full[:, :N // 2]) * full[:, N // 2:] if epi == 3 else full
        err = (got - want).norm(dim=0) / want.norm(dim=0)
        assert float(err.max()) < 1.5e-2 and not bool(ws[:4096].any()) and bool(ws[4096:].any())


def test_qmm_wide_tiles_at_4_bits_keep_their_last_round(ops):
    """Rounds of 4-bit tiles are too short for a second launch: 744 row blocks, five rounds of 148 and four blocks, in one launch that leaves the workspace alone."""
    M, N, K = 256, 744 * 128, 8192
    g = torch.Generator(device="cuda").manual_seed(N)
    w = torch.randint(-2 ** 31, 2 ** 31, (N, K // 8), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    s = ((torch.rand((N, K // 64), generator=g, device="cuda") + 0.5) * 2 / 15 / K ** 0.5).bfloat16()
    x, ws = torch.randn((M, K), generator=g, device="cuda").bfloat16(), torch.zeros(ops.qmm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    got = ops.qmm(x, w, s, (-s.float() * 15 / 2).bfloat16(), 64, 4, 0, workspace=ws, small_scale=True)
    assert bool(got.isfinite().all()) and not bool(ws.any())


@pytest.mark.parametrize("M,N,K,bits,dtype", [(201, 2048, 4096, 8, "bfloat16"), (250, 18944, 1024, 8, "bfloat16"), (300, 4096, 2048, 4, "float16")])
def test_qmm_wide_tiles_repeat_bit_for_bit(ops, M, N, K, bits, dtype):
    """Whole tiles are summed in a fixed order: hundreds of launches over the same operands agree in every bit.  (A k-block of one row that is
    lost on its way to the tensor core shows as a column that differs.)"""
    g = torch.Generator(device="cuda")
    g.manual_seed(M)
    dt = TD[dtype]
    w = torch.randint(-2 ** 31, 2 ** 31, (N, K * bits // 32), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    s = ((torch.rand((N, K // 64), generator=g, device="cuda") + 0.5) * 2 / (2 ** bits - 1) / K ** 0.5).to(dt)
    b = (-s.float() * (2 ** bits - 1) / 2).to(dt)
    x, ws = torch.randn((M, K), generator=g, device="cuda").to(dt), torch.zeros(ops.qmm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    first = ops.qmm(x, w, s, b, 64, bits, 1, workspace=ws, small_scale=True)
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(300):
        bad += (ops.qmm(x, w, s, b, 64, bits, 1, workspace=ws, small_scale=True) != first).sum()
    assert int(bad) == 0


@pytest.mark.parametrize("M,N,K,dtype,epi,small", [
    (8, 4096, 576, "bfloat16", 0, True),          # nine k-blocks: a stage with one, scales that the copy engine cannot fetch, whole row blocks
    (32, 4112, 2368, "float16", 3, False),        # three slots of the ring; rows past N / 2 in the last block
    (33, 8200, 1024, "bfloat16", 1, True),        # two slots
    (64, 40960, 512, "float16", 0, True),         # more tiles than SMs: two accumulators, one unit on each side of the border
    (96, 4096, 512, "bfloat16", 2, True),         # the largest token tile of two k-blocks ...
    (97, 4096, 512, "bfloat16", 2, True),         # ... and the smallest of one
    (20, 2056, 1216, "float16", 2, False),        # ranges of K that end inside a tile
])
def test_qmm_units_of_two_k_blocks(ops, M, N, K, dtype, epi, small):
    """The tile kernels hand over two k-blocks at a time at 4 bits up to 96 tokens: against the oracle, tolerances as for the other 16-bit paths."""
    got, exp = qmm_case(ops, M, N, K, 4, dtype, epi, seed=M + N, path=2, small_scale=small)
    assert rel_err(got, exp) < {"float16": 3e-3, "bfloat16": 2e-2}[dtype]


def test_qmm_forced_tiles():
    """B200P_TC_R and B200P_TC_S force rows per block and K splits, also on 4-bit matrices that take whole blocks by themselves: two splits meet in the workspace."""
    import os
    import subprocess
    import sys
    code = ("import torch\nfrom mlx_parallm_b200 import ops, _lib\n_lib.lib().b200p_qmm_set_path(2)\n"
            "w = torch.randint(-2**31, 2**31 - 1, (4096, 512), device='cuda', dtype=torch.int32)\n"
            "s, x = torch.full((4096, 64), 0.001, device='cuda').half(), torch.randn(24, 4096, device='cuda').half()\n"
            "ws = torch.zeros(ops.qmm_workspace_bytes(24, 4096, 4096), dtype=torch.uint8, device='cuda')\n"
            "y = ops.qmm(x, w, s, -s, 64, 4, 0, workspace=ws)\nprint(bool(y.isfinite().all()), bool(ws[4096:].any()))\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    for splits, used in (("1", "False"), ("2", "True")):
        env = dict(os.environ, PYTHONPATH=root, B200P_TC_R="64", B200P_TC_S=splits)
        out = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
        assert out.stdout.split() == ["True", used], out.stdout + out.stderr


@pytest.mark.parametrize("M,N,K,bits,dtype", [(250, 18944, 1024, 8, "bfloat16"), (64, 8192, 4096, 4, "float16"), (40, 4096, 8192, 8, "bfloat16"), (1, 8192, 8192, 4, "bfloat16")])
def test_qmm_between_memory_bound_kernels(ops, M, N, K, bits, dtype):
    """A product that starts while an elementwise kernel still fills the SM's memory pipeline: the weights' slots must not be refilled
    while reads from them wait their turn (before, about one launch in 500 of the first case had a column that differed)."""
    g = torch.Generator(device="cuda").manual_seed(M)
    dt = TD[dtype]
    w = torch.randint(-2 ** 31, 2 ** 31, (N, K * bits // 32), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    s = ((torch.rand((N, K // 64), generator=g, device="cuda") + 0.5) * 2 / (2 ** bits - 1) / K ** 0.5).to(dt)
    b = (-s.float() * (2 ** bits - 1) / 2).to(dt)
    x, ws = torch.randn((M, K), generator=g, device="cuda").to(dt), torch.zeros(ops.qmm_workspace_bytes(M, N, K), dtype=torch.uint8, device="cuda")
    first, bad = ops.qmm(x, w, s, b, 64, bits, 1, workspace=ws, small_scale=True), torch.zeros((), dtype=torch.int64, device="cuda")
    other = torch.zeros(1 << 21, device="cuda")
    for _ in range(2000):
        other.add_(1.0)
        bad += (ops.qmm(x, w, s, b, 64, bits, 1, workspace=ws, small_scale=True) != first).sum()
    assert int(bad) == 0


# ---------------------------------------------------------------- TMA-ring GEMV of b200p_qmm (M <= 16)
@pytest.mark.parametrize("M,N,K,bits,dtype,epi,small", [
    (1, 16, 512, 4, "float16", 1, True),          # one unit: seven of eight warps have nothing to do
    (2, 48, 1024, 4, "bfloat16", 3, False),       # two units per tile: runs end inside a tile, idle warps in between
    (3, 2400, 1536, 4, "float16", 0, False),      # three chunks per tile against eight warps, 16-bit store
    (4, 4096, 4096, 4, "float16", 2, True),       # accumulate: tiles shared by two CTAs
    (5, 96, 17408, 4, "bfloat16", 2, False),      # accumulate: several panels of k, few tiles
    (8, 1024, 5120, 4, "float16", 3, True),       # 16-warp CTAs
    (9, 256, 2048, 4, "bfloat16", 1, False),      # second n-tile, one token in it
    (16, 512, 2048, 4, "float16", 2, False),
    (1, 512, 2048, 8, "float16", 3, True),
    (7, 80, 1024, 8, "bfloat16", 0, False),
    (13, 64, 4096, 8, "float16", 2, False),
])
def test_qmm_ring_gemv(ops, M, N, K, bits, dtype, epi, small):
    """csrc/qmv_ring.cu against the oracle at the edges of its schedule.  Tolerances as for the other 16-bit paths: A is q*s+b rounded to
    the storage type, sums are fp32, 16-bit epilogues round once more."""
    from mlx_parallm_b200 import _lib
    got, exp = qmm_case(ops, M, N, K, bits, dtype, epi, seed=M + N, path=6, ragged_ld=(M in (3, 9)), small_scale=small)
    assert _lib.lib().b200p_qmv_fault() == 0
    assert rel_err(got, exp) < {"float16": 3e-3, "bfloat16": 2e-2}[dtype]


# ---------------------------------------------------------------- mma.sync register GEMV of b200p_qmm (M <= 16)
MMA_CASES = [  # M, N, K, dtype, epilogue (1 = fp32 store, 2 = += into fp32, split-K with red.add)
    (1, 256, 256, "float16", 1), (3, 512, 1024, "float16", 2), (8, 96, 512, "bfloat16", 1), (9, 1024, 4096, "float16", 2),
    (16, 2048, 256, "bfloat16", 2), (5, 64, 768, "float16", 1), (2, 4096, 4096, "float16", 2), (13, 160, 1280, "float16", 1),
]


@pytest.mark.parametrize("M,N,K,dtype,epi", MMA_CASES)
def test_qmm_mma_gemv_matches_oracle(ops, M, N, K, dtype, epi):
    got, exp = qmm_case(ops, M, N, K, 4, dtype, epi, seed=M + N + K, path=3, ragged_ld=(M == 5))
    tol = {"float16": 3e-3, "bfloat16": 2e-2}[dtype]     # A = storage-rounded q*s+b, fp32 accumulation in the MMA
    assert rel_err(got, exp) < tol


def test_qmm_mma_gemv_agrees_with_the_other_paths_and_is_the_auto_choice(ops):
    from mlx_parallm_b200 import _lib
    m, _ = qmm_case(ops, 4, 512, 2048, 4, "float16", 1, seed=9, path=3)
    t, _ = qmm_case(ops, 4, 512, 2048, 4, "float16", 1, seed=9, path=2) if \
        _lib.lib().b200p_qmm_tensor_supported(4, 512, 2048, 64, 4, 1, 1) else (m, None)
    g, _ = qmm_case(ops, 4, 512, 2048, 4, "float16", 1, seed=9, path=1)
    a, _ = qmm_case(ops, 4, 512, 2048, 4, "float16", 1, seed=9, path=0)
    assert rel_err(m, t) < 1e-5 and rel_err(m, g) < 1e-3
    assert np.array_equal(a, m)                          # small matrix, M <= 4: auto == the mma.sync GEMV, bit for bit
    assert _lib.lib().b200p_qmm_set_path(5) == -1


@pytest.mark.parametrize("dtype,M", [("float16", 1), ("bfloat16", 3), ("float16", 8), ("float16", 13)])
def test_qmv_mma_silu_mul_pairs_gate_and_up_rows(ops, dtype, M):
    """SILU_MUL through the mma.sync GEMV (forced path 3): a warp takes 8 gate rows and the 8 matching up rows."""
    from mlx_parallm_b200 import _lib
    got, exp = qmm_case(ops, M, 256, 512, 4, dtype, _lib.EPI_SILU_MUL, seed=40 + M, path=3)
    assert got.shape == (M, 128)
    assert rel_err(got, exp) < {"float16": 2e-3, "bfloat16": 1e-2}[dtype]
    tile, _ = qmm_case(ops, M, 256, 512, 4, dtype, _lib.EPI_SILU_MUL, seed=40 + M, path=2)
    assert rel_err(got, tile) < {"float16": 1.1e-3, "bfloat16": 8.1e-3}[dtype]      # one rounding of the same fp32 value


# ---------------------------------------------------------------- mma.sync small-matrix GEMM (csrc/qmm_mma.cu)
@pytest.mark.parametrize("dtype,M,N,K", [
    ("float16", 5, 128, 512),        # NT = 1, two steps, no K split
    ("float16", 8, 256, 1024),
    ("bfloat16", 16, 128, 2048),     # NT = 2
    ("float16", 23, 384, 1024),      # NT = 4 with zero-filled token lines
    ("float16", 64, 256, 2048),      # NT = 8, K split
    ("bfloat16", 64, 128, 256),      # a single step
    ("float16", 33, 1024, 4096),     # many row blocks x splits: partial sums meet through the bulk reduce-add
])
def test_qmm_mma_small_matrix_gemm_matches_oracle(ops, dtype, M, N, K):
    from mlx_parallm_b200 import _lib
    got, exp = qmm_case(ops, M, N, K, 4, dtype, _lib.EPI_ADD_RESIDUAL, seed=M + N, path=4, ragged_ld=(M == 23))
    assert rel_err(got, exp) < {"float16": 1e-3, "bfloat16": 6e-3}[dtype]     # bound: rounding of the dequantised weights
    auto, _ = qmm_case(ops, M, N, K, 4, dtype, _lib.EPI_ADD_RESIDUAL, seed=M + N, path=0)
    assert rel_err(auto, got) < 1e-5                     # auto (this kernel up to 16 rows, stream-K tiles above): same dequantised
                                                         # weights, fp32 sums in another order


def test_qmm_mma_perm8_activations_and_unsupported_shapes(ops):
    from mlx_parallm_b200 import _lib
    from test_gpu_layouts import to_perm8
    rng = np.random.default_rng(77)
    M, N, K = 64, 256, 1024
    wq = rng.integers(0, 2 ** 32, (N, K // 8), dtype=np.uint32)
    s = ref.round_to(rng.uniform(0.5, 1.5, (N, K // 64)) * (2 / 15) / np.sqrt(K), "float16")
    b = ref.round_to(-s * 7.5, "float16")
    x = ref.round_to(rng.standard_normal((M, K)), "float16")
    _lib.check(_lib.lib().b200p_qmm_set_path(4))
    try:
        nat = torch.zeros((M, N), dtype=torch.float32, device="cuda")
        per = torch.zeros((M, N), dtype=torch.float32, device="cuda")
        ops.qmm(t_(x, "float16"), w_(wq), t_(s, "float16"), t_(b, "float16"), 64, 4, _lib.EPI_ADD_RESIDUAL, out=nat)
        ops.qmm(t_(to_perm8(x), "float16"), w_(wq), t_(s, "float16"), t_(b, "float16"), 64, 4, _lib.EPI_ADD_RESIDUAL, out=per,
                x_perm=True)
        assert rel_err(per.cpu().numpy(), nat.cpu().numpy()) < 1e-6
        assert rel_err(nat.cpu().numpy(), ref.quantized_matmul(x, wq, s, b, 64, 4)) < 1e-3
        with pytest.raises(_lib.B200PError):                  # N not a multiple of 128: forced path refuses, nothing is launched
            ops.qmm(t_(x, "float16"), w_(wq[:96]), t_(s[:96], "float16"), t_(b[:96], "float16"), 64, 4, _lib.EPI_ADD_RESIDUAL,
                    out=nat[:, :96].contiguous())
        with pytest.raises(_lib.B200PError):                  # STORE epilogue: not this kernel's
            ops.qmm(t_(x, "float16"), w_(wq), t_(s, "float16"), t_(b, "float16"), 64, 4, _lib.EPI_STORE_F32)
    finally:
        _lib.lib().b200p_qmm_set_path(0)


# ---------------------------------------------------------------- split-K tensor decode attention
@pytest.mark.parametrize("dtype,Hq,Hkv,lengths", [
    ("float16", 8, 2, [0, 5, 130]),             # ragged rows incl. an empty cache (only the new token)
    ("bfloat16", 5, 1, [15, 16, 17]),           # G = 5 (Qwen3-14B at TP=8), tile-boundary lengths
    ("float16", 32, 8, [700, 3]),               # Llama-3-8B head layout
    ("float16", 8, 1, [5000, 4999, 1, 2500]),   # G = 8 (70B), long rows -> sequence split across CTAs
])
def test_attention_tensor_decode(ops, dtype, Hq, Hkv, lengths):
    got, exp = attn_case(ops, len(lengths), 1, Hq, Hkv, 128, lengths, dtype, path=2)
    assert rel_err(got, exp) < {"float16": 2e-3, "bfloat16": 1.2e-2}[dtype]


@pytest.mark.parametrize("dtype,Hq,Hkv,lengths", [
    ("float16", 16, 1, [763]),                  # 767 keys of capacity: whole; 768 and 769: in 64s
    ("bfloat16", 16, 1, [764]),
    ("float16", 32, 8, [765]),
    ("float16", 32, 16, [508, 70]),             # 512 keys, two splits become four (32 (row, key head) pairs on 7/8 of 148 SMs)
    ("float16", 16, 16, [508]),                 # ... eight: 64 keys each
    ("bfloat16", 8, 8, [2040]),                 # as many splits as 7/8 of the SMs hold
    ("float16", 4, 1, [2047, 0, 63, 64, 1000]), # 25 splits: most of them empty in the short rows
    ("bfloat16", 4, 4, [700] * 32),             # as many (row, key head) pairs as SMs to spread over: not spread further
])
def test_attention_tensor_decode_spread_over_idle_sms(ops, dtype, Hq, Hkv, lengths):
    """Few key heads in all: more splits of fewer keys, rows that end before most of the splits begin."""
    got, exp = attn_case(ops, len(lengths), 1, Hq, Hkv, 128, lengths, dtype, path=2)
    assert rel_err(got, exp) < {"float16": 2e-3, "bfloat16": 1.2e-2}[dtype]


def test_attention_tensor_matches_generic(ops):
    a, _ = attn_case(ops, 2, 1, 8, 2, 128, [1000, 37], "float16", path=2, seed=9)
    g, _ = attn_case(ops, 2, 1, 8, 2, 128, [1000, 37], "float16", path=1, seed=9)
    assert rel_err(a, g) < 2e-3


# ---------------------------------------------------------------- bounded waits that give up
def test_waits_that_give_up_are_reported(ops):
    """A wait of a millisecond for an arrival that nothing makes: the host sees it without synchronising on anything but the launch, every
    launch of a kernel with bounded waits is refused until the report has been taken, and then runs again."""
    from mlx_parallm_b200 import _lib
    L = _lib.lib()
    q, k, v = prefill_inputs("float16", 1, 300, 4, 2, 300, seed=1)
    before = prefill(ops, q, k, v, [0], 0.1)
    x, w = torch.ones((200, 64), dtype=torch.float16, device="cuda"), torch.ones((64, 64), dtype=torch.float16, device="cuda")
    wq, s = torch.zeros((256, 64), dtype=torch.int32, device="cuda"), torch.ones((256, 8), dtype=torch.float16, device="cuda")
    xq, ws = torch.ones((200, 512), dtype=torch.float16, device="cuda"), torch.zeros(ops.qmm_workspace_bytes(200, 256, 512), dtype=torch.uint8, device="cuda")
    calls = [lambda: prefill(ops, q, k, v, [0], 0.1), lambda: ops.gemm(x, w, 0), lambda: ops.qmm(xq, wq, s, s, workspace=ws)]
    assert L.b200p_wait_fault() == 0
    _lib.check(L.b200p_wait_probe(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert L.b200p_wait_fault() == 256 * 3 + 1
    for call in calls:
        with pytest.raises(_lib.B200PError, match="gave up"):
            call()
    with pytest.raises(_lib.B200PError, match="gave up"):
        ops.check_waits()
    assert L.b200p_attn_tc_fault() == 0 and L.b200p_qmv_fault() == 1 and L.b200p_qmv_fault() == 0
    ops.check_waits()
    assert torch.equal(calls[0](), before)
    for call in calls[1:]:
        call()
