"""Dogulorn on the GPU against the slow float64 oracle (tests/dogulorn_oracle.py): each mechanism alone, prompts against
token-by-token decoding, portions, ragged batches, rows given back and used again, window edges and far keys, other sizes,
greedy generation through generate_step."""
import math

import numpy as np
import pytest
import torch

import dogulorn_oracle as O

pytestmark = pytest.mark.gpu

F32_TOL = 2e-4        # float32 model against the float64 oracle (centred rms over the vocabulary, relative)
BF16_TOL = 6e-2       # bfloat16 matrix products


def build(cfg, seed=0, dtype=torch.float32):
    from mlx_parallm_b200.utils import _get_classes
    Model, Args = _get_classes(cfg)
    w = O.random_weights(cfg, seed)
    return Model(Args.from_dict(cfg)).load_weights(w, device="cuda", dtype=dtype), w


def toks(cfg, n, seed):
    return np.random.default_rng(seed).integers(0, cfg["vocab"], n).tolist()


MLP = {"kind": "dense", "ff": 40, "limit": 1.5}
CONFIGS = {
    # every branch: own latents, shared latents, delta with and without feed-forward, attention without feed-forward, no window
    "mixed": lambda: O.make_config([
        O.attn_layer(3, 8, 16, 24, 32, window=7, scale=0.3, mlp=MLP),
        O.delta_layer(4, 2, 16, 8, conv=4),
        O.attn_layer(2, 16, 8, 16, 32, window=5, kv_from=0),
        O.delta_layer(3, 3, 8, 24, conv=2, mlp={"kind": "dense", "ff": 56, "limit": 0.75}),
        O.attn_layer(5, 8, 8, 8, 16, window=0, mlp=MLP),
    ]),
    # sizes off the fast paths (odd width and ranks), one kv head for three heads, no bigram, no token input, window 1
    "odd": lambda: O.make_config([
        O.delta_layer(3, 1, 5, 7, conv=3),
        O.attn_layer(1, 6, 10, 9, 11, window=1, mlp={"kind": "dense", "ff": 13, "limit": 3.0}),
        O.attn_layer(2, 6, 10, 9, 11, window=3, kv_from=1),
    ], vocab=31, width=27, eps=1e-3, emb_scale=1.0, bigram=None, side_dim=0),
    # wider heads: key size 40 pads to 64 state rows, value size 160 spans two thread blocks, rank 72
    "wide": lambda: O.make_config([
        O.delta_layer(2, 1, 40, 160, conv=1, mlp=MLP),
        O.attn_layer(4, 16, 24, 40, 72, window=33),
    ], vocab=130, width=64, bigram=(7, 3, 1), side_dim=4),
}


@pytest.fixture(scope="module")
def models():
    out = {}
    for name, mk in CONFIGS.items():
        cfg = mk()
        m, w = build(cfg, seed=len(name))
        out[name] = (cfg, m, w)
    return out


# ---- mechanisms alone ---------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", [(1, 10, 16), (3, 7, 5), (8, 64, 48), (9, 130, 72), (70, 33, 40), (200, 96, 128), (300, 64, 24)])
def test_gemm_shapes(dtype, M, N, K):
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator().manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g).to(dtype)
    w = torch.randn(N, K, generator=g).to(dtype)
    want = x.double() @ w.double().T
    got = ops.gemm(x.cuda(), w.cuda(), _lib.GEMM_STORE_F32)
    tol = 1e-5 if dtype == torch.float32 else 1e-5          # same products and fp32 accumulation: only summation order differs
    assert (got.double().cpu() - want).abs().max() <= tol * math.sqrt(K) * 8
    got16 = ops.gemm(x.cuda(), w.cuda(), _lib.GEMM_STORE)
    assert got16.dtype == dtype and (got16.double().cpu() - want).abs().max() <= (1e-4 if dtype == torch.float32 else 0.05) * math.sqrt(K)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M", [2, 40])
def test_gemm_gated_epilogue_and_heads(dtype, M):
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator().manual_seed(5)
    K, F, lim = 32, 24, 0.8
    x = torch.randn(M, K, generator=g).to(dtype)
    gate, up = torch.randn(F, K, generator=g).to(dtype), torch.randn(F, K, generator=g).to(dtype)
    gu = torch.stack([gate, up], 1).reshape(2 * F, K)
    a = torch.clamp(x.double() @ gate.double().T, max=lim)
    u = torch.clamp(x.double() @ up.double().T, -lim, lim)
    want = a * torch.sigmoid(1.702 * a) * (u + 1)
    got = ops.gemm(x.cuda(), gu.cuda().contiguous(), _lib.GEMM_GLU_CLAMP, act=(lim, 0.0))
    assert got.shape == (M, F) and (got.double().cpu() - want).abs().max() < (1e-4 if dtype == torch.float32 else 0.04)
    # one weight block per head, operands strided inside wider rows
    H, dk, R = 3, 8, 16
    q = torch.randn(M, H * dk, generator=g).to(dtype)
    wk = torch.randn(H, R, dk, generator=g).to(dtype)
    out = torch.empty(M, H * R, dtype=torch.float32, device="cuda")
    ops.gemm(q.cuda(), wk.cuda(), _lib.GEMM_STORE_F32, out=out, batch=H, strides=(dk, R * dk, R), M=M, N=R, K=dk, ldx=H * dk, ldw=dk,
             ldy=H * R)
    want = torch.einsum("mhd,hrd->mhr", q.double().view(M, H, dk), wk.double()).reshape(M, H * R)
    assert (out.double().cpu() - want).abs().max() < 1e-4


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(9, 130, 72), (17, 72, 64), (40, 264, 200), (64, 520, 128), (65, 8, 64), (128, 72, 72), (300, 264, 200), (1000, 520, 512), (129, 1100, 64), (4100, 640, 136),
                                   (33, 9700, 64), (20, 9500, 200), (32, 2048, 2080), (50, 1000, 1700)])
def test_gemm_tcgen05_tiles(dtype, M, N, K):
    """Nine rows and more with K >= 64 run on tcgen05: ragged tile edges in all three dimensions, every tile width, all epilogues,
    against float64 and against the mma.sync kernel.  Up to 64 rows take the decode variant (weights on the M side, a 32- or
    64-token N side, transposed store, K split over several CTAs where the output is narrow and K long)."""
    from mlx_parallm_b200 import _lib, ops
    L = _lib.lib()
    g = torch.Generator().manual_seed(M + N + K)
    x = (torch.randn(M, K, generator=g) / 4).to(dtype).cuda()
    w = (torch.randn(N, K, generator=g) / 4).to(dtype).cuda()
    want = x.double() @ w.double().T
    got = ops.gemm(x, w, _lib.GEMM_STORE_F32)
    got16 = ops.gemm(x, w, _lib.GEMM_STORE)
    L.b200p_gemm_set_path(1)
    try:
        other = ops.gemm(x, w, _lib.GEMM_STORE_F32)
    finally:
        L.b200p_gemm_set_path(0)
    assert L.b200p_gemm_tc_fault() == 0
    assert (got.double() - want).abs().max() <= 2e-5 * math.sqrt(K)
    assert (got - other).abs().max() <= 2e-5 * math.sqrt(K)
    assert got16.dtype == dtype and (got16.double() - want).abs().max() <= 0.02 * math.sqrt(K) / 4
    if N % 2 == 0:
        lim = 0.7
        a = torch.clamp(want[:, 0::2], max=lim)
        u = torch.clamp(want[:, 1::2], -lim, lim)
        glu = ops.gemm(x, w, _lib.GEMM_GLU_CLAMP, act=(lim, 0.0))
        assert glu.shape == (M, N // 2) and (glu.double() - a * torch.sigmoid(1.702 * a) * (u + 1)).abs().max() < 0.02


@pytest.mark.parametrize("M,N,K,batch", [(1, 35, 520, 1), (2, 16, 504, 2), (2, 17, 512, 3), (3, 50, 1032, 1), (4, 31, 2056, 2), (8, 40, 6144, 1), (8, 16, 6152, 1), (5, 3, 4096, 2)])
def test_gemv_of_few_rows(M, N, K, batch):
    """Up to eight rows: x staged in shared memory (512 <= K, up to 96 KB) or read in place, pieces of K that end inside a warp's four, odd
    numbers of columns and warps without any, rows and products strided; a row's bits do not depend on how many others there are."""
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = (torch.randn(M, batch, K, generator=g, device="cuda") / 4).to(torch.bfloat16)
    w = (torch.randn(batch, N, K, generator=g, device="cuda") / 4).to(torch.bfloat16)
    out = torch.full((M, batch, N), 7.0, device="cuda")
    args = dict(batch=batch, strides=(K, N * K, N), N=N, K=K, ldx=batch * K, ldw=K, ldy=batch * N)
    ops.gemm(x, w, _lib.GEMM_STORE_F32, out=out, M=M, **args)
    want = torch.einsum("mbk,bnk->mbn", x.double(), w.double())
    assert (out.double() - want).abs().max() <= 2e-5 * math.sqrt(K)
    one = torch.empty((1, batch, N), device="cuda")
    ops.gemm(x[M - 1:], w, _lib.GEMM_STORE_F32, out=one, M=1, **args)
    assert torch.equal(one[0], out[M - 1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K,batch", [(65, 2, 64, 1), (96, 256, 72, 1), (257, 300, 200, 1), (512, 257, 448, 1), (777, 1030, 136, 1), (1000, 640, 64, 3),
                                         (4100, 5000, 320, 1), (65, 2, 1032, 1), (257, 300, 1096, 1), (513, 257, 1032, 1), (777, 1030, 1032, 1), (300, 640, 1032, 3),
                                         (1030, 31, 1032, 1), (129, 200, 768, 2), (200, 130, 1024, 1), (2100, 128, 512, 2)])
def test_gemm_pairs_of_ctas(dtype, M, N, K, batch):
    """More than 64 rows: two CTAs on one tile of 256 output columns x up to 256 tokens, or one on 128 tokens x 64 to 256 columns (stores and the
    squared relu at a short K or a narrow output): ragged edges in all three dimensions, columns that end in the first CTA's half, one tile for
    a pair and several, batches, all kinds of stores."""
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = (torch.randn(batch, M, K, generator=g, device="cuda") / 4).to(dtype)
    w = (torch.randn(batch, N, K, generator=g, device="cuda") / 4).to(dtype)
    want = torch.einsum("bmk,bnk->mbn", x.double(), w.double())
    for epi in (_lib.GEMM_STORE_F32, _lib.GEMM_STORE, _lib.GEMM_RELU_SQ, _lib.GEMM_CAP_F32, _lib.GEMM_GLU_SILU):
        gated = epi == _lib.GEMM_GLU_SILU
        if gated and N % 2:
            continue
        cols = N // 2 if gated else N
        out = torch.full((M, batch, cols), 7.0, dtype=torch.float32 if _lib.gemm_is_f32(epi) else dtype, device="cuda")
        ops.gemm(x, w, epi, out=out, act=(3.0, 0.0), batch=batch, strides=(M * K, N * K, cols), M=M, N=N, K=K, ldx=K, ldw=K, ldy=batch * cols)
        ref, tol = want, 2e-5 * math.sqrt(K)                        # sums of K products of about 1 / 16 in fp32
        if epi == _lib.GEMM_RELU_SQ:
            ref = want.clamp(min=0).square()
        elif epi == _lib.GEMM_CAP_F32:
            ref = 3.0 * torch.tanh(want / 3.0)
        elif gated:
            ref = torch.nn.functional.silu(want[..., 0::2]) * want[..., 1::2]
        if not _lib.gemm_is_f32(epi):                               # one rounding to 8 or 11 bits of the largest result
            tol += float(ref.abs().max()) * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11)
        assert (out.double() - ref).abs().max() <= tol, epi
    assert _lib.lib().b200p_gemm_tc_fault() == 0


@pytest.mark.parametrize("M", [330, 24, 57])
def test_gemm_tcgen05_heads_and_strides(M):
    """One weight block per head, operands and outputs strided inside wider rows (3-d tensor maps)."""
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator().manual_seed(11)
    H, dk, R = 3, 64, 40
    q = (torch.randn(M, H * dk, generator=g) / 4).to(torch.bfloat16).cuda()
    wk = (torch.randn(H, R, dk, generator=g) / 4).to(torch.bfloat16).cuda()
    want = torch.einsum("mhd,hrd->mhr", q.double().view(M, H, dk), wk.double()).reshape(M, H * R)
    for epi, dt, tol in ((_lib.GEMM_STORE_F32, torch.float32, 2e-4), (_lib.GEMM_STORE, torch.bfloat16, 0.03)):
        out = torch.full((M, H * R), 7.0, dtype=dt, device="cuda")
        ops.gemm(q, wk, epi, out=out, batch=H, strides=(dk, R * dk, R), M=M, N=R, K=dk, ldx=H * dk, ldw=dk, ldy=H * R)
        assert (out.double() - want).abs().max() < tol
    assert _lib.lib().b200p_gemm_tc_fault() == 0


def test_norm_add_norm_parts():
    from mlx_parallm_b200 import ops
    g = torch.Generator().manual_seed(1)
    M, W, eps = 5, 37, 1e-3
    h, y = torch.randn(M, W, generator=g), torch.randn(M, W, generator=g) * 3
    wp, wn = torch.randn(W, generator=g), torch.randn(W, generator=g)
    hd = h.cuda()
    x = torch.empty(M, W, device="cuda")
    raw = torch.empty(M, W, device="cuda")
    ops.norm_add_norm(hd, eps, torch.float32, y=y.cuda(), w_post=wp.cuda(), w_next=wn.cuda(), x_out=x, raw_out=raw)
    h2 = h.double() + O.rms_norm(y.double(), wp.double(), eps)
    assert (hd.double().cpu() - h2).abs().max() < 1e-5 and (raw.double().cpu() - h2).abs().max() < 1e-5
    assert (x.double().cpu() - O.rms_norm(h2, wn.double(), eps)).abs().max() < 1e-5


def test_hashed_embedding_across_portions():
    """The pair (previous, current) must also be right at the start of a portion (previous token from the row's state) and at
    the very first token (the extra row); large multipliers must not overflow."""
    cfg = O.make_config([O.delta_layer(1, 1, 4, 4, conv=1)], vocab=50, width=8, bigram=(47, 2 ** 30 + 3, 2 ** 29 + 1), side_dim=0)
    m, w = build(cfg)
    t = toks(cfg, 9, 3)
    P = {k: v.double() for k, v in w.items()}
    big = cfg["embedding"]["bigram"]
    want = O.hashed_embedding(t, P["embed"], P["bigram"], cfg["embedding"]["scale"], big["buckets"], big["mul_prev"], big["mul_cur"])
    got = []
    from mlx_parallm_b200 import ops
    for lo, hi in ((0, 1), (1, 4), (4, 5), (5, 9)):          # the kernel alone, one portion at a time, in row 1 of 2
        n = hi - lo
        ids = torch.tensor(t[lo:hi], dtype=torch.int32, device="cuda")
        i32 = dict(dtype=torch.int32, device="cuda")
        cu, rows = torch.tensor([0, n], **i32), torch.tensor([1], **i32)
        lengths = torch.tensor([0, lo], **i32)
        last = torch.tensor([0, t[lo - 1] if lo else 0], **i32)
        tr, tp, to = (torch.empty(n, **i32) for _ in range(3))
        ops.ragged_plan(cu, rows, lengths, tr, tp, to, 1, n)
        h = torch.empty(n, 8, device="cuda")
        ops.embed_hashed(ids, tr, tp, to, last, m.embed.weight, m.embed.bigram, h, m.embed.scale, m.embed.buckets, m.embed.mul_prev,
                         m.embed.mul_cur)
        got.append(h.cpu())
    assert (torch.cat(got).double() - want).abs().max() < 1e-6


def _attn_kernel_case(T, H, R, window, hot_query, hot_key, dtype=torch.float32):
    """Random latents and queries; query ``hot_query`` and latent ``hot_key`` are made parallel and long, so that head 0 of
    that query puts nearly all its weight on that key exactly when it may see it."""
    g = torch.Generator().manual_seed(T + R)
    c = torch.randn(T, R, generator=g) * 0.3
    q = torch.randn(T, H, R, generator=g) * 0.3
    d = torch.randn(R, generator=g)
    d = d / d.norm()
    c[hot_key] = 6.0 * d
    q[hot_query, 0] = 6.0 * d
    c = c.to(dtype)
    want = torch.zeros(T, H, R, dtype=torch.float64)
    for i in range(T):
        lo = 0 if window <= 0 else max(0, i - window + 1)
        p = torch.softmax(torch.einsum("hr,jr->hj", q[i].double(), c[lo:i + 1].double()) * 0.5, -1)
        want[i] = p @ c[lo:i + 1].double()
    return q, c, want


@pytest.mark.parametrize("T,window,dist", [(80, 16, 15), (80, 16, 16), (70, 33, 32), (70, 33, 33), (600, 0, 577), (90, 64, 63), (90, 64, 64),
                                           (40, 1, 0), (40, 1, 1)])
def test_latent_attention_window_edges_prompt_and_decode(T, window, dist):
    """A dominant key ``dist`` positions back: just inside the window it decides the output, one further it must be unseen.
    The same positions through one prompt pass and through single-token steps over the cache."""
    from mlx_parallm_b200 import ops
    H, R = 3, 40
    iq = T - 2
    q, c, want = _attn_kernel_case(T, H, R, window, iq, iq - dist)
    i32 = dict(dtype=torch.int32, device="cuda")
    cache = torch.zeros(2, T + 5, R, device="cuda")
    cache[1, :T] = c.cuda()
    rows, pos = torch.full((T,), 1, **i32), torch.arange(T, **i32)
    out = torch.empty(T, H * R, device="cuda")
    ops.latent_attn(q.reshape(T, H * R).cuda().contiguous(), cache, rows, pos, out, H, R, window, 0.5)
    assert (out.double().cpu().view(T, H, R) - want).abs().max() < 1e-4
    inside = window <= 0 or dist < window
    assert (want[iq, 0] - c[iq - dist].double()).abs().max() < 0.2 if inside else (want[iq, 0] - c[iq - dist].double()).abs().max() > 1.0
    for i in (iq - 1, iq, iq + 1):          # decoded alone
        o1 = torch.empty(1, H * R, device="cuda")
        ops.latent_attn(q[i].reshape(1, H * R).cuda().contiguous(), cache, rows[:1], pos[i:i + 1], o1, H, R, window, 0.5)
        assert torch.equal(o1[0], out[i])


# ---- whole models -------------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("name", list(CONFIGS))
def test_prompt_logits_and_residuals_match_the_oracle(models, name):
    cfg, m, w = models[name]
    t = toks(cfg, 45, 1)
    res = []
    want = O.forward(cfg, w, t, res)
    got_res = {}
    m.residual_tap = lambda layer, kind, h: got_res.__setitem__(layer, h.clone())
    try:
        got = m.forward_ragged([t], m.make_cache(1), want=[list(range(len(t)))])
    finally:
        m.residual_tap = None
    for i, r in enumerate(res):
        assert (got_res[i].double().cpu() - r).abs().max() < 2e-4 * max(1.0, float(r.abs().max())), f"residual after layer {i}"
    assert O.logits_error(got, want) < F32_TOL


@pytest.mark.parametrize("name", list(CONFIGS))
def test_bfloat16_model(name):
    cfg = CONFIGS[name]()
    m, w = build(cfg, seed=3, dtype=torch.bfloat16)
    t = toks(cfg, 60, 2)
    got = m.forward_ragged([t], m.make_cache(1), want=[list(range(len(t)))])
    want = O.forward(cfg, w, t)
    per_pos = sorted(O.logits_error(got[i:i + 1], want[i:i + 1]) for i in range(len(t)))
    # 8 mantissa bits through several narrow layers: a few percent at the typical position, never a different answer
    assert per_pos[len(t) // 2] < BF16_TOL and per_pos[-1] < 1.0, per_pos[-3:]


@pytest.mark.parametrize("name", list(CONFIGS))
def test_portions_and_single_tokens_equal_one_pass(models, name):
    """A prompt cut into portions of 1, 2, 3, ... tokens, and fed token by token, gives the logits of one pass; the portions
    cross every window edge and the convolution's reach."""
    cfg, m, w = models[name]
    t = toks(cfg, 50, 4)
    want = O.forward(cfg, w, t)
    for cuts in ([50], [1, 2, 3, 5, 8, 13, 18], [2] * 25, [1] * 50, [47, 1, 2], [49, 1]):
        cache = m.make_cache(3)
        got, lo = [], 0
        for n in cuts:
            got.append(m.forward_ragged([t[lo:lo + n]], cache, rows=[2], want=[list(range(n))]))
            lo += n
        assert O.logits_error(torch.cat(got), want) < F32_TOL, cuts


@pytest.mark.parametrize("name", ["mixed", "wide"])
def test_decode_step_graph_against_prompt(models, name):
    """Most of a prompt in one pass, the rest through the engine's captured decode step (the generation path), 70 tokens long:
    past every window of the config."""
    from mlx_parallm_b200 import utils
    cfg, m, w = models[name]
    t = toks(cfg, 100, 5)
    want = O.forward(cfg, w, t)
    cache = utils._kv_pool.get_for(m, 1)
    got = [m.forward_ragged([t[:30]], cache, want=[[29]])]
    st = utils._decode_step_for(m, cache, 1, False)
    for tok in t[30:]:
        st.tok.copy_(torch.tensor([tok], dtype=torch.int32))
        st.run()
        got.append(st.logits.clone())
    assert O.logits_error(torch.cat(got), want[29:]) < F32_TOL
    assert cache[-1].offsets == [100]
    # a second group of the same batch size, stepped in turns with the first one whose row list differs: the scratch (and the
    # row list the captured graph reads) is shared by both steps and must be rewritten when the other one ran in between
    big = utils._kv_pool.get_for(m, 3)
    m.forward_ragged([t[:30]], big, rows=[2])
    st2 = utils._decode_step_for(m, big, 1, False)
    st2.set_rows([2])
    cache1 = m.make_cache(1)
    m.forward_ragged([t[:30]], cache1)
    st1 = utils._decode_step_for(m, cache1, 1, False)
    for k, tok in enumerate(t[30:36]):
        for s_ in (st2, st1):
            s_.tok.copy_(torch.tensor([tok], dtype=torch.int32))
            s_.run()
            assert torch.equal(s_.logits, got[1 + k]), (k, s_ is st1)


def test_ragged_batch_equals_each_alone_and_rows_end_early(models):
    """Four prompts of 1, 2, 17 and 40 tokens in one pass, then decoded together while the short ones end: bit-equal to each
    request alone in a cache of its own, and right against the oracle."""
    from mlx_parallm_b200 import utils
    cfg, m, w = models["mixed"]
    lens, extra = [1, 2, 17, 40], [0, 3, 12, 12]
    seqs = [toks(cfg, n + e, 10 + n) for n, e in zip(lens, extra)]
    cache = utils._kv_pool.get_for(m, 4)
    rows = [2, 0, 3, 1]
    first = m.forward_ragged([s[:n] for s, n in zip(seqs, lens)], cache, rows=rows, want=[list(range(n)) for n in lens])
    together = {i: [] for i in range(4)}
    o = 0
    for i, n in enumerate(lens):
        together[i].append(first[o:o + n])
        o += n
    m.release_rows(cache, [rows[0]])
    for k in range(12):
        live = [i for i in range(1, 4) if k < extra[i]]
        st = utils._decode_step_for(m, cache, len(live), False)
        st.set_rows([rows[i] for i in live])
        st.tok.copy_(torch.tensor([seqs[i][lens[i] + k] for i in live], dtype=torch.int32))
        st.run()
        for j, i in enumerate(live):
            together[i].append(st.logits[j:j + 1].clone())
        if k + 1 == extra[1]:
            m.release_rows(cache, [rows[1]])
    for i in range(4):
        got = torch.cat(together[i])
        assert O.logits_error(got, O.forward(cfg, w, seqs[i])) < F32_TOL
        alone_cache = m.make_cache(1)
        alone = [m.forward_ragged([seqs[i][:lens[i]]], alone_cache, want=[list(range(lens[i]))])]
        for tok in seqs[i][lens[i]:]:
            alone.append(m.forward_ragged([[tok]], alone_cache))
        assert torch.equal(torch.cat(alone), got), f"request {i} depends on its batch"


def test_rows_given_back_start_from_nothing(models):
    """A row that held a long sequence is released and takes a new one, alone and beside a row that goes on: the new sequence
    sees no state, no latents and no previous token of the old one."""
    cfg, m, w = models["mixed"]
    cache = m.make_cache(2)
    old, keep, new = toks(cfg, 60, 20), toks(cfg, 30, 21), toks(cfg, 25, 22)
    m.forward_ragged([old, keep[:20]], cache)
    m.release_rows(cache, [0])
    assert cache[0].offsets == [0, 20]
    got = m.forward_ragged([new[:3], keep[20:]], cache, want=[[0, 1, 2], list(range(10))])
    assert O.logits_error(got[:3], O.forward(cfg, w, new)[:3]) < F32_TOL
    assert O.logits_error(got[3:], O.forward(cfg, w, keep)[20:]) < F32_TOL
    rest = m.forward_ragged([new[3:]], cache, rows=[0], want=[list(range(22))])
    assert O.logits_error(rest, O.forward(cfg, w, new)[3:]) < F32_TOL


def test_first_tokens_and_short_sequences(models):
    """Sequences shorter than the convolution, one-token sequences in a batch, and the first-token bucket."""
    cfg, m, w = models["mixed"]
    seqs = [toks(cfg, n, 30 + n) for n in (1, 1, 2, 3, 4)]
    got = m.forward_ragged(seqs, m.make_cache(5), want=[list(range(len(s))) for s in seqs])
    want = torch.cat([O.forward(cfg, w, s) for s in seqs])
    assert O.logits_error(got, want) < F32_TOL


def test_far_memory_of_the_recurrence():
    """With decay close to one and wide keys a write is still readable 150 tokens later (every later write erases only the part
    along its own key): the state must survive a long prompt and a portion boundary in between."""
    cfg = O.make_config([O.delta_layer(1, 1, 64, 8, conv=2)], vocab=40, width=16, bigram=None, side_dim=0)
    w = O.random_weights(cfg, 9)
    w["l0.mix.A_log"] = torch.full((1,), -9.0).to(torch.bfloat16)          # decay = exp(-exp(-9) * softplus) ~ 1
    from mlx_parallm_b200.utils import _get_classes
    Model, Args = _get_classes(cfg)
    m = Model(Args.from_dict(cfg)).load_weights(w, device="cuda", dtype=torch.float32)
    t = toks(cfg, 160, 6)
    t2 = list(t)
    t2[3] = (t[3] + 1) % 40
    a, b = O.forward(cfg, w, t)[-1], O.forward(cfg, w, t2)[-1]
    assert O.logits_error(a[None], b[None]) > 1e-3                        # the oracle itself remembers token 3
    cache = m.make_cache(1)
    m.forward_ragged([t[:80]], cache)
    got = m.forward_ragged([t[80:]], cache)
    assert O.logits_error(got, a[None]) < F32_TOL
    lost = m.forward_ragged([t[80:]], m.make_cache(1))                    # without the first portion's state: clearly different
    assert O.logits_error(lost, a[None]) > 1e-2


def test_long_decoding(models):
    from mlx_parallm_b200 import utils
    cfg, m, w = models["odd"]
    t = toks(cfg, 330, 8)
    want = O.forward(cfg, w, t)
    cache = utils._kv_pool.get_for(m, 1)
    m.forward_ragged([t[:5]], cache)
    st = utils._decode_step_for(m, cache, 1, False)
    got = []
    for tok in t[5:]:
        st.tok.copy_(torch.tensor([tok], dtype=torch.int32))
        st.run()
        got.append(st.logits.clone())
    assert O.logits_error(torch.cat(got), want[5:]) < F32_TOL


def test_greedy_generation_through_generate_step(models):
    """The engine's own entry point: left-padded prompts with their lengths, prefill, then the captured decode step feeding
    its own argmax back.  Compared with greedy decoding of the oracle, request by request (float32: no near-ties expected at
    these sizes; a differing token must be a near-tie of the oracle)."""
    from mlx_parallm_b200 import utils
    cfg, m, w = models["mixed"]
    prompts = [toks(cfg, n, 40 + n) for n in (3, 9, 6)]
    L = max(len(p) for p in prompts)
    padded = torch.tensor([[0] * (L - len(p)) + p for p in prompts])
    n_new = 8
    gen = utils.generate_step(padded, m, prompt_lengths=[len(p) for p in prompts])
    got = torch.cat([y for _, (y, _) in zip(range(n_new), gen)], 1).cpu().tolist()
    for p, g in zip(prompts, got):
        seq = list(p)
        for tok in g:
            lg = O.forward(cfg, w, seq)[-1]
            best = int(lg.argmax())
            assert tok == best or float(lg[best] - lg[tok]) < 1e-3 * float(lg.abs().max())
            seq.append(tok)
    # the rectangular call without lengths feeds the padding like any token (the other models' behaviour)
    gen = utils.generate_step(padded[1:2, L - 9:], m)
    again = torch.cat([y for _, (y, _) in zip(range(n_new), gen)], 1).cpu().tolist()[0]
    assert again == got[1]


def test_batch_generate_front_end(models):
    from fake_tokenizer import FakeTokenizer
    from mlx_parallm_b200 import utils
    from mlx_parallm_b200.tokenizer_utils import TokenizerWrapper
    cfg, m, w = models["mixed"]
    tok = TokenizerWrapper(FakeTokenizer(vocab_size=cfg["vocab"]))
    out = utils.batch_generate(m, tok, ["w5 w6", "w5 w6 w7 w8 w9 w10 w11"], max_tokens=5, format_prompts=False)
    alone = utils.batch_generate(m, tok, ["w5 w6"], max_tokens=5, format_prompts=False)
    assert len(out) == 2 and out[0] == alone[0]


@pytest.mark.parametrize("R,window", [(32, 0), (64, 9), (96, 64), (256, 65), (512, 40), (576, 0), (640, 70), (544, 64)])
def test_latent_attention_tile_kernel(R, window):
    """The tensor-core prompt kernel against float64, on a ragged batch whose entries start at different positions of
    different cache rows (1 to 70 tokens, so tiles are full, partial and single), with a dominant key placed exactly at the
    window's edge of one query: inside for one entry, one position too far for another."""
    from mlx_parallm_b200 import ops
    H, scale = 3, 0.4
    starts, counts, rows = [0, 3, 100, 0, 20], [1, 5, 16, 17, 70], [4, 0, 2, 1, 3]
    g = torch.Generator().manual_seed(R + window)
    Tcap = 192
    cache = (torch.randn(5, Tcap, R, generator=g) * 0.3).to(torch.bfloat16)
    M = sum(counts)
    q = torch.randn(M, H, R, generator=g) * 0.3
    cu = [0]
    for n in counts:
        cu.append(cu[-1] + n)
    d = torch.randn(R, generator=g)
    d = d / d.norm()
    if window > 1:
        # entry 2 (row 2): query at position 110, key window - 1 back (seen); entry 4 (row 3): query at position 80, key window back
        cache[2, 110 - (window - 1)] = (5.0 * d).to(torch.bfloat16)
        q[cu[2] + 10, 0] = 5.0 * d
        cache[3, 80 - window] = (5.0 * d).to(torch.bfloat16)
        q[cu[4] + 60, 0] = 5.0 * d
    i32 = dict(dtype=torch.int32, device="cuda")
    t_row = torch.tensor([r for r, n in zip(rows, counts) for _ in range(n)], **i32)
    t_pos = torch.tensor([s + i for s, n in zip(starts, counts) for i in range(n)], **i32)
    cd, qd = cache.cuda(), q.reshape(M, H * R).cuda().contiguous()
    tiles = torch.empty(M, H * R, dtype=torch.bfloat16, device="cuda")
    ops.latent_attn(qd, cd, t_row, t_pos, tiles, H, R, window, scale, cu=torch.tensor(cu, **i32), rows=torch.tensor(rows, **i32),
                    nb=5, max_n=70)
    from mlx_parallm_b200 import _lib
    for buffers in (1, 2):                 # one chunk buffer, or the next chunk in flight during the products: the same numbers
        other = torch.empty_like(tiles)
        _lib.lib().b200p_latent_attn_set_buffers(buffers)
        try:
            ops.latent_attn(qd, cd, t_row, t_pos, other, H, R, window, scale, cu=torch.tensor(cu, **i32), rows=torch.tensor(rows, **i32),
                            nb=5, max_n=70)
        finally:
            _lib.lib().b200p_latent_attn_set_buffers(0)
        assert torch.equal(other, tiles), buffers
    single = torch.empty_like(tiles)
    ops.latent_attn(qd, cd, t_row, t_pos, single, H, R, window, scale)
    want = torch.zeros(M, H, R, dtype=torch.float64)
    c64 = cache.double()
    for t in range(M):
        r, p = int(t_row[t]), int(t_pos[t])
        lo = 0 if window <= 0 else max(0, p - window + 1)
        pr = torch.softmax(torch.einsum("hr,jr->hj", q[t].double(), c64[r, lo:p + 1]) * scale, -1)
        want[t] = pr @ c64[r, lo:p + 1]
    want = want.reshape(M, H * R)
    assert (single.double().cpu() - want).abs().max() < 0.02
    assert (tiles.double().cpu() - want).abs().max() < 0.04
    if window > 1:
        seen, unseen, hot = want[cu[2] + 10, :R], want[cu[4] + 60, :R], 5.0 * d.double()
        assert (seen - hot).norm() < 0.2 * hot.norm() and (unseen - hot).norm() > 0.6 * hot.norm()


@pytest.mark.parametrize("splits", [0, 1, 2, 4, 8])
@pytest.mark.parametrize("H,R,window", [(20, 64, 33), (8, 128, 0), (16, 32, 64), (3, 512, 130), (9, 576, 0), (32, 640, 100)])
def test_latent_attention_decode_tiles_over_heads(H, R, window, splits):
    """A decode step (one token per entry) tiles over the heads of each token: against float64 and against the per-token
    kernel, entries at different positions (also position 0), a head count that leaves the last tile partial.  With the keys
    of a tile shared between the CTAs of a cluster (2, 4, 8; 0 = the launch's own choice), some of which get no key at all
    at the early positions."""
    from mlx_parallm_b200 import _lib, ops
    L = _lib.lib()
    g = torch.Generator().manual_seed(H + R)
    pos, rows = [0, 1, 63, 64, 150], [1, 4, 0, 3, 2]
    cache = (torch.randn(5, 160, R, generator=g) * 0.3).to(torch.bfloat16)
    q = torch.randn(5, H, R, generator=g) * 0.3
    i32 = dict(dtype=torch.int32, device="cuda")
    t_row, t_pos = torch.tensor(rows, **i32), torch.tensor(pos, **i32)
    cd, qd = cache.cuda(), q.reshape(5, H * R).cuda().contiguous()
    tiles, single = torch.empty(5, H * R, dtype=torch.bfloat16, device="cuda"), torch.empty(5, H * R, dtype=torch.bfloat16, device="cuda")
    L.b200p_latent_attn_set_splits(splits)
    try:
        ops.latent_attn(qd, cd, t_row, t_pos, tiles, H, R, window, 0.3, cu=torch.arange(6, **i32), rows=t_row, nb=5, max_n=1)
    finally:
        L.b200p_latent_attn_set_splits(0)
    ops.latent_attn(qd, cd, t_row, t_pos, single, H, R, window, 0.3)
    c64 = cache.double()
    for t in range(5):
        lo = 0 if window <= 0 else max(0, pos[t] - window + 1)
        keys = c64[rows[t], lo:pos[t] + 1]
        want = (torch.softmax(q[t].double() @ keys.T * 0.3, -1) @ keys).reshape(-1)
        assert (single[t].double().cpu() - want).abs().max() < 0.02 and (tiles[t].double().cpu() - want).abs().max() < 0.04


def test_latent_attention_tiles_sharing_keys_between_heads():
    """One, two or four 16-row tiles per CTA read the same staged keys: identical numbers, also when the head count leaves
    groups of the last CTA without a head."""
    from mlx_parallm_b200 import _lib, ops
    L = _lib.lib()
    g = torch.Generator().manual_seed(3)
    H, R, window, nb, T = 5, 128, 21, 2, 37
    cache = (torch.randn(nb, 64, R, generator=g) * 0.3).to(torch.bfloat16).cuda()
    q = (torch.randn(nb * T, H * R, generator=g) * 0.3).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    t_row = torch.arange(nb, **i32).repeat_interleave(T)
    t_pos = torch.arange(T, **i32).repeat(nb) + 9
    outs = []
    try:
        for groups in (1, 2, 4, 0):
            L.b200p_latent_attn_set_groups(groups)
            out = torch.empty(nb * T, H * R, dtype=torch.bfloat16, device="cuda")
            ops.latent_attn(q, cache, t_row, t_pos, out, H, R, window, 0.2, cu=torch.tensor([0, T, 2 * T], **i32), rows=torch.arange(nb, **i32),
                            nb=nb, max_n=T)
            outs.append(out)
    finally:
        L.b200p_latent_attn_set_groups(0)
    single = torch.empty_like(outs[0])
    ops.latent_attn(q, cache, t_row, t_pos, single, H, R, window, 0.2)
    assert all(torch.equal(o, outs[0]) for o in outs[1:])
    assert (outs[0].float() - single.float()).abs().max() < 0.03


def test_latent_attention_rank_above_the_tile_kernel():
    """Rank 672 runs on the per-token kernel (the tile kernel stops at 640)."""
    from mlx_parallm_b200 import ops
    g = torch.Generator().manual_seed(8)
    H, R, window, T = 2, 672, 6, 19
    cache = (torch.randn(1, 32, R, generator=g) * 0.2).to(torch.bfloat16)
    q = torch.randn(T, H, R, generator=g) * 0.2
    i32 = dict(dtype=torch.int32, device="cuda")
    t_row, t_pos = torch.zeros(T, **i32), torch.arange(T, **i32) + 4
    out = torch.empty(T, H * R, dtype=torch.bfloat16, device="cuda")
    ops.latent_attn(q.reshape(T, H * R).cuda().contiguous(), cache.cuda(), t_row, t_pos, out, H, R, window, 0.25,
                    cu=torch.tensor([0, T], **i32), rows=torch.zeros(1, **i32), nb=1, max_n=T)
    c64 = cache[0].double()
    for t in range(T):
        p = t + 4
        keys = c64[max(0, p - window + 1):p + 1]
        want = (torch.softmax(q[t].double() @ keys.T * 0.25, -1) @ keys).reshape(-1)
        assert (out[t].double().cpu() - want).abs().max() < 0.02


@pytest.mark.parametrize("dk,dv,H,KH", [(16, 100, 2, 1), (128, 64, 4, 2), (200, 24, 2, 2), (300, 70, 3, 1)])
def test_delta_scan_key_and_value_sizes(dk, dv, H, KH):
    """The recurrence kernel alone against a float64 loop: key sizes that put 4, 8 and 16 lanes on a column, value sizes that
    leave column slots empty or need several thread blocks; one entry continues a stored state, one starts from nothing."""
    import ctypes as C
    from mlx_parallm_b200 import _lib
    L = _lib.lib()
    g = torch.Generator().manual_seed(dk + dv)
    counts, rows, lengths = [11, 3], [2, 0], [5, 0]
    M = sum(counts)
    qn = torch.randn(M, KH, dk, generator=g) / dk
    kn = torch.nn.functional.normalize(torch.randn(M, KH, dk, generator=g), dim=-1)
    v = torch.randn(M, H, dv, generator=g)
    beta, decay = torch.rand(M, H, generator=g), 0.5 + 0.5 * torch.rand(M, H, generator=g)
    state0 = torch.randn(3, H, dk, dv, generator=g) * 0.3
    want_o, want_s = torch.zeros(M, H, dv, dtype=torch.float64), state0.double().clone()
    t = 0
    for n, r, ln in zip(counts, rows, lengths):
        for h in range(H):
            S = want_s[r, h].clone() if ln > 0 else torch.zeros(dk, dv, dtype=torch.float64)
            for i in range(t, t + n):
                k, q_ = kn[i, h // (H // KH)].double(), qn[i, h // (H // KH)].double()
                S = S * decay[i, h].double()
                u = beta[i, h].double() * (v[i, h].double() - S.T @ k)
                S = S + torch.outer(k, u)
                want_o[i, h] = S.T @ q_
            want_s[r, h] = S
        t += n
    i32 = dict(dtype=torch.int32, device="cuda")
    dev = [x.contiguous().cuda() for x in (qn.reshape(M, -1), kn.reshape(M, -1), v.reshape(M, -1), beta, decay, state0)]
    cu, rw, ln = torch.tensor([0, counts[0], M], **i32), torch.tensor(rows, **i32), torch.tensor([0, 0, 5], **i32)
    o = torch.empty(M, H * dv, device="cuda")
    p = lambda x: C.c_void_p(x.data_ptr())
    assert L.b200p_delta_scan(p(dev[0]), p(dev[1]), p(dev[2]), p(dev[3]), p(dev[4]), p(dev[5]), p(cu), p(rw), p(ln), p(o), 2, H, KH, dk, dv,
                              0, None) == 0
    assert (o.double().cpu().view(M, H, dv) - want_o).abs().max() < 1e-4
    assert (dev[5].double().cpu()[[0, 2]] - want_s[[0, 2]]).abs().max() < 1e-4
    assert torch.equal(dev[5].cpu()[1], state0[1])               # a row that no entry names is not touched


@pytest.mark.parametrize("mode,dk", [(0, 128), (1, 128), (1, 100), (2, 128)])
def test_delta_scan_of_more_ctas_than_sms_equals_its_parts(mode, dk):
    """12 entries x 16 heads of 128 value columns are 384 CTAs, run two per SM; the same entries four at a time are 128, run one per SM:
    one summation order, bit for bit, partial chunks and decode entries among them."""
    from mlx_parallm_b200 import ops
    H, KH, dv, lens = 16, 8, 128, [1, 9, 17, 8, 2, 30, 1, 16, 3, 24, 7, 11]
    g, nb, M = torch.Generator(device="cuda").manual_seed(mode), len(lens), sum(lens)
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")
    qn, kn, v = rnd(M, KH * dk) / dk, torch.nn.functional.normalize(rnd(M, KH, dk), dim=-1).reshape(M, -1), rnd(M, H * dv)
    beta, decay = torch.rand(M, H, generator=g, device="cuda"), 0.5 + 0.5 * torch.rand(M, H * (dk if mode == 1 else 1), generator=g, device="cuda")
    states = [(rnd(nb, H, dk, dv) * 0.3)]
    states.append(states[0].clone())
    i32, off = dict(dtype=torch.int32, device="cuda"), [0]
    for n in lens:
        off.append(off[-1] + n)
    rows, lengths, o = torch.arange(nb, **i32), torch.tensor([3] * nb, **i32), [torch.zeros(M, H * dv, device="cuda") for _ in range(2)]
    ops.delta_scan(qn, kn, v, beta, decay, states[0], torch.tensor(off, **i32), rows, lengths, o[0], nb, H, KH, dk, dv, mode)
    for e in range(0, nb, 4):
        ops.delta_scan(qn, kn, v, beta, decay, states[1], torch.tensor(off[e:e + 5], **i32), rows[e:e + 4].contiguous(), lengths, o[1], 4, H, KH, dk, dv, mode)
    assert torch.equal(o[0], o[1]) and torch.equal(states[0], states[1])


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("dk,dv,H,KH,shift", [(16, 31, 2, 1, 0), (32, 64, 4, 4, 1), (50, 66, 2, 2, 0), (64, 64, 3, 1, 0), (100, 96, 4, 2, 0), (128, 128, 20, 4, 1)])
def test_delta_scan_of_decode_steps_equals_the_scan_of_prompts(mode, dk, dv, H, KH, shift):
    """Told that an entry has few tokens, the call runs another kernel than it does for prompts: the same bits, whatever the entries hold in
    fact (none, one, a whole prompt), states of odd widths and at odd addresses (shift), carried and fresh ones."""
    from mlx_parallm_b200 import _lib
    lens, nb = [1, 0, 1, 19, 8, 1], 6
    g, M = torch.Generator(device="cuda").manual_seed(dk + mode), sum(lens)
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")
    qn, kn, v = rnd(M, KH * dk) / dk, torch.nn.functional.normalize(rnd(M, KH, dk), dim=-1).reshape(M, -1).contiguous(), rnd(M, H * dv)
    beta, decay = torch.rand(M, H, generator=g, device="cuda"), 0.5 + 0.5 * torch.rand(M, H * (dk if mode == 1 else 1), generator=g, device="cuda")
    state0 = rnd(nb + 1, H, dk, dv) * 0.3
    i32 = dict(dtype=torch.int32, device="cuda")
    cu, rows = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32), torch.tensor([4, 6, 1, 0, 5, 2], **i32)
    lengths, got = torch.tensor([3, 7, 0, 2, 5, 0, 1], **i32), []
    for tokens in (0, 1, M):
        state = torch.empty(state0.numel() + 2, device="cuda")[shift:shift + state0.numel()]
        state.copy_(state0.reshape(-1))
        o = torch.zeros(M, H * dv, device="cuda")
        p = lambda t: t.data_ptr()
        _lib.check(_lib.lib().b200p_delta_scan_tokens(p(qn), p(kn), p(v), p(beta), p(decay), p(state), p(cu), p(rows), p(lengths), p(o), tokens, nb, H, KH,
                                                      dk, dv, mode, torch.cuda.current_stream().cuda_stream))
        got.append((o, state.clone()))
    assert all(torch.equal(got[0][i], other[i]) for other in got[1:] for i in (0, 1))
    assert torch.equal(got[0][1].view_as(state0)[3], state0[3])             # a row that no entry names is not touched


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dk,dv,H,KH,shift", [(128, 128, 4, 2, 0), (65, 31, 2, 1, 0), (100, 66, 4, 4, 1), (128, 192, 2, 2, 1)])
def test_delta_scan_of_long_entries(mode, dk, dv, H, KH, shift):
    """Entries of 32 tokens and more go in chunks: against a float64 loop, odd lengths, lengths around the border, carried and fresh
    states, widths and addresses that forbid 16-byte accesses; an entry's bits are the same alone and among others, short and long."""
    from mlx_parallm_b200 import _lib
    lens = [32, 33, 31, 1, 71, 0]
    g, nb, M = torch.Generator(device="cuda").manual_seed(dk + mode), len(lens), sum(lens)
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")
    qn, kn, v = rnd(M, KH * dk) / dk ** 0.5, torch.nn.functional.normalize(rnd(M, KH, dk), dim=-1).reshape(M, -1).contiguous(), rnd(M, H * dv)
    beta, decay = torch.rand(M, H, generator=g, device="cuda"), 0.5 + 0.5 * torch.rand(M, H * (dk if mode else 1), generator=g, device="cuda")
    state0 = rnd(nb + 1, H, dk, dv) * 0.3
    i32 = dict(dtype=torch.int32, device="cuda")
    cu, rows, lengths = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), **i32), torch.tensor([4, 6, 1, 0, 5, 2], **i32), torch.tensor([3, 7, 0, 2, 0, 9, 1], **i32)

    def scan(tokens, cu, rows, n):
        state = torch.empty(state0.numel() + 2, device="cuda")[shift:shift + state0.numel()]
        state.copy_(state0.reshape(-1))
        o = torch.zeros(M, H * dv, device="cuda")
        p = lambda t: t.data_ptr()
        _lib.check(_lib.lib().b200p_delta_scan_tokens(p(qn), p(kn), p(v), p(beta), p(decay), p(state), p(cu), p(rows), p(lengths), p(o), tokens, n, H, KH,
                                                      dk, dv, mode, torch.cuda.current_stream().cuda_stream))
        return o, state.view_as(state0)

    o, state = scan(0, cu, rows, nb)
    for e, n in enumerate(lens):
        lo, r = int(cu[e]), int(rows[e])
        if n:
            alone = scan(n, cu[e:e + 2].contiguous(), rows[e:e + 1].contiguous(), 1)
            assert torch.equal(alone[0][lo:lo + n], o[lo:lo + n]) and torch.equal(alone[1][r], state[r]), e
        S = (state0[r] * (int(lengths[r]) > 0)).double() if n else state0[r].double()
        out = []
        for t in range(lo, lo + n):
            k, q_ = (x[t].double().view(KH, dk).repeat_interleave(H // KH, 0) for x in (kn, qn))
            S = S * decay[t].double().view(H, -1, 1)
            u = beta[t].double().unsqueeze(1) * (v[t].double().view(H, dv) - torch.einsum("hkv,hk->hv", S, k))
            S = S + k.unsqueeze(2) * u.unsqueeze(1)
            out.append(torch.einsum("hkv,hk->hv", S, q_).reshape(-1))
        assert (state[r].double() - S).abs().max() < 2e-5                # 71 tokens of fp32 sums over 128 rows of about 0.3, unit keys
        assert not out or (o[lo:lo + n].double() - torch.stack(out)).abs().max() < 2e-5
    assert torch.equal(state[3], state0[3])                              # a row that no entry names is not touched


@pytest.mark.parametrize("lens,H,KH,dv,channel", [([3, 1, 20], 2, 1, 128, True), ([257], 1, 1, 128, False), ([1, 300, 2], 3, 1, 256, True),
                                                  ([130, 3, 129, 9], 4, 2, 128, True), ([5, 600, 2, 30], 2, 2, 128, False)])
def test_delta_prep_rows_equals_the_per_token_kernel(lens, H, KH, dv, channel):
    """Heads of 128 channels and four taps (a warp per 128 channels and 1, 4 or 8 tokens) against the kernel of a block per token, which takes the
    same convolution as five taps, the oldest of weight zero: bit for bit, entries that begin inside a warp's tokens and carried inputs among them."""
    from mlx_parallm_b200 import ops
    dk, taps, M, nb = 128, 4, sum(lens), len(lens)
    C, f32, i32 = 2 * KH * dk + H * dv, torch.float32, torch.int32
    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")        # noqa: E731
    n_dec = H * (dk if channel else 1)
    proj, a, conv_w, state = rnd(M, C + H + 3), rnd(M, n_dec), rnd(C, taps), rnd(nb, taps - 1, C)
    A_log, dt_bias = rnd(H), rnd(n_dec)
    cu = torch.tensor([0] + np.cumsum(lens).tolist(), dtype=i32, device="cuda")
    rows = torch.arange(nb, dtype=i32, device="cuda").flip(0).contiguous()
    lengths = torch.tensor([0, 2, 1, 7][:nb], dtype=i32, device="cuda")  # nothing carried, fewer than taps - 1 inputs, all of them
    t = [torch.zeros(M, dtype=i32, device="cuda") for _ in range(3)]
    ops.ragged_plan(cu, rows, lengths, *t, nb, M)

    def run(conv_w, state, taps):
        out = [torch.zeros((M, n), dtype=f32, device="cuda") for n in (KH * dk, KH * dk, H * dv, H, n_dec)]
        ops.delta_prep(proj, C, a, conv_w, state, A_log, dt_bias, *t, *out, H, KH, dk, dv, taps)
        return out

    per_token = run(torch.cat([torch.zeros(C, 1, device="cuda"), conv_w], 1), torch.cat([rnd(nb, 1, C), state], 1), taps + 1)
    for w, p in zip(run(conv_w, state, taps), per_token):
        assert torch.equal(w, p)


@pytest.mark.parametrize("M,H,KH,dv,channel", [(1, 3, 1, 128, True), (128, 2, 2, 256, False), (131, 2, 1, 128, True), (512, 1, 1, 128, False), (513, 1, 1, 128, False),
                                                 (1025, 2, 1, 128, True)])
def test_delta_prep_of_128_channel_heads(M, H, KH, dv, channel):
    """A warp per 128 channels and 1, 4 or 8 tokens (by their number), one sequence that carries inputs: against float64."""
    from mlx_parallm_b200 import ops
    dk, taps, C = 128, 4, 2 * KH * 128 + H * dv
    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")        # noqa: E731
    nd, i32 = H * (dk if channel else 1), dict(dtype=torch.int32, device="cuda")
    proj, a, conv_w, state, A_log, dt_bias = rnd(M, C + H + 1), rnd(M, nd), rnd(C, taps), rnd(1, taps - 1, C), rnd(H), rnd(nd)
    pos = torch.arange(M, **i32)
    out = [torch.zeros((M, n), device="cuda") for n in (KH * dk, KH * dk, H * dv, H, nd)]
    ops.delta_prep(proj, C, a, conv_w, state, A_log, dt_bias, torch.zeros(M, **i32), pos + 2, pos, *out, H, KH, dk, dv, taps)
    past = torch.cat([state[0].double(), proj[:, :C].double()])
    past[0] = 0                                                         # position 2: two inputs lie before the portion, not three
    act = torch.nn.functional.silu(sum(conv_w.double()[:, j] * past[j:j + M] for j in range(taps)))
    q, k = act[:, :KH * dk].view(M, KH, dk), act[:, KH * dk:2 * KH * dk].view(M, KH, dk)
    unit = lambda z: z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6)        # noqa: E731
    step = torch.nn.functional.softplus(a.double() + dt_bias.double())
    want = [(unit(q) * dk ** -0.5).reshape(M, -1), unit(k).reshape(M, -1), act[:, 2 * KH * dk:], torch.sigmoid(proj[:, C:C + H].double()),
            torch.exp(-A_log.double().exp().repeat_interleave(nd // H) * step)]
    for got, ref in zip(out, want):
        assert (got.double() - ref).abs().max() <= 4e-6 * max(1.0, float(ref.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,dv,col", [(3, 128, 0), (2, 256, 4), (5, 512, 0), (3, 384, 0), (3, 128, 1), (2, 100, 0)])
def test_delta_out_widths(dtype, H, dv, col):
    """Norm, weight and gate per head: 16-byte pieces for groups of 128, 256 and 512 values, the general kernel for other widths and for
    gates that start between 16-byte boundaries."""
    from mlx_parallm_b200 import ops
    M = 7
    g = torch.Generator(device="cuda").manual_seed(dv)
    o, gate = torch.randn(M, H * dv, generator=g, device="cuda"), torch.randn(M, H * dv + 8, generator=g, device="cuda")
    w = 1 + 0.1 * torch.randn(dv, generator=g, device="cuda")
    for act in (0, 1):
        out = torch.zeros(M, H * dv, dtype=dtype, device="cuda")
        gt = gate[:, col:col + H * dv]
        ops.delta_out(o, gt, w, out, H, dv, 1e-5, act)
        x, z = o.double().view(M, H, dv), gt.double()
        s = z * torch.sigmoid(z) if act == 0 else torch.sigmoid(z)
        want = (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w.double()).reshape(M, -1) * s
        tol = {torch.float32: 4e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]      # one rounding
        assert (out.double() - want).abs().max() <= tol * float(want.abs().max())


def test_silu_of_the_delta_kernels_keeps_its_fp32_range():
    """silu(z) for z = -88.5 .. 88.5 wherever the recurrent mixers apply it (convolved q, k, v, the plain accumulation's inputs, the head norm's
    gate of a float32 model) against float64, relative to each value: the smallest, -88 e^-88 = -5e-37, is a normal fp32 number.  Bound:
    __expf's documented error of 2 + 1.173 * 88.5 units in the last place of 2^-23, and two more roundings."""
    from mlx_parallm_b200 import ops
    H, KH, dk, dv, taps, M, bound = 1, 1, 128, 128, 4, 3, 1.3e-5
    z = torch.linspace(-88.5, 88.5, 2 * dk + dv, dtype=torch.float64).float().cuda().repeat(M, 1)
    want = z.double() * torch.sigmoid(z.double())
    rel = lambda got, ref: float(((got.double() - ref).abs() / ref.abs().clamp(min=1e-300)).max())        # noqa: E731
    f32, i32 = dict(dtype=torch.float32, device="cuda"), dict(dtype=torch.int32, device="cuda")
    q, k, v, decay = (torch.zeros(M, n, **f32) for n in (dk, dk, dv, H))
    ops.linear_attn_prep(z, torch.ones(H, **f32), q, k, v, decay, H, dk, dv)
    assert rel(torch.cat([q, k, v], 1), want) < bound
    conv_w = torch.zeros(2 * dk + dv, taps, **f32)
    conv_w[:, -1] = 1                                                  # the convolution hands its newest input through
    proj, beta, pos = torch.cat([z, z[:, :H]], 1), torch.zeros(M, H, **f32), torch.arange(M, **i32)
    ops.delta_prep(proj, 2 * dk + dv, z[:, :H], conv_w, torch.zeros(1, taps - 1, 2 * dk + dv, **f32), torch.zeros(H, **f32), torch.zeros(H, **f32),
                   torch.zeros(M, **i32), pos, pos, q, k, v, beta, decay, H, KH, dk, dv, taps)
    assert rel(v, want[:, 2 * dk:]) < bound                            # (q and k are made unit vectors)
    for heads in (3, 1):                                               # heads of 128 values in 16-byte pieces; one group of all
        gate, o, out = z[:, :dv * 3].contiguous(), torch.ones(M, 3 * dv, **f32), torch.zeros(M, 3 * dv, **f32)
        ops.delta_out(o, gate, torch.ones(3 * dv // heads, **f32), out, heads, 3 * dv // heads, 0.0)
        assert rel(out, want) < bound


@pytest.mark.parametrize("M", [9, 33, 65, 300])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gated_units_of_the_tcgen05_products_keep_their_range(dtype, M):
    """Gates of -88 .. 88 (silu) and -51 .. 51 (clamped, whose sigmoid has 1.702 z) beside an up value of 2^100 in bf16, 1 in f16: each result
    against float64, relative to itself: half a unit of the storage type, and __expf's documented error (2 + 1.17 * 88 units of 2^-23) with
    the few roundings of the unit."""
    from mlx_parallm_b200 import _lib, ops
    up = 2.0 ** 100 if dtype == torch.bfloat16 else 1.0
    half, tiny = (2.0 ** -8, 2.0 ** -126) if dtype == torch.bfloat16 else (2.0 ** -11, 2.0 ** -14)
    for epi, c, most, add in ((_lib.GEMM_GLU_SILU, 1.0, 88.0, 0.0), (_lib.GEMM_GLU_CLAMP, 1.702, 51.0, 1.0)):
        gates = torch.linspace(-most, most, 200, dtype=torch.float64).to(dtype).cuda()
        w = torch.zeros(400, 64, dtype=dtype, device="cuda")
        w[0::2, 0], w[1::2, 0] = gates, up
        x = torch.zeros(M, 64, dtype=dtype, device="cuda")
        x[:, 0] = 1
        got = ops.gemm(x, w, epi, act=(2.0 ** 101, 0.0)).double()
        z = gates.double()
        want = (z * torch.sigmoid(c * z) * (up + add)).expand(M, -1)
        err = (got - want).abs() / want.abs().clamp(min=tiny)          # (below the normal numbers: of the smallest of them)
        assert float(err.max()) <= half + 1.4e-5


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("lens,H", [([40, 1, 1, 3, 0, 33, 2], 3), ([1] * 40 + [32], 8), ([5, 9, 20], 20), ([0] * 30 + [50] + [0] * 40, 2), ([16, 31, 32, 20, 70, 15], 6)])
def test_delta_scan_of_long_entries_among_short_ones(mode, lens, H):
    """The two launches of such a batch overlap, with more CTAs than fit and without; what reads the results behind them sees both.  A call that is
    told its tokens and its longest entry gives the bits of one that is not (which takes both launches), also beside as many empty entries as a
    decode step would have; a length that is told too small changes no more than the order of the sums."""
    from mlx_parallm_b200 import _lib
    g, nb, M, KH, dk, dv = torch.Generator(device="cuda").manual_seed(H + mode), len(lens), sum(lens), 1, 128, 128
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")        # noqa: E731
    qn, kn, v = rnd(M, KH * dk) / dk ** 0.5, torch.nn.functional.normalize(rnd(M, KH, dk), dim=-1).reshape(M, -1).contiguous(), rnd(M, H * dv)
    beta, decay = torch.rand(M, H, generator=g, device="cuda"), 0.5 + 0.5 * torch.rand(M, H * (dk if mode else 1), generator=g, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    cu, rows, lengths = torch.tensor([0] + np.cumsum(lens).tolist(), **i32), torch.arange(nb, **i32), torch.full((nb,), 3, **i32)
    state0, got = rnd(nb, H, dk, dv) * 0.3, []
    for tokens, longest in ((0, 0), (M, max(lens)), (M, 1)):
        state, o = state0.clone(), torch.zeros(M, H * dv, device="cuda")
        _lib.check(_lib.lib().b200p_delta_scan_entries(*(t.data_ptr() for t in (qn, kn, v, beta, decay, state, cu, rows, lengths, o)), tokens, longest, nb,
                                                       H, KH, dk, dv, mode, torch.cuda.current_stream().cuda_stream))
        got.append((o * 1, state * 1))
        state.zero_()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert (got[0][0] - got[2][0]).abs().max() < 4e-5 and (got[0][1] - got[2][1]).abs().max() < 4e-5        # (2e-5 each: the test above)
    for e in [e for e in range(nb) if lens[e]]:              # and each entry those that it has alone
        a, b = int(cu[e]), int(cu[e + 1])
        state, o = state0[e:e + 1].clone(), torch.zeros(b - a, H * dv, device="cuda")
        one, alone = torch.tensor([0, b - a], **i32), [t[a:b].contiguous() for t in (qn, kn, v, beta, decay)]
        _lib.check(_lib.lib().b200p_delta_scan_entries(*(t.data_ptr() for t in (*alone, state, one, rows, lengths, o)), b - a, b - a, 1, H, KH, dk, dv, mode,
                                                       torch.cuda.current_stream().cuda_stream))
        assert torch.equal(o, got[1][0][a:b]) and torch.equal(state[0], got[1][1][e])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dk,dv,in_place", [(128, 16, False), (128, 17, False), (72, 64, False), (128, 129, False), (128, 128, True)])
def test_delta_scan_in_chunks(mode, dk, dv, in_place):
    """Entries of 32 tokens and more, 16 at a time, against float64 with the recurrence's fp32 bound (the test of long entries): last chunks of 1, 15 and 16
    tokens, the narrowest outputs that hold a chunk's intermediate numbers and the widest that do not, outputs in the memory of v, decays of zero and
    of 1e-30 (quotients of decays would be infinite); a key of NaN reaches no token before it and no other entry."""
    from mlx_parallm_b200 import ops
    H, KH, lens, bad = 2, 1, [33, 48, 63, 47], 20
    g, nb, M = torch.Generator(device="cuda").manual_seed(dk + dv + mode), len(lens), sum(lens)
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")        # noqa: E731
    nd = dk if mode else 1
    qn, kn, v = rnd(M, KH * dk) / dk ** 0.5, torch.nn.functional.normalize(rnd(M, KH, dk), dim=-1).reshape(M, -1).contiguous(), rnd(M, H * dv)
    beta, decay = torch.rand(M, H, generator=g, device="cuda"), 0.5 + 0.5 * torch.rand(M, H * nd, generator=g, device="cuda")
    decay[5::11, ::3], decay[7::13, ::2] = 0.0, 1e-30
    i32, off = dict(dtype=torch.int32, device="cuda"), [0]
    for n in lens:
        off.append(off[-1] + n)
    cu, rows, lengths, state0 = torch.tensor(off, **i32), torch.arange(nb, **i32), torch.full((nb,), 3, **i32), rnd(nb, H, dk, dv) * 0.3

    def scan(kn):
        state, vals = state0.clone(), v.clone()
        o = vals if in_place else torch.empty(M, H * dv, device="cuda")
        ops.delta_scan(qn, kn, vals, beta, decay, state, cu, rows, lengths, o, nb, H, KH, dk, dv, mode, longest=max(lens))
        return o, state

    o, state = scan(kn)
    for e in range(nb):
        S = state0[e].double()
        for t in range(off[e], off[e + 1]):
            S = S * decay[t].double().view(H, -1, 1)
            u = beta[t].double().unsqueeze(1) * (v[t].double().view(H, dv) - torch.einsum("hkv,k->hv", S, kn[t].double()))
            S = S + kn[t].double().view(1, dk, 1) * u.unsqueeze(1)
            assert (o[t].double() - torch.einsum("hkv,k->hv", S, qn[t].double()).reshape(-1)).abs().max() < 2e-5
        assert (state[e].double() - S).abs().max() < 2e-5
    spoilt = kn.clone()
    spoilt[off[1] + bad, 3] = float("nan")
    o2, state2 = scan(spoilt)
    keep = [t for t in range(M) if not off[1] + bad <= t < off[2]]
    assert (o2[keep] - o[keep]).abs().max() < 2e-5 and o2[off[1] + bad:off[2]].isnan().all()
    assert torch.equal(state2[[0, 2, 3]], state[[0, 2, 3]]) and state2[1].isnan().any()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("slow", [False, True])
def test_delta_scan_in_chunks_is_as_exact_as_token_by_token(mode, slow):
    """The products of long entries run on the tensor cores with nothing lost against fp32: the distance from 64 bits is that of the token-by-token kernel
    (which outputs in the memory of v take).  1.25: both are a few roundings per number (measured 0.60 to 1.07; operands short of their last bits: 2)."""
    from mlx_parallm_b200 import ops
    F = torch.nn.functional
    H, KH, dk, dv, lens = 16, 8, 128, 128, [300, 260, 33, 100]
    g, nb, M = torch.Generator(device="cuda").manual_seed(mode), len(lens), sum(lens)
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")        # noqa: E731
    qn, kn = (F.normalize(F.silu(rnd(M, KH, dk)), dim=-1) for _ in range(2))
    qn, v, beta, nd = qn * dk ** -0.5, F.silu(rnd(M, H, dv)), rnd(M, H).sigmoid(), dk if mode else 1
    a = (torch.rand(H, generator=g, device="cuda") * 3 - 2).exp().view(1, H, 1)
    decay = 1 - 0.02 * torch.rand(M, H, nd, generator=g, device="cuda") if slow else torch.exp(-a * F.softplus(rnd(M, H, nd) + rnd(1, H, nd)))
    i32, off = dict(dtype=torch.int32, device="cuda"), [0]
    for n in lens:
        off.append(off[-1] + n)
    cu, rows, lengths, state0 = torch.tensor(off, **i32), torch.arange(nb, **i32), torch.full((nb,), 3, **i32), rnd(nb, H, dk, dv) * 0.3
    S, want = state0.double(), torch.empty(M, H, dv, dtype=torch.float64, device="cuda")
    for i in range(max(lens)):
        es = [e for e in range(nb) if i < lens[e]]
        t = torch.tensor([off[e] + i for e in es], device="cuda")
        k, q = (x[t].double().repeat_interleave(H // KH, 1) for x in (kn, qn))
        new = S[es] * decay[t].double().unsqueeze(-1)
        u = beta[t].double().unsqueeze(-1) * (v[t].double() - torch.einsum("bhkv,bhk->bhv", new, k))
        new = new + k.unsqueeze(-1) * u.unsqueeze(-2)
        want[t], S[es] = torch.einsum("bhkv,bhk->bhv", new, q), new
    err = []
    for in_place in (False, True):
        state, vals = state0.clone(), v.reshape(M, -1).clone()
        o = vals if in_place else torch.empty_like(vals)
        ops.delta_scan(qn.reshape(M, -1), kn.reshape(M, -1), vals, beta, decay.reshape(M, -1).contiguous(), state, cu, rows, lengths, o, nb, H, KH, dk, dv, mode,
                       longest=max(lens))
        err.append([float((x.double() - y).norm() / y.norm()) for x, y in ((o.view(M, H, dv), want), (state, S))])
    assert err[0][0] < 1.25 * err[1][0] and err[0][1] < 1.25 * err[1][1], err


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dv", [65, 3088, 4097])                # two slices; a remainder of 16, of 1 beside slices of 64
def test_delta_scan_in_chunks_of_wide_values(mode, dv):
    """A chunk's intermediate numbers lie in each slice of its rows of the output, so every slice has to be wide enough for them: against float64 with the
    recurrence's fp32 bound; rows behind the output stay as they were."""
    from mlx_parallm_b200 import ops
    dk, lens = 128, [33, 48]
    g, nb, M = torch.Generator(device="cuda").manual_seed(dv + mode), len(lens), sum(lens)
    rnd = lambda *sh: torch.randn(*sh, generator=g, device="cuda")        # noqa: E731
    qn, kn, v = rnd(M, dk) / dk ** 0.5, torch.nn.functional.normalize(rnd(M, dk), dim=-1), rnd(M, dv)
    beta, decay = torch.rand(M, 1, generator=g, device="cuda"), 0.5 + 0.5 * torch.rand(M, dk if mode else 1, generator=g, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    cu, rows, lengths, state0 = torch.tensor([0, 33, M], **i32), torch.arange(nb, **i32), torch.full((nb,), 3, **i32), rnd(nb, 1, dk, dv) * 0.3
    state, buf = state0.clone(), torch.full((M + 300, dv), 7.0, device="cuda")
    ops.delta_scan(qn, kn, v, beta, decay, state, cu, rows, lengths, buf[:M], nb, 1, 1, dk, dv, mode, longest=max(lens))
    assert bool((buf[M:] == 7).all())
    for e, (a, b) in enumerate([(0, 33), (33, M)]):
        S = state0[e, 0].double()
        for t in range(a, b):
            S = S * decay[t].double().view(-1, 1)
            u = beta[t].double() * (v[t].double() - S.t() @ kn[t].double())
            S = S + kn[t].double().view(-1, 1) * u
            assert (buf[t].double() - S.t() @ qn[t].double()).abs().max() < 2e-5
        assert (state[e, 0].double() - S).abs().max() < 2e-5


@pytest.mark.parametrize("M,N,K,batch", [(1, 64, 128, 9), (2, 512, 128, 16), (5, 128, 512, 64), (8, 130, 512, 3), (3, 128, 1024, 40), (1, 128, 520, 64)])
def test_gemv_of_short_rows(M, N, K, batch):
    """Few rows over many short weight rows (per-head products): one piece of a row at a time; from 512 channels, where the CTAs fit the GPU
    twice, and from 1024 four of them and staged x."""
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = (torch.randn(M, batch, K, generator=g, device="cuda") / 4).bfloat16()
    w = (torch.randn(batch, N, K, generator=g, device="cuda") / 4).bfloat16()
    out = torch.full((M, batch, N), 7.0, device="cuda")
    ops.gemm(x, w, _lib.GEMM_STORE_F32, out=out, batch=batch, strides=(K, N * K, N), M=M, N=N, K=K, ldx=batch * K, ldw=K, ldy=batch * N)
    want = torch.einsum("mbk,bnk->mbn", x.double(), w.double())
    assert (out.double() - want).abs().max() <= 2e-5 * math.sqrt(K)


@pytest.mark.parametrize("M,N,K,ld,shift", [(130, 96, 64, 96, 1), (130, 96, 128, 97, 0), (200, 33, 256, 40, 4), (129, 64, 72, 200, 8), (1025, 32, 1032, 32, 2)])
def test_gemm_rows_at_any_output_address(M, N, K, ld, shift):
    """Short K and narrow outputs store a token's outputs as 16-byte pieces where address and row stride allow it: others, and columns that are
    not theirs, stay right."""
    from mlx_parallm_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(M + N + ld)
    x, w = (torch.randn(n, K, generator=g, device="cuda").bfloat16() for n in (M, N))
    want = x.double() @ w.double().T
    for epi, dt in ((_lib.GEMM_STORE_F32, torch.float32), (_lib.GEMM_STORE, torch.bfloat16)):
        buf = torch.full((M * ld + 16,), 7.0, dtype=dt, device="cuda")
        ops.gemm(x, w, epi, out=buf[shift:shift + M * ld].view(M, ld)[:, :N], ldy=ld)
        rows = buf[shift:shift + M * ld].view(M, ld)
        tol = 2e-5 * math.sqrt(K) + (2.0 ** -8 * float(want.abs().max()) if dt == torch.bfloat16 else 0.0)
        assert (rows[:, :N].double() - want).abs().max() <= tol and bool((rows[:, N:] == 7).all())
        assert bool((buf[:shift] == 7).all()) and bool((buf[shift + M * ld:] == 7).all())
    assert _lib.lib().b200p_gemm_tc_fault() == 0
