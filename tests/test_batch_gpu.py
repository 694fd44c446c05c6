"""Token batches at the edges of the batched kernels' tiles: the tensor-core projections against the dp4a ones, the hybrid
layers against the step-by-step route (needs a B200)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from taraference_b200 import synth as S  # noqa: E402
from tests.test_engine_gpu import TF_WORST, _rel, margin_gated_equal  # noqa: E402

# rows that fill neither row tiles nor row groups' tiles (FF = 1 280, K = 768: three and five blocks), a vocabulary of odd size
ODD = dict(arch="qwen2", n_layer=1, n_embd=768, n_head=6, n_kv=2, head_dim=128, n_ff=1280, n_vocab=3001,
           rope_theta=1e6, eps=1e-6, tied=True, qkv_bias=True)
WIDE = dict(ODD, n_embd=1024, n_head=8, n_kv=1, n_ff=2816, n_vocab=2000)


@pytest.fixture(scope="module")
def E(cuda_lib):
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    from taraference_b200 import engine
    return engine


def _state(m, kv, cfg, n):
    kvdim = cfg["n_kv"] * cfg["head_dim"]
    return [m.debug_read(w, n * kvdim, np.uint16, kv=kv, layer=0) for w in "kv"]


# Sums of the same int8 products by two kernels, of the largest value.  Measured against float64: no kernel is off by more than
# 2e-6 of a result's rms, and a largest value is three to four rms: 1.3e-6.  One and a half times that.
SAME_INT8 = 2e-6


@pytest.mark.parametrize("cfg", [ODD, WIDE], ids=["odd", "wide"])
@pytest.mark.parametrize("n", [5, 16, 17, 32, 33, 48, 80, 81, 128, 129, 224, 256, 257, 640])
def test_projections_of_batches_at_tile_edges(E, oracle, cfg, n, monkeypatch):
    """One layer, all tokens in one batch: 16- and 32-token paddings, mma.sync up to 80 tokens (Q6_K: 32), the tcgen05 forms, several
    token tiles, tiles that end inside a column group.  V rows are the dp4a route's bits, K rows the same up to f16 steps.  The last
    token's vectors are held against the decode kernels stage by stage, each fed the batch's own vector, so that both round the
    same values to int8 and only the order of the fp32 sums differs."""
    tens = S.make_dense_model(cfg, seed=31)
    m = E.CudaModel.load_with(cfg, tens)
    K, FF, nq = cfg["n_embd"], cfg["n_ff"], cfg["n_head"] * cfg["head_dim"]
    taps = [("layer_attn", nq), ("layer_mid", K), ("layer_h", FF), ("layer_x", K)]
    for name, width in taps:
        m.debug_read(name, width)  # switch the taps on
    prompt = [int(t) for t in np.random.default_rng(n).integers(0, cfg["n_vocab"], n)]
    out = []
    for dp4a in (True, False):
        (monkeypatch.setenv if dp4a else monkeypatch.delenv)(*(("TFR_GEMM_DP4A", "1") if dp4a else ("TFR_GEMM_DP4A",)))
        kv = m.alloc_kv(n + 8)
        m.forward_greedy(prompt, kv)
        out.append((*_state(m, kv, cfg, n), [m.debug_read(*t) for t in taps]))
        kv.free()
    (ka, va, ta), (kb, vb, tb) = out
    logits = m.current_logits()
    assert np.array_equal(va, vb)
    f = lambda a: a.view(np.float16).astype(np.float32)
    assert _rel(f(kb), f(ka)) < 5e-4
    assert _rel(tb[0], ta[0]) < 1e-4  # K values that fell to the other f16: 5e-4 of the largest, fewer than one in a hundred
    attn, mid, h, x = (torch.from_numpy(v).cuda() for v in tb)
    mats = {k: E.GpuMat(*tens[k][:3], tens[k][3]) for k in tens if k == "token_embd.weight" or ("blk" in k and isinstance(tens[k], tuple))}
    vec = lambda k: torch.from_numpy(tens[k]).cuda()
    wtype, k, _, raw = tens["token_embd.weight"]
    row = np.ascontiguousarray(raw.reshape(cfg["n_vocab"], -1)[prompt[-1]])
    want = [torch.from_numpy(oracle.dequant_rows(wtype, row, k, 1).reshape(-1)).cuda(), torch.empty(FF, device="cuda"), mid.clone(),
            torch.empty(cfg["n_vocab"], device="cuda")]
    E.op_gemv(mats["blk.0.attn_output.weight"], attn, want[0], use_res=2)
    E.op_ffn_gate_up(mats["blk.0.ffn_gate.weight"], mats["blk.0.ffn_up.weight"], mid, want[1], norm_w=vec("blk.0.ffn_norm.weight"), eps=cfg["eps"])
    E.op_gemv(mats["blk.0.ffn_down.weight"], h, want[2], use_res=2)
    E.op_gemv(mats["token_embd.weight"], x, want[3], norm_w=vec("output_norm.weight"), eps=cfg["eps"])
    for name, got, w in zip(("mid", "h", "x", "logits"), (mid, h, x, torch.from_numpy(logits)), want):
        assert _rel(got.cpu().numpy(), w.cpu().numpy()) < SAME_INT8, name
    for w in mats.values():
        w.free()
    m.destroy()


@pytest.mark.parametrize("n", [64, 65, 72, 80, 81])
def test_projections_of_a_batch_on_both_tensor_core_kernels(E, oracle, n, monkeypatch):
    """The same where gate and up rows are on tcgen05 beside Q, K and output rows on mma.sync: 65 to 80 tokens, more than 4 096 rows."""
    test_projections_of_batches_at_tile_edges(E, oracle, dict(ODD, n_ff=5120), n, monkeypatch)


def _q4_k_exact(raw, K, N):
    """GGUF bytes -> float64 weights, exactly (kernels/common.cu:40-84)."""
    b = raw.reshape(N, K // 256, 144)
    d, dmin = (b[..., i:i + 2].copy().view(np.float16)[..., 0].astype(np.float64) for i in (0, 2))
    s = b[..., 4:16].astype(np.int64)
    sc = np.concatenate([s[..., :4] & 63, (s[..., 8:] & 15) | (s[..., :4] >> 6 << 4)], -1)
    mn = np.concatenate([s[..., 4:8] & 63, (s[..., 8:] >> 4) | (s[..., 4:8] >> 6 << 4)], -1)
    q = b[..., 16:].astype(np.int64).reshape(N, K // 256, 4, 32)
    q = np.stack([q & 15, q >> 4], axis=3).reshape(N, K // 256, 8, 32)
    return (d[..., None, None] * sc[..., None] * q - (dmin[..., None] * mn)[..., None]).reshape(N, K)


def _q6_k_exact(raw, K, N):
    """GGUF bytes -> float64 weights, exactly (kernels/gemv.cu:302-337)."""
    b = raw.reshape(N, K // 256, 210)
    ql, qh = b[..., :128].astype(np.int64).reshape(N, -1, 2, 64), b[..., 128:192].astype(np.int64).reshape(N, -1, 2, 32)
    sc = b[..., 192:208].copy().view(np.int8).astype(np.float64).reshape(N, -1, 2, 8)
    w = np.empty((N, K // 256, 2, 128))
    for j in range(4):
        q = (ql[..., 32 * (j & 1):32 * (j & 1) + 32] >> (4 * (j >> 1)) & 15) | (qh >> (2 * j) & 3) << 4
        w[..., 32 * j:32 * j + 32] = sc[..., 2 * j:2 * j + 2].repeat(16, axis=-1) * (q - 32)
    return (w * b[..., 208:].copy().view(np.float16).astype(np.float64)[..., None]).reshape(N, K)


DP4A, MMA, TC = 0, 1, 2


def _matrix(E, wtype, K, N, rng, scale=0.02):
    raw = S.quantize(wtype, (rng.standard_normal((N, K)) * scale).astype(np.float32)).reshape(-1)
    exact = (_q4_k_exact if wtype == S.Q4_K else _q6_k_exact)(raw, K, N)
    return E.GpuMat(wtype, K, N, raw), torch.from_numpy(exact).cuda()


def _exact_q8(E, x):
    """The int8 activations and their scales as float64."""
    M, K = x.shape
    q8, d8 = torch.empty(M * K, dtype=torch.int8, device="cuda"), torch.empty(M * K // 32, device="cuda")
    E.op_quantize_q8(x.view(-1), q8, d8)
    return (q8.view(-1, 32).double() * d8.view(-1, 1).double()).view(M, K)


def _errors(E, w, exact, x, routes, **kw):
    """Relative error (2-norm) of a batch's projection against float64 sums of the same int8 activations, by route."""
    ref = _exact_q8(E, x) @ exact.T
    errs = []
    for route in routes:
        out = torch.full((x.shape[0], w.N), float("nan"), device="cuda")
        E.op_project_rows(w, x, out, x.shape[0], route=route, **kw)
        errs.append(float((out.double() - ref).norm() / ref.norm()))
    return errs


@pytest.mark.parametrize("wtype", [S.Q4_K, S.Q6_K], ids=["q4", "q6"])
@pytest.mark.parametrize("K,N", [(256, 3), (768, 130), (2816, 257), (11008, 64)])
def test_projection_routes_agree_on_equal_int8(E, wtype, K, N):
    """The three projection kernels on the same int8 activations, against float64, where tiles, token paddings, clusters over
    the k range and pairs of CTAs end; then residuals added, and gate/up pairs with a fused norm."""
    rng = np.random.default_rng(K + N)
    w, exact = _matrix(E, wtype, K, N, rng)
    for M in (5, 16, 17, 32, 33, 80, 81, 128, 129, 257):
        x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
        routes = [DP4A, TC] + ([MMA] if M <= (80 if wtype == S.Q4_K else 32) else [])
        assert max(_errors(E, w, exact, x, routes)) < SAME_INT8, M
    M, norm = 37, torch.from_numpy(rng.uniform(0.5, 2, K).astype(np.float32)).cuda()
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
    w2, _ = _matrix(E, wtype, K, N, rng)
    res = torch.randn((M, N), device="cuda")
    for kw in (dict(use_res=2), dict(b=w2, norm_w=norm) if K < 4096 else dict(b=w2)):
        outs = []
        for route in (DP4A, TC, -1):
            out = res.clone() if "use_res" in kw else torch.full_like(res, float("nan"))
            E.op_project_rows(w, x, out, M, route=route, **kw)
            outs.append(out.cpu().numpy())
        assert _rel(outs[1], outs[0]) < SAME_INT8 and _rel(outs[2], outs[0]) < SAME_INT8, kw.keys()
    w.free()
    w2.free()


@pytest.mark.parametrize("wtype,N,M,pair,route", [
    (S.Q4_K, 512, 4, False, DP4A), (S.Q4_K, 512, 5, False, MMA), (S.Q4_K, 4097, 64, False, MMA), (S.Q4_K, 4097, 65, False, TC), (S.Q4_K, 4096, 65, False, MMA),
    (S.Q4_K, 4096, 80, False, MMA), (S.Q4_K, 4096, 81, False, TC), (S.Q4_K, 4096, 65, True, MMA), (S.Q4_K, 4100, 65, True, TC),
    (S.Q6_K, 512, 32, False, MMA), (S.Q6_K, 512, 33, False, TC)])
def test_route_of_a_batch(E, wtype, N, M, pair, route):
    """The engine's own choice on both sides of every line is the kernel whose bits it leaves; all kernels agree up to the order of sums."""
    rng = np.random.default_rng(N + M)
    w, b = (_matrix(E, wtype, 1024, N, rng)[0] for _ in range(2))
    x, out = torch.from_numpy(rng.standard_normal((M, 1024)).astype(np.float32)).cuda(), {}
    for r in (-1, DP4A, TC) + ((MMA,) if M <= (80 if wtype == S.Q4_K else 32) else ()):
        out[r] = torch.full((M, N), float("nan"), device="cuda")
        E.op_project_rows(w, x, out[r], M, route=r, b=b if pair else None)
    for r in out:
        assert torch.equal(out[r], out[-1]) == (r in (-1, route)), r
        assert _rel(out[r].cpu().numpy(), out[DP4A].cpu().numpy()) < SAME_INT8
    w.free()
    b.free()


# Rounding errors of fp32 sums of exact products grow with the kernel's order of additions alone: dp4a adds a row's blocks as a
# tree, the tensor-core kernels one by one, which measures up to 1.17 times dp4a's error (Q4_K, 11 008 inputs 1.02; the int8
# kernel for chunks before them: 1.05 to 1.17).  The rest is the spread of a sample of a few thousand results.
PRECISION = 1.25


@pytest.mark.parametrize("wtype", [S.Q4_K, S.Q6_K], ids=["q4", "q6"])
@pytest.mark.parametrize("K", [768, 2048, 11008])
def test_small_batches_are_as_precise_as_dp4a(E, wtype, K):
    """Error of k_gemm_mma against float64 sums of the same int8 activations, against dp4a's."""
    rng = np.random.default_rng(K)
    w, exact = _matrix(E, wtype, K, 200, rng)
    for M in (16, 32, 77) if wtype == S.Q4_K else (16, 32):
        x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
        dp4a, mma = _errors(E, w, exact, x, (DP4A, MMA))
        assert mma < PRECISION * dp4a, (M, dp4a, mma)
    w.free()


@pytest.mark.parametrize("wtype", [S.Q4_K, S.Q6_K], ids=["q4", "q6"])
@pytest.mark.parametrize("K,N,M", [(768, 200, 81), (2048, 500, 128), (2048, 500, 300), (11008, 500, 100), (11008, 1536, 1300)])
def test_larger_batches_are_as_precise_as_dp4a(E, wtype, K, N, M):
    """Error of k_gemm_tc against float64 sums of the same int8 activations, against dp4a's.  Also with blocks of the input spread
    over five decades and weights that make up for it, so that small groups count as much as the token's largest; the last shape
    has so many tiles that nothing but the length of a row's chain of additions asks for parts of the k range."""
    from taraference_b200 import synth_gpu as G
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K + M)
    for spread in (0, 5):
        f = 10.0 ** (-spread * torch.rand(K // 256, generator=gen, device="cuda")).repeat_interleave(256)
        w32 = torch.randn((N, K), generator=gen, device="cuda") * (0.005 / f)
        raw = torch.empty(N * K // 256 * S.BLOCK_BYTES[wtype], dtype=torch.uint8, device="cuda")
        E.synth_quantize(wtype, w32, raw)
        raw = raw.cpu().numpy()
        exact = torch.from_numpy((_q4_k_exact if wtype == S.Q4_K else _q6_k_exact)(raw, K, N)).cuda()
        w = E.GpuMat(wtype, K, N, raw)
        dp4a, tc = _errors(E, w, exact, torch.randn((M, K), generator=gen, device="cuda") * f, (DP4A, TC))
        assert tc < PRECISION * dp4a, (spread, dp4a, tc)
        w.free()


@pytest.mark.parametrize("wtype,K,N,M", [(S.Q4_K, 512, 20000, 300), (S.Q4_K, 7680, 3000, 1000), (S.Q6_K, 7680, 3000, 1000), (S.Q6_K, 27648, 5120, 500),
                                         (S.Q4_K, 27648, 97, 66), (S.Q6_K, 2048, 2048, 65)])
def test_larger_batches_beyond_one_tile_a_cta(E, wtype, K, N, M):
    """k_gemm_tc where a CTA works on several tiles, where a row's chain of additions is cut and its pieces wait in memory (in one
    part, and in two), in tiles of 64 rows: against dp4a on the same int8 activations."""
    from taraference_b200 import synth_gpu as G
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K + N)
    w = E.GpuMat(wtype, K, N, G.quantized_matrix(wtype, K, N, gen, 0.02))
    x, res = torch.randn((M, K), generator=gen, device="cuda"), torch.randn((M, N), generator=gen, device="cuda")
    outs = [res.clone(), res.clone()]
    for route, out in zip((DP4A, TC), outs):
        E.op_project_rows(w, x, out, M, route=route, use_res=2)
    assert _rel(outs[1].cpu().numpy(), outs[0].cpu().numpy()) < SAME_INT8
    w.free()


@pytest.mark.parametrize("wtype", [S.Q4_K, S.Q6_K], ids=["q4", "q6"])
@pytest.mark.parametrize("K,N,M", [(20736, 888, 1792), (27648, 885, 1790)])
def test_larger_batches_whose_chains_have_middle_pieces(E, wtype, K, N, M):
    """81 and 108 blocks a row on 10 x 14 tiles of 96 rows x 128 tokens, which is one round of CTAs with the k range in one part: chains of
    additions in three and four pieces, whose middle ones read parked sums and park again.  Error against float64, against dp4a's."""
    rng = np.random.default_rng(K)
    w, exact = _matrix(E, wtype, K, N, rng)
    x = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).cuda()
    dp4a, tc = _errors(E, w, exact, x, (DP4A, TC))
    assert tc < PRECISION * dp4a, (dp4a, tc)
    w.free()


@pytest.mark.parametrize("K,N,M", [(512, 11008, 300), (512, 5003, 300), (256, 3600, 640)])
def test_gate_up_pairs_beyond_one_tile_a_cta(E, K, N, M):
    """Interleaved pairs where a CTA works on several tiles: whole tiles that leave from the registers, a last tile with rows that do not
    exist, outputs that are no multiple of four.  All values against dp4a on the same int8 activations.  The bound of the sums holds
    for their product: an error e of both branches moves it by at most (1.1 |up| + |gate|) e, which at the largest value, a few rms in
    either branch, is below e times that value."""
    from taraference_b200 import synth_gpu as G
    gen = torch.Generator(device="cuda")
    gen.manual_seed(K + N)
    w, b = (E.GpuMat(S.Q4_K, K, N, G.quantized_matrix(S.Q4_K, K, N, gen, 0.04)) for _ in range(2))
    x, outs = torch.randn((M, K), generator=gen, device="cuda"), []
    for route in (DP4A, TC):
        outs.append(torch.full((M, N), float("nan"), device="cuda"))
        E.op_project_rows(w, x, outs[-1], M, route=route, b=b)
    assert _rel(outs[1].cpu().numpy(), outs[0].cpu().numpy()) < SAME_INT8
    w.free()
    b.free()


def test_q_and_k_rows_beyond_one_tile_a_cta(E, monkeypatch):
    """A matrix that follows another in one launch (K rows behind Q rows) where a CTA works on several tiles of both: 43 + 6 row tiles x 5
    token tiles.  K rows of all tokens against the dp4a route's, up to f16 steps; the second layer's, which depend on the first
    one's Q rows of every token, up to what a flipped rounding moves."""
    cfg = dict(ODD, n_layer=2, n_embd=512, n_head=32, n_kv=4, n_ff=1024, n_vocab=2000)
    m, n = E.CudaModel.load_with(cfg, S.make_dense_model(cfg, seed=37)), 640
    prompt = [int(t) for t in np.random.default_rng(3).integers(0, cfg["n_vocab"], n)]
    out = []
    for dp4a in (True, False):
        (monkeypatch.setenv if dp4a else monkeypatch.delenv)(*(("TFR_GEMM_DP4A", "1") if dp4a else ("TFR_GEMM_DP4A",)))
        kv = m.alloc_kv(n + 8)
        m.forward_greedy(prompt, kv)
        out.append([m.debug_read("k", n * 512, np.uint16, kv=kv, layer=i).view(np.float16).astype(np.float32) for i in range(2)])
        kv.free()
    (a0, a1), (b0, b1) = out
    assert _rel(b0, a0) < 5e-4
    assert _rel(b1, a1) < 2 * TF_WORST
    m.destroy()


@pytest.mark.parametrize("chunk,n", [(2, 7), (16, 16), (16, 45), (64, 19), (2048, 41)])
def test_hybrid_prompt_in_batches_equals_step_by_step(E, chunk, n):
    """Batches of a hybrid model: conv history across batches (shorter ones than the kernel, too), scan tiles of 16 tokens,
    gated attention; then decode steps that continue from the state a batch left."""
    cfg = S.TINY_HYBRID
    m = E.CudaModel.load_with(cfg, S.make_model(cfg, seed=5))
    prompt = [int(t) for t in np.random.default_rng(n).integers(0, cfg["n_vocab"], n)]
    logits = []
    for tokens in (0, chunk):
        m.set_prefill_chunk(tokens)
        kv = m.alloc_kv(96)
        m.forward_greedy(prompt[:3], kv)
        m.forward_greedy(prompt, kv)
        row = [m.current_logits()]
        for t in prompt[:3]:
            m.forward_greedy([t], kv)
            row.append(m.current_logits())
        logits.append(row)
        kv.free()
    rels = [_rel(b, a) for a, b in zip(*logits)]
    assert max(rels) < cfg["n_layer"] * TF_WORST, rels
    m.destroy()


def _mixed_types(cfg, seed):
    """The tensor mix of real hybrid files: of a linear layer's four projections one is Q8_0 (from Q5_K) and three are Q4_K, so
    that they stay four matrices; attn_output is Q8_0."""
    tens, rng = S.make_model(cfg, seed=seed), np.random.default_rng(seed)
    for name, t in list(tens.items()):
        if name.endswith(("attn_qkv.weight", "ssm_out.weight")):
            tens[name] = (S.Q5_K, *t[1:3], S.random_q5_k(rng, t[2] * (t[1] // 256), d_sigma=0.0015).reshape(-1))
        elif name.endswith("attn_output.weight"):
            tens[name] = (S.Q8_0, *t[1:3], S.quantize_q8_0(rng.normal(0, 0.02, (t[2], t[1])).astype(np.float32)).reshape(-1))
    return tens


def _recurrent_state(m, kv, cfg):
    return [m.debug_read("ssm_state", cfg["ssm_n_v"] * 128 * 128, kv=kv, layer=i) for i in range(cfg["n_layer"]) if S.is_linear_layer(cfg, i)]


@pytest.mark.parametrize("mixed", [False, True], ids=["q4", "mixed"])
@pytest.mark.parametrize("n", [2, 9, 16, 23])
def test_hybrid_verification_in_one_pass(E, n, mixed):
    """forward_greedy_all of a hybrid model as batches (its default) against one decode step per token: the greedy token after every
    position wherever the step's margin is above what a flip moves, the logits, the recurrent state, and a step that continues
    from it.  23 tokens take two passes."""
    cfg = S.TINY_HYBRID
    m = E.CudaModel.load_with(cfg, _mixed_types(cfg, 6) if mixed else S.make_model(cfg, seed=6))
    toks = [int(t) for t in np.random.default_rng(n).integers(0, cfg["n_vocab"], n)]
    m.set_prefill_chunk(0)
    kv = m.alloc_kv(64)
    m.forward_greedy([1, 2, 3], kv)
    want, margins = [], []
    for t in toks:
        want.append(m.forward_greedy([t], kv))
        top = np.sort(m.current_logits())[-2:]
        margins.append(float(top[1] - top[0]))
    a = [m.current_logits(), *_recurrent_state(m, kv, cfg)]
    m.forward_greedy([4], kv)
    a.append(m.current_logits())
    kv.free()
    m.set_prefill_chunk(64)
    kv = m.alloc_kv(64)
    m.forward_greedy([1, 2, 3], kv)
    launches = m.launch_count()
    got = m.forward_greedy_all(toks, kv)
    launches = m.launch_count() - launches
    assert kv.len == 3 + n
    b = [m.current_logits(), *_recurrent_state(m, kv, cfg)]
    m.forward_greedy([4], kv)
    b.append(m.current_logits())
    assert launches < n * 10 * cfg["n_layer"] or n == 2, launches  # a pass over the layers, not one for every token
    scale = float(np.abs(a[0]).max())
    assert margin_gated_equal(list(got), want, margins, gate=cfg["n_layer"] * TF_WORST * scale)
    rels = [_rel(y, x) for x, y in zip(a, b)]
    assert max(rels) < cfg["n_layer"] * TF_WORST, rels
    kv.free()
    m.destroy()


@pytest.mark.parametrize("n", [3, 7, 40, 100])
def test_hybrid_prompt_of_mixed_types_equals_step_by_step(E, n):
    """Four projections of different types in a batch: Q8_0 ones on dp4a beside Q4_K ones on mma.sync and tcgen05."""
    cfg = S.TINY_HYBRID
    m = E.CudaModel.load_with(cfg, _mixed_types(cfg, 7))
    prompt = [int(t) for t in np.random.default_rng(n).integers(0, cfg["n_vocab"], n)]
    out = []
    for tokens in (0, 2048):
        m.set_prefill_chunk(tokens)
        kv = m.alloc_kv(128)
        m.forward_greedy(prompt, kv)
        out.append([m.current_logits(), *_recurrent_state(m, kv, cfg)])
        kv.free()
    rels = [_rel(y, x) for x, y in zip(*out)]
    assert max(rels) < cfg["n_layer"] * TF_WORST, rels
    m.destroy()


def test_prefill_chunk_of_a_hybrid_model(E):
    """tfr_prefill_chunk reports the batches of models whose layers take all tokens at once and 0 for hybrid models (callers rely on
    it), whose prompts go through in batches all the same: far fewer launches than with batches switched off."""
    cfg = S.TINY_HYBRID
    m = E.CudaModel.load_with(cfg, S.make_model(cfg, seed=2))
    launches = []
    for tokens in (0, 64):
        m.set_prefill_chunk(tokens)
        assert m.prefill_chunk() == 0
        kv = m.alloc_kv(64)
        before = m.launch_count()
        m.forward_greedy([int(t) for t in np.random.default_rng(1).integers(0, cfg["n_vocab"], 48)], kv)
        launches.append(m.launch_count() - before)
        kv.free()
    assert launches[1] < launches[0] / 5, launches
    m.destroy()
