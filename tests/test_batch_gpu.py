"""Token batches at the edges of the batched kernels' tiles: the tensor-core projections against the dp4a ones, the hybrid
layers against the step-by-step route (needs a B200)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from taraference_b200 import synth as S  # noqa: E402
from tests.test_engine_gpu import TF_WORST, _rel  # noqa: E402

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


@pytest.mark.parametrize("cfg", [ODD, WIDE], ids=["odd", "wide"])
@pytest.mark.parametrize("n", [5, 16, 17, 32, 33, 48, 80, 81, 128, 129, 224, 256, 257, 640])
def test_projections_of_batches_at_tile_edges(E, cfg, n, monkeypatch):
    """One layer, all tokens in one batch: 16- and 32-token paddings, mma.sync up to 80 tokens (Q6_K: 32), the tcgen05 forms, several
    token tiles, tiles that end inside a column group.  V rows are the same bits, the logits differ by a flip at most."""
    m = E.CudaModel.load_with(cfg, S.make_dense_model(cfg, seed=31))
    prompt = [int(t) for t in np.random.default_rng(n).integers(0, cfg["n_vocab"], n)]
    out = []
    for dp4a in (True, False):
        (monkeypatch.setenv if dp4a else monkeypatch.delenv)(*(("TFR_GEMM_DP4A", "1") if dp4a else ("TFR_GEMM_DP4A",)))
        kv = m.alloc_kv(n + 8)
        m.forward_greedy(prompt, kv)
        out.append((m.current_logits(), *_state(m, kv, cfg, n)))
        kv.free()
    (la, ka, va), (lb, kb, vb) = out
    assert np.array_equal(va, vb)
    f = lambda a: a.view(np.float16).astype(np.float32)
    assert _rel(f(kb), f(ka)) < 5e-4
    assert _rel(lb, la) < TF_WORST
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
