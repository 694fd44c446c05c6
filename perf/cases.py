"""What a user of this framework has it do, as measurable cases.

A program loads one model, keeps it, opens a KV cache per conversation and then feeds prompts, decodes bursts of greedy
tokens, fetches single tokens (and their logits, to sample on the host) or verifies drafted tokens.  Every state here is
one conversation: a KV cache of its own on the model that all conversations of a process share, with a prompt drawn from
the seed.  A few cases call the stand-alone operators with device tensors instead.

Weights are N(0, sigma) in the repository's Q4_K_M mix, sigma as in the benchmark at its width (0.02 at 2 048 inputs) and
falling with the square root of the inputs.  Two things about them follow trained models instead of a bare initialisation,
because results have to be comparable: the two projections that write to the residual stream are scaled with the depth,
and the head is the embedding with its rows moved, so that every token has one likely successor and the greedy choice does
not hang on the rounding of an activation to int8.
"""
import functools
import math

import numpy as np
import torch

from taraference_b200 import engine as E
from taraference_b200 import synth as S
from taraference_b200 import synth_gpu as G

# shape -> (configuration, layers).  Where the layers are fewer than the configuration's, the case is about the width.
SHAPES = {
    "tiny": (S.TINY_DENSE, 2),
    "3b": (S.QWEN25_3B, 36),
    "3b-12": (S.QWEN25_3B, 12),
    "32b-8": (S.QWEN25_32B, 8),
    "4b-hybrid": (S.QWEN35_4B, 32),
}
SIGMA_EMBD = 2.0


def _sigma(K):
    return 0.02 * math.sqrt(2048 / K)


def listed():
    return [
        # the smallest call there is: one token of a very small model, launches and host work only
        {"name": "token-tiny", "kind": "token", "shape": "tiny", "past": 20, "ctx": 256},
        # a host that samples by itself: one token, then its logits
        {"name": "token-3b", "kind": "token", "shape": "3b", "past": 500, "ctx": 4096},
        # the ordinary answer to a short prompt (the benchmark's default workload, fewer tokens)
        {"name": "burst-3b", "kind": "burst", "shape": "3b", "past": 32, "n": 64, "ctx": 4096},
        # an answer about a long document: attention over an odd number of keys near 16 K
        {"name": "burst-3b-long", "kind": "burst", "shape": "3b-12", "past": 16001, "n": 32, "ctx": 32768},
        # the widest layers the framework is used with
        {"name": "burst-32b", "kind": "burst", "shape": "32b-8", "past": 128, "n": 32, "ctx": 4096},
        # reading a long prompt
        {"name": "prompt-3b-2048", "kind": "prompt", "shape": "3b", "past": 0, "n": 2048, "ctx": 4096},
        # a question of a few lines, ragged against every tile
        {"name": "prompt-3b-77", "kind": "prompt", "shape": "3b", "past": 0, "n": 77, "ctx": 4096},
        # a page more for a conversation that has one already, on wide layers
        {"name": "prompt-32b-500", "kind": "prompt", "shape": "32b-8", "past": 301, "n": 500, "ctx": 4096},
        # speculative decoding: nine drafted tokens checked in one pass
        {"name": "verify-3b-9", "kind": "verify", "shape": "3b", "past": 300, "n": 9, "ctx": 4096},
        # a whole turn of the hybrid model: prompt and answer, recurrent layers included
        {"name": "turn-4b-hybrid", "kind": "turn", "shape": "4b-hybrid", "prompt": 64, "n": 32, "ctx": 4096},
        # the feed-forward block as an operator
        {"name": "ffn-3b", "kind": "ffn", "K": 2048, "FF": 11008, "host": False},
        # attention over a long cache as an operator
        {"name": "attention-16896", "kind": "attention", "n_head": 16, "n_kv": 2, "head_dim": 128, "keys": 16896, "gated": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "burst", "burst", "prompt", "prompt", "verify", "turn", "ffn", "attention"])
    if kind == "ffn":
        return {"kind": kind, "K": 256 * _log(rng, 2, 20), "FF": 256 * _log(rng, 4, 108), "host": rng.random() < 0.3}
    if kind == "attention":
        n_kv = rng.choice([1, 2, 4, 8])
        hd = rng.choice([64, 128, 256])
        return {"kind": kind, "n_head": n_kv * rng.choice([2, 4, 5, 8]) if hd < 256 else n_kv * 4, "n_kv": n_kv, "head_dim": hd,
                "keys": _log(rng, 17, 32768), "gated": rng.random() < 0.3}
    if kind == "turn":
        return {"kind": kind, "shape": "4b-hybrid", "prompt": _log(rng, 3, 100), "n": _log(rng, 4, 64), "ctx": 4096}
    shape = rng.choice(["3b", "3b", "32b-8", "3b-12"] + (["tiny"] if kind == "token" else []))
    past = _log(rng, 2, 200 if shape == "tiny" else 3000)
    case = {"kind": kind, "shape": shape, "past": past, "ctx": 256 if shape == "tiny" else 4096}
    if kind == "burst":
        case["n"] = _log(rng, 4, 100)
    elif kind == "prompt":
        case["past"] = rng.choice([0, 0, past // 4])
        case["n"] = _log(rng, 6, 1900 if shape == "3b" else 1000)
    elif kind == "verify":
        case["n"] = rng.randint(3, 24)
    return case


# ------------------------------------------------------------------ models and conversations

class _Model:
    def __init__(self, shape):
        base, layers = SHAPES[shape]
        self.cfg = cfg = dict(base, n_layer=layers, tied=False)
        gen = torch.Generator(device="cuda")
        gen.manual_seed(11)
        self.m = m = E.CudaModel(torch.cuda.current_device())
        m.set_config(cfg, 4096)
        for name, t, K, N in S.tensor_plan(cfg):
            if name == "output.weight":
                continue  # made from the embedding below
            residual = name.endswith(("attn_output.weight", "ffn_down.weight", "ssm_out.weight"))
            sigma = SIGMA_EMBD if name == "token_embd.weight" else _sigma(K) / (math.sqrt(2 * layers) if residual else 1)
            q = G.quantized_matrix(t, K, N, gen, sigma)
            m.upload_tensor(name, t, K, N, q)
            if name == "token_embd.weight":
                self.successor = torch.randperm(N, generator=gen, device="cuda")
                head = torch.empty_like(q).view(N, -1)
                head[self.successor] = q.view(N, -1)  # the row that scores successor[i] is the embedding of i
                torch.cuda.synchronize()
                m.upload_tensor("output.weight", t, K, N, head.view(-1))
        rng = np.random.default_rng(11)
        for name, n, kind in S.vector_plan(cfg):
            v = S.make_vector(kind, n, rng, 0.02)
            m.upload_tensor(name, E.TYPE_F32, n, 1, v)
        m.finalize_load()


@functools.lru_cache(maxsize=None)
def _model(shape):
    return _Model(shape)


class _Conversation:
    """A KV cache on a shared model, with what the next pass feeds."""

    def __init__(self, case, seed):
        self.model = _model(case["shape"])
        self.kv = self.model.m.alloc_kv(case["ctx"])
        rng = np.random.default_rng(seed)
        tokens = lambda n: rng.integers(0, self.model.cfg["n_vocab"], n).astype(np.uint32)
        kind, m = case["kind"], self.model.m
        self.past, self.n = case.get("past", 0), case.get("n", 1)
        if self.past:
            self.first = m.forward_greedy(tokens(self.past), self.kv)
        self.feed = tokens(case["prompt"] if kind == "turn" else self.n)

    def __del__(self):
        self.kv.free()


class _Mats:
    def __init__(self, K, FF, gen):
        make = lambda t, k, n: E.GpuMat(t, k, n, G.quantized_matrix(t, k, n, gen, _sigma(k)))
        self.gate, self.up, self.down = make(S.Q4_K, K, FF), make(S.Q4_K, K, FF), make(S.Q6_K, FF, K)

    def __del__(self):
        for m in (self.gate, self.up, self.down):
            m.free()


def prepare(case, seed):
    kind = case["kind"]
    if kind not in ("ffn", "attention"):
        return {"kind": kind, "c": _Conversation(case, seed)}
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    randn = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    if kind == "ffn":
        x = randn(case["K"])
        s = {"kind": kind, "host": case["host"], "w": _Mats(case["K"], case["FF"], gen), "x": x,
             "h": torch.empty(case["FF"], device="cuda"), "y": torch.empty(case["K"], device="cuda")}
        if case["host"]:
            s["x"], s["y"] = x.cpu().numpy(), np.empty(case["K"], np.float32)
        return s
    H, Hkv, hd, T = case["n_head"], case["n_kv"], case["head_dim"], case["keys"]
    return {"kind": kind, "shape": (H, Hkv, hd, T - 1), "q": randn(H * hd), "k": randn(T, Hkv * hd).half(), "v": randn(T, Hkv * hd).half(),
            "gate": randn(H * hd) if case["gated"] else None, "out": torch.empty(H * hd, device="cuda")}


# ------------------------------------------------------------------ one pass

def run(s):
    kind = s["kind"]
    if kind == "ffn":
        w = s["w"]
        if s["host"]:
            E.ffn_block_host(w.gate, w.up, w.down, s["x"], s["y"])
        else:
            E.op_ffn_block(w.gate, w.up, w.down, s["x"], s["h"], s["y"])
        return s["y"]
    if kind == "attention":
        if s["gate"] is None:
            E.op_attention(s["q"], s["k"], s["v"], s["out"], *s["shape"])
        else:
            E.op_attention_gated(s["q"], s["k"], s["v"], s["gate"], s["out"], *s["shape"])
        return s["out"]
    c = s["c"]
    m, kv = c.model.m, c.kv
    kv.len = c.past
    if kind == "verify":
        tokens = m.forward_greedy_all(c.feed, kv)
    elif kind == "burst":
        tokens = m.decode_burst(c.first, c.n, kv)
    else:  # token, prompt, turn
        if kind == "turn":
            m.zero_recurrent(kv)
        first = m.forward_greedy([c.first] if kind == "token" else c.feed, kv)
        tokens = [first]
        if kind == "turn":
            tokens = np.concatenate([tokens, m.decode_burst(first, c.n, kv)])
    return {"tokens": np.asarray(tokens, np.int64), "logits": m.current_logits()}


# ------------------------------------------------------------------ what a pass cannot do without

def _sizes(cfg):
    """(bytes, weights) of the layers, and of the head."""
    layer_b = layer_n = 0
    for name, t, K, N in S.tensor_plan(cfg):
        if name not in ("token_embd.weight", "output.weight"):
            layer_b += N * (K // 256) * S.BLOCK_BYTES[t]
            layer_n += N * K
    head_n = cfg["n_vocab"] * cfg["n_embd"]
    return layer_b, layer_n, head_n // 256 * S.BLOCK_BYTES[S.Q6_K], head_n


def work(case):
    kind = case["kind"]
    if kind == "ffn":
        K, FF = case["K"], case["FF"]
        return {"bytes": 2 * FF * K // 256 * 144 + K * FF // 256 * 210 + 8 * K, "flops": 6 * K * FF}
    if kind == "attention":
        H, Hkv, hd, T = case["n_head"], case["n_kv"], case["head_dim"], case["keys"]
        return {"bytes": 4 * T * Hkv * hd + 4 * H * hd * (3 if case["gated"] else 2), "flops": 4 * H * hd * T}
    base, layers = SHAPES[case["shape"]]
    cfg = dict(base, n_layer=layers, tied=False)
    layer_b, layer_n, head_b, head_n = _sizes(cfg)
    kv_b = G.kv_bytes_per_position(cfg)
    state_b = G.recurrent_state_bytes(cfg)
    full = sum(1 for i in range(layers) if not S.is_linear_layer(cfg, i))
    att = 4 * cfg["n_head"] * cfg["head_dim"] * full  # operations of one query token and one key
    past, n, out_b = case.get("past", 0), case.get("n", 1), 4 * cfg["n_vocab"]

    def block(p, k, heads):  # k tokens behind p positions in one pass over the weights
        return (layer_b + head_b + kv_b * (p + k) + state_b, 2 * (layer_n * k + head_n * heads) + att * (k * p + k * (k + 1) // 2))

    if kind == "token":
        parts = [block(past, 1, 1)]
    elif kind == "prompt":
        parts = [block(past, n, 1)]
    elif kind == "verify":
        parts = [block(past, n, n)]
    else:
        parts = [block(0, case["prompt"], 1)] if kind == "turn" else []
        p = past + case.get("prompt", 0)
        parts += [block(p + i, 1, 1) for i in range(n)]
    return {"bytes": sum(b for b, _ in parts) + out_b, "flops": sum(f for _, f in parts)}


def tolerance(case):
    if case["kind"] == "attention":
        return {"rel": 1e-5}
    if case["kind"] == "ffn":
        return {"rel": 1e-3}  # the product of the two branches is rounded to int8: a value on the border may fall either way
    # Every projection rounds its input to int8: sums in another order move a few values across a rounding border in
    # every layer, and the next layers carry that on.  The tokens' margins are far above it.
    return {"rel": 1e-2, "max": 0.1}
