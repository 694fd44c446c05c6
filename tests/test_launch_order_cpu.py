"""Kernels of a decode step read the decode state, the recurrent state and earlier cache rows ahead of their dependency wait.  That is
sound only behind a kernel that lets its successor start after its own wait; the launchers ask for such a predecessor (WaitsFirst).
What the type cannot say is held here, on the sources: that the kernels that make one do wait first, and that the readers are launched
with a state through those launchers alone."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "taraference_b200" / "csrc"
ENGINE = (CSRC / "tfr_engine.cu").read_text()
ALL = ENGINE + "".join(p.read_text() for p in sorted(CSRC.glob("*.cuh")))
READERS = ("k_gdn_step", "k_qk_norm_rope_store")


def _body(name):
    """Text of a kernel from its name to the brace that closes it."""
    at = re.search(r"__global__[^;{]*?\b%s\(" % name, ALL).end()
    at = ALL.index("{", at)
    depth = 0
    for i in range(at, len(ALL)):
        depth += {"{": 1, "}": -1}.get(ALL[i], 0)
        if depth == 0:
            return ALL[at:i]
    raise AssertionError(name)


def test_kernels_that_start_their_successor_behind_their_wait():
    makers = set(re.findall(r"WaitsFirst\{launch_pdl\((\w+)", ALL))
    assert {"k_gemv", "k_qk_norm_rope_store"} <= makers
    for name in makers:
        body = _body(name)
        assert 0 <= body.index("griddep_wait()") < body.index("griddep_launch_dependents()"), name
    assert "k_gemm_tc" not in makers


def test_readers_ahead_of_their_wait_follow_such_a_kernel():
    for name in READERS:
        behind = re.search(r"_behind\(WaitsFirst before[^}]*launch_pdl\(%s\b" % name, ENGINE)
        assert behind, name
        for m in re.finditer(r"launch_pdl\(%s\b[^;]*;|%s<<<[^;]*;" % (name, name), ALL):
            assert "nullptr)" in m.group() or behind.start() < m.start() < behind.end(), m.group()
    behind = re.search(r"launch_attention_behind\(WaitsFirst before[^}]*\}", ENGINE)
    calls = [m for m in re.finditer(r"(?<!cudaError_t )\blaunch_attention\([^;{]*;", ENGINE) if not behind.start() < m.start() < behind.end()]
    assert calls and all("nullptr)" in m.group() for m in calls), calls
