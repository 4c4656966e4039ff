"""What a kernel of the chain reads of its predecessors' output goes through plain loads.

A read-only load (__ldg) and a load through a __restrict__ argument that the kernel does not write may be moved ahead of
griddepcontrol.wait, where the predecessor may still be writing.  Only weights and tables, which nothing in flight writes,
may be read that way; __restrict__ may also stand on buffers that a kernel only writes."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "rvllm_b200" / "csrc"
WEIGHTS = {"gamma", "weight", "scale"}  # (`scale`: block scales of the block-scaled GEMV's weight)
WRITTEN = {"out", "scales", "output", "out_fp8", "out_scale", "q_fp8", "k_cache", "v_cache", "k_scale", "v_scale", "q_scale"}
# operands of read-only loads: norm gains, RoPE tables, block-scaled weights and their scales, embedding rows, the helper itself
READ_ONLY = re.compile(r"\b(gamma|rk\.cos_t|rk\.sin_t|w_row|srow|p)\b|^reinterpret_cast<const uint4\*>\(src\) \+ v$")


def code():
    for f in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh"))):
        yield f.name, re.sub(r"//[^\n]*", "", f.read_text())


def argument(text, at):
    """The parenthesised text that begins at text[at] == '('."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError("unbalanced")


def test_restrict_only_on_weights_and_pure_outputs():
    bad = []
    for name, text in code():
        for m in re.finditer(r"(const\s+)?[\w:<> ]+\*\s*__restrict__\s+(\w+)", text):
            const, arg = bool(re.search(r"\bconst\b", m.group(0))), m.group(2)
            if arg not in (WEIGHTS if const else WRITTEN):
                bad.append(f"{name}: {' '.join(m.group(0).split())}")
    assert not bad, bad


def test_read_only_loads_touch_weights_only():
    bad = []
    for name, text in code():
        for m in re.finditer(r"\b(__ldg|ldg128)\(", text):
            arg = argument(text, m.end() - 1)
            if arg == "const void* p":  # the helper's own declaration
                continue
            if name == "common.cuh" and arg == "reinterpret_cast<const uint4*>(p)":
                continue
            if arg == "reinterpret_cast<const uint4*>(src) + v" and name != "rope_kv_write.cu":
                bad.append(f"{name}: {arg}")
            elif not READ_ONLY.search(arg) or re.search(r"\bp\.", arg):
                bad.append(f"{name}: {arg}")
    assert not bad, bad
