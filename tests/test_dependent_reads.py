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


# A bounded wait that depends on what the preceding kernel writes may only start once that kernel is complete: its limit counts
# polls, and would otherwise run while the predecessor does.  Per wait: the file, the text that begins the warp role it is in,
# the wait.  (The others of these kernels' waits follow one of these, or griddepcontrol.wait of the whole block.)
BOUNDED = [
    ("paged_decode_fp8_items.cuh", "if (warp == 0) {", "alive = wait_one(item_free"),
    ("paged_decode_fp8_items.cuh", "} else if (warp == 1) {", "test(item_full"),
    ("paged_decode_fp8_items.cuh", "if (use > 0) {", "alive = alive && wait_one(empty"),
    ("paged_decode_fp8_umma.cuh", "if (use > 0) {", "mbar_wait(empty + slot"),
    ("paged_decode_fp8_umma.cuh", "if (warp != 0) {", "mbar_try_wait(s_free"),
    ("fp8_gemm_pair.cuh", "if (warp == 0) {", "mbar_wait(empty + s"),
    ("fp8_gemm_pair.cuh", "} else if (warp == 1) {", "mbar_wait_cluster(acc_empty"),
    ("fp8_gemm_tc.cuh", "} else if (warp == 1) {", "mbar_wait(full + s, ph, 2)"),
    ("fp8_layer_block.cuh", "if (stage == 0) {", "alive = slot_free(it + i);"),
    ("fp8_layer_block.cuh", "} else if (warp == 1) {", "mbar_wait(acc_free"),
]


def test_bounded_waits_start_after_the_dependency_wait():
    bad = []
    for name, role, wait in BOUNDED:
        text = dict(code())[name]
        at, end = -1, -1
        while True:  # the role's text: from its last beginning ahead of the wait up to the wait
            begin = text.find(role, at + 1)
            if begin < 0 or (end > 0 and begin > end):
                break
            at, end = begin, text.find(wait, begin)
        assert at < 0 or end > 0, (name, wait)
        if at < 0 or not re.search(r"pdl_wait\(\)|send_q\(\)", text[at:end]):
            bad.append(f"{name}: {wait}")
    assert not bad, bad
