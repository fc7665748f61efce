"""What the kernels' sources keep to where neither the compiler nor a run would show a breach.

A kernel that waits for the kernel before it (`pdl_wait`, `pdl_prologue`) may declare `__restrict__` only for memory that no earlier
kernel of the stream can have written, or that the kernel itself only writes: reads through any other such pointer could be made
ahead of the wait (csrc/common.cuh, at `pdl_wait`)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "x0ne_engine_b200", "csrc")
WEIGHTS = {"w", "W", "w_d", "w0", "u", "mu", "weight", "bias", "bias_d", "norm_q", "norm_k", "norm_w", "correction", "lambda", "step", "table", "rope_table",
           "freq", "inv_freq"}
TABLES = {"rows", "tokens", "row_slot", "row_pos", "seq_first_row", "seq_slot", "seq_pos0", "tile_seq", "tile_row0"}
WRITTEN_ONLY = {"out", "q_out", "cq_out", "Y", "C", "o", "xs", "mixes", "coef", "gates", "chosen", "weights", "sgate", "resid"}


def kernels(text):
    """(name, parameters, body) of every __global__ function of a source."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        start = text.index("{", m.start())
        head = text[m.start():start]
        depth, close = 0, head.rindex(")")
        for k in range(close, -1, -1):
            depth += (head[k] == ")") - (head[k] == "(")
            if depth == 0:
                break
        depth = 0
        for end in range(start, len(text)):
            depth += (text[end] == "{") - (text[end] == "}")
            if depth == 0:
                break
        yield re.search(r"(\w+)\s*$", head[:k]).group(1), [re.sub(r"\s+", " ", p).strip() for p in head[k + 1:close].split(",")], text[start:end]


def breaches(text):
    found = []
    for name, params, body in kernels(text):
        if "pdl_wait()" not in body and "pdl_prologue()" not in body:
            continue
        for p in params:
            if "__restrict__" not in p:
                continue
            var = p.split()[-1].lstrip("*")
            if p.startswith("const "):
                ok = var in WEIGHTS or var in TABLES
            else:
                # (a pointer that is written only: every mention is a store's address or the start of one)
                ok = var in WRITTEN_ONLY and not re.search(r"\bload\w*\(\s*%s\b" % var, body) and not re.search(r"[^=!<>]=\s*(to_f32\()?%s\[" % var, body)
            if not ok:
                found.append("%s: %s" % (name, p))
    return found


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_only_weights_tables_and_results_are_restrict_behind_the_wait(path):
    with open(path) as f:
        assert breaches(f.read()) == []


def test_the_check_sees_breaches():
    src = "__global__ void %s(const float* __restrict__ w, const float* __restrict__ x, float* __restrict__ out) { pdl_prologue(); out[0] = w[0] * x[0]; }"
    assert breaches(src % "k") == ["k: const float* __restrict__ x"]
    assert breaches((src % "k").replace("pdl_prologue();", "")) == []
    assert breaches("__global__ void k(float* __restrict__ resid) { pdl_wait(); float v = resid[0]; }") == ["k: float* __restrict__ resid"]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*tcgen05.cu"))), ids=os.path.basename)
def test_kernels_let_their_successors_start_only_with_their_tensor_memory_in_hand(path):
    """A block that waits for tensor memory which a block of its successor holds, while that one waits for it, waits for good."""
    with open(path) as f:
        own = [(name, body) for name, _, body in kernels(f.read()) if "tcgen05.alloc" in body]
    assert own
    for name, body in own:
        assert re.search(r"tcgen05\.alloc.*__syncthreads\(\);.*pdl_launch_dependents\(\);", body, re.S), name
        assert "pdl_launch_dependents" not in body[:body.index("tcgen05.alloc")], name


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_rules_ask_the_device_for_its_multiprocessors(path):
    with open(path) as f:
        assert not re.search(r"\b148\b", re.sub(r"//[^\n]*", "", f.read()))


def defined(source, name):
    """The whole number that a source defines `name` as, through other names of the same source."""
    with open(os.path.join(CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    value = re.search(rf"#define\s+{name}\s+(.+)", text).group(1)
    return eval(re.sub(r"[A-Z][A-Z0-9_]*", lambda m: str(defined(source, m.group(0))), value))


def test_sizes_that_python_repeats_are_the_kernels():
    from x0ne_engine_b200.csrc import ops
    assert ops.F32_SPLIT_K == defined("gemm_f32.cu", "F32_SPLIT_K")
    assert (ops.WKV_CHUNK, ops.WKV_CHUNK_UNIT) == (defined("wkv_chunk.cu", "WC_L"), defined("wkv_chunk.cu", "WC_UNIT"))
    assert ops.MOE_TC_TILE_ROWS == defined("moe_tcgen05.cu", "MT_BM")
