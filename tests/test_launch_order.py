"""Kernels that are launched while the kernel before them still runs (csrc/cuda/pdl.cuh) read what the step computes only
behind their dependency wait.  Read from the sources: a race does not show on every run."""
import glob
import os
import re

import pytest

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kv-cache-manager_b200", "csrc", "cuda")
# Weights, and the integers of the batch and the keys and values of earlier tokens, which no kernel of a step writes.
CONSTANTS = {"W", "wr", "wgu", "wd", "w", "weight", "wq", "wc", "wb", "wn", "w0", "w1", "mix", "outw", "inw", "lambda",
             "inv_freq", "v_inv_freq", "decay", "positions", "slot_mapping", "rows", "row_seq", "seq_q_start", "seq_q_len",
             "seq_ctx_len", "order", "seq_state_slot", "block_tables", "tile_seq", "tile_q0"}
# Named above the wait: keys below the newest (written by earlier steps), and rows that a lambda copies behind it.
BEHIND_IT = {"attn_decode_kernel": {"k_cache", "v_cache"}, "gemm_f32_kernel": {"X"}}


def _closing(text, at, pair):
    depth = 1
    while depth:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[at], 0)
        at += 1
    return at


def _sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CUDA, "*.cu*"))):
        with open(f) as fh:
            out[os.path.basename(f)] = re.sub(r"//[^\n]*", "", fh.read())
    return out


def _pointer_fields(text):
    """Struct name -> names of its pointers."""
    out = {}
    for m in re.finditer(r"struct\s+(\w+)\s*\{", text):
        body = text[m.end():_closing(text, m.end(), "{}") - 1]
        out[m.group(1)] = set(re.findall(r"\*\s*(\w+)\s*[;,]", body)) | set(re.findall(r"\*\s*(\w+)\[\w+\]\s*;", body))
    return out


def _early_kernels():
    head = re.compile(r"__global__\s+void\s*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(")
    for name, text in _sources().items():
        structs = _pointer_fields(text)
        for m in head.finditer(text):
            end = _closing(text, m.end(), "()")
            start = text.index("{", end) + 1
            body = text[start:_closing(text, start, "{}")]
            launched = re.search(r"pdl_launch(?:_cluster)?\(\(?%s\b" % m.group(1), text)
            if "pdl_launch_dependents" in body or "pdl_wait" in body or launched:
                params = [re.sub(r"\s+", " ", p).strip() for p in text[m.end():end - 1].split(",")]
                yield pytest.param(m.group(1), params, body, structs, id=f"{name}:{m.group(1)}")


EARLY = list(_early_kernels())


def test_the_sources_were_read():
    names = {p.values[0] for p in EARLY}
    assert len(names) > 60 and {"moe_few_down_kernel", "attn_decode_kernel", "gemm_f32_kernel", "sample_kernel"} <= names


@pytest.mark.parametrize("name,params,body,structs", EARLY)
def test_only_constants_are_read_before_the_wait(name, params, body, structs):
    assert "pdl_wait();" in body, "launched early, and never waits"
    before = body[:body.index("pdl_wait();")]
    allowed = CONSTANTS | BEHIND_IT.get(name, set())
    data = []
    for p in params:
        arg = p.split()[-1]
        if "*" in p:
            data += [r"(?<![\w.])%s" % arg] if arg not in allowed else []
        for s in structs:
            if re.search(r"\b%s\b" % s, p):
                data += [r"\b%s\.%s" % (arg, f) for f in structs[s] - allowed]
    for statement in re.split(r"[;{}]", before):
        if re.search(r"\*\s*(const\s+)?\w+\s*=[^=]", statement):
            continue                                        # (an address is formed)
        for d in data:
            assert not re.search(d + r"\s*(\[|,|\+)|\*" + d.replace(r"(?<![\w.])", "") + r"\b", statement), f"before the wait: {statement.strip()}"


# What `__restrict__` may promise of such a kernel: that nothing writes the data while the kernel is there.  It is there before
# the kernel before it has ended, so that holds of the constants alone.
PROMISED = CONSTANTS | {"ids", "prev", "table", "pair", "place", "bias", "conv_w", "a_log", "dt_bias", "skip_coef", "coef", "alpha", "sink",
                        "temperature", "seed", "request_id", "position"}
PROMISED_OF = {"dyt_norm_kernel": {"b"}, "dyt_norm_vec_kernel": {"b"}}
STEP_TABLE = {"rope_cache_table_kernel"}                    # its table of angles is the step's


@pytest.mark.parametrize("name,params,body,structs", EARLY)
def test_restrict_qualifies_constants_and_results_only(name, params, body, structs):
    for p in params:
        arg = p.split()[-1]
        if "__restrict__" not in p:
            continue
        if p.startswith("const "):
            assert arg in (PROMISED - ({"table"} if name in STEP_TABLE else set())) | PROMISED_OF.get(name, set()), p
        else:
            assert not re.search(r"\b%s\[[^;=]*\]\s*[-+*/]=" % arg, body), f"{p}: changed in place"
    assert not re.search(r"const\s+\w+\*\s*__restrict__\s+(qkv|state)\b", body)
