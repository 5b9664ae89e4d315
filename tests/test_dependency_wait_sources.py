"""Every kernel may start while the kernel before it in the stream still runs, and waits
(``pdl_wait``) before it touches what that kernel writes.  A parameter that is ``__restrict__`` promises
the compiler that nobody else writes there while the kernel runs; it may then read it above the wait.
So only what no kernel of a step writes may be read through one: weights, tables of constants and the
step's integers, which are copied to the device before its first kernel."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "minfer_b200", "csrc")
SOURCES = sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu")))

WEIGHTS = {"W", "w", "wg", "wu", "wd", "w2t", "w0", "bias", "weight", "norm_w", "table", "rows", "row_idx", "vec",
           "coef", "shift", "mu", "lam", "sink_logit", "correction", "inv_freq"}
STEP_INTEGERS = {"positions", "token_row", "seq_end", "cu_seqlens", "slots", "page_table"}
# outputs that the kernel only writes
WRITTEN = {"out", "y", "x_out", "q_out", "k_out", "v_out", "k_cache", "v_cache", "status", "logits", "idx", "wts",
           "hidden", "counts", "offsets", "order", "where"}


def kernels(source):
    """(name, parameters) of every kernel of a file."""
    with open(os.path.join(CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), [" ".join(p.split()) for p in text[m.end():end - 1].split(",")]


def test_the_kernels_are_found():
    names = [name for source in SOURCES for name, _ in kernels(source)]
    assert len(names) > 80 and "rmsnorm_vec_kernel" in names and "splitk_reduce_kernel" in names


@pytest.mark.parametrize("source", SOURCES)
def test_what_a_kernel_of_the_step_writes_is_not_restrict(source):
    bad = []
    for name, parameters in kernels(source):
        for p in parameters:
            if "__restrict__" not in p:
                continue
            allowed = WEIGHTS | STEP_INTEGERS if p.startswith("const ") else WRITTEN
            if p.split()[-1].lstrip("*&") not in allowed:
                bad.append(f"{name}: {p}")
    assert not bad, bad


@pytest.mark.parametrize("source", SOURCES)
def test_no_load_is_marked_read_only(source):
    with open(os.path.join(CSRC, source)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert not re.search(r"\b__ldg\s*\(|ld\.global(\.\w+)*\.nc\b", text)
