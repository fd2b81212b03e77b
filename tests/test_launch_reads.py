"""Kernels that are launched before their predecessor has finished must not
read what it writes through the read-only path: `__ldg`, `ldg_n` and
`const ... __restrict__` parameters promise data that is constant while the
kernel is resident, and the compiler may move such loads ahead of the wait.
Checked on the sources: in those kernels, and in the device functions that they
may call, only the operator's arrays are read that way."""

import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "imate_b200", "csrc")

# written when the operator is built, constant from then on
OPERATOR = {"indptr", "indices", "vals", "gptr", "gcol", "gval", "inv",
            # places in them
            "val"}
# device functions of operator set-up and of kernels launched in stream order
SETUP = {"perm_row", "rcm_start_component", "blk_col_range", "blk_bitmap",
         "ldg_n"}


def _text(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _functions(text):
    """(name, parameters, body) of every device function and kernel."""
    for m in re.finditer(r"\b(?:__global__|__device__)\b[^;{}]*?"
                         r"\b(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


def _early():
    """Kernels launched with launch_pdl, and those launched in stream order."""
    text = _text("slq_engine.cu")
    early = set(re.findall(r"launch_pdl\(\s*L\s*,\s*(k_\w+)", text))
    plain = set(re.findall(r"\b(k_\w+)(?:<[^<>]*>)?\s*<<<", text))
    return early, plain


def test_every_early_kernel_is_found_and_waits():
    early, _ = _early()
    assert {"k_spmm", "k_spmm_rows", "k_spmm_rg", "k_spmm_blk", "k_finalize",
            "k_ql", "k_quad", "k_dots", "k_stream", "k_reorth",
            "k_three_term", "k_dense_tc", "k_dense_epi", "k_dense_split_t",
            "k_probe_parity", "k_probe_starts"} <= early
    found = set()
    for f in ("slq_kernels.cuh", "slq_blk.cuh"):
        for name, _, body in _functions(_text(f)):
            if name in early:
                found.add(name)
                assert "pdl_wait()" in body, name
    assert found == early


@pytest.mark.parametrize("f", ["slq_kernels.cuh", "slq_blk.cuh", "slq_tc.cuh",
                               "slq_ql.cuh"])
def test_only_operator_arrays_are_read_as_constant(f):
    early, plain = _early()
    wrong = []
    for name, params, body in _functions(_text(f)):
        if name in SETUP or (name.startswith("k_") and name not in early):
            continue
        for p in params.split(","):
            if "__restrict__" in p and "const" in p:
                arg = re.findall(r"\w+", p)[-1]
                if arg not in OPERATOR:
                    wrong.append("%s: const __restrict__ %s" % (name, arg))
        for m in re.finditer(r"\b(?:__ldg|ldg_n(?:<[^<>]*>)?)\s*\(\s*"
                             r"(?:reinterpret_cast<[^<>]*>\(\s*)?([\w.]+)",
                             body):
            if m.group(1) not in OPERATOR:
                wrong.append("%s: read-only load of %s" % (name, m.group(1)))
    assert not wrong, "\n".join(wrong)


def test_a_product_of_the_caller_waits_for_the_caller_s_kernels():
    # its predecessor in the stream may be any kernel, one that lets its
    # dependents start early and writes the operator's arrays among them
    text = _text("slq_engine.cu")
    body = text[text.index('extern "C" slq_status slq_operator_dot('):]
    body = body[:body.index("\n}\n")]
    assert body.index("L.early = false") < body.index("op_spmm<")
