"""Loads of kernels that overlap their predecessor (programmatic stream serialization).

Such a kernel is resident while its predecessor still writes its operands, so the read-only data path
(``__ldg``, or a ``const ... *__restrict__`` parameter, which lets the compiler choose that path) is closed
to them: CUDA allows it for data that is read-only for the kernel's whole life.  Checked on the source,
because a broken promise need not show in a result."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nessi_b200", "csrc")
# uploaded by the host and waited for before the call returns: no kernel writes these
HOST_WRITTEN = {"gt", "probs", "udiag"}


def _source():
    text = ""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                text += fh.read()
    return re.sub(r"//[^\n]*", "", text)


def _functions(text):
    """{name: (parameters, body)} of the __global__ and __device__ functions."""
    out = {}
    for m in re.finditer(r"__(?:global|device)__\s", text):
        i = text.find("(", m.end())
        while i > 0:  # the parameter list: the first (...) followed by a body
            depth, j = 0, i
            while True:
                depth += {"(": 1, ")": -1}.get(text[j], 0)
                j += 1
                if depth == 0:
                    break
            name = re.search(r"(\w+)\s*$", text[m.end():i])
            if re.match(r"\s*(const\s*)?\{", text[j:]):
                break
            if not re.match(r"\s*\w", text[j:]):  # a declaration
                name = None
                break
            i = text.find("(", j)  # __launch_bounds__(...) and the like
        if not name:
            continue
        params, i = text[i:j], text.find("{", j)
        depth, j = 0, i
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                break
        out[name.group(1)] = (params, text[i:j])
    return out


FUNCTIONS = _functions(_source())
CHAINED = sorted(n for n, (_, body) in FUNCTIONS.items() if re.search(r"\bpdl_(wait|entry)\(\)", body) and n.startswith("k_"))


def _reached(name, seen):
    """The device functions that a kernel calls, itself among them."""
    if name in seen:
        return seen
    seen.add(name)
    for callee in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\s*\(", FUNCTIONS[name][1])) & set(FUNCTIONS):
        _reached(callee, seen)
    return seen


def test_the_chained_kernels_are_found():
    assert {"k_prep", "k_mat_operator", "k_zgemm", "k_zgemm_split", "k_zgemm_split1", "k_vol_block", "k_vol_trail",
            "k_vol_trail_split", "k_gloc", "k_gloc_final", "k_sigma_2b", "k_extrapolate"} <= set(CHAINED)


@pytest.mark.parametrize("kernel", CHAINED)
def test_no_read_only_loads_of_data_a_predecessor_writes(kernel):
    for f in _reached(kernel, set()):
        params, body = FUNCTIONS[f]
        assert "__ldg(" not in body and "ld.global.nc" not in body, (kernel, f)
        for p in params.strip("()").split(","):
            if "__restrict__" in p and "const" in p:
                assert re.search(r"(\w+)\s*$", p).group(1) in HOST_WRITTEN, (kernel, f, p.strip())
