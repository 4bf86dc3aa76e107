"""Kernels that may start while the kernel in front of them is running (they execute griddepcontrol.wait) read what it writes.  A
const __restrict__ parameter promises memory that nothing writes meanwhile, and allows the compiler to load from it before the wait:
none of these kernels takes an input that way.  Read off the sources, since a stale read shows itself only now and then."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "landmark_attention_b200", "csrc")
PROMISE = re.compile(r"const\s+[\w:<>\s]*\*\s*(?:const\s+)?__restrict__")


def closing(text, at, pair):
    """Index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def functions(text):
    """name -> (parameters, body) of the kernels of a source."""
    text = re.sub(r"//[^\n]*", "", text)
    found = {}
    for m in re.finditer(r"__global__", text):
        at, params, name = m.end(), None, None
        while text[at] not in "{;":
            if text[at] == "(":
                name = re.search(r"(\w+)\s*$", text[m.end():at]).group(1)
                end = closing(text, at, "()")
                params, at = text[at:end], end
            else:
                at += 1
        if text[at] == "{":
            found[name] = (params, text[at:closing(text, at, "{}")])
    return found


@pytest.mark.parametrize("source,kernels", [("attn_sm100.cu", ("sm100_bwd_dq_kernel", "sm100_bwd_dkv_kernel"))])
def test_waiting_kernels_promise_nothing_about_their_inputs(source, kernels):
    with open(os.path.join(CSRC, source)) as f:
        found = functions(f.read())
    for name in kernels:
        params, body = found[name]
        assert "grid_dep_wait()" in body, name
        assert not PROMISE.search(params), name
