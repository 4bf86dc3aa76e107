"""Kernels that may start while the kernel in front of them is running (they execute griddepcontrol.wait) read what it writes.  A
__restrict__ parameter promises memory that nobody else touches meanwhile, and allows the compiler to load from it before the wait, and
so does __ldg: none of these kernels uses them.  And a thread that has read a tile from shared memory lets TMA overwrite it only
behind a fence between the two proxies.  Read off the sources, since either fault shows itself only now and then."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "landmark_attention_b200", "csrc")
PROMISE = re.compile(r"__restrict__|__ldg|ld\.global\.nc")


def closing(text, at, pair):
    """Index behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def functions(text):
    """(kernels, device functions) of a source: name -> [(parameters, body)]."""
    text = re.sub(r"//[^\n]*", "", text)
    kernels, device = {}, {}
    for m in re.finditer(r"__global__|__device__", text):
        at, params, name = m.end(), None, None
        while text[at] not in "{;=":
            if text[at] == "(":
                name = re.search(r"(\w*)\s*$", text[m.end():at]).group(1)       # "": an operator
                end = closing(text, at, "()")
                params, at = text[at:end], end
            else:
                at += 1
        if text[at] == "{" and name:
            kept = kernels if m.group() == "__global__" else device
            kept.setdefault(name, []).append((params, text[at:closing(text, at, "{}")]))
    return kernels, device


def reached(body, device):
    """The device functions of the same source that a body calls, directly or not."""
    names, queue = set(), [body]
    while queue:
        for name in set(re.findall(r"\w+", queue.pop())) & device.keys() - names:
            names.add(name)
            queue += [b for _, b in device[name]]
    return names


def read(source):
    with open(os.path.join(CSRC, source)) as f:
        return f.read()


SHARED = "".join(read(f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cuh", ".h")))
WAITING = [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu") and "grid_dep_wait()" in read(f)]


@pytest.mark.parametrize("source", WAITING)
def test_waiting_kernels_promise_nothing_about_their_inputs(source):
    kernels, device = functions(SHARED + read(source))
    waiting = 0
    for kernel, forms in kernels.items():
        for params, body in forms:
            if "grid_dep_wait()" not in body:
                continue
            waiting += 1
            for name, (p, b) in [(kernel, (params, body)), *[(n, f) for n in reached(body, device) for f in device[n]]]:
                assert not PROMISE.search(p + b), f"{kernel}: {name}"
    assert waiting


def test_every_source_that_launches_before_the_end_is_looked_at():
    launching = [f for f in os.listdir(CSRC) if f.endswith(".cu") and re.search(r"launch_overlapped|ProgrammaticStream", read(f))]
    assert set(launching) <= set(WAITING)


def test_tiles_read_by_threads_are_released_behind_a_proxy_fence():
    (_, body), = functions(read("attn_sm100.cu"))[0]["sm100_bwd_dq_kernel"]
    release = body.index("mbar_arrive(smem_u32(&sm->delta_read))")
    assert body.rindex("fence_proxy_async_smem()", 0, release) > body.rindex("ld.shared", 0, release)
    assert body.count("ld.shared") == body[:release].count("ld.shared")
