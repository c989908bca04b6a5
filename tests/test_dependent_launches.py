"""Kernels launched as dependents of the one before begin before it has ended.  What a kernel of the same chain
writes must then be read behind the wait: through a pointer that the wait ties (a __restrict__ parameter's
loads may otherwise pass it), and not through the non-coherent path.  Read from the sources, no GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "render_engine_gb300", "csrc")

# kernel -> its __restrict__ parameters that an earlier kernel of its chain writes and it reads
READ_BEHIND = {
    ("rc_mlp.cu", "k_mlp_train"): [],
    ("rc_mlp.cu", "k_mlp_gsum"): ["part"],
    ("rc_mlp.cu", "k_mlp_adam"): ["gsum", "w", "m1", "m2"],
    ("rc_taa.cu", "k_post"): ["x", "H", "react", "ref"],
    ("rc_kernels.cu", "k_taa_pt"): ["cur"],
    ("rc_kernels.cu", "k_frame"): [],
    ("rc_kernels.cu", "k_pretrace"): [],
    ("rc_kernels.cu", "k_update"): [],
    ("rc_kernels.cu", "k_event"): [],
    ("rc_kernels.cu", "k_ref"): [],
}


def _kernels(name):
    """(kernel, parameter text, body) of every __global__ function of a source file."""
    text = open(os.path.join(CSRC, name)).read()
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\) )?(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, j = text[m.end():i - 1], text.index("{", i)
        depth, k = 1, j + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), params, text[j:k]


def _waiting():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            for kernel, params, body in _kernels(name):
                if "pdl_wait(" in body:
                    yield name, kernel, params, body


def test_the_table_names_every_waiting_kernel():
    assert {(n, k) for n, k, _, _ in _waiting()} == set(READ_BEHIND)


@pytest.mark.parametrize("name,kernel", sorted(READ_BEHIND))
def test_reads_are_tied_to_the_wait(name, kernel):
    (params, body), = [(p, b) for n, k, p, b in _waiting() if (n, k) == (name, kernel)]
    for p in READ_BEHIND[name, kernel]:
        assert re.search(r"__restrict__ %s\b" % p, params) or re.search(r"\* *%s\b" % p, params)
        assert "%s = pdl_wait(%s);" % (p, p) in body, p
    if name == "rc_mlp.cu":   # its inputs, weights and state are all written between or by the steps
        assert "__ldg(" not in body
