"""Kernels that are launched before their predecessor has finished: what their sources may promise the compiler about memory."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlxforge_b200", "csrc")

# weights and constant tables: nothing writes them while steps run
CONSTANTS = {"w", "w1", "w2", "W", "wt", "w_gu", "w_down", "wq", "wkv", "g", "weight", "bias", "delta_bias", "logit_bias", "dt_bias", "a_log", "A",
             "decay", "mix", "win", "wout", "table", "freqs", "inv_f", "inv_d"}


def _closing(s, i, pair):
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(s[i], 0)
        i += 1
        if depth == 0:
            return i


def _dependent_kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as f:
            s = f.read()
        for m in re.finditer(r"__global__\s+void\s*(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\))?\s*(\w+)\s*\(", s):
            end = _closing(s, m.end() - 1, "()")
            start = s.index("{", end)
            body = s[start:_closing(s, start, "{}")]
            if "pdl_wait" in body:
                yield f"{name}:{m.group(1)}", s[m.end():end - 1], body


def test_the_kernels_are_found():
    assert len(list(_dependent_kernels())) > 40


@pytest.mark.parametrize("kernel,params,body", [pytest.param(*k, id=k[0]) for k in _dependent_kernels()])
def test_what_a_predecessor_writes_is_not_promised_to_stay(kernel, params, body):
    """A ``const __restrict__`` pointer (or ``__ldg``) says that nobody writes the memory while the kernel lives, and the compiler then may
    read it ahead of the wait for the kernel before, which is still writing it."""
    promised = set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params))
    assert promised <= CONSTANTS, (kernel, promised - CONSTANTS)
    assert "__ldg" not in body and "global.nc" not in body, kernel
