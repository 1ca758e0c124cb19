"""Tensor maps describe memory that is allocated and no more: a copy unit given a map that reaches beyond a pool faulted where the pool stood
at the end of what was mapped."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlxforge_b200", "csrc")


def test_no_map_has_an_extent_of_its_own_making():
    """The extents of every map come from the caller's sizes."""
    makers = re.compile(r"\b(bf16_map|bf16_map_chunked|bf16_map_pages|map_3d)\(([^;{]*)\)|\bdims\[\d\] = \{([^}]*)\}")
    seen = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                for m in makers.finditer(f.read()):
                    seen += 1
                    assert "<<" not in m.group(0), (name, m.group(0))
    assert seen > 20


def _case(form, T, held, pages, first):
    """Outputs of ``form`` for a sequence whose pages are the pool's from ``first`` on, in a pool of ``pages``."""
    import torch
    from mlxforge_b200.csrc import ops
    nh, nkv, hd, vd = {"plain64": (4, 2, 64, 64), "plain128": (4, 2, 128, 128), "options": (4, 2, 128, 128), "latent": (3, 1, 160, 128),
                       "wide_latent": (2, 1, 256, 208), "talking": (8, 2, 64, 128), "decode64": (8, 2, 64, 64), "decode128": (8, 2, 128, 128)}[form]
    g = torch.Generator(device="cuda").manual_seed(T + hd)
    bf, ctx = torch.bfloat16, T + held
    n, q = -(-ctx // 16), torch.randn((T, nh * hd), generator=g, device="cuda").to(bf)
    keys, values = (torch.randn((n, nkv, 16, d), generator=g, device="cuda").to(bf) for d in (hd, vd))
    kp, vp = (torch.full((pages, nkv, 16, d), float("nan"), device="cuda", dtype=bf) for d in (hd, vd))
    kp[first:first + n], vp[first:first + n] = keys, values
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    table, out = torch.arange(first, first + n, dtype=torch.int32, device="cuda")[None].contiguous(), torch.zeros((T, nh * vd), device="cuda", dtype=bf)
    seqs = (i32([0]), i32([T]), i32([ctx]), 0, T, table, 16, nh, nkv, hd)
    if form.startswith("plain"):
        ops.attention_prefill(q, kp, vp, out, *seqs, hd ** -0.5, 0)
    elif form == "talking":
        splits = ops.attention_talking_prefill_splits(ctx + 64)
        f = lambda m: torch.zeros(max(m, 1), device="cuda")
        ops.attention_talking_tc(q, kp, vp, out, *seqs, vd, hd ** -0.5, 0.0, torch.eye(nh, device="cuda"), 0, 0, splits, f(T * splits * nh * vd),
                                 f(T * splits * nh * 2))
    elif form.startswith("decode"):
        f = lambda m: torch.zeros(m, device="cuda")
        o, ml = ops.attention_decode_scratch(T, nh, hd, ctx)
        ops.attention_decode(q, kp, vp, out, f(o), f(ml), i32([ctx - 1] * T), i32([0] * T), table, 16, nh, nkv, hd, hd ** -0.5, 0, ctx)
    else:
        own = form == "options"
        sink = torch.zeros(nh, device="cuda") if own else None
        ops.attention_prefill_ex(q, kp, vp if own else kp, out, *seqs, hd ** -0.5, 0, vd, not own, 0, sink)
    ops.check_kernel_status()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain64", "plain128", "options", "latent", "wide_latent", "talking", "decode64", "decode128"])
@pytest.mark.parametrize("held", [0, 77])
def test_the_last_pages_of_a_pool(form, held):
    """A sequence in the last pages of a pool, alone in it or behind others, gets the bits that it gets in the first pages of a longer one."""
    import torch
    T = 1 if form.startswith("decode") else 243
    n = -(-(T + held) // 16)
    want = _case(form, T, held, 3 * n, 0)
    assert not bool(torch.isnan(want).any())
    assert torch.equal(_case(form, T, held, n, 0), want) and torch.equal(_case(form, T, held, n + 5, 5), want)
