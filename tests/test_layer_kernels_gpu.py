"""Kernels of single layers at the sizes where they can go wrong: edges of tiles, remainders, the smallest and largest of
their range, against 64-bit references."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ran(before):
    from mlxforge_b200.csrc import binding
    return {k: v - before[k] for k, v in binding.kernel_launches().items() if v - before[k]}


# ----------------------------------------------------------------------------- experts, few tokens

@pytest.mark.parametrize("H,ff,E,top,T,act", [
    (2048, 768, 64, 6, 8, None), (64, 64, 4, 1, 1, None), (72, 24, 5, 2, 9, None), (136, 200, 7, 3, 17, "silu"),
    (256, 128, 2, 2, 63, None), (4160, 64, 3, 2, 20, None), (128, 72, 3, 3, 33, "relu2"), (1024, 512, 1024, 8, 63, None)])
def test_experts_few_tokens(H, ff, E, top, T, act):
    """Every chosen expert's matrices once; passes of 8 and 16 tokens, experts with more than one pass, identity experts
    (a choice beyond the matrices), ragged rows and slices."""
    import torch
    from mlxforge_b200.csrc import binding, ops
    g = torch.Generator(device="cuda").manual_seed(H + ff + T)
    bf = torch.bfloat16
    x = torch.randn((T, H), generator=g, device="cuda").to(bf)
    w_gu = (torch.randn((E, 1 if act else 2, ff, H), generator=g, device="cuda") * H ** -0.5).to(bf)
    w_down = (torch.randn((E, H, ff), generator=g, device="cuda") * ff ** -0.5).to(bf)
    # a choice without repetition out of the experts and one identity expert behind them
    ids = torch.rand((T, E + 1), generator=g, device="cuda").topk(top, 1).indices.to(torch.int32).contiguous()
    slices = ops.moe_rows_slices(ff)
    y = torch.full((T, top * slices, H), float("nan"), device="cuda")
    before = binding.kernel_launches()
    ops.moe_rows(x, w_gu, w_down, ids, y, 7.0, 1.702, 1.0, act)
    assert _ran(before).get("moe_rows_mma", 0) == 1
    got = y.view(T, top, slices, H).double().sum(2)
    for t in range(T):
        for k in range(top):
            e = int(ids[t, k])
            if e >= E:
                assert bool(torch.isnan(y.view(T, top, slices, H)[t, k]).all())
                continue
            r = w_gu[e].double() @ x[t].double()
            if act == "silu":
                a = r[0] * torch.sigmoid(r[0])
            elif act == "relu2":
                a = r[0].clamp(min=0) ** 2
            else:
                gate, up = r[0].clamp(max=7.0), r[1].clamp(-7.0, 7.0)
                a = gate * torch.sigmoid(1.702 * gate) * (up + 1.0)
            a = a.to(bf).double()
            terms = w_down[e].double() * a
            # an activation next to a tie of its rounding may fall on the other side (a bfloat16 step, 2^-8 of it, in at most
            # a few of ff: 32-bit sums differ by 1e-6 of a step's 4e-3); the rest is 32-bit summation
            bound = 4 * 2 ** -8 * terms.abs().amax(1) + 1e-5 * terms.abs().sum(1)
            assert bool(((got[t, k] - terms.sum(1)).abs() <= bound).all()), (t, k)
    alone = torch.empty((1, top * slices, H), device="cuda")
    ops.moe_rows(x[T // 2:T // 2 + 1].contiguous(), w_gu, w_down, ids[T // 2:T // 2 + 1].contiguous(), alone, 7.0, 1.702, 1.0, act)
    here = (ids[T // 2] < E).repeat_interleave(slices)
    assert torch.equal(alone[0][here], y[T // 2][here]), "a token's result depends on what else is in the step"


@pytest.mark.parametrize("act", ["silu", "relu2", None])
@pytest.mark.parametrize("ff", [72, 128, 200])
@pytest.mark.parametrize("bad", ["nan", "inf"])
def test_experts_few_tokens_that_are_not_finite(ff, bad, act):
    """A token that is not finite beside others of its experts' passes: theirs keep their bits, and its own outputs are those of its
    ff columns, not of the zeros that fill a slice.  An infinity that every column's first factor has, with the sign of ``act``'s case:
    infinite throughout, zero throughout, or clamped to finite numbers."""
    import torch
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(ff)
    bf, H, E, T, top = torch.bfloat16, 128, 3, 12, 2
    x = torch.randn((T, H), generator=g, device="cuda").to(bf)
    w_gu = torch.randn((E, 1 if act else 2, ff, H), generator=g, device="cuda").to(bf)
    w_gu[:, 0, :, 17] = (w_gu[:, 0, :, 17].abs() + 0.5) * (-1 if act == "relu2" else 1)
    w_down = (torch.rand((E, H, ff), generator=g, device="cuda") + 0.1).to(bf)
    ids = torch.rand((T, E), generator=g, device="cuda").topk(top, 1).indices.to(torch.int32).contiguous()
    slices, ys = ops.moe_rows_slices(ff), []
    for value in (None, float(bad)):
        y = torch.full((T, top * slices, H), 7.0, device="cuda")
        if value is not None:
            x[5, 17] = value
        ops.moe_rows(x, w_gu, w_down, ids, y, 7.0, 1.702, 1.0, act)
        ys.append(y)
    ops.check_kernel_status()
    others = torch.arange(T, device="cuda") != 5
    assert torch.equal(ys[0][others], ys[1][others])
    if bad == "inf":
        assert bool(((ys[1][5] == float("inf")) if act == "silu" else (ys[1][5] == 0) if act == "relu2" else ys[1][5].isfinite()).all())


@pytest.mark.parametrize("E,groups,keep,top", [(64, 8, 4, 6), (33, 0, 0, 5), (6, 3, 1, 2), (200, 0, 0, 9)])
def test_router_ties_and_values_that_are_not_finite(E, groups, keep, top):
    """Equal scores go to the lower expert (groups: the higher one leaves first); a score that is not a number is never chosen
    and its group never leaves."""
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(E)
    T = 37
    z = rng.integers(-2, 3, (T, E)).astype(np.float32)
    z[3, :] = 0.0
    z[5, 1] = np.nan
    z[6, 2] = -np.inf
    z[7, 4] = np.inf
    bias = rng.integers(-1, 2, E).astype(np.float32) if groups == 0 else None
    ids = torch.empty((T, top), dtype=torch.int32, device="cuda")
    wts = torch.empty((T, top), dtype=torch.float32, device="cuda")
    ops.moe_route(torch.from_numpy(z).cuda(), groups, keep, top, 1.0, ids, wts,
                  bias=None if bias is None else torch.from_numpy(bias).cuda())
    s = torch.sigmoid(torch.from_numpy(z)).numpy()          # equal inputs, equal scores: all that the choice needs
    for t in range(T):
        sel = s[t] + (bias if bias is not None else 0)
        if groups:
            pairs = np.sort(s[t].reshape(groups, -1), 1)[:, -2:].sum(1)
            left = list(range(groups))
            for _ in range(groups - keep):
                low = [g for g in left if not np.isnan(pairs[g])]
                left.remove(max(g for g in low if pairs[g] == min(pairs[h] for h in low)))
            sel = np.where(np.isin(np.arange(E) // (E // groups), left), sel, -np.inf)
        if t == 5 and groups:
            continue                                        # which two of a group's scores count when one is NaN is not defined
        order = sorted((e for e in range(E) if sel[e] > -np.inf), key=lambda e: (-sel[e], e))[:top]
        assert ids[t].tolist()[:len(order)] == order, t


@pytest.mark.parametrize("H,top,slices,T,kind", [(2048, 6, 12, 8, 0), (132, 9, 3, 5, 1), (1028, 2, 1, 70, 2), (128, 17, 2, 3, 3),
                                                  (130, 3, 2, 4, 3), (2048, 6, 1, 100, 3),
                                                  (2048, 1, 12, 8, 0), (132, 1, 2, 5, 3), (1028, 1, 1, 70, 1), (132, 2, 2, 5, 3)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_weighted_sum_of_experts(H, top, slices, T, kind, dtype):
    """kind 0: plain; 1: identity experts; 2: rows by slot; 3: a shared branch with its gate as well."""
    import torch
    from mlxforge_b200.csrc import ops
    dt = getattr(torch, dtype)
    g = torch.Generator(device="cuda").manual_seed(H + top)
    y = torch.randn((T * top, slices, H), generator=g, device="cuda")
    w = torch.rand((T, top), generator=g, device="cuda")
    x, shared = (torch.randn((T, H), generator=g, device="cuda").to(dt) for _ in range(2))
    gate = torch.randn((T, 3), generator=g, device="cuda")
    ids = torch.randint(0, 6, (T, top), generator=g, device="cuda", dtype=torch.int32)
    slot = torch.randperm(T * top, generator=g, device="cuda").to(torch.int32)
    out = torch.empty((T, H), dtype=dt, device="cuda")
    ops.moe_combine(y.view(T, top * slices, H) if kind != 2 else y, w, slot if kind >= 2 else None, out, slices,
                    ids if kind in (1, 3) else None, 4, x if kind in (1, 3) else None, shared if kind == 3 else None,
                    gate[:, 2:] if kind == 3 else None, 3)
    rows = (slot.long() if kind >= 2 else torch.arange(T * top, device="cuda")).view(T, top)
    parts = y.double().sum(1)[rows]
    if kind in (1, 3):
        parts = torch.where((ids >= 4)[..., None], x.double()[:, None], parts)
    want = (w.double()[..., None] * parts).sum(1)
    if kind == 3:
        want = want + torch.sigmoid(gate[:, 2:].double()) * shared.double()
    mag = (w.double()[..., None] * y.double().abs().sum(1)[rows]).sum(1) + x.double().abs() * top + shared.double().abs()
    bound = (top + slices + 4) * 2 ** -24 * mag + (want.abs() * 2 ** -8 if dtype == "bfloat16" else 0)
    assert bool(((out.double() - want).abs() <= bound).all())


# ----------------------------------------------------------------------------- attention of prompts: pages that follow one another

@pytest.mark.parametrize("form", ["plain", "options", "latent"])
@pytest.mark.parametrize("lens,held", [([128, 191], [0, 0]), ([129, 300], [63, 500]), ([257], [1000])])
def test_prefill_attention_does_not_depend_on_where_the_pages_are(form, lens, held):
    """A tile of keys whose pages follow one another comes as one copy, any other page by page: the same bits from a cache laid
    out in order, one in reverse and one with every page elsewhere (what the kernel does not fetch is NaN), near a 64-bit result."""
    import torch
    from mlxforge_b200.csrc import binding, ops
    nh, nkv, hd, vd, window, keep = {"plain": (4, 2, 128, 128, 0, 0), "options": (4, 2, 128, 128, 150, 4), "latent": (3, 1, 160, 128, 0, 0)}[form]
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + hd)
    bf, T, ctx = torch.bfloat16, sum(lens), [n + h for n, h in zip(lens, held)]
    q = torch.randn((T, nh * hd), generator=g, device="cuda").to(bf)
    gate = torch.randn((T, nh * vd), generator=g, device="cuda").to(bf) if form == "options" else None
    sink = torch.randn(nh, generator=g, device="cuda") if form == "options" else None
    ks = [torch.randn((c, nkv, hd), generator=g, device="cuda").to(bf) for c in ctx]
    vs = [k[..., :vd] if form == "latent" else torch.randn((c, nkv, vd), generator=g, device="cuda").to(bf) for k, c in zip(ks, ctx)]
    per = [-(-c // 16) for c in ctx]
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    outs = []
    for order in ("in order", "reverse", "elsewhere"):
        ids = {"in order": np.arange(sum(per)), "reverse": np.arange(sum(per))[::-1],
               "elsewhere": np.random.default_rng(1).permutation(3 * sum(per))[:sum(per)]}[order]
        kp = torch.full((3 * sum(per) + 1, nkv, 16, hd), float("nan"), device="cuda", dtype=bf)
        vp = torch.full((3 * sum(per) + 1, nkv, 16, vd), float("nan"), device="cuda", dtype=bf)
        table, at = np.full((len(lens), max(per)), -1, np.int32), 0
        for s, n in enumerate(per):
            table[s, :n] = ids[at:at + n]
            at += n
            for b in range(n):
                k, v = ks[s][b * 16:b * 16 + 16], vs[s][b * 16:b * 16 + 16]
                kp[int(table[s, b]), :, :k.shape[0]] = k.transpose(0, 1)
                vp[int(table[s, b]), :, :k.shape[0]] = v.transpose(0, 1)
        out = torch.full((T, nh * vd), float("nan"), device="cuda", dtype=bf)
        before = binding.kernel_launches()
        args = (i32(np.cumsum([0] + lens[:-1]).tolist()), i32(lens), i32(ctx), 0, max(lens), torch.from_numpy(table).cuda(), 16, nh, nkv, hd, hd ** -0.5)
        if form == "plain":
            ops.attention_prefill(q, kp, vp, out, *args, 0)
        else:
            ops.attention_prefill_ex(q, kp, kp if form == "latent" else vp, out, *args, window, vd, form == "latent", keep, sink, gate, nh * vd,
                                     0.0, min(lens))
        ops.check_kernel_status()
        assert _ran(before).get("attn_prefill_tc", 0) == 1
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    at = 0
    for n, h, k, v in zip(lens, held, ks, vs):
        i, j = torch.arange(h, h + n, device="cuda")[:, None], torch.arange(h + n, device="cuda")[None]
        seen = (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i
        for head in range(nh):
            kv = head // (nh // nkv)
            s = (q[at:at + n, head * hd:(head + 1) * hd].double() @ k[:, kv].double().T * hd ** -0.5).masked_fill_(~seen, -np.inf)
            if sink is not None:
                s = torch.cat((s, sink[head].double().expand(n, 1)), 1)
            p = torch.softmax(s, 1)[:, :h + n]
            want, mag = p @ v[:, kv].double(), p @ v[:, kv].double().abs()
            if gate is not None:
                sg = torch.sigmoid(gate[at:at + n, head * vd:(head + 1) * vd].double())
                want, mag = want * sg, mag * sg
            # a probability is rounded to 8 bits once, the result once more
            got = outs[0][at:at + n, head * vd:(head + 1) * vd].double()
            assert bool(((got - want).abs() <= 2 ** -8 * mag + 2 ** -8 * want.abs() + 1e-6).all()), (head, n)
        at += n


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n,held", [(137, 0), (130, 200), (161, 1000)])
def test_prefill_attention_does_not_depend_on_the_next_portion(hd, n, held):
    """A portion whose last tile of queries is partly another portion's, whose scores are hundreds of times as large: the bits that it
    has alone."""
    import torch
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(n + hd)
    nh, nkv, bf, other = 4, 2, torch.bfloat16, 140
    per, per2 = -(-(n + held) // 16), -(-other // 16)
    q = torch.randn((n + other, nh * hd), generator=g, device="cuda")
    q[n:] *= 300.0
    q = q.to(bf)
    kp, vp = (torch.randn((per + per2, nkv, 16, hd), generator=g, device="cuda").to(bf) for _ in range(2))
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    table = torch.full((2, max(per, per2)), -1, dtype=torch.int32, device="cuda")
    table[0, :per], table[1, :per2] = torch.arange(per), per + torch.arange(per2)
    outs = []
    for seqs in (1, 2):
        T = n if seqs == 1 else n + other
        out = torch.empty((T, nh * hd), device="cuda", dtype=bf)
        ops.attention_prefill(q[:T].contiguous(), kp, vp, out, i32([0, n][:seqs]), i32([n, other][:seqs]), i32([n + held, other][:seqs]), 0,
                              max(n, other if seqs == 2 else 0), table[:seqs].contiguous(), 16, nh, nkv, hd, hd ** -0.5, 0)
        outs.append(out[:n].clone())
    ops.check_kernel_status()
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("form", ["plain", "latent"])
@pytest.mark.parametrize("chain", [0, 1])
@pytest.mark.parametrize("what", ["value nan", "value inf", "key nan", "tile unseen"])
def test_prefill_attention_joins_what_is_not_finite(form, chain, what):
    """Two running results over alternate tiles of 64 keys: a NaN or an infinity that one of them holds is in the joined one where a
    64-bit softmax has it, one whose scores all are minus infinity has no part, and query tiles that see none of it keep their bits."""
    import torch
    from mlxforge_b200.csrc import binding, ops
    nh, nkv, hd, vd = (4, 2, 128, 128) if form == "plain" else (3, 1, 160, 128)
    g = torch.Generator(device="cuda").manual_seed(hd)
    bf, n = torch.bfloat16, 300
    q = (0.3 * torch.randn((n, nh, hd), generator=g, device="cuda")).to(bf)
    q[..., -1] = 1
    k = torch.randn((n, nkv, hd), generator=g, device="cuda").to(bf)
    v = k[..., :vd] if form == "latent" else torch.randn((n, nkv, vd), generator=g, device="cuda").to(bf)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    per, outs, at = -(-n // 16), [], 64 * (2 + chain) + 5
    first = 0 if what == "tile unseen" else at            # the first row that sees it
    for spoilt in (False, True):
        if spoilt and what == "tile unseen":              # all that this chain has of the first 128 keys
            k[64 * chain:64 * chain + 64, :, -1] = -float("inf")
        elif spoilt and what == "key nan":
            k[at, :, -1] = float("nan")
        elif spoilt:
            v[at, :, 7] = float(what.split()[1])
        kp, vp = (torch.full((per, nkv, 16, x.shape[2]), float("nan"), device="cuda", dtype=bf) for x in (k, v))
        for b in range(per):
            for pool, x in ((kp, k), (vp, v)):
                pool[b, :, :x[b * 16:b * 16 + 16].shape[0]] = x[b * 16:b * 16 + 16].transpose(0, 1)
        out = torch.full((n, nh * vd), float("nan"), device="cuda", dtype=bf)
        args = (i32([0]), i32([n]), i32([n]), 0, n, i32([list(range(per))]), 16, nh, nkv, hd, hd ** -0.5)
        before = binding.kernel_launches()
        if form == "plain":
            ops.attention_prefill(q.view(n, -1), kp, vp, out, *args, 0)
        else:
            ops.attention_prefill_ex(q.view(n, -1), kp, kp, out, *args, 0, vd, True, 0, None, None, 0, 0.0, n)
        ops.check_kernel_status()
        assert _ran(before).get("attn_prefill_tc", 0) == 1
        outs.append(out)
    if first >= 128:
        assert torch.equal(outs[0][:128], outs[1][:128])
    i, j = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
    for h in range(nh):
        kd, vd64 = k[:, h // (nh // nkv)].double(), v[:, h // (nh // nkv)].double()
        p = torch.softmax((q[:, h].double() @ kd.T * hd ** -0.5).masked_fill(j > i, -np.inf), 1)
        # a row's own keys only: a zero times what is not finite would not be zero
        for row in range(64 if what == "tile unseen" else first, n, 7):
            want, mag = p[row, :row + 1] @ vd64[:row + 1], p[row, :row + 1] @ vd64[:row + 1].abs()
            got, ok = outs[1][row, h * vd:(h + 1) * vd].double(), want.isfinite()
            assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[~ok & ~want.isnan()], want[~ok & ~want.isnan()])
            assert bool(((got - want).abs() <= 2 ** -8 * mag + 2 ** -8 * want.abs() + 1e-6)[ok].all()), (h, row)


# ----------------------------------------------------------------------------- rotations, biases and norms of prompts

def _store_case(kind, T, g, pages):
    """A launch of ``kind`` for tokens a..b of T tokens: a function of (a, b) that returns the outputs of those tokens' rows."""
    import torch
    from mlxforge_b200.csrc import ops
    bf, f32 = torch.bfloat16, torch.float32
    r = lambda *s, dt=bf: torch.randn(s, generator=g, device="cuda").to(dt)
    pos = torch.randint(0, 5000, (T,), generator=g, device="cuda", dtype=torch.int32)
    table = torch.arange(T, device="cuda", dtype=torch.int32)[:, None].repeat(1, 5000 // 16 + 1).contiguous()       # a page a token
    seq = torch.arange(T, device="cuda", dtype=torch.int32)
    inv = 50000.0 ** (-torch.arange(32, device="cuda", dtype=f32) / 32)
    pool = lambda heads, d: torch.full((T, heads, 16, d), float("nan"), device="cuda", dtype=bf)

    def kv(p, a, b):
        return p[torch.arange(a, b, device="cuda"), :, pos[a:b].long() % 16]

    if kind == "pairs":
        x, nh, nkv, hd = r(T, 8 * 128), 4, 2, 128
        def go(a, b):
            q, k, v = r(b - a, nh * hd), pool(nkv, hd), pool(nkv, hd)
            ops.rope_store(x[a:b], pos[a:b], seq[a:b], table, 16, inv[:24].contiguous(), None, q, k, v, nh, nkv, hd, 48, True, True, True, ld=8 * 128)
            return q, kv(k, a, b), kv(v, a, b)
    elif kind == "halves":
        nh, nkv, hd = 6, 2, 64
        x, freqs = r(T, (nh + 2 * nkv) * hd), (1 / inv[:16]).contiguous()
        def go(a, b):
            q, k, v = r(b - a, nh * hd), pool(nkv, hd), pool(nkv, hd)
            ops.rope_kv_write(x[a:b], pos[a:b], seq[a:b], table, 16, freqs, q, k, v, nh, nkv, hd, 32, True, False)
            return q, kv(k, a, b), kv(v, a, b)
    elif kind == "retention":
        x = r(T, 1000)
        def go(a, b):
            qk = r(b - a, 2 * 3 * 64, dt=f32)
            ops.retention_prepare(x[a:b], 3, 64, 48, 0.125, pos[a:b], inv[:24].contiguous(), None, qk, silu=True)
            return (qk,)
    elif kind == "biases":
        nh, nkv, d, dv = 5, 1, 36, 20
        x, bias = r(T, nh * d + d + dv, dt=f32), r(nh * d + d + dv, dt=f32)
        def go(a, b):
            q, k, v = r(b - a, nh * d), pool(nkv, d), pool(nkv, dv)
            ops.biased_kv_store(x[a:b], bias, pos[a:b], seq[a:b], table, 16, q, k, v, nh, nkv, d, dv, True)
            return q, kv(k, a, b), kv(v, a, b)
    else:
        x, wq, wkv = r(T, 1208), r(1032, dt=f32), r(104, dt=f32)
        def go(a, b):
            cq, k = r(b - a, 1032), pool(1, 104 + 64)
            ops.latent_prepare(x[a:b], 1032, 1040, 104, 64, wq, wkv, 1e-6, pos[a:b], seq[a:b], table, 16, inv, None, cq, k, True)
            return cq, kv(k, a, b)
        xd = x.double()
        want = xd[:, :1032] / (xd[:, :1032].square().mean(1, keepdim=True) + 1e-6).sqrt() * wq.double()
        assert bool(((go(0, T)[0].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all())         # one rounding
    return go


@pytest.mark.parametrize("kind", ["pairs", "halves", "retention", "biases", "latent"])
def test_several_tokens_a_block(kind):
    """Steps of so many tokens that a block takes several, with a last block that has fewer: every token's bits are those it has
    in a step of few."""
    import torch
    T = 8 * torch.cuda.get_device_properties(0).multi_processor_count + 3
    g = torch.Generator(device="cuda").manual_seed(len(kind))
    go = _store_case(kind, T, g, None)
    many = go(0, T)
    assert all(not bool(torch.isnan(m).any()) for m in many)
    for a, b in ((0, 1), (5, 9), (T - 2, T)):
        for m, f in zip(many, go(a, b)):
            assert torch.equal(m[a:b], f), (kind, a)


@pytest.mark.parametrize("kind,sizes,per_sm", [
    ("pairs", (4, 1, 64, 48), 8), ("pairs", (4, 2, 128, 48), 13), ("pairs", (16, 4, 128, 128), 24), ("pairs", (17, 4, 128, 64), 40), ("pairs", (3, 1, 72, 0), 8),
    ("halves", (4, 2, 64, 32), 8), ("halves", (6, 2, 64, 32), 13), ("halves", (24, 6, 64, 64), 24), ("halves", (16, 4, 128, 128), 24), ("halves", (32, 16, 64, 16), 40), ("halves", (1, 1, 4096, 4096), 40),
    ("retention", (3, 64, 48), 8), ("retention", (8, 128, 64), 24), ("retention", (16, 128, 64), 40), ("retention", (1, 72, 0), 8), ("retention", (8, 128, 128), 8),
    ("biases", (3, 1, 36, 20), 8), ("biases", (5, 1, 36, 20), 13), ("biases", (9, 1, 112, 128), 24), ("biases", (16, 4, 128, 128), 40),
    ("latent", (1032, 104, 64, 32), 8), ("latent", (0, 256, 32, 32), 8), ("latent", (2048, 8, 16, 0), 8)])
def test_stored_rows(kind, sizes, per_sm):
    """Steps around the sizes from which a block takes several tokens, of rows that start on a 16-byte boundary and of rows that do not
    (the general kernels): both stay within the roundings of the same in 64 bits, and what is only copied or added keeps its bits."""
    import torch
    from mlxforge_b200.csrc import ops
    bf, f32, f64 = torch.bfloat16, torch.float32, torch.float64
    edge = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(sum(sizes))
    page = 16

    def rows(T, width, dt, off):              # [T, width], `off` elements behind a 16-byte boundary
        x = torch.empty(T * width + 8, device="cuda", dtype=dt)[off:off + T * width].view(T, width)
        return x.copy_(torch.randn((T, width), generator=g, device="cuda"))

    def turned(x, cos, sin, pairs):           # 64 bits; also the size of what was added up
        r, n = 2 * cos.shape[-1], cos.shape[-1]
        a, b = (x[..., 0:r:2], x[..., 1:r:2]) if pairs else (x[..., :n], x[..., n:r])
        y, m = x.clone(), x.abs()
        ya, yb, size = a * cos - b * sin, b * cos + a * sin, a.abs() + b.abs()
        for z, u, v in ((y, ya, yb), (m, size, size)):
            if pairs:
                z[..., 0:r:2], z[..., 1:r:2] = u, v
            else:
                z[..., :n], z[..., n:r] = u, v
        return y, m

    def near(got, want, size, slack=0.0):
        # sine and cosine to 2 ulp, three roundings of 2^-24 each, what the caller adds; a rounding to the result's type
        tol = (2 ** -21 + slack) * size + (2 ** -8 * want.abs() if got.dtype == bf else 0)
        assert bool(((got.double() - want).abs() <= tol).all())

    for T, off in ((1, 0), (3, 1), (edge - 1, 0), (edge, 0), (edge + 3, 0), (edge + 3, 1)):
        pages = -(-T // page)
        table = torch.randperm(pages + 1, generator=g, device="cuda")[:pages].to(torch.int32)[None].contiguous()
        pos, seq = torch.arange(T, device="cuda", dtype=torch.int32), torch.zeros(T, device="cuda", dtype=torch.int32)
        pool = lambda heads, d: torch.full((pages + 1, heads, page, d), float("nan"), device="cuda", dtype=bf)
        kept = lambda p: p[table[0, (pos // page).long()].long(), :, (pos % page).long()]          # [T, heads, d]
        table_f = lambda n: 50000.0 ** (-torch.arange(n, device="cuda", dtype=f32) / max(n, 1))
        turn = lambda angles: (angles.double().cos()[:, None], angles.double().sin()[:, None])
        if kind in ("pairs", "halves"):
            nh, nkv, hd, rot = sizes
            pairs, heads = kind == "pairs", nh + (1 if kind == "pairs" else 2) * nkv
            x, q, k, v = rows(T, heads * hd, bf, off), torch.full((T, nh * hd), float("nan"), device="cuda", dtype=bf), pool(nkv, hd), pool(nkv, hd)
            inv = table_f(rot // 2)
            if pairs:
                ops.rope_store(x, pos, seq, table, page, inv, None, q, k, v, nh, nkv, hd, rot, True, True, True, ld=heads * hd)
                angles = pos.to(f32)[:, None] * inv
            else:
                ops.rope_kv_write(x, pos, seq, table, page, 1 / inv, q, k, v, nh, nkv, hd, rot, True, False)
                angles = pos.to(f32)[:, None] / (1 / inv)
            xs = x.view(T, heads, hd)
            want, size = turned(xs[:, :nh + nkv].double(), *turn(angles), pairs)
            got = torch.cat([q.view(T, nh, hd), kept(k)], 1)
            near(got[..., :rot], want[..., :rot], size[..., :rot])
            assert torch.equal(got[..., rot:], xs[:, :nh + nkv, rot:]) and torch.equal(kept(v), xs[:, -nkv:])
        elif kind == "retention":
            nh, d, rot = sizes
            x, qk, inv = rows(T, 3 * nh * d, bf, off), torch.full((T, 2 * nh * d), float("nan"), device="cuda"), table_f(rot // 2)
            ops.retention_prepare(x, nh, d, rot, 0.3, pos, inv, None, qk, silu=True)
            xd = x.view(T, 3 * nh, d)[:, :2 * nh].double()
            y, size = turned(xd * torch.sigmoid(xd), *turn(pos.to(f32)[:, None] * inv), False)
            f = torch.tensor([1.0] * nh + [0.3] * nh, device="cuda", dtype=f32).double()[None, :, None]
            near(qk.view(T, 2 * nh, d), y * f, size * f, 2 ** -20)            # the sigmoid: an exponential of 2 ulp, a sum and a quotient
        elif kind == "biases":
            nh, nkv, d, dv = sizes
            w = nh * d + nkv * (d + dv)
            x, b, q = rows(T, w, f32, off), torch.randn(w, generator=g, device="cuda"), torch.full((T, nh * d), float("nan"), device="cuda", dtype=bf)
            k, v = pool(nkv, d), pool(nkv, dv)
            ops.biased_kv_store(x, b, pos, seq, table, page, q, k, v, nh, nkv, d, dv, True)
            y = (x + b).to(bf)
            assert torch.equal(q, y[:, :nh * d]) and torch.equal(kept(k).reshape(T, -1), y[:, nh * d:(nh + nkv) * d])
            assert torch.equal(kept(v).reshape(T, -1), y[:, (nh + nkv) * d:])
        else:
            qr, rank, part, rot = sizes
            x, inv = rows(T, qr + 8 + rank + part, bf, off), table_f(rot // 2)
            wq, wkv = (torch.randn(max(n, 4), generator=g, device="cuda") for n in (qr, rank))
            cq, k, pairs = torch.full((T, max(qr, 1)), float("nan"), device="cuda", dtype=bf), pool(1, rank + part), T % 2 == 1
            ops.latent_prepare(x, qr, qr + 8, rank, part, wq if qr else None, wkv, 1e-6, pos, seq, table, page, inv, None, cq if qr else None, k,
                               True, pairs=pairs, rot_dims=rot, magnitude=1.25)
            normed = lambda a, w: a / (a.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
            xd, row = x.double(), kept(k)[:, 0]
            if qr:
                want = normed(xd[:, :qr], wq)
                near(cq, want, want.abs(), 2 ** -20)                          # the sum of up to 2048 squares, by lanes; root and quotient
            want = normed(xd[:, qr + 8:qr + 8 + rank], wkv[:rank])
            near(row[:, :rank], want, want.abs(), 2 ** -20)
            key = xd[:, None, qr + 8 + rank:]
            want, size = turned(key, *(1.25 * c for c in turn(pos.to(f32)[:, None] * inv)), pairs)
            near(row[:, rank:rank + rot], want[:, 0, :rot], 1.25 * size[:, 0, :rot])
            assert torch.equal(row[:, rank + rot:], x[:, qr + 8 + rank + rot:])


@pytest.mark.parametrize("V,heads,T,parts", [(64, 3, 5, 1), (128, 5, 3, 4), (128, 1, 1, 1)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_read_out_norms(V, heads, T, parts, dtype):
    """Retention's and the delta rule's norms over whole heads, broken last blocks, several partial read-outs."""
    import torch
    from mlxforge_b200.csrc import ops
    dt, n = getattr(torch, dtype), heads * V
    g = torch.Generator(device="cuda").manual_seed(V + T)
    o = torch.randn((parts, T, n), generator=g, device="cuda")
    x = torch.randn((T, n + 8), generator=g, device="cuda").to(dt)
    out = torch.empty((T, n), dtype=dt, device="cuda")
    ops.retention_output(o, x[:, 8:], n + 8, 1e-6, out, heads, V)
    rms = lambda a: (a / (a.view(T, heads, V).square().mean(-1, keepdim=True) + 1e-6).sqrt().expand(T, heads, V).reshape(T, n))
    gd = x[:, 8:].double()
    # sums of up to 128 squares and a few roundings of 2^-24, one of the result's type
    tol = 2 ** -8 if dtype == "bfloat16" else 2 ** -19
    want = rms(o.double().sum(0)) * gd * torch.sigmoid(gd)
    assert bool(((out.double() - want).abs() <= tol * want.abs() + 2 ** -20 * gd.abs() * parts).all())
    gate, w = torch.randn((T, n + 4), generator=g, device="cuda"), torch.randn(V, generator=g, device="cuda")
    ops.delta_output(o[0].contiguous(), gate[:, 4:], n + 4, w, 1e-6, out, heads, V)
    want = rms(o[0].double()) * w.double().repeat(heads) * gate[:, 4:].double()
    assert bool(((out.double() - want).abs() <= tol * want.abs() + 1e-12).all())


# ----------------------------------------------------------------------------- talking heads: keys and values by tensor copies

@pytest.mark.parametrize("H,G,dim,vdim,page,lens,held,window,chunk", [
    (16, 4, 128, 128, 16, [33, 17], [0, 700], 0, 0), (8, 2, 128, 64, 32, [48], [15], 0, 32), (6, 3, 64, 128, 16, [70], [1100], 40, 0),
    (4, 4, 64, 64, 48, [1, 31, 64], [5, 0, 0], 0, 0), (16, 1, 128, 128, 16, [130], [2000], 0, 2048), (4, 2, 80, 96, 16, [40], [9], 0, 0)])
def test_talking_heads_portions(H, G, dim, vdim, page, lens, held, window, chunk):
    """Head sizes with and without tensor copies, pages of other sizes, first and last granules that are partly unseen (NaN stands
    wherever no key is), windows and chunks that begin inside a granule, key ranges that are cut."""
    import torch
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(H + dim + sum(lens))
    bf, T, ctx = torch.bfloat16, sum(lens), [n + h for n, h in zip(lens, held)]
    q = torch.randn((T, H * dim), generator=g, device="cuda").to(bf)
    talk = torch.eye(H, device="cuda") + 0.1 * torch.randn((H, H), generator=g, device="cuda")
    per = [-(-c // page) for c in ctx]
    ids = np.random.default_rng(0).permutation(sum(per) + 3)[:sum(per)]
    kp, vp = (torch.full((sum(per) + 3, G, page, d), float("nan"), device="cuda", dtype=bf) for d in (dim, vdim))
    table, ks, vs, at = np.full((len(lens), max(per)), -1, np.int32), [], [], 0
    for s, (n, c) in enumerate(zip(per, ctx)):
        table[s, :n] = ids[at:at + n]
        at += n
        ks.append(torch.randn((c, G, dim), generator=g, device="cuda").to(bf))
        vs.append(torch.randn((c, G, vdim), generator=g, device="cuda").to(bf))
        for b in range(n):
            for pool, x in ((kp, ks[-1]), (vp, vs[-1])):
                x = x[b * page:(b + 1) * page]
                pool[int(table[s, b]), :, :x.shape[0]] = x.transpose(0, 1)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    out = torch.full((T, H * vdim), float("nan"), device="cuda", dtype=bf)
    seen = max(min(c, chunk or c, window or c) for c in ctx) + 64
    splits = ops.attention_talking_prefill_splits(seen, window, chunk)
    f = lambda n: torch.full((max(n, 1),), float("nan"), device="cuda")
    ops.attention_talking_tc(q, kp, vp, out, i32(np.cumsum([0] + lens[:-1]).tolist()), i32(lens), i32(ctx), 0, max(lens), torch.from_numpy(table).cuda(),
                             page, H, G, dim, vdim, dim ** -0.5, 30.0, talk, window, chunk, splits, f(T * splits * H * vdim), f(T * splits * H * 2))
    ops.check_kernel_status()
    at = 0
    for n, h, k, v in zip(lens, held, ks, vs):
        i, j = torch.arange(h, h + n, device="cuda")[:, None], torch.arange(h + n, device="cuda")[None]
        ok = (j <= i) & ((i - j < window) if window else True) & ((i // chunk == j // chunk) if chunk else True)
        s = torch.einsum("ihd,jhd->hij", q[at:at + n].double().view(n, H, dim), k.double().repeat_interleave(H // G, 1)) * dim ** -0.5
        s = torch.einsum("hg,gij->hij", talk.double(), 30.0 * torch.tanh(s / 30.0))
        p = torch.softmax(s.masked_fill(~ok, -np.inf), 2)
        vv = v.double().repeat_interleave(H // G, 1)
        want, mag = torch.einsum("hij,jhd->ihd", p, vv).flatten(1), torch.einsum("hij,jhd->ihd", p, vv.abs()).flatten(1)
        # a probability is rounded to 8 bits once, the result once more
        assert bool(((out[at:at + n].double() - want).abs() <= 2 ** -8 * mag + 2 ** -8 * want.abs() + 1e-6).all()), n
        at += n


@pytest.mark.parametrize("H,page,lens,held,window,chunk,cap,talking", [
    (16, 16, [33, 17, 250, 1], [0, 700, 0, 0], 0, 0, 30.0, True),          # both kernels in one launch, a sequence each by its own length
    (8, 48, [70, 24], [1100, 60], 40, 0, 0.0, True),                       # every window short: the other kernel alone
    (8, 32, [130, 100], [2000, 3], 300, 0, 20.0, True), (16, 16, [130], [2000], 1030, 0, 30.0, True),
    (16, 16, [600], [1500], 0, 2048, 30.0, True), (8, 16, [70], [250], 0, 300, 30.0, True),       # tiles that begin inside a chunk, cut ranges
    (16, 16, [20], [3000], 0, 0, 5.0, False), (8, 16, [300], [0], 0, 0, 0.0, False), (16, 64, [256, 192], [0, 0], 0, 0, 0.0, True)])
def test_talking_heads_prompt_kernel(H, page, lens, held, window, chunk, cap, talking):
    """Tiles of 16 queries and 128 keys with broken ends on all sides, pages in any order (NaN wherever no key is), keys cut at 1024, the rule
    by a sequence's own length, with and without cap and matrix."""
    import torch
    from mlxforge_b200.csrc import binding, ops
    g = torch.Generator(device="cuda").manual_seed(H + sum(lens))
    G, D, bf, T, ctx = H // 4, 128, torch.bfloat16, sum(lens), [n + h for n, h in zip(lens, held)]
    q = torch.randn((T, H * D), generator=g, device="cuda").to(bf)
    talk = torch.eye(H, device="cuda") + 0.1 * torch.randn((H, H), generator=g, device="cuda") if talking else None
    per = [-(-c // page) for c in ctx]
    ids = np.random.default_rng(1).permutation(sum(per) + 3)[:sum(per)] if T % 2 else np.arange(sum(per))
    kp, vp = (torch.full((sum(per) + 3, G, page, D), float("nan"), device="cuda", dtype=bf) for _ in range(2))
    table, ks, vs, at = np.full((len(lens), max(per)), -1, np.int32), [], [], 0
    for s, (n, c) in enumerate(zip(per, ctx)):
        table[s, :n] = ids[at:at + n]
        at += n
        ks.append(torch.randn((c, G, D), generator=g, device="cuda").to(bf))
        vs.append(torch.randn((c, G, D), generator=g, device="cuda").to(bf))
        for b in range(n):
            for pool, x in ((kp, ks[-1]), (vp, vs[-1])):
                x = x[b * page:(b + 1) * page]
                pool[int(table[s, b]), :, :x.shape[0]] = x.transpose(0, 1)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    seen = [min(c, chunk or c, window or c) for c in ctx]
    splits = ops.attention_talking_prefill_splits(max(seen), window, chunk)
    f = lambda n: torch.full((max(n, 1),), float("nan"), device="cuda")
    outs = []
    for bounds in ((min(ctx), max(ctx)), (0, 0)):
        out, before = torch.full((T, H * D), float("nan"), device="cuda", dtype=bf), binding.kernel_launches()
        ops.attention_talking_tc(q, kp, vp, out, i32(np.cumsum([0] + lens[:-1]).tolist()), i32(lens), i32(ctx), 0, max(lens), torch.from_numpy(table).cuda(),
                                 page, H, G, D, D, D ** -0.5, cap, talk, window, chunk, splits, f(T * splits * H * D), f(T * splits * H * 2), 0, *bounds)
        ops.check_kernel_status()
        outs.append(out)
        assert (_ran(before).get("attn_talking_prompt", 0) == 1) == (max(seen) >= (192 if H == 16 else 80))
    assert torch.equal(*outs)
    at = 0
    for n, h, k, v in zip(lens, held, ks, vs):
        i, j = torch.arange(h, h + n, device="cuda")[:, None], torch.arange(h + n, device="cuda")[None]
        ok = (j <= i) & ((i - j < window) if window else True) & ((i // chunk == j // chunk) if chunk else True)
        s = torch.einsum("ihd,jhd->hij", q[at:at + n].double().view(n, H, D), k.double().repeat_interleave(4, 1)) * D ** -0.5
        s = cap * torch.tanh(s / cap) if cap else s
        s = torch.einsum("hg,gij->hij", talk.double(), s) if talking else s
        p = torch.softmax(s.masked_fill(~ok, -np.inf), 2)
        vv = v.double().repeat_interleave(4, 1)
        want, mag = torch.einsum("hij,jhd->ihd", p, vv).flatten(1), torch.einsum("hij,jhd->ihd", p, vv.abs()).flatten(1)
        # a probability is rounded to 8 bits once, the result once more
        assert bool(((out[at:at + n].double() - want).abs() <= 2 ** -8 * mag + 2 ** -8 * want.abs() + 1e-6).all()), n
        at += n


@pytest.mark.parametrize("H,lens,held,window,chunk,cap,talking", [
    (16, 300, 0, 0, 0, 30.0, True), (16, 300, 0, 0, 0, 0.0, False), (8, 300, 0, 0, 0, 30.0, False), (8, 331, 5, 0, 0, 0.0, True),
    (16, 90, 1000, 250, 0, 20.0, True), (8, 90, 1000, 250, 0, 0.0, False), (16, 60, 1490, 0, 2048, 0.0, False), (8, 200, 420, 0, 512, 30.0, True),
    (16, 31, 1000, 0, 0, 0.0, False), (8, 30, 299, 0, 256, 30.0, True)])
def test_talking_heads_prompt_kernel_keeps_what_is_not_finite_apart(H, lens, held, window, chunk, cap, talking):
    """One number of a key or a value of one key head NaN or infinite, at places over all of a tile of 128 and at the ends of the range: the rows
    that do not see it keep their bits (of a value up to the own 16 rows and its own channel, as the weights of a tile are one product),
    values never pass to another key head's query heads, keys only through a matrix; an infinite key under a cap is what 64 bits say."""
    import torch
    from mlxforge_b200.csrc import binding, ops
    g = torch.Generator(device="cuda").manual_seed(H + lens)
    G, D, bf, ctx, page = H // 4, 128, torch.bfloat16, lens + held, 16
    n = -(-ctx // page)
    q = torch.randn((lens, H * D), generator=g, device="cuda").to(bf)
    talk = torch.eye(H, device="cuda") + 0.1 * torch.randn((H, H), generator=g, device="cuda") if talking else None
    pools = [torch.randn((n, G, page, D), generator=g, device="cuda").to(bf) for _ in range(2)]
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    table = torch.arange(n, dtype=torch.int32, device="cuda")[None]
    splits = ops.attention_talking_prefill_splits(min(ctx, chunk or ctx, window or ctx), window, chunk)

    def run(kp, vp):
        f = lambda m: torch.full((max(m, 1),), float("nan"), device="cuda")
        out, before = torch.full((lens, H * D), 7.0, device="cuda", dtype=bf), binding.kernel_launches()
        ops.attention_talking_tc(q, kp, vp, out, i32([0]), i32([lens]), i32([ctx]), 0, lens, table, page, H, G, D, D, D ** -0.5, cap, talk, window, chunk,
                                 splits, f(lens * splits * H * D), f(lens * splits * H * 2), 0, ctx, ctx)
        ops.check_kernel_status()
        assert _ran(before)["attn_talking_prompt"] == 1
        return out.view(lens, H, D)

    pos = torch.arange(held, ctx, device="cuda")
    first = max(0, held - window + 1) if window else held // chunk * chunk if chunk else 0
    whole = lens > 64 or -(-(held % 16 + lens) // 16) == -(-lens // 16) or chunk and held // chunk != (ctx - 1) // chunk
    tile = pos // 16 if whole else (pos - held) // 16          # of positions; of rows where a short portion has fewer so
    at = {first, first + 1, first + 17, held, ctx - 1, ctx - 2, ctx - 17} | {t for t in range(first, ctx, 37)} | {t for t in range(held // 128 * 128, ctx, 64)}
    bits = lambda x: x.view(torch.int16)
    clean, same = run(*pools), lambda a, b: torch.equal(bits(a), bits(b))
    assert bool(clean.isfinite().all())
    for i, t in enumerate(sorted(t for t in at if first <= t < ctx)):
        kv = i % G
        own = slice(4 * kv, 4 * kv + 4)
        other = [h for h in range(H) if h // 4 != kv]
        sees = (pos >= t) & ((pos - t < window) if window else True) & ((pos // chunk == t // chunk) if chunk else True)
        # rows of a tile that holds a row which sees it
        near = torch.isin(tile, tile[sees]) & ~sees
        for bad in (float("nan"), float("inf"), float("-inf")):
            kp, vp = (x.clone() for x in pools)
            vp[t // page, kv, t % page, 5] = bad
            out = run(pools[0], vp)
            assert same(out[:, other], clean[:, other]), (t, bad)
            assert same(out[..., [c for c in range(D) if c != 5]], clean[..., [c for c in range(D) if c != 5]]), (t, bad)
            assert same(out[~(sees | near)], clean[~(sees | near)]), (t, bad)
            assert not bool(out[sees][:, own, 5].isfinite().any()), (t, bad)
            kp[t // page, kv, t % page, 9] = bad
            out = run(kp, pools[1])
            assert same(out[~sees], clean[~sees]), (t, bad)
            if not talking:
                assert same(out[:, other], clean[:, other]), (t, bad)
            if bad != bad:
                assert not bool(out[sees][:, own].isfinite().any()), t
            elif cap:
                k = kp.transpose(1, 2).reshape(n * page, G, D)[:ctx].double().repeat_interleave(4, 1)
                v = pools[1].transpose(1, 2).reshape(n * page, G, D)[:ctx].double().repeat_interleave(4, 1)
                key = torch.arange(ctx, device="cuda")[None]
                ok = (key <= pos[:, None]) & ((pos[:, None] - key < window) if window else True) & ((pos[:, None] // chunk == key // chunk) if chunk else True)
                s = cap * torch.tanh(torch.einsum("ihd,jhd->hij", q.double().view(lens, H, D), k) * D ** -0.5 / cap)
                s = torch.einsum("hg,gij->hij", talk.double(), s) if talking else s
                p = torch.softmax(s.masked_fill(~ok, -np.inf), 2)
                want, mag = torch.einsum("hij,jhd->ihd", p, v), torch.einsum("hij,jhd->ihd", p, v.abs())
                # a probability is rounded to 8 bits once, the result once more
                assert bool(((out.double() - want).abs() <= 2 ** -8 * mag + 2 ** -8 * want.abs() + 1e-6).all()), (t, bad)


@pytest.mark.parametrize("H,window,chunk", [(16, 0, 0), (8, 250, 0), (16, 0, 2048), (8, 0, 512), (16, 0, 500)])
def test_talking_heads_prompt_kernel_portions_give_the_bits_of_the_whole_prompt(H, window, chunk):
    """A prompt at once and its tokens from any place on as a portion of their own: tiles of queries then begin elsewhere, reach over a chunk's
    start or over a cut of the keys, and a row's numbers are the same."""
    import torch
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(H + window)
    G, D, bf, T, page = H // 4, 128, torch.bfloat16, 1200, 16
    q = torch.randn((T, H * D), generator=g, device="cuda").to(bf)
    talk = torch.eye(H, device="cuda") + 0.1 * torch.randn((H, H), generator=g, device="cuda")
    kp, vp = (torch.randn((T // page, G, page, D), generator=g, device="cuda").to(bf) for _ in range(2))
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    splits = ops.attention_talking_prefill_splits(min(T, chunk or T, window or T), window, chunk)
    f = lambda n: torch.full((max(n, 1),), float("nan"), device="cuda")

    def portion(start, end):
        n = end - start
        out = torch.full((n, H * D), float("nan"), device="cuda", dtype=bf)
        ops.attention_talking_tc(q[start:end].contiguous(), kp, vp, out, i32([0]), i32([n]), i32([end]), 0, n, torch.arange(T // page, dtype=torch.int32, device="cuda")[None],
                                 page, H, G, D, D, D ** -0.5, 30.0, talk, window, chunk, splits, f(n * splits * H * D), f(n * splits * H * 2), 0, end, end)
        ops.check_kernel_status()
        return out

    whole = portion(0, T)
    for start, end in ((1009, 1100), (1023, 1025), (491, 520), (300, 1200), (517, 560), (1, 700), (1003, 1031), (1009, 1025)):
        assert torch.equal(portion(start, end), whole[start:end]), (start, end)


@pytest.mark.parametrize("H,dim,ctx,chunk,bounds,prompt,mma,merge", [
    (16, 128, [300, 90], 0, True, 1, 1, 0), (16, 128, [300, 90], 0, False, 1, 1, 0), (16, 128, [90, 70], 0, True, 0, 1, 0), (8, 128, [90, 300], 0, True, 1, 0, 0),
    (16, 128, [2048, 90], 2048, True, 1, 1, 1), (16, 128, [2048], 2048, True, 1, 0, 1), (8, 128, [1024], 1024, True, 1, 0, 0), (4, 64, [1100], 1100, True, 0, 1, 1),
    (4, 64, [90], 0, False, 0, 1, 0)])
def test_talking_heads_launches_are_counted(H, dim, ctx, chunk, bounds, prompt, mma, merge):
    """The library's count of launches and of each kernel, whichever of the two the portions go to and whether keys are cut."""
    import torch
    from mlxforge_b200.csrc import binding, ops
    G, bf, page, i32 = H // 4, torch.bfloat16, 16, lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    lens, T = [20] * len(ctx), 20 * len(ctx)
    q, out = (torch.zeros((T, H * dim), device="cuda", dtype=bf) for _ in range(2))
    kp = torch.zeros((128, G, page, dim), device="cuda", dtype=bf)
    table = torch.arange(128, dtype=torch.int32, device="cuda").repeat(len(ctx), 1)
    splits = ops.attention_talking_prefill_splits(min(max(ctx), chunk or max(ctx)), 0, chunk)
    part = [torch.empty((max(T * splits * H * n, 1),), device="cuda") for n in (dim, 2)]
    launches, before = binding.launch_count(), binding.kernel_launches()
    ops.attention_talking_tc(q, kp, kp, out, i32([20 * i for i in range(len(ctx))]), i32(lens), i32(ctx), 0, 20, table, page, H, G, dim, dim, 1.0, 0.0, None, 0, chunk,
                             splits, *part, 0, *((min(ctx), max(ctx)) if bounds else (0, 0)))
    ops.check_kernel_status()
    ran = _ran(before)
    assert [ran.get("attn_talking_" + k, 0) for k in ("prompt", "mma", "merge")] == [prompt, mma, merge] and ran["attn_talking_tc"] == 1
    assert binding.launch_count() - launches == prompt + mma + merge


# ----------------------------------------------------------------------------- latents: rotated query parts

@pytest.mark.parametrize("T,heads,dim,rot,rank,rot_dims,pairs,extra", [
    (1, 3, 64, 32, 192, 32, False, 0), (9, 16, 64, 32, 128, 32, False, 8), (17, 5, 16, 64, 24, 32, False, 0), (40, 2, 128, 64, 512, 64, True, 0),
    (7, 4, 8, 24, 16, 8, True, 16), (12, 3, 64, 24, 64, 24, False, 0), (12, 3, 60, 32, 64, 32, False, 0), (5, 2, 64, 32, 64, 0, False, 0)])
def test_latent_query_pieces(T, heads, dim, rot, rank, rot_dims, pairs, extra):
    """Whole pieces in halves and in pairs, parts that pass unturned, broken blocks of tokens, and sizes that are no whole pieces: the rotation
    in 64 bits to a rounding of bfloat16 of the pair's size, what is not rotated to the bit."""
    import torch
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(T + rot)
    ld = heads * (dim + rot) + extra
    q = torch.randn((T, ld), generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.randint(0, 500, (T,), generator=g, device="cuda", dtype=torch.int32)
    half = rot_dims // 2
    inv = 100.0 ** (-torch.arange(max(half, 1), device="cuda", dtype=torch.float32) / max(half, 1))
    out = torch.full((T, heads * (rank + rot)), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.latent_query(q, heads, dim, rot, rank, pos, inv, None, out, ld, pairs, rot_dims, 1.25)
    got, src = out.view(T, heads, rank + rot), q[:, :heads * (dim + rot)].view(T, heads, dim + rot)[..., dim:]
    assert bool((got[..., :rank] == 7).all()) and torch.equal(got[..., rank + rot_dims:], src[..., rot_dims:])
    x = src[..., :rot_dims].double()
    u, v = (x[..., 0::2], x[..., 1::2]) if pairs else (x[..., :half], x[..., half:])
    a = (pos[:, None].float() * inv[None, :half]).double()[:, None]
    c, s = torch.cos(a) * 1.25, torch.sin(a) * 1.25
    w = got[..., rank:rank + rot_dims].double()
    gu, gv = (w[..., 0::2], w[..., 1::2]) if pairs else (w[..., :half], w[..., half:])
    size = 1.25 * (u.square() + v.square()).sqrt()
    # one rounding to 8 bits; a few of 24 before it
    assert bool(((gu - (u * c - v * s)).abs() <= 2.0 ** -8 * size).all()) and bool(((gv - (v * c + u * s)).abs() <= 2.0 ** -8 * size).all())


# ----------------------------------------------------------------------------- 32-bit products

@pytest.mark.parametrize("M,N,K", [(300, 3001, 36), (449, 1409, 67), (150, 2900, 52), (45, 700, 20)])
def test_gemm_f32_every_tile(M, N, K):
    """Sizes that choose 64 x 128, 48 x 128, 64 x 64 and 32 x 64 results a block, with broken tiles on both sides: rows have the bits
    they have alone; sums of K products of unit normals in four chains within 2^-22 sqrt(K) of their norm sqrt(K)."""
    import torch
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(M)
    a, w = torch.randn((M, K), generator=g, device="cuda"), torch.randn((N, K), generator=g, device="cuda")
    out, few = torch.full((M, N), float("nan"), device="cuda"), torch.empty((5, N), device="cuda")
    ops.gemm_f32(a, w, out)
    assert bool(((out.double() - a.double() @ w.double().T).abs() < 2.0 ** -22 * K).all())
    ops.gemm_f32(a[M - 5:].contiguous(), w, few)
    assert torch.equal(few, out[M - 5:])


@pytest.mark.parametrize("nh,nkv,hd,vd,n", [(8, 2, 64, 64, 40), (16, 4, 128, 128, 100), (3, 1, 96, 192, 70), (20, 1, 32, 32, 9)])
def test_attention_f32_tiles_of_every_height(nh, nkv, hd, vd, n):
    """A portion alone (tiles of 16 or 32 rows), beside a few and beside so many others that tiles of 64 rows are taken: the same bits,
    within 2^-18 of a 64-bit result's weighted magnitudes (chains of at most 64 roundings of 2^-24 a tile, few tiles)."""
    import torch
    from types import SimpleNamespace
    from mlxforge_b200.csrc import ops
    g = torch.Generator(device="cuda").manual_seed(n)
    held, per = 130, -(-(130 + n) // 16)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    q = torch.randn((n, nh * hd), generator=g, device="cuda")
    kp, vp = (torch.randn((per + 2, nkv, 16, d), generator=g, device="cuda") for d in (hd, vd))
    order = np.random.default_rng(n).permutation(per + 2)[:per].astype(np.int32)
    outs = []
    for copies in (1, 6, 60):
        out = torch.full((copies * n, nh * vd), float("nan"), device="cuda")
        batch = SimpleNamespace(seq_q_start=i32([c * n for c in range(copies)]), seq_q_len=i32([n] * copies), seq_ctx_len=i32([held + n] * copies),
                                n_seqs=copies, q_len=[n] * copies)
        table = torch.from_numpy(np.tile(order, (copies, 1))).cuda()
        if vd == hd:
            ops.attention_f32(q.repeat(copies, 1), kp, vp, out, batch, table, 16, nh, nkv, hd, hd ** -0.5, 0, vd, vd)
        else:
            ops.attention_f32(q.repeat(copies, 1), kp, vp, out, batch, table, 16, nh, nkv, hd, hd ** -0.5, 90, vd, vd, 20)
        outs.append(out[-n:])
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    k, v = (p[torch.from_numpy(order).long().cuda()].transpose(1, 2).reshape(per * 16, nkv, -1)[:held + n].double() for p in (kp, vp))
    i, j = torch.arange(held, held + n, device="cuda")[:, None], torch.arange(held + n, device="cuda")[None]
    seen = j <= i if vd == hd else (j <= i) & ((i - j < 90) | (j < 20))
    for h in range(nh):
        s = (q[:, h * hd:(h + 1) * hd].double() @ k[:, h // (nh // nkv)].T * hd ** -0.5).masked_fill(~seen, -np.inf)
        p = torch.softmax(s, 1)
        want, mag = p @ v[:, h // (nh // nkv)], p @ v[:, h // (nh // nkv)].abs()
        assert bool(((outs[0][:, h * vd:(h + 1) * vd].double() - want).abs() <= 2 ** -18 * mag).all())


# ----------------------------------------------------------------------------- experts, many tokens

@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (37, 3, 33), (2048, 8, 1024), (16385, 1, 64), (5001, 7, 200), (4099, 12, 2)])
def test_sorted_pairs_and_gathered_rows(T, top, E):
    """Pairs that the block loads at once (up to 8,192) and those beyond, experts in part of a warp up to all of the block's
    threads, identity experts in between, gathers whose last block has a rest: whole numbers and copies, so equality."""
    import torch
    from mlxforge_b200.csrc import ops
    rng, H = np.random.default_rng(T + E), 64
    ids = rng.integers(0, E + max(E // 4, 1), (T, top)).astype(np.int32)
    ids[0, 0] = 0
    n, tile_rows, bf = T * top, ops.moe_tc_rows(), torch.bfloat16
    empty = lambda m: torch.full((m,), -7, dtype=torch.int32, device="cuda")
    slot, row_token, meta, tiles = empty(n), empty(n), empty(4), empty(3 * ops.moe_grouped_max_tiles(T, top, E))
    ops.moe_sort(torch.from_numpy(ids).cuda(), E, slot, row_token, meta, tiles, tile_rows)
    slots, tokens = slot.cpu().numpy().reshape(T, top), row_token.cpu().numpy()
    real = ids < E
    m = int(real.sum())
    assert np.all(slots[~real] == -1) and np.array_equal(np.sort(slots[real]), np.arange(m)) and np.all(tokens[m:] == 0)
    assert np.array_equal(tokens[slots[real]], np.nonzero(real)[0])
    of_row = np.empty(m, np.int64)
    of_row[slots[real]] = ids[real]
    assert np.all(np.diff(of_row) >= 0)                       # the experts' rows one expert after another
    cuts = tiles.cpu().numpy()[:3 * int(meta[0])].reshape(-1, 3)
    assert all(np.all(of_row[r:r + k] == e) and 0 < k <= tile_rows for e, r, k in cuts) and cuts[:, 2].sum() == m
    x = torch.from_numpy(rng.standard_normal((T, H)).astype(np.float32)).cuda().to(bf)
    xg, act = torch.zeros((n, H), dtype=bf, device="cuda"), torch.empty((n, 64), dtype=bf, device="cuda")
    wg = torch.zeros((E, 2, 64, H), dtype=bf, device="cuda")
    ops.moe_tc_up(x, row_token, xg, wg, meta, tiles, act, 1.5, 1.702, 1.0, None)
    ops.check_kernel_status()
    assert torch.equal(xg, x[row_token.long()])
