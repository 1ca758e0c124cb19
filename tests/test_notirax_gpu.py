"""The Notirax parts and models on the GPU against the plain implementation (plain_notirax.py).

Part by part (each built from its registry with its own sizes, given a runtime, a step batch and a
cache lane, run over portions and single tokens of two sequences), then whole models of three
configurations through the trace replayer's functions -- whole prompts, the last tokens decoded
one by one, portions down to two tokens, mixed batches on a pool so small that pages and slots are
used again, every request decoded from its first token -- in float32 and bfloat16, and greedy
generation through the engine's entry point and scheduler."""
import io
from types import SimpleNamespace

import numpy as np
import pytest

import plain_notirax as P
import trace_tools as TT
from helpers import bf16_round
from notirax_helpers import CONFIGS, make_model, prompt

pytestmark = pytest.mark.gpu

LENGTHS = [45, 23]
STEPS = [(20, 0), (7, 5), (0, 16), (17, 1), (1, 1)]     # tokens of (sequence 0, sequence 1) per step


def tdt(name):
    import torch
    return {"float32": torch.float32, "bfloat16": torch.bfloat16}[name]


def dev(a, dtype=None):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.to(dtype)


def host(t):
    import torch
    return t.detach().to("cpu", torch.float32).numpy().astype(np.float64)


def tol(dtype, scale):
    return (3e-5 if dtype == "float32" else 3e-2) * max(1.0, scale)


def rand(rng, *shape, std=1.0):
    return bf16_round(rng.standard_normal(shape).astype(np.float32) * std)


class Harness:
    """A runtime, a cache with one lane of the given need (or one of each of several) and the runner's metadata builder."""

    def __init__(self, dtype, need, lengths=LENGTHS, steps=STEPS, page_size=16, max_tokens=512):
        import torch
        from mlxforge_b200.cache.manager import CacheLayout, CacheManager, GroupLayout
        from mlxforge_b200.engine.runtime import Runtime
        from mlxforge_b200.engine.step import ModelRunner
        from mlxforge_b200.parts.base import PagedKV
        self.rt = Runtime(tdt(dtype))
        needs = need if isinstance(need, tuple) else (need,)
        paged = tuple(n for n in needs if isinstance(n, PagedKV))
        state = tuple(n for n in needs if not isinstance(n, PagedKV))
        lanes = tuple(("paged", paged.index(n), 0) if isinstance(n, PagedKV) else ("state", state.index(n), 0) for n in needs)
        layout = CacheLayout(paged=tuple(GroupLayout(n, 1) for n in paged), state=tuple(GroupLayout(n, 1) for n in state),
                             item_lane=(lanes if isinstance(need, tuple) else lanes[0],))
        self.cache = CacheManager(layout, page_size=page_size, max_tokens=max_tokens, max_seqs=4, dtype=tdt(dtype),
                                  device="cuda")
        for pool in self.cache._k + self.cache._v:
            pool.fill_(float("nan"))
        self.cache.open_sequence()                                     # so that the sequences do not sit in slot 0
        for st in self.cache._state:
            st.fill_(float("nan"))                                     # a slot is zeroed when a sequence opens
        stub = SimpleNamespace(graph_safe=False, spec=SimpleNamespace(vocab_size=1 << 20))
        self.runner = ModelRunner(stub, self.cache, self.rt)
        self.lengths, self.plan = lengths, steps
        self.seqs = [self.cache.open_sequence() for _ in lengths]
        torch.cuda.synchronize()

    def steps(self):
        """Yields (batch, rows): rows[i] = (sequence, position) of the step's i-th token."""
        from mlxforge_b200.engine.step import StepEntry
        done = [0] * len(self.lengths)
        for counts in self.plan:
            entries, per_seq = [], []
            for s, n in enumerate(counts):
                if n:
                    entries.append(StepEntry(self.seqs[s], [0] * n, []))
                    per_seq.append((s, n))
            self.cache.reserve([(e.seq, len(e.tokens)) for e in entries])
            batch = self.runner._build(entries)
            order = sorted(range(len(per_seq)), key=lambda i: (per_seq[i][1] != 1, i))
            rows = [(per_seq[i][0], done[per_seq[i][0]] + j) for i in order for j in range(per_seq[i][1])]
            yield batch, rows
            for e in entries:
                self.cache.commit(e.seq, len(e.tokens))
            for s, n in per_seq:
                done[s] += n
        assert done == list(self.lengths)

    def run_mixer(self, part, xs, dtype):
        """The mixer's output for every token of the sequences ``xs`` (arrays [len, H]), fed in steps."""
        got = [np.zeros((len(x), part.hidden)) for x in xs]
        lane = self.cache.lane(0)
        for batch, rows in self.steps():
            x = np.stack([xs[s][p] for s, p in rows])
            out = host(part.forward(dev(x, tdt(dtype)), batch, lane))
            bias = getattr(part, "output_bias", None)
            if bias is not None:
                out = out + host(bias)
            for i, (s, p) in enumerate(rows):
                got[s][p] = out[i]
        return got


# ----------------------------------------------------------------------------- streams, norm, embedding

@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("S,groups,H", [(1, 1, 40), (3, 4, 96), (5, 3, 33 * 3), (8, 2, 2048)])
def test_stream_write_read_and_grouped_norm(dtype, S, groups, H):
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(S * 100 + groups)
    T, eps = 7, 1e-5
    x = rng.standard_normal((T, S, H)).astype(np.float32) * 2
    y, bias = rand(rng, T, H), rng.standard_normal(H).astype(np.float32)
    mix = (np.eye(S) + 0.3 * rng.standard_normal((S, S))).astype(np.float32)
    w_out, w_in = rng.standard_normal(S).astype(np.float32), rng.standard_normal(S).astype(np.float32)
    w = (1 + 0.2 * rng.standard_normal(H)).astype(np.float32)
    f = np.float64
    new = P.hyper_write(x.transpose(1, 0, 2).astype(f), y.astype(f) + bias, mix.astype(f), w_out.astype(f))
    want = P.group_rms_norm(P.hyper_read(new, w_in.astype(f)), w.astype(f), eps, groups)
    streams = dev(x.reshape(T, S * H))
    out = torch.empty((T, H), dtype=tdt(dtype), device="cuda")
    ops.hyper_update_norm(streams, dev(y, tdt(dtype)), dev(bias), dev(mix), dev(w_out), dev(w_in), dev(w), eps, groups,
                          out, S)
    assert np.max(np.abs(host(out) - want)) < tol(dtype, np.abs(want).max())
    assert np.max(np.abs(host(streams).reshape(T, S, H).transpose(1, 0, 2) - new)) < 1e-5 * np.abs(new).max()
    # selected rows only: the streams stay, the result is that of the rows; no read weights: the plain sum
    streams = dev(x.reshape(T, S * H))
    rows = dev(np.array([5, 0, 5], dtype=np.int32))
    out = torch.empty((3, H), dtype=tdt(dtype), device="cuda")
    ops.hyper_update_norm(streams, dev(y, tdt(dtype)), None, dev(mix), dev(w_out), None, dev(w), eps, groups, out, S, rows)
    new = P.hyper_write(x.transpose(1, 0, 2).astype(f), y.astype(f), mix.astype(f), w_out.astype(f))
    want = P.group_rms_norm(new.sum(0), w.astype(f), eps, groups)[[5, 0, 5]]
    assert np.max(np.abs(host(out) - want)) < tol(dtype, np.abs(want).max())
    assert np.array_equal(host(streams), x.reshape(T, S * H).astype(f))
    # nothing pending, identity write: the ordinary residual sum
    streams = dev(x.reshape(T, S * H))
    out = torch.empty((T, H), dtype=tdt(dtype), device="cuda")
    ops.hyper_update_norm(streams, None, None, None, None, dev(w_in), dev(w), eps, groups, out, S)
    want = P.group_rms_norm(P.hyper_read(x.transpose(1, 0, 2).astype(f), w_in.astype(f)), w.astype(f), eps, groups)
    assert np.max(np.abs(host(out) - want)) < tol(dtype, np.abs(want).max())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_embedding_with_sinusoid_into_every_stream(dtype):
    import torch
    from mlxforge_b200.parts.base import EMBEDDINGS, PartSpec, build_part
    from mlxforge_b200.engine.runtime import Runtime
    rng = np.random.default_rng(0)
    V, H, S = 50, 37, 3
    part = build_part(EMBEDDINGS, PartSpec("token_embedding", {"vocab_size": V, "hidden_size": H, "tensor": "embed",
                                                               "positions": "sinusoid"}), Runtime(tdt(dtype)))
    table = rand(rng, V, H)
    part.bind({"embed": dev(table)})
    tokens = np.array([3, 49, 0, 7], dtype=np.int32)
    positions = np.array([0, 1, 1500, 40000], dtype=np.int32)
    out = torch.empty((4, S * H), dtype=torch.float32, device="cuda")
    part.embed(SimpleNamespace(tokens=dev(tokens), positions=dev(positions)), out, S)
    want = P.embed(table.astype(np.float64), tokens, positions)
    got = host(out).reshape(4, S, H)
    for s in range(S):
        assert np.max(np.abs(got[:, s] - want)) < (2e-6 if dtype == "float32" else 5e-3)


# ----------------------------------------------------------------------------- attention

ATTN_CASES = {
    # heads, kv, dim, vdim, chunk, window, softcap, talking
    "odd": (6, 2, 24, 40, 7, 0, 4.0, True),
    "page_chunk": (4, 4, 16, 16, 16, 0, 0.0, True),
    "no_talk_no_chunk": (3, 1, 32, 8, 0, 0, 30.0, False),
    "window": (4, 2, 16, 24, 0, 9, 0.0, True),
    "tiles": (4, 2, 64, 64, 40, 0, 10.0, True),
    "long": (4, 2, 64, 32, 0, 0, 10.0, True),        # no chunk and 1,300 tokens: the key range is cut across blocks
    "two_heads": (2, 1, 32, 32, 24, 0, 5.0, True),   # fewer heads than the tensor-core kernel has warps
    "sixteen_heads": (16, 4, 16, 96, 50, 0, 8.0, True),
}
ATTN_PLANS = {"tiles": ([150, 70], [(129, 0), (2, 40), (18, 29), (1, 1)]),
              "long": ([1300, 70], [(1100, 0), (150, 40), (49, 29), (1, 1)])}


def _attention_part(dtype, case, rng, H=56, gain=1.0):
    from mlxforge_b200.parts.base import MIXERS, PartSpec, build_part
    nh, nkv, d, dv, chunk, window, cap, talking = ATTN_CASES[case]
    params = {"hidden_size": H, "n_heads": nh, "n_kv_heads": nkv, "head_dim": d, "v_head_dim": dv,
              "softmax_scale": 1.7 * d ** -0.5, "softcap": cap, "talking": talking, "chunk": chunk, "window": window}
    part = build_part(MIXERS, PartSpec("talking_attention", params, prefix="a."), None)
    w = {}
    for name, spec in part.tensor_specs().items():
        if name.endswith("talk"):
            w[name] = bf16_round((np.eye(nh) + 0.3 * rng.standard_normal((nh, nh))).astype(np.float32))
        elif len(spec.shape) == 1:
            w[name] = rand(rng, *spec.shape, std=0.3)
        else:
            g = gain if name in ("a.q", "a.k") else 1.0
            w[name] = rand(rng, *spec.shape, std=g / np.sqrt(spec.shape[1]))
    p = {"heads": nh, "kv_heads": nkv, "dim": d, "vdim": dv, "scale": params["softmax_scale"], "softcap": cap,
         "mask": {"size": chunk} if chunk else None}
    return params, w, p, window


def _plain_attention(x, p, w, window):
    f = {k[2:]: v.astype(np.float64) for k, v in w.items()}
    if not window:
        return P.talking_chunk_attention(x, p, f.get)
    # a window is not in the plain model: the same function on every window's keys alone
    out = np.zeros((x.shape[0], f["o"].shape[0]))
    q_only = dict(p)
    for i in range(x.shape[0]):
        lo = max(0, i - window + 1)
        out[i] = P.talking_chunk_attention(x[lo:i + 1], q_only, f.get)[-1]
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("case", list(ATTN_CASES))
def test_talking_attention_part(dtype, case):
    from mlxforge_b200.parts.base import MIXERS, PartSpec, build_part
    rng = np.random.default_rng(sum(map(ord, case)))
    params, w, p, window = _attention_part(dtype, case, rng)
    lengths, steps = ATTN_PLANS.get(case, (LENGTHS, STEPS))
    part = build_part(MIXERS, PartSpec("talking_attention", params, prefix="a."), None)
    need = part.cache_need()
    h = Harness(dtype, need, lengths, steps, max_tokens=2048)
    part = build_part(MIXERS, PartSpec("talking_attention", params, prefix="a."), h.rt)
    part.bind({n: dev(a) for n, a in w.items()})
    xs = [rand(rng, n, params["hidden_size"]) for n in lengths]
    got = h.run_mixer(part, xs, dtype)
    for s, x in enumerate(xs):
        want = _plain_attention(x.astype(np.float64), p, w, window)
        assert np.max(np.abs(got[s] - want)) < tol(dtype, np.abs(want).max()), (case, s)
    if params["chunk"]:
        # pages before the chunk of the next query went back to the pool
        held = h.seqs[0].pages_held(0)
        assert held == (lengths[0] + 15) // 16 - (lengths[0] // params["chunk"] * params["chunk"]) // 16


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("case", ["odd", "page_chunk", "tiles"])
def test_keys_at_the_edges_of_chunks_and_pages_decide(dtype, case):
    """The keys at the last place of a chunk, the first of the next, and at both sides of every page
    border are made to stand out (their scores are far above the others'), with values of their own:
    a query that sees one key too many or too few ends somewhere else.  In prompts and decoding."""
    from mlxforge_b200.parts.base import MIXERS, PartSpec, build_part
    rng = np.random.default_rng(5)
    params, w, p, window = _attention_part(dtype, case, rng, gain=1.0)
    chunk, H = params["chunk"], params["hidden_size"]
    lengths = [4 * chunk + 3, 2 * chunk + 1] if chunk < 30 else [150, 90]
    steps = [(lengths[0] - chunk - 2, 3), (2, lengths[1] - 5)] + [(1, 1)] * 2 + [(chunk - 2, 0)]
    steps[-1] = (lengths[0] - sum(s[0] for s in steps[:-1]), lengths[1] - sum(s[1] for s in steps[:-1]))
    part = build_part(MIXERS, PartSpec("talking_attention", params, prefix="a."), None)
    h = Harness(dtype, part.cache_need(), lengths, steps)
    part = build_part(MIXERS, PartSpec("talking_attention", params, prefix="a."), h.rt)
    # every token's input has a common direction e: queries and keys both project it strongly for the
    # edge tokens, so an edge key outweighs all others for every later query of its chunk
    e = rand(rng, H)
    xs = []
    for n in lengths:
        x = rand(rng, n, H, std=0.3)
        for j in range(n):
            if chunk and (j % chunk in (0, chunk - 1)) or j % 16 in (0, 15):
                x[j] = bf16_round(x[j] + 1.5 * e)
        xs.append(x)
    part.bind({n: dev(a) for n, a in w.items()})
    got = h.run_mixer(part, xs, dtype)
    for s, x in enumerate(xs):
        want = _plain_attention(x.astype(np.float64), p, w, window)
        assert np.max(np.abs(got[s] - want)) < tol(dtype, np.abs(want).max()), (case, s)


# ----------------------------------------------------------------------------- gated delta rule

DELTA_CASES = {
    # heads, kv, dim, vdim, taps, decay rank, gate rank
    "odd": (6, 2, 20, 12, 4, 5, 3),
    "one_tap": (2, 2, 16, 16, 1, 4, 4),
    "wide": (2, 1, 128, 48, 2, 8, 8),
    "long_taps": (3, 3, 40, 24, 6, 2, 7),
    "unaligned": (2, 1, 18, 10, 3, 3, 3),            # sizes that are no multiple of 4: the kernel without 16-byte copies
}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("case", list(DELTA_CASES))
def test_channel_delta_part(dtype, case):
    from mlxforge_b200.parts.base import MIXERS, PartSpec, build_part
    rng = np.random.default_rng(len(case))
    nh, nkv, d, dv, taps, ra, rg = DELTA_CASES[case]
    H, eps = 48, 1e-5
    params = {"hidden_size": H, "n_heads": nh, "n_kv_heads": nkv, "head_dim": d, "v_head_dim": dv, "conv": taps,
              "eps": eps, "decay_rank": ra, "gate_rank": rg}
    part = build_part(MIXERS, PartSpec("channel_delta", params, prefix="m."), None)
    # portions shorter than the convolution's history, single tokens in between
    lengths, steps = [60, 31], [(20, 0), (2, 5), (1, 1), (1, 0), (3, 16), (17, 1), (1, 1), (15, 7)]
    h = Harness(dtype, part.cache_need(), lengths, steps)
    part = build_part(MIXERS, PartSpec("channel_delta", params, prefix="m."), h.rt)
    w = {}
    for name, spec in part.tensor_specs().items():
        leaf = name.split(".")[-1]
        if leaf == "norm":
            w[name] = bf16_round((1 + 0.1 * rng.standard_normal(spec.shape)).astype(np.float32))
        elif leaf in ("conv", "A_log", "dt_bias"):
            w[name] = rand(rng, *spec.shape, std=0.6)
        else:
            w[name] = rand(rng, *spec.shape, std=1.5 / np.sqrt(spec.shape[1]))
    part.bind({n: dev(a) for n, a in w.items()})
    xs = [rand(rng, n, H) for n in lengths]
    got = h.run_mixer(part, xs, dtype)
    p = {"heads": nh, "kv_heads": nkv, "dim": d, "vdim": dv, "conv": taps}
    f = {k[2:]: v.astype(np.float64) for k, v in w.items()}
    for s, x in enumerate(xs):
        want = P.channel_delta(x.astype(np.float64), p, f.get, eps)
        assert np.max(np.abs(got[s] - want)) < tol(dtype, np.abs(want).max()), (case, s)


def test_delta_state_carries_a_far_token():
    """One early token writes into key channels that no other token touches (their keys are zero
    there), the state hardly decays, and the last token asks with a query in those channels: its
    read-out is the early token's value, hundreds of tokens and several steps later.  A state that
    is lost, restarted or decayed wrongly shows."""
    from mlxforge_b200.parts.base import MIXERS, PartSpec, build_part
    rng = np.random.default_rng(9)
    nh, d, dv, H = 2, 16, 16, 32
    params = {"hidden_size": H, "n_heads": nh, "n_kv_heads": nh, "head_dim": d, "v_head_dim": dv, "conv": 1,
              "eps": 1e-6, "decay_rank": 2, "gate_rank": 2}
    part = build_part(MIXERS, PartSpec("channel_delta", params, prefix="m."), None)
    lengths = [300, 5]
    steps = [(100, 1), (1, 1), (50, 1), (2, 1), (146, 1), (1, 0)]
    h = Harness("float32", part.cache_need(), lengths, steps)
    part = build_part(MIXERS, PartSpec("channel_delta", params, prefix="m."), h.rt)
    w = {n: rand(rng, *s.shape, std=0.3 if len(s.shape) > 1 else 0.1) for n, s in part.tensor_specs().items()}
    w["m.a1"] *= 0.0
    w["m.dt_bias"] = np.full(nh * d, -14.0, dtype=np.float32)            # softplus ~ 1e-6: the state hardly decays
    w["m.q.conv"], w["m.k.conv"], w["m.v.conv"] = (np.ones_like(w[n]) for n in ("m.q.conv", "m.k.conv", "m.v.conv"))
    w["m.norm"] = np.ones(dv, dtype=np.float32)
    # ordinary tokens live in the first half of the width; the second half is read by the upper key
    # and query channels of every head only, and by nothing else of q and k
    for n in ("m.q", "m.k"):
        m = w[n].reshape(nh, d, H)
        m[:, :d // 2, H // 2:] = 0.0
        m[:, d // 2:, :H // 2] = 0.0
        m[:, d // 2:, H // 2:] = np.abs(m[:, d // 2:, H // 2:])
    xs = [rand(rng, n, H, std=0.5) for n in lengths]
    for x in xs:
        x[:, H // 2:] = 0.0
    e = np.zeros(H, dtype=np.float32)
    e[H // 2:] = bf16_round(np.abs(rng.standard_normal(H // 2)).astype(np.float32) + 1.0)
    xs[0][3] += e                                                        # the far token
    xs[0][299] += e                                                      # the query that asks for it
    part.bind({n: dev(a) for n, a in w.items()})
    got = h.run_mixer(part, xs, "float32")
    p = {"heads": nh, "kv_heads": nh, "dim": d, "vdim": dv, "conv": 1}
    f = {k[2:]: v.astype(np.float64) for k, v in w.items()}
    want = P.channel_delta(xs[0].astype(np.float64), p, f.get, 1e-6)
    without = xs[0].astype(np.float64).copy()
    without[3] -= e
    assert np.max(np.abs(P.channel_delta(without, p, f.get, 1e-6)[299] - want[299])) > 0.2 * np.abs(want[299]).max(), \
        "the far token does not decide: the test would show nothing"
    assert np.max(np.abs(got[0] - want)) < 3e-5 * max(1.0, np.abs(want).max())


# ----------------------------------------------------------------------------- mixture of experts

@pytest.mark.parametrize("E,groups,keep,top", [(12, 4, 2, 3), (8, 0, 0, 2), (6, 6, 3, 2), (64, 8, 3, 6), (4, 1, 1, 4),
                                               (160, 8, 3, 8)])
def test_router_kernel(E, groups, keep, top):
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(E)
    T = 301
    z = (rng.standard_normal((T, E)) * 2).astype(np.float32)
    ids = torch.empty((T, top), dtype=torch.int32, device="cuda")
    wts = torch.empty((T, top), dtype=torch.float32, device="cuda")
    ops.moe_route(dev(z), groups, keep, top, 1.5, ids, wts)
    r = {"top": top, "scale": 1.5}
    if groups:
        r["groups"] = {"count": groups, "keep": keep}
    chosen, weight = P.grouped_router(z.astype(np.float64), np.eye(E), r)
    assert np.array_equal(ids.cpu().numpy(), chosen)
    assert np.max(np.abs(wts.cpu().numpy() - weight)) < 1e-6
    if groups > 1 and keep < groups and E // groups > 1:      # with one expert a group the rule cannot change a choice
        free, _ = P.grouped_router(z.astype(np.float64), np.eye(E), {"top": top, "scale": 1.5})
        assert (np.sort(free, -1) != np.sort(chosen, -1)).any(-1).mean() > 0.1, "the groups never decide in this test"


@pytest.mark.parametrize("own_tiles", [False, True])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,ff,E,groups,keep,top,T", [(40, 24, 6, 3, 2, 2, 9), (64, 64, 8, 0, 0, 3, 150),
                                                       (128, 32, 16, 4, 2, 4, 300), (72, 20, 5, 0, 0, 1, 70)])
def test_routed_experts_part(dtype, H, ff, E, groups, keep, top, T, own_tiles, monkeypatch):
    """``own_tiles``: many tokens in bfloat16 through the mma.sync tiles instead of the tcgen05 products (the other
    cases take the same kernels either way)."""
    from mlxforge_b200.csrc import binding
    from mlxforge_b200.engine.runtime import Runtime
    if own_tiles and (dtype != "bfloat16" or T < 64 or H % 8 or ff % 8):
        pytest.skip("the path does not differ here")
    monkeypatch.setenv("MLXFORGE_MOE_TILES", "1" if own_tiles else "0")
    before = binding.kernel_launches()
    from mlxforge_b200.parts.base import FEED_FORWARDS, PartSpec, build_part
    rng = np.random.default_rng(H + T)
    params = {"hidden_size": H, "intermediate_size": ff, "n_experts": E, "top": top, "n_groups": groups,
              "keep_groups": keep, "route_scale": 1.3, "limit": 0.8}
    part = build_part(FEED_FORWARDS, PartSpec("routed_experts", params, prefix="f."), Runtime(tdt(dtype)))
    w = {n: rand(rng, *s.shape, std=(4.0 if n.endswith("router") else 1.5) / np.sqrt(s.shape[1]))
         for n, s in part.tensor_specs().items()}
    part.bind({n: dev(a) for n, a in w.items()})
    x = rand(rng, T, H)
    p = {"expert": {"limit": 0.8}, "router": {"top": top, "scale": 1.3}}
    if groups:
        p["router"]["groups"] = {"count": groups, "keep": keep}
    f = {k[2:]: v.astype(np.float64) for k, v in w.items()}
    want = P.moe(x.astype(np.float64), p, f.get)
    got = host(part.forward(dev(x, tdt(dtype)), None))
    # a token whose choice hangs on a close call may differ in bfloat16 (the router reads the same
    # bfloat16 inputs, so here it does not); all others must agree
    assert np.max(np.abs(got - want)) < tol(dtype, np.abs(want).max())
    ran = {k: v - before[k] for k, v in binding.kernel_launches().items() if v - before[k]}
    if dtype == "bfloat16" and T >= 64 and H % 8 == 0 and ff % 8 == 0:
        assert ran.get("moe_grouped", 0) == 2 and ran.get("moe_sort", 0) == 1, ran
        assert ran.get("moe_grouped_tc", 0) == (0 if own_tiles else 2), ran
    else:
        assert ran.get("moe_rows", 0) == 1, ran
    # each token alone gives the same as inside the batch
    alone = host(part.forward(dev(x[7:8], tdt(dtype)), None))
    assert np.max(np.abs(alone[0] - got[7])) < (1e-5 if dtype == "float32" else 2e-2) * max(1.0, np.abs(want).max())


# ----------------------------------------------------------------------------- whole models through the replayer

REQUEST_LENGTHS = {"A": [1, 9, 40, 75, 131, 58], "B": [2, 17, 33, 64, 100], "C": [300, 45, 520, 203]}
PORTIONS = {"A": (7, 2, 5, 3, 2, 11, 4, 2, 16, 1, 9), "B": (7, 2, 5, 3, 2, 11, 4, 2, 16, 1, 9),
            "C": (150, 2, 129, 7, 64, 3, 131, 200)}
PEAKED = {"A": 6.0, "B": 6.0, "C": 3.0}


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("notirax")
    out = {}
    for which in CONFIGS:
        for peaked in (False, True):
            d, cfg, w = make_model(tmp, which, seed=ord(which), qk_gain=PEAKED[which] if peaked else 1.0)
            reqs = {f"r{i}": prompt(cfg, n, i) for i, n in enumerate(REQUEST_LENGTHS[which])}
            expected = {rid: P.forward(cfg, w, toks) for rid, toks in reqs.items()}
            P.ROUND = P.round_bf16
            try:
                noise = max(float(np.max(np.abs(P.forward(cfg, w, toks) - expected[rid]))) for rid, toks in reqs.items())
            finally:
                P.ROUND = None
            scale = max(float(np.max(np.abs(e))) for e in expected.values())
            out[(which, peaked)] = (d, cfg, reqs, expected, {"float32": 1e-4 * max(1.0, scale), "bfloat16": 3.0 * noise}, w)
    return out


def _replay(model_dir, dtype, trace, tmp_path, max_tokens=None, max_seqs=4):
    from mlxforge_b200.csrc import binding
    from mlxforge_b200.engine.replay import make_runner, replay
    runner = make_runner(model_dir, dtype, max_tokens or trace.live_tokens_rounded(), max_seqs=max_seqs)
    for pool in runner.cache._k + runner.cache._v + runner.cache._state:
        pool.fill_(float("nan"))
    out_dir = str(tmp_path / "out")
    before = binding.kernel_launches()
    replay(runner, trace.lines(), out_dir, done=io.StringIO())
    runner.cache.check()
    assert runner.cache.free_pages() == runner.cache.total_pages() and runner.cache.slots.n_free == max_seqs
    ran = {k: v - before[k] for k, v in binding.kernel_launches().items() if v - before[k]}
    return out_dir, ran


def _check(models, which, peaked, dtype, trace, tmp_path, **kw):
    d, cfg, reqs, expected, tols, _ = models[(which, peaked)]
    out_dir, ran = _replay(d, dtype, trace, tmp_path, **kw)
    got = TT.read_outputs(trace, out_dir, cfg["vocab"])
    assert got, "the trace asked for nothing"
    worst, where = TT.worst(got, expected)
    assert worst <= tols[dtype], (which, peaked, dtype, worst, tols[dtype], where, TT.first_bad(got, expected, tols[dtype]))
    return ran


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("peaked", [False, True])
@pytest.mark.parametrize("which", list(CONFIGS))
def test_whole_prompts_and_decoded_tails(models, which, peaked, dtype, tmp_path):
    reqs = models[(which, peaked)][2]
    _check(models, which, peaked, dtype, TT.whole(reqs), tmp_path)
    _check(models, which, peaked, dtype, TT.decode_tail(reqs, tail=32), tmp_path / "tail")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("which", list(CONFIGS))
def test_portions_down_to_two_tokens(models, which, dtype, tmp_path):
    reqs = models[(which, True)][2]
    _check(models, which, True, dtype, TT.portions(reqs, PORTIONS[which]), tmp_path)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("which", list(CONFIGS))
def test_mixed_batches_on_a_pool_where_pages_and_slots_are_used_again(models, which, dtype, tmp_path):
    reqs = models[(which, True)][2]
    trace = TT.mixed(reqs, max_live=3, seed=3, decode_last=6, max_portion=9 if which != "C" else 140)
    assert trace.live_tokens_rounded() < sum((len(t) + 63) // 64 * 64 for t in reqs.values())
    _check(models, which, True, dtype, trace, tmp_path, max_seqs=3)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("which", ["A", "B"])
def test_every_request_decoded_from_its_first_token(models, which, dtype, tmp_path):
    """Long decoding in a batch that shrinks: the first tokens of a sequence, chunk edges and page
    borders met token by token, decode steps replayed from graphs."""
    reqs = models[(which, False)][2]
    _check(models, which, False, dtype, TT.lockstep(reqs), tmp_path, max_seqs=len(reqs))


@pytest.mark.parametrize("own_tiles", [False, True])
def test_serving_shapes_take_the_fast_kernels(models, tmp_path, own_tiles, monkeypatch):
    """Configuration C in bfloat16: which kernels its prompts and its decoding go through, with the experts of
    many tokens through the tcgen05 products and through the mma.sync tiles."""
    monkeypatch.setenv("MLXFORGE_MOE_TILES", "1" if own_tiles else "0")
    reqs = models[("C", False)][2]
    ran = _check(models, "C", False, "bfloat16", TT.decode_tail(reqs, tail=8), tmp_path)
    for k in ("hyper_norm", "delta_recurrence", "moe_route", "embed_positions", "kv_store"):
        assert ran.get(k, 0) > 0, (k, ran)
    assert ran.get("attn_talking_tc", 0) > 0 and ran.get("attn_talking_merge", 0) > 0, ran
    assert ran.get("moe_grouped", 0) > 0 and ran.get("moe_rows", 0) > 0, ran
    assert (ran.get("moe_grouped_tc", 0) > 0) != own_tiles, ran


# ----------------------------------------------------------------------------- generation through the entry point

@pytest.mark.parametrize("which", ["A", "C"])
def test_greedy_generation_through_the_engine(models, which):
    import mlxforge_b200 as mf
    d, cfg, reqs, expected, _, w = models[(which, False)]
    prompts = [reqs["r2"], reqs["r1"], reqs["r3"][:50]]
    # portions of at most 16 tokens under a budget of 24: prompts are cut and run beside decoding
    eng = mf.Engine(model_spec=d, dtype="float32", kv_pool_tokens=1024, prefill_chunk=16, token_budget=24, max_running=4)
    got = eng.generate(prompts, max_tokens=6)
    clear = agree = 0
    for p, g in zip(prompts, got):
        seq = list(p)
        for t in g:
            row = P.forward(cfg, w, seq)[-1]
            top2 = np.sort(row)[-2:]
            if top2[1] - top2[0] > 1e-3:
                clear += 1
                agree += int(t == int(np.argmax(row)))
            seq.append(t)
    assert clear >= 10 and agree == clear, (got, clear, agree)
    assert eng.metrics()["completed"] == 3
    eng16 = mf.Engine(model_spec=d, dtype="bfloat16", kv_pool_tokens=1024, max_running=4)
    out16 = eng16.generate(prompts, max_tokens=6)
    assert all(len(o) == 6 for o in out16)


def test_cli_generate_and_trace_run_for_notirax(models, tmp_path, capsys):
    """The command line's own entry points: `generate` prints the plain implementation's greedy tokens, and the
    replayer's program (four slots unless told otherwise) writes the logits of a small trace."""
    from mlxforge_b200 import cli
    from mlxforge_b200.engine import replay as R
    d, cfg, reqs, expected, tols, w = models[("B", False)]
    prompt_ids = reqs["r2"][:20]
    capsys.readouterr()
    assert cli.main(["generate", d, ",".join(map(str, prompt_ids)), "5", "--dtype", "float32"]) == 0
    got = [int(t) for t in capsys.readouterr().out.split()]
    seq, want = list(prompt_ids), []
    for _ in range(5):
        row = P.forward(cfg, w, seq)[-1]
        want.append(int(np.argmax(row)))
        seq.append(want[-1])
    assert got == want, (got, want)
    trace = TT.mixed(reqs, max_live=4, seed=1, decode_last=4)
    out_dir = tmp_path / "out"
    import sys
    old = sys.stdin
    sys.stdin = trace.lines()
    try:
        assert R.main(["--model", d, "--dtype", "float32", "--out", str(out_dir), "--max-tokens",
                       str(trace.live_tokens_rounded())]) == 0
    finally:
        sys.stdin = old
    capsys.readouterr()
    worst, where = TT.worst(TT.read_outputs(trace, str(out_dir), cfg["vocab"]), expected)
    assert worst <= tols["float32"], (worst, where)


# ----------------------------------------------------------------------------- the delta rule over runs of tokens

@pytest.mark.parametrize("lens,heads,n_kv,dim,vdim,strong", [
    ([48], 1, 1, 64, 16, False), ([49, 1, 16, 17], 4, 2, 64, 48, True), ([95, 0, 2], 2, 2, 128, 128, False),
    ([64, 15], 6, 3, 128, 32, True), ([300], 10, 10, 128, 128, False),
])
def test_delta_runs_against_the_rule(lens, heads, n_kv, dim, vdim, strong):
    """Whole and broken runs, blocks of 8 and of 16 columns, sequences without a token, decays down to exp(-1000).
    A result is a chain of at most ~300 roundings of 2^-24, which add like a random walk: 1e-6 of the result's norm."""
    import torch
    from types import SimpleNamespace
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(len(lens) + dim)
    T, rep = sum(lens), heads // n_kv
    q, k = (a / np.linalg.norm(a, axis=-1, keepdims=True) for a in rng.standard_normal((2, T, n_kv, dim)))
    v = rng.standard_normal((T, heads, vdim))
    g = np.exp(-np.exp(3 * rng.standard_normal((T, heads, dim)))) if strong else np.exp(-0.1 * rng.random((T, heads, dim)))
    beta = rng.random((T, heads))
    state = 0.1 * rng.standard_normal((len(lens), heads * dim * vdim + 24))
    f32 = lambda a: a.astype(np.float32)
    qkv = f32(np.concatenate([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], axis=1))
    ag, b32, s32 = f32(np.concatenate([g.reshape(T, -1), rng.random((T, heads * vdim))], axis=1)), f32(beta), f32(state)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    starts = np.cumsum([0] + lens[:-1]).astype(np.int32)
    batch = SimpleNamespace(q_len=lens, n_seqs=len(lens), seq_q_start=dev(starts), seq_q_len=dev(np.array(lens, np.int32)),
                            slots=dev(np.arange(len(lens), dtype=np.int32)[::-1].copy()))
    runs, floats = ops.delta_runs(batch, heads, dim, vdim)
    assert runs == sum(-(-n // 16) for n in lens)
    st, o = dev(s32), torch.full((T, heads * vdim), float("nan"), device="cuda")
    ops.delta_recurrence_runs(dev(qkv), dev(b32), dev(ag), st, batch, o, heads, n_kv, dim, vdim, runs,
                              torch.full((floats,), float("nan"), device="cuda"))
    ops.check_kernel_status()
    got_o, got_s = o.cpu().numpy().astype(np.float64).reshape(T, heads, vdim), st.cpu().numpy()
    d = lambda a: a.astype(np.float64)
    qd = np.repeat(d(qkv[:, :n_kv * dim]).reshape(T, n_kv, dim), rep, axis=1)
    kd = np.repeat(d(qkv[:, n_kv * dim:2 * n_kv * dim]).reshape(T, n_kv, dim), rep, axis=1)
    vd, gd, bd = d(qkv[:, 2 * n_kv * dim:]).reshape(T, heads, vdim), d(ag[:, :heads * dim]).reshape(T, heads, dim), d(b32)
    for i, (t0, n) in enumerate(zip(starts, lens)):
        slot = len(lens) - 1 - i
        S = d(s32[slot, :heads * dim * vdim]).reshape(heads, dim, vdim)
        for t in range(t0, t0 + n):
            S = gd[t][:, :, None] * S
            u = bd[t][:, None] * (vd[t] - np.einsum("hdv,hd->hv", S, kd[t]))
            S = S + kd[t][:, :, None] * u[:, None]
            want = np.einsum("hdv,hd->hv", S, qd[t])
            assert np.linalg.norm(got_o[t] - want) < 1e-6 * max(np.linalg.norm(want), 1e-2)
        got = got_s[slot, :heads * dim * vdim].reshape(heads, dim, vdim)
        assert np.linalg.norm(got - S) < 1e-6 * np.linalg.norm(S)
    assert np.array_equal(got_s[:, heads * dim * vdim:], s32[:, heads * dim * vdim:]), "what stands behind S is not touched"


@pytest.mark.parametrize("lens,heads,n_kv,dim,vdim,taps", [
    ([255, 1, 2, 3], 2, 1, 128, 64, 4), ([100, 200], 3, 3, 64, 128, 3), ([1, 1, 1], 2, 2, 128, 128, 4), ([1, 2, 1], 4, 2, 64, 64, 2),
    ([300], 1, 1, 64, 64, 1),
])
def test_delta_prepare_by_heads(lens, heads, n_kv, dim, vdim, taps):
    """Runs of tokens over sequences' borders and beyond the last token, portions shorter than the history, the history
    moved on in the kernel (one token each) and behind it.  Convolution and SiLU to 2^-20 of the result, histories to the bit."""
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(sum(lens))
    T, C, n_low = sum(lens), 2 * n_kv * dim + heads * vdim, 12
    ld = C + heads + n_low + (-(C + heads + n_low) % 4)
    proj = rng.standard_normal((T, ld)).astype(np.float32)
    w = rng.standard_normal((C, taps)).astype(np.float32)
    state = rng.standard_normal((len(lens), 8 + (taps - 1) * C)).astype(np.float32)
    starts = np.cumsum([0] + lens[:-1])
    i32 = lambda a: dev(np.asarray(a, np.int32))
    batch = SimpleNamespace(q_len=lens, n_seqs=len(lens), positions=i32(np.zeros(T)), slots=i32(np.arange(len(lens))[::-1]),
                            seq_of_token=i32(np.repeat(np.arange(len(lens)), lens)), seq_q_start=i32(starts), seq_q_len=i32(lens))
    st, qkv, beta = dev(state), torch.full((T, C), np.nan, device="cuda"), torch.full((T, heads), np.nan, device="cuda")
    low = torch.full((T, n_low), np.nan, device="cuda")
    ops.delta_prepare(dev(proj), dev(w), taps, st, 8, batch, qkv, beta, low, heads, n_kv, dim, vdim)
    want_state = state.copy()
    for i, (t0, n) in enumerate(zip(starts, lens)):
        tail = state[len(lens) - 1 - i, 8:].reshape(taps - 1, C)
        rows = np.concatenate([tail, proj[t0:t0 + n, :C]]).astype(np.float64)
        want_state[len(lens) - 1 - i, 8:] = rows[n:].ravel()
        y = sum(rows[j:j + n] * w[:, j].astype(np.float64) for j in range(taps))
        y = y / (1 + np.exp(-y))
        qk = y[:, :2 * n_kv * dim].reshape(n, 2 * n_kv, dim)
        qk /= np.sqrt((qk * qk).sum(-1, keepdims=True) + 1e-6)
        qk[:, :n_kv] *= dim ** -0.5
        assert np.max(np.abs(host(qkv[t0:t0 + n]) - y)) < 2.0 ** -20 * max(1.0, np.abs(y).max())
    assert np.array_equal(st.cpu().numpy(), want_state)
    assert np.max(np.abs(host(beta) - 1 / (1 + np.exp(-proj[:, C:C + heads].astype(np.float64))))) < 2.0 ** -21
    assert np.array_equal(low.cpu().numpy(), proj[:, C + heads:C + heads + n_low])


@pytest.mark.parametrize("dim,vdim,taps", [(128, 128, 4), (64, 128, 3), (128, 64, 2), (64, 64, 1)])
def test_delta_prepare_in_runs_keeps_the_bits_of_single_tokens(dim, vdim, taps):
    """A step long enough for runs of eight tokens, its sequences' borders at every place of a run, against the same
    sequences a step each, short enough for one token at a time: the same sums in the same order, so the same bits."""
    import torch
    from mlxforge_b200.csrc import ops
    lens, heads, n_kv, n_low = [1, 2, 3, 4, 5, 6, 7, 9, 10, 220, 1, 200], 3, 1, 300
    gen = torch.Generator(device="cuda").manual_seed(dim + taps)
    T, C = sum(lens), 2 * n_kv * dim + heads * vdim
    ld = C + heads + n_low + (-(C + heads + n_low) % 4)
    proj, w = torch.randn((T, ld), generator=gen, device="cuda"), torch.randn((C, taps), generator=gen, device="cuda")
    state = torch.randn((len(lens), 8 + (taps - 1) * C), generator=gen, device="cuda")
    i32 = lambda a: dev(np.asarray(a, np.int32))

    def prepare(rows, own, st):
        n = sum(own)
        batch = SimpleNamespace(q_len=own, n_seqs=len(own), positions=i32(np.zeros(n)), slots=i32(np.arange(len(own))),
                                seq_of_token=i32(np.repeat(np.arange(len(own)), own)), seq_q_start=i32(np.cumsum([0] + own[:-1])),
                                seq_q_len=i32(own))
        out = [torch.full((n, m), float("nan"), device="cuda", dtype=t)
               for m, t in ((C, torch.float32), (heads, torch.float32), (n_low, torch.bfloat16))]
        ops.delta_prepare(rows, w, taps, st, 8, batch, *out, heads, n_kv, dim, vdim)
        return out

    st = state.clone()
    whole, at = prepare(proj, lens, st), 0
    for i, n in enumerate(lens):
        own = state[i:i + 1].clone()
        for a, b in zip(whole, prepare(proj[at:at + n], [n], own)):
            assert torch.equal(a[at:at + n], b)
        assert torch.equal(st[i:i + 1], own)
        at += n


@pytest.mark.parametrize("heads,kv,dim,vdim,chunk,window,cap,seqs", [
    (16, 4, 128, 128, 2048, 0, 30.0, [(17, 1100), (1, 700), (2, 18)]),       # key ranges cut at 512, a tile of one query
    (12, 3, 64, 96, 0, 600, 0.0, [(40, 900), (16, 16)]),                     # a window cut at 512; heads that are no power of two
    (8, 8, 16, 32, 33, 0, 5.0, [(70, 100), (1, 33), (1, 34)]),               # chunks that end inside a tile
    (5, 1, 48, 64, 0, 0, 20.0, [(31, 31), (1, 260)]),
    (16, 1, 32, 64, 0, 65, 30.0, [(1, 1), (1, 63), (1, 64), (1, 65), (1, 129)]),        # decoding: ends of a split, 16 heads on one
    (10, 5, 144, 128, 100, 0, 0.0, [(1, 99), (1, 100), (1, 101), (1, 200), (1, 1000)]),
    (12, 12, 16, 128, 0, 0, 10.0, [(1, 70), (1, 300)]),                      # values too wide for the decode kernel
])
def test_talking_kernels_mix_in_32_bits(heads, kv, dim, vdim, chunk, window, cap, seqs):
    """The tensor-core kernel against the block-per-token one with a mixing matrix of unit normals, so that scores of up to
    ~30 cancel: mixing them in bfloat16 would move a score by 0.1 and a weight by a tenth.  Both round their result to bfloat16 (2^-8 of
    it) and the first its weights (2^-9, averaged over the keys): 2^-6 of the largest result."""
    import torch
    from mlxforge_b200.csrc import ops
    from mlxforge_b200.engine.runtime import Runtime
    from mlxforge_b200.parts.talking_attention import talking_paged_attention
    rng = np.random.default_rng(heads)
    seqs = sorted(seqs, key=lambda s: s[0] != 1)
    page, T, bf = 16, sum(n for n, _ in seqs), torch.bfloat16
    blocks = [-(-c // page) for _, c in seqs]
    perm, at = rng.permutation(sum(blocks) + 2), 0
    table = np.full((len(seqs), max(blocks)), -1, np.int32)
    k, v = (np.full((len(perm), kv, page, d), np.nan, np.float32) for d in (dim, vdim))
    for i, (n, c) in enumerate(seqs):
        for b in range(blocks[i]):
            table[i, b], at, m = perm[at], at + 1, min(page, c - b * page)
            k[table[i, b], :, :m], v[table[i, b], :, :m] = rng.standard_normal((kv, m, dim)), rng.standard_normal((kv, m, vdim))
    i32 = lambda a: dev(np.asarray(a, np.int32))
    lens, ctx = [n for n, _ in seqs], [c for _, c in seqs]
    starts = np.cumsum([0] + lens[:-1])
    batch = SimpleNamespace(n_decode=sum(n == 1 for n in lens), n_tokens=T, max_ctx=max(ctx), q_len=lens, block_table=lambda g: dev(table),
                            seq_q_start=i32(starts), seq_q_len=i32(lens), seq_ctx_len=i32(ctx))
    lane = SimpleNamespace(group=0, k=dev(k, bf), v=dev(v, bf), page_size=page)
    m = SimpleNamespace(n_heads=heads, n_kv=kv, dim=dim, vdim=vdim, scale=dim ** -0.5 * 3, softcap=cap, window=window, chunk=chunk,
                        talk=dev(rng.standard_normal((heads, heads)).astype(np.float32) * 0.5))
    q = dev(rng.standard_normal((T, heads * dim)).astype(np.float32), bf)
    got, want = (torch.full((T, heads * vdim), float("nan"), device="cuda", dtype=bf) for _ in range(2))
    before = dict(ops_launches())
    talking_paged_attention(Runtime(bf), batch, q, lane, got, m)
    assert ops_launches()["attn_talking_tc"] > before["attn_talking_tc"]
    fits = kv * 64 * (vdim + 8) * 2 + heads * (68 * 4 + 72 * 2) <= 200 * 1024        # the values of a split of 64 keys, scores, weights
    decode = ops_launches()["attn_talking_decode"] - before["attn_talking_decode"]
    assert decode == (1 if batch.n_decode and fits else 0)
    pos = np.concatenate([np.arange(c - n, c) for n, c in seqs])
    ops.attention_talking(q, lane.k, lane.v, want, i32(pos), i32(np.repeat(np.arange(len(seqs)), lens)), dev(table), page, heads, kv,
                          dim, vdim, m.scale, cap, m.talk, window, chunk)
    assert torch.isfinite(want).all()
    assert (got.float() - want.float()).abs().max() < 2.0 ** -6 * want.float().abs().max()


def ops_launches():
    from mlxforge_b200.csrc import binding
    return binding.kernel_launches()


@pytest.mark.parametrize("T,H,ff,E,top,kind", [
    (70, 72, 40, 3, 2, None), (64, 128, 136, 5, 1, None), (600, 192, 264, 4, 3, None), (700, 64, 128, 2, 2, None),
    (100, 200, 88, 9, 4, "relu2"), (65, 2048, 768, 64, 6, None), (520, 136, 128, 1, 1, "silu"),
])
def test_sorted_experts_on_tcgen05(T, H, ff, E, top, kind):
    """Remainders of every tile (rows of the matrices, K steps, pairs), experts without a pair, with a few and with more than a
    unit holds, identity experts in between; both result types.  Sums of bfloat16 products in 32-bit, the activation rounded once: 2^-8 of
    a row's largest value, and the wide result to 2^-8 of what the rounded activations give."""
    import torch
    from mlxforge_b200.csrc import ops
    rng, bf = np.random.default_rng(T + E), torch.bfloat16
    x, wg = (dev(rng.standard_normal(s).astype(np.float32) * H ** -0.25, bf) for s in ((T, H), (E, 1 if kind else 2, ff, H)))
    wd = dev(rng.standard_normal((E, H, ff)).astype(np.float32) * ff ** -0.5, bf)
    skew = rng.random((T, E + 1)) ** np.linspace(0.2, 4, E + 1)                 # output E is an identity expert
    ids = np.argsort(-skew, axis=1)[:, :top].astype(np.int32)
    n, tile_rows = T * top, ops.moe_tc_rows()
    empty = lambda *s, t=torch.int32: torch.full(s, -7, dtype=t, device="cuda")
    slot, row_token, meta, tiles = empty(n), empty(n), empty(4), empty(3 * ops.moe_grouped_max_tiles(T, top, E))
    ops.moe_sort(dev(ids), E, slot, row_token, meta, tiles, tile_rows)
    slots, cuts = slot.cpu().numpy().reshape(T, top), tiles.cpu().numpy()[:3 * int(meta[0])].reshape(-1, 3)
    real = ids < E
    assert np.array_equal(np.sort(slots[real]), np.arange(real.sum())) and np.all(slots[~real] == -1)
    covered = np.concatenate([np.arange(r, r + k) for _, r, k in cuts])
    assert np.array_equal(covered, np.arange(real.sum())) and cuts[:, 2].max() <= tile_rows
    act = torch.full((n, ff), float("nan"), dtype=bf, device="cuda")
    ops.moe_tc_up(x, row_token, torch.empty((n, H), dtype=bf, device="cuda"), wg, meta, tiles, act, 1.5, 1.702, 1.0, kind)
    y16, y32 = (torch.full((n, H), float("nan"), dtype=t, device="cuda") for t in (bf, torch.float32))
    ops.moe_tc_down(act, wd, meta, tiles, y16)
    ops.moe_tc_down(act, wd, meta, tiles, y32)
    ops.check_kernel_status()
    for t in range(T):
        for k in range(top):
            e, r = ids[t, k], slots[t, k]
            if e == E:
                continue
            assert int(row_token[r]) == t if T < 100 else True
            p = [x[t].double() @ m.double().T for m in wg[e]]
            want = P_activation(p, kind)
            assert (act[r].double() - want).abs().max() < 2.0 ** -8 * max(want.abs().max(), 1e-2)
            down = act[r].double() @ wd[e].double().T
            assert (y32[r].double() - down).abs().max() < 2.0 ** -17 * max(down.abs().max(), 1e-2)
            assert (y16[r].double() - down).abs().max() < 2.0 ** -8 * max(down.abs().max(), 1e-2)


def P_activation(p, kind):
    if kind == "relu2":
        return p[0].clamp(min=0) ** 2
    if kind == "silu":
        return p[0].sigmoid() * p[0]
    g, u = p[0].clamp(max=1.5), p[1].clamp(-1.5, 1.5)
    return g * (1.702 * g).sigmoid() * (u + 1)


@pytest.mark.parametrize("n,heads,n_kv,dim,vdim", [(1, 1, 1, 64, 32), (5, 4, 2, 128, 96), (3, 2, 2, 128, 128), (2, 3, 1, 64, 160)])
def test_delta_step_against_the_rule(n, heads, n_kv, dim, vdim):
    """One token of every sequence: within 1e-6 of the rule in 64 bits (sums of at most 128 terms in 32-bit)."""
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(n + dim)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    qkv, beta, ag, state = f(n, 2 * n_kv * dim + heads * vdim), rng.random((n, heads)).astype(np.float32), rng.random((n, heads * dim + 4)).astype(np.float32), f(n, heads * dim * vdim + 8)
    qkv[:, :2 * n_kv * dim] *= dim ** -0.5
    i32 = lambda a: dev(np.asarray(a, np.int32))
    slots = np.arange(n)[::-1]
    st, o = dev(state), torch.full((n, heads * vdim), np.nan, device="cuda")
    batch = SimpleNamespace(q_len=[1] * n, n_seqs=n, seq_q_start=i32(np.arange(n)), seq_q_len=i32(np.ones(n)), slots=i32(slots))
    before = ops_launches()["delta_step"]
    ops.delta_recurrence(dev(qkv), dev(beta), dev(ag), st, batch, o, heads, n_kv, dim, vdim)
    assert ops_launches()["delta_step"] == before + 1
    d, rep = lambda a: a.astype(np.float64), heads // n_kv
    for t in range(n):
        q, k = (np.repeat(d(qkv[t, i * n_kv * dim:(i + 1) * n_kv * dim]).reshape(n_kv, dim), rep, axis=0) for i in (0, 1))
        v = d(qkv[t, 2 * n_kv * dim:]).reshape(heads, vdim)
        S = d(ag[t, :heads * dim]).reshape(heads, dim, 1) * d(state[slots[t], :heads * dim * vdim]).reshape(heads, dim, vdim)
        u = d(beta[t])[:, None] * (v - np.einsum("hdv,hd->hv", S, k))
        S = S + k[:, :, None] * u[:, None]
        want, got = np.einsum("hdv,hd->hv", S, q), host(o[t]).reshape(heads, vdim)
        assert np.linalg.norm(got - want) < 1e-6 * np.linalg.norm(S) / np.sqrt(dim)
        assert np.linalg.norm(host(st[slots[t], :heads * dim * vdim]).reshape(S.shape) - S) < 1e-6 * np.linalg.norm(S)
    assert np.array_equal(st[:, heads * dim * vdim:].cpu().numpy(), state[:, heads * dim * vdim:])


@pytest.mark.parametrize("t,what", [(0, "v"), (5, "v"), (15, "k"), (16, "v"), (40, "g"), (62, "k"), (30, "q"), (33, "b")])
@pytest.mark.parametrize("dim,vdim,heads", [(128, 32, 2), (64, 64, 80)])
def test_delta_runs_keep_what_is_not_finite_from_earlier_tokens(t, what, dim, vdim, heads):
    """As for the retention's chunks: what is not finite at a token (of any operand) reaches neither the tokens before it, those of its
    own run of 16 among them, nor the other heads; blocks of 8 and of 16 columns."""
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(t)
    T, f = 63, lambda *s: rng.standard_normal(s).astype(np.float32)
    C = 2 * heads * dim + heads * vdim
    qkv, beta, ag, state = f(T, C), rng.random((T, heads)).astype(np.float32), rng.random((T, heads * dim)).astype(np.float32), f(1, heads * dim * vdim)
    qkv[:, :2 * heads * dim] *= dim ** -0.5
    i32 = lambda a: dev(np.asarray(a, np.int32))
    batch = SimpleNamespace(q_len=[T], n_seqs=1, seq_q_start=i32([0]), seq_q_len=i32([T]), slots=i32([0]))
    runs, floats = ops.delta_runs(batch, heads, dim, vdim)
    res = []
    for bad in (None, np.nan, np.inf):
        x, g, b = qkv.copy(), ag.copy(), beta.copy()
        if bad is not None:
            if what == "g":
                g[t, 7] = bad
            elif what == "b":
                b[t, 0] = bad
            else:
                x[t, {"q": 0, "k": heads * dim, "v": 2 * heads * dim}[what] + 3] = bad
        st, o = dev(state), torch.full((T, heads * vdim), float("nan"), device="cuda")
        ops.delta_recurrence_runs(dev(x), dev(b), dev(g), st, batch, o, heads, heads, dim, vdim, runs, torch.empty(floats, device="cuda"))
        res.append(o)
    ops.check_kernel_status()
    for o in res[1:]:
        assert torch.equal(o[:t], res[0][:t])
        assert not torch.isfinite(o[t]).all()
        assert torch.equal(o[:, vdim:], res[0][:, vdim:])


RECURRENT = {
    "channel_delta": {"n_kv_heads": 2, "conv": 4, "decay_rank": 16, "gate_rank": 16},
    "retention": {"rotary_dim": 128, "rope_base": 1e4, "decay": [0.97, 0.999]},
}


def recurrent_part(kind, rt, rng, hidden=64):
    """A mixer with a state, two heads of 128 channels."""
    from mlxforge_b200.parts.base import MIXERS, PartSpec, build_part
    part = build_part(MIXERS, PartSpec(kind, dict(RECURRENT[kind], hidden_size=hidden, n_heads=2, head_dim=128, eps=1e-6), "m."), rt)
    part.bind({n: dev(rand(rng, *s.shape, std=s.shape[-1] ** -0.5)) for n, s in part.tensor_specs().items()})
    return part


def recurrent_runner(part, n):
    """A runner over ``n`` open sequences with states drawn from one seed."""
    from mlxforge_b200.cache.manager import CacheLayout, CacheManager, GroupLayout
    from mlxforge_b200.engine.step import ModelRunner
    layout = CacheLayout(paged=(), state=(GroupLayout(part.cache_need(), 1),), item_lane=(("state", 0, 0),))
    cache = CacheManager(layout, page_size=16, max_tokens=64, max_seqs=n, dtype=part.rt.dtype, device="cuda")
    seqs, states = [cache.open_sequence() for _ in range(n)], cache.lane(0).tensor
    rng = np.random.default_rng(n)
    for s in seqs:
        states[s.slot] = dev(rng.standard_normal(states.shape[1]).astype(np.float32))
    stub = SimpleNamespace(graph_safe=False, spec=SimpleNamespace(vocab_size=1 << 20))
    return ModelRunner(stub, cache, part.rt), seqs, states


@pytest.mark.parametrize("kind", list(RECURRENT))
def test_a_sequence_has_the_same_bits_alone_and_beside_others(kind):
    """Single tokens, portions that go token after token and portions that go over runs or chunks, in one step and each in a step of
    its own: outputs and states to the bit (float32)."""
    import torch
    from mlxforge_b200.engine.runtime import Runtime
    from mlxforge_b200.engine.step import StepEntry
    lens = [1, 300, 40, 1, 20, 700, 90, 64, 48, 130, 257]          # enough behind one another for blocks of 16 columns
    rng = np.random.default_rng(0)
    part = recurrent_part(kind, Runtime(torch.float32), rng)
    xs, results = [rand(rng, n, 64) for n in lens], []
    for steps in ([range(len(lens))], [[i] for i in range(len(lens))]):
        runner, seqs, states = recurrent_runner(part, len(lens))
        got = [None] * len(lens)
        for step in steps:
            entries = [StepEntry(seqs[i], [0] * lens[i], []) for i in step]
            runner.cache.reserve([(e.seq, len(e.tokens)) for e in entries])
            order = sorted(step, key=lambda i: (lens[i] != 1, i))
            out, at = part.forward(dev(np.concatenate([xs[i] for i in order])), runner._build(entries), runner.cache.lane(0)), 0
            for i in order:
                got[i], at = out[at:at + lens[i]].clone(), at + lens[i]
        results.append((got, [states[s.slot].clone() for s in seqs]))
    (together, s_together), (alone, s_alone) = results
    differ = [lens[i] for i in range(len(lens)) if not (torch.equal(together[i], alone[i]) and torch.equal(s_together[i], s_alone[i]))]
    assert not differ, differ


@pytest.mark.parametrize("kind", list(RECURRENT))
def test_scratch_of_runs_and_chunks_does_not_move_within_the_token_budget(kind):
    """A buffer that moves makes every captured decode graph void: the first long portion makes room for all that the budget allows."""
    import torch
    from mlxforge_b200.engine.runtime import Runtime
    from mlxforge_b200.engine.step import StepEntry
    rt = Runtime(torch.bfloat16)
    rt.reserve_rows = 2048
    part = recurrent_part(kind, rt, np.random.default_rng(0))
    seen = []
    for lens in ([300], [1, 40], [2048], [48] * 42, [257] * 7 + [1] * 3, [600, 1400]):
        runner, seqs, _ = recurrent_runner(part, len(lens))
        entries = [StepEntry(s, [0] * n, []) for s, n in zip(seqs, lens)]
        runner.cache.reserve([(e.seq, len(e.tokens)) for e in entries])
        part.forward(dev(rand(np.random.default_rng(1), sum(lens), 64), torch.bfloat16), runner._build(entries), runner.cache.lane(0))
        seen.append(rt.generation)
    assert len(set(seen)) == 1, seen


def test_delta_prepare_takes_a_sequence_without_a_token_beside_single_ones():
    """Its history stays as it is, the others' move on."""
    import torch
    from mlxforge_b200.csrc import ops
    rng = np.random.default_rng(3)
    lens, heads, dim, taps = [1, 0, 1], 2, 64, 4
    C = 3 * heads * dim
    proj, w = rng.standard_normal((2, C + 4)).astype(np.float32), rng.standard_normal((C, taps)).astype(np.float32)
    state = rng.standard_normal((3, 3, C)).astype(np.float32)
    i32 = lambda a: dev(np.asarray(a, np.int32))
    batch = SimpleNamespace(q_len=lens, n_seqs=3, positions=i32([0, 0]), slots=i32([2, 1, 0]), seq_of_token=i32([0, 2]),
                            seq_q_start=i32([0, 1, 1]), seq_q_len=i32(lens))
    st, qkv, beta, low = dev(state.reshape(3, -1)), *(torch.empty((2, n), device="cuda") for n in (C, heads, 2))
    ops.delta_prepare(dev(proj), dev(w), taps, st, 0, batch, qkv, beta, low, heads, heads, dim, dim)
    for slot, t in ((2, 0), (0, 1)):
        state[slot] = np.concatenate([state[slot, 1:], proj[t:t + 1, :C]])
    assert np.array_equal(st.cpu().numpy(), state.reshape(3, -1)) and torch.isfinite(qkv).all()


@pytest.mark.parametrize("gemm", ["auto", "tcgen05"])
def test_the_type_of_an_experts_result(gemm):
    """32-bit in every step that decodes, recorded or not, of few tokens or many, and for prompts too with the ``tcgen05`` backend:
    a token's result then has the same bits in a step of 511 tokens and of 600, and in a replayed one."""
    import torch
    from mlxforge_b200.engine.runtime import Runtime
    from mlxforge_b200.parts.base import FEED_FORWARDS, PartSpec, build_part
    rng, rt = np.random.default_rng(0), Runtime(torch.bfloat16)
    rt.gemm_backend = gemm
    part = build_part(FEED_FORWARDS, PartSpec("routed_experts", {"hidden_size": 128, "intermediate_size": 64, "n_experts": 8, "top": 4,
                                                                "n_groups": 0, "keep_groups": 0, "limit": 7.0}, prefix="f."), rt)
    part.bind({n: dev(rand(rng, *s.shape, std=s.shape[-1] ** -0.5)) for n, s in part.tensor_specs().items()})
    x = dev(rand(rng, 600, 128), torch.bfloat16)
    decode = lambda n: SimpleNamespace(n_decode=n) if gemm == "auto" else None
    few, many = part.forward(x[:511], decode(511)).clone(), part.forward(x, decode(600)).clone()
    prompt = part.forward(x, SimpleNamespace(n_decode=0)).clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = part.forward(x, decode(600))
    graph.replay()
    assert torch.equal(few, many[:511]) and torch.equal(out, many)
    assert torch.equal(prompt, many) == (gemm == "tcgen05")


def talking_case(seqs, heads, kv, k, v, q, scale, talk=None):
    """(tensor-core kernels, block-per-token kernel) [T, heads, vdim] over sequences of (new tokens, context) with the keys and values
    k[i], v[i] [context, kv, .]."""
    import torch
    from mlxforge_b200.csrc import ops
    from mlxforge_b200.engine.runtime import Runtime
    from mlxforge_b200.parts.talking_attention import talking_paged_attention
    bf, page, T, dim, vdim = torch.bfloat16, 16, sum(n for n, _ in seqs), k[0].shape[2], v[0].shape[2]
    blocks = [-(-c // page) for _, c in seqs]
    table, at = np.full((len(seqs), max(blocks)), -1, np.int32), 0
    kp, vp = (np.zeros((sum(blocks), kv, page, d), np.float32) for d in (dim, vdim))
    for i, (n, c) in enumerate(seqs):
        for b in range(blocks[i]):
            table[i, b], m = at, min(page, c - b * page)
            kp[at, :, :m], vp[at, :, :m] = (x[i][b * page:b * page + m].transpose(1, 0, 2) for x in (k, v))
            at += 1
    i32 = lambda a: dev(np.asarray(a, np.int32))
    lens, ctx = [n for n, _ in seqs], [c for _, c in seqs]
    starts = np.cumsum([0] + lens[:-1])
    batch = SimpleNamespace(n_decode=sum(n == 1 for n in lens), n_tokens=T, max_ctx=max(ctx), q_len=lens, block_table=lambda g: dev(table),
                            seq_q_start=i32(starts), seq_q_len=i32(lens), seq_ctx_len=i32(ctx))
    lane = SimpleNamespace(group=0, k=dev(kp, bf), v=dev(vp, bf), page_size=page)
    m = SimpleNamespace(n_heads=heads, n_kv=kv, dim=dim, vdim=vdim, scale=scale, softcap=0.0, window=0, chunk=0, talk=talk)
    got, want = (torch.full((T, heads * vdim), float("nan"), device="cuda", dtype=bf) for _ in range(2))
    talking_paged_attention(Runtime(bf), batch, dev(q.reshape(T, -1), bf), lane, got, m)
    pos = np.concatenate([np.arange(c - n, c) for n, c in seqs])
    ops.attention_talking(dev(q.reshape(T, -1), bf), lane.k, lane.v, want, i32(pos), i32(np.repeat(np.arange(len(seqs)), lens)), dev(table),
                          page, heads, kv, dim, vdim, scale, 0.0, talk, 0, 0)
    return host(got).reshape(T, heads, vdim), host(want).reshape(T, heads, vdim)


@pytest.mark.parametrize("seqs", [[(1, 300)], [(2, 300)], [(16, 2000)]])
@pytest.mark.parametrize("base", [3.0, 2.0 ** 20])
def test_talking_weights_of_large_scores(seqs, base):
    """Scores of base + j / 4 (exact in every type used), the maximum rising from tile to tile: however large they are, a weight is
    e^(j / 4).  Weights and results are rounded to bfloat16 (2^-8 each); a maximum rounded in one place and not in another moves a weight
    by up to 2^-4.5 at the larger base."""
    heads, kv, dim, vdim = 2, 1, 16, 32
    n, c = seqs[0]
    k, v, q = np.zeros((c, kv, dim), np.float32), np.zeros((c, kv, vdim), np.float32), np.zeros((n, heads, dim), np.float32)
    k[:, 0, 0], k[:, 0, 1], q[:, :, :2] = base, np.arange(c) // 32 % 8 * 0.25, 1.0
    v[np.arange(c), 0, np.arange(c) // 32 % vdim] = 1.0
    got, other = talking_case(seqs, heads, kv, [k], [v], q, 1.0)
    for i in range(n):
        p = np.exp(k[:c - n + 1 + i, 0, 1].astype(np.float64))
        want = p @ v[:c - n + 1 + i, 0].astype(np.float64) / p.sum()
        assert np.all(np.abs(got[i] - want) <= 2.0 ** -7 * 1.02 * want) and np.all(np.abs(other[i] - want) <= 2.0 ** -8 * 1.02 * want)


@pytest.mark.parametrize("seqs", [[(1, 200)], [(20, 200)]])
@pytest.mark.parametrize("heads,kv", [(4, 2), (16, 4)])
def test_talking_heads_without_a_mixing_matrix_stay_apart(heads, kv, seqs):
    """A query that is not finite in one head leaves the others as they are."""
    rng = np.random.default_rng(0)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    k, v, q = f(200, kv, 64), f(200, kv, 64), f(seqs[0][0], heads, 64)
    clean, _ = talking_case(seqs, heads, kv, [k], [v], q, 0.125)
    q[:, 1, 5] = np.nan
    got, want = talking_case(seqs, heads, kv, [k], [v], q, 0.125)
    others = np.arange(heads) != 1
    assert np.isfinite(want[:, others]).all() and np.array_equal(got[:, others], clean[:, others])
    assert not np.isfinite(want[:, 1]).any() and not np.isfinite(got[:, 1]).any()
