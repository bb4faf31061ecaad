"""Each mechanism that the Sonalorn design brought, alone, against the plain
implementation's function for it: the stream's sum through an output norm and a
per-channel scale, the embedding with learned positions, the gated delta rule
(state carried over steps, slots used again, planted far keys), the routed
feed-forward (choice by groups with corrected scores, pass-through experts,
clamps), attention with values of another size, a query temperature and a sink of
logit zero."""
import math

import pytest
import torch

from plain import sonalorn as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.float32: dict(atol=3e-5, rtol=3e-4), torch.bfloat16: dict(atol=0.03, rtol=0.03)}


def close(got, want, dtype, what=""):
    got, want = got.detach().double().cpu(), want.detach().double().cpu()
    assert got.shape == want.shape, (what, got.shape, want.shape)
    err = (got - want).abs()
    bound = TOL[dtype]["atol"] + TOL[dtype]["rtol"] * want.abs()
    assert bool((err <= bound).all()), f"{what}: max err {err.max().item():.3g} at {int(err.argmax())}"


def rnd(*shape, seed=0, scale=1.0, dtype=torch.float32):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype)


class Step:
    """The fields of a step that the kernels read, for sequences given as (slot, start, n)."""

    def __init__(self, seqs):
        from grout_b200.engine.batch import make_context
        self.ctx = make_context([(s, st, [0] * n) for s, st, n in seqs], None, DEV)


# ------------------------------------------------------------------ the stream's sum
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N", [24, 320, 1000, 5120])
def test_stream_sum_through_norm_and_scale(dtype, N):
    from grout_b200.kernels import ops
    T = 7
    res, d = rnd(T, N, seed=1, scale=3.0), rnd(T, N, seed=2, scale=0.2).to(dtype)
    pw, sc, w = 1 + rnd(N, seed=3, scale=0.2), rnd(N, seed=4), 1 + rnd(N, seed=5, scale=0.2)
    c = plain.rms_norm(d, pw, 1e-5) * sc.double()
    want_res = res.double() + c
    g = lambda t: t.to(DEV)
    r, y = ops.add_postnorm(g(res).clone(), g(d), dtype=dtype, post_weight=g(pw), post_eps=1e-5, scale=g(sc))
    close(r, want_res, torch.float32, "stream")
    close(y, want_res, dtype, "the stream as the next sublayer reads it")
    rows = torch.tensor([5, 0, 5], dtype=torch.int32)
    r2, y2 = ops.add_postnorm(g(res).clone(), g(d), dtype=dtype, post_weight=g(pw), post_eps=1e-5,
                              scale=g(sc), weight=g(w), eps=1e-6, rows=g(rows))
    close(r2, want_res[rows.long()], torch.float32, "gathered rows")
    close(y2, plain.rms_norm(want_res[rows.long()], w, 1e-6), dtype, "final norm of gathered rows")
    parts = torch.stack([d.float() * 0.25, d.float() * 0.5, d.float() * 0.25]).contiguous()
    r3, _ = ops.add_postnorm(g(res).clone(), g(parts), dtype=dtype, post_weight=g(pw), post_eps=1e-5, scale=g(sc))
    close(r3, want_res, torch.float32, "partial sums")
    r4, y4 = ops.add_postnorm(g(res).clone(), None, dtype=dtype)
    assert torch.equal(r4.cpu(), res) and torch.equal(y4.cpu(), res.to(dtype))
    r5, _ = ops.add_postnorm(None, g(d), dtype=dtype)                 # nothing but the delta
    close(r5, d.double(), torch.float32, "delta alone")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,S", [(4, 1), (1001, 2), (4096, 5), (4100, 9), (8196, 3), (12288, 5), (16384, 4), (16388, 2)])
def test_stream_sum_at_the_widths_where_its_kernel_changes(N, S, dtype):
    from grout_b200.kernels import ops
    res, parts = rnd(3, N, seed=1), rnd(S, 3, N, seed=2)
    pw, w = 1 + rnd(N, seed=3, scale=0.2), 1 + rnd(N, seed=4, scale=0.2)
    want = res.double() + plain.rms_norm(parts.double().sum(0), pw, 1e-5)
    r, y = ops.add_postnorm(res.to(DEV), parts.to(DEV), dtype=dtype, post_weight=pw.to(DEV), post_eps=1e-5,
                            weight=w.to(DEV), eps=1e-6)
    close(r, want, torch.float32, "stream")
    close(y, plain.rms_norm(want, w, 1e-6), dtype, "its norm")


def _just_computed(vectors, call):
    """``call()`` eight times, each right behind the kernels that write ``vectors`` and let their successor in on entry:
    waited for one by one, then in one graph, with the same bits."""
    from grout_b200.kernels import ops
    first = [v.clone() for v in vectors]

    def play(wait):
        out = []
        for i in range(8):
            for v in vectors:
                ops.scale_softcap_(v, 0.5 + 0.25 * i, None)
            if wait:
                torch.cuda.synchronize()
            out += call()
        return out

    want, graph = play(True), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got = play(False)
    for v, f in zip(vectors, first):
        v.copy_(f)
    graph.replay()
    assert len(got) == len(want) and all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("N", [1001, 2048, 8192, 10240])
def test_stream_sum_with_vectors_that_were_just_computed(N):
    from grout_b200.kernels import ops
    res, d = rnd(3, N, seed=1).to(DEV), rnd(3, N, seed=2).to(DEV)
    vectors = [(1 + rnd(N, seed=3 + i, scale=0.2)).to(DEV) for i in range(3)]
    rows = torch.arange(3, dtype=torch.int32, device=DEV)
    for on in ([vectors[0]], [vectors[1]], [vectors[2]], vectors):
        _just_computed(on, lambda: ops.add_postnorm(res, d, dtype=torch.float32, rows=rows, post_weight=vectors[0],
                                                    post_eps=1e-5, scale=vectors[1], weight=vectors[2], eps=1e-6))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_with_positions(dtype):
    from grout_b200.kernels import ops
    V, P, H = 37, 50, 72
    table, pos, w = rnd(V, H, seed=1).to(dtype), rnd(P, H, seed=2).to(dtype), 1 + rnd(H, seed=3, scale=0.1)
    ids = torch.tensor([3, 36, 0, 3], dtype=torch.int32)
    tp = torch.tensor([0, 49, 7, 8], dtype=torch.int32)
    got = ops.embed_pos_norm(table.to(DEV), pos.to(DEV), ids.to(DEV), tp.to(DEV), w.to(DEV), 1e-5)
    x = table.double()[ids.long()] + pos.double()[tp.long()]
    close(got, plain.rms_norm(x, w, 1e-5), torch.float32)            # 32-bit whatever the tables' type


def test_gelu_tanh_gate():
    from grout_b200.kernels import ops
    gu = rnd(5, 2 * 24, seed=1, scale=2.0)
    got = ops.gelu_tanh_mul(gu.to(DEV), 0)
    close(got, plain.gelu_tanh(gu[:, :24].double()) * gu[:, 24:].double(), torch.float32)


@pytest.mark.parametrize("rows", [3, 64, 300])
def test_gelu_tanh_gate_as_the_products_epilogue(rows):
    """The gated feed-forward part in bfloat16: a decode step's product and a prompt's
    apply the gate's activation before they store (gate and up rows interleaved in eights);
    all product choices give the plain result."""
    from grout_b200.parts import BuildContext, PartSpec, ProductChoice, build_part
    W, F = 64, 96
    w = {"gate": rnd(F, W, seed=1, scale=0.3).bfloat16(), "up": rnd(F, W, seed=2, scale=0.3).bfloat16(),
         "down": rnd(W, F, seed=3, scale=0.2).bfloat16()}
    x = rnd(rows, W, seed=4).bfloat16()
    want = plain.dense_ff(x, {"m." + k: v for k, v in w.items()}, "m.")
    for choice in (ProductChoice("tc", "auto"), ProductChoice("tc", "pair"), ProductChoice("skinny", "library")):
        part = build_part("feedforward", PartSpec("gated_mlp", dict(
            hidden=W, intermediate=F, activation="gelu_tanh", names={"gate": "gate", "up": "up", "down": "down"})),
            BuildContext(torch.bfloat16, torch.device(DEV), choice))
        part.load({k: v.to(DEV) for k, v in w.items()})
        assert part.interleave == 8
        got = part.forward(x.to(DEV), None)
        got = (got.sum(0) if got.dim() == 3 else got).double().cpu()
        # the unfused path rounds gate and up before the activation: a bar on the whole
        assert float((got - want).pow(2).mean().sqrt() / want.pow(2).mean().sqrt()) < 0.02, (rows, choice)


# ------------------------------------------------------------------ the gated delta rule
def _delta_weights(H, G, dk, dv, taps, W, seed, slow=True):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s, sc=1.0: torch.randn(*s, generator=g) * sc
    w = {"q": r(G * dk, W, sc=0.3), "k": r(G * dk, W, sc=0.3), "v": r(H * dv, W, sc=0.3),
         "g": r(H * dv, W, sc=0.3), "b": r(H, W, sc=0.3), "a": r(H, W, sc=0.3),
         "q.conv": r(G * dk, taps, sc=0.6), "k.conv": r(G * dk, taps, sc=0.6), "v.conv": r(H * dv, taps, sc=0.6),
         # decays from "forgets at once" to "keeps for hundreds of tokens"
         "A_log": torch.linspace(-6.0 if slow else -1.0, 0.5, H), "dt_bias": r(H, sc=0.5),
         "norm": 1 + r(dv, sc=0.2), "o": r(W, H * dv, sc=0.2)}
    return w


def _delta_run(w, m, xs, cuts, dtype, state=None, slot=0, n_slots=3):
    """Feeds rows xs [T, W] through the kernels in steps of the given sizes."""
    from grout_b200.kernels import ops
    H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
    g = lambda t: t.float().to(DEV).contiguous()
    wp = torch.cat([w[k] for k in ("q", "k", "v", "g", "b", "a")], 0).double()
    conv = g(torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], 0))
    if state is None:
        state = torch.zeros(n_slots + 1, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV)
    outs, start = [], 0
    for n in cuts:
        step = Step([(slot, start, n)]).ctx
        proj = g(xs[start:start + n].double() @ wp.T)
        y = ops.delta_forward(proj, state, conv, g(w["A_log"]), g(w["dt_bias"]), g(w["norm"]), H=H, G=G,
                              dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5,
                              token_seq=step.token_seq, cu_q=step.cu_q, slots=step.slots, dtype=dtype)
        outs.append(y.float().cpu())
        start += n
    return torch.cat(outs), state


def _delta_plain(w, m, xs):
    W = dict({"m." + k: v for k, v in w.items()})
    W["m.o"] = torch.eye(m["heads"] * m["vdim"])          # the read-out before the o projection
    return plain.delta_mixer(xs, W, "m.", m, 1e-5)


DELTA_SHAPES = [dict(heads=4, kv_heads=2, dim=16, vdim=8, conv=3),
                dict(heads=3, kv_heads=3, dim=40, vdim=20, conv=4),     # sizes that fill no lane group
                dict(heads=2, kv_heads=1, dim=64, vdim=48, conv=2),
                dict(heads=2, kv_heads=2, dim=128, vdim=16, conv=1),    # no convolution to speak of
                dict(heads=2, kv_heads=1, dim=30, vdim=10, conv=5)]     # sizes that are no multiple of four


@pytest.mark.parametrize("m", DELTA_SHAPES)
def test_delta_rule_whole_in_portions_and_token_by_token(m):
    W, T = 24, 150
    w = _delta_weights(m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"], W, seed=3)
    xs = rnd(T, W, seed=4)
    want = _delta_plain(w, m, xs)
    whole, _ = _delta_run(w, m, xs, [T], torch.float32)
    close(whole, want, torch.float32, "whole")
    for cuts in ([2] * 75, [1] * T, [1, 2, 3, 100, 44], [149, 1]):
        got, _ = _delta_run(w, m, xs, cuts, torch.float32)
        # the same recurrence however the rows are cut (rows are walked in groups that
        # start where a step starts, so the rounding differs)
        assert float((got - whole).abs().max()) < 1e-5, cuts
    half, _ = _delta_run(w, m, xs, [T], torch.bfloat16)
    close(half, want, torch.bfloat16, "bfloat16 output")


@pytest.mark.parametrize("m", [dict(heads=2, kv_heads=2, dim=128, vdim=128, conv=4), DELTA_SHAPES[0], DELTA_SHAPES[1],
                               dict(heads=8, kv_heads=1, dim=64, vdim=48, conv=8), DELTA_SHAPES[3],
                               dict(heads=16, kv_heads=4, dim=12, vdim=128, conv=3),
                               dict(heads=2, kv_heads=1, dim=128, vdim=144, conv=2)])
def test_delta_rule_chunk_by_chunk_and_step_by_step(m, monkeypatch):
    """When the host knows how many rows a sequence brings at most, prompts go chunk by chunk (32 rows) and decode
    steps through one kernel: sequences of 1, 31, 32, 33, 64 and 100 rows in one step, a padding sequence and one
    without rows between them, go on with 3 decode steps.  Against the plain rule, and against the kernels that
    take any rows; strong and weak decays side by side; 32-bit sums of values of order one, a bar of 1e-5."""
    from grout_b200.kernels import ops
    monkeypatch.setattr(ops, "delta_chunks_pay", lambda T, n_seqs, max_rows: max_rows >= 64)
    H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
    W, lens, more = 24, [1, 31, 32, 33, 64, 100], 3
    w = _delta_weights(H, G, dk, dv, taps, W, seed=13)
    xs = [rnd(n + more, W, seed=14 + i) for i, n in enumerate(lens)]
    g = lambda t: t.float().to(DEV).contiguous()  # noqa: E731
    wp = torch.cat([w[k] for k in ("q", "k", "v", "g", "b", "a")], 0).double()
    conv = g(torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], 0))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731

    def play(known):
        state = torch.zeros(len(lens) + 1, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV)
        outs = [[] for _ in lens]

        def step(parts, max_rows):            # parts: (sequence or -1, rows [n, W])
            ns = [len(x) for _i, x in parts]
            y = ops.delta_forward(
                g(torch.cat([x for _i, x in parts]).double() @ wp.T), state, conv, g(w["A_log"]), g(w["dt_bias"]),
                g(w["norm"]), H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5, dtype=torch.float32,
                token_seq=i32([k for k, n in enumerate(ns) for _ in range(n)]),
                cu_q=i32([0] + torch.tensor(ns).cumsum(0).tolist()), slots=i32([i for i, _x in parts]),
                max_rows=max_rows if known else None).cpu()
            for (i, _x), rows in zip(parts, torch.split(y, ns)):
                if 0 <= i < len(lens):
                    outs[i].append(rows)

        firsts = [(i, x[:n]) for i, (n, x) in enumerate(zip(lens, xs))]
        step(firsts[:3] + [(-1, rnd(40, W, seed=1)), (6, xs[0][:0])] + firsts[3:], max(lens))
        for k in range(more):
            order = [5, 0, 3, 1, 4, 2]
            step([(i, xs[i][lens[i] + k:lens[i] + k + 1]) for i in order] + [(-1, xs[0][:1])], 1)
        assert float(state[6].abs().max()) == 0.0
        return [torch.cat(o) for o in outs], state

    got, state = play(True)
    old, old_state = play(False)
    for i, x in enumerate(xs):
        close(got[i], _delta_plain(w, m, x), torch.float32, str(lens[i]))
        # (a read-out is normalised and gated, which scales its rounding, some 1e-7 of its largest terms, up with it: the
        # bar goes with the largest value, which is beyond one)
        assert float((got[i] - old[i]).abs().max()) < 1e-5 * max(1.0, float(old[i].abs().max())), lens[i]
    assert float((state - old_state).abs().max()) < 1e-5 * max(1.0, float(old_state.abs().max()))


def _delta_in_64_bits(proj, lens, conv, a_log, dt_bias, norm, H, G, dk, dv, taps):
    """The rule on the projection's 32-bit sums, all in 64 bits: (read-outs, states [sequence, head, value, key])."""
    conv, a_log, dt_bias, norm = (t.double() for t in (conv, a_log, dt_bias, norm))
    Cc, outs, states = 2 * G * dk + H * dv, [], []
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    for x in torch.split(proj.double(), lens):
        n = len(x)
        c = sum(conv[:, j] * torch.cat([torch.zeros(taps - 1 - j, Cc).double(), x[:, :Cc]])[:n] for j in range(taps))
        q, k, v = torch.split(c * torch.sigmoid(c), [G * dk, G * dk, H * dv], 1)
        q, k = (unit(t.view(n, G, dk)).repeat_interleave(H // G, 1) for t in (q, k))
        v, gate, b, a = v.view(n, H, dv), x[:, Cc:Cc + H * dv].view(n, H, dv), x[:, -2 * H:-H], x[:, -H:]
        g = torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(a + dt_bias))
        S, o = torch.zeros(H, dv, dk).double(), torch.empty(n, H, dv).double()
        for t in range(n):
            S = S * g[t][:, None, None]
            u = torch.sigmoid(b[t])[:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None]
            o[t] = torch.einsum("hvk,hk->hv", S, q[t]) * dk ** -0.5
        y = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * norm * gate * torch.sigmoid(gate)
        outs.append(y.reshape(n, -1)), states.append(S)
    return torch.cat(outs), torch.stack(states)


@pytest.mark.parametrize("fit,parts", [(1000, 0), (12, 2), (8, 3), (3, 2)])
def test_delta_rule_by_groups_and_windows_of_chunks(fit, parts, monkeypatch):
    """However many records the scratch holds: groups of sequences and windows of chunks give the bits of all at once,
    read-outs and states; without room for any scratch a step goes row by row."""
    from grout_b200.kernels import ops
    H, G, dk, dv, taps, lens = 4, 2, 32, 64, 3, [300, 65, 1, 130, 32]
    monkeypatch.setattr(ops, "delta_chunks_pay", lambda T, n_seqs, max_rows: max_rows > 4)
    Cc, i32 = 2 * G * dk + H * dv, lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    proj = rnd(sum(lens), Cc + H * dv + 2 * H, seed=51).to(DEV)
    w = [t.to(DEV) for t in (rnd(Cc, taps, seed=52), rnd(H, seed=53), rnd(H, seed=54), rnd(dv, seed=55))]

    def run(max_rows=max(lens)):
        state = rnd(6, ops.delta_state_floats(H, G, dk, dv, taps), seed=56, scale=0.1).to(DEV)
        y = ops.delta_forward(proj, state, *w, H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5,
                              dtype=torch.float32, token_seq=i32([k for k, n in enumerate(lens) for _ in range(n)]),
                              cu_q=i32([0] + torch.tensor(lens).cumsum(0).tolist()), slots=i32([4, 0, 2, 5, 1]),
                              max_rows=max_rows)
        return y, state

    want = run()
    monkeypatch.setattr(ops, "DELTA_CHUNK_BYTES", fit * 4 * H * ops.delta_record(dk, dv))
    records, group, window = ops.delta_chunk_plan(sum(lens), len(lens), max(lens), H, dk, dv)
    assert records <= fit and (-(-10 // window) * -(-5 // group) >= parts if parts else not window)
    got = run()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    monkeypatch.setattr(ops, "delta_chunk_plan", lambda *a: ((1 << 42) // (4 * H * ops.delta_record(dk, dv)), 0, 0))
    got, want = run(), run(None)                  # (four terabytes)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("dk", [64, 44])
@pytest.mark.parametrize("at", [0, 63, 149, 282])
def test_delta_rule_by_chunks_rows_in_front_of_one_that_is_not_finite(at, dk):
    """A row of infinities (its products are NaN) leaves the rows in front of it as they are, to the bit, and the other
    sequence too."""
    from grout_b200.kernels import ops
    H, G, dv, taps, lens = 4, 2, 48, 3, [300, 120]
    assert ops.delta_chunks_pay(sum(lens), 2, max(lens))
    Cc, i32 = 2 * G * dk + H * dv, lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    proj = rnd(sum(lens), Cc + H * dv + 2 * H, seed=61)
    w = [t.to(DEV) for t in (rnd(Cc, taps, seed=62), rnd(H, seed=63), rnd(H, seed=64), rnd(dv, seed=65))]

    def run(x):
        state = torch.zeros(2, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV)
        return ops.delta_forward(x.to(DEV), state, *w, H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5,
                                 dtype=torch.float32, token_seq=i32([0] * 300 + [1] * 120), cu_q=i32([0, 300, 420]),
                                 slots=i32([0, 1]), max_rows=300).cpu()

    want = run(proj)
    proj[at] = float("inf")
    got = run(proj)
    assert torch.equal(got[:at], want[:at]) and torch.equal(got[300:], want[300:])
    assert not torch.isfinite(got[at:300]).all(1).any()


@pytest.mark.parametrize("decay", [0.0, -4.0])
def test_delta_rule_by_chunks_is_as_exact_as_row_by_row(decay):
    """The relative error against 64 bits of read-outs and states, chunk by chunk and row by row: both are 32-bit sums in
    short chains, so neither is more than a tenth above the other (sums over a whole head in one chain, and products of
    decays that lose each rounding, were a third to two thirds above)."""
    from grout_b200.kernels import ops
    H, G, dk, dv, taps, lens = 4, 2, 128, 128, 4, [300, 90]
    assert ops.delta_chunks_pay(sum(lens), 2, max(lens))
    Cc = 2 * G * dk + H * dv
    proj, conv = rnd(sum(lens), Cc + H * dv + 2 * H, seed=41), 1 + rnd(Cc, taps, seed=42, scale=0.1)
    a_log, dt, norm = decay + rnd(H, seed=43, scale=0.1), rnd(H, seed=44, scale=0.1), 1 + rnd(dv, seed=45, scale=0.1)
    want, want_state = _delta_in_64_bits(proj, lens, conv, a_log, dt, norm, H, G, dk, dv, taps)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    off = lambda x, y: float((x.double() - y).norm() / y.norm())  # noqa: E731
    errors = []
    for max_rows in (max(lens), None):
        state = torch.zeros(2, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV)
        y = ops.delta_forward(proj.to(DEV), state, *(t.to(DEV).contiguous() for t in (conv, a_log, dt, norm)),
                              H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5, dtype=torch.float32,
                              token_seq=i32([0] * lens[0] + [1] * lens[1]), cu_q=i32([0, lens[0], sum(lens)]),
                              slots=i32([0, 1]), max_rows=max_rows)
        errors.append((off(y.cpu(), want), off(state[:, (taps - 1) * Cc:].cpu().view(2, H, dv, dk), want_state)))
    (chunks, chunk_state), (rows, row_state) = errors
    assert chunks < 1.1 * rows and chunk_state < 1.1 * row_state, errors


@pytest.mark.parametrize("n_seqs,m", [(1, dict(heads=16, kv_heads=16, dim=128, vdim=128, conv=4)),
                                      (3, dict(heads=8, kv_heads=2, dim=64, vdim=96, conv=3)),
                                      (40, dict(heads=16, kv_heads=4, dim=64, vdim=64, conv=4))])
def test_delta_decode_steps_queued_behind_one_another(n_seqs, m):
    """Decode steps of one state with nothing between them (all arguments made beforehand, then captured in one graph)
    give the bits of steps that are waited for one by one: a step sees the state and the kept inputs that the step in
    front of it left."""
    from grout_b200.kernels import ops
    H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
    W, steps = 24, 12
    w = _delta_weights(H, G, dk, dv, taps, W, seed=23)
    g = lambda t: t.float().to(DEV).contiguous()  # noqa: E731
    wp = torch.cat([w[k] for k in ("q", "k", "v", "g", "b", "a")], 0).double()
    projs = [g(rnd(n_seqs, W, seed=30 + i).double() @ wp.T) for i in range(steps)]
    args = (g(torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], 0)), g(w["A_log"]), g(w["dt_bias"]), g(w["norm"]))
    i32 = lambda n: torch.arange(n, dtype=torch.int32, device=DEV)  # noqa: E731
    kw = dict(H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5, dtype=torch.float32, max_rows=1,
              token_seq=i32(n_seqs), cu_q=i32(n_seqs + 1), slots=i32(n_seqs))
    state = torch.zeros(n_seqs, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV)

    def play(wait):
        out = []
        for p in projs:
            out.append(ops.delta_forward(p, state, *args, **kw))
            if wait:
                torch.cuda.synchronize()
        return out

    want, last = play(True), state.clone()
    assert float((want[1] - want[0]).abs().max()) > 0.01
    state.zero_()
    torch.cuda.synchronize()
    got = play(False)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and torch.equal(state, last)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = play(False)
    state.zero_()
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and torch.equal(state, last)


@pytest.mark.parametrize("rows", [1, 3, 300])
def test_delta_rule_with_weights_that_were_just_computed(rows):
    from grout_b200.kernels import ops
    m = dict(heads=16, kv_heads=8, dim=64, vdim=64, conv=4)
    H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
    w = _delta_weights(H, G, dk, dv, taps, 24, seed=24)
    g = lambda t: t.float().to(DEV).contiguous()  # noqa: E731
    wp = torch.cat([w[k] for k in ("q", "k", "v", "g", "b", "a")], 0).double()
    proj = g(rnd(rows, 24, seed=29).double() @ wp.T)
    args = (g(torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], 0)), g(w["A_log"]), g(w["dt_bias"]), g(w["norm"]))
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)  # noqa: E731
    kw = dict(H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5, dtype=torch.float32, max_rows=rows,
              token_seq=torch.zeros(rows, dtype=torch.int32, device=DEV), cu_q=i32(0, rows), slots=i32(0))
    # a state for each call, made beforehand, so that nothing stands between the weights' kernel and the rule's
    states = [torch.zeros(1, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV) for _ in range(32)]

    def call():
        s = states.pop()
        return [ops.delta_forward(proj, s, *args, **kw), s]

    for on in ([args[0]], [args[3]]):
        _just_computed(on, call)


def test_delta_rule_batches_slots_used_again_and_padding():
    from grout_b200.kernels import ops
    m = DELTA_SHAPES[0]
    H, G, dk, dv, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
    W = 24
    w = _delta_weights(H, G, dk, dv, taps, W, seed=5)
    xa, xb = rnd(40, W, seed=6), rnd(9, W, seed=7)
    alone_a, _ = _delta_run(w, m, xa, [40], torch.float32)
    alone_b, _ = _delta_run(w, m, xb, [9], torch.float32)
    g = lambda t: t.float().to(DEV).contiguous()
    wp = torch.cat([w[k] for k in ("q", "k", "v", "g", "b", "a")], 0).double()
    conv = g(torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], 0))
    state = torch.zeros(4, ops.delta_state_floats(H, G, dk, dv, taps), device=DEV)
    state[1].fill_(7.0)                                               # a slot that someone left dirty ...
    state[1].zero_()                                                  # ... is zeroed when it is opened
    args = dict(H=H, G=G, dk=dk, dv=dv, taps=taps, unit_eps=1e-6, norm_eps=1e-5, dtype=torch.float32)
    run = lambda step, rows: ops.delta_forward(g(rows.double() @ wp.T), state, conv, g(w["A_log"]), g(w["dt_bias"]),
                                               g(w["norm"]), token_seq=step.token_seq, cu_q=step.cu_q,
                                               slots=step.slots, **args).cpu()
    # a in slot 2 and b in slot 1 start together with a padding sequence between them
    s1 = Step([(2, 0, 30), (-1, 0, 3), (1, 0, 8)]).ctx
    y = run(s1, torch.cat([xa[:30], rnd(3, W, seed=8), xb[:8]]))
    same = lambda p, q: float((p - q).abs().max()) < 1e-5
    assert same(y[:30], alone_a[:30]) and same(y[33:], alone_b[:8])
    assert float(state[3].abs().max()) == 0.0                         # padding rows store nothing
    s2 = Step([(1, 8, 1), (2, 30, 1)]).ctx                            # then decoded together, other order
    y = run(s2, torch.cat([xb[8:9], xa[30:31]]))
    assert same(y[0], alone_b[8]) and same(y[1], alone_a[30])
    state[1].zero_()                                                  # b ends; its slot serves a new request
    s3 = Step([(2, 31, 9), (1, 0, 9)]).ctx
    y = run(s3, torch.cat([xa[31:], xb]))
    assert same(y[:9], alone_a[31:]) and same(y[9:], alone_b)


def test_delta_rule_reads_a_far_key():
    """One head keeps what it wrote 400 tokens ago (slow decay): the planted value
    comes back when its key is asked for, and does not with a fast decay."""
    m = dict(heads=1, kv_heads=1, dim=16, vdim=8, conv=1)
    W = 32
    w = _delta_weights(1, 1, 16, 8, 1, W, seed=9)
    for k in ("q.conv", "k.conv", "v.conv"):
        w[k] = torch.ones_like(w[k])
    w["q"], w["k"] = torch.eye(16, W) * 4, torch.eye(16, W) * 4
    w["v"] = torch.zeros(8, W)
    w["v"][:, 16:24] = torch.eye(8) * 4
    w["b"] = torch.full((1, W), 0.0)
    w["b"][0, 31] = 8.0                                               # beta near one where channel 31 is set
    w["a"], w["dt_bias"] = torch.zeros(1, W), torch.zeros(1)
    xs = torch.zeros(402, W)
    xs[:, 3] = 0.3                                                    # every token asks for "key 3" a little
    xs[0, 5], xs[0, 16:24], xs[0, 31] = 5.0, torch.arange(1.0, 9.0), 1.0   # the planted pair: key 5 -> value
    xs[401, 5] = 5.0                                                  # the last token asks for key 5
    for a_log, keeps in ((-9.0, True), (0.0, False)):
        w["A_log"] = torch.tensor([a_log])
        got, _ = _delta_run(w, m, xs, [300, 101, 1], torch.float32)
        close(got, _delta_plain(w, m, xs), torch.float32, f"A_log {a_log}")
        w2 = dict(w)
        x2 = xs.clone()
        x2[0, 16:24] = 0.0
        other, _ = _delta_run(w2, m, x2, [402], torch.float32)
        moved = float((got[401] - other[401]).abs().max())
        assert (moved > 0.1) == keeps, (a_log, moved)


# ------------------------------------------------------------------ routed experts
def _moe_weights(E, ident, F, W, seed, router_scale=3.0):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s, sc=1.0: torch.randn(*s, generator=g) * sc
    w = {"router": r(E + ident, W, sc=router_scale / math.sqrt(W)), "correction": r(E + ident, sc=0.15) - 0.1}
    for j in range(E):
        w[f"e{j}.gate"], w[f"e{j}.up"] = r(F, W, sc=2.0 / math.sqrt(W)), r(F, W, sc=2.0 / math.sqrt(W))
        w[f"e{j}.down"] = r(W, F, sc=1.0 / math.sqrt(F))
    return w


def _moe_run(w, mlp, x, dtype):
    from grout_b200.kernels import ops
    r = mlp["router"]
    E = r["experts"]
    st = lambda what: torch.stack([w[f"e{j}.{what}"] for j in range(E)]).to(dtype).to(DEV).contiguous()
    g = r.get("groups") or {"count": 1, "keep": 1}
    return ops.moe_forward(x.to(dtype).to(DEV), w["router"].float().to(DEV), w["correction"].float().to(DEV),
                           st("gate"), st("up"), st("down"), top=r["top"], n_identity=r.get("identity", 0),
                           n_groups=g["count"], keep_groups=g["keep"], limit=mlp["expert"]["limit"],
                           slope=1.702, want_choice=True)


MOES = [{"kind": "moe", "expert": {"ff": 24, "limit": 0.8},
         "router": {"experts": 6, "identity": 2, "top": 3, "groups": {"count": 4, "keep": 2}}},
        {"kind": "moe", "expert": {"ff": 50, "limit": 2.5},
         "router": {"experts": 9, "identity": 0, "top": 1, "groups": {"count": 3, "keep": 1}}},
        {"kind": "moe", "expert": {"ff": 17, "limit": 0.3},
         "router": {"experts": 5, "identity": 1, "top": 4}},                       # no groups
        {"kind": "moe", "expert": {"ff": 64, "limit": 1.0},
         "router": {"experts": 30, "identity": 2, "top": 2, "groups": {"count": 8, "keep": 3}}}]


@pytest.mark.parametrize("mlp", MOES)
def test_routed_experts_choice_and_output(mlp):
    W, T = 40, 70
    r = mlp["router"]
    w = _moe_weights(r["experts"], r.get("identity", 0), mlp["expert"]["ff"], W, seed=11)
    x = rnd(T, W, seed=12)
    out, ids, wts = _moe_run(w, mlp, x, torch.float32)
    chosen, weights = plain.route(x, w["router"], w["correction"], r)
    assert torch.equal(ids.cpu().long(), chosen)
    close(wts, weights, torch.float32, "weights are the uncorrected scores")
    want = plain.routed_ff(x, {"m." + k: v for k, v in w.items()}, "m.", mlp)
    close(out.sum(0), want, torch.float32, "output")
    # what the test is for: corrected scores below zero, clamps that bite, pass-through experts chosen
    c = torch.softmax(x.double() @ w["router"].double().T, -1) + w["correction"].double()
    if r["top"] >= 3:
        assert bool((c.gather(1, chosen) < 0).any())
    if r.get("identity", 0) * 8 >= w["router"].shape[0]:
        assert bool((chosen >= r["experts"]).any())
    # a token's result does not depend on the rows around it
    alone, _, _ = _moe_run(w, mlp, x[17:18], torch.float32)
    assert torch.equal(alone[:, 0], out[:, 17])
    xb = x.to(torch.bfloat16)
    outb, idsb, _ = _moe_run(w, mlp, xb, torch.bfloat16)
    wb = {k: (v if k in ("router", "correction") else v.to(torch.bfloat16)) for k, v in w.items()}
    same = (idsb.cpu().long() == plain.route(xb, w["router"], w["correction"], r)[0]).all(dim=1)
    wantb = plain.routed_ff(xb, {"m." + k: v for k, v in wb.items()}, "m.", mlp)
    close(outb.sum(0)[same], wantb[same], torch.bfloat16, "bfloat16 output")
    assert int(same.sum()) >= T - 2


# ------------------------------------------------------------------ attention
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(4, 2, 16, 16), (4, 2, 16, 40), (6, 3, 48, 16), (2, 1, 96, 96)])
def test_attention_value_size_temperature_and_sink(dtype, shape):
    """Through the mixer part: q/k norms, the query factor, the sink of logit zero,
    values narrower and wider than the keys; a prompt and its continuation."""
    from grout_b200.cache import CacheLayout, SequenceCache
    from grout_b200.parts import BuildContext, PartSpec, build_part
    H, G, dk, dv = shape
    W, T, eps = 32, 100, 1e-5
    m = dict(heads=H, kv_heads=G, dim=dk, vdim=dv, scale=1.7 / math.sqrt(dk), q_temp={"coef": 0.8, "every": 7})
    g = torch.Generator().manual_seed(21)
    r = lambda *s, sc=1.0: torch.randn(*s, generator=g) * sc
    w = {"q": r(H * dk, W), "k": r(G * dk, W), "v": r(G * dv, W), "o": r(W, H * dv, sc=0.2),
         "q.norm": 1 + r(dk, sc=0.3), "k.norm": 1 + r(dk, sc=0.3)}
    w = {k: v.to(dtype) for k, v in w.items()}
    x = r(T, W).to(dtype)
    want = plain.attention_mixer(x, {"m." + k: v for k, v in w.items()}, "m.", m, eps)
    ctx = BuildContext(dtype, torch.device(DEV))
    part = build_part("mixer", PartSpec("gqa_attention", dict(
        hidden=W, n_heads=H, n_kv_heads=G, head_dim=dk, v_head_dim=dv, position=PartSpec("none", {}),
        qk_norm_eps=eps, scale=m["scale"], sink_logit=0.0, q_temp=(0.8, 7),
        names={"q": "q", "k": "k", "v": "v", "o": "o", "q_norm": "q.norm", "k_norm": "k.norm"})), ctx)
    part.load({k: v.to(DEV) for k, v in w.items()})
    cache = SequenceCache(CacheLayout.from_specs([part.cache_spec()]), max_tokens=512, max_slots=2,
                          max_seq_len=256, dtype=dtype, device=DEV)
    slot = cache.open()
    outs, start = [], 0
    for n in (63, 2, 34, 1):
        cache.reserve(slot, n)
        cache.flush()
        step = Step([(slot, start, n)]).ctx
        outs.append(part.forward(x[start:start + n].to(DEV), step, cache.view(0)))
        outs[-1] = (outs[-1].sum(0) if outs[-1].dim() == 3 else outs[-1]).float().cpu()
        cache.advance(slot, n)
        start += n
    got = torch.cat(outs)
    if dtype == torch.float32:
        close(got, want, dtype)
    else:
        d = (got.double() - want)
        assert float(d.pow(2).mean().sqrt() / want.pow(2).mean().sqrt()) < 0.03
    # the sink and the temperature are there: the plain result without them differs
    m2 = dict(m, q_temp=None)
    assert float((plain.attention_mixer(x, {"m." + k: v for k, v in w.items()}, "m.", m2, eps) - want).abs().max()) > 0.05


def test_attention_finds_a_far_key_beside_the_sink():
    """One key far back is made to stand out for the last query: with the sink's
    share known, the output is that key's value times exp(s) / (1 + sum exp)."""
    dk = dv = 16
    T = 700
    k = rnd(T, dk, seed=31, scale=0.05).double()
    v = rnd(T, dv, seed=32).double()
    q = torch.zeros(T, dk, dtype=torch.float64)
    k[3] = 0
    k[3, 2] = 4.0
    q[T - 1, 2] = 2.0
    out = plain.sink_attention(q, k, v, 1.0)[T - 1]
    e = torch.exp(q[T - 1] @ k.T)
    assert torch.allclose(out, (e[:, None] * v).sum(0) / (1 + e.sum()))
    assert float(e[3] / (1 + e.sum())) > 0.7
    from grout_b200.kernels import ops
    from grout_b200.cache import CacheLayout, KVSpec, SequenceCache
    for dtype in (torch.float32, torch.bfloat16):
        cache = SequenceCache(CacheLayout.from_specs([KVSpec(1, dk, None)]), max_tokens=1024, max_slots=1,
                              max_seq_len=1024, dtype=dtype, device=DEV)
        slot = cache.open()
        cache.reserve(slot, T)
        cache.flush()
        step = Step([(slot, 0, T)]).ctx
        view = cache.view(0)
        qkv = torch.cat([q, k, v], dim=1).to(dtype).to(DEV).contiguous()
        qq, _ = ops.qk_prepare(qkv, 1, 1, dk, token_seq=step.token_seq, token_pos=step.token_pos,
                               slots=step.slots, block_table=view.block_table, k_pages=view.k_pages,
                               v_pages=view.v_pages, page=view.page)
        sinks = torch.zeros(1, device=DEV)
        got = ops.attention(qq, view.k_pages, view.v_pages, view.block_table, step=step, page=view.page,
                            scale=1.0, sinks=sinks)[T - 1, 0].float().cpu()
        close(got, out, dtype, "prompt")
        # the same query alone, as a decode step over the cached keys
        step1 = Step([(slot, T - 1, 1)]).ctx
        got1 = ops.attention(qq[T - 1:].contiguous(), view.k_pages, view.v_pages, view.block_table,
                             step=step1, page=view.page, scale=1.0, sinks=sinks)[0, 0].float().cpu()
        close(got1, out, dtype, "decoded")
