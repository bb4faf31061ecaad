"""Argmax and sampling kernels against the plain sampler, fed the same draws."""
import itertools
import random

import pytest
import torch

from plain import sampling as plain_sampling

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from grout_b200.kernels import ops
    return ops


def test_argmax_first_maximum_wins():
    g = torch.Generator().manual_seed(0)
    logits = torch.randn(6, 1003, generator=g)
    logits[1, 17] = logits[1, 900] = 9.0           # a tie: the lower index wins
    logits[2, 1002] = 11.0                         # the last element
    logits[3, 0] = 11.0
    logits[4, 5] = float("nan")                    # NaN never wins
    logits[5] = 0.25                               # all equal
    got = _ops().argmax(logits.to(DEV)).cpu().tolist()
    want = [plain_sampling.argmax_first([v if v == v else float("-inf") for v in row.tolist()])
            for row in logits]
    assert got == want and got[1] == 17 and got[5] == 0


CASES = [(1.0, 0, 1.0), (0.8, 0, 1.0), (0.8, 20, 1.0), (0.8, 0, 0.9), (0.7, 50, 0.95),
         (1.5, 1, 1.0), (1.0, 0, 0.0), (0.3, 5, 0.5), (2.0, 1002, 0.999), (1e-6, 10, 0.5)]


@pytest.mark.parametrize("quantised", [False, True])
def test_sample_matches_plain_sampler(quantised):
    """Rows with continuous logits, and rows rounded to a coarse grid so that the
    thresholds of top-k and top-p fall on ties."""
    rng = random.Random(1)
    g = torch.Generator().manual_seed(2)
    V = 1003
    rows, temps, ks, ps, us = [], [], [], [], []
    for t, k, p in CASES:
        for _ in range(6):
            row = torch.randn(V, generator=g) * 2.0
            if quantised:
                row = (row * 2).round() / 2
            rows.append(row)
            temps.append(t), ks.append(k), ps.append(p), us.append(rng.random())
    logits = torch.stack(rows)
    got = _ops().sample(logits.to(DEV), torch.tensor(temps, device=DEV),
                        torch.tensor(ks, dtype=torch.int32, device=DEV),
                        torch.tensor(ps, device=DEV), torch.tensor(us, device=DEV)).cpu().tolist()
    us32 = torch.tensor(us).tolist()               # the kernel sees float32 draws
    for i in range(len(rows)):
        want = plain_sampling.sample_next(rows[i].tolist(), temps[i], ks[i], ps[i], us32[i])
        assert got[i] == want, (i, temps[i], ks[i], ps[i], us32[i], got[i], want)


def test_sample_stays_inside_top_k_and_follows_the_distribution():
    V, n = 257, 4000
    g = torch.Generator().manual_seed(3)
    row = torch.randn(V, generator=g)
    logits = row.repeat(n, 1).to(DEV)
    u = torch.rand(n, generator=g).to(DEV)
    got = _ops().sample(logits, torch.full((n,), 0.9, device=DEV),
                        torch.full((n,), 8, dtype=torch.int32, device=DEV),
                        torch.ones(n, device=DEV), u).cpu()
    top = torch.topk(row, 8).indices
    assert set(got.tolist()) <= set(top.tolist())
    p = torch.softmax(row[top] / 0.9, 0)
    for j, idx in enumerate(top.tolist()):
        assert abs((got == idx).float().mean().item() - p[j].item()) < 0.03


def test_host_sampler_agrees_with_plain():
    from grout_b200.sampling import SamplingParams, choose_one
    rng = random.Random(4)
    g = torch.Generator().manual_seed(5)
    for t, k, p in CASES:
        row = ((torch.randn(300, generator=g) * 4).round() / 2)
        u = rng.random()
        want = plain_sampling.sample_next(row.tolist(), t, k, p, u)
        got = choose_one(row.numpy(), SamplingParams(True, t, k, p).normalised(), u)
        assert got == want, (t, k, p)


def _rows_for_thresholds(V, g):
    """Rows on which a threshold falls in every way: among distinct scores, among more equal
    scores than are ranked directly, in a range stretched by far outliers, beside masked
    scores, and with a NaN that top-k leaves out."""
    normal = torch.randn(V, generator=g) * 2.0
    rows = {"normal": normal, "equal": torch.full((V,), 0.75), "two values": (normal > 0).float(),
            "outliers": normal.clone(), "masked": torch.where(normal > 1.0, normal, torch.tensor(float("-inf"))),
            "flat": 1.0 + 1e-3 * torch.rand(V, generator=g)}
    rows["outliers"][0], rows["outliers"][V // 2] = -3.0e4, 60.0
    rows["masked"][V - 1] = 0.5                    # at least one score is there
    return rows


def _check_thresholds(V, asked, draw):
    """Every row of _rows_for_thresholds with everything asked, against the plain sampler."""
    g = torch.Generator().manual_seed(V)
    rows, prm = [], []
    for name, row in _rows_for_thresholds(V, g).items():
        for t, k, p in asked:
            rows.append(row)
            prm.append((t, max(k, 0), p, draw()))
    logits = torch.stack(rows).to(DEV)
    t, k, p, u = zip(*prm)
    args = [torch.tensor(x, dtype=d) for x, d in ((t, torch.float32), (k, torch.int32), (p, torch.float32), (u, torch.float32))]
    got = _ops().sample(logits, *(a.to(DEV) for a in args)).cpu().tolist()
    assert got == _ops().sample_host(logits, *(a.numpy() for a in args)).cpu().tolist()
    for i, row in enumerate(rows):
        # scaled as the kernel scales, in 32 bits: two scores that this makes equal are a tie
        scaled = (row * (1.0 / args[0][i])).tolist()
        u = args[3][i].item()
        # masses are 32-bit exponentials (2^-22 off) against 64-bit ones here: a draw that close
        # to an element's edge may fall on either side of it
        near = {plain_sampling.sample_next(scaled, 1.0, *prm[i][1:3], min(max(u + d, 0.0), 1.0 - 2.0 ** -24))
                for d in (-2.0 ** -21, 0.0, 2.0 ** -21)}
        assert got[i] in near, (i, prm[i], got[i], near)


# around the cluster kernel's shares of a row (eight blocks of sixteen warps), and the first
# length that takes the one-block kernel
@pytest.mark.parametrize("V", [1, 7, 8, 9, 127, 129, 4095, 33000, 400001])
def test_sample_thresholds_of_every_kind(V):
    asked = [(1.0, 0, 1.0), (0.7, 20, 0.9), (0.8, 0, 0.95), (1.0, 1500, 1.0), (1.0, V - 1, 0.5), (50.0, 3, 0.7)]
    _check_thresholds(V, asked[1:3] if V > 40000 else asked, random.Random(V).random)


# a block's share takes more than one turn of its loads: a vocabulary, one whose rows do not start
# on 16 bytes, and the longest row of the cluster kernel (all of a block's shared memory)
@pytest.mark.parametrize("V", [151936, 151939, 400000])
def test_sample_whole_vocabularies(V):
    draws = itertools.cycle([random.Random(V).random(), 0.0, 1.0 - 2.0 ** -24])
    _check_thresholds(V, [(0.7, 20, 0.9), (1.0, 1500, 1.0)], lambda: next(draws))


@pytest.mark.parametrize("n", [63, 64, 65, 130])
def test_sample_host_rows_beyond_one_launch(n):
    """What a launch carries is for 64 rows: more go in several launches, each row with its own."""
    rng = random.Random(n)
    logits = torch.randn(n, 1003, generator=torch.Generator().manual_seed(n)).to(DEV)
    args = [torch.tensor([rng.choice(c) for _ in range(n)], dtype=d) for c, d in
            (((0.5, 0.9, 1.3), torch.float32), ((0, 1, 40), torch.int32), ((0.6, 1.0), torch.float32))]
    args.append(torch.tensor([rng.random() for _ in range(n)]))
    got = _ops().sample_host(logits, *(a.numpy() for a in args)).cpu().tolist()
    assert got == _ops().sample(logits, *(a.to(DEV) for a in args)).cpu().tolist()
    assert got == [_ops().sample(logits[i:i + 1], *(a[i:i + 1].to(DEV) for a in args)).item() for i in range(n)]


def test_sample_with_nan_and_without_a_finite_maximum():
    nan, inf = float("nan"), float("inf")
    rows = torch.randn(5, 300, generator=torch.Generator().manual_seed(8))
    rows[0, 7] = nan                               # left out by top-k
    rows[1, 7] = nan                               # in the kept set: the sum is void, the maximum is taken
    rows[2, 250] = inf
    rows[3] = -inf
    rows[4] = nan
    k = torch.tensor([5, 0, 0, 0, 0], dtype=torch.int32)
    got = _ops().sample(rows.to(DEV), torch.ones(5, device=DEV), k.to(DEV), torch.ones(5, device=DEV),
                        torch.full((5,), 0.5, device=DEV)).cpu().tolist()
    finite = [v if v == v else -inf for v in rows[0].tolist()]
    assert got[0] in sorted(range(300), key=lambda i: -finite[i])[:5]
    assert got[1:] == [plain_sampling.argmax_first([v if v == v else -inf for v in rows[1].tolist()]), 250, 0, 0]
