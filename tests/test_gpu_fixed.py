"""Solves in one fixed sequence (instances a batch routes to the all-SM pipeline):
nothing is read back in the middle of one, so it must end whatever the lists --
in its last step of the rounds, the last segment of the tail, the retry, or one of
the paths a rank-mode instance takes."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


def order_sample(i, samples, n):
    """The women whose ranks set the starting order (common.cuh)."""
    start, end = i * n // samples, (i + 1) * n // samples
    h = (i + 1) * 0x9E3779B9 & 0xFFFFFFFF
    h = (h ^ (h >> 15)) * 0x85EBCA6B & 0xFFFFFFFF
    h ^= h >> 13
    return start + h % (end - start)


def worst_order(n):
    # The 64 women whose ranks set the starting order like the men in one order, all
    # others in the reverse: every man who starts displaces all who started before
    # him, and the steps run out before the men have all started.
    pm = np.tile(np.arange(n, dtype=np.int32), (n, 1))
    pm[n // 2, [n - 2, n - 1]] = pm[n // 2, [n - 1, n - 2]]  # not one shared list
    pw = np.tile(np.arange(n, dtype=np.int32)[::-1], (n, 1))
    for i in range(64):
        pw[order_sample(i, 64, n)] = np.arange(n, dtype=np.int32)
    return pm, pw


def near_shared(n):
    pm, pw = oracle.generate(pb.SMP_GEN_CONGESTED, n, 7)
    pm = pm.copy()
    pm[n // 2, [n - 2, n - 1]] = pm[n // 2, [n - 1, n - 2]]
    return pm, pw


def shuffled_solo(n):
    rng = np.random.default_rng(n)
    pm, pw = oracle.generate(pb.SMP_GEN_SOLO, n, 3)
    number = rng.permutation(n).astype(np.int32)
    return number[pm], np.ascontiguousarray(pw[np.argsort(number)])


def mixed(n, men, women):
    return oracle.generate(*men[:1], n, 7, 0, men[1])[0], oracle.generate(*women[:1], n, 7, 0, women[1])[1]


UNIFORM, CONGESTED = (pb.SMP_GEN_UNIFORM, 0), (pb.SMP_GEN_CONGESTED, 0)
CASES = {
    "worst 1500": lambda: worst_order(1500),
    "worst 5000": lambda: worst_order(5000),
    "solo 601": lambda: shuffled_solo(601),
    "solo 1777": lambda: shuffled_solo(1777),
    "uniform 400": lambda: mixed(400, UNIFORM, UNIFORM),
    "uniform 3001": lambda: mixed(3001, UNIFORM, UNIFORM),
    "uniform 12001": lambda: mixed(12001, UNIFORM, UNIFORM),  # the tail's lists in L2
    "correlated 300": lambda: mixed(300, (pb.SMP_GEN_CORRELATED, 500), (pb.SMP_GEN_CORRELATED, 500)),
    "correlated 3001": lambda: mixed(3001, (pb.SMP_GEN_CORRELATED, 500), (pb.SMP_GEN_CORRELATED, 500)),
    "random5 1301": lambda: mixed(1301, (pb.SMP_GEN_GROUPED, 5), (pb.SMP_GEN_GROUPED, 5)),
    "perfect 900": lambda: mixed(900, (pb.SMP_GEN_PERFECT, 0), (pb.SMP_GEN_PERFECT, 0)),
    "shared 303": lambda: mixed(303, CONGESTED, UNIFORM),
    "shared 2501": lambda: mixed(2501, CONGESTED, UNIFORM),
    "shared by both 1100": lambda: mixed(1100, (pb.SMP_GEN_REF_CONGESTED, 0), (pb.SMP_GEN_REF_CONGESTED, 0)),
    "shared, women alike 1200": lambda: mixed(1200, CONGESTED, (pb.SMP_GEN_CORRELATED, 20)),
    "near shared 1501": lambda: near_shared(1501),
    "near shared 2501": lambda: near_shared(2501),
    "men alike 1281": lambda: mixed(1281, (pb.SMP_GEN_CORRELATED, 300), UNIFORM),
    "men alike 3001": lambda: mixed(3001, (pb.SMP_GEN_CORRELATED, 300), UNIFORM),
}


@pytest.mark.parametrize("case", CASES)
def test_fixed_sequence(ctx, case):
    import torch

    pm, pw = CASES[case]()
    n = pm.shape[0]
    want, props = oracle.gs_seq(pm, pw)
    small = oracle.generate(pb.SMP_GEN_UNIFORM, 50, 2)
    insts = [(torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda(),
              torch.from_numpy(np.ascontiguousarray(b, dtype=np.int32)).cuda(),
              torch.full((a.shape[0],), -1, dtype=torch.int32, device="cuda")) for a, b in ((pm, pw), small)]
    for use_graph in (False, True):
        insts[0][2].fill_(-1)
        with pb.Batch(ctx, insts, threshold_n=60, use_graph=use_graph, tune=False) as batch:
            for _ in range(2):  # and replayed
                status, proposals, _ = batch.run()
                assert status == [0, 0] and proposals[0] == props
                assert np.array_equal(insts[0][2].cpu().numpy(), want)


@pytest.mark.parametrize("n", [700, 1500, 5000])
def test_worst_order_in_steps_that_are_added(n):
    pm, pw = worst_order(n)
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context() as c:
        match, st = c.solve(pm, pw)
        assert np.array_equal(match, want) and st["proposals"] == props and st["mode"] == 0


@pytest.mark.parametrize("case", ["uniform 400", "correlated 3001", "shared 2501", "near shared 2501", "men alike 1281"])
@pytest.mark.parametrize("side", [0, 1])
def test_fixed_sequence_bad_input(ctx, case, side):
    import torch

    lists = [np.array(x, dtype=np.int32) for x in CASES[case]()]
    n = lists[0].shape[0]
    lists[side][n // 3, 2] = n if side == 0 else lists[side][n // 3, 3]
    pm, pw = (torch.from_numpy(x).cuda() for x in lists)
    good = [torch.from_numpy(x).cuda() for x in oracle.generate(pb.SMP_GEN_CONGESTED, 700, 4)]
    out = [torch.empty(k, dtype=torch.int32, device="cuda") for k in (n, 700)]
    with pb.Batch(ctx, [(pm, pw, out[0]), (*good, out[1])], threshold_n=60, tune=False) as batch:
        status, _, _ = batch.run()
    assert status == [pb.SMP_ERR_INVALID_INPUT, 0]
    want, _ = oracle.gs_seq(*(x.cpu().numpy() for x in good))
    assert np.array_equal(out[1].cpu().numpy(), want)


def test_short_prefix_is_retried(ctx):
    # uniform women, men whose choices crowd a few women after the first: the query mode
    # ends beyond the prefix and the sequence goes on with the rank mode
    import torch

    n = 1500
    rng = np.random.default_rng(4)
    pm = np.stack([np.concatenate([[m], rng.permutation(np.delete(np.arange(n), m))]) for m in range(n)])
    pw = np.stack([rng.permutation(n) for _ in range(n)])
    crowd = np.arange(400)  # these men's lists begin alike, 400 deep
    head = rng.permutation(400)
    for m in crowd:
        rest = pm[m][~np.isin(pm[m], head)]
        pm[m] = np.concatenate([head, rest])
    pm, pw = (x.astype(np.int32) for x in (pm, pw))
    want, props = oracle.gs_seq(pm, pw)
    _, st = ctx.solve(pm, pw)
    assert st["mode"] == 2
    dm, dw = torch.from_numpy(pm).cuda(), torch.from_numpy(pw).cuda()
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    with pb.Batch(ctx, [(dm, dw, out)], threshold_n=60, tune=False) as batch:
        status, proposals, _ = batch.run()
    assert status == [0] and proposals == [props] and np.array_equal(out.cpu().numpy(), want)
