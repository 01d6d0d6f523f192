"""The query-mode tail (tail_kernels.cuh) against the oracle: every depth of
the lists it keeps in shared memory, the sizes where that changes, men handed
over at once or late, lists used up, and hand-overs in segments."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


# 16, 8, 4 and no list entries per man in shared memory; the first and last
# sizes of each, and the last below which one launch does it all
@pytest.mark.parametrize("n", [767, 768, 769, 3317, 3350, 6330, 6500, 10300, 11900, 12001])
def test_tail_matches_checker(ctx, n):
    for seed in (3, 4):
        pm, pw = ctx.generate(pb.SMP_GEN_UNIFORM, n, seed)
        match, st = ctx.solve(pm, pw)
        assert st["mode"] == 1
        if n <= 3400:
            want, props = oracle.gs_seq(pm.cpu().numpy(), pw.cpu().numpy())
            assert np.array_equal(match.cpu().numpy(), want) and st["proposals"] == props
        assert ctx.check(pm, pw, match) == (0, st["proposals"])
        again, st2 = ctx.solve(pm, pw, check=True)  # a fixed number of segments
        assert np.array_equal(again.cpu().numpy(), match.cpu().numpy())
        assert st2["proposals"] == st["proposals"] and st2["blocking_pairs"] == 0


@pytest.mark.parametrize("threshold", [1, 3, 4, 700, 5000])
@pytest.mark.parametrize("n", [800, 2001, 11000])
def test_tail_hand_over(threshold, n):
    # one free woman to all of them when the chains move to one CTA
    with pb.Context(tail_threshold=threshold) as c:
        pm, pw = c.generate(pb.SMP_GEN_UNIFORM, n, 9)
        want, _ = c.solve(pm, pw, check=True)
        match, st = c.solve(pm, pw)
        assert np.array_equal(match.cpu().numpy(), want.cpu().numpy())
        assert c.check(pm, pw, match) == (0, st["proposals"])


@pytest.mark.parametrize("prefix_k,mode", [(6, 2), (24, 2), (1500, 1)])
def test_tail_runs_out_of_prefix(prefix_k, mode):
    # a short prefix sends the solve to the rank mode; one as long as the
    # lists never does
    n = 1500
    with pb.Context(prefix_k=prefix_k) as c:
        pm, pw = c.generate(pb.SMP_GEN_UNIFORM, n, 2)
        want, props = oracle.gs_seq(pm.cpu().numpy(), pw.cpu().numpy())
        for check in (False, True):
            match, st = c.solve(pm, pw, check=check)
            assert np.array_equal(match.cpu().numpy(), want) and st["proposals"] == props and st["mode"] == mode
