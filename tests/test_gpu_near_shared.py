"""Rank-mode men who are alike among women who are not: through k_bulk and
k_tail instead of the rounds, from n = 1280 on (2304 where most men are the same)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


def twisted(n, how):
    """One list for all men but `how` of them (spread over `how` first choices)."""
    pm, pw = oracle.generate(pb.SMP_GEN_CONGESTED, n, 7)
    pm = pm.copy()
    rng = np.random.default_rng(n)
    for i, m in enumerate(rng.choice(n, how, replace=False)):
        if i == 0:  # the same first choice: the screen finds the difference
            pm[m, [n - 2, n - 1]] = pm[m, [n - 1, n - 2]]
        else:
            pm[m] = rng.permutation(n)
    return pm, pw


@pytest.mark.parametrize("n", [1279, 1280, 2303, 2304, 2305, 4200])
@pytest.mark.parametrize("how", [0, 1, 12, 40, 700, "correlated", "grouped"])
def test_men_alike(n, how):
    if how == "correlated":
        pm, pw = oracle.generate(pb.SMP_GEN_CORRELATED, n, 7, 0, 300)[0], oracle.generate(pb.SMP_GEN_UNIFORM, n, 7)[1]
    elif how == "grouped":
        pm, pw = oracle.generate(pb.SMP_GEN_GROUPED, n, 7, 0, 20)[0], oracle.generate(pb.SMP_GEN_UNIFORM, n, 7)[1]
    else:
        pm, pw = twisted(n, how)
    want, props = oracle.gs_seq(pm, pw)
    for mode in (0, 1):
        with pb.Context(mode=mode) as c:
            for check in (False, True):  # n >= 4096 from the host: streamed unless checked
                match, st = c.solve(pm, pw, check=check)
                assert np.array_equal(match, want) and st["proposals"] == props
                few = 4 * len(np.unique(pm[:, 0])) < n  # else the query mode is tried first
                assert not (few or mode == 1) or st["mode"] == (3 if how == 0 and mode == 0 else 0)
            engine = pb.SmpEngineB200(pb.SmpObj(pm, pw), n, c)
            for _ in range(2):
                assert np.array_equal(engine.FindStableMatching(), want) and c.stats()["proposals"] == props


@pytest.mark.parametrize("where", ["men", "women"])
def test_men_alike_bad_input(where):
    n = 2600  # (the bulk)
    pm, pw = (x.copy() for x in twisted(n, 3))
    side = pm if where == "men" else pw
    side[n // 3, n // 2] = n if where == "men" else side[n // 3, 0]
    with pb.Context() as c, pytest.raises(pb.SmpError) as e:
        c.solve(pm, pw)
    assert e.value.status == pb.SMP_ERR_INVALID_INPUT
