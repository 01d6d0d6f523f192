"""The stability checker against the oracle's: sizes at the edges of its
256-bit tiles, its 64 choices read ahead and its 16-byte rows; matchings that
are stable, random, and with the wife last or first."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 63, 64, 65, 127, 128, 129, 255, 256, 257, 319, 513, 1030])
@pytest.mark.parametrize("kind,param", [(pb.SMP_GEN_UNIFORM, 0), (pb.SMP_GEN_CORRELATED, 500)])
def test_checker_matches_oracle(ctx, kind, param, n):
    pm, pw = oracle.generate(kind, n, 23, 0, param)
    rng = np.random.default_rng(n)
    stable, _ = oracle.gs_seq(pm, pw)
    for match in (stable, rng.permutation(n).astype(np.int32), np.roll(stable, 1)):
        assert ctx.check(pm, pw, match) == oracle.check(pm, pw, match)


def test_checker_refuses_bad_input(ctx):
    n = 300
    pm, pw = oracle.generate(pb.SMP_GEN_UNIFORM, n, 4)
    match, _ = oracle.gs_seq(pm, pw)
    twice, off = match.copy(), match.copy()
    twice[0] = twice[1]
    off[7] = n
    bad_w, bad_m, no_wife = pw.copy(), pm.copy(), pm.copy()
    bad_w[n - 1, 3] = bad_w[n - 1, 4]
    bad_m[5, 0] = -1
    no_wife[9][no_wife[9] == match[9]] = -1
    for m, w, mt in ((pm, pw, twice), (pm, pw, off), (pm, bad_w, match), (bad_m, pw, match), (no_wife, pw, match)):
        with pytest.raises(pb.SmpError) as e:
            ctx.check(m, w, mt)
        assert e.value.status == pb.SMP_ERR_INVALID_INPUT
    assert ctx.check(pm, pw, match)[0] == 0
