"""Solves without a tail and with a configured tail window: every
mode and hand-over from one pass to the next, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu

KINDS = [(pb.SMP_GEN_UNIFORM, 0), (pb.SMP_GEN_CONGESTED, 0), (pb.SMP_GEN_CORRELATED, 500), (pb.SMP_GEN_PERFECT, 0),
         (pb.SMP_GEN_REF_CONGESTED, 0), (pb.SMP_GEN_GROUPED, 5), (pb.SMP_GEN_SOLO, 0)]


@pytest.mark.parametrize("cfg", [{"tail_threshold": -1}, {"tail_threshold": -1, "prefix_k": 6},
                                 {"tail_threshold": -1, "mode": 1}, {"tail_threshold": -1, "rank_bytes": 4},
                                 {"tail_window": 64}, {"tail_window": 32, "rank_bytes": 4}])
@pytest.mark.parametrize("kind,param", KINDS)
def test_configured_tails(kind, param, cfg):
    with pb.Context(**cfg) as c:
        for n in (3, 97, 300, 1100):
            pm, pw = oracle.generate(kind, n, 14, 0, param)
            want, props = oracle.gs_seq(pm, pw)
            for check in (False, True):
                match, st = c.solve(pm, pw, check=check)
                assert np.array_equal(match, want) and st["proposals"] == props, (n, check)
            bad = pw.copy()
            bad[n - 1, 0] = n
            if not st["perfect"]:
                with pytest.raises(pb.SmpError) as e:
                    c.solve(pm, bad)
                assert e.value.status == pb.SMP_ERR_INVALID_INPUT


@pytest.mark.parametrize("kind,mode", [(pb.SMP_GEN_UNIFORM, 1), (pb.SMP_GEN_PERFECT, 1), (pb.SMP_GEN_CONGESTED, 3)])
def test_too_large_for_a_tail(ctx, kind, mode):
    n = 38700  # 6 n bytes of bids and positions: above one SM's shared memory
    pm, pw = ctx.generate(kind, n, 2)
    match, st = ctx.solve(pm, pw)
    assert st["mode"] == mode
    assert ctx.check(pm, pw, match) == (0, st["proposals"])
