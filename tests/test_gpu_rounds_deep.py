"""Rounds whose chains pass whole windows of their lists (SOLO: one chain that
jumps through lists as long as n), where eight lanes hand over to warps."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [592, 593, 600, 801, 1024, 1025, 1190])
def test_one_deep_chain(n, mode):
    rng = np.random.default_rng(n)
    pm, pw = oracle.generate(pb.SMP_GEN_SOLO, n, 3)
    number = rng.permutation(n).astype(np.int32)
    pm, pw = number[pm], np.ascontiguousarray(pw[np.argsort(number)])
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context(mode=mode) as c:
        match, st = c.solve(pm, pw)
        assert np.array_equal(match, want) and st["proposals"] == props


@pytest.mark.parametrize("n", [700, 1024, 1300])
def test_deep_chains_among_shallow_ones(n):
    # uniform lists for most, the last sixteenth of the men at the end of everyone's
    rng = np.random.default_rng(n)
    pm, pw = (np.stack([rng.permutation(n) for _ in range(n)]).astype(np.int32) for _ in range(2))
    late = rng.choice(n, n // 16, replace=False)
    for w in range(n):
        pw[w] = np.concatenate([pw[w][~np.isin(pw[w], late)], rng.permutation(late)])
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context(mode=1) as c:
        match, st = c.solve(pm, pw)
        assert np.array_equal(match, want) and st["proposals"] == props
