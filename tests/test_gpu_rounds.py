"""Rank-mode solves in rounds (round_kernels.cuh) against the oracle: sizes at
the edges of a batch of men (592), of a candidate list (1024) and of the
16-byte rows, lists that resemble one another in every way the generator
knows, and men that start in the worst possible order."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 8, 31, 33, 257, 591, 593, 1023, 1024, 1025, 1187, 2055)


def lists(kind, n, param=0, seed=11):
    if kind == pb.SMP_GEN_SOLO and n < 3:
        kind = pb.SMP_GEN_UNIFORM
    return oracle.generate(kind, n, seed, 0, param)


@pytest.mark.parametrize("kind,param", [
    (pb.SMP_GEN_UNIFORM, 0), (pb.SMP_GEN_CORRELATED, 500), (pb.SMP_GEN_CORRELATED, 20), (pb.SMP_GEN_GROUPED, 5),
    (pb.SMP_GEN_CONGESTED, 0), (pb.SMP_GEN_REF_CONGESTED, 0), (pb.SMP_GEN_SOLO, 0), (pb.SMP_GEN_PERFECT, 0),
])
def test_rounds_match_oracle(kind, param):
    with pb.Context(mode=1) as c:  # rank mode whatever the lists
        for n in SIZES:
            pm, pw = lists(kind, n, param)
            want, props = oracle.gs_seq(pm, pw)
            match, st = c.solve(pm, pw)  # steps added until the matching is complete
            assert np.array_equal(match, want) and st["proposals"] == props, n
            match, st = c.solve(pm, pw, check=True)  # a fixed sequence of steps
            assert np.array_equal(match, want) and st["proposals"] == props and st["blocking_pairs"] == 0, n


@pytest.mark.parametrize("n", [1500, 5000])
def test_rounds_in_the_worst_order(n):
    # The 64 women whose ranks set the starting order like the men in one
    # order, all others in the reverse: every man who starts displaces all
    # who started before him, lists are used up at once, and at n = 5000 the
    # fixed sequence runs out of steps and ends in its last one.
    pm = np.tile(np.arange(n, dtype=np.int32), (n, 1))
    pm[n // 2, [n - 2, n - 1]] = pm[n // 2, [n - 1, n - 2]]  # not one shared list
    pw = np.tile(np.arange(n, dtype=np.int32)[::-1], (n, 1))
    for i in range(64):
        pw[i * n // 64] = np.arange(n, dtype=np.int32)
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context() as c:
        for check in (False, True):
            match, st = c.solve(pm, pw, check=check)
            assert np.array_equal(match, want) and st["proposals"] == props and st["mode"] == 0


@pytest.mark.parametrize("where", ["first", "deep", "late_man"])
def test_rounds_refuse_an_entry_out_of_range(where):
    # every entry of the men's lists is checked, also those no man reaches
    n = 1300
    pm, pw = oracle.generate(pb.SMP_GEN_CORRELATED, n, 5, 0, 500)
    pm = pm.copy()
    pm[{"first": 3, "deep": 700, "late_man": n - 1}[where], {"first": 0, "deep": n - 1, "late_man": 640}[where]] = n
    with pb.Context(mode=1) as c:
        for check in (False, True):
            with pytest.raises(pb.SmpError) as e:
                c.solve(pm, pw, check=check)
            assert e.value.status == pb.SMP_ERR_INVALID_INPUT


@pytest.mark.parametrize("n", [23216, 23217])
def test_rounds_at_the_table_limit(n):
    # the largest n whose refresh steps have the table of next entries, and the next
    with pb.Context() as c:
        pm, pw = c.generate(pb.SMP_GEN_SOLO, n, 3)
        match, st = c.solve(pm, pw)
        again, st2 = c.solve(pm, pw, check=True)
        assert bool((match == again).all()) and st["proposals"] == st2["proposals"] and st2["blocking_pairs"] == 0


@pytest.mark.parametrize("kind,n,param", [
    (pb.SMP_GEN_UNIFORM, 3001, 0), (pb.SMP_GEN_CORRELATED, 5003, 1000), (pb.SMP_GEN_CORRELATED, 4100, 3000),
    (pb.SMP_GEN_GROUPED, 3301, 400), (pb.SMP_GEN_SOLO, 1777, 0),
])
def test_rounds_by_eight_lanes(kind, n, param):
    # steps after the first work their chains by eight lanes where few proposals come too late
    pm, pw = lists(kind, n, param)
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context(mode=1) as c:
        for check in (False, True):
            match, st = c.solve(pm, pw, check=check)
            assert np.array_equal(match, want) and st["proposals"] == props


@pytest.mark.parametrize("kind,n,param", [
    ("worst", 5000, 0), (pb.SMP_GEN_SOLO, 1777, 0), (pb.SMP_GEN_CORRELATED, 3001, 500), (pb.SMP_GEN_UNIFORM, 3001, 0),
    (pb.SMP_GEN_UNIFORM, 9001, 0), (pb.SMP_GEN_PERFECT, 900, 0),
])
def test_fixed_sequences(kind, n, param):
    # phase by phase nothing is read back in the middle of one: a fixed number of
    # steps and a last one, or of the tail's segments and one without a limit
    if kind == "worst":
        pm = np.tile(np.arange(n, dtype=np.int32), (n, 1))
        pm[n // 2, [n - 2, n - 1]] = pm[n // 2, [n - 1, n - 2]]
        pw = np.tile(np.arange(n, dtype=np.int32)[::-1], (n, 1))
        for i in range(64):
            pw[i * n // 64] = np.arange(n, dtype=np.int32)
    else:
        pm, pw = lists(kind, n, param)
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context() as c:
        c.stage(pm, pw, n)
        if not c.precheck():
            c.init()
            c.core()
        assert np.array_equal(c.post(), want)
        match, st = c.solve(pm, pw, check=True)  # the checker after the passes
        assert np.array_equal(match, want) and st["proposals"] == props and st["blocking_pairs"] == 0
