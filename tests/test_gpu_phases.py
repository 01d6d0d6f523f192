"""The phase calls on a context that has already done something: the whole
sequence again on one staging, and after a solve on the same context."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle
import pactae_b200 as pb
from pactae_b200._lib import lib

pytestmark = pytest.mark.gpu


def phases(c, n):
    """precheck .. post of what the context holds; the matching on the host."""
    perfect = ctypes.c_int32()
    assert lib.smp_b200_precheck(c.handle, ctypes.byref(perfect)) == pb.SMP_OK
    if not perfect.value:
        assert lib.smp_b200_init(c.handle) == pb.SMP_OK
        assert lib.smp_b200_core(c.handle) == pb.SMP_OK
    return post(c, n)


def post(c, n):
    match = np.full(n, -1, dtype=np.int32)
    assert lib.smp_b200_post(c.handle, ctypes.c_void_p(match.ctypes.data), 0) == pb.SMP_OK
    return match


# with a prefix too short for the query mode (the rank-mode retry), in the query
# mode to its end, in the rank mode, and with distinct first choices
@pytest.mark.parametrize("kind,n,param,prefix_k", [
    (pb.SMP_GEN_UNIFORM, 1500, 0, 6), (pb.SMP_GEN_UNIFORM, 400, 0, 6), (pb.SMP_GEN_UNIFORM, 1500, 0, 0),
    (pb.SMP_GEN_CORRELATED, 1300, 500, 0), (pb.SMP_GEN_CONGESTED, 600, 0, 0), (pb.SMP_GEN_PERFECT, 700, 0, 0),
])
def test_phases_again_on_one_staging(kind, n, param, prefix_k):
    pm, pw = oracle.generate(kind, n, 8, 0, param)
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context(prefix_k=prefix_k) as c:
        engine = pb.SmpEngineB200(pb.SmpObj(pm, pw), n, c)
        for _ in range(3):
            assert np.array_equal(engine.FindStableMatching(), want)
            assert c.stats()["proposals"] == props


@pytest.mark.parametrize("n", [300, 900])
def test_phases_after_a_device_solve_leave_its_match_alone(n):
    # the array of a call that has returned is not written again
    with pb.Context() as c:
        pm, pw = c.generate(pb.SMP_GEN_UNIFORM, n, 6)
        out, _ = c.solve(pm, pw)
        want = out.cpu().numpy()
        out.fill_(-1)
        assert np.array_equal(phases(c, n), want)
        assert bool((out == -1).all())


# one launch, the one-launch tail, the segments, distinct first choices, the
# rounds, and men who share one list; each the first call on its context
@pytest.mark.parametrize("device", [True, False])
@pytest.mark.parametrize("kind,n,param", [
    (pb.SMP_GEN_UNIFORM, 97, 0), (pb.SMP_GEN_PERFECT, 40, 0), (pb.SMP_GEN_CONGESTED, 200, 0),
    (pb.SMP_GEN_UNIFORM, 400, 0), (pb.SMP_GEN_UNIFORM, 900, 0), (pb.SMP_GEN_PERFECT, 900, 0),
    (pb.SMP_GEN_CORRELATED, 700, 500), (pb.SMP_GEN_CONGESTED, 700, 0),
])
def test_phases_that_follow_a_solve(kind, n, param, device):
    pm, pw = oracle.generate(kind, n, 12, 0, param)
    want, props = oracle.gs_seq(pm, pw)
    if device:
        import torch

        pm, pw = torch.from_numpy(pm).cuda(), torch.from_numpy(pw).cuda()
    with pb.Context() as c:
        _, st = c.solve(pm, pw)
        for _ in range(2):  # post returns what the solve found
            assert np.array_equal(post(c, n), want)
            assert (c.stats()["proposals"], c.stats()["mode"]) == (props, st["mode"])
        # init and core start from the precheck
        assert lib.smp_b200_init(c.handle) == pb.SMP_OK
        for _ in range(2):
            assert lib.smp_b200_core(c.handle) == pb.SMP_OK
            assert np.array_equal(post(c, n), want) and c.stats()["proposals"] == props
    with pb.Context() as c:
        c.solve(pm, pw)
        assert lib.smp_b200_core(c.handle) == pb.SMP_OK
        assert np.array_equal(post(c, n), want) and c.stats()["proposals"] == props


@pytest.mark.parametrize("kind", [pb.SMP_GEN_PERFECT, pb.SMP_GEN_UNIFORM])
@pytest.mark.parametrize("n", [200, 600, 5000])
def test_match_may_lie_in_a_list_that_is_not_needed_again(ctx, kind, n):
    # the matching is copied over a row once everything has been read
    for side in (0, 1):
        for row in (0, n // 2, n - 1):
            lists = ctx.generate(kind, n, 4)
            want, _ = ctx.solve(*lists)
            match, _ = ctx.solve(*lists, out=lists[side][row])
            assert bool((match == want).all()) and match.data_ptr() == lists[side][row].data_ptr()
