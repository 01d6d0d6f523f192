"""Solves of at most 256 people in one launch (small_kernels.cuh) against the
oracle and against the general pipeline, which a configured hand-over takes:
the matching, the proposals, and what the statistics say about the instance."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu

KINDS = [(pb.SMP_GEN_UNIFORM, 0), (pb.SMP_GEN_CONGESTED, 0), (pb.SMP_GEN_CORRELATED, 500), (pb.SMP_GEN_PERFECT, 0),
         (pb.SMP_GEN_REF_CONGESTED, 0), (pb.SMP_GEN_GROUPED, 5), (pb.SMP_GEN_SOLO, 0)]


@pytest.mark.parametrize("kind,param", KINDS)
def test_small_matches_oracle_and_pipeline(ctx, kind, param):
    with pb.Context(tail_threshold=96) as general:
        for n in (1, 2, 3, 4, 5, 31, 32, 33, 64, 97, 191, 192, 193, 255, 256, 257):
            if kind == pb.SMP_GEN_SOLO and n < 3:
                continue
            pm, pw = ctx.generate(kind, n, 40 + n, param=param)
            want, props = oracle.gs_seq(pm.cpu().numpy(), pw.cpu().numpy())
            ref, rst = general.solve(pm, pw)
            for precheck in (True, False):
                match, st = ctx.solve(pm, pw, precheck=precheck)
                assert np.array_equal(match.cpu().numpy(), want) and st["proposals"] == props
                if precheck:
                    assert {k: st[k] for k in ("mode", "perfect", "n", "rank_bytes", "proposals")} == {
                        k: rst[k] for k in ("mode", "perfect", "n", "rank_bytes", "proposals")}, n
            host, hst = ctx.solve(pm.cpu().numpy(), pw.cpu().numpy())
            assert np.array_equal(host, want) and hst["proposals"] == props and hst["mode"] == rst["mode"]
            assert st["kernel_launches"] == (1 if n <= 256 else st["kernel_launches"])


@pytest.mark.parametrize("n", [2, 40, 256])
@pytest.mark.parametrize("kind,param", KINDS[:5])
def test_small_refuses_what_the_pipeline_refuses(ctx, kind, param, n):
    rng = np.random.default_rng(n)
    base_m, base_w = oracle.generate(kind, n, 8, 0, param)
    with pb.Context(tail_threshold=96) as general:
        for where in range(10):
            pm, pw = base_m.copy(), base_w.copy()
            side = pm if where % 2 else pw
            row, col = int(rng.integers(n)), int(rng.integers(n))
            side[row, col] = [n, -1, side[row, (col + 1) % n], 1 << 20, side[row, 0]][where // 2]
            outcome = []
            for c in (ctx, general):
                try:
                    match, st = c.solve(pm, pw)
                    outcome.append((match.tolist(), st["proposals"]))
                except pb.SmpError as e:
                    outcome.append(e.status)
            assert outcome[0] == outcome[1], (where, row, col)


@pytest.mark.parametrize("n", [97, 300, 927])
def test_match_where_no_kernel_may_write(n):
    # pinned host memory as the device solve's output: copied there, as ever
    import torch

    with pb.Context() as c:
        pm, pw = c.generate(pb.SMP_GEN_UNIFORM, n, 5)
        want, _ = c.solve(pm, pw)
        out = torch.full((n,), -1, dtype=torch.int32).pin_memory()
        match, _ = c.solve(pm, pw, out=out)
        assert bool((match == want.cpu()).all())


@pytest.mark.parametrize("n", [257, 767, 768, 4097])
def test_perfect_without_the_tail(n):
    # every man a first choice of his own; then two who share one
    import torch

    def device(*lists):
        return [torch.from_numpy(x).cuda() for x in lists]

    rng = np.random.default_rng(n)
    pm = np.stack([rng.permutation(n) for _ in range(n)]).astype(np.int32)
    pw = np.stack([rng.permutation(n) for _ in range(n)]).astype(np.int32)
    for m, w in enumerate(rng.permutation(n)):
        k = int(np.nonzero(pm[m] == w)[0][0])
        pm[m, [0, k]] = pm[m, [k, 0]]
    with pb.Context() as c:
        match, st = c.solve(*device(pm, pw))
        assert np.array_equal(match.cpu().numpy(), pm[:, 0]) and st["proposals"] == n
        pm[0] = pm[1]
        want, props = oracle.gs_seq(pm, pw)
        match, st = c.solve(*device(pm, pw))
        assert np.array_equal(match.cpu().numpy(), want) and st["proposals"] == props
