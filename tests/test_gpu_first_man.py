"""Men who all make the same first choice, and a first man whose list names a woman
twice: a solve refuses it (they may share that list); checked solves, batches and
served requests take the men's own proposals for an answer."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


def _men_propose(pm, pw):
    n = len(pm)
    rank = np.empty((n, n), dtype=np.int32)
    np.put_along_axis(rank, pw, np.arange(n, dtype=np.int32)[None, :].repeat(n, 0), axis=1)
    husband, place, proposals = [-1] * n, [0] * n, 0
    for man in range(n):
        m = man
        while m >= 0:
            w = int(pm[m, place[m]])
            place[m] += 1
            proposals += 1
            if husband[w] < 0 or rank[w, m] < rank[w, husband[w]]:
                husband[w], m = m, husband[w]
    match = np.empty(n, dtype=np.int32)
    match[husband] = np.arange(n)
    return match, proposals


@pytest.mark.parametrize("n", [5, 8, 200, 256, 257, 900, 2400])
@pytest.mark.parametrize("others", ["alike", "different"])
def test_first_list_names_a_woman_twice(ctx, n, others):
    import torch

    rng = np.random.default_rng(n)
    pm, pw = (np.array(x, dtype=np.int32) for x in oracle.generate(pb.SMP_GEN_CONGESTED, n, 3))
    if others == "different":  # but for the first choice
        for m in range(1, n):
            pm[m, 1:] = rng.permutation(pm[m, 1:])
    pm[0, n - 1] = pm[0, n - 2]
    row = pw[pm[0, 0]]  # her first choice is the first man, who so ends with her
    at = int(np.flatnonzero(row == 0)[0])
    row[0], row[at] = row[at], row[0]
    want, props = _men_propose(pm, pw)
    dm, dw = torch.from_numpy(pm).cuda(), torch.from_numpy(pw).cuda()
    for lists in ((pm, pw), (dm, dw)):
        with pytest.raises(pb.SmpError) as e:
            ctx.solve(*lists)
        assert e.value.status == pb.SMP_ERR_INVALID_INPUT
    match, st = ctx.solve(dm, dw, check=True)
    assert np.array_equal(match.cpu().numpy(), want) and st["proposals"] == props
    for threshold in (1, 4096):
        out = torch.empty(n, dtype=torch.int32, device="cuda")
        with pb.Batch(ctx, [(dm, dw, out)], threshold_n=threshold, tune=False, use_graph=False) as batch:
            status, proposals, _ = batch.run()
        assert status[0] == 0 and proposals[0] == props and np.array_equal(out.cpu().numpy(), want)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    with pb.Server(route_n=1) as srv:
        result = srv.poll(srv.submit(dm, dw, out))
    assert result["status"] == 0 and result["proposals"] == props and np.array_equal(out.cpu().numpy(), want)
