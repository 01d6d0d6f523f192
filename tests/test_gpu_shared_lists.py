"""Men who share one list, the women's lists alike in several degrees: their
proposals run beside the screen, after it, or not at all."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


def women(kind, n, rng):
    if kind == "alike":
        return np.tile(rng.permutation(n), (n, 1))
    if kind == "one differs":
        pw = np.tile(rng.permutation(n), (n, 1))
        pw[n // 2, [0, n - 1]] = pw[n // 2, [n - 1, 0]]
        return pw
    if kind == "same first":
        pw = np.stack([rng.permutation(n) for _ in range(n)])
        k = np.argmax(pw == 0, axis=1)
        pw[np.arange(n), k] = pw[:, 0]
        pw[:, 0] = 0
        return pw
    if kind == "quarter":  # n / 4 distinct first choices, where the rule turns
        pw = np.stack([rng.permutation(n) for _ in range(n)])
        for w in range(n):
            k = int(np.argmax(pw[w] == w % (n // 4)))
            pw[w, [0, k]] = pw[w, [k, 0]]
        return pw
    return oracle.generate(pb.SMP_GEN_CORRELATED, n, 5, 0, kind)[1]


@pytest.mark.parametrize("kind", ["alike", "one differs", "same first", "quarter", 3, 500])
@pytest.mark.parametrize("n", [257, 300, 1025, 2049])
def test_women_alike(kind, n):
    rng = np.random.default_rng(n)
    pm = np.tile(rng.permutation(n), (n, 1)).astype(np.int32)
    pw = np.ascontiguousarray(women(kind, n, rng), dtype=np.int32)
    want, props = oracle.gs_seq(pm, pw)
    with pb.Context() as c:
        for lists in ((pm, pw), (pm, pw)):
            match, st = c.solve(*lists)
            assert np.array_equal(match, want) and st["proposals"] == props and st["mode"] == 3
        bad = pw.copy()
        bad[n - 1, n - 1] = bad[n - 1, 0]
        with pytest.raises(pb.SmpError) as e:
            c.solve(pm, bad)
        assert e.value.status == pb.SMP_ERR_INVALID_INPUT
