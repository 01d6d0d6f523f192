"""The shape a batch runs with: fields the caller fixed stay fixed whatever
batches of the same size were tuned before, and a reported shape can be asked
for again."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import pactae_b200 as pb

pytestmark = pytest.mark.gpu


def uniform_batch(c, count, n_lo):
    import torch

    insts = []
    for b in range(count):
        n = n_lo + b
        pm, pw = c.generate(pb.SMP_GEN_UNIFORM, n, 3, salt=b)
        insts.append((pm, pw, torch.full((n,), -1, dtype=torch.int32, device="cuda")))
    return insts


def assert_solved(insts, batch):
    status, props, _ = batch.run()
    assert not any(status)
    for (pm, pw, mt), p in zip(insts, props):
        want, wp = oracle.gs_seq(pm.cpu().numpy(), pw.cpu().numpy())
        assert np.array_equal(mt.cpu().numpy(), want) and p == wp


@pytest.mark.parametrize("first", [{}, {"window": 256}, {"block_threads": 64, "ctas_per_sm": 1}])
def test_fixed_fields_are_not_taken_from_another_batch(ctx, first):
    insts = uniform_batch(ctx, 40, 40)
    for fixed in (first, {"block_threads": 128, "ctas_per_sm": 2}, {"window": 128}, {"rank_smem_kb": -1},
                  {"cta_width": 2}, {}):
        with pb.Batch(ctx, insts, **fixed) as batch:
            cfg = {**batch.config(), "cta_width": batch.cta_width}
            assert {k: cfg[k] for k in fixed} == fixed
            assert_solved(insts, batch)


@pytest.mark.parametrize("width", [1, 2])
@pytest.mark.parametrize("block", [64, 512])
def test_reported_shape_can_be_asked_for(ctx, block, width):
    insts = uniform_batch(ctx, 12, 90)
    shape = {"block_threads": block, "ctas_per_sm": 1, "window": 64, "rank_smem_kb": 32}
    with pb.Batch(ctx, insts, cta_width=width if width == 2 else 0, **shape) as batch:
        cfg = batch.config()
        assert {k: cfg[k] for k in shape} == shape and batch.cta_width == width
        assert_solved(insts, batch)
