"""Scratch of the plan and of the router never shrinks as a batch grows: a buffer sized for the largest batch serves every
smaller one.  (The scratch of the split-K GEMMs, and with it a forward's workspace, is largest at 64 rows: it is sized per
batch, or for the largest of the batches it serves.)"""

import pytest

import blackwell_moe_b200 as bw


@pytest.mark.parametrize("E,K", [(8, 2), (64, 6), (256, 8)])
def test_plan_and_router_scratch_grow_with_the_batch(E, K):
    lib = bw.lib()
    tokens = sorted({*range(1, 6000, 13), *(n // K + d for n in (1024, 2048, 262144, 524288, 600000) for d in (-1, 0, 1, 2)), 300000})
    for size in (lambda t: lib.bwmoe_plan_scratch_bytes(t, E, K), lambda t: lib.bwmoe_router_scratch_bytes(t, 2048, E, K)):
        sizes = [size(t) for t in tokens]
        assert sizes == sorted(sizes)
