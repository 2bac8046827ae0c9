"""The mixed contraction's FP64 staging ring (csrc/fk_tc_contract.cuh): stages of 32
k-values arrive in quarters of eight through a ring of five slots, 128 rows at a
time.  Sizes on both sides of a quarter, of a stage and of the ring's length, with
rows on both sides of the tile, against the oracle.

Tolerance: the mixed gate of the other tests, 1e-6 relative to each output's scale.
"""
import pytest

from conftest import gpp_scales, mixed_gate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 7, 8, 9, 24, 31, 33, 39, 41, 256, 519])
@pytest.mark.parametrize("nb", [3, 129])
def test_ring_edges(ctx, fk, orc, nb, nc):
    p = fk.inputs.gpp_synthetic(nb, 2, nc, min(5, nc), seed=nb + nc, dist="branch", index="reference", wx="stress")
    mixed_gate(ctx.gpp(p, "mixed"), orc.gpp(p), gpp_scales(p, orc), 1e-6)
