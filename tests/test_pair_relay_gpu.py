"""The mixed contraction on CTA pairs without a pre-split A image (ngpown 22..63,
device arrays, csrc/fk_tc_contract.cuh): the odd CTA's rows are stored by its own
converter warps and used by MMAs that the even CTA issues, after the odd CTA's
relay has reported each stage.  More than 128 bands, so that the odd CTA holds rows
of the result; the same bits in every call, and the mixed gate against the oracle.
(No input makes a missing ordering show every time; the calls are repeated.)
"""
import numpy as np
import pytest

from conftest import gpp_scales, mixed_gate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ng", [22, 42, 63])
@pytest.mark.parametrize("nb, nc", [(130, 1056), (514, 4100)])
def test_odd_rows_repeat_bit_for_bit(ctx, fk, orc, nb, nc, ng):
    import torch
    p = fk.inputs.gpp_synthetic(nb, 2, nc, ng, seed=nb + ng, dist="branch", wx="stress")
    d = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v for k, v in p.items()}
    torch.cuda.synchronize()
    first = {k: np.array(v) for k, v in ctx.gpp(d, "mixed").items() if v is not None}
    mixed_gate(first, orc.gpp(p), gpp_scales(p, orc), 1e-6)
    for _ in range(20):
        again = ctx.gpp(d, "mixed")
        for k, v in first.items():
            np.testing.assert_array_equal(np.asarray(again[k]), v)
