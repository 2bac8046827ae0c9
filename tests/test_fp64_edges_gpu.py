"""FP64 calls at the edges of what the FP32 branch tests of the FP64 preps
(csrc/fk_gpp.cu) can hold, against the oracle.

Tolerance: the FP64 gate of the other tests, 1e-12 relative, normwise.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-12
KEYS = ("achtemp", "asxtemp", "acht_n1_loc")


@pytest.mark.parametrize("wx", [(1e17, 3e17, 9e17), (1e30, 1e40, 1e50), (1e62, 1e70, 1e80), (1e85, 1e90, 1e95)],
                         ids=lambda w: "%g" % w[0])
def test_huge_frequencies(ctx, fk, orc, wx):
    """|wx - wtilde|^2 beyond FP32's range: each frequency's sums by themselves (asxtemp
    is 0 where (wx^2)^2 overflows, as in the reference)."""
    p = fk.inputs.gpp_synthetic(20, 3, 300, 7, seed=2)
    p["wx_array"] = np.array(wx)
    res, ref = ctx.gpp(p, "fp64"), orc.gpp(p)
    for k in ("achtemp", "asxtemp"):
        for iw in range(3):
            assert rel(res[k][iw:iw + 1], ref[k][iw:iw + 1]) <= TOL, (k, iw)
    assert rel(res["acht_n1_loc"], ref["acht_n1_loc"]) <= TOL


def test_tiny_frequencies(ctx, fk, orc):
    """(wx^2)^2 underflows: the reference divides by zero, and so does the call."""
    p = fk.inputs.gpp_synthetic(20, 3, 300, 7, seed=2)
    p["wx_array"] = np.array([1e-90, 1e-85, 0.5])
    res, ref = ctx.gpp(p, "fp64"), orc.gpp(p)
    np.testing.assert_array_equal(np.isfinite(res["asxtemp"]), np.isfinite(ref["asxtemp"]))
    assert not np.isfinite(ref["asxtemp"][0]) and np.isfinite(ref["asxtemp"][2])
    assert rel(res["achtemp"], ref["achtemp"]) <= TOL
    assert rel(res["asxtemp"][2:], ref["asxtemp"][2:]) <= TOL


@pytest.mark.parametrize("bad", [complex(np.inf, 0.0), complex(0.0, -np.inf), complex(np.nan, 1.0)], ids=str)
@pytest.mark.parametrize("band", [0, 2])
@pytest.mark.parametrize("flags", [0, 8])
def test_not_finite_over_a_zero_term(ctx, fk, orc, band, bad, flags):
    """A value of an occupied band's aqsntemp that is not finite where wtilde is 0: at wx = 0.4
    neither sch nor ssx is taken there, and 0 times the value is NaN as in the reference."""
    p = fk.inputs.gpp_synthetic(12, 3, 600, 7, seed=3, wx="stress")
    p["wtilde_array"][:, 77] = 0.0
    p["aqsntemp"][band, 77] = bad
    res, ref = ctx.gpp(p, "fp64", flags), orc.gpp(p, flags=flags)
    for k in KEYS:
        np.testing.assert_array_equal(np.isnan(res[k]), np.isnan(ref[k]), err_msg=k)
        ok = np.isfinite(ref[k])
        if ok.any():
            assert rel(res[k][ok], ref[k][ok]) <= TOL, k
    assert np.isnan(ref["asxtemp"]).all()


@pytest.mark.parametrize("log2", [59, 61, 130, 260, 450])
def test_half_sum_break_beyond_fp32(ctx, fk, orc, log2):
    """Epsilon beyond FP32's range in one column: the half sum's search for the first
    |Omega2| < 1e-6 of a column must not stop there."""
    p = fk.inputs.gpp_synthetic(40, 3, 700, 9, seed=4, dist="branch", wx="stress")
    p["I_eps_array"][3] *= 2.0 ** log2
    res, ref = ctx.gpp(p, "fp64", fk.FK_GPP_HALF_SUM), orc.gpp(p, flags=orc.ORC_GPP_HALF_SUM)
    for k in KEYS:
        assert rel(res[k], ref[k]) <= TOL, k
