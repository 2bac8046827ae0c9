"""FP64 calls whose rows the digit products cannot hold to FP64's own precision
(csrc/fk_tc64.cuh): large and small magnitudes in one k-slice.  The contraction
must notice where its error is not small beside the row's sums and leave those
tiles to the DMMA kernel.

Tolerance: the FP64 gate of the other tests, 1e-12 relative, normwise over each
output.  A tile stays on the digit products while their error, 2^-57.2 sqrt(2 K)
times the product of the rows' powers of two (rms of the dropped classes), is below
2^-48 of the row's largest term; over at most 2^9 columns and slices of a row these
add to 2^-48 * 2^4.5 = 8e-14.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu
TOL = 1e-12
KEYS = ("achtemp", "asxtemp", "acht_n1_loc")
FFKEYS = ("achsDtemp", "asxDtemp", "achDtemp", "achDtemp_cor", "ach2Dtemp", "schDt_matrix")


def check(res, ref, keys=KEYS, tol=TOL):
    for k in keys:
        if np.max(np.abs(ref[k])) > 0:
            assert rel(np.atleast_1d(res[k]), np.atleast_1d(ref[k])) <= tol, k


@pytest.mark.parametrize("decades", [3, 6, 12])
def test_opposite_gradings_in_one_slice(ctx, fk, orc, decades):
    """aqsntemp falls by `decades` along ncouls and epsilon rises by as many, every
    product of the same size.  With 16 planes of eight column tiles the plan keeps
    all 2000 k-values in one slice."""
    p = fk.inputs.ff_synthetic(40, 2, 2000, 512, 16, 3, seed=3)
    fall = 10.0 ** np.linspace(0.0, -float(decades), 2000)
    p["aqsntemp"] = np.ascontiguousarray(p["aqsntemp"] * fall)
    for k in ("I_epsR_array", "I_epsA_array"):
        p[k] = np.ascontiguousarray(p[k] / fall)
    check(ctx.ff(p, "fp64", 5), orc.ff(p, flags=5), FFKEYS)


@pytest.mark.parametrize("log2", [10, 20, 30, 40, 60, 200])
@pytest.mark.parametrize("flags", [0, 2, 4, 8])
def test_one_large_value_over_zero_epsilon(ctx, fk, orc, log2, flags):
    """One value of a row of aqsntemp is 2^log2; epsilon is zero there in every column,
    so the value enters no sum: full sum, static remainder, half sum, physics mode."""
    p = fk.inputs.gpp_synthetic(70, 2, 3000, 9, seed=log2 + flags, dist="branch", wx="stress")
    p["I_eps_array"][:, 1234] = 0.0
    p["aqsntemp"][10, 1234] = 2.0 ** log2
    res, ref = ctx.gpp(p, "fp64", flags), orc.gpp(p, flags=flags)
    check(res, ref)
    if flags == 2:
        assert rel(res["achstemp"], [ref["achstemp"]]) <= TOL


@pytest.mark.parametrize("log2", [20, 60])
def test_one_large_value_over_zero_epsilon_real(ctx, fk, orc, log2):
    p = fk.inputs.gpp_real_synthetic(70, 2, 3000, 9, seed=log2)
    p["I_eps_array"][:, 1234] = 0.0
    p["aqsntemp"][10, 1234] = 2.0 ** log2
    check(ctx.gpp_real(p, "fp64"), orc.gpp_real(p))


def test_real_rows_whose_halves_differ(ctx, fk, orc):
    """The real-valued sum contracts pairs of plane waves as complex values and uses
    the real part only.  Even plane waves large in aqsntemp and small in epsilon, odd
    ones the other way: the real part is small beside the unused imaginary one."""
    p = fk.inputs.gpp_real_synthetic(40, 2, 4000, 9, seed=8)
    s = np.where(np.arange(4000) % 2 == 0, 1e6, 1e-6)
    p["aqsntemp"] = np.ascontiguousarray(p["aqsntemp"] * s)
    p["I_eps_array"] = np.ascontiguousarray(p["I_eps_array"] / s)
    check(ctx.gpp_real(p, "fp64"), orc.gpp_real(p))


def test_full_size_slice_with_one_large_value(ctx, fk):
    """512 x 32768 x 20: 38 slices of 864 k-values, against torch in FP64."""
    import torch
    nb, nc, ng = 512, 32768, 20
    p = fk.inputs.gpp_synthetic(nb, 2, nc, ng, seed=5)
    p["I_eps_array"][:, 20001] = 0.0
    for n, e in ((7, 10), (200, 20), (300, 30), (511, 60)):
        p["aqsntemp"][n, 20001] = 2.0 ** e
    res = ctx.gpp(p, "fp64")
    t = lambda k: torch.from_numpy(p[k]).cuda()  # noqa: E731
    wt, eps = t("wtilde_array"), t("I_eps_array")
    wd = float(p["wx_array"][2]) - wt
    n = wd.real ** 2 + wd.imag ** 2
    delw = wt * torch.conj(wd) / n
    D = torch.where((n > 0.25) & (delw.real ** 2 + delw.imag ** 2 < 250000.0), delw * eps, torch.zeros_like(eps))
    igp = torch.from_numpy(p["inv_igp_index"].astype(np.int64)).cuda()
    w = torch.conj(t("aqsmtemp")[:, igp]) * (0.5 * t("vcoul")[igp])
    want = (w * (t("aqsntemp") @ D.T)).sum(1).cpu().numpy()
    err = np.abs(res["acht_n1_loc"] - want)
    assert np.max(err / np.maximum(np.abs(want), np.median(np.abs(want)))) <= TOL


def test_extreme_digits(ctx, fk):
    """Constant rows whose digits are the extreme ones (64, then -256): the drained
    class sums are the largest that occur, 14.7e6 < 2^24.  schDt_matrix with unit
    weights is K (2 v^2 + 0 i) for a = (v, v), b = (v, -v)."""
    v = float(64 * 2 ** 54 - 256 * (2 ** 45 + 2 ** 36 + 2 ** 27)) * 2.0 ** -59
    for K in (32, 96, 8192):
        p = fk.inputs.ff_synthetic(3, 1, K, 1, 2, 2, seed=1)
        p["aqsmtemp"] = np.ones_like(p["aqsmtemp"])
        p["aqsntemp"] = np.full_like(p["aqsntemp"], complex(v, v))
        p["I_epsR_array"] = np.full_like(p["I_epsR_array"], complex(v, -v))
        got = ctx.ff(p, "fp64", 5)["schDt_matrix"]
        want = 2.0 * K * v * v
        assert np.max(np.abs(got - want)) <= 4e-16 * want, K


@pytest.mark.parametrize("which, planes", [("I_epsR_array", 7), ("I_epsA_array", 7), ("I_epsR_array", 70)])
def test_ff_planes_out_of_range_go_to_dmma(ctx, fk, orc, which, planes):
    """A plane scaled beyond 2^400 (of R, of A, and with two groups of planes one of the
    second): every plane of its launch is contracted by the DMMA kernel, with the band order, the
    second epsilon array and the plane list of the tensor-core launch."""
    p = fk.inputs.ff_synthetic(150, 3, 200, 40, planes, 4, seed=planes)
    want = orc.ff(p, flags=5)
    q = dict(p)
    q[which] = p[which].copy()
    f = planes - 2
    q[which][f] *= 2.0 ** 450
    got = ctx.ff(q, "fp64", 5)
    m = got["schDt_matrix"].copy()
    if which == "I_epsR_array":
        m[:, f] /= 2.0 ** 450
    assert rel(m, want["schDt_matrix"]) <= TOL
    if which == "I_epsA_array":
        check(got, orc.ff(q, flags=5), FFKEYS)
    check(ctx.ff(p, "fp64", 5), want, FFKEYS)


@pytest.mark.parametrize("flags", [0, 2, 4])
def test_d_rows_out_of_range_go_to_dmma(ctx, fk, orc, flags):
    p = fk.inputs.gpp_synthetic(70, 2, 700, 9, seed=4, dist="branch", wx="stress")
    p["I_eps_array"][3] *= 2.0 ** 450
    res, ref = ctx.gpp(p, "fp64", flags), orc.gpp(p, flags=flags)
    check(res, ref)
    if flags == 2:
        assert rel(res["achstemp"], [ref["achstemp"]]) <= TOL


def test_real_rows_out_of_range_go_to_dmma(ctx, fk, orc):
    p = fk.inputs.gpp_real_synthetic(70, 2, 700, 9, seed=4)
    p["aqsntemp"][10] *= 2.0 ** 450
    got, want = ctx.gpp_real(p, "fp64")["acht_n1_loc"], orc.gpp_real(p)["acht_n1_loc"]
    got[10] /= 2.0 ** 450
    want[10] /= 2.0 ** 450
    assert rel(got, want) <= TOL


def test_more_units_than_pairs_and_long_slices(ctx, fk):
    """300 bands x 640 columns x 8 planes: 160 tiles on 76 CTA pairs, slices of 8192
    k-values (converted without shared memory), against torch in FP64."""
    import torch
    p = fk.inputs.ff_synthetic_device(300, 2, 8192, 640, 8, 3, seed=9)
    torch.cuda.synchronize()
    got = ctx.ff(p, "fp64", 5)["schDt_matrix"]
    w = torch.conj(p["aqsmtemp"][:, :640])
    want = np.stack([(w * (p["aqsntemp"] @ p["I_epsR_array"][f].T)).sum(1).cpu().numpy() for f in range(8)], 1)
    assert rel(got, want) <= TOL


@pytest.mark.parametrize("path", ["gpp", "ff"])
def test_wait_timeout_is_reported(ctx, fk, orc, path):
    """A wait bound of 0 cycles: the call reports FK_ETIMEOUT and the context stays usable."""
    if path == "gpp":
        p = fk.inputs.gpp_synthetic(48, 2, 1536, 12, seed=1, dist="branch", index="reference", wx="reference")
        call, ref, keys = (lambda: ctx.gpp(p, "fp64")), orc.gpp(p), KEYS
    else:
        p = fk.inputs.ff_synthetic(40, 2, 640, 48, 6, 5, seed=2)
        call, ref, keys = (lambda: ctx.ff(p, "fp64", 5)), orc.ff(p, flags=5), FFKEYS
    ctx.set_wait_limit(0)
    try:
        with pytest.raises(fk.FKError) as e:
            call()
        assert e.value.status == fk._native.FK_ETIMEOUT
    finally:
        ctx.set_wait_limit(-1)
    ctx.synchronize()
    check(call(), ref, keys)


def test_half_sum_weights_out_of_range(ctx, fk, orc):
    """A band of aqsmtemp beyond 2^400: the half sum's second contraction (rows of aqsmtemp)
    goes to DMMA, the other bands keep their values."""
    p = fk.inputs.gpp_synthetic(70, 2, 700, 9, seed=6, dist="branch", wx="stress")
    want = orc.gpp(p, flags=orc.ORC_GPP_HALF_SUM)["acht_n1_loc"]
    q = dict(p, aqsmtemp=p["aqsmtemp"].copy())
    q["aqsmtemp"][10] *= 2.0 ** 450
    got, ref = ctx.gpp(q, "fp64", fk.FK_GPP_HALF_SUM)["acht_n1_loc"], orc.gpp(q, flags=orc.ORC_GPP_HALF_SUM)["acht_n1_loc"]
    keep = np.arange(70) != 10
    assert rel(got[keep], want[keep]) <= TOL
    assert rel(got[10:11], ref[10:11]) <= TOL
