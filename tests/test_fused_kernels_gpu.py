"""The kernels that do several steps of a call at once, at the sizes where their
splits have edges, against the oracle.

FF (ff_bands_kernel, ff_epilogue_kernel, csrc/fk_ff.cu): frequencies on both sides
of a group of lanes and of a warp, one output and more outputs than threads, more
planes than warps.  A planes of several k-slices per unit: long rows, few tiles.
GPP (setup_kernel, rows_flag_block, csrc/fk_gpp.cu): fewer and more plane waves
than the half sum's 64 break chunks, more columns than the 1024 items a block of
the band reduction takes at a time, several occupied bands.

Tolerances: the gates of the other tests, FP64 1e-12, mixed 1e-6.
"""
import numpy as np
import pytest

from conftest import ff_scales, gpp_scales, mixed_gate, rel

pytestmark = pytest.mark.gpu
FFKEYS = ("achsDtemp", "asxDtemp", "achDtemp", "achDtemp_cor", "ach2Dtemp", "schDt_matrix")


# nb, nv, nc, ng, nf, ne
@pytest.mark.parametrize("case", [(3, 1, 33, 2, 2, 1), (20, 2, 64, 8, 33, 7), (9, 4, 100, 4, 70, 300),
                                  (130, 3, 1500, 70, 16, 3)], ids=lambda c: "x".join(map(str, c)))
def test_ff_bands(ctx, fk, orc, case):
    p = fk.inputs.ff_synthetic(*case, seed=sum(case))
    f = fk.FK_FF_SCHDT_GEMM | fk.FK_FF_SPLIT_ACHD
    want, res = orc.ff(p, flags=f), ctx.ff(p, "fp64", f)
    for k in FFKEYS:
        if np.max(np.abs(want[k])) > 0:
            assert rel(np.atleast_1d(res[k]), np.atleast_1d(want[k])) <= 1e-12, k
    mixed_gate(ctx.ff(p, "mixed", f), want, ff_scales(p, orc), 1e-6, keys=FFKEYS)


@pytest.mark.parametrize("nc", [5, 63, 65, 200])
def test_half_sum_break_chunks(ctx, fk, orc, nc):
    p = fk.inputs.gpp_synthetic(20, 5, nc, min(nc, 9), seed=nc, dist="branch", index="even", wx="stress")
    want = orc.gpp(p, flags=orc.ORC_GPP_HALF_SUM)
    res = ctx.gpp(p, "fp64", fk.FK_GPP_HALF_SUM)
    for k in ("achtemp", "asxtemp", "acht_n1_loc"):
        if np.max(np.abs(want[k])) > 0:
            assert rel(res[k], want[k]) <= 1e-12, k
    mixed_gate(ctx.gpp(p, "mixed", fk.FK_GPP_HALF_SUM), res, gpp_scales(p, orc, orc.ORC_GPP_HALF_SUM), 1e-6)


@pytest.mark.parametrize("nv, ng", [(1, 31), (7, 33), (2, 1100)])
def test_occupied_bands_over_many_columns(ctx, fk, orc, nv, ng):
    p = fk.inputs.gpp_synthetic(12, nv, 1200, ng, seed=ng, dist="branch", index="even", wx="stress")
    want = orc.gpp(p)
    res = ctx.gpp(p, "fp64")
    for k in ("achtemp", "asxtemp", "acht_n1_loc"):
        assert rel(res[k], want[k]) <= 1e-12, k
    mixed_gate(ctx.gpp(p, "mixed"), want, gpp_scales(p, orc), 1e-6)
