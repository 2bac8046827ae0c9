"""The FP64 contraction on the tensor cores (csrc/fk_tc64.cuh) against the
oracle, at the sizes where its tiles, slices and digits have edges: 256-row and
64-column tiles, 32-wide stages, one and several k-slices, rows whose values
spread over many decades, and rows it must leave to the DMMA kernel (not
finite, or beyond 2^+-400).

Tolerance: the FP64 gate of the other tests, 1e-12 relative, normwise over each
output (the digit products keep 59 bits of the rows' largest product per term,
so K = 4096 terms stay below 1e-14 of the sum's scale).
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


# bands on both sides of the 128- and 256-row tiles, 3 * ngpown around 64 and 128, ncouls around the stage width
@pytest.mark.parametrize("nb, ng, nc", [(1, 1, 1), (2, 21, 31), (127, 22, 32), (130, 42, 33), (257, 43, 65),
                                        (258, 5, 4097), (514, 21, 1000)])
@pytest.mark.parametrize("achstemp", [0, 2])
def test_gpp_tile_edges(ctx, fk, orc, nb, ng, nc, achstemp):
    p = fk.inputs.gpp_synthetic(nb, min(2, nb - 1), nc, min(ng, nc), seed=nb + nc, dist="branch", wx="stress")
    res, ref = ctx.gpp(p, "fp64", achstemp), orc.gpp(p, flags=achstemp)
    check(res, ref)
    if achstemp:
        assert rel(res["achstemp"], [ref["achstemp"]]) <= TOL


@pytest.mark.parametrize("nb, ng, nc, nf", [(3, 1, 33, 2), (128, 63, 96, 5), (257, 65, 1000, 3), (20, 8, 64, 70)])
def test_ff_tile_edges(ctx, fk, orc, nb, ng, nc, nf):
    p = fk.inputs.ff_synthetic(nb, min(2, nb), nc, ng, nf, 3, seed=nb + nc)
    for flags in (0, 5):
        check(ctx.ff(p, "fp64", flags), orc.ff(p, flags=flags), FFKEYS)


def test_rows_of_many_decades(ctx, fk, orc):
    """Rows falling by twelve decades along ncouls (aqsntemp) and epsilon rows
    rising by as many: every product is of the same size, far from both rows'
    largest magnitudes."""
    p = fk.inputs.ff_synthetic(40, 2, 2000, 48, 4, 3, seed=3)
    fall = 10.0 ** np.linspace(0.0, -12.0, 2000)
    p["aqsntemp"] = np.ascontiguousarray(p["aqsntemp"] * fall)
    for k in ("I_epsR_array", "I_epsA_array"):
        p[k] = np.ascontiguousarray(p[k] / fall)
    check(ctx.ff(p, "fp64", 5), orc.ff(p, flags=5), FFKEYS)


def test_rows_out_of_range_go_to_dmma(ctx, fk, orc):
    p = fk.inputs.gpp_synthetic(70, 2, 700, 9, seed=4, dist="branch", wx="stress")
    want = orc.gpp(p)
    check(ctx.gpp(p, "fp64"), want)
    # a band scaled beyond 2^400: its acht_n1_loc scales with it, the other bands keep theirs
    q = dict(p, aqsntemp=p["aqsntemp"].copy())
    q["aqsntemp"][10] *= 1e150
    got = ctx.gpp(q, "fp64")["acht_n1_loc"].copy()
    got[10] /= 1e150
    assert rel(got, want["acht_n1_loc"]) <= TOL
    # infinities and NaN stay in the band they are in
    for bad in (np.inf, np.nan):
        q["aqsntemp"] = p["aqsntemp"].copy()
        q["aqsntemp"][10, 123] = bad
        got = ctx.gpp(q, "fp64")["acht_n1_loc"]
        assert not np.isfinite(got[10])
        keep = np.arange(70) != 10
        assert rel(got[keep], want["acht_n1_loc"][keep]) <= TOL
    check(ctx.gpp(p, "fp64"), want)  # and the next call is an ordinary one


def test_capture_without_room_for_the_images(fk, orc):
    """A caller's own stream capture cannot grow the workspace: with only the
    DMMA path's workspace there the call takes that path, as it did before the
    tensor-core one."""
    import torch
    c = fk.Context(0)
    nb, nc, ng = 64, 2048, 8
    p = fk.inputs.gpp_synthetic(nb, 2, nc, ng, seed=6)
    d = dict(p)
    for k, v in p.items():
        if isinstance(v, np.ndarray):
            d[k] = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    out = {k: torch.zeros(n, dtype=torch.complex128, device="cuda")
           for k, n in (("achtemp", 3), ("asxtemp", 3), ("acht_n1_loc", nb))}
    stream = torch.cuda.Stream()
    c.set_stream(stream.cuda_stream)
    c.reserve(48 * ng * nc + (1 << 21))  # D and the partial sums, not the images
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        with pytest.raises(fk.FKError):
            c.reserve(1 << 30)  # growing is refused during capture
        c.gpp(d, "fp64", out=out)
    g.replay()
    torch.cuda.synchronize()
    ref = orc.gpp(p)
    check({k: v.cpu().numpy() for k, v in out.items()}, ref)
    c.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_ff_small_arrays_wherever_they_are(ctx, fk, prec):
    """The small arrays as numpy, as GPU tensors and as GPU tensors off a
    16-byte boundary (copied), and calls queued behind one another without a
    wait: the same bits every time."""
    import torch
    p = fk.inputs.ff_synthetic(40, 2, 640, 48, 6, 5, seed=8)
    want = ctx.ff(p, prec, 5)
    small = ("vcoul", "inv_igp_index", "indinv", "ekq", "dFreqGrid", "dFreqBrd", "pref")
    d = {k: torch.from_numpy(v).cuda() if isinstance(v, np.ndarray) and k not in small else v for k, v in p.items()}
    dev, off = dict(d), dict(d)
    for k in small:
        dev[k] = torch.from_numpy(p[k]).cuda()
        if k != "dFreqBrd":  # torch's complex loads want 16 bytes themselves
            raw = torch.zeros(8 + p[k].nbytes, dtype=torch.uint8, device="cuda")
            raw[8:] = torch.from_numpy(p[k].view(np.uint8)).cuda()
            off[k] = raw[8:].view(dev[k].dtype)
    torch.cuda.synchronize()
    outs = []
    for q in (d, dev, off, d, d, d):
        o = {k: torch.zeros(v.shape, dtype=torch.complex128, device="cuda") for k, v in want.items()}
        ctx.ff(q, prec, 5, out=o)
        outs.append(o)
    ctx.synchronize()
    for o in outs:
        for k in FFKEYS:
            np.testing.assert_array_equal(o[k].cpu().numpy(), want[k])
