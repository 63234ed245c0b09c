"""The pair scan through a workspace (rr_zscan_pairs_ws) against the one
without (rr_zscan_pairs): the same sums in the same order, so every output is
compared for equality -- all basis sizes, solve methods, chunk remainders, two
exposures on one grid, rounds that do not divide the pairs, and pairs whose
redshift puts a bin outside the template."""

import ctypes

import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

from redrock_b200 import synth  # noqa: E402


def _both(rows, src, pt, pz, round_pairs, bounds=None):
    """Host (chi2, coeff, penalty, status) of both entry points."""
    import torch
    from redrock_b200 import _lib
    from redrock_b200.device import ptr, to_device
    L = _lib.lib()
    segs = (_lib.PairSegment * len(rows.segments))(*rows.segments)
    hb = None if bounds is None else np.ascontiguousarray(bounds, dtype=np.float64)
    tm = _lib.PairTemplate(ptr(src.x), src.nx, ptr(src.y), src.nbasis, src.igm, src.method, 0, None,
                           ptr(src.oii_dev),
                           None if hb is None else hb.ctypes.data_as(ctypes.c_void_p))
    n = len(pz)
    dt, dz = to_device(np.asarray(pt, np.int32), torch.int32), to_device(pz)
    out = []
    for ws in (False, True):
        c2 = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
        co = torch.full((n, src.nbasis), -1.0, dtype=torch.float64, device="cuda")
        pe = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        a = (ctypes.byref(tm), segs, len(segs), ptr(rows.rows), ptr(rows.fwf), ptr(rows.wsum),
             rows.npix_row, ptr(dt), ptr(dz), n, ptr(c2), ptr(co), ptr(pe))
        if ws:
            nb = int(L.rr_zscan_pairs_ws_bytes(segs, len(segs), src.nbasis, round_pairs))
            w = torch.empty(nb, dtype=torch.uint8, device="cuda")
            assert L.rr_zscan_pairs_ws(*a, ptr(w), nb, ptr(st), None) == 0
        else:
            assert L.rr_zscan_pairs(*a, ptr(st), None) == 0
        torch.cuda.synchronize()
        out.append([x.cpu().numpy() for x in (c2, co, pe, st)])
    return out


def _same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("nb,npix,method,igm", [
    (10, (2751, 2326, 2881), "PCA", "Inoue14"), (4, (246, 247), "PCA", "Inoue14"),
    (5, (245, 1, 30), "PCA", "None"), (1, (493,), "PCA", "Calura12"),
    (7, (300, 700), "NNLS", "None"), (3, (500,), "BVLS", "Inoue14"), (9, (246, 492), "PCA", "None"),
    (2, (738,), "PCA", "Kamble20"), (6, (256,), "UNKNOWN", "None"), (8, (1000,), "NNLS", "None"),
])
def test_ws_equals_direct(nb, npix, method, igm):
    from redrock_b200 import targets as T
    from redrock_b200.engine import GridLayout, RowPack, TargetBatch, TemplateSource
    from redrock_b200.templates import solve_code_of
    rng = np.random.default_rng(nb)
    grids, lo = {}, 3700.0
    for i, n in enumerate(npix):
        grids[f"c{i}"] = lo + 0.8 * np.arange(max(n, 2))[:max(n, 2)]
        lo += 0.8 * n + 9.0
    tg = []
    for t in range(5):
        sp = []
        for band, w in grids.items():
            for _ in range(2 if t == 1 else 1):
                rd, ro = synth.resolution_dia(len(w), rng.uniform(0.8, 1.2))
                iv = rng.uniform(0.3, 4.0, len(w)) * (rng.uniform(size=len(w)) > 0.2)
                if t == 3:
                    iv[:] = 0.0
                sp.append(synth.SpectrumSpec(band, w, rng.normal(size=len(w)) + 1.0, iv, rd, ro))
        tg.append(synth.TargetSpec(t, sp))
    layout = GridLayout.from_dwave(grids)
    rows = RowPack(TargetBatch(T.from_synth(tg), layout).to_device())
    w = np.arange(900.0, 10500.0, 0.9)
    flux = np.stack([1.0 + np.sin(w / (20.0 + 7.0 * i)) for i in range(nb)])
    src = TemplateSource(w, flux, np.array([0.5]), igm, oii=rng.normal(size=nb),
                         method=solve_code_of(method))
    n = 37
    pt = rng.integers(0, 5, n)
    z = rng.uniform(0.1, 2.5, n)
    bounds = None if method != "BVLS" else np.stack([np.full(nb, -0.4), np.full(nb, 0.6)])
    for per in (2, 8, 40):
        a, b = _both(rows, src, pt, z, per, bounds)
        _same(a, b)
    z[5] = 9.0                                # bins below the template's first sample
    a, b = _both(rows, src, pt, z, 16, bounds)
    assert a[3][0] == 2 and np.isnan(a[0][5])
    _same(a, b)


def test_ws_arguments():
    from redrock_b200 import _lib
    L = _lib.lib()
    seg = (_lib.PairSegment * 1)(_lib.PairSegment(None, None, 100, 0, 1.0))
    one = int(L.rr_zscan_pairs_ws_bytes(seg, 1, 4, 1))
    assert one >= 110 * 4 * 8
    assert int(L.rr_zscan_pairs_ws_bytes(seg, 1, 4, 10)) == 10 * one
    big = 2 ** (8 * ctypes.sizeof(ctypes.c_size_t)) - 1
    assert int(L.rr_zscan_pairs_ws_bytes(seg, 1, 11, 1)) == big
    assert int(L.rr_zscan_pairs_ws_bytes(seg, 0, 4, 1)) == big


@pytest.mark.parametrize("nb,npix,igm", [(10, (2751, 2326), "Inoue14"), (4, (246, 247, 5), "Inoue14"),
                                         (5, (500,), "None"), (7, (300, 41), "Calura12")])
def test_grad_ws_equals_direct(nb, npix, igm):
    """Gradients: chi2, coefficients, penalty and dchi2/dflux are the same
    bits.  dT/dz divides by reciprocals, two roundings of e y / (w (1 + z)),
    about 1e-12 of |T| here, against |dT/dz| of order |T|: the derivative
    sums agree within 1e-9 of their largest value."""
    import torch
    from redrock_b200 import _lib, targets as T
    from redrock_b200.device import ptr, to_device
    from redrock_b200.engine import GridLayout, RowPack, TargetBatch, TemplateSource
    rng = np.random.default_rng(nb)
    grids, lo = {}, 3700.0
    for i, n in enumerate(npix):
        grids[f"c{i}"] = lo + 0.8 * np.arange(n)
        lo += 0.8 * n + 9.0
    tg = []
    for t in range(4):
        sp = []
        for band, w in grids.items():
            rd, ro = synth.resolution_dia(len(w), rng.uniform(0.8, 1.2))
            iv = rng.uniform(0.3, 4.0, len(w)) * (rng.uniform(size=len(w)) > 0.2) * (t != 2)
            sp.append(synth.SpectrumSpec(band, w, rng.normal(size=len(w)) + 1.0, iv, rd, ro))
        tg.append(synth.TargetSpec(t, sp))
    layout = GridLayout.from_dwave(grids)
    rows = RowPack(TargetBatch(T.from_synth(tg), layout).to_device())
    w = np.arange(900.0, 10500.0, 0.9)
    flux = np.stack([1.0 + np.sin(w / (20.0 + 7.0 * i)) for i in range(nb)])
    src = TemplateSource(w, flux, np.array([0.5]), igm, oii=rng.normal(size=nb))
    segs = (_lib.PairSegment * len(rows.segments))(*rows.segments)
    tm = _lib.PairTemplate(ptr(src.x), src.nx, ptr(src.y), nb, src.igm, 0, 0, None,
                           ptr(src.oii_dev), None)
    n = 23
    dt = to_device(rng.integers(0, 4, n).astype(np.int32), torch.int32)
    z = rng.uniform(0.1, 2.5, n)
    z[3] = 9.0
    dz = to_device(z)
    L = _lib.lib()
    out = []
    for per in (0, 4, 24):
        o = [torch.full(s, -1.0, dtype=torch.float64, device="cuda")
             for s in ((n,), (n, nb), (n,), (n,), (n,), (n, rows.npix_row), (n,))]
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        a = (ctypes.byref(tm), segs, len(segs), ptr(rows.rows), ptr(rows.sw), ptr(rows.fwf),
             ptr(rows.wsum), rows.npix_row, ptr(dt), ptr(dz), n) + tuple(ptr(x) for x in o)
        if per:
            nbytes = int(L.rr_zscan_pairs_grad_ws_bytes(segs, len(segs), nb, per))
            ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            assert L.rr_zscan_pairs_grad_ws(*a, ptr(ws), nbytes, ptr(st), None) == 0
        else:
            assert L.rr_zscan_pairs_grad(*a, ptr(st), None) == 0
        torch.cuda.synchronize()
        out.append([x.cpu().numpy() for x in o] + [st.cpu().numpy()])
    ref = out[0]
    assert ref[-1][0] == 2 and np.isnan(ref[3][3])
    for got in out[1:]:
        for k in (0, 1, 2, 5, 7):
            np.testing.assert_array_equal(got[k], ref[k])
        for k in (3, 4, 6):
            ok = np.isfinite(ref[k])
            np.testing.assert_array_equal(np.isfinite(got[k]), ok)
            assert np.max(np.abs(got[k] - ref[k])[ok]) <= 1e-9 * np.max(np.abs(ref[k][ok]))
