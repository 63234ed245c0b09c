"""The gradient pair scan through a workspace against the one without: every
output the same bits, dT/dz too (its quotients are exactly rounded in both),
also where quotients leave the fast divisions' range or are zero."""
import ctypes

import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("nb,igm,extreme", [(10, "None", False), (4, "Inoue14", False),
                                            (5, "None", True), (3, "Inoue14", True),
                                            (7, "Calura12", True),
                                            # more gradient sums than M and y
                                            (1, "Inoue14", True), (2, "None", False)])
def test_gradients_are_the_same_bits(nb, igm, extreme):
    import torch
    from redrock_b200 import _lib, synth, targets as T
    from redrock_b200.device import ptr, to_device
    from redrock_b200.engine import GridLayout, RowPack, TargetBatch, TemplateSource
    rng = np.random.default_rng(nb)
    grids = {"a": 3700.0 + 0.8 * np.arange(500), "b": 4200.0 + 0.8 * np.arange(247)}
    tg = []
    for t in range(3):
        sp = []
        for band, w in grids.items():
            rd, ro = synth.resolution_dia(len(w), 1.0)
            sp.append(synth.SpectrumSpec(band, w, rng.normal(size=len(w)) + 1.0,
                                         rng.uniform(0.3, 4.0, len(w)), rd, ro))
        tg.append(synth.TargetSpec(t, sp))
    layout = GridLayout.from_dwave(grids)
    rows = RowPack(TargetBatch(T.from_synth(tg), layout).to_device())
    w = np.arange(900.0, 10500.0, 0.9)
    flux = np.stack([1.0 + np.sin(w / (20.0 + 7.0 * i)) for i in range(nb)])
    if extreme:
        flux[-1, 2000:2400] = 0.0
        flux[-1, 2500:2540] = 1e-300
        flux[0, 3000:3003] = [5e-324, -5e-324, 0.0]
    src = TemplateSource(w, flux, np.array([0.5]), igm, oii=rng.normal(size=nb))
    segs = (_lib.PairSegment * len(rows.segments))(*rows.segments)
    tm = _lib.PairTemplate(ptr(src.x), src.nx, ptr(src.y), nb, src.igm, 0, 0, None,
                           ptr(src.oii_dev), None)
    n = 61
    dt = to_device(rng.integers(0, 3, n).astype(np.int32), torch.int32)
    dz = to_device(rng.uniform(0.0, 2.5, n))
    L = _lib.lib()
    out = []
    for ws in (False, True):
        o = [torch.full(s, -1.0, dtype=torch.float64, device="cuda")
             for s in ((n,), (n, nb), (n,), (n,), (n,), (n, rows.npix_row), (n,))]
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        a = (ctypes.byref(tm), segs, len(segs), ptr(rows.rows), ptr(rows.sw), ptr(rows.fwf),
             ptr(rows.wsum), rows.npix_row, ptr(dt), ptr(dz), n) + tuple(ptr(x) for x in o)
        if ws:
            size = int(L.rr_zscan_pairs_grad_ws_bytes(segs, len(segs), nb, n))
            buf = torch.empty(size, dtype=torch.uint8, device="cuda")
            assert L.rr_zscan_pairs_grad_ws(*a, ptr(buf), size, ptr(st), None) == 0
        else:
            assert L.rr_zscan_pairs_grad(*a, ptr(st), None) == 0
        out.append([x.cpu().numpy() for x in o] + [st.cpu().numpy()])
    assert out[0][-1][0] == 0 and np.all(np.isfinite(out[0][3])) and np.any(out[0][3] != 0)
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
