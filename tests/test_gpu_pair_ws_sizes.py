"""The pair scan with exactly the workspace that its size query names, for odd
numbers of pairs too, with and without gradients."""
import ctypes

import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.test_gpu_pairs_ws import _both, _same

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def _case(nb):
    from redrock_b200 import synth, targets as T
    from redrock_b200.engine import GridLayout, RowPack, TargetBatch, TemplateSource
    rng = np.random.default_rng(nb)
    grid = 3700.0 + 0.8 * np.arange(301)
    tg = []
    for t in range(2):
        rd, ro = synth.resolution_dia(len(grid), 1.0)
        tg.append(synth.TargetSpec(t, [synth.SpectrumSpec(
            "c", grid, rng.normal(size=301) + 1.0, rng.uniform(0.3, 4.0, 301), rd, ro)]))
    layout = GridLayout.from_dwave({"c": grid})
    rows = RowPack(TargetBatch(T.from_synth(tg), layout).to_device())
    w = np.arange(900.0, 10500.0, 0.9)
    flux = np.stack([1.0 + np.sin(w / (20.0 + 7.0 * i)) for i in range(nb)])
    return rows, TemplateSource(w, flux, np.array([0.5]), "Inoue14", oii=rng.normal(size=nb))


@pytest.mark.parametrize("nb", [1, 3, 4, 5])
@pytest.mark.parametrize("n,per", [(1, 1), (3, 3), (5, 1), (7, 3)])
def test_exact_workspace(nb, n, per):
    rows, src = _case(nb)
    rng = np.random.default_rng(n)
    a, b = _both(rows, src, rng.integers(0, 2, n), rng.uniform(0.1, 2.5, n), per)
    _same(a, b)


@pytest.mark.parametrize("nb", [1, 4, 5])
@pytest.mark.parametrize("n,per", [(1, 1), (3, 3), (5, 1)])
def test_exact_gradient_workspace(nb, n, per):
    import torch
    from redrock_b200 import _lib
    from redrock_b200.device import ptr, to_device
    L = _lib.lib()
    rows, src = _case(nb)
    rng = np.random.default_rng(n)
    dt = to_device(rng.integers(0, 2, n).astype(np.int32), torch.int32)
    dz = to_device(rng.uniform(0.1, 2.5, n))
    segs = (_lib.PairSegment * len(rows.segments))(*rows.segments)
    tm = _lib.PairTemplate(ptr(src.x), src.nx, ptr(src.y), nb, src.igm, 0, 0, None,
                           ptr(src.oii_dev), None)
    out = []
    for pairs in (per, 64):
        o = [torch.full(s, -1.0, dtype=torch.float64, device="cuda")
             for s in ((n,), (n, nb), (n,), (n,), (n,), (n, rows.npix_row), (n,))]
        st = torch.zeros(1, dtype=torch.int32, device="cuda")
        size = int(L.rr_zscan_pairs_grad_ws_bytes(segs, len(segs), nb, pairs))
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        assert L.rr_zscan_pairs_grad_ws(
            ctypes.byref(tm), segs, len(segs), ptr(rows.rows), ptr(rows.sw), ptr(rows.fwf),
            ptr(rows.wsum), rows.npix_row, ptr(dt), ptr(dz), n, *(ptr(x) for x in o), ptr(ws), size,
            ptr(st), None) == 0
        out.append([x.cpu().numpy() for x in o] + [st.cpu().numpy()])
    assert out[0][-1][0] == 0
    _same(*out)
