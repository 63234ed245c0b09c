"""The few-target scan (rr_zscan_few) against the oracle at the sizes where
its steps and lanes end, and its independence of the batch around a target.

Tolerances: those of the fused scan's parity tests -- |dchi2| <= 2e-5,
identical best-z index, coefficients within 1e-5 of max|c| per redshift."""

import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

from oracle import oracle as O  # noqa: E402
from redrock_b200 import synth  # noqa: E402


def _cameras(npix):
    """Grids of the given lengths at 0.8 A from 3700 A on."""
    out, lo = [], 3700.0
    for i, n in enumerate(npix):
        out.append((f"c{i}", lo, lo + 0.8 * (n - 1)))
        lo += 0.8 * n + 10.0
    return tuple(out)


def _basis(nb):
    """Sinusoids of 25 to 60 A: full rank on the shortest grids below
    (condition number of M up to 3e7 there), which the galaxy basis is not."""
    w = np.arange(1500.0, 10000.0, 0.4)
    f = [1.0 + 0.5 * np.sin(2 * np.pi * w / (25.0 + 4.0 * i) + i) + 0.05 * i for i in range(nb)]
    return w, np.stack(f)


@pytest.mark.parametrize("nb,npix,count,nz", [
    (10, (96, 97), 1, 9),        # one step, one step and a lane of the next
    (10, (95, 300, 191), 3, 8),  # ragged steps over three grids
    (7, (288, 120), 2, 1),       # whole steps; one redshift of the eight
    (4, (2751, 2326, 2881), 10, 17),
    (5, (49, 1000), 5, 16),
    (1, (24, 25), 2, 7),
])
def test_few_vs_oracle(nb, npix, count, nz):
    from redrock_b200 import targets as T, templates as TM
    from redrock_b200.engine import (DeviceBasis, GridLayout, TargetBatch, TargetPack,
                                     TemplateSource, run_fused)
    cams = _cameras(npix)
    tg = synth.make_targets(count, seed=300 + nb, cameras=cams, mask_range=(0.0, 0.3))
    grids = {c: synth.camera_wave(lo, hi) for c, lo, hi in cams}
    gw, gf = _basis(nb)
    z = np.linspace(0.1, 0.9, nz)
    ts = synth.TemplateSpec("GALAXY", f"n{nb}", gw, gf, z, "Inoue14")
    layout = GridLayout.from_dwave(grids)
    basis = DeviceBasis.build(TemplateSource.from_template(TM.from_synth(ts)), layout)
    pack = TargetPack(TargetBatch(T.from_synth(tg), layout).to_device())
    res, st = run_fused(pack, [basis], tail=count)
    st.check("few")
    tdata = O.template_basis(ts.wave, ts.flux, z, grids, ts.igm_model)
    ospec = [[O.OSpectrum(s.band, s.wave, s.flux, s.ivar, s.rdata, s.roffsets)
              for s in t.spectra] for t in tg]
    ozc, oco, ope = O.calc_zchi2(ospec, tdata, nz, nb, OIItemplate=O.oii_template(gw, gf))
    zc, co = res[0].zchi2.cpu().numpy(), res[0].zcoeff.cpu().numpy()
    assert np.max(np.abs(zc - ozc)) <= 2e-5
    np.testing.assert_array_equal(np.argmin(zc, axis=1), np.argmin(ozc, axis=1))
    scale = np.maximum(np.abs(oco).max(axis=-1, keepdims=True), 1e-300)
    assert np.all(np.abs(co - oco) <= 1e-5 * scale)
    np.testing.assert_allclose(res[0].penalty.cpu().numpy(), ope, rtol=1e-6, atol=1e-8)
    # one target alone gives the same bits
    one = TargetPack(TargetBatch(T.from_synth(tg[count - 1:]), layout).to_device())
    r1, st = run_fused(one, [basis], tail=1)
    st.check("few")
    assert np.array_equal(r1[0].zchi2.cpu().numpy()[0], zc[-1])
    assert np.array_equal(r1[0].zcoeff.cpu().numpy()[0], co[-1])


def test_few_all_masked_and_resweep():
    """An all-masked target keeps HUGE_CHI2 and zero coefficients; the
    ill-conditioned fits of a dropped camera take the residual sweep."""
    import torch
    from redrock_b200 import targets as T, templates as TM, zscan
    from redrock_b200.engine import run_fused
    tg = synth.make_targets(3, seed=97, amp=50.0, drop_camera_frac=1.0, zrange=(1.3, 1.5))
    for s in tg[1].spectra:
        s.ivar[:] = 0.0
    gal = synth.template_set()[0]
    gal.redshifts = gal.redshifts[-400::16]
    rt = T.from_synth(tg)
    dt = TM.DistTemplate(TM.from_synth(gal), synth.camera_grids())
    zc, co, pe = zscan.calc_zchi2([t.id for t in rt], rt, dt)
    assert np.all(zc[1] == 9999999.0) and np.all(co[1] == 0.0) and np.all(pe[1] == 0.0)
    counter = run_fused.last_counter.cpu().numpy()
    assert counter[2] > 0 and counter[3] > 0
    torch.cuda.synchronize()
    tdata = O.template_basis(gal.wave, gal.flux, gal.redshifts, synth.camera_grids(),
                             gal.igm_model)
    ospec = [[O.OSpectrum(s.band, s.wave, s.flux, s.ivar, s.rdata, s.roffsets)
              for s in t.spectra] for t in tg]
    ozc, _, _ = O.calc_zchi2(ospec, tdata, len(gal.redshifts), 10,
                             OIItemplate=O.oii_template(gal.wave, gal.flux))
    assert np.max(np.abs(zc - ozc)) <= 2e-5


@pytest.mark.parametrize("method,nb,n", [("NMF", 5, 3), ("NMF", 10, 1), ("BVLS", 4, 2)])
def test_bounded_scan_equals_plain_chain(method, nb, n):
    """A bounded template's scan against the plain per-target chain it
    replaced, with a dropped camera, a masked target and a negative weight
    (which keeps the plain chain): chi2 within 1e-9 relative (both sum 8000
    squared residuals in FP64), identical active sets."""
    from redrock_b200 import targets as T, templates as TM, zscan
    from redrock_b200.engine import ScanResult
    tg = synth.make_targets(n, seed=11, amp=1.0, drop_camera_frac=0.4)
    gal = synth.template_set(zsub=211)[0]
    tm = TM.Template(spectype="GALAXY", subtype="b", redshifts=gal.redshifts, wave=gal.wave,
                     flux=gal.flux[:nb].copy(), method="NMF", igm_model=gal.igm_model)
    tm._method = method
    rt = T.from_synth(tg)
    if n > 2:
        rt[1].spectra[0].ivar[100] = -1e-3
        for s in rt[2].spectra:
            s.ivar[:] = 0.0
    dt = TM.DistTemplate(tm, synth.camera_grids())
    zc, co, _ = zscan.calc_zchi2([t.id for t in rt], rt, dt)
    ref = ScanResult(n, dt.basis, dt.basis.basis.device)
    for i, t in enumerate(rt):
        zscan._plain_target(t, dt.basis, dt.layout, ref, i)
    rz, rc = ref.zchi2.cpu().numpy(), ref.zcoeff.cpu().numpy()
    np.testing.assert_allclose(zc, rz, rtol=1e-9)
    np.testing.assert_array_equal(co == 0, rc == 0)
    scale = np.maximum(np.abs(rc).max(axis=-1, keepdims=True), 1e-300)
    assert np.all(np.abs(co - rc) <= 1e-5 * scale)


@pytest.mark.parametrize("n", [32, 70])
def test_y_choice_per_template(n):
    """The default y is the scan's own FP64 sum for the templates y_in_scan
    names -- bit-identical to ygemm="fp64" there -- and the INT8 GEMM for the
    others; the choice follows the whole batch, not the chunk."""
    import torch
    from redrock_b200 import targets as T, templates as TM, zscan
    from redrock_b200.engine import TargetBatch, TargetPack, run_fused, y_in_scan
    tg = T.from_synth(synth.make_targets(n, seed=87))
    tset = synth.template_set()
    sel = [tset[0], tset[2]]                       # GALAXY at full length, one STAR
    dts = [TM.DistTemplate(TM.from_synth(t), synth.camera_grids()) for t in sel]
    bases = [d.basis for d in dts]
    assert not y_in_scan(bases[0], n) and y_in_scan(bases[1], n)
    pack = TargetPack(TargetBatch(tg, dts[0].layout).to_device())
    tail = n % 32
    got, st = run_fused(pack, bases, tail=tail)
    ref, st2 = run_fused(pack, bases, ygemm="fp64", tail=tail)
    st.check("mixed")
    st2.check("fp64")
    assert torch.equal(got[1].zchi2, ref[1].zchi2) and torch.equal(got[1].zcoeff, ref[1].zcoeff)
    assert float((got[0].zchi2 - ref[0].zchi2).abs().max()) <= 2e-5
    chunked = zscan.scan_device(tg, dts, chunk=16)
    for a, b in zip(chunked, got):
        assert torch.equal(a.zchi2, b.zchi2) and torch.equal(a.zcoeff, b.zcoeff)
