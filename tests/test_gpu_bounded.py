"""Scans of templates with a bounded solve (NMF) through calc_zchi2."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def _nmf(nbasis, zsub=211):
    from redrock_b200 import synth, templates as TM
    gal = synth.template_set(zsub=zsub)[0]
    return TM.Template(spectype="GALAXY", subtype=f"n{nbasis}", redshifts=gal.redshifts,
                       wave=gal.wave, flux=np.abs(gal.flux[:nbasis]) + 0.1, method="NMF",
                       igm_model=gal.igm_model)


def _targets(n, seed=11):
    from redrock_b200 import synth, targets as T
    return T.from_synth(synth.make_targets(n, seed=seed))


def test_flux_changed_in_place():
    """The same target objects with other contents give the other contents'
    results, as the per-target chain always did: nothing is kept between
    calls.  Several bounded templates of one call share the packing."""
    from redrock_b200 import synth, templates as TM, zscan
    dts = [TM.DistTemplate(_nmf(nb), synth.camera_grids()) for nb in (5, 3)]
    tg = _targets(3)
    zscan.scan_device(tg, dts, host=True)
    for t in tg:
        for s in t.spectra:
            s.flux *= 2.0
            s.ivar[::7] = 0.0
    got = zscan.scan_device(tg, dts, host=True)
    fresh = _targets(3)
    for t in fresh:
        for s in t.spectra:
            s.flux *= 2.0
            s.ivar[::7] = 0.0
    for dt, g in zip(dts, got):
        ref = zscan.calc_zchi2([t.id for t in fresh], fresh, dt)
        for x, y in zip((g.zchi2, g.zcoeff, g.penalty), ref):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("weight", [np.inf, np.nan, -0.5])
def test_weights_without_a_square_root(weight):
    """A target with a weight that the packed rows cannot hold keeps the
    plain chain's results; the others of its batch keep theirs."""
    from redrock_b200 import synth, templates as TM, zscan
    from redrock_b200.engine import ScanResult
    dt = TM.DistTemplate(_nmf(5), synth.camera_grids())
    tg = _targets(3)
    clean = zscan.calc_zchi2([t.id for t in tg], tg, dt)
    tg[1].spectra[0].ivar[100] = weight
    got = zscan.calc_zchi2([t.id for t in tg], tg, dt)
    ref = ScanResult(3, dt.basis, dt.basis.basis.device)
    zscan._plain_target(tg[1], dt.basis, dt.layout, ref, 1)
    for x, y, z in zip(got, clean, (ref.zchi2, ref.zcoeff, ref.penalty)):
        np.testing.assert_array_equal(x[1], z.cpu().numpy()[1])
        np.testing.assert_array_equal(x[[0, 2]], y[[0, 2]])
