"""Arrays that are not as long as their wavelength grid (CPU): refused before
anything reads past their end, or completed where scipy defines the rest."""
import numpy as np
import pytest
import scipy.sparse

from redrock_b200 import coadd, synth
from redrock_b200.engine import GridLayout, TargetBatch, spectrum_dia
from redrock_b200.targets import from_synth


def _target():
    return from_synth(synth.make_targets(1, seed=2))[0]


@pytest.mark.parametrize("name", ["ivar", "flux"])
@pytest.mark.parametrize("change", [lambda a: a[:-1], lambda a: np.append(a, 1.0)])
def test_short_and_long_arrays(name, change):
    t = _target()
    setattr(t.spectra[1], name, change(getattr(t.spectra[1], name)))
    with pytest.raises(ValueError):
        TargetBatch([t], GridLayout.from_dwave(synth.camera_grids()))
    with pytest.raises(ValueError):
        coadd.coadd_targets([t])


@pytest.mark.parametrize("form", [scipy.sparse.csr_matrix, lambda r: scipy.sparse.dia_matrix(
    (np.pad(r.data, ((0, 0), (0, 1))), r.offsets), shape=r.shape)])
def test_coadd_of_another_resolution_form(form):
    """numpy refuses R.data * ivar of these in redrock too (ValueError)."""
    t = _target()
    s = t.spectra[0]
    s.R = form(s.R)
    with pytest.raises(ValueError):
        s.R.data * s.ivar
    with pytest.raises(ValueError):
        coadd.coadd_targets([t])


def test_resolution_without_its_last_columns():
    t = _target()
    s = t.spectra[0]
    npix = len(s.wave)
    full = s.R.tocsr().toarray()
    full[:, npix - 7:] = 0.0
    s.R = scipy.sparse.csr_matrix(full)
    d, o = spectrum_dia(s)
    assert d.shape == (len(o), npix) and not d[:, npix - 7:].any()
    got = scipy.sparse.dia_matrix((d, o), shape=(npix, npix)).toarray()
    np.testing.assert_array_equal(got, full)
    b = TargetBatch([t], GridLayout.from_dwave(synth.camera_grids()))
    assert b.rdata.size == sum(len(q.wave) * len(spectrum_dia(q)[1]) for q in t.spectra)
