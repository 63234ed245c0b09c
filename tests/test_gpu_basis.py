"""The basis builder's register path (rr_build_basis): shared exactly
corrected divisions, redshifts taken 16 to a block, IGM terms kept between
redshifts.  Every value is bit-identical to the oracle's rebin (redrock's
operations in its order), and with IGM to that rebin times the standalone
transmission kernel's factor -- so the comparisons are for equality."""

import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

from oracle import oracle as O  # noqa: E402


def _template(nb, uneven, seed):
    rng = np.random.default_rng(seed)
    n = 4001
    wave = np.linspace(900.0, 9000.0, n)
    if uneven:
        wave = wave + np.cumsum(rng.uniform(0.0, 0.5, n))
    flux = rng.normal(size=(nb, n))
    flux[0, 1000:1400] = 0.0                 # flat zero: 0 / dx
    flux[-1, 2000:2040] = 1e-300             # quotients below the fast range
    flux[-1, 2100:2110] *= 1e250
    flux[nb // 2, 2500:2503] = [5e-324, -5e-324, 0.0]
    return wave, flux


def _build(wave, flux, z, grid, igm="None"):
    from redrock_b200.engine import DeviceBasis, GridLayout, TemplateSource
    layout = GridLayout.from_dwave({"g": grid})
    return DeviceBasis.build(TemplateSource(wave, flux, z, igm), layout).data_dict()["g"]


@pytest.mark.parametrize("nb,uneven,npix,nz", [
    (1, True, 1, 1), (2, False, 127, 15), (3, True, 128, 16), (4, False, 129, 17),
    (5, True, 118, 33), (7, False, 1000, 2), (10, True, 501, 16), (10, False, 246, 31),
])
def test_build_equals_oracle(nb, uneven, npix, nz):
    wave, flux = _template(nb, uneven, 100 + nb)
    rng = np.random.default_rng(nz)
    z = rng.uniform(0.05, 2.0, nz)           # no order
    # bins from a tenth of a sample to several samples wide
    grid = 3300.0 + np.cumsum(rng.choice([0.3, 1.1, 5.0, 9.0], size=max(npix, 2)))[:max(npix, 2)]
    np.testing.assert_array_equal(_build(wave, flux, z, grid),
                                  O.trapz_rebin(wave, flux, xnew=grid, myz=z))


def test_build_nbasis_above_ten_and_range_error():
    """11 to 16 bases keep the general kernel; a bin outside the template
    raises, as before."""
    import ctypes

    import torch
    from redrock_b200 import _lib
    from redrock_b200.device import ptr, to_device
    from redrock_b200.engine import GridLayout
    wave, flux = _template(11, False, 3)
    grid = np.linspace(3400.0, 3500.0, 40)
    z = np.array([0.3, 0.9])
    layout = GridLayout.from_dwave({"g": grid})
    e, w, emin, emax = layout.device_arrays(0)
    gd = (_lib.GridDesc * 1)(_lib.GridDesc(ptr(e), ptr(w), layout.npix[0], layout.npix_pad[0],
                                           layout.pix_offset[0], emin, emax, 0, 0))
    out = torch.empty((2, layout.pix_stride, 12), dtype=torch.float64, device="cuda")
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    x, y, dz = to_device(wave), to_device(flux), to_device(z)
    rc = _lib.lib().rr_build_basis(ptr(x), len(wave), ptr(y), 11, ptr(dz), 2,
                                   float(wave[0] * (1 + z.max())), float(wave[-1] * (1 + z.min())),
                                   gd, 1, 0, layout.pix_stride, 12, ptr(out), ptr(st), None)
    assert rc == 0 and int(st.item()) == 0
    got = out[:, 5:45, :11].cpu().numpy()
    np.testing.assert_array_equal(got, O.trapz_rebin(wave, flux, xnew=grid, myz=z))
    with pytest.raises(ValueError):
        _build(wave, flux[:4], np.array([0.3, 5.0]), grid)


@pytest.mark.parametrize("model", ["Inoue14", "Calura12", "Kamble20"])
@pytest.mark.parametrize("order", ["up", "down", "mixed"])
def test_build_igm_equals_rebin_times_transmission(model, order):
    from redrock_b200.igm import transmission_Lyman
    wave = np.arange(500.0, 9000.0, 0.7)
    flux = np.stack([1.0 + 0.1 * np.sin(wave / 7.0), (wave / 3000.0) ** -1.3])
    grid = np.arange(3600.0, 6800.0, 11.7)
    # through every branch: z < 1.2, < 2, < 4.7 and above
    z = np.exp(np.linspace(np.log(1.05), np.log(7.0), 61)) - 1.0
    if order == "down":
        z = z[::-1].copy()
    elif order == "mixed":
        z = np.random.default_rng(4).permutation(z)
    got = _build(wave, flux, z, grid, igm=model)
    t = transmission_Lyman(z, grid, model=model)
    want = O.trapz_rebin(wave, flux, xnew=grid, myz=z) * t[:, :, None]
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("nb,npix,nz", [(1, 33, 1), (3, 128, 2), (4, 129, 5), (8, 31, 3), (10, 300, 4),
                                        (11, 65, 2)])
def test_trapz_rebin_equals_oracle(nb, npix, nz):
    """The drop-in rebin in registers (up to ten bases) and the general kernel
    (eleven), and rebin_template's grids from one upload."""
    from types import SimpleNamespace

    from redrock_b200 import rebin
    wave, flux = _template(nb, True, 200 + nb)
    z = np.random.default_rng(nz).uniform(0.05, 2.0, nz)
    grid = 3300.0 + np.cumsum(np.random.default_rng(1).choice([0.3, 1.1, 5.0, 9.0], size=npix))
    want = O.trapz_rebin(wave, flux, xnew=grid, myz=z)
    np.testing.assert_array_equal(rebin.trapz_rebin(wave, flux, xnew=grid, myz=z), want)
    t = SimpleNamespace(wave=wave, flux=flux, minwave=wave[0], maxwave=wave[-1])
    got = rebin.rebin_template(t, z, dwave={"a": grid, "b": grid[:20]})
    np.testing.assert_array_equal(got["a"], want)
    np.testing.assert_array_equal(got["b"], O.trapz_rebin(wave, flux, xnew=grid[:20], myz=z))
    if nb == 1:
        np.testing.assert_array_equal(rebin.trapz_rebin(wave * 1.3, flux[0], xnew=grid),
                                      O.trapz_rebin(wave * 1.3, flux[0], xnew=grid))
