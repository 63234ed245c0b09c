"""The basis builder's redshifts per block, which go by the length of the
redshift grid: the same bits as the oracle's rebin times the standalone
transmission on both sides of every change."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

from oracle import oracle as O  # noqa: E402


@pytest.mark.parametrize("igm", ["Inoue14", "None"])
@pytest.mark.parametrize("nz", [1, 28, 29, 57, 150, 455, 520])
def test_any_redshift_grid(nz, igm):
    """8000 pixels: 63 columns of blocks, so 1 redshift to a block up to 56,
    more from there on and all 16 (Inoue14) from 452, in any order."""
    from redrock_b200.engine import DeviceBasis, GridLayout, TemplateSource
    from redrock_b200.igm import transmission_Lyman
    wave = np.arange(500.0, 9900.0, 1.1)
    flux = np.stack([1.0 + 0.1 * np.sin(wave / 7.0), (wave / 3000.0) ** -1.3])
    grid = 3600.0 + 0.75 * np.arange(8000)
    z = np.random.default_rng(nz).uniform(0.0, 6.0, nz)
    layout = GridLayout.from_dwave({"g": grid})
    got = DeviceBasis.build(TemplateSource(wave, flux, z, igm), layout).data_dict()["g"]
    want = O.trapz_rebin(wave, flux, xnew=grid, myz=z)
    if igm != "None":
        t = transmission_Lyman(z, grid, model=igm)
        if t is not None:
            want = want * t[:, :, None]
    np.testing.assert_array_equal(got, want)
