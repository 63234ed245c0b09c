"""Which batches are gathered by threads (CPU, with a stand-in for pinned
memory): the large ones only, with the same contents either way."""
import types

import numpy as np
import pytest
import torch

from redrock_b200 import _lib, engine


@pytest.mark.parametrize("ntarget,threads", [(2, False), (5, False), (6, True), (7, True)])
def test_small_batches_are_copied_in_place(monkeypatch, ntarget, threads):
    """Six targets of 3 MB make 16 MB and more."""
    npix = 33000
    rng = np.random.default_rng(0)
    data = [rng.normal(size=(11, npix)) for _ in range(ntarget)]
    spectra = [types.SimpleNamespace(wave=np.arange(float(npix)), wavehash="g", ivar=d[0], flux=d[1],
                                     R=types.SimpleNamespace(data=d, offsets=np.arange(-5, 6)))
               for d in data]
    targets = [types.SimpleNamespace(spectra=[s]) for s in spectra]
    layout = engine.GridLayout([("g", npix, np.arange(float(npix)))])
    calls = []
    lib = _lib.lib()

    class Lib:
        def rr_host_gather(self, *a):
            calls.append(a)
            return lib.rr_host_gather(*a)
    real = torch.empty
    monkeypatch.setattr(_lib, "lib", lambda: Lib())
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch, "empty", lambda n, dtype=None, pin_memory=False: real(n, dtype=dtype))
    b = engine.TargetBatch(targets, layout)
    assert (b.rdata.nbytes >= 16 << 20) == threads
    np.testing.assert_array_equal(b.rdata, np.concatenate([d.ravel() for d in data]))
    np.testing.assert_array_equal(b.ivar, np.concatenate([d[0] for d in data]))
    np.testing.assert_array_equal(b.flux, np.concatenate([d[1] for d in data]))
    assert bool(calls) == threads


@pytest.mark.parametrize("ntarget,threads", [(2, False), (6, True)])
def test_spectra_of_many_targets(monkeypatch, ntarget, threads):
    """The band rows of an archetype batch go by the same rule."""
    npix = 33000
    d = np.random.default_rng(0).normal(size=(11, npix))
    s = types.SimpleNamespace(wave=np.arange(float(npix)), wavehash="g", ivar=d[0], flux=d[1],
                              R=types.SimpleNamespace(data=d, offsets=np.arange(-5, 6)))
    layout = engine.GridLayout([("g", npix, np.arange(float(npix)))])
    calls = []

    class Lib:
        def rr_host_gather(self, *a):
            calls.append(a)
            return 0

        def rr_pack_band_rows(self, *a):
            return 0
    real = torch.empty
    monkeypatch.setattr(_lib, "lib", lambda: Lib())
    monkeypatch.setattr(engine, "device", lambda: torch.device("cpu"))
    monkeypatch.setattr(engine, "to_device",
                        lambda a, dtype=torch.float64: torch.as_tensor(a).to(dtype))
    monkeypatch.setattr(engine, "StatusWord", lambda dev: types.SimpleNamespace(ptr=0))
    monkeypatch.setattr(engine, "stream_handle", lambda s=None: None)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(torch, "empty",
                        lambda n, dtype=None, pin_memory=False, device=None: real(n, dtype=dtype))
    engine.PlainTarget([s] * ntarget, layout)
    assert bool(calls) == threads
