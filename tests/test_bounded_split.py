"""How a bounded scan splits its targets (CPU, with stand-ins)."""
import types

import numpy as np
import torch

from redrock_b200 import device, zscan


def test_split_is_one_pass(monkeypatch):
    """The targets that need the plain chain are found without a set of them
    built per target (ten thousand such targets: 10^8 steps)."""
    made = []
    monkeypatch.setattr(zscan, "set", lambda *a: made.append(1) or set(*a), raising=False)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch, "zeros", lambda *a, **kw: None)
    monkeypatch.setattr(device, "StatusWord",
                        lambda *a: types.SimpleNamespace(check=lambda what: None))
    monkeypatch.setattr(zscan, "ScanResult", lambda n, b, dev: [None] * n)
    done = []
    monkeypatch.setattr(zscan, "_plain_target", lambda t, b, lay, res, i: done.append(i))
    bad = types.SimpleNamespace(spectra=[types.SimpleNamespace(ivar=np.array([1.0, -1.0]))])
    basis = types.SimpleNamespace(stride=2, nbasis=1)
    zscan._bounded_scan([bad] * 500, [basis], None)
    assert done == list(range(500))
    assert len(made) <= 1
