"""The pair-scan workspace of zfind(graph=True)'s device plan (CPU, with
stand-ins for the GPU side)."""
import contextlib
import types

import numpy as np
import torch

from redrock_b200 import _lib, autotune, device, engine, zfind, zscan


def test_templates_of_a_plan_share_one_workspace(monkeypatch):
    """One workspace, made before any capture (outside the graphs' memory
    pools) and large enough for the largest template, serves the fine-grid
    scans of all templates."""
    n, nminima, nfine = 5, 3, 15
    seg = _lib.PairSegment(None, None, 100, 0, 1.0)
    rows = types.SimpleNamespace(segments=[seg], rows=torch.zeros(1))
    batch = types.SimpleNamespace(batch=types.SimpleNamespace(nblock=1))
    got, made, capturing = [], [], []

    def capture(fn):
        capturing.append(True)
        out = fn()
        capturing.pop()
        return None, out

    def ws(nbytes, segs, nbasis, pairs, dev):
        assert not capturing
        made.append((nbasis, pairs))
        return torch.zeros(1)
    monkeypatch.setattr(device, "StatusWord", lambda *a: types.SimpleNamespace(ptr=0))
    monkeypatch.setattr(device, "to_device", lambda a, *b: a)
    monkeypatch.setattr(device, "capture_graph", capture)
    monkeypatch.setattr(engine, "TargetBatch",
                        lambda *a: types.SimpleNamespace(to_device=lambda: batch))
    monkeypatch.setattr(engine, "TargetPack", lambda *a, **kw: None)
    monkeypatch.setattr(engine, "TemplateSource",
                        types.SimpleNamespace(from_template=lambda t: t))
    monkeypatch.setattr(engine, "run_fused", lambda pack, bases, **kw: (
        [types.SimpleNamespace(zchi2=None, penalty=None) for _ in bases], None))
    monkeypatch.setattr(engine, "FitzCandidates", lambda *a: types.SimpleNamespace(
        pair_t=None, pair_z=torch.zeros(n * nminima * nfine)))
    monkeypatch.setattr(engine, "run_pairs_device",
                        lambda *a, ws=None, **kw: got.append(ws) or (None, None, None))
    monkeypatch.setattr(engine, "_pair_ws", ws)
    monkeypatch.setattr(zfind, "RowPack", lambda b: rows)
    monkeypatch.setattr(zscan, "_bases_for", lambda ts, lay: [
        types.SimpleNamespace(oii=None) for _ in ts])
    monkeypatch.setattr(autotune, "choice", lambda *a, **kw: {4: 1})
    monkeypatch.setattr(zfind, "_warm_devices", {0})
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    ts = [types.SimpleNamespace(template=types.SimpleNamespace(nbasis=nb, redshifts=np.arange(9.0)))
          for nb in (4, 10, 5)]
    for graph in (True, False):
        del got[:], made[:]
        plan = zfind.DeviceFitzPlan(list(range(n)), ts, None, nminima=nminima, nfine=nfine,
                                    graph=graph)
        if not graph:
            monkeypatch.setattr(torch.cuda, "Event",
                                lambda: types.SimpleNamespace(record=lambda: None))
            monkeypatch.setattr(zfind, "_read_stream", contextlib.nullcontext)
            plan.launch()
        assert made == [(10, n * nminima * nfine)]
        assert len(got) == 3 and all(g is plan.pair_ws for g in got)
