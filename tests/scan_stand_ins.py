"""Stand-ins for the scan's GPU side (streams, events, packing, launches), so
that the host code around the launches runs on the CPU and its order is
recorded."""
import contextlib
import types

import numpy as np
import torch

from redrock_b200 import _lib, device, zscan
from redrock_b200.engine import GridLayout


class Stream:
    def __init__(self, rec, name):
        self.rec, self.name, self.cuda_stream = rec, name, 16

    def wait_event(self, ev):
        self.rec.log.append(("wait", self.name, ev.on))

    def synchronize(self):
        pass


class Recorder:
    """The streams of one device and what was done on them, in order:
    ("wait", stream, stream waited for), ("digits", stream, nbasis),
    ("scan", stream, target ids, targets of the few-target scan among them,
    batch size given for the y rule)."""

    def __init__(self):
        self.log = []
        self.main, self.lane = Stream(self, "main"), Stream(self, "lane")
        self.side = Stream(self, "side")
        self.current = self.main

    @contextlib.contextmanager
    def on(self, s):
        was, self.current = self.current, s
        try:
            yield
        finally:
            self.current = was

    def scans(self):
        return [e for e in self.log if e[0] == "scan"]


class _Host:
    def __init__(self, ntarget, basis):
        self.t = [torch.zeros((ntarget, basis.nz)), torch.zeros((ntarget, basis.nz, basis.nbasis)),
                  torch.zeros((ntarget, basis.nz))]
        self.zchi2, self.zcoeff, self.penalty = (x.numpy() for x in self.t)


class _Result:
    def __init__(self, n, basis):
        self.zchi2 = torch.zeros((n, basis.nz))
        self.zcoeff = torch.zeros((n, basis.nz, basis.nbasis))
        self.penalty = torch.zeros((n, basis.nz))


class Target:
    def __init__(self, i):
        self.id = i
        self.spectra = []


def template(full_type="GALAXY", nbasis=4, nz=11):
    """A DistTemplate as far as the stand-ins look."""
    layout = GridLayout([("b", 240, np.arange(240.0))])
    basis = types.SimpleNamespace(method=_lib.RR_SOLVE_PCA, stride=nbasis + nbasis % 2,
                                  nbasis=nbasis, nz=nz, layout=layout)
    return types.SimpleNamespace(basis=basis, layout=layout, comm=None,
                                 template=types.SimpleNamespace(full_type=full_type,
                                                                redshifts=np.arange(float(nz)),
                                                                nbasis=nbasis))


def install(monkeypatch):
    """Put the stand-ins in place of zscan's GPU side; the Recorder."""
    rec = Recorder()

    class Event:
        on = None

        def record(self, stream=None):
            self.on = (stream or rec.current).name

    def run(pack, bases, status=None, tiles=None, tail=None, ntarget=None):
        rec.log.append(("scan", rec.current.name, [t.id for t in pack.targets], tail, ntarget))
        return [_Result(len(pack.targets), b) for b in bases], status

    def pack(targets, layout, *a):
        return types.SimpleNamespace(targets=list(targets), ntarget=len(targets), layout=layout,
                                     nblock=max(1, -(-len(targets) // 32)))

    def bases_for(dts, layout):
        for d in dts:
            d.basis.i8_digits = lambda kpad, variant, n=d.basis.nbasis: rec.log.append(
                ("digits", rec.current.name, n))
        return [d.basis for d in dts]
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: rec.current)
    monkeypatch.setattr(torch.cuda, "stream", rec.on)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda self, s: None)
    monkeypatch.setattr(device, "StatusWord",
                        lambda *a: types.SimpleNamespace(check=lambda what: None, ptr=0))
    for name, v in dict(_lane_stream=lambda: rec.lane, _side_stream=lambda: rec.side,
                        HostResult=_Host, run_fused=run, _bases_for=bases_for, _pack=pack,
                        _pack_overlapped=pack, AUTOTUNE=False,
                        _pack_cache=zscan.IdCache(4)).items():
        monkeypatch.setattr(zscan, name, v)
    return rec
