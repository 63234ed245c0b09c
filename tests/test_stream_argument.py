"""Calls given a stream of their own (CPU, with stand-ins for the library and
the streams): the buffers they make are ready before the launches on that
stream read or write them, and are kept from reuse until it is done."""
import gc
import types
import weakref

import numpy as np
import pytest
import torch

from redrock_b200 import _lib, engine


class _Pack(types.SimpleNamespace):
    pass


class _Stream:
    def __init__(self, log, name):
        self.log, self.name, self.cuda_stream = log, name, 8

    def wait_stream(self, other):
        self.log.append(("wait", self.name, other.name))


@pytest.fixture
def calls(monkeypatch):
    """(log, current stream, another stream): the log of waits, held buffers
    (their addresses) and library calls with the addresses they get."""
    log = []
    main, side = _Stream(log, "main"), _Stream(log, "side")

    class Lib:
        def __getattr__(self, name):
            if name.endswith("_ws_bytes"):
                return lambda segs, nseg, nb, n: 64 * n
            if name == "rr_few_rows_doubles":
                return lambda tgs: 10

            def call(*a):
                log.append((name, {int(v) for v in a if isinstance(v, int)}))
                return 0
            return call
    monkeypatch.setattr(_lib, "lib", lambda: Lib())
    monkeypatch.setattr(engine, "device", lambda: torch.device("cpu"))
    monkeypatch.setattr(engine, "to_device", lambda a, dtype=torch.float64: torch.as_tensor(
        np.asarray(a)).to(dtype))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: main)
    monkeypatch.setattr(torch.Tensor, "record_stream",
                        lambda t, s: log.append(("hold", s.name, t.data_ptr())))
    return log, main, side


def _check(log, launch):
    """Every buffer the launches get that is held is held, and the wait comes
    first; the held ones include what the call allocated for itself."""
    at = next(i for i, e in enumerate(log) if e[0] == launch)
    assert ("wait", "side", "main") in log[:at]
    held = {e[2] for e in log if e[0] == "hold"}
    assert all(e[1] == "side" for e in log if e[0] == "hold")
    return held, log[at][1]


def _rows():
    return types.SimpleNamespace(rows=torch.zeros(4), fwf=torch.zeros(1), wsum=torch.zeros(1),
                                 sw=torch.zeros(4), npix_row=4,
                                 segments=[_lib.PairSegment(None, None, 4, 0, 1.0)])


def _src():
    z = torch.zeros(4, dtype=torch.float64)
    return types.SimpleNamespace(x=z, nx=4, y=z, nbasis=1, igm=0, method=0, oii_dev=None)


def _st():
    return types.SimpleNamespace(ptr=0)


def test_pair_scan_workspace(calls, monkeypatch):
    log, main, side = calls
    made = []
    real = engine._pair_ws
    monkeypatch.setattr(engine, "_pair_ws", lambda *a: made.append(real(*a)) or made[-1])
    engine.run_pairs(_rows(), _src(), [0, 0], [0.1, 0.2], stream=side, status=_st())
    held, args = _check(log, "rr_zscan_pairs_ws")
    assert made[0].data_ptr() in held & args
    del log[:]
    engine.run_pairs_grad(_rows(), _src(), [0, 0], [0.1, 0.2], stream=side, status=_st())
    held, args = _check(log, "rr_zscan_pairs_grad_ws")
    assert made[1].data_ptr() in held & args
    # on the current stream there is nothing to wait for or to hold
    del log[:]
    for s in (None, main):
        engine.run_pairs(_rows(), _src(), [0, 0], [0.1, 0.2], stream=s, status=_st())
    assert {e[0] for e in log} == {"rr_zscan_pairs_ws"}


@pytest.mark.parametrize("n,tail", [(20, 20), (40, 10)])
def test_scan_tail(calls, n, tail):
    """The few-target scan's rows, and the fused scan's row numbers without
    the tail's."""
    log, main, side = calls
    layout = types.SimpleNamespace(signature=(), pix_stride=64)
    nblock = -(-n // 32)
    pack = _Pack(
        ntarget=n, nblock=nblock, layout=layout, rw=torch.zeros(1),
        rows=torch.arange(32 * nblock, dtype=torch.int32),
        scan_targets_struct=lambda nb=None, rows=None: _lib.ScanTargets(
            1, 1, 1, None if rows is None else rows.data_ptr(), None, nb or nblock, 1, 64))
    basis = types.SimpleNamespace(layout=layout, method=_lib.RR_SOLVE_PCA, stride=2, nbasis=1,
                                  nz=3, basis=torch.zeros(2), prior=None, oii=None)
    res, _ = engine.run_fused(pack, [basis], stream=side, status=_st(), ygemm="fp64", tail=tail)
    lrows, rows = res[0].few
    held, args = _check(log, "rr_pack_few")
    assert lrows.data_ptr() in held & args
    if n > tail:
        held, _ = _check(log, "rr_zscan_fused")
        assert rows.data_ptr() in held
        assert rows[n - tail:].eq(-1).all() and rows[:n - tail].ge(0).all()
    # results a caller keeps do not keep the packed targets (0.8 MB each)
    ref = weakref.ref(pack)
    del pack
    gc.collect()
    assert ref() is None and res
