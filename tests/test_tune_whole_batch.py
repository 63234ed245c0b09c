"""The tile tuner times the kernels that run (CPU, with stand-ins): a chunk is
tuned with the size of its whole batch, which decides where y is summed, and
the two kernels' choices are kept apart."""
import types

import torch

from redrock_b200 import autotune, engine, zscan
from tests import scan_stand_ins as S


def test_tuner_times_the_kernel_that_runs(monkeypatch):
    rec = S.install(monkeypatch)
    ran = []

    def run(pack, bases, tiles=None, kernel_events=None, tail=None, ntarget=None, scan_tail=True):
        ran.append((ntarget, tuple(tiles.items())))
        if kernel_events is not None:
            kernel_events.append((types.SimpleNamespace(elapsed_time=lambda e: 1.0), None))
    monkeypatch.setattr(engine, "run_fused", run)
    # y in the scan for batches below 100 targets, as y_in_scan has it for STAR
    monkeypatch.setattr(engine, "y_in_scan", lambda basis, n: n < 100)
    monkeypatch.setattr(zscan, "y_in_scan", lambda basis, n: n < 100)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)
    monkeypatch.setattr(zscan, "AUTOTUNE", True)
    monkeypatch.setattr(autotune, "_cache", {})
    targets = [S.Target(i) for i in range(192)]
    zscan.scan_device(targets, [S.template()], chunk=64, host=True)
    assert ran and {n for n, _ in ran} == {192}
    assert {n for *_, n in rec.scans()} == {192}
    # another batch of chunks as large, with y in the scan: tuned by itself
    del ran[:]
    zscan.scan_device(targets[:64], [S.template()], host=True)
    assert ran and {n for n, _ in ran} == {64}
    # and neither again
    del ran[:]
    zscan.scan_device(targets, [S.template()], chunk=64, host=True)
    zscan.scan_device(targets[:64], [S.template()], host=True)
    assert not ran
