"""zfind(graph=True) with a pair-scan workspace that takes several rounds per
template: the eager table bit for bit, and one workspace for the plan."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


def test_graph_in_rounds_equals_eager(monkeypatch):
    from redrock_b200 import engine, synth, targets as T, templates as TM, zscan
    from redrock_b200.zfind import zfind
    dz = T.DistTargetsCopy(T.from_synth(synth.make_targets(6, seed=49, first_id=100)))
    tset = synth.template_set()
    dts = []
    for i, step in ((0, 29), (1, 37), (2, 4)):
        tset[i].redshifts = tset[i].redshifts[::step]
        dts.append(TM.DistTemplate(TM.from_synth(tset[i]), dz.wavegrids()))
    _, eager = zfind(dz, dts, nminima=3)
    zscan.clear_caches()
    monkeypatch.setattr(engine, "PAIR_WS_BYTES", 20 << 20)   # 31 of 270 GALAXY pairs
    _, graph = zfind(dz, dts, nminima=3, graph=True)
    plan = next(iter(zscan._plan_cache.d.values()))[1]
    assert plan.pair_ws.numel() == 20 << 20
    for k in eager:
        np.testing.assert_array_equal(graph[k], eager[k], err_msg=k)
