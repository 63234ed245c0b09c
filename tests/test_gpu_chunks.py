"""A batch that the few-target scan takes whole, in chunks on two streams,
right after its templates were built: the same bits as in one launch."""
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("n,chunk", [(20, 8), (12, 5)])
def test_chunked_few_targets_equal_one_launch(n, chunk):
    import torch
    from redrock_b200 import synth, targets as T, templates as TM, zscan
    tg = T.from_synth(synth.make_targets(n, seed=51))
    tms = [TM.from_synth(t) for t in synth.template_set(zsub=7)[:3]]
    grids = synth.camera_grids()
    zscan.clear_caches()
    a = zscan.scan_device(tg, [TM.DistTemplate(t, grids) for t in tms], chunk=chunk)
    b = zscan.scan_device(tg, [TM.DistTemplate(t, grids) for t in tms])
    for x, y in zip(a, b):
        for k in ("zchi2", "zcoeff", "penalty"):
            assert torch.equal(getattr(x, k), getattr(y, k)), k
