"""zfind on two ranks (processes sharing cuda:0, their kernels independent) of
a batch whose split leaves other numbers of targets over a block than the
whole has: the one-process table bit for bit, eager and captured."""
import os

import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.test_gpu_multirank import _free_port

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(), reason="needs a CUDA GPU")]

N = 48     # one process: 32 fused and 16 few targets; two ranks: 24 each


def _zfind(comm, graph):
    from redrock_b200 import synth, targets as T, templates as TM
    from redrock_b200.zfind import zfind
    tg = synth.make_targets(N, seed=43, amp=2.0, drop_camera_frac=0.2, first_id=7000)
    dtg = T.DistTargetsCopy(T.from_synth(tg), comm=comm)
    dwave = dtg.wavegrids()
    dts = []
    for ts, step in zip(synth.template_set()[:3], (23, 31, 4)):
        ts.redshifts = ts.redshifts[::step]
        dts.append(TM.DistTemplate(TM.from_synth(ts), dwave, comm=comm))
    return len(dtg.local()), zfind(dtg, dts, nminima=3, graph=graph)[1]


def _worker(rank, world, port, graph, q):
    import datetime

    import torch
    import torch.distributed as dist
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    torch.cuda.set_device(0)
    dist.init_process_group("gloo", rank=rank, world_size=world,
                            timeout=datetime.timedelta(seconds=120))
    try:
        from redrock_b200.shard import TorchComm
        q.put((rank,) + _zfind(TorchComm(), graph))
    finally:
        dist.destroy_process_group()


@pytest.mark.parametrize("graph", [False, True])
def test_split_with_other_tails_equals_one_process(graph):
    import torch.multiprocessing as mp
    _, ref = _zfind(None, graph)
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = _free_port()
    procs = [ctx.Process(target=_worker, args=(r, 2, port, graph, q)) for r in range(2)]
    for p in procs:
        p.start()
    out = {}
    for _ in range(2):
        r, nlocal, zf = q.get(timeout=600)
        out[r] = (nlocal, zf)
    for p in procs:
        p.join(timeout=120)
        assert p.exitcode == 0
    assert out[0][0] == out[1][0] == N // 2 and out[1][1] is None
    zf = out[0][1]
    assert list(zf.keys()) == list(ref.keys())
    for k in zf:
        np.testing.assert_array_equal(zf[k], ref[k], err_msg=k)
