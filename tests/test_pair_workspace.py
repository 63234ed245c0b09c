"""The workspace that a pair scan allocates (CPU, with stand-ins): what its size
query says, capped, and less where the device has less left."""
import pytest
import torch

from redrock_b200 import engine


@pytest.mark.parametrize("n,cap,left,size", [
    (1, 1000, 10 ** 6, 100), (3, 1000, 10 ** 6, 300), (40, 1000, 10 ** 6, 1000),
    (40, 50, 10 ** 6, 100), (40, 1000, 300, 250), (40, 1000, 100, 100), (40, 1000, 99, None),
])
def test_size(monkeypatch, n, cap, left, size):
    def empty(k, dtype=None, device=None):
        if k > left:
            raise torch.cuda.OutOfMemoryError("stand-in")
        return k
    monkeypatch.setattr(torch, "empty", empty)
    monkeypatch.setattr(engine, "PAIR_WS_BYTES", cap)

    def ws():
        return engine._pair_ws(lambda segs, nseg, nb, pairs: 100 * pairs, [], 4, n, None)
    if size is None:
        with pytest.raises(torch.cuda.OutOfMemoryError):
            ws()
    else:
        assert ws() == size
