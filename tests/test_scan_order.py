"""The order that the chunked scan puts on its streams (CPU, with stand-ins
for the GPU side)."""
import pytest

from redrock_b200 import zscan
from tests import scan_stand_ins as S


@pytest.mark.parametrize("n,chunk", [(20, 8), (12, 5), (3, 1), (21, 8), (70, 16)])
def test_second_stream_waits_for_the_first(monkeypatch, n, chunk):
    """Chunks on the second stream read what the first stream made (the bases,
    the status word): it waits for the first before its first scan, whether
    or not the batch has targets for the fused scan."""
    rec = S.install(monkeypatch)
    zscan.scan_device([S.Target(i) for i in range(n)], [S.template()], chunk=chunk, host=True)
    assert sorted({e[1] for e in rec.scans()}) == ["lane", "main"]
    assert [i for e in rec.scans() for i in e[2]] == list(range(n))
    first = next(i for i, e in enumerate(rec.log) if e[0] == "scan" and e[1] == "lane")
    assert ("wait", "lane", "main") in rec.log[:first]
    # what the scans share is made before that wait
    wait = rec.log.index(("wait", "lane", "main"))
    assert all(e[1] == "main" for e in rec.log[:wait])
    assert not any(e[0] == "digits" for e in rec.log[wait:])
