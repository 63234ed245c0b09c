"""Which scan takes a target does not depend on how many ranks share the
batch (CPU, with stand-ins for the GPU side)."""
import types

import pytest

from redrock_b200 import zscan
from redrock_b200.targets import distribute_targets
from tests import scan_stand_ins as S


def _rank(ids, sizes, world, rank):
    """A DistTargets as rank `rank` of `world` sees it (None: one process)."""
    made = []
    for i in ids:
        t = S.Target(i)
        t.spectra = [None] * sizes[i]
        made.append(t)
    by_id = {t.id: t for t in made}
    mine = ids if world is None else distribute_targets(made, world)[rank]
    comm = None if world is None else types.SimpleNamespace(rank=rank, size=world)
    return types.SimpleNamespace(comm=comm, all_target_ids=ids,
                                 local=lambda: [by_id[i] for i in mine],
                                 local_target_ids=lambda: list(mine))


@pytest.mark.parametrize("n", [9, 20, 40, 48, 52, 70, 500])
def test_routes_do_not_depend_on_the_ranks(monkeypatch, n):
    ids = list(range(1000, 1000 + n))
    sizes = {i: 2 + i % 2 for i in ids}          # uneven shares, another local order
    routes = {}
    for world in (None, 1, 2, 3):
        got = {}
        for rank in range(world or 1):
            rec = S.install(monkeypatch)
            tg = _rank(ids, sizes, world, rank)
            res = zscan.calc_zchi2_targets(tg, [S.template()])
            assert list(res) == tg.local_target_ids()
            for _, _, part, few, ntarget in rec.scans():
                for k, i in enumerate(part):
                    got[i] = (k >= len(part) - few, ntarget)
        routes[world] = got
        assert sorted(got) == ids
    assert routes[1] == routes[None] and routes[2] == routes[None] and routes[3] == routes[None]
    assert sum(few for few, _ in routes[None].values()) == zscan.few_tail(n)
