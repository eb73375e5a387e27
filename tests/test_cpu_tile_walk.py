r"""How a persistent grouped GEMM cuts its tiles among the CTA pairs (host code of the same header)."""
import random

import pytest


@pytest.mark.parametrize("seed", range(40))
def test_every_block_once_and_every_sum_collected(seed):
    from fastmoe_b200.ops import native
    if not native.available():
        pytest.skip("native extension not built")
    walk = native.get().tile_walk
    rng = random.Random(seed)
    groups, pairs = rng.randint(1, 12), rng.choice([1, 3, 74, 74])
    cost_kb, equal = rng.choice([0, 1, 4, 16]), rng.randint(1, 40)
    per_tile = [equal if seed % 2 else rng.randint(1, 40) for _ in range(groups)]
    count = [rng.choice([0, rng.randint(0, 40)]) for _ in range(groups)]
    tiles, units = [0], [0]
    for t, kb in zip(count, per_tile):
        tiles.append(tiles[-1] + t)
        units.append(units[-1] + t * kb)
    parts = [walk(tiles, units, p, pairs, cost_kb) for p in range(pairs)]
    blocks = sorted((g, t, kb) for mine in parts for g, t, kb0, kb1, _n, _l in mine for kb in range(kb0, kb1))
    assert blocks == [(g, t, kb) for g in range(groups) for t in range(count[g]) for kb in range(per_tile[g])]
    handed = 0
    for p, mine in enumerate(parts):
        # at most one sum handed over, before the pair's one tile that has to be collected, its last
        foreign = [i for i, part in enumerate(mine) if part[2] != 0]
        collect = [i for i, part in enumerate(mine) if part[5] >= 0]
        assert len(foreign) <= 1 and collect in ([], [len(mine) - 1]) and not set(foreign) & set(collect)
        handed += len(foreign)
        for i in collect:
            g, t, _kb0, end, num_kb, last = mine[i]
            for q in range(p + 1, last + 1):
                (part,) = [x for x in parts[q] if x[2] != 0]
                assert part[:3] == [g, t, end]
                end = part[3]
                handed -= 1
            assert end == num_kb
    assert handed == 0
    if cost_kb == 0:
        assert all(part[2] == 0 and part[3] == part[4] for mine in parts for part in mine)
