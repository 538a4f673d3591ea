"""How the streaming kernel deals tiles and K pieces to CTA pairs (host-only, no GPU)."""
import ctypes as C
import itertools

import pytest


def _plan(clib, m, n, k, batch, tile_n, clusters):
    out = [C.c_uint32() for _ in range(5)]
    assert clib.cuMpSGEMM_plan_stream(m, n, k, batch, tile_n, clusters, *map(C.byref, out)) == 0
    return tuple(o.value for o in out)


def _items(total, units, whole, pieces, cluster, clusters):
    """The work items of one pair, as the kernel walks them: (tile, first unit, units, slot)."""
    for t in range(cluster, whole, clusters):
        yield t, 0, units, 0
    if cluster < pieces:
        u_all = (total - whole) * units
        u, end = cluster * u_all // pieces, (cluster + 1) * u_all // pieces
        slot = 0
        while u < end:
            t, u0 = divmod(u, units)
            un = min(units - u0, end - u)
            yield whole + t, u0, un, slot
            slot, u = 1, u + un


@pytest.mark.parametrize("clusters", [1, 2, 66, 74])
@pytest.mark.parametrize("tile_n", [256, 128])
def test_every_unit_of_every_tile_is_done_once(clib, tile_n, clusters):
    sizes = [(256, 200, 65536, 1), (512, 256, 512, 512), (300, 300, 1000, 32), (2560, 960, 3000, 1),
             (1, 1, 1, 1), (256, 256, 64, 75), (1000, 1000, 1000, 9), (256, 128, 4096, 40),
             (2048, 2048, 2048, 1), (512, 512, 130, 37), (256, 256, 16384, 30)]
    for m, n, k, batch in sizes:
        total, units, whole, pieces, slices = _plan(clib, m, n, k, batch, tile_n, clusters)
        assert total == -(-m // 256) * -(-n // tile_n) * batch and units == -(-k // 64)
        assert pieces <= clusters and whole <= total and (pieces > 0) == (whole < total)
        done, pieces_of, scratch = {}, {}, set()
        grid = min(clusters, max(whole, pieces))
        for c in range(grid):
            for tile, u0, un, slot in _items(total, units, whole, pieces, c, grid):
                assert un > 0
                done.setdefault(tile, []).append((u0, un))
                if un != units:
                    # a partial item: its scratch tile is its own
                    assert slices > 1 or (c, slot) not in scratch
                    scratch.add((c, slot))
                    pieces_of.setdefault(tile, []).append((u0, c, slot))
        assert sorted(done) == list(range(total))
        for tile, parts in done.items():
            parts.sort()
            assert [p[0] for p in parts] == list(itertools.accumulate([0] + [p[1] for p in parts[:-1]]))
            assert sum(p[1] for p in parts) == units
        for tile, parts in pieces_of.items():
            # ascending k is ascending cluster, without gaps, and every piece but the first is its
            # cluster's first item: what the kernel that adds them relies on
            parts.sort()
            cs = [p[1] for p in parts]
            assert cs == list(range(cs[0], cs[0] + len(cs)))
            assert all(p[2] == 0 for p in parts[1:])
            first_unit = (tile - whole) * units
            starts_here = cs[0] * ((total - whole) * units) // pieces == first_unit
            assert parts[0][2] == (0 if starts_here else 1)
        if slices > 1:
            assert whole == 0 and pieces == slices * total
            assert all(len(p) == slices for p in done.values())
            for c in range(pieces):   # one item per pair: slice index = pair modulo slices
                (item,) = _items(total, units, whole, pieces, c, grid)
                assert item[0] == c // slices
        else:
            assert total - whole < clusters


def test_plan_rejects_bad_arguments(clib):
    out = [C.c_uint32() for _ in range(5)]
    for bad in ((0, 1, 1, 1, 256, 74), (1, 0, 1, 1, 256, 74), (1, 1, 0, 1, 256, 74),
                (1, 1, 1, 0, 256, 74), (1, 1, 1, 1, 64, 74), (1, 1, 1, 1, 256, 0)):
        assert clib.cuMpSGEMM_plan_stream(*bad, *map(C.byref, out)) == 1
