"""How the CTA-pair kernel deals tiles and K pieces to CTA pairs (host-only, no GPU): every unit of
every tile exactly once, whichever way the left-over tiles are cut."""
import ctypes as C

import pytest


def _plan(clib, tiles, clusters, k_pad, tf32):
    out = [C.c_uint32() for _ in range(5)]
    assert clib.cuMpSGEMM_plan_pair(tiles, clusters, k_pad, tf32, *map(C.byref, out)) == 0
    return tuple(o.value for o in out)


def _piece_start(c, whole, total, units, pieces, slices, slice_units):
    """First unit of pair c's piece, in the K loops of the left-over tiles laid end to end."""
    if slice_units == 0:
        return c * (total - whole) * units // pieces
    tile, i = divmod(c, slices)
    return tile * units + i * slice_units


def _items(cluster, grid, total, units, whole, pieces, slices, slice_units):
    """The work items of one pair, as the kernel walks them: (tile, first unit, units, slot)."""
    for t in range(cluster, whole, grid):
        yield t, 0, units, 0
    if cluster < pieces:
        args = (whole, total, units, pieces, slices, slice_units)
        u, end, slot = _piece_start(cluster, *args), _piece_start(cluster + 1, *args), 0
        while u < end:
            t, u0 = divmod(u, units)
            un = min(units - u0, end - u)
            yield whole + t, u0, un, slot
            slot, u = 1, u + un


@pytest.mark.parametrize("tf32", [0, 1])
@pytest.mark.parametrize("clusters", [1, 2, 66, 74])
def test_every_unit_of_every_tile_is_done_once(clib, clusters, tf32):
    kinds = set()
    for tiles in (1, 4, 5, 36, 37, 38, 40, 64, 73, 74, 75, 96, 111, 112, 148, 256, 300, 1000):
        for k_pad in (64, 1024, 1600, 2816, 4096, 8256, 65536):
            units, whole, pieces, slices, slice_units = _plan(clib, tiles, clusters, k_pad, tf32)
            assert units == k_pad // 64 and whole <= tiles and (pieces > 0) == (whole < tiles)
            assert pieces <= clusters and tiles - whole in (0, tiles % clusters)
            if pieces == 0:
                kinds.add("whole")
                continue
            kinds.add("slices" if slice_units else "shared")
            if slice_units:
                assert pieces == (tiles - whole) * slices and slices >= 2
                assert slice_units * 64 >= 1024 and slice_units * (slices - 1) < units <= slice_units * slices
            else:
                assert pieces == clusters
            done, scratch = {}, set()
            grid = min(clusters, max(whole, pieces))
            for c in range(grid):
                for tile, u0, un, slot in _items(c, grid, tiles, units, whole, pieces, slices, slice_units):
                    assert un > 0
                    done.setdefault(tile, []).append((u0, un, c, slot))
                    if un != units:
                        assert (c, slot) not in scratch    # a partial item's scratch tile is its own
                        scratch.add((c, slot))
            assert sorted(done) == list(range(tiles))
            for tile, parts in done.items():
                parts.sort()
                at = 0
                for u0, un, _, _ in parts:
                    assert u0 == at
                    at += un
                assert at == units
                if tile >= whole:
                    # ascending k is ascending pair, without gaps, and every piece but the first is
                    # its pair's first item: what the kernel that adds the pieces relies on
                    cs = [p[2] for p in parts]
                    assert len(parts) > 1 and cs == list(range(cs[0], cs[0] + len(cs)))
                    assert all(p[3] == 0 for p in parts[1:])
    if clusters >= 66:
        assert kinds == {"whole", "slices", "shared"}


def test_agrees_with_the_slice_query(clib):
    """cuMpSGEMM_plan_pair_tail describes the plans that cut tiles into slices, and calls the others
    uncut."""
    for tiles in (1, 4, 37, 38, 64, 96, 256, 1000):
        for k_pad in (1024, 4096, 65536):
            units, whole, pieces, slices, slice_units = _plan(clib, tiles, 74, k_pad, 0)
            out = [C.c_uint32() for _ in range(4)]
            assert clib.cuMpSGEMM_plan_pair_tail(tiles, 74, k_pad, 0, *map(C.byref, out)) == 0
            got = tuple(o.value for o in out)
            if slice_units:
                assert got == (whole, slices, 64 * slice_units, whole + pieces)
            else:
                assert got == (tiles, 1, k_pad, tiles)


def test_plan_rejects_bad_arguments(clib):
    out = [C.c_uint32() for _ in range(5)]
    for bad in ((0, 74, 4096, 0), (1, 0, 4096, 0), (1, 74, 0, 0), (1, 74, 100, 0)):
        assert clib.cuMpSGEMM_plan_pair(*bad, *map(C.byref, out)) == 1
