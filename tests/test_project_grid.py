"""The grids that the projection lays over its passes, computed without a device."""
import ctypes

import pytest

from trak_b200 import _lib

RAD, NOR = 0, 1


def grid(B, F, N, T=148, p=RAD, sms=148):
    out = (ctypes.c_uint32 * 8)()
    rc = _lib.lib().tb_project_grid(B, F, N, T, p, sms, out)
    assert rc == 0, rc
    names = ("columns", "groups", "ctas_per_sm", "tiles", "tiles_per_cta", "bundles", "stages", "chain")
    return dict(zip(names, out))


def busiest_sm(g, N, sms=148):
    """Column tiles x feature tiles that the busiest SM works through, CTAs handed out one by one."""
    per_sm = [0.0] * (sms * g["ctas_per_sm"])
    left = g["tiles"]
    for _ in range(g["bundles"]):
        walked = min(left, g["tiles_per_cta"])
        left -= walked
        for _ in range(N // g["columns"]):
            i = per_sm.index(min(per_sm))
            per_sm[i] += walked
    assert left == 0
    return max(per_sm)


@pytest.mark.parametrize("T,sms", [(148, 148), (132, 132)])
@pytest.mark.parametrize("F", [1_000_003, 11_173_962])
@pytest.mark.parametrize("N", range(512, 4097, 512))
@pytest.mark.parametrize("B", [65, 96, 128])
def test_rademacher_batches_of_65_to_128_rows_fill_the_gpu(B, N, F, T, sms):
    """These are bound by the MMAs: a pass takes as long as the tiles of its busiest SM, whose share must be near the mean
    where the tiles are long.  Tiles of 256 columns cannot be shared: a whole one above the mean is allowed."""
    g = grid(B, F, N, T, RAD, sms)
    mean = g["tiles"] * (N // g["columns"]) / sms
    assert busiest_sm(g, N, sms) <= max(1.16 * mean, -(-g["tiles"] * (N // g["columns"]) // sms))


@pytest.mark.parametrize("F,stages,chain", [(9_472, 1, 1), (28_416, 3, 3), (28_417, 4, 2), (37_889, 5, 3), (100_003, 11, 6),
                                            (1_000_003, 106, 53), (11_173_962, 1180, 256)])
def test_four_groups_drain_in_mid_tile_only_where_the_tile_is_long(F, stages, chain):
    """Chains of up to 48 MMA steps do not drift beyond the rounding of the sums; longer tiles take two chains or more."""
    g = grid(128, F, 1024)
    assert (g["groups"], g["stages"], g["chain"]) == (4, stages, chain)


@pytest.mark.parametrize("p", [RAD, NOR])
@pytest.mark.parametrize("N", [512, 1024, 1536, 4096])
@pytest.mark.parametrize("B", [1, 16, 64, 128])
def test_a_grid_of_at_most_one_cta_per_sm_is_not_packed(B, N, p):
    """The SMs that become free first would otherwise take two CTAs and the others none."""
    g = grid(B, 1_000_003, N, 148, p)
    assert g["ctas_per_sm"] == 1 or g["bundles"] * N // g["columns"] > 148
    assert N != 512 or g["bundles"] * N // g["columns"] == 148


def test_wide_grid_of_short_tiles_takes_fewer_ctas():
    """Eight column tiles: two CTAs of four tiles to an SM where a tile is long, one of eight where the CTA itself costs more."""
    for F, tiles, bundles in ((3_000, 8, 18), (9_472, 8, 19), (20_011, 8, 19), (1_000_003, 4, 37)):
        g = grid(512, F, 1024, 148, NOR)
        assert (g["tiles_per_cta"], g["bundles"]) == (tiles, bundles)
