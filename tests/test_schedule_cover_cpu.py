"""The work lists of ts_plan_schedule: every (tile, 64-row granule) once, whatever the number of units per SM."""
import pytest

from test_schedule_cpu import check_cover, plan


@pytest.mark.parametrize("n_ctas", [1, 7, 148])
@pytest.mark.parametrize("tiles,M,K,keep", [(12, 12800, 768, 384), (24, 12800, 768, 384), (1, 64 * 1000, 2048, 900), (148, 3 * 256 + 8, 4096, 512),
                                            (37, 20000, 3072, 700), (5, 30008, 2048, 64), (300, 12800, 768, 128)])
def test_every_granule_once(tiles, M, K, keep, n_ctas):
    kc, nc = [keep] * tiles, [128] * tiles
    urows, grid, units, cost = plan(kc, nc, K, M, n_ctas)
    check_cover(units, kc, nc, M, urows, n_ctas)
    assert len(cost) == grid <= n_ctas
