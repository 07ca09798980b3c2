"""Work units of two widths where the last round of equal ones would be nearly empty (ts_plan_schedule): every
(tile, 64-row granule) once, whatever the number of units per SM, and no worse balanced than the whole units are."""
import numpy as np
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


def test_few_units_per_sm_are_balanced():
    """12 tiles of 12800 rows: 600 whole units are 4.05 per SM, so one SM in five would run a fifth one."""
    kc, nc = [384] * 12, [128] * 12
    urows, grid, units, cost = plan(kc, nc, 768, 12800)
    width = units[:, 3]           # (the ends of the tiles' lines give a few narrower ones)
    assert (width == 192).sum() >= 148 and (width == 256).sum() >= 148 and urows == 256 and grid == 148
    assert cost.mean() / cost.max() > 0.9
    skewed = np.array([384] * 6 + [100] * 6)
    _, _, units, cost = plan(skewed, nc, 768, 12800)
    check_cover(units, skewed, nc, 12800, 256, 148)
    assert cost.mean() / cost.max() > 0.85
