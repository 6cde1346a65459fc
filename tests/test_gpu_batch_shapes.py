"""Launch shapes of a batch's groups: their defaults, and that the tuner leaves one
of its grids (one CTA per tile, or whole waves of 4 CTAs per SM) and nothing else
changed."""
import pytest

import penguin_2_0_b200 as pg


@pytest.mark.gpu
def test_default_and_tuned_shapes(gpu):
    import torch
    wave = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    p = [pg.params(0, imax=72, jmax=150, precision=k, endtime=1e6, tmovie=1e6) for k in (0, 1)]
    runs = [pg.Run(q, 0).load(pg.build_ic(q)) for q in p]
    with pg.Batch(0) as b:
        assert b.shape(0) == dict(grid_x=0, grid_y=0, minb=8)
        assert b.shape(1) == dict(grid_x=0, grid_y=0, minb=4)
        for r in runs:
            r.clock_reset(0)
            b.add(r)
        b.tune(1)
        for g, minb in ((0, 8), (1, 4)):
            s = b.shape(g)
            assert s["minb"] == minb and s["grid_x"] == s["grid_y"]
            assert s["grid_x"] in [k * wave for k in (0, 1, 2, 3, 4, 6)]
        for r in runs:
            b.remove(r)
            r.close()
