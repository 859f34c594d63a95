"""The terrain generator's corner table against the restatement, bit for bit:
scales whose lattice box fits the table, just about fits, and does not (the
corners are then hashed per cell), coordinates past the integer split's range,
maps that leave blocks partly empty, and every field but the heights zero."""
import numpy as np
import pytest

import hydrogen as H
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 72, 136])
@pytest.mark.parametrize("kw", [dict(), dict(scale=0.003), dict(scale=0.006), dict(scale=0.05),
                                dict(scale=0.05, seed=2.0e4), dict(scale=0.002, seed=3.0e6, octaves=3),
                                dict(domain_warp=2, domain_warp_scale=900.0), dict(domain_warp=0, octaves=12),
                                dict(octaves=0), dict(lacunarity=-1.7, persistance=-0.5, scale=0.004)])
def test_corner_table_bitwise(n, kw):
    ms = H.map_settings(mask_exp=0, hmap_dims=(n, n), **kw)
    w = H.World(n, layers=2)
    for f in ("rock", "dirt", "water", "sediment", "flux_l", "vel_u", "sediment_dirt"):
        w.upload(f, np.full((n, n), 7.0, np.float32))
    w.init_reference_heightmap(ms)
    rock, dirt = O.ref_heightmap(ms, n)
    assert np.array_equal(w.download("rock"), rock, equal_nan=True)
    assert np.array_equal(w.download("dirt"), dirt, equal_nan=True)
    for f in ("water", "sediment", "flux_l", "flux_r", "flux_t", "flux_b", "vel_u", "vel_v", "vel_z", "sediment_dirt"):
        assert not np.any(w.download(f)), f
