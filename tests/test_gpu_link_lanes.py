"""2D link detection and link cells on either side of the rule for a surface's
lanes per segment (32 lanes up to 16 segments per SM, 8 beyond), at the ends of
the link-cell kernel's range: four segments of many cells each, and thousands
far shorter than a cell.  Links must be the oracle's, entry for entry; moments
within 4e-6 after a few steps (test_gpu_random_flags.py), forces within 1e-4 of
the largest."""
import numpy as np
import pytest

from freeflow_b200 import workloads as W

from helpers import make_gpu, make_oracle, max_abs, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nseg", [4, 128, 2500, 9000])
def test_cylinder_segments(cuda, nseg):
    def make():
        return W.cylinder_channel_2d(nx=200, ny=120, radius=35.0, center=(80.3, 60.2), nseg=nseg, seed=nseg)

    wl = make()
    g, surf = make_gpu(wl)
    o = make_oracle(wl)
    v, u = wl.surface_at(0)
    surf.update(v, u)
    gcq, gkey = g.debug_links(surf)
    o.step(v, u, wl.elements, None)
    ocq, okey = o.links()
    g.close()
    o.close()
    assert len(ocq) > 200
    assert np.array_equal(gcq, ocq) and np.array_equal(gkey, okey)
    gm, om, gf, of, _ = run_pair(make(), 4)
    assert max_abs(gm, om) <= 4e-6
    assert max_abs(gf, of) <= 1e-4 * np.abs(of).max()
