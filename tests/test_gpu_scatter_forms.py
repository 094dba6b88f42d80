"""The density scatter's forms against the oracle, bit for bit: one and two
window words per bin, values past 32 bits (bins of 4e10 square DBU), cells
inside the window and outside it, up to 3 x 3 bins and more, gcells past the
core's edges, and bin sizes with every remainder."""

import numpy as np
import pytest

from replace_gb300 import netlist as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,chunk", [(0, 0), (16, 1024), (64, 2048)])
@pytest.mark.parametrize("bins_x,bins_y", [(2, 2), (8, 4), (32, 64), (64, 64), (128, 256)])
def test_bin_areas_equal_oracle(gpu_lib, oracle_mod, bins_x, bins_y, tile, chunk):
    from replace_gb300 import Placer
    nl = N.generate(9_000, 9_450, n_io=60, n_macros=6, seed=bins_x + 3 * bins_y, macro_rows=(8, 14))
    kw = dict(target_density=0.75, initial_place_max_iter=0, bin_grid_cnt_x=bins_x, bin_grid_cnt_y=bins_y,
              poisson_path=1)
    p = Placer(nl, scatter_tile=tile, scatter_chunk=chunk, **kw)
    p.initial_place()
    p.nesterov_init()                     # fixes the scatter's shape
    o = oracle_mod.Oracle(nl, **kw)
    o.initial_place()
    assert o.nesterov_base() == 0
    n = o.info.n_gcells
    rng = np.random.default_rng(bins_x * 100 + bins_y)
    lx, ly, ux, uy = nl.core
    # a third anywhere, a third in a corner of the core, a third on bin edges
    xy = np.stack([rng.uniform(lx, ux, n), rng.uniform(ly, uy, n)], 1)
    xy[::3] = rng.uniform(0, 3_000, (len(xy[::3]), 2))
    edge = (ux - lx) / bins_x
    xy[1::3, 0] = lx + edge * rng.integers(0, bins_x + 1, len(xy[1::3]))
    xy = xy.astype(np.float32)
    _, _, st = p.eval(xy, 1e-4)
    _, _, ost, _ = o.eval(xy, 1e-4)
    b, ob = p.bins(bins_x, bins_y), o.bins()
    assert np.array_equal(b["inst_area"], ob["inst_area"])
    assert np.array_equal(b["filler_area"], ob["filler_area"])
    assert st.hpwl == ost.hpwl
    p.close()
