"""The totals that an evaluation forms on the device, against 64-bit sums of
its outputs."""

import numpy as np
import pytest

from replace_gb300 import netlist as N

pytestmark = pytest.mark.gpu

# rms relative error of the gradient totals over the same 40 placements when
# every block summed fewer, shorter warps (six blocks on a multiprocessor)
SIX_BLOCKS = 4.51e-10


def test_gradient_totals_as_exact_as_with_shorter_sums(gpu_lib):
    from replace_gb300 import Placer
    nl = N.generate(500_000, 525_000, n_io=200, seed=7)
    p = Placer(nl, target_density=0.7, bin_grid_cnt_x=512, bin_grid_cnt_y=512, initial_place_max_iter=0,
               poisson_path=1)
    p.initial_place()
    p.nesterov_init()
    n = p.info.n_gcells
    lx, ly, ux, uy = nl.core
    err = []
    for seed in range(40):
        rng = np.random.default_rng(seed)
        xy = np.stack([rng.uniform(lx + 3000, ux - 3000, n), rng.uniform(ly + 3000, uy - 3000, n)], 1)
        wl, dg, st = p.eval(xy.astype(np.float32), 2e-4)
        for grad, total in ((wl, st.wire_length_grad_sum), (dg, st.density_grad_sum)):
            want = (np.abs(grad[:, 0]) + np.abs(grad[:, 1])).astype(np.float64).sum()
            err.append((total - want) / want)
    p.close()
    assert np.sqrt(np.mean(np.square(err))) <= SIX_BLOCKS
