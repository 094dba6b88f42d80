"""The Poisson solve's group form (grids of 256 to 2048 bins per axis) against
64-bit transforms, at every pair of transform lengths, and its batched use.

Tolerance 2e-6 relative L2: an FP32 FFT of n points has a relative error of
about 0.6e-7 sqrt(log2 n), four transforms of up to 2048 points and the
spectral division stay below 1e-6; a wrong element of one row or column would
show as 1e-3 and more.
"""

import math

import numpy as np
import pytest

from conftest import rel_l2
from replace_gb300 import netlist as N

pytestmark = pytest.mark.gpu

SIZES = [256, 512, 1024, 2048]


def fp64_solve(d, bsx, bsy):
    """(phi, Ex, Ey) by cosine and sine matrices in float64."""
    import torch
    ny, nx = d.shape
    x = torch.from_numpy(d).double().cuda()

    def mats(n):
        k = torch.arange(n, dtype=torch.float64, device="cuda")
        a = math.pi * k[:, None] * (k[None, :] + 0.5) / n       # [k, m]
        return torch.cos(a), torch.sin(a)
    cx, sx = mats(nx)
    cy, sy = mats(ny)
    c = (cy @ x @ cx.T) * (4.0 / (nx * ny))
    c[0] *= 0.5
    c[:, 0] *= 0.5
    wx = math.pi * torch.arange(nx, dtype=torch.float64, device="cuda") / nx
    wy = math.pi * torch.arange(ny, dtype=torch.float64, device="cuda") / ny * (bsy / bsx)
    w2 = wx[None] ** 2 + wy[:, None] ** 2
    w2[0, 0] = 1.0
    ph = c / w2
    ph[0, 0] = 0.0
    return [t.cpu().numpy() for t in (cy.T @ ph @ cx, cy.T @ (ph * wx[None]) @ sx, sy.T @ (ph * wy[:, None]) @ cx)]


@pytest.mark.parametrize("phi", [True, False])
@pytest.mark.parametrize("ny", SIZES)
@pytest.mark.parametrize("nx", SIZES)
def test_solve_matches_fp64(gpu_lib, nx, ny, phi):
    import torch
    from replace_gb300.placer import poisson_solve
    rng = np.random.default_rng(nx * 7 + ny)
    d = (0.7 + 0.4 * rng.random((ny, nx)) + np.outer(np.linspace(0, 1, ny), np.linspace(0.5, 0, nx))).astype(np.float32)
    dd = torch.from_numpy(d).cuda()
    out = [torch.full_like(dd, 7.0) for _ in range(3)]
    poisson_solve(dd.data_ptr(), out[0].data_ptr() if phi else 0, out[1].data_ptr(), out[2].data_ptr(), nx, ny, 380, 1400)
    torch.cuda.synchronize()
    ref = fp64_solve(d, 380, 1400)
    for got, want in list(zip(out, ref))[0 if phi else 1:]:
        assert rel_l2(got.cpu().numpy(), want) < 2e-6


def test_batch_takes_group_form_grids(gpu_lib):
    """Jobs on group-form grids that are not square beside one on a
    block-form grid, batched: each equals the job alone bit for bit."""
    from replace_gb300 import Placer, batch_nesterov_run
    nl = N.generate(6_000, 6_300, n_io=100, seed=31)
    grids = [(512, 256), (64, 64), (256, 512)]

    def job(bx, by):
        p = Placer(nl, target_density=0.75, poisson_path=1, bin_grid_cnt_x=bx, bin_grid_cnt_y=by,
                   initial_place_max_iter=2)
        p.initial_place()
        p.nesterov_init()
        return p
    ps = [job(*g) for g in grids]
    batch_nesterov_run(ps, 20)
    for p, g in zip(ps, grids):
        q = job(*g)
        q.nesterov_run(20)
        assert np.array_equal(p.gcell_coords(), q.gcell_coords()), g
        p.close()
        q.close()
