"""The work that users of the placement library have it do, as cases to time.

Seven kinds, each through the public Python entry points over the C ABI:

* ``poisson``     the electrostatic solve alone on device arrays
                  (``poisson_solve``): the call of a framework that has its
                  own density and wants the field.
* ``eval``        one physics evaluation from host coordinates
                  (``Placer.eval``): the gradient-check hook, here with movable
                  macros and per-net weights.
* ``loop``        a chunk of Nesterov iterations of a prepared job
                  (``Placer.nesterov_run``), as a server or a timing-driven
                  caller steps a placement, with the read-back of the
                  coordinates; from the clustered placement that the initial
                  place leaves, or from a spread one (incremental mode).
* ``place``       a whole job from host arrays: create, initial place, init, a
                  first chunk of iterations, coordinates.
* ``ip``          the initial place alone (``Placer.initial_place``): 20 rounds
                  of B2B assembly and BiCGSTAB, with the instance locations.
* ``batch_ip``    the initial places of many small jobs together.
* ``batch_loop``  the Nesterov loops of many small jobs together.

The netlists come from the repository's seeded generator with its sizes: 2k to
1M cells, mixed-size jobs with 10 to 40 macros, bin grids from 64 to 2048 per
axis.  The loop cases hold the density penalty (both phi coefficients 1) and
set the target overflow to 0, so that a chunk can be run again and again at
about the same state: a job's cost per iteration does not depend on the
penalty, and the loop's stop rule would otherwise end a case that is timed for
longer than one placement takes.  The Poisson form is the FFT passes, which
the automatic choice also takes on these grids; pinned, so that no timing
decides what is computed.  The chunks are short: the loop amplifies a
difference of one rounding by about ten in eight iterations of a spread
placement, and of a clustered one in thirty.
"""

import functools
import math

import numpy as np
import torch

from replace_gb300 import Placer, batch_initial_place, batch_nesterov_run
from replace_gb300 import netlist as N
from replace_gb300.placer import poisson_solve


def listed():
    return [
        # the smallest call: a small block's grid, with the potential; launches count
        {"name": "poisson_128_phi", "kind": "poisson", "nx": 128, "ny": 128, "bin_x": 1530, "bin_y": 1460,
         "phi": True},
        # a grid that is not square
        {"name": "poisson_512x256", "kind": "poisson", "nx": 512, "ny": 256, "bin_x": 1701, "bin_y": 1855,
         "phi": False},
        # the grid of a million-cell design, field only (what a loop needs)
        {"name": "poisson_1024", "kind": "poisson", "nx": 1024, "ny": 1024, "bin_x": 1776, "bin_y": 1656,
         "phi": False},
        # the grid of a four-million-cell design, with the potential
        {"name": "poisson_2048_phi", "kind": "poisson", "nx": 2048, "ny": 2048, "bin_x": 2033, "bin_y": 1912,
         "phi": True},
        # one evaluation of a mixed-size design with timing weights
        {"name": "eval_40k_macros", "kind": "eval", "cells": 40_000, "macros": 20, "bins": 256, "weights": True},
        # a small block's loop: latency and launches
        {"name": "loop_10k", "kind": "loop", "cells": 10_000, "macros": 0, "bins": 128, "spread": False,
         "weights": False, "iters": 32},
        # a mixed-size design's loop
        {"name": "loop_200k_macros", "kind": "loop", "cells": 200_000, "macros": 40, "bins": 512, "spread": False,
         "weights": False, "iters": 16},
        # the headline design's loop, from a spread placement
        {"name": "loop_1m", "kind": "loop", "cells": 1_000_000, "macros": 0, "bins": 1024, "spread": True,
         "weights": False, "iters": 6},
        # a whole small job as a user's script runs it
        {"name": "place_30k", "kind": "place", "cells": 30_000, "iters": 64},
        # the initial place of a large block
        {"name": "ip_400k", "kind": "ip", "cells": 400_000},
        # a batch of small blocks: initial places, then loops
        {"name": "batch_ip_16", "kind": "batch_ip", "jobs": 16, "cells_lo": 2_000, "cells_hi": 50_000},
        {"name": "batch_loop_16", "kind": "batch_loop", "jobs": 16, "cells_lo": 2_000, "cells_hi": 50_000,
         "iters": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "eval", "loop", "loop", "place", "ip", "batch_ip", "batch_loop"])
    if kind == "poisson":
        a = rng.randint(6, 11)
        b = min(11, max(6, a + rng.choice([-1, 0, 0, 0, 1])))
        return {"kind": kind, "nx": 1 << a, "ny": 1 << b, "bin_x": rng.randint(700, 2400),
                "bin_y": rng.randint(700, 2400), "phi": rng.random() < 0.5}
    if kind == "eval":
        return {"kind": kind, "cells": _log_int(rng, 2_000, 200_000), "macros": rng.choice([0, rng.randint(10, 40)]),
                "bins": rng.choice([128, 256, 512]), "weights": rng.random() < 0.5}
    if kind == "loop":
        cells = _log_int(rng, 2_000, 600_000)
        spread = rng.random() < 0.5
        # the generator's mixed-size jobs have 10 to 40 macros on 5k to 500k cells
        macros = rng.randint(10, 40) if not spread and cells >= 50_000 and rng.random() < 0.5 else 0
        bins = 1 << min(10, max(6, int(round(math.log2(math.sqrt(1.25 * cells))))))
        return {"kind": kind, "cells": cells, "macros": macros, "bins": bins, "spread": spread,
                "weights": rng.random() < 0.3, "iters": rng.randint(4, 6) if spread else rng.randint(8, 24)}
    if kind == "place":
        return {"kind": kind, "cells": _log_int(rng, 2_000, 100_000), "iters": rng.randint(16, 64)}
    if kind == "ip":
        return {"kind": kind, "cells": _log_int(rng, 2_000, 400_000)}
    jobs = rng.randint(4, 16)
    case = {"kind": kind, "jobs": jobs, "cells_lo": 2_000, "cells_hi": _log_int(rng, 10_000, 50_000)}
    if kind == "batch_loop":
        case["iters"] = rng.randint(8, 24)
    return case


# ------------------------------------------------------------------ inputs
def _curve(n, order=12):
    """n points along a Hilbert curve over the unit square: neighbours in
    index order, which the generator's nets join, are neighbours in space."""
    t = np.arange(n, dtype=np.int64) * (4 ** order) // n
    x = np.zeros(n, np.int64)
    y = np.zeros(n, np.int64)
    s = 1
    while s < 2 ** order:
        rx = 1 & (t // 2)
        ry = 1 & (t ^ rx)
        flip = (ry == 0) & (rx == 1)
        fx, fy = np.where(flip, s - 1 - x, x), np.where(flip, s - 1 - y, y)
        x, y = np.where(ry == 0, fy, fx) + s * rx, np.where(ry == 0, fx, fy) + s * ry
        t //= 4
        s *= 2
    return (x + 0.5) / 2 ** order, (y + 0.5) / 2 ** order


def _spread_centres(nl, rng, jitter=0.005):
    """Cell centres of a placement that is spread over the core: the curve
    with a seeded displacement of a few bins."""
    lx, ly, ux, uy = nl.core
    n = nl.n_insts
    w, h = nl.inst_ux - nl.inst_lx, nl.inst_uy - nl.inst_ly
    fx, fy = _curve(n)
    x = lx + fx * (ux - lx) + rng.normal(0, jitter * (ux - lx), n)
    y = ly + fy * (uy - ly) + rng.normal(0, jitter * (uy - ly), n)
    return np.clip(x, lx + w / 2, ux - w / 2), np.clip(y, ly + h / 2, uy - h / 2)


@functools.lru_cache(maxsize=64)
def _library(cells, macros, util):
    """The instances' sizes and the core of a design: the same for every seed,
    so that all of a case's inputs have the same gcells."""
    return N.generate(cells, 1, n_io=200, n_macros=macros, util=util, seed=cells)


def _design(cells, macros, util, seed):
    """A generated netlist of this seed's nets and pins over the case's
    instances."""
    lib = _library(cells, macros, util)
    nl = N.generate(cells, int(round(1.05 * cells)), n_io=200, n_macros=macros, util=util, seed=int(seed))
    rng = np.random.default_rng(seed + 1)
    on = nl.pin_inst >= 0
    i = nl.pin_inst[on]
    for off, lo, hi in ((nl.pin_ox, lib.inst_lx, lib.inst_ux), (nl.pin_oy, lib.inst_ly, lib.inst_uy)):
        off[on] = np.floor((rng.random(len(i)) - 0.5) * (hi - lo)[i]).astype(np.int32)
    for pos, k in ((nl.pin_x, 2), (nl.pin_y, 3)):
        pos[~on] = (pos[~on].astype(np.int64) * lib.core[k] // nl.core[k]).astype(np.int32)
    nl.core, nl.die, nl.rows = lib.core, lib.die, lib.rows
    nl.inst_lx, nl.inst_ly = lib.inst_lx.copy(), lib.inst_ly.copy()
    nl.inst_ux, nl.inst_uy = lib.inst_ux.copy(), lib.inst_uy.copy()
    nl._update_pins()
    return nl


def _netlist(case, seed):
    return _design(case["cells"], case.get("macros", 0), 0.60, seed)


def _weights(nl, seed):
    return np.random.default_rng(seed + 7).lognormal(0.0, 0.5, nl.n_nets).astype(np.float32)


# a loop that holds its penalty and does not stop (see above)
_HELD = dict(max_phi_coef=1.0, min_phi_coef=1.0, target_overflow=0.0, nesterov_place_max_iter=60_000, poisson_path=1)


def _batch(case, seed):
    sizes = np.random.default_rng(case["jobs"])
    out = []
    for k in range(case["jobs"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["cells_lo"]), math.log(case["cells_hi"])))))
        td = float(sizes.uniform(0.60, 0.85))
        out.append((_design(n, 0, min(0.60, td - 0.02), int(seed) * 131 + k), td))
    return out


def _eval_inputs(case, seed):
    nl = _netlist(case, seed)
    rng = np.random.default_rng(seed + 3)
    x, y = _spread_centres(nl, rng)
    return nl, rng, x, y


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        nx, ny = case["nx"], case["ny"]
        d = _density(case, seed)
        out = [torch.empty((ny, nx), dtype=torch.float32, device="cuda") for _ in range(3)]
        return {"case": case, "density": d, "phi": out[0] if case["phi"] else None, "fx": out[1], "fy": out[2]}
    if kind == "eval":
        nl, rng, x, y = _eval_inputs(case, seed)
        p = Placer(nl, target_density=0.70, bin_grid_cnt_x=case["bins"], bin_grid_cnt_y=case["bins"],
                   initial_place_max_iter=0, poisson_path=1)
        if case["weights"]:
            p.set_net_weights(_weights(nl, seed))
        p.initial_place()
        p.nesterov_init()
        lx, ly, ux, uy = nl.core
        fill = p.info.n_gcells - nl.n_insts
        xy = np.empty((p.info.n_gcells, 2), np.float32)
        xy[:nl.n_insts, 0], xy[:nl.n_insts, 1] = x, y
        xy[nl.n_insts:, 0] = rng.uniform(lx + 6_000, ux - 6_000, fill)
        xy[nl.n_insts:, 1] = rng.uniform(ly + 6_000, uy - 6_000, fill)
        return {"case": case, "placer": p, "xy": xy, "cells": nl.n_insts, "coef": _EVAL_COEF}
    if kind == "loop":
        nl = _netlist(case, seed)
        kw = dict(_HELD, target_density=0.75, bin_grid_cnt_x=case["bins"], bin_grid_cnt_y=case["bins"])
        if case["spread"]:
            x, y = _spread_centres(nl, np.random.default_rng(seed + 3))
            w, h = nl.inst_ux - nl.inst_lx, nl.inst_uy - nl.inst_ly
            nl.set_inst_locations(np.arange(nl.n_insts), (x - w / 2).astype(np.int32), (y - h / 2).astype(np.int32))
            p = Placer(nl, incremental_place_mode=1, initial_place_max_iter=0, init_density_penalty=0.003, **kw)
        else:
            p = Placer(nl, init_density_penalty=0.1, **kw)
        if case["weights"]:
            p.set_net_weights(_weights(nl, seed))
        p.initial_place()
        p.nesterov_init()
        return {"case": case, "placer": p}
    if kind == "place":
        return {"case": case, "netlist": _netlist(case, seed)}
    if kind == "ip":
        return {"case": case, "placer": Placer(_netlist(case, seed), target_density=0.70)}
    if kind == "batch_ip":
        return {"case": case, "placers": [Placer(nl, target_density=td) for nl, td in _batch(case, seed)]}
    ps = [Placer(nl, target_density=td, init_density_penalty=0.1, **_HELD) for nl, td in _batch(case, seed)]
    batch_initial_place(ps)
    for p in ps:
        p.nesterov_init()
    return {"case": case, "placers": ps}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "poisson":
        phi = state["phi"]
        poisson_solve(state["density"].data_ptr(), 0 if phi is None else phi.data_ptr(), state["fx"].data_ptr(),
                      state["fy"].data_ptr(), case["nx"], case["ny"], case["bin_x"], case["bin_y"],
                      stream=torch.cuda.current_stream().cuda_stream)
        out = {"fx": state["fx"], "fy": state["fy"]}
        if phi is not None:
            out["phi"] = phi
        return out
    if kind == "eval":
        wl, dg, st = state["placer"].eval(state["xy"], state["coef"])
        n = state["cells"]
        return {"wl_cells": wl[:n], "wl_fillers": wl[n:], "dg": dg, "hpwl": int(st.hpwl),
                "overflow": float(st.overflow_area_f64), "sum_phi": float(st.sum_phi),
                "wl_sum": float(st.wire_length_grad_sum), "dg_sum": float(st.density_grad_sum)}
    if kind == "loop":
        p = state["placer"]
        _, st, _ = p.nesterov_run(case["iters"])
        return {"xy": p.gcell_coords(), "overflow": float(st.overflow)}
    if kind == "place":
        p = Placer(state["netlist"], target_density=0.70, poisson_path=1)
        p.initial_place()
        p.nesterov_init()
        _, st, _ = p.nesterov_run(case["iters"])
        out = {"xy": p.gcell_coords(), "overflow": float(st.overflow)}
        p.close()
        return out
    if kind == "ip":
        state["placer"].initial_place()
        return state["placer"].inst_locations()
    if kind == "batch_ip":
        batch_initial_place(state["placers"])
        return [np.stack(p.inst_locations()) for p in state["placers"]]
    batch_nesterov_run(state["placers"], case["iters"])
    return [p.gcell_coords() for p in state["placers"]]


# -------------------------------------------------------------------- work
def _sizes(cells):
    """(gcells, pins, nets, entries of both B2B matrices) of a generated
    netlist: fillers add about a quarter, nets average 4.6 pins."""
    return 1.25 * cells, 4.8 * cells, 1.05 * cells, 2 * 12.4 * cells


def _eval_work(cells, bins, weights=False):
    g, p, n, _ = _sizes(cells)
    # per gcell: coordinates and gradients in and out (48 bytes), size, scale,
    # kind and preconditioner (21); per pin its cell and offset; per net its
    # start; per bin the fixed area
    b = 69 * g + 12 * p + (8 if weights else 4) * n + 8 * bins
    # four exponentials of 22 operations and about 40 more per pin; six bins
    # of about 20 operations per gcell; a forward and three inverse transforms
    f = 128 * p + 2 * 120 * g + 4 * 2.5 * bins * math.log2(bins)
    return b, f


def _ip_work(cells):
    g, p, n, e = _sizes(cells)
    # the netlist once and the locations out; per round the matrices out and
    # in once (the solver's iterations can hold them on the chip)
    b = 16 * p + 8 * n + 16 * cells + 20 * (2 * 6 * e)
    f = 20 * (100 * (2 * 2 * e + 2 * 24 * cells) + 10 * e)
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "poisson":
        n = case["nx"] * case["ny"]
        outs = 3 if case["phi"] else 2
        return {"bytes": 4.0 * n * (1 + outs), "flops": (1 + outs) * 2.5 * n * math.log2(n)}
    if kind == "eval":
        b, f = _eval_work(case["cells"], case["bins"] ** 2, case["weights"])
    elif kind == "loop":
        b, f = (case["iters"] * v for v in _eval_work(case["cells"], case["bins"] ** 2, case["weights"]))
    elif kind == "place":
        i, e = _ip_work(case["cells"]), _eval_work(case["cells"], 2.0 * case["cells"])
        b, f = (u + case["iters"] * v for u, v in zip(i, e))
    elif kind == "ip":
        b, f = _ip_work(case["cells"])
    else:
        # cell counts are log-uniform
        lo, hi = case["cells_lo"], case["cells_hi"]
        cells = case["jobs"] * (hi - lo) / math.log(hi / lo)
        if kind == "batch_ip":
            b, f = _ip_work(cells)
        else:
            b, f = (case["iters"] * v for v in _eval_work(cells, 2.0 * cells))
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------- exact
_EVAL_COEF = 2e-4


def _density(case, seed):
    """A density as a placement has it: near the target on the whole, denser
    in places, noisy from bin to bin."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    nx, ny = case["nx"], case["ny"]
    coarse = torch.rand((1, 1, 9, 9), generator=g, device="cuda")
    smooth = torch.nn.functional.interpolate(coarse, size=(ny, nx), mode="bilinear", align_corners=True)[0, 0]
    noise = torch.rand((ny, nx), generator=g, device="cuda")
    return (0.5 + smooth + 0.3 * noise).to(torch.float32).contiguous()


def _cos_sum(a, sine):
    """Along the last axis of length n: sum_k a[k] cos(pi k (m + 1/2) / n), or
    with sine the same sum of sines, for every m, in float64."""
    n = a.shape[-1]
    k = torch.arange(n, dtype=torch.float64, device=a.device)
    z = torch.zeros(a.shape[:-1] + (2 * n,), dtype=torch.complex128, device=a.device)
    z[..., :n] = a * torch.exp(1j * math.pi * k / (2 * n))
    r = torch.fft.ifft(z, dim=-1)[..., :n] * (2 * n)
    return r.imag if sine else r.real


def _dct2(x):
    """sum_m x[m] cos(pi k (m + 1/2) / n) along the last axis, float64."""
    n = x.shape[-1]
    k = torch.arange(n, dtype=torch.float64, device=x.device)
    z = torch.zeros(x.shape[:-1] + (2 * n,), dtype=torch.complex128, device=x.device)
    z[..., :n] = x
    return (torch.fft.fft(z, dim=-1)[..., :n] * torch.exp(-1j * math.pi * k / (2 * n))).real


def _exact_poisson(case, seed):
    nx, ny = case["nx"], case["ny"]
    sx, sy = case["bin_x"], case["bin_y"]
    d = _density(case, seed).double()
    # rho^ with the constant term dropped; the y frequencies are scaled by the
    # bins' aspect ratio
    c = _dct2(_dct2(d).transpose(0, 1)).transpose(0, 1) * (4.0 / (nx * ny))
    c[0, :] *= 0.5
    c[:, 0] *= 0.5
    wx = math.pi * torch.arange(nx, dtype=torch.float64, device=d.device) / nx
    wy = math.pi * torch.arange(ny, dtype=torch.float64, device=d.device) / ny * (sy / sx)
    w2 = wx[None, :] ** 2 + wy[:, None] ** 2
    w2[0, 0] = 1.0
    ph = c / w2
    ph[0, 0] = 0.0

    def inverse(a, sin_x, sin_y):
        return _cos_sum(_cos_sum(a, sin_x).transpose(0, 1), sin_y).transpose(0, 1).contiguous()

    out = {"fx": inverse(ph * wx[None, :], True, False), "fy": inverse(ph * wy[:, None], False, True)}
    if case["phi"]:
        out["phi"] = inverse(ph, False, False)
    return out


def _exact_wl(case, seed):
    """The weighted-average wirelength gradient of every gcell (fillers have
    none), with the library's exponential (1 + a / 1024)^1024."""
    nl, _, x, y = _eval_inputs(case, seed)
    cx = x.astype(np.float32).astype(np.int64)
    cy = y.astype(np.float32).astype(np.int64)
    net = np.repeat(np.arange(nl.n_nets), np.diff(nl.net_start))
    first = nl.net_start[:-1]
    on = nl.pin_inst >= 0
    w = _weights(nl, seed).astype(np.float64) if case["weights"] else np.ones(nl.n_nets)
    grad = np.zeros((nl.n_insts, 2))
    coef = float(np.float32(_EVAL_COEF))
    for axis, (c, off, fixed) in enumerate(((cx, nl.pin_ox, nl.pin_x), (cy, nl.pin_oy, nl.pin_y))):
        pos = np.where(on, c[np.maximum(nl.pin_inst, 0)] + off, fixed).astype(np.int64)
        lo, hi = np.minimum.reduceat(pos, first), np.maximum.reduceat(pos, first)
        g = np.zeros(len(pos))
        for a, sign in (((lo[net] - pos) * coef, 1.0), ((pos - hi[net]) * coef, -1.0)):
            e = np.where(a > -300.0, np.power(1.0 + a / 1024.0, 1024.0), 0.0)
            # positions from the net's centre: the same gradient, no cancellation
            q = pos - 0.5 * (lo + hi)[net]
            s0, s1 = np.add.reduceat(e, first)[net], np.add.reduceat(q * e, first)[net]
            g += sign * e / s0 * (1.0 - sign * coef * (q - s1 / s0))
        grad[:, axis] = np.bincount(nl.pin_inst[on], weights=(g * w[net])[on], minlength=nl.n_insts)
    return grad


def exact(case, seed):
    if case["kind"] == "poisson":
        return _exact_poisson(case, seed)
    if case["kind"] == "eval":
        return {"wl_cells": _exact_wl(case, seed)}
    return None
