"""Every way in which the initial place sums a matrix row, on netlists wired so
that it occurs (the counts that verbose_level 2 prints show that it does):
locations, rounds and solver iterations equal the ones recorded from the form
that reads every row from the CSR arrays.
"""

import hashlib
import re

import numpy as np
import pytest

from replace_gb300 import netlist as N

pytestmark = pytest.mark.gpu


def wired(n, nets):
    """A generated design of n cells whose nets are replaced; a net is a list
    of cells, with one IO pin where it holds -1."""
    nl = N.generate(n, 10, n_io=10, seed=n)
    rng = np.random.default_rng(n)
    flat = np.concatenate(nets).astype(np.int32)
    nl.net_start = np.concatenate([[0], np.cumsum([len(k) for k in nets])]).astype(np.int32)
    nl.pin_inst = flat
    on = flat >= 0
    nl.pin_ox, nl.pin_oy = (np.where(on, rng.integers(-150, 150, len(flat)), 0).astype(np.int32) for _ in range(2))
    nl.pin_x = np.where(on, 0, rng.integers(nl.core[0], nl.core[2], len(flat))).astype(np.int32)
    nl.pin_y = np.where(on, 0, rng.integers(nl.core[1], nl.core[3], len(flat))).astype(np.int32)
    nl.io_box = None
    order = np.nonzero(on)[0][np.argsort(flat[on], kind="stable")]
    nl.inst_pins = order.astype(np.int32)
    counts = np.bincount(flat[on], minlength=nl.n_insts)
    nl.inst_pin_start = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    nl._update_pins()
    return nl


def chain(n, every=0):
    """Cells in a row, with an IO pin at both ends and on every `every`-th net."""
    nets = [[-1, 0]] + [[k, k + 1] for k in range(n - 1)] + [[n - 1, -1]]
    if every:
        nets += [[k, -1] for k in range(0, n, every)]
    return nets


def far_half(n):
    """The upper half of a chain also wired at random within that half."""
    rng = np.random.default_rng(n)
    return chain(n, 50) + [[int(k), int(n // 2 + rng.integers(n // 2))] for k in range(n // 2, n)]


def stars(n, degree, step):
    """A chain, and nets of `degree` neighbouring cells every `step` cells."""
    return chain(n, 100) + [list(range(k, k + degree)) for k in range(0, n - degree, step)]


# netlist, the forms that have to occur, sha256 of the locations after three
# rounds of 100 solver iterations
CASES = {
    # (padded to four entries a row, a chain needs more room than its share)
    "no room": (lambda: wired(4000, chain(4000, 40)), {"sliced", "in CSR form"},
        "aca7525e32a82ffc54d94da12199bb38e626cbbcca74e308f37c527802293be2"),
    "wide windows": (lambda: wired(16000, far_half(16000)), {"sliced", "in CSR form"},
        "e8c2fffe9f1f75833727d930096d40d1768c725f1475860c4e50a9eb983e5430"),
    "staged": (lambda: wired(3000, stars(3000, 40, 25)), {"sliced", "staged"},
        "ee46fdd79665ae68feeee0d2936e4ee83e9cbf981168b288c9669147d7a8d9ae"),
    "long among many": (lambda: wired(3000, stars(3000, 90, 3)), {"sliced", "staged", "long ones among many"},
        "4fcb6c4a78f13867016d186820667623eb3b1d49afcab52bc64aba74c30ad3d2"),
    "longer than the stage": (lambda: wired(3000, stars(3000, 190, 38)), {"longer than the stage"},
        "12638e988b49b242af240acfd1e9c2b8114e0e90fb5adb4431e817b2c69c8cfb"),
}


@pytest.mark.parametrize("case", CASES)
def test_row_forms_equal_csr_form(gpu_lib, case, capfd):
    from replace_gb300 import Placer
    build, forms, want = CASES[case]
    p = Placer(build(), target_density=0.7, initial_place_max_iter=3, verbose_level=2)
    st = p.initial_place()
    lx, ly = p.inst_locations()
    p.close()
    lines = re.findall(r"rows of [xy]: (.*)", capfd.readouterr().out)
    assert len(lines) == 2
    for line in lines:
        rows = {form.strip(): int(k) for k, form in re.findall(r"(\d+) ([a-zA-Z ]+)", line.split("(")[0])}
        assert all(rows[f] > 0 for f in forms), (forms, rows)
    assert (st.iterations, st.solver_iters_x, st.solver_iters_y) == (3, 100, 100)
    assert hashlib.sha256(lx.tobytes() + ly.tobytes()).hexdigest() == want
