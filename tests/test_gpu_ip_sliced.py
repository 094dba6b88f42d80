"""The initial place's sliced matrix form gives the sums of the CSR form bit
for bit: locations, rounds and solver iterations of netlists whose rows reach
each of its branches equal the ones recorded from the CSR form (one lane sums
a row's products in entry order; rows over 32 entries in a window of 32 rows
with more than 1024 take the warp-wide order).

Cases: a single SpMV block and a partial last slice (40), blocks that are not
256 rows (700), several rows per thread (70,000), rows longer than every slice
(nets joined to degree about 100: special and warp-wide rows), and macros with
hundreds of pins.
"""

import hashlib

import numpy as np
import pytest

from replace_gb300 import netlist as N

pytestmark = pytest.mark.gpu

# (cells, nets joined per net, macros) -> (rounds, iterations x, y, sha256 of the locations)
RECORDED = {
    (40, 1, 0): (3, 30, 30,
        "c236087d9d15f63db94526e76eee8f9b532aa95aff3d2818309b7b27a80b18d7"),
    (257, 1, 0): (3, 76, 69,
        "6489dc0595144a158441ce36ba30afaed76ded61e0a286c5105813e18700e0e0"),
    (700, 1, 0): (3, 99, 81,
        "5d1a9bf5e01964cee12277397af21209be30496622566a5cfeafc23bcdcce8ac"),
    (10000, 1, 0): (3, 100, 100,
        "4261e1cf015bd6556e2c0b4c3d48cc0411dba6f8a2bdb563c1cd6de8e4ffe3b1"),
    (70000, 1, 0): (3, 100, 100,
        "4e28fe482b3057e60f4cc9ba3faead168cad42043065b73eb6936318d6f38516"),
    (5000, 20, 0): (3, 100, 100,
        "994edca1f89ba455384fadf2233809ef2fe084399706c167e26bd6f3042ca633"),
    (40000, 30, 0): (3, 100, 100,
        "9fd361cbb0ffe0074a6ec3fc94c824574fa64417d32776d657f3003c385dbce6"),
    (20000, 1, 12): (3, 100, 100,
        "74c8220e3fee72fc1734097bb7adb3a7ab60e5aaa53675ebff42d8c6a7dd917f"),
    (100000, 20, 5): (3, 100, 100,
        "4f9c3e5c819ba93aeb2cd0a659412d8544ef2046ffec87903277c117d2c7afd9"),
}


def build(cells, join, macros):
    nl = N.generate(cells, int(round(1.05 * cells)) + 7, n_io=50, n_macros=macros, seed=cells + join + macros,
                    macro_rows=(6, 9))
    if join > 1:
        keep = np.arange(0, nl.n_nets, join)
        nl.net_start = np.concatenate([nl.net_start[keep], nl.net_start[-1:]]).astype(np.int32)
    if macros:
        # every 50th pin of a cell moves to a macro
        mac = np.nonzero(nl.inst_uy - nl.inst_ly > N.ROW_H)[0]
        on = np.nonzero(nl.pin_inst >= 0)[0][::50]
        nl.pin_inst[on] = mac[np.arange(len(on)) % len(mac)].astype(np.int32)
        nl.pin_ox[on] = nl.pin_oy[on] = 0
        m = nl.pin_inst >= 0
        pins = np.nonzero(m)[0]
        order = pins[np.argsort(nl.pin_inst[pins], kind="stable")]
        counts = np.bincount(nl.pin_inst[order], minlength=nl.n_insts)
        nl.inst_pin_start = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
        nl.inst_pins = order.astype(np.int32)
        nl._update_pins()
    return nl


def outcome(cells, join, macros):
    from replace_gb300 import Placer
    nl = build(cells, join, macros)
    p = Placer(nl, target_density=0.7, initial_place_max_iter=3)
    st = p.initial_place()
    lx, ly = p.inst_locations()
    p.close()
    return st.iterations, st.solver_iters_x, st.solver_iters_y, hashlib.sha256(lx.tobytes() + ly.tobytes()).hexdigest()


@pytest.mark.parametrize("case", RECORDED)
def test_sliced_form_equals_csr_form(gpu_lib, case):
    assert outcome(*case) == RECORDED[case]
