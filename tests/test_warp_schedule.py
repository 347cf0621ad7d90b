"""The warp schedule's first-pass potentials on the golden fixtures, bit for bit: its float
operations, their fused multiply-adds and the order of its partial sums are
fixed, and the lane schedule's changes must not reach them."""
import hashlib

import pytest

from helpers import FIRST_PASS_CASES, load_case

POTENTIALS = {  # walk_leaf_runs 0 and 1
    "first_pass_corner_2200": ("f6d7bbe8155aba1b", "3dec2d85c931ef33"),
    "first_pass_nfw_3300": ("01af9c237da29b24", "0797059435afa6d8"),
}


@pytest.mark.gpu
@pytest.mark.parametrize("leaf_runs", [0, 1])
@pytest.mark.parametrize("case", FIRST_PASS_CASES)
def test_potentials(case, leaf_runs):
    from hbtplus_gb300.unbind import Unbinder
    par, inp, _ = load_case(case)
    with Unbinder(par) as ub:
        ub.set_option("walk_schedule", 1)
        ub.set_option("walk_leaf_runs", leaf_runs)
        _, pot = ub.binding_energies(inp["pos"], inp["vel"], inp["mass"], inp["ref_pos"],
                                     inp["ref_vel"])
    assert hashlib.sha1(pot.tobytes()).hexdigest()[:16] == POTENTIALS[case][leaf_runs]
