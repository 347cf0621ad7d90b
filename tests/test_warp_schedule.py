"""The warp schedule on the golden fixtures, bit for bit: its float operations, their fused
multiply-adds and its partial sums, which depend on which targets share a warp
(in correction passes too), are fixed, and the lane schedule's changes must
not reach them."""
import hashlib

import numpy as np
import pytest

from helpers import FIRST_PASS_CASES, load_case

POTENTIALS = {  # walk_leaf_runs 0 and 1
    "first_pass_corner_2200": ("f6d7bbe8155aba1b", "3dec2d85c931ef33"),
    "first_pass_nfw_3300": ("01af9c237da29b24", "0797059435afa6d8"),
}

UNBOUND = {
    "nfw_2200_bulk": "69690340c505301d",
    "nfw_3300_corner": "d0159d6b2348b49f",
    "nfw_4400_sampled": "c3cbac14304308f0",
    "nfw_1650_theta07": "653734e3f859589f",
    "batch_48": "bca4454bacd6790b",
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


@pytest.mark.gpu
@pytest.mark.parametrize("case", UNBOUND)
def test_unbinding(case):
    from hbtplus_gb300.unbind import Unbinder
    par, inp, _ = load_case(case)
    with Unbinder(par) as ub:
        ub.set_option("walk_schedule", 1)
        order, energy, _ = (ub.unbind_batch if "offsets" in inp else ub.unbind)(inp)
    energy[np.isnan(energy)] = np.nan
    assert hashlib.sha1(order.tobytes() + energy.tobytes()).hexdigest()[:16] == UNBOUND[case]
