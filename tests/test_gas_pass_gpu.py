"""GPU: the first pass of the pure-fluid search (passGas), which decides the plainly
gaseous cells in registers. Its results must be the work queue's: every bit of
the states, transport states and flags equals the search with the two-phase bound
off (where the queue solves every cell), and p, T equal the oracle flash's."""
import numpy as np
import pytest

from oracle import oracle
from spuma_multiphysics_b200 import _abi as A, cases, thermo_data as td
from spuma_multiphysics_b200.eos import PureFluid
from spuma_multiphysics_b200.thermo_data import N2O, N2O_FLASH
import flash_cases as F
from test_two_phase_bound_gpu import assert_same, both

pytestmark = pytest.mark.gpu


def gas_states(n, shift, seed=5):
    """Single-phase gas states over the bound's outside (T 150-1500 K, up to 60 bar),
    each seeded `shift` (relative) off its own temperature."""
    rng = np.random.default_rng(seed)
    T = np.exp(rng.uniform(np.log(150.0), np.log(1500.0), n))
    p = np.exp(rng.uniform(np.log(2e3), np.log(6e6), n))
    props = PureFluid(N2O).tp(T, p, root="gas")
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = p, T * (1 + shift), props["rho"]
    return np.ascontiguousarray(props["rho"]), np.ascontiguousarray(props["rho"] * props["e"]), guess


# 0 and 1e-12: accepted at the seed; 1e-4, 4e-3: a Newton inside half the bracket's
# radius (1% of T); 6e-3 and more, either way: past it, so the general pass
@pytest.mark.parametrize("shift", [0.0, 1e-12, 1e-4, -1e-4, 4e-3, -4e-3, 6e-3, 2e-2, -2e-2, .3])
def test_gas_cells_equal_the_queue_bitwise_and_the_oracle(shift):
    rho, e, guess = gas_states(4000, shift)
    on, off = both(rho, e, guess)
    assert_same(on, off)
    got = np.frombuffer(on[0], dtype=A.THERMO_DTYPE)
    pick = slice(0, 400)
    ref, ref_ok, _ = F.oracle_flash(oracle, td.model_bytes(td.pure_model()), rho[pick], e[pick], guess[pick])
    s = F.compare(got[pick], on[2][pick], ref, ref_ok)
    assert s["success_equal"] and s["label_mismatch"] == 0, s
    # both stop at an energy residual of 1e-9 of max(1e5 rho, rho cp T), which cp/cv < 1.5
    # here and the pressure's T-slope turn into less than 1e-8 of p and T
    assert s["p_rel"] <= 1e-8 and s["T_rel"] <= 1e-8, s


# about the liquid range's end, above which no liquid is evaluated, and up to past the
# critical pressure there
@pytest.mark.parametrize("shift", [0.0, 4e-3, -4e-3])
def test_cells_at_the_end_of_the_liquid_range(shift):
    n, rng = 3000, np.random.default_rng(9)
    end = N2O_FLASH["liquidTc"] * (1 - 1e-10)
    step = np.resize([0.0, 1e-15, -1e-15, 1e-12, -1e-12, 1e-9, -1e-9, 1e-6, -1e-6, 1e-3, -1e-3, .1], n)
    T, p = end * (1 + step), np.exp(rng.uniform(np.log(1e5), np.log(1.2e7), n))
    props = PureFluid(N2O).tp(T, p, root="gas")
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = p, T * (1 + shift), props["rho"]
    on, off = both(np.ascontiguousarray(props["rho"]), np.ascontiguousarray(props["rho"] * props["e"]), guess)
    assert_same(on, off)
    assert on[2].mean() > .9


# one thread, a warp's edges, a block's edges, and a mix of gas, dome and liquid
# cells inside one warp (the staged write must leave the others' records alone)
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 1000])
def test_partial_warps_and_mixed_cells(n):
    rho, e, guess = cases.flash_batch(max(n, 8), seed=100 + n, two_phase_share=.4)
    on, off = both(rho[:n], e[:n], np.ascontiguousarray(guess[:n]))
    assert_same(on, off)
