"""GPU: partitions that provably cannot become a stable candidate (an all-gas or
all-liquid state of a cell inside the dome) are not solved: every bit of states and
flags equals the exhaustive search's."""
import numpy as np
import pytest

from spuma_multiphysics_b200 import _abi as A, cases
from spuma_multiphysics_b200.eos import PureFluid
from spuma_multiphysics_b200.thermo_data import N2O
from test_two_phase_bound_gpu import assert_same, both

pytestmark = pytest.mark.gpu


def seeded(rho, T, p=4e6):
    guess = np.zeros(len(rho), dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = p, T, rho
    return guess


def tie_line_states(T, beta):
    """Two-phase states at temperature T and liquid mass fraction beta: (rho, e, guess)."""
    ps, gas, liq = PureFluid(N2O).saturation(T)
    rho = 1 / ((1 - beta) / gas["rho"] + beta / liq["rho"])
    e = rho * ((1 - beta) * gas["e"] + beta * liq["e"])
    guess = seeded(rho, T, ps)
    guess["liquidMass"][:, 0] = beta * rho
    guess["activeLiquids"] = 1
    return rho, e, guess


def mesh_states(part):
    rng = np.random.default_rng(31)
    if part == "fixed seeds":
        return cases.flash_batch(3000, seed=61, seed_policy="fixed")
    if part == "compressed liquid":
        T, p = rng.uniform(185.0, 305.0, 1500), np.exp(rng.uniform(np.log(6e6), np.log(4e7), 1500))
        s = PureFluid(N2O).tp(T, p, root="liquid")
        ok = np.isfinite(s["rho"]) & (s["rho"] > 0)
        rho, e = s["rho"][ok], (s["rho"] * s["e"])[ok]
        return rho, e, seeded(rho, 250.0)
    if part == "all densities":     # the whole (rho, e) box around and inside the dome
        rho = np.exp(rng.uniform(np.log(2.0), np.log(1200.0), 3000))
        u = rng.uniform(-4.2e5, 2e5, 3000)
        return rho, rho * u, seeded(rho, rng.uniform(160.0, 320.0, 3000))
    T = {"near critical": (308.5, 309.45), "cold end": (148.0, 160.0)}[part]
    return tie_line_states(rng.uniform(*T, 1500), rng.uniform(0.0, 1.0, 1500))


@pytest.mark.parametrize("part", ["fixed seeds", "compressed liquid", "all densities", "near critical", "cold end"])
def test_skipped_partitions_change_no_bit(part):
    rho, e, guess = mesh_states(part)
    rho, e = np.ascontiguousarray(rho), np.ascontiguousarray(e)
    on, off = both(rho, e, guess)
    assert_same(on, off)
