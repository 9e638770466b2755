"""GPU: the pure-fluid search's passes that leave work out or rewrite it.

* Partitions that provably cannot converge (an all-gas or all-liquid state of a
  cell inside the dome) are not solved: every bit of states and flags equals the
  exhaustive search's.
* The two-phase candidates in registers (analytic Jacobian) against the general
  evaluation of the one-thread-per-cell form and against the oracle flash.
"""
import numpy as np
import pytest
import torch

from oracle import oracle
from spuma_multiphysics_b200 import _abi as A, cases, thermo_data as td
from spuma_multiphysics_b200.eos import PureFluid
from spuma_multiphysics_b200.hem import GpuHem
from spuma_multiphysics_b200.thermo_data import N2O
import flash_cases as F
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
        u = rng.uniform(1.3e6, 2.2e6, 3000)  # N2O's saturated liquid at 148 K has 1.34e6, its gas at 700 K 2.1e6
        return rho, rho * u, seeded(rho, rng.uniform(160.0, 320.0, 3000))
    T = {"near critical": (308.5, 309.45), "cold end": (148.0, 160.0)}[part]
    return tie_line_states(rng.uniform(*T, 1500), rng.uniform(0.0, 1.0, 1500))


@pytest.mark.parametrize("part", ["fixed seeds", "compressed liquid", "all densities", "near critical", "cold end"])
def test_skipped_partitions_change_no_bit(part):
    rho, e, guess = mesh_states(part)
    rho, e = np.ascontiguousarray(rho), np.ascontiguousarray(e)
    on, off = both(rho, e, guess)
    assert_same(on, off)
    assert on[2].mean() > .1  # states that have an answer


# one cell, a warp's and a block's edges; liquid fractions from both ends of the tie line
@pytest.mark.parametrize("n", [1, 31, 33, 129, 3000])
@pytest.mark.parametrize("beta", [(0.0, 1.0), (1e-7, 1e-4), (1 - 1e-4, 1 - 1e-7)])
def test_two_phase_candidates_equal_the_general_evaluation(n, beta):
    rng = np.random.default_rng(7 * n + 1)
    rho, e, guess = tie_line_states(rng.uniform(185.0, 306.0, n), rng.uniform(*beta, n))
    guess["T"] += rng.uniform(-3.0, 3.0, n)
    guess["p"] *= rng.uniform(.9, 1.1, n)
    hem = GpuHem(capacity=n)
    try:
        cons = torch.zeros((5, n), dtype=torch.float64, device="cuda")
        cons[0], cons[4] = torch.from_numpy(rho).cuda(), torch.from_numpy(e).cuda()
        seed = torch.from_numpy(guess.view(np.uint8).copy()).cuda()
        out = []
        for per_cell in (False, True):
            state, ok = torch.zeros_like(seed), torch.zeros(n, dtype=torch.int32, device="cuda")
            hem.run_device(cons, n, n, 5, seed, state, None, ok, torch.cuda.current_stream().cuda_stream, per_cell)
            torch.cuda.synchronize()
            out.append((state.cpu().numpy().view(A.THERMO_DTYPE), ok.cpu().numpy()))
    finally:
        hem.close()
    (got, ok), (general, general_ok) = out
    ref, ref_ok, _ = F.oracle_flash(oracle, td.model_bytes(td.pure_model()), rho, e, guess)
    for other, other_ok in ((general, general_ok), (ref, ref_ok)):
        s = F.compare(got, ok, other, other_ok)
        assert s["success_equal"] and s["label_mismatch"] == 0, s
        # both stop at residuals below 1e-9: in the energy, of at most 2000 T per mass, which
        # over cv > 1500 is 1.4e-9 of T each, and by Clausius-Clapeyron (h_fg W / RT < 13 from
        # 185 K) 13 times that of p
        assert s["p_rel"] <= 4e-8 and s["T_rel"] <= 3e-9 and s["ml_rel"] <= F.STATE_TOL, s
