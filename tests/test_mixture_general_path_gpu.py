"""GPU: the multi-species flash where its two-phase residual is not formed alone: a
liquid whose table is not the gas species' own, and points that the residual formed
alone leaves to the general evaluation. A stored candidate must be the converged
point itself, not one of the Jacobian's side points beside it: the reference's
captured results, the oracle flash and the residuals of the stored states."""

import numpy as np
import pytest

from oracle import oracle
from spuma_multiphysics_b200 import _abi as A, thermo_data as td
from spuma_multiphysics_b200.eos import PureFluid
from spuma_multiphysics_b200.hem import GpuHem
import flash_cases as F
from test_mixture_flash_gpu import GOLDEN, check, gpu_flash
from test_mixture_residual import residuals, shim  # noqa: F401 (fixture)
from test_two_phase_pass_gpu import tie_line_states

pytestmark = pytest.mark.gpu
# a liquid table of its own: chemical potentials move by this times kappa's terms (< 100),
# far below the affinity tolerance of 1e-7 and the comparisons' 1e-9
OWN = 1 + 1e-13


def test_own_liquid_tables_match_the_captured_results():
    d = np.load(GOLDEN)
    model = td.two_liquid_model()
    for i in (1, 2):
        model.phase[i].species[0].kappa *= OWN
    got, ok, _ = gpu_flash(td.model_bytes(model), d["q"], d["energy"], d["guess"].view(A.THERMO_DTYPE))
    check(got, ok, d["out"].view(A.THERMO_DTYPE), d["success"], min_success=1.0)


# both searches of an equilibrium batch without a jump: liquid fractions, and (nearly
# all liquid) log vapour fractions
@pytest.mark.parametrize("beta", [(.05, .95), (1 - 5e-5, 1 - 1e-6)])
def test_own_liquid_table_of_a_pure_fluid_matches_the_oracle(beta):
    n = 200
    rng = np.random.default_rng(11)
    rho, e, guess = tie_line_states(rng.uniform(190.0, 300.0, n), rng.uniform(*beta, n))
    guess["T"] += rng.uniform(-2.0, 2.0, n)
    model = td.pure_model(analytic_jacobian=0)
    ref, ref_ok, _ = F.oracle_flash(oracle, td.model_bytes(model), rho, e, guess)
    model.phase[1].species[0].kappa *= OWN
    hem = GpuHem(model=td.model_bytes(model), capacity=n)
    try:
        got = guess.copy()
        inputs = np.zeros(n, dtype=A.CAPILLARY_DTYPE)
        inputs["equilibrium"] = 1
        ok, _ = hem.run_capillary(rho[:, None].copy(), e, inputs, got)
    finally:
        hem.close()
    assert ref_ok.all()
    s = F.compare(got, ok, ref, ref_ok)
    assert s["success_equal"] and s["label_mismatch"] == 0, s
    # both stop at residuals below 1e-9, as in test_two_phase_candidates_equal_the_general_evaluation
    assert s["p_rel"] <= 4e-8 and s["T_rel"] <= 3e-9 and s["ml_rel"] <= F.STATE_TOL, s


def test_undecided_points_match_the_general_evaluation(shim):  # noqa: F811
    """A condensable of three times N2O's a (Tc = 929 K): beside it the gas's
    reported-phase line lies where the residual formed alone decides nothing."""
    heavy = dict(td.N2O, name="heavy", a=3 * td.N2O["a"])
    tc = td.critical_point(heavy)[0]
    model = td.production_model(species=(td.N2, td.O2, td.N2O, heavy), condensable="heavy", analytic_jacobian=0,
                                controls=dict(td.N2O_FLASH, liquidTc=.999 * tc, pmax=1e9))
    n = 300
    rng = np.random.default_rng(5)
    T, beta = rng.uniform(.75, .93, n) * tc, rng.uniform(.1, .9, n)
    ps, gas, liq = PureFluid(heavy).saturation(T)
    rho = 1 / ((1 - beta) / gas["rho"] + beta / liq["rho"])
    q = np.zeros((n, 4))
    q[:, 0], q[:, 3] = 1e-3 * rho, rho
    e = rho * ((1 - beta) * gas["e"] + beta * liq["e"])
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = ps, T + rng.uniform(-3.0, 3.0, n), q.sum(axis=1)
    guess["liquidMass"][:, 0], guess["activeLiquids"] = beta * rho, 1
    got, ok, _ = gpu_flash(td.model_bytes(model), q, e, guess)
    own = td.HemModel.from_buffer_copy(model)
    own.phase[1].species[0].kappa *= OWN
    general, general_ok, _ = gpu_flash(td.model_bytes(own), q, e, guess)
    assert ok.all() and general_ok.all()
    s = F.compare(got, ok, general, general_ok)
    assert s["label_mismatch"] == 0 and s["p_rel"] <= 4e-8 and s["T_rel"] <= 3e-9 and s["ml_rel"] <= F.STATE_TOL, s
    for states, image in ((got, model), (general, own)):
        two = states["liquidMass"][:, 0] > 0
        assert two.mean() > .9
        scale = np.maximum(np.maximum(1e5 * states["rho"], np.abs(e)),
                           states["rho"] * 2000 * np.maximum(guess["T"], model.Tmin))
        x = np.column_stack([np.log(states["p"]), np.log(states["T"]), states["liquidMass"][:, 0] / q[:, 3], 0 * e])
        # the general evaluation on the host (it needs a model with the gas species' own tables)
        _, codes, accepted, _, g = residuals(shim, model, q[two], e[two], np.ones(two.sum()), False, (0.0, 0.0), x[two],
                                             scale[two])
        assert (codes == -1).all() and accepted.all()
        # the search's tolerances, and (own table) what 1e-13 of kappa moves
        assert np.abs(g[:, 0]).max() <= model.vtol * 1.01 and np.abs(g[:, 1]).max() <= model.etol * 1.01
        assert np.abs(g[:, 2]).max() <= model.mutol * 1.01
        for field, column in (("volumeResidual", 0), ("energyResidual", 1), ("chemicalResidual", 2)):
            assert np.abs(states[field][two] - np.abs(g[:, column])).max() <= 1e-10
