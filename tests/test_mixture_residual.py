"""CPU: the two-phase residual formed alone (spuma-multiphysics_b200/csrc/
mixture_residual.cuh, host and device code from one source) against the residual
of the general mixture evaluation, over compositions with traces, liquid
fractions, log vapour fractions and a pressure jump, inside and outside the
liquids' ranges: accepted exactly where the general evaluation accepts, undecided
(left to it) on a vanishing share, and equal to the rounding of the sums."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from spuma_multiphysics_b200 import thermo_data as td

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    out = tmp_path_factory.mktemp("residual") / "libmixture_residual.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-I", str(ROOT / "spuma-multiphysics_b200" / "csrc"),
                    str(ROOT / "tests" / "native" / "mixture_residual_shim.cpp"), "-o", str(out)], check=True)
    return C.CDLL(str(out))


def residuals(shim, model, q, energy, mask, adaptive, offsets, x, scale):
    n = len(energy)
    codes, general = np.zeros(n, np.int32), np.zeros(n, np.int32)
    f, g = np.zeros((n, 4)), np.zeros((n, 4))
    p = lambda a: np.ascontiguousarray(a).ctypes.data_as(C.c_void_p)
    keep = [np.ascontiguousarray(a) for a in (q, energy, mask.astype(np.int32), x, scale)]
    valid = shim.mix_residuals(C.byref(model), C.c_long(n), p(keep[0]), p(keep[1]), p(keep[2]), int(adaptive),
                               C.c_double(offsets[0]), C.c_double(offsets[1]), p(keep[3]), p(keep[4]),
                               p(codes), p(general), p(f), p(g))
    return valid, codes, general, f, g


@pytest.mark.parametrize("name", ["one liquid", "two liquids"])
@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("T_range", [(145.0, 320.0), (300.0, 520.0)])
@pytest.mark.parametrize("offsets", [(0.0, 0.0), (3e4, -7e4)])
def test_residual_equals_the_general_evaluation(shim, name, adaptive, T_range, offsets):
    one = name == "one liquid"
    model = td.production_model(analytic_jacobian=0) if one else td.two_liquid_model()
    rng = np.random.default_rng(17)
    n = 6000
    Y = rng.dirichlet([.3] * 4, n)
    Y[: n // 8, 0] = 0.0  # absent species
    rho = np.exp(rng.uniform(np.log(.5), np.log(900.0), n))
    q = Y * rho[:, None]
    energy = rho * rng.uniform(-3e6, 2e6, n)
    p = np.exp(rng.uniform(np.log(2e4), np.log(4e7), n))
    T = rng.uniform(*T_range, n)
    fractions = -np.exp(rng.uniform(-3, 3, (n, 2))) if adaptive else rng.uniform(0, 1, (n, 2))
    x = np.column_stack([np.log(p), np.log(T), fractions])
    mask = np.ones(n, int) if one else rng.integers(1, 4, n)
    scale = np.maximum(1e5 * rho, np.abs(energy))
    valid, codes, general, f, g = residuals(shim, model, q, energy, mask, adaptive, offsets, x, scale)
    assert valid == 1
    decided = codes >= 0
    assert decided.mean() > .99
    assert np.array_equal(codes[decided], general[decided])
    both = decided & (codes == 1)
    assert both.sum() > 10
    # a root carries a few ulp over its distance from the covolume (a hundred at most
    # in these liquids); the chemical potentials' terms are below a thousand
    assert np.max(np.abs(f - g)[both, 0] / (1 + np.abs(g[both, 0]))) <= 1e-13
    assert np.max(np.abs(f - g)[both, 1]) <= 1e-12
    assert np.max(np.abs(f - g)[both, 2:]) <= 2e-12


def test_terms_refuse_a_liquid_that_is_not_the_gas_species(shim):
    model = td.production_model(analytic_jacobian=0)
    model.phase[1].species[0].kappa *= 1 + 1e-12
    one = np.ones(1)
    assert residuals(shim, model, np.ones((1, 4)), one, np.ones(1), False, (0, 0), np.zeros((1, 4)), one)[0] == 0
