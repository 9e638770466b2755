"""GPU: the ideal-gas closure's way to the temperature (the Newton between the iterates
on either side of the solution) recovers the generating temperature, whatever the
distance of the seed and the number of species, and fails where the range ends first."""
import numpy as np
import pytest
import torch

from spuma_multiphysics_b200 import cases
from spuma_multiphysics_b200.adjoint import IdealGasBox
from spuma_multiphysics_b200.thermo_data import ideal_cv, ideal_energy, N2, N2O

pytestmark = pytest.mark.gpu


# at the seed; a Newton inside the first radius (1% of T); far up, far down and from
# either end of the range, where the first steps overshoot it
@pytest.mark.parametrize("species", [(N2O,), (N2O, N2), (N2, N2O, N2), (N2O, N2, N2, N2O)], ids=len)
@pytest.mark.parametrize("seed_T", [150.0, 300.0, 1000.0, 3000.0])
def test_recovers_the_generating_temperature(species, seed_T):
    n = 8
    spec = cases.blast_box(n, edge=n * 1e-3, radius=2e-3, species=(N2O, N2))
    box = IdealGasBox(spec["faces"], spec["volume"], species, T_guess=seed_T)
    try:
        rng = np.random.default_rng(len(species))
        cells, ns = n ** 3, len(species)
        T = np.exp(rng.uniform(np.log(160.0), np.log(2900.0), cells))
        T[: cells // 4] = seed_T * (1 + rng.uniform(-2e-3, 2e-3, cells // 4)) if 160 < seed_T < 2900 else 500.0
        Y = rng.dirichlet(np.ones(ns), cells)
        rho = rng.uniform(.5, 20.0, cells)
        u = sum(Y[:, k] * np.array([ideal_energy(sp, t) for t in T]) for k, sp in enumerate(species))
        q = np.zeros((ns + 4, cells))
        q[:ns] = (rho[:, None] * Y).T
        mom = rng.uniform(-30, 30, (3, cells)) * rho
        q[ns:ns + 3] = mom
        q[ns + 3] = rho * u + .5 * (mom ** 2).sum(0) / rho
        got, _ = box.closure(torch.from_numpy(q).cuda())
        torch.cuda.synchronize()
        assert (box.success.cpu().numpy() == 1).all()
        # e's round-off (sums of terms below 1e7 J/kg, cv above 500) is 1e-11 K; the
        # accepted residual, 2.5e-14 of cp T, is corrected by its own Newton step
        assert np.max(np.abs(got.cpu().numpy() - T) / T) <= 1e-12
    finally:
        box.close()


# solutions beyond either end of [150, 3000] K (a cell's energy shifted by cv times the
# distance), at the ends themselves and just inside them
@pytest.mark.parametrize("seed_T", [150.0, 300.0, 2999.0, 3000.0])
def test_solutions_at_and_beyond_the_range(seed_T):
    n = 4
    spec = cases.blast_box(n, edge=n * 1e-3, radius=2e-3, species=(N2O, N2))
    box = IdealGasBox(spec["faces"], spec["volume"], (N2O, N2), T_guess=seed_T)
    try:
        cells = n ** 3
        T = np.resize([150.0, 150.0 + 1e-9, 160.0, 2990.0, 3000.0 - 1e-9, 3000.0], cells)
        shift = np.resize([0.0, 0.0, -20.0, 20.0, 0.0, 0.0, -1.0], cells)  # K
        inside = shift == 0
        u = sum(.5 * np.array([ideal_energy(sp, t) + ideal_cv(sp, t) * d for t, d in zip(T, shift)]) for sp in (N2O, N2))
        q = np.zeros((6, cells))
        q[:2], q[5] = 1.0, 2.0 * u
        got, _ = box.closure(torch.from_numpy(q).cuda())
        torch.cuda.synchronize()
        ok = box.success.cpu().numpy()
        beyond = (T + shift < 149.5) | (T + shift > 3000.5)
        assert (ok[inside] == 1).all() and (ok[beyond] == 0).all() and beyond.any()
        # 1e-12 as above: the ends are within the closure's own tolerance of themselves
        assert np.max(np.abs(got.cpu().numpy() - T)[inside] / T[inside]) <= 1e-12
    finally:
        box.close()
