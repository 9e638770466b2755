"""GPU: the restart search, a warp a cell with its twenty two-phase solves on as many
lanes. States over the whole density range and beyond both ends of it, from seeds far
off, against the oracle flash's serial search: the same cells recovered, among them ones
that only a restart solves, and the same cells left as their seeds."""
import numpy as np
import pytest
import torch

from oracle import oracle
from spuma_multiphysics_b200 import _abi as A, thermo_data as td
from spuma_multiphysics_b200.hem import GpuHem
import flash_cases as F

pytestmark = pytest.mark.gpu


def far_seeds(n, seed):
    """(rho, e, seeds at 250 K and random pressures and liquid fractions): gas, the whole
    dome, compressed liquid, and energies that no state of N2O has."""
    rng = np.random.default_rng(seed)
    rho = np.exp(rng.uniform(np.log(1.0), np.log(1300.0), n))
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = np.exp(rng.uniform(np.log(1e4), np.log(4e7), n)), 250.0, rho
    liquid = rng.uniform(0, 1, n) * (rng.uniform(0, 1, n) < .5)
    guess["liquidMass"][:, 0], guess["gasMass"] = liquid * rho, (1 - liquid) * rho
    return rho, rho * rng.uniform(1.3e6, 2.2e6, n), guess


@pytest.mark.parametrize("options", [{}, dict(analytic_jacobian=0)], ids=["registers", "queue"])
def test_restarts_match_the_oracle_s_serial_search(options):
    n = 1200
    rho, e, guess = far_seeds(n, 3)
    image = td.model_bytes(td.pure_model(**options))
    ref, ref_ok, counts = F.oracle_flash(oracle, image, rho, e, guess)
    restarted = counts[:, 2] > 5  # two-phase candidates: five, and twenty by restarts
    hem = GpuHem(model=image, capacity=n)
    try:
        cons = torch.zeros((5, n), dtype=torch.float64, device="cuda")
        cons[0], cons[4] = torch.from_numpy(rho).cuda(), torch.from_numpy(e).cuda()
        seed = torch.from_numpy(guess.view(np.uint8).copy()).cuda()
        # any number of queued cells: one cell, a few warps of them, all
        picks = [np.nonzero(restarted & (ref_ok != 0))[0][:1], np.nonzero(restarted)[0][:37], np.arange(n)]
        for pick in picks:
            m, index = len(pick), torch.from_numpy(pick).cuda()
            q = cons[:, index].contiguous()
            s = seed.view(n, -1)[index].contiguous()
            state, ok = torch.zeros_like(s), torch.zeros(m, dtype=torch.int32, device="cuda")
            hem.run_device(q, m, m, 5, s, state, None, ok, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            got, got_ok = state.cpu().numpy().reshape(-1).view(A.THERMO_DTYPE), ok.cpu().numpy()
            summary = F.compare(got, got_ok, ref[pick], ref_ok[pick])
            assert summary["success_equal"] and summary["label_mismatch"] == 0, (m, summary)
            # both stop at residuals below 1e-9, as in test_two_phase_candidates_equal_the_general_evaluation
            assert summary["p_rel"] <= 4e-8 and summary["T_rel"] <= 3e-9, (m, summary)
            failed = got_ok == 0
            assert got[failed].tobytes() == guess[pick][failed].tobytes()
    finally:
        hem.close()
    assert (restarted & (ref_ok != 0)).sum() >= 5 and (ref_ok == 0).sum() >= 100
