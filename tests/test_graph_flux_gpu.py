"""GPU: the face graph's finished-flux form (up to 12 conserved variables) and the
form it replaces there (more variables): the combined CFL + stage entry equals the
two calls bit for bit, and both equal the oracle's rates."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle
from spuma_multiphysics_b200 import _lib
import transport_cases as T

pytestmark = pytest.mark.gpu


# nv = 5, 12 (the last with finished fluxes), 13; one cell, a block's edges; boundary
# faces within one ledger block (256) and past it
@pytest.mark.parametrize("ns", [1, 8, 9])
@pytest.mark.parametrize("nc,extra,wale", [(1, 0, None), (255, 0, .325), (257, 0, None), (300, 700, None)])
def test_combined_entry_equals_the_two_calls_and_the_oracle(ns, nc, extra, wale):
    L = _lib.load()
    lib = T.bind(L)
    case = T.make_case(ns, nc, 3, spatial=nc > 1, extra_boundary=extra, viscous_only=True, conduction=wale is None)
    nv = case["nv"]
    h = T.create(lib, 1, case, wale_cw=wale)
    try:
        sizes = [C.c_size_t() for _ in range(4)]
        assert L.reactive_transport_layout_v3(h, *(C.byref(x) for x in sizes)) == 0
        all_ = nc + sizes[1].value
        s = torch.cuda.current_stream().cuda_stream
        q0 = torch.zeros((nv, all_), dtype=torch.float64, device="cuda")
        q0[:, :nc] = torch.from_numpy(case["q"].T.copy()).cuda()
        st = torch.zeros((all_, 7), dtype=torch.float64, device="cuda")
        st[:nc] = torch.from_numpy(case["states"].view(np.float64).reshape(nc, 7)).cuda()
        assert L.reactive_transport_fill_fixed_v3(h, q0.data_ptr(), st.data_ptr(), s) == 0
        states = case["states"].ctypes.data_as(C.c_void_p)
        cw = -1.0 if wale is None else wale
        dt = .1 * oracle.transport_stable_dt(case, case["q"], states, .23, .1, wale_cw=cw)
        out = []
        for combined in (False, True):
            q1, br = q0.clone(), torch.zeros(nv, dtype=torch.float64, device="cuda")
            d = torch.zeros(1, dtype=torch.float64, device="cuda")
            if combined:
                assert L.reactive_transport_stage_cfl_device_v3(h, q0.data_ptr(), q1.data_ptr(), st.data_ptr(), dt, 0,
                                                                br.data_ptr(), .23, .1, d.data_ptr(), s) == 0
            else:
                assert L.reactive_transport_stable_step_device_v3(h, q0.data_ptr(), st.data_ptr(), .23, .1,
                                                                  d.data_ptr(), s) == 0
                assert L.reactive_transport_stage_device_v3(h, q0.data_ptr(), q1.data_ptr(), st.data_ptr(), dt, 0,
                                                            br.data_ptr(), s) == 0
            torch.cuda.synchronize()
            out.append((d.item(), q1.cpu().numpy(), br.cpu().numpy()))
        assert out[0][0] == out[1][0] > 0
        assert np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
        rates, ledger, _, _, status = oracle.transport_rhs(case, case["q"], states, case["y"], case["h"], wale_cw=cw)
        assert status == 0
        assert abs(out[0][0] / (10 * dt) - 1) < T.DT_TOL
        # q + dt rate: the rate's bound, the rounding of the sum divided by dt, and that of
        # the face fluxes that cancel in it: p A / V up to 1.25e5 x 1.5 / 0.1 (and u times
        # as much in the energy, within its own scale), one ulp for each of four faces
        got = (out[0][1][:, :nc].T - case["q"]) / dt
        scale = np.maximum(1.0, np.abs(rates).max(axis=0))
        rounding = 4e-16 * np.abs(case["q"]).max(axis=0) / dt
        rounding[ns:ns + 3] += 4 * 2.3e-16 * 1.25e5 * 1.5 / .1
        assert (np.abs(got - rates).max(axis=0) <= T.RHS_TOL * scale + rounding).all()
        assert T.scaled_error(out[0][2][None], ledger[None]) <= T.RHS_TOL
    finally:
        lib.reactive_transport_destroy(h)
