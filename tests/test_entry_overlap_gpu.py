"""GPU: the host entries that only move conserved variables (upload, download) share
no array with the device stage entries: run while device stages of the same handle are
in flight on another stream, they leave every bit of the stages' results."""
import ctypes as C

import numpy as np
import pytest
import torch

from spuma_multiphysics_b200 import _abi as A, _lib
import transport_cases as T
from test_structured_gpu import box_case, mixed_kinds

pytestmark = pytest.mark.gpu


# enough cells that a run of stages outlasts the entries; one and four species, the
# structured box and the face graph
@pytest.mark.parametrize("ns", [1, 4])
@pytest.mark.parametrize("structured", [1, 0])
def test_moving_conserved_variables_leaves_stages_in_flight_alone(ns, structured):
    L = _lib.load()
    lib = T.bind(L)
    dims, stages, moves = (48, 40, 44), 200, 12
    case = box_case(dims, ns, mixed_kinds(dims, 3), viscous=True, conduction=True)
    nc, nv = case["nc"], case["nv"]
    h = T.create(lib, 1, case, wale_cw=.325)
    try:
        assert L.reactive_transport_structured_v3(h, structured, None) == 0
        fixed = C.c_size_t()
        sizes = [C.byref(C.c_size_t()), C.byref(fixed), C.byref(C.c_size_t()), C.byref(C.c_size_t())]
        assert L.reactive_transport_layout_v3(h, *sizes) == 0
        all_ = nc + fixed.value
        stream = torch.cuda.Stream()
        q0 = torch.zeros((nv, all_), dtype=torch.float64, device="cuda")
        q0[:, :nc] = torch.from_numpy(case["q"].T.copy()).cuda()
        st = torch.zeros((all_, 7), dtype=torch.float64, device="cuda")
        st[:nc] = torch.from_numpy(case["states"].view(np.float64).reshape(nc, 7)).cuda()
        assert L.reactive_transport_fill_fixed_v3(h, q0.data_ptr(), st.data_ptr(), 0) == 0
        torch.cuda.synchronize()
        assert L.reactive_transport_begin_attempt(h, b"", 1) == 0, lib.reactive_transport_error(h)
        back, version, out = np.empty_like(case["q"]), 0, []
        for move in (False, True):
            a, b = q0.clone(), q0.clone()
            done = torch.cuda.Event()
            torch.cuda.synchronize()
            for _ in range(stages):
                assert L.reactive_transport_stage_device_v3(h, a.data_ptr(), b.data_ptr(), st.data_ptr(), 1e-9, 0, None,
                                                            stream.cuda_stream) == 0
                a, b = b, a
            done.record(stream)
            overlapped = 0
            for _ in range(moves if move else 0):
                overlapped += not done.query()
                version += 1
                assert L.reactive_transport_upload_conserved(h, T.dp(case["q"]), version) == 0
                assert L.reactive_transport_download_conserved(h, A.Token(1, 0, version), T.dp(back)) == 0
                assert np.array_equal(back, case["q"])
            torch.cuda.synchronize()
            out.append(a.cpu().numpy())
        assert overlapped >= 1  # an entry began while the stages ran
        assert np.isfinite(out[0]).all() and not np.array_equal(out[0], q0.cpu().numpy())
        assert np.array_equal(out[0], out[1])
    finally:
        lib.reactive_transport_destroy(h)
