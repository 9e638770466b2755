"""GPU: the rate VJP by the dot-product test on boxes from two cells a side (every cell
a corner) past a block's 128 cells, one to four species, each with and without the
viscous terms."""
import ctypes as C

import numpy as np
import pytest
import torch

from spuma_multiphysics_b200 import _abi as A, _lib
import transport_cases as T
from test_structured_gpu import box_case, mixed_kinds

pytestmark = pytest.mark.gpu
FIELDS = ("p", "T", "rho", "sound")


@pytest.mark.parametrize("dims,ns", [((2, 2, 2), 1), ((2, 2, 2), 4), ((43, 3, 2), 2), ((3, 2, 22), 3), ((5, 9, 3), 1)])
@pytest.mark.parametrize("wale,viscous", [(None, False), (None, True), (.325, False), (.325, True)])
def test_rate_vjp_dot_product(dims, ns, wale, viscous):
    L = _lib.load()
    lib = T.bind(L)
    case = box_case(dims, ns, mixed_kinds(dims, 7), viscous=viscous, conduction=viscous, seed=9)
    h = T.create(lib, 1, case, wale_cw=wale)
    nc, nv = case["nc"], case["nv"]
    rng = np.random.default_rng(2)
    try:
        q, st = case["q"], case["states"]

        def rhs(qq, ss):
            out, br = np.empty_like(qq), np.empty(nv)
            assert lib.reactive_transport_rhs(h, T.dp(np.ascontiguousarray(qq)), T.states_ptr(ss), None, None,
                                              T.dp(out), T.dp(br)) == 0, lib.reactive_transport_error(h)
            return out

        vq = rng.normal(size=q.shape) * np.abs(q).max(axis=0)
        vs = {f: rng.normal(size=nc) * np.abs(st[f]).max() * .1 for f in FIELDS}
        w = rng.normal(size=q.shape)
        eps, sp, sm = 1e-6, st.copy(), st.copy()
        for f in FIELDS:
            sp[f] += eps * vs[f]
            sm[f] -= eps * vs[f]
        up, down = rhs(q + eps * vq, sp), rhs(q - eps * vq, sm)
        fd = float(np.sum(w * (up - down) / (2 * eps)))
        sizes = [C.c_size_t() for _ in range(4)]
        assert L.reactive_transport_layout_v3(h, *(C.byref(x) for x in sizes)) == 0
        all_ = nc + sizes[1].value
        stream = torch.cuda.current_stream().cuda_stream
        qd = torch.zeros((nv, all_), dtype=torch.float64, device="cuda")
        qd[:, :nc] = torch.from_numpy(q.T.copy()).cuda()
        sd = torch.zeros((all_, 7), dtype=torch.float64, device="cuda")
        sd[:nc] = torch.from_numpy(st.view(np.float64).reshape(nc, 7)).cuda()
        assert L.reactive_transport_fill_fixed_v3(h, qd.data_ptr(), sd.data_ptr(), stream) == 0
        wd = torch.from_numpy(w.T.copy()).cuda()
        q_bar = torch.empty((nv, nc), dtype=torch.float64, device="cuda")
        s_bar = torch.empty((nc, 7), dtype=torch.float64, device="cuda")
        assert L.reactive_transport_rate_vjp_v3(h, qd.data_ptr(), sd.data_ptr(), wd.data_ptr(), q_bar.data_ptr(),
                                                s_bar.data_ptr(), stream) == 0, lib.reactive_transport_error(h)
        torch.cuda.synchronize()
        sb = s_bar.cpu().numpy().view(A.STATE_DTYPE).reshape(nc)
        adj = float(np.sum(q_bar.cpu().numpy().T * vq)) + sum(float(np.sum(sb[f] * vs[f])) for f in FIELDS)
        # truncation 1e-6 of the sum (as the larger boxes' test), and the differences' own
        # rounding: an ulp of the largest rate a term over the step
        rounding = 2.3e-16 * np.abs(up).max(axis=0) @ np.abs(w).sum(axis=0) / eps
        assert abs(adj - fd) <= 1e-6 * abs(fd) + rounding, (adj, fd, rounding)
    finally:
        lib.reactive_transport_destroy(h)
