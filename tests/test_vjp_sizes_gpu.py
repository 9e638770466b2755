"""GPU: the hand-written adjoints at the sizes and states where a cell's sides are few:
the rate VJP by the dot-product test on boxes from two cells a side (every cell a
corner) past a block's 128 cells, one to four species, each with and without the
viscous terms; the flash VJP of single-phase cells, gas to 1500 K and compressed
liquid, against central differences of the flash."""
import ctypes as C

import numpy as np
import pytest
import torch

from spuma_multiphysics_b200 import _abi as A, _lib
from spuma_multiphysics_b200.eos import PureFluid
from spuma_multiphysics_b200.hem import GpuHem
from spuma_multiphysics_b200.thermo_data import N2O
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


@pytest.mark.parametrize("phase", ["gas", "liquid"])
def test_single_phase_flash_vjp(phase):
    n = 600
    rng = np.random.default_rng(3)
    if phase == "gas":
        t, p = np.exp(rng.uniform(np.log(250.0), np.log(1500.0), n)), np.exp(rng.uniform(np.log(5e4), np.log(1.5e6), n))
    else:
        # to 10 MPa: denser liquids' cubics fall into the absolute near-repeated-root band of the
        # root rules (|disc| < 1e-14, volumes below 0.04 m^3/kmol), where no search solves them
        # (the oracle solves none above 13 MPa)
        t, p = rng.uniform(190.0, 295.0, n), rng.uniform(6.5e6, 1e7, n)
    s = PureFluid(N2O).tp(t, p, root=phase)
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = p, t, s["rho"]
    if phase == "liquid":
        guess["liquidMass"][:, 0], guess["activeLiquids"] = s["rho"], 1
    q = np.zeros((5, n))
    q[0], q[4] = s["rho"], s["rho"] * s["e"]
    q[1:4] = rng.normal(0, 20, (3, n)) * q[0]
    q[4] += .5 * (q[1:4] ** 2).sum(0) / q[0]
    hem = GpuHem(capacity=n)
    seed = torch.from_numpy(guess.view(np.uint8).copy()).cuda()

    def flash(x):
        cons, state = torch.from_numpy(np.ascontiguousarray(x)).cuda(), torch.zeros_like(seed)
        tr, ok = torch.zeros((n, 7), dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        hem.run_device(cons, n, n, 5, seed, state, tr, ok, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert ok.cpu().numpy().all()
        return cons, state, tr.cpu().numpy()

    try:
        cons, state, tr = flash(q)
        scale = np.abs(tr).max(axis=0)
        scale[scale == 0] = 1.0
        bar = rng.normal(size=(n, 7)) / scale
        bar[:, 6] = 0
        q_bar = torch.zeros((5, n), dtype=torch.float64, device="cuda")
        failed, err = torch.zeros(1, dtype=torch.int32, device="cuda"), C.create_string_buffer(512)
        assert _lib.load().reactive_gpu_hem_vjp_device_v3(
            hem.handle, cons.data_ptr(), n, n, 5, state.data_ptr(), torch.from_numpy(bar).cuda().data_ptr(),
            q_bar.data_ptr(), n, failed.data_ptr(), torch.cuda.current_stream().cuda_stream, err, len(err)) == 0
        torch.cuda.synchronize()
        assert failed.item() == 0
        v, eps = rng.normal(size=q.shape) * np.abs(q), 1e-4
        fd = np.sum(bar * (flash(q + eps * v)[2] - flash(q - eps * v)[2]) / (2 * eps), axis=1)
        adj = np.sum(q_bar.cpu().numpy() * v, axis=0)
        # steps of 1e-4: truncation 1e-8 of third derivatives of order one (a hundred in the
        # liquid, whose volume sits near the covolume), the flash's 1e-9 over the step 1e-5
        size = np.abs(bar * scale).sum(axis=1) * (100.0 if phase == "liquid" else 1.0)
        assert np.max(np.abs(adj - fd) / np.maximum(np.abs(fd), size)) <= 1e-4
    finally:
        hem.close()
