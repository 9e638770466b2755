"""GPU: the flash's autotuner varies the grid of the launches that search the model's
candidates. Read from the kernel nodes of a captured batch: the search launches with
the blocks the tuner reports, and the restart search keeps its grid."""
import ctypes as C

import numpy as np
import pytest
import torch

from spuma_multiphysics_b200 import _lib, cases, thermo_data as td
from spuma_multiphysics_b200.hem import GpuHem

pytestmark = pytest.mark.gpu


class NodeParams(C.Structure):  # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def grids(launch):
    """{kernel name: grid} of the kernels `launch(stream)` launches (captured, never run)."""
    cuda = C.CDLL("libcuda.so.1")
    g = torch.cuda.CUDAGraph(keep_graph=True)
    stream = torch.cuda.Stream()
    with torch.cuda.graph(g, stream=stream):
        launch(stream.cuda_stream)
    handle, count = C.c_void_p(g.raw_cuda_graph()), C.c_size_t(0)
    assert cuda.cuGraphGetNodes(handle, None, C.byref(count)) == 0
    nodes = (C.c_void_p * count.value)()
    assert cuda.cuGraphGetNodes(handle, nodes, C.byref(count)) == 0
    out, kind, name = {}, C.c_int(), C.c_char_p()
    for node in nodes[:count.value]:
        assert cuda.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value:
            continue
        p = NodeParams()
        assert cuda.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
        assert (cuda.cuFuncGetName(C.byref(name), C.c_void_p(p.func)) if p.func
                else cuda.cuKernelGetName(C.byref(name), C.c_void_p(p.kern))) == 0
        for kernel in ("passSearch", "passQueue", "passRestarts"):
            if kernel.encode() in name.value:
                out[kernel] = p.grid[0]
    return out


# the search in registers; the work queue (finite-difference Jacobian); both
@pytest.mark.parametrize("options,searches", [({}, {"passSearch"}), (dict(analytic_jacobian=0), {"passQueue"}),
                                              (dict(stable_gas_prune=1), {"passQueue", "passSearch"})])
def test_search_launches_with_the_tuned_blocks(options, searches):
    n = 20000
    rho, e, guess = cases.flash_batch(n, seed=8, two_phase_share=.4, saturation_levels=64)
    cons = torch.zeros((5, n), dtype=torch.float64, device="cuda")
    cons[0], cons[4] = torch.from_numpy(rho).cuda(), torch.from_numpy(e).cuda()
    seed = torch.from_numpy(guess.view(np.uint8).copy()).cuda()
    state, ok = torch.zeros_like(seed), torch.zeros(n, dtype=torch.int32, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    hem = GpuHem(model=td.model_bytes(td.pure_model(**options)), capacity=n)
    try:
        run = lambda stream: hem.run_device(cons, n, n, 5, seed, state, None, ok, stream)
        run(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        untuned, expected = grids(run), state.clone()
        blocks, err = C.c_int(), C.create_string_buffer(512)
        assert _lib.load().reactive_gpu_hem_autotune_v3(hem.handle, cons.data_ptr(), n, n, 5, seed.data_ptr(),
                                                        torch.cuda.current_stream().cuda_stream, C.byref(blocks), err,
                                                        len(err)) == 0, err.value
        tuned = grids(run)
        assert set(untuned) == set(tuned) == searches | {"passRestarts"}
        assert tuned["passRestarts"] == untuned["passRestarts"]
        limit = max(untuned[k] for k in searches) // sms
        assert 1 <= blocks.value <= limit
        for k in searches:
            assert tuned[k] == min(blocks.value * sms, untuned[k]), (k, blocks.value, tuned, untuned)
        state.zero_()
        run(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert torch.equal(state, expected)
    finally:
        hem.close()
