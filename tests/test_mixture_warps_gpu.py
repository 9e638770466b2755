"""GPU: the multi-species flash spreads a cell's evaluations over a warp. A cell's
result must not depend on its place in the batch: batches of every remainder, in
any order, give each cell the bits it has in the whole batch, and the captured
results of the reference."""
import numpy as np
import pytest

from oracle import oracle
from spuma_multiphysics_b200 import _abi as A, thermo_data as td
from test_mixture_flash_gpu import GOLDEN, check, gpu_flash

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def whole():
    d = np.load(GOLDEN)
    guess = d["guess"].view(A.THERMO_DTYPE)
    image = td.model_bytes(td.two_liquid_model())
    out, ok, _ = gpu_flash(image, d["q"], d["energy"], guess)
    return d, guess, image, out, ok


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 33, 127, 129])
def test_any_part_of_a_batch_gives_the_whole_batch_s_bits(whole, n):
    d, guess, image, out, ok = whole
    pick = np.random.default_rng(n).permutation(len(ok))[:n]
    got, got_ok, prof = gpu_flash(image, d["q"][pick], d["energy"][pick], np.ascontiguousarray(guess[pick]))
    assert np.array_equal(got_ok, ok[pick])
    assert got.tobytes() == out[pick].tobytes()
    check(got, got_ok, d["out"].view(A.THERMO_DTYPE)[pick], d["success"][pick], min_success=1.0)
    assert prof.submitted == n and prof.stableCandidates >= n and prof.flashCandidates >= n
