"""Up to 32 beams (voltages kept as input bytes, widened inside the beam GEMM)
against the general path: a run over 40 beams (two beam tiles, 16-bit
voltages in memory) whose first beams are the same. A beam's products, their
order and its epilogue are the same in both, so Stokes, bytes, offsets and
scales have to agree bit for bit."""
import numpy as np
import pytest

from helpers import torch_cuda
from test_gpu_multibeam import make_case, run_mb

pytestmark = pytest.mark.gpu


# the smallest array and run, one and two integrations left over after a whole sample tile, an odd count of
# integrations, several integration shares of the 8-bit stage, a wide array, the last full beam tile
@pytest.mark.parametrize("nant,npnt,nfine,ns", [(16, 1, 1, 10), (48, 5, 3, 260), (32, 20, 33, 770), (128, 32, 32, 2600),
                                                (528, 3, 2, 250), (144, 31, 128, 500)])
@pytest.mark.parametrize("precision,nstokes,int8", [(0, 4, False), (0, 1, True), (1, 1, False), (1, 4, True), (2, 4, False),
                                                    (2, 1, True)])
def test_few_beams_match_the_general_path(oracle_mod, nant, npnt, nfine, ns, precision, nstokes, int8):
    torch = torch_cuda()
    import vgb

    case = make_case(oracle_mod, nant, 40, nfine, ns, seed=nant + ns, int8=int8)
    # two inputs, in a random input order: the Gaussian voltages of the case, and every byte value (-128 included),
    # where 10 samples of 8-bit power overflow the FP16 coherencies in either path: the same non-finite values then
    rng = np.random.default_rng(ns + nant)
    every = rng.integers(0, 256, size=case["v_dev"].shape, dtype=np.uint8)
    order = rng.permutation(2 * nant).astype(np.uint32)
    case["polQ"], case["polP"] = np.ascontiguousarray(order[0::2]), np.ascontiguousarray(order[1::2])
    for v in (every, case["v_dev"]):
        c = dict(case, v_dev=v)
        many = run_mb(vgb, torch, c, nant, 40, nfine, ns, nstokes, precision, int8=int8, invw=1.0, psrfits=True)
        c = dict(c, unit=np.ascontiguousarray(case["unit"][:npnt]), B=np.ascontiguousarray(case["B"][:npnt]))
        few = run_mb(vgb, torch, c, nant, npnt, nfine, ns, nstokes, precision, int8=int8, invw=1.0, psrfits=True)
        assert few["launches"] == many["launches"] == 5
        assert np.array_equal(few["S"], many["S"][:, :npnt], equal_nan=True)
        for k in ("out", "off", "scl"):
            assert np.array_equal(few[k], many[k][:npnt], equal_nan=k != "out"), k
    assert np.isfinite(few["S"]).all() and np.abs(few["S"]).max() > 0
