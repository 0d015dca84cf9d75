"""The many-beam beamformer on 8-bit voltages of full range, every byte value.

Ten samples of a tile's power reach 327,680, past FP16's largest number, where
the coherencies' halves are FP16. Stokes of both voltage paths (up to 32 beams
and more) and every precision are finite and match the FP64 oracle within
each mode's tolerance (test_gpu_multibeam): uniform random bytes, and every
value at -128, the largest power there is."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import torch_cuda
from test_gpu_multibeam import make_case, oracle_stokes, run_mb, stokes_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npnt", [7, 40])
@pytest.mark.parametrize("precision,tol", [(0, 1e-3), (2, 4e-3), (1, 3e-2), (3, 2e-5)])
@pytest.mark.parametrize("constant", [False, True])
def test_full_range_voltages(oracle_mod, npnt, precision, tol, constant):
    torch = torch_cuda()
    import vgb

    nant, nfine, ns, nst = 48, 3, 510, 4
    case = make_case(oracle_mod, nant, npnt, nfine, ns, int8=True)
    shape = case["v_dev"].shape
    raw = np.full(shape, -128, np.int8) if constant else np.random.default_rng(5).integers(-128, 128, shape, dtype=np.int8)
    case["v_dev"] = raw.view(np.uint8)
    case["v_oracle"] = raw[..., 0].astype(np.float64) + 1j * raw[..., 1].astype(np.float64)
    invw = 1.0 / (2 * nant)
    res = run_mb(vgb, torch, case, nant, npnt, nfine, ns, nst, precision, int8=True, invw=invw, psrfits=True)
    assert np.isfinite(res["S"]).all() and np.isfinite(res["off"]).all() and np.isfinite(res["scl"]).all()
    for st, err in enumerate(stokes_err(res["S"], oracle_stokes(oracle_mod, case, nst, invw))):
        assert err < tol, (st, err)
