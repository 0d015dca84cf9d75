"""vgb_renormalise of runs so short that blocks of a cluster have no samples.

Eight blocks share a row's samples and read one another's extremes before they
leave, so with fewer samples than blocks, or about as many, the idle ones reach
their end while the others still read. Many rows at once, repeated, against
NumPy's extremes and the oracle's bytes, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, host, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nstep", [1, 2, 3, 7, 8, 9, 15, 17])
def test_blocks_without_samples(nstep, oracle_mod):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(nstep)
    ncc, npnt, nst, nchan = 3, 5, 4, 256
    S = (rng.standard_normal((ncc, npnt, nstep, nst, nchan)) * 100).astype(np.float32)
    want = [oracle_mod.renormalise(S[cc]) for cc in range(ncc)]
    d, per = dev(S), nstep * nst * nchan
    for _ in range(20):
        out = torch.full((S.size,), 0x5A, dtype=torch.uint8, device="cuda")
        off = torch.full((ncc * npnt * nst * nchan,), float("nan"), device="cuda")
        scl = torch.full_like(off, float("nan"))
        vgb.renormalise(d, ncc, npnt, nstep, nst, nchan, out, npnt * per, per, nst * nchan, nchan, off, scl)
        torch.cuda.synchronize()
        off, scl, out = host(off).reshape(ncc, npnt, nst, nchan), host(scl).reshape(ncc, npnt, nst, nchan), host(out).reshape(S.shape)
        assert np.array_equal(off, S.min(axis=2))
        for cc, (o, s, u) in enumerate(want):
            assert np.array_equal(off[cc], o) and np.array_equal(scl[cc], s) and np.array_equal(out[cc], u)
