"""The legacy-input beamformer at the edges of its tiles, against NumPy in 64 bits.

The tile depends on the input type and the tile count: 64, 32, 16, 8 or 4
samples x 32 channels for 4+4-bit voltages, 32, 16, 8, 4 or 2 samples x 8
channels for complex doubles, and the one-row kernel for arrays whose voltages
do not fit a tile (more than 768 or 877 tiles). The cases take each tile, with
channels and samples that leave its last block partly filled, one and several
pointings, Stokes I and IQUV, and input lists that are no permutation.

Tolerance: a sum over n tiles of products of FP32 values is off by at most
(n + 8) 2^-24 of the sum of the magnitudes; the Stokes values are differences
of two such sums of squares, each at most (sum |W v|)^2, so 4 (n + 8) 2^-24 of
that bounds them.
"""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, host, torch_cuda

pytestmark = pytest.mark.gpu


def reference(v, W, polQ, polP, invw, nstokes):
    """S [p][s][st][c], e [p][s][c][2] and the bound of |ex|, |ey| [p][s][c]."""
    q, p = v[:, :, polQ], v[:, :, polP]
    S, e, bound = [], [], []
    for w in W.transpose(0, 2, 1, 3, 4).astype(np.complex128):  # [c][a][2][2]
        ex = w[..., 0, 0] * q + w[..., 0, 1] * p
        ey = w[..., 1, 0] * q + w[..., 1, 1] * p
        X, Y = ex.sum(-1), ey.sum(-1)
        xx = abs(X) ** 2 - (abs(ex) ** 2).sum(-1)
        yy = abs(Y) ** 2 - (abs(ey) ** 2).sum(-1)
        xy = X * Y.conj() - (ex * ey.conj()).sum(-1)
        S.append(np.stack([invw * (xx + yy), invw * (xx - yy), 2 * invw * xy.real, -2 * invw * xy.imag][:nstokes], 1))
        e.append(np.stack([X, Y], -1))
        mag = np.abs(w)
        bound.append(np.maximum((mag[..., 0, 0] * abs(q) + mag[..., 0, 1] * abs(p)).sum(-1),
                                (mag[..., 1, 0] * abs(q) + mag[..., 1, 1] * abs(p)).sum(-1)))
    return np.array(S), np.array(e), np.array(bound)


CASES = [  # double, tiles, channels, samples, pointings, Stokes
    (False, 2, 1, 1, 1, 1), (False, 6, 33, 65, 2, 4), (False, 18, 31, 63, 1, 4), (False, 36, 64, 17, 3, 1),
    (False, 66, 40, 23, 1, 4), (False, 128, 33, 9, 2, 4), (False, 160, 32, 8, 1, 4), (False, 258, 5, 7, 2, 4),
    (False, 770, 3, 5, 1, 4),
    (True, 1, 1, 1, 1, 1), (True, 5, 9, 33, 2, 4), (True, 17, 7, 31, 1, 4), (True, 33, 16, 17, 3, 1),
    (True, 65, 9, 9, 1, 4), (True, 128, 9, 5, 2, 4), (True, 145, 8, 3, 1, 4), (True, 255, 3, 5, 2, 4),
    (True, 890, 2, 3, 1, 4),
    # enough blocks for several sample groups a block, with a partial last group; pointings over the blocks
    (False, 6, 128, 619, 1, 4), (False, 36, 120, 333, 2, 4), (False, 8, 128, 21, 5, 4), (False, 130, 64, 9, 7, 1),
    (True, 5, 127, 615, 1, 4), (True, 20, 128, 307, 2, 4), (True, 33, 128, 157, 1, 1), (True, 128, 128, 78, 2, 4),
    (True, 21, 64, 11, 6, 4),
]


@pytest.mark.parametrize("double,nant,nchan,ns,npnt,nst", CASES)
def test_legacy_tiles_against_numpy(double, nant, nchan, ns, npnt, nst):
    import vgb

    torch = torch_cuda()
    rng = np.random.default_rng(nant * 1000 + ns)
    ni = 2 * nant
    if double:
        v = rng.standard_normal((ns, nchan, ni)) + 1j * rng.standard_normal((ns, nchan, ni))
        v[0, 0, : min(4, ni)] = [0.0, 1e-42 + 0j, 3e-39j, -0.0][: min(4, ni)]  # zero and FP32 subnormals
        raw = v
        v = v.real.astype(np.float32).astype(np.float64) + 1j * v.imag.astype(np.float32)
    else:
        raw = rng.integers(0, 256, size=(ns, nchan, ni), dtype=np.uint8)  # every nibble, -8 included
        sign = lambda n: ((n.astype(np.int64) ^ 8) - 8).astype(np.float64)  # noqa: E731
        v = sign(raw >> 4) + 1j * sign(raw & 15)
    # any input lists: repeated and unused inputs too
    polQ = rng.integers(0, ni, nant).astype(np.uint32)
    polP = rng.integers(0, ni, nant).astype(np.uint32)
    W = (rng.standard_normal((npnt, nant, nchan, 2, 2)) + 1j * rng.standard_normal((npnt, nant, nchan, 2, 2))).astype(np.complex64)
    invw = 1.0 / ni
    S = torch.full((npnt, ns, nst, nchan), float("nan"), device="cuda")
    e = torch.full((npnt, ns, nchan, 2, 2), float("nan"), device="cuda")
    inc = None if double else torch.full((ns, nchan), float("nan"), device="cuda")
    vgb.beamform_legacy(dev(raw), vgb.DBL if double else vgb.INT4, ns, nchan, nant, dev(polQ), dev(polP), dev(W), npnt,
                        invw, nst, S, e, inc)
    torch.cuda.synchronize()
    Sref, eref, bound = reference(v, W, polQ, polP, invw, nst)
    eps = (nant + 8) * 2.0 ** -24
    got = host(e).astype(np.float64)
    assert np.all(np.abs(got[..., 0] + 1j * got[..., 1] - eref) <= 2 * eps * bound[..., None])
    assert np.all(np.abs(host(S) - Sref) <= 8 * eps * invw * (bound ** 2)[:, :, None])
    if inc is not None:
        assert np.array_equal(host(inc), (np.abs(v) ** 2).round().sum(-1).astype(np.float32))
    assert vgb.check_device_status() == 0
