"""The legacy-input beamformer on runs of more than 65,535 sample tiles.

A call takes up to 262,140 samples whatever the tile. Arrays of 208 tiles of
complex doubles take tiles of two samples, so a run past 131,070 samples has
more of them than one grid dimension but x counts. Every sample is summed by
itself: the long run equals the same samples in calls of 65,000, bit for bit,
and a call of one sample more than the limit is refused."""
from __future__ import annotations

import pytest

from helpers import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("double,nant,ns", [(True, 208, 131_072), (True, 2, 262_140), (False, 2, 262_140), (False, 258, 262_140)])
def test_long_run(double, nant, ns):
    import vgb

    torch = torch_cuda()
    g = torch.Generator(device="cuda").manual_seed(nant)
    ni = 2 * nant
    v = torch.empty((ns, ni, 2), dtype=torch.float64, device="cuda") if double else torch.empty((ns, ni), dtype=torch.uint8, device="cuda")
    v.normal_(generator=g) if double else v.random_(0, 256, generator=g)
    W = torch.randn((nant, 1, 8), device="cuda", generator=g)
    polQ = torch.arange(0, ni, 2, dtype=torch.int32, device="cuda")
    polP = polQ + 1

    def run(v, n):
        S = torch.full((n, 4), float("nan"), device="cuda")
        e = torch.full((n, 4), float("nan"), device="cuda")
        inc = None if double else torch.full((n,), float("nan"), device="cuda")
        vgb.beamform_legacy(v, vgb.DBL if double else vgb.INT4, n, 1, nant, polQ, polP, W, 1, 1 / ni, 4, S, e, inc)
        return [x for x in (S, e, inc) if x is not None]

    whole = run(v, ns)
    parts = [run(v[s:s + 65_000], min(65_000, ns - s)) for s in range(0, ns, 65_000)]
    torch.cuda.synchronize()
    for k, x in enumerate(whole):
        assert not torch.isnan(x).any()
        assert torch.equal(x, torch.cat([p[k] for p in parts]))
    assert vgb.check_device_status() == 0
    with pytest.raises(vgb.VGBError):
        run(v, 262_141)
