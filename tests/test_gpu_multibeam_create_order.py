"""vgb_multibeam_create beside a busy default stream.

The handle's padding is zeroed at creation. A run on a non-blocking stream is
not ordered behind the default stream, so that zeroing has to be complete when
create returns: with about 0.2 s of work queued on the default stream, a run on
another stream gives the Stokes and bytes of a run on an idle GPU."""
from __future__ import annotations

import numpy as np
import pytest

from helpers import dev, host, torch_cuda
from test_gpu_multibeam import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 2, 3])
@pytest.mark.parametrize("npnt", [5, 40])
def test_run_on_another_stream(oracle_mod, precision, npnt):
    torch = torch_cuda()
    import vgb

    nant, nfine, ns, nst = 32, 4, 500, 4
    case = make_case(oracle_mod, nant, npnt, nfine, ns)
    t = {k: dev(case[k]) for k in ("unit", "east", "north", "height", "cable", "D", "B", "freqs", "polQ", "polP", "v_dev")}
    side = torch.cuda.Stream()

    def run(busy):
        S = torch.full((nfine * npnt * nst * ns // 10,), float("nan"), device="cuda")
        out = torch.zeros(npnt * ns // 10 * nst * nfine, dtype=torch.uint8, device="cuda")
        off, scl = (torch.zeros(npnt * nst * nfine, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(400_000_000)
        mb = vgb.Multibeam(1, nfine, nant, npnt, ns, nstokes=nst, precision=precision)
        mb.set_geometry(t["unit"], t["east"], t["north"], t["height"], t["cable"], stream=side)
        mb.set_jones(t["D"], t["B"], t["freqs"], t["polQ"], t["polP"], stream=side)
        mb.run(t["v_dev"], S=S, out=out, offsets=off, scales=scl, stream=side)
        side.synchronize()
        torch.cuda.synchronize()
        mb.close()
        return [host(x) for x in (S, out, off, scl)]

    want = run(False)
    assert not np.isnan(want[0]).any()
    for x, y in zip(run(True), want):
        assert np.array_equal(x, y)
    assert vgb.check_device_status() == 0
