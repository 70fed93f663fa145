"""Largest bond component and shortest bond of a neighbour list against
numpy.  The squared length is a fused multiply-add chain: at most two
roundings off numpy's sum, so its root is within 4e-16 of numpy's."""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


@pytest.mark.parametrize("n,width,form", [
    (1, 8, "none"), (9, 8, "none"), (9, 32, "plain"), (257, 16, "plain"),
    (257, 256, "plain"), (20_000, 64, "plain"), (257, 64, "nan"),
    (257, 64, "equal")])
def test_extent(n, width, form):
    import torch
    from probabilistic_peridynamics_gb300._lib import check, lib
    rng = np.random.default_rng(n + width)
    r0 = rng.uniform(-1.0, 1.0, (n, 3))
    nl = rng.integers(-1, n, (n, width)).astype(np.int32)
    own = nl == np.arange(n)[:, None]
    nl[own] = -1
    if form == "none":
        nl[:] = -1
    if form == "nan":
        r0[3, 1] = np.nan
    if form == "equal":
        r0[5] = r0[6]
        nl[5, 0] = 6
    d = r0[nl] - r0[:, None]
    size = np.abs(d)[nl >= 0]
    length = np.sqrt((d[nl >= 0] ** 2).sum(1))
    length = length[~np.isnan(length)]
    want = (np.nanmax(size) if size.size else 0.0,
            length.min() if length.size else 1e300)
    dev = [torch.from_numpy(x).cuda() for x in (nl, r0)]
    out = torch.empty(2, dtype=torch.float64, device="cuda")
    check(lib().pp_bond_extent(
        dev[0].data_ptr(), dev[1].data_ptr(), n, width, out.data_ptr(),
        torch.cuda.current_stream().cuda_stream), "pp_bond_extent")
    got = out.cpu().numpy()
    assert got[0] == want[0]
    assert abs(got[1] - want[1]) <= 4e-16 * want[1]
