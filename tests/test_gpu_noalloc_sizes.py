"""ccx_ccd_energy_noalloc over channel tables of every kind its scan meets, against numpy in FP64.
The sum of n products in either order is within n eps sum |t v|; with the pairwise parts of both
sums 1e-14 times log2 n covers it by far, 1e-13 is asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch,hmax,pmax", [
    (1, 1, 1), (1, 8, 32), (1, 9, 33),      # one task, and one beyond it in each direction
    (25, 26, 70), (1024, 5, 9), (1025, 5, 9),  # one chunk of the scan, and one channel more
    (16384, 3, 3), (3, 40, 3000),
])
@pytest.mark.parametrize("shift", [0, 1])
def test_channel_tables(ccx, nch, hmax, pmax, shift):
    torch = pytest.importorskip("torch")
    r = np.random.RandomState(nch + hmax + pmax)
    dims = np.stack([r.randint(0 if nch > 1 else hmax, hmax + 1, nch), r.randint(0 if nch > 1 else pmax, pmax + 1, nch)], 1)
    n = int((dims[:, 0] * dims[:, 1]).sum())
    t, v = (r.standard_normal(2 * n).view(np.complex128) for _ in range(2))
    want, size, at = 0.0, 0.0, 0
    for h, p in dims:
        a, b = t[at:at + h * p].reshape(h, p), v[at:at + h * p].reshape(p, h).T
        want += 0.25 * (a * b).sum()
        size += np.abs(a * b).sum()
        at += h * p

    def device(x):  # shift doubles beyond a 16-byte boundary
        d = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")
        d[shift:shift + 2 * n] = torch.from_numpy(x.view(np.float64).copy())
        return d, d.data_ptr() + 8 * shift

    td, tp = device(t)
    vd, vp = device(v)
    dd = torch.tensor(dims.reshape(-1), dtype=torch.int32, device="cuda")
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    for _ in range(2):
        ccx.ccd_energy_noalloc(nch, dd.data_ptr(), tp, vp, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        got = complex(*out.tolist())
        assert abs(got - want) <= 1e-13 * max(size, 1e-300)
