"""Lists of page-locked interaction blocks that end in an error or hold unused channels: the
engine is left as by the same blocks given one by one from pageable memory."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def give(ccx, e, kind, chs, ptrs):
    n = len(chs)
    return ccx.lib().ccx_set_vblocks(e._h, kind, n, (C.c_int32 * n)(*chs), (C.c_void_p * n)(*ptrs))


def test_blocks_before_an_invalid_channel(ccx):
    """[c, c, out of range] after a mixed solve: EINVAL, and the next mixed solve uses the V that
    was given throughout, not digit planes of the old one beside it."""
    torch = pytest.importorskip("torch")
    L = ccx.Layout.from_basis(2, 14, 0.08)
    opts = dict(mode=ccx.MODE_STANDARD, precision=ccx.PREC_MIXED, rebase=ccx.REBASE_DIGITS, tol=1e-9, max_iter=100)
    dims = L.hhpp_dims()
    ch = max(range(len(dims)), key=lambda c: dims[c][0] * dims[c][1])
    energy = []
    for pinned in (False, True):
        e = ccx.Engine(L, real=True)
        e.generate()
        e.setup_t_amplitudes()
        first = e.ccd_iter(**opts)["e_ccd"].real
        flat = np.ascontiguousarray((0.5 * e.vblock(ccx.V_PPPP, ch)).reshape(-1, order="F")).view(np.float64)
        t = torch.empty(flat.size, dtype=torch.float64, pin_memory=pinned)
        t.numpy()[:] = flat
        assert give(ccx, e, ccx.V_PPPP, [ch, ch, 10 ** 6], [t.data_ptr()] * 3) == 1
        e.setup_t_amplitudes()
        energy.append(e.ccd_iter(**opts)["e_ccd"].real)
        assert abs(energy[-1] - first) > 1e-6 * abs(first)
        e.close()
    assert abs(energy[0] - energy[1]) < 1e-11 * abs(energy[0])


def test_unused_hhhh_channel_changes_nothing(ccx):
    """An hhhh channel without an hhpp partner is not stored: the generated family stays the one
    that is read back."""
    torch = pytest.importorskip("torch")
    L = ccx.Layout.from_basis(1, 38, 0.16)
    e = ccx.Engine(L, real=True)
    e.generate()
    qn = [{c: tuple(L.channel(k, c)[0]) for c in range(L.counts()[n])}
          for k, n in ((ccx.CH_HHHH, "hhhh"), (ccx.CH_HHPP, "hhpp"))]
    unused = [c for c, q in qn[0].items() if q not in qn[1].values()]
    assert unused
    want = e.vblock(ccx.CH_HHHH, unused[0])
    t = torch.zeros(2 * want.size, dtype=torch.float64, pin_memory=True)
    assert give(ccx, e, ccx.CH_HHHH, [unused[0]], [t.data_ptr()]) == 0
    assert np.array_equal(e.vblock(ccx.CH_HHHH, unused[0]), want)
    e.close()
