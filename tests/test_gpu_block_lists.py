"""Whole families of blocks in one launch: interaction blocks in page-locked memory, and the
amplitudes unpacked for all channels, against the single-block calls, bit for bit (copies)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pinned_copy(torch, a, shift):
    """A block in page-locked memory, shift doubles beyond a 16-byte boundary."""
    flat = np.ascontiguousarray(a.reshape(-1, order="F")).view(np.float64)
    t = torch.empty(flat.size + 2, dtype=torch.float64, pin_memory=True)
    t.numpy()[shift:shift + flat.size] = flat
    return t, t.data_ptr() + 8 * shift


@pytest.mark.parametrize("nmax,A,snm,real", [(1, 2, False, True), (2, 14, False, True), (2, 28, True, False)])
@pytest.mark.parametrize("shift", [0, 1])
def test_families_in_one_launch(ccx, nmax, A, snm, real, shift):
    torch = pytest.importorskip("torch")
    L = ccx.Layout.from_basis(nmax, A, 0.16, snm=snm)
    src = ccx.Engine(L, real=real)
    src.generate(potential=ccx.POT_MINNESOTA if real else ccx.POT_CHIRAL_LIKE)
    src.setup_t_amplitudes()
    c = L.counts()
    a, b = ccx.Engine(L, real=real), ccx.Engine(L, real=real)
    for e in (a, b):
        e.set_fock(src.fock(), src.e0())
    keep = []
    for kind, n in ((ccx.CH_HHPP, c["hhpp"]), (ccx.V_PPPP, c["hhpp"]), (ccx.CH_HHHH, c["hhhh"]), (ccx.CH_HPHP, c["hphp"])):
        blocks = [src.vblock(kind, ch) for ch in range(n)]
        for ch, x in enumerate(blocks):
            a.set_vblock(kind, ch, x)
        # every channel, the first one twice: the last block given counts
        chs = [0] + list(range(n))
        bufs = [pinned_copy(torch, 2.0 * blocks[0], shift)] + [pinned_copy(torch, x, shift) for x in blocks]
        keep += bufs
        ccx._check(ccx.lib().ccx_set_vblocks(b._h, kind, len(chs), (C.c_int32 * len(chs))(*chs),
                                             (C.c_void_p * len(chs))(*[p for _, p in bufs])))
    for e in (a, b):
        e.setup_t_amplitudes()
        e.t2_intermediate()
    for ch in range(c["hhpp"]):
        assert np.array_equal(a.t2(ch), b.t2(ch)) and np.array_equal(a.t2_eqn(ch), b.t2_eqn(ch)), ch
    want = np.concatenate([b.t2(ch).reshape(-1, order="F") for ch in range(c["hhpp"])])
    assert np.array_equal(b.t2_all(), want)
    t, ptr = pinned_copy(torch, np.zeros(c["amps"], np.complex128), shift)
    ccx._check(ccx.lib().ccx_get_t2_all(b._h, C.c_void_p(ptr)))
    assert np.array_equal(t.numpy()[shift:shift + 2 * c["amps"]].view(np.complex128), want)
