"""Shared memory of the stem + pool kernel (csrc/stem_pool.cu), called directly: no GPU is involved."""
import ctypes as C

import pytest

from occamy_b200 import runtime as rt


class Layout(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("tiled", "ring", "chunk", "bk", "in_at", "in_row", "slot_bytes", "mr_bytes", "smem")]


def row_bytes(taps, stride_w, Cp, Q):
    """Bytes of a padded input row (a multiple of 8 pixels) whose last window ends inside it."""
    return ((Q - 1) * stride_w + taps + 7) // 8 * 8 * Cp * 2


@pytest.mark.parametrize("may_tile", [True, False])
@pytest.mark.parametrize("Cp,stride_w", [(4, 2), (8, 1)])   # 16 bytes from one column to the next
def test_every_read_stays_in_the_allocation(native_libs, Cp, stride_w, may_tile):
    fn = getattr(C.CDLL(rt.LIB_PATH), "_ZN3occ16stem_pool_layoutEiiiiibPNS_14StemPoolLayoutE")
    fn.restype, fn.argtypes = C.c_bool, [C.c_int] * 5 + [C.c_bool, C.POINTER(Layout)]
    seen = set()
    for Cf in (16, 32, 48, 64):
        for R in range(1, 12):
            for stride_h in range(1, 5):
                for Q in range(1, 129):
                    pitch = row_bytes(Cf // Cp, stride_w, Cp, Q)
                    m = Layout()
                    if not fn(R, Cf, stride_h, Q, pitch, may_tile, m):
                        continue
                    seen.add((m.tiled, m.bk if m.tiled else 0))
                    window = 2 * m.bk if m.tiled else 16           # bytes from one window to the next
                    width = 2 * m.bk if m.tiled else 2 * Cf        # bytes of one
                    # the 128 windows from the start of the ring's last row
                    end = m.in_at + m.ring * m.slot_bytes - m.in_row + 127 * window + width
                    assert end <= m.smem - 1024, (Cf, R, stride_h, Q)
                    assert m.smem <= 227 * 1024
                    assert m.in_row == ((Q + 7) // 8 * 8 * 2 * m.bk if m.tiled else pitch)
                    assert m.slot_bytes == stride_h * m.in_row
                    assert m.in_at >= R * (m.bk if m.tiled else Cf) * 64 * 2
                    # the row maxima, biases and barriers behind the ring
                    assert m.in_at + m.ring * m.slot_bytes + 3 * m.mr_bytes + 256 + 8 * 33 <= m.smem - 1024
                    # rows a convolution row needs at once, and the chunks they lie in
                    groups = (R - 1) // stride_h + 1
                    if groups <= 6:
                        assert (groups + m.chunk - 2) // m.chunk + 1 <= m.ring // m.chunk
    assert seen == ({(1, 16), (1, 32), (1, 64), (0, 0)} if may_tile else {(0, 0)})
