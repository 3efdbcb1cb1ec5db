"""Shared-memory layout of the response tile kernel (select.cu, tile_kernel) as it is now, restated on the CPU: the
response rows of 80 floats and the NMS rows of 72 fit the planes they alias, every phase reads what an earlier
one wrote, inside its region, and the cell scan's vectors hold the pixels that its ranks stand for."""

import numpy as np

TW, TH = 64, 32
RW, GW, GH = TW + 2, TW + 10, TH + 8
GS, HS, RS, NS = 76, 68, 80, 72
OFF_G = 3 * GH * HS  # floats: three planes of sums, then two gradient planes
THREADS = 256


def test_regions():
    assert (OFF_G + 2 * GH * GS) * 4 == 56960
    assert TH * NS <= GH * HS          # the NMS map in the first plane of sums
    assert (TH + 2) * RS <= 2 * GH * GS  # the response in the gradient planes
    for stride in (GS, HS, RS, NS):
        assert stride * 4 % 16 == 0
    assert OFF_G * 4 % 128 == 0 and GH * GS * 4 % 128 == 0  # TMA targets


def test_horizontal_pass():
    """Three 16-byte loads a plane from column q0: inside the row; the ten columns that the sums use are staged, the
    last two of a row are not and no sum uses them."""
    for q0 in range(0, HS, 4):
        assert q0 + 12 <= GS
        # taps: pairs of columns q0 + j and q0 + j + 2, j = 0..6
        used = {q0 + j + d + e for j in range(7) for d in (0, 2) for e in (0, 1)}
        assert max(used) == q0 + 9 < GW


def test_vertical_pass_and_nms():
    resp, strip = np.zeros((TH + 2, RS), bool), 5
    strips = -(-(TH + 2) // strip)
    assert strips * (RW // 2) <= THREADS
    for tid in range(strips * (RW // 2)):
        s, q = tid // (RW // 2), tid % (RW // 2) * 2
        r0 = min(s * strip, TH + 2 - strip)
        assert r0 + strip + 6 <= GH and q + 1 < HS
        for o in range(s * strip - r0, strip):
            assert not resp[r0 + o, q]
            resp[r0 + o, q:q + 2] = True
    assert resp[:, :RW].all() and not resp[:, RW:].any()
    nms = np.zeros((TH, NS), bool)
    for i in range(TW * TH // 4):
        r, q = i // (TW // 4), i % (TW // 4) * 4
        assert resp[r:r + 3, q:q + 6].all()
        nms[r, q:q + 4] = True
    assert nms[:, :TW].all()


def test_cell_scan():
    """Thread g of a cell takes pixels f = 4 g + (k >> 1) + 32 (k & 1) in this order from two 16-byte loads."""
    for tid in range(THREADS):
        cc, g = tid >> 3, tid & 7
        ccx, ccy = cc & 7, cc >> 3
        base = (ccy * 8 + (g >> 1)) * NS + ccx * 8 + 4 * (g & 1)
        assert base % 4 == 0 and (base + 4 * NS) % 4 == 0
        loads = [base + d for d in range(4)], [base + 4 * NS + d for d in range(4)]
        vals = [loads[k & 1][k >> 1] for k in range(8)]
        for k in range(8):
            f = 4 * g + (k >> 1) + 32 * (k & 1)
            assert vals[k] == (ccy * 8 + (f >> 3)) * NS + ccx * 8 + (f & 7)
            assert vals[k] < TH * NS and vals[k] % NS < TW


def test_sub_tile_sums():
    """Each lane's eight values lie in the response's core; after the three halving stages lane k < 8 holds value k,
    joined from the partial sums that a butterfly over the lanes joins."""
    for wid in range(8):
        for lane in range(32):
            for s8 in range(8):
                row, col = (s8 >> 2) * 16 + 2 * wid + (lane >> 4) + 1, (s8 & 3) * 16 + (lane & 15) + 1
                assert 1 <= row <= TH and 1 <= col <= TW
    # a partial sum as a nested pair of the lanes it joins (sums commute: as sets)
    v = [[frozenset([(lane, k)]) for k in range(8)] for lane in range(32)]
    for st in range(3):
        new = [row[:] for row in v]
        for lane in range(32):
            up, other = (lane >> st) & 1, lane ^ (1 << st)
            for k in range(4 >> st):
                keep = v[lane][2 * k + 1] if up else v[lane][2 * k]
                sent = v[other][2 * k] if (other >> st) & 1 else v[other][2 * k + 1]
                new[lane][k] = frozenset([keep, sent])
        v = new
    b = [[frozenset([(lane, k)]) for lane in range(32)] for k in range(8)]
    for st in range(3):
        b = [[frozenset([row[lane], row[lane ^ (1 << st)]]) for lane in range(32)] for row in b]
    for lane in range(32):
        assert v[lane][0] == b[lane & 7][lane]
