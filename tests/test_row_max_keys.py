"""Host models of the integer identities of the 16x2 cells (gotoh.cu): a row
maximum's key H * S + S - 1 - t, whose largest is the largest score's least column
block t; its score by a product instead of a division; and the opened-gap flags of two
states by one exclusive or."""
import numpy as np


def test_score_of_a_key():
    keys = np.arange(1 << 16, dtype=np.uint64)
    sizes = sorted({4 * k for k in range(1, 700)} | {1 << k for k in range(2, 17)} | {65532, 43692, 21848})
    for s in sizes:
        inv = np.uint64((0xFFFFFFFF // s + 1) & 0xFFFFFFFF)
        assert ((keys * inv) >> np.uint64(32) == keys // np.uint64(s)).all(), s


def test_key_order():
    for s in (4, 8, 64, 1024):
        h, t = (a.ravel() for a in np.meshgrid(np.arange(65536 // s), np.arange(s)))
        key = h * s + s - 1 - t
        assert key.max() < 1 << 16 and len(np.unique(key)) == len(key)
        order = np.argsort(-key)  # larger scores first, then smaller column blocks
        assert (order == np.lexsort((t, -h))).all()
        base = key // s * s
        assert (base + s - 1 - key == t).all()


def test_opened_flags():
    for e in range(-64, 64, 4):
        for f in range(-64, 64, 4):
            for a in (0, 1):
                for b in (0, 2):
                    assert ((e + a) ^ (f + b)) & 3 == a + b
