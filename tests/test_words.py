"""The word-wise byte functions the kernels hash, compare and sum text and
numerics with (xb_hash.h), against their byte-wise and general forms: every
alignment, lengths around the word and mixing steps, every on-disk numeric
form.  They are host functions too, so this needs no GPU."""
import ctypes

import numpy as np
import pytest

import xb_producer as P
import xpu_b200


@pytest.fixture(scope="module")
def L():
    lib = ctypes.CDLL(xpu_b200.LIB_PATH)
    lib.xb_hash_words_of.restype = ctypes.c_uint32
    lib.xb_hash_words_of.argtypes = [ctypes.c_void_p, ctypes.c_uint32]
    lib.xb_words_eq_of.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32]
    lib.xb_numeric_sum_of.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p,
                                      ctypes.c_void_p]
    return lib


def _aligned(n):
    a = np.zeros(n + 64, dtype=np.uint8)
    o = -a.ctypes.data % 64
    return a[o:o + n]


def test_hash_and_equality(L):
    r = np.random.default_rng(3)
    buf, other = _aligned(512), _aligned(512)
    buf[:] = r.integers(0, 256, 512)
    for off in range(8):
        for n in list(range(0, 75)) + [126, 127, 128, 191, 300, 401]:
            p = buf.ctypes.data + off
            want = P.hash_any(buf[off:off + n].tobytes())
            assert L.xb_hash_words_of(p, n) == want, (off, n)
            at = int(r.integers(0, 8))
            other[:] = r.integers(0, 256, 512)              # other bytes around it
            other[at:at + n] = buf[off:off + n]
            q = other.ctypes.data + at
            assert L.xb_words_eq_of(p, q, n) == 1, (off, at, n)
            for k in {0, n // 2, n - 1} if n else ():
                other[at + k] ^= 0x80
                assert L.xb_words_eq_of(p, q, n) == 0, (off, at, n, k)
                other[at + k] ^= 0x80


def _sum(L, p, weight, general):
    kind, lo, hi = ctypes.c_uint8(), ctypes.c_uint64(), ctypes.c_uint64()
    rc = L.xb_numeric_sum_of(p, weight, general, ctypes.byref(kind), ctypes.byref(lo), ctypes.byref(hi))
    return (1,) if rc else (0, kind.value, lo.value, hi.value)


VALUES = [0, 1, -1, 5, 99, 100, 101, 9999, 10000, 10001, 123456, -123456, 99999999, 100000000, 10 ** 12, -10 ** 12,
          10 ** 15 + 7, -(10 ** 16) - 12345, 10 ** 20 + 3, 4 * 10 ** 30]


@pytest.mark.parametrize("scale", [0, 1, 2, 3, 4, 6, 9, 20])
def test_numeric_sum_value(L, scale):
    """every header form, at every alignment, rescaled up and down; special
    and corrupt images too"""
    images = [P.encode_numeric(v, scale, long_fmt=lf, hdr4=h4) for v in VALUES for lf in (0, 1) for h4 in (0, 1)]
    images += [P.encode_varlena(b, h4) for b in (b"\x00\xc0", b"\x00\xd0", b"\x00\xf0", b"\x00\xe0", b"\x00", b"\x00\x81\x01")
               for h4 in (False, True)]
    images += [b"\x01\x12" + b"\0" * 16, b"\x02\x00\x00\x00" + b"\0" * 16]
    buf = _aligned(128)
    r = np.random.default_rng(scale)
    for img in images:
        for off in range(8):
            buf[:] = r.integers(0, 256, 128)
            buf[off:off + len(img)] = np.frombuffer(img, dtype=np.uint8)
            p = buf.ctypes.data + off
            for weight in (-5, -1, 0, 1, 2, 3, 4, 7, 12):
                assert _sum(L, p, weight, 0) == _sum(L, p, weight, 1), (img.hex(), off, weight)
