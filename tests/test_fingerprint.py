"""The fingerprint that tells whether a constant's host buffer changed (csrc/host/fingerprint.cpp),
called directly: no GPU is involved."""
import ctypes as C

import numpy as np
import pytest

from occamy_b200 import runtime as rt

SIZES = (4, 60, 64, 508, 512, 516, 1020, 1024, 1028, 1087, 1088, 1092, 4096, 17000, 16 * 1024 + 1088, 1 << 20)


@pytest.fixture(scope="module")
def fns():
    lib = C.CDLL(rt.LIB_PATH)
    out = []
    for name in ("_ZN3occ9host_hashEPKvm", "_ZN3occ15host_hash_plainEPKvm"):
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = C.c_uint64, [C.c_void_p, C.c_size_t]
        out.append(fn)
    return out


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("shift", (0, 4, 60))
def test_vector_and_plain_forms_agree(fns, size, shift):
    a = np.random.default_rng(size).integers(0, 256, size + 64, dtype=np.uint8)
    p = a.ctypes.data + shift
    assert fns[0](p, size) == fns[1](p, size)


@pytest.mark.parametrize("size", SIZES)
def test_changes_are_seen(fns, size):
    a = np.random.default_rng(size).integers(0, 256, size, dtype=np.uint8)
    h = fns[0](a.ctypes.data, size)
    assert fns[0](a.ctypes.data, size) == h
    # every byte of the head and the tail counts; up to 17 KB every byte does
    dense = range(size) if size <= 1088 else list(range(512)) + list(range(size - 512, size))
    if 1088 < size <= 17000:
        dense = list(dense) + list(range(512, size - 512, 61))
    for i in dense:
        a[i] ^= 1
        assert fns[0](a.ctypes.data, size) != h, i
        a[i] ^= 1
    if size >= 4096:   # two sampled lines exchanged
        b = a.copy()
        b[:64], b[64:128] = a[64:128].copy(), a[:64].copy()
        c = np.frombuffer(b.tobytes(), np.uint8)
        b2 = a
        b2[:128] = c[:128]
        assert fns[0](b2.ctypes.data, size) != h
