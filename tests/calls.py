"""One inference by direct calls of the runtime's ABI, for tests that need a sequence no graph of
``occamy_b200.graphs`` gives: an unusual order of uploads, a stop in the middle, tensors outside the pool."""
import ctypes as C

import numpy as np

from occamy_b200 import runtime as rt


class Inference:
    """``with Inference(pool_bytes) as f:`` -- the handle and the pool of one inference; tensors are placed one
    after the other (``at`` puts one at an offset of its own)."""

    def __init__(self, pool_bytes=1 << 22):
        self.L, self.bytes = rt.lib(), pool_bytes

    def __enter__(self):
        self.h, self.pool, self.at = C.c_void_p(), C.c_void_p(), 0
        self.L.cudnnCreate(C.byref(self.h))
        self.L.wrapDNNMemPoolInit(C.byref(self.pool), self.bytes)
        return self

    def __exit__(self, *_):
        self.L.wrapDNNDealloc(self.pool)
        self.L.cudnnDestroy(self.h)

    def place(self, nbytes, at=None):
        p = C.c_void_p()
        if at is None:
            at, self.at = self.at, self.at + (nbytes + 31) // 32 * 32
        self.L.wrapDNNMemOffset(C.byref(p), self.pool, at, nbytes)
        return p.value

    def put(self, a, at=None):
        """A host array into a tensor of its own (a constant, or a batch)."""
        p = self.place(a.nbytes, at)
        self.L.wrapDNNMemcpy(p, a.ctypes.data, a.nbytes, 1, None)
        return p

    def copy(self, ptr, nbytes, at=None):
        """Device memory into a tensor of its own."""
        p = self.place(nbytes, at)
        self.L.wrapDNNMemcpy(p, ptr, nbytes, 3, None)
        return p

    def get(self, p, shape):
        out = np.empty(shape, np.float32)
        self.L.wrapDNNMemcpy(out.ctypes.data, p, out.nbytes, 2, None)
        return out

    def conv(self, x, xs, w, ws, b=None, pads=(0, 0), strides=(1, 1), groups=1, act=None, y=None, at=None):
        """Convolution; with `act` the fused call (0 sigmoid, 1 ReLU, 2 tanh, 5 none)."""
        o = (xs[0], ws[0]) + tuple((xs[2 + i] + 2 * pads[i] - ws[2 + i]) // strides[i] + 1 for i in (0, 1))
        if y is None:
            y = self.place(int(np.prod(o)) * 4, at)
        d = rt.dims
        if act is None:
            self.L.DNNConvFunc(self.h, x, d(xs), w, d(ws), None, 0, 0, groups, d(pads), d(strides), y)
        else:
            self.L.DNNConvBiasActivFunc(self.h, x, d(xs), w, d(ws), b, d((1, ws[0], 1, 1)), None, 0, 0, d(pads),
                                        d(strides), act, y)
        return y, o

    def clip(self, x, xs, lo, hi):
        y = self.place(int(np.prod(xs)) * 4)
        self.L.CUDAClipFunc(x, y, rt.dims(xs), lo, hi, len(xs))
        return y

    def relu(self, x, xs):
        y = self.place(int(np.prod(xs)) * 4)
        self.L.DNNActiveFunc(self.h, x, rt.dims(xs), 1, y)
        return y

    def op(self, mode, a, as_, b, bs, y=None):
        """Element-wise: 0 a + b, 1 a * b."""
        if y is None:
            y = self.place(int(np.prod(as_)) * 4)
        self.L.DNNTensorOpFunc(self.h, mode, a, rt.dims(as_), len(as_), b, rt.dims(bs), len(bs), y, rt.dims(as_),
                               len(as_), 1.0)
        return y

    def matmul(self, a, as_, b, bs, trans_b=1):
        n = bs[0] if trans_b else bs[1]
        y = self.place(as_[0] * n * 4)
        d = rt.dims
        self.L.CUBLASMatmul2dFunc(2, a, d(as_), b, d(bs), y, d((as_[0], n)), y, d((as_[0], n)), 1.0, 0.0, 0, trans_b)
        return y, (as_[0], n)


def rand(seed, *shape, scale=1.0):
    return (np.random.default_rng(seed).standard_normal(shape) * scale).astype(np.float32)
