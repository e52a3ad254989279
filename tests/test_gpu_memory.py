"""Device memory that the library takes from the device's pool, against the
bytes of the arrays that it is for."""
import ctypes as C

import numpy as np
import pytest

import libapr_b200 as A
from tests.helpers import lib_params, volume

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrUsedMemHigh


class Pool:
    """The default memory pool of device 0, which the library allocates from."""

    def __init__(self):
        import torch
        torch.cuda.init()
        self.rt, self.pool = C.CDLL("libcudart.so.12"), C.c_void_p()
        assert self.rt.cudaDeviceGetDefaultMemPool(C.byref(self.pool), 0) == 0

    def get(self, attr):
        import torch
        torch.cuda.synchronize()
        v = C.c_uint64()
        assert self.rt.cudaMemPoolGetAttribute(self.pool, attr, C.byref(v)) == 0
        return v.value


def test_small_aprs_kept_together():
    """APRs of small volumes hold their arrays and at most an eighth more (and
    the pool's 512-byte granules)."""
    pool = Pool()
    conv = A.APRConverter("float")
    conv.par = lib_params()
    imgs = [volume((24, 30 + k % 5, 34 + k % 7), 3 + k % 4, k) for k in range(30)]
    first = A.APR()
    assert conv.get_apr(first, volume((24, 34, 40), 6, 99))  # the converter's own buffers
    before, held, arrays = pool.get(USED_CURRENT), [], 0
    for img in imgs:
        apr = A.APR()
        assert conv.get_apr(apr, img)
        i = apr.info()
        arrays += 2 * int(i.total_number_particles) + 8 * int(i.n_xz)
        held.append(apr)
    used = pool.get(USED_CURRENT) - before
    assert used <= 1.125 * arrays + 1024 * len(held), (used, arrays)
