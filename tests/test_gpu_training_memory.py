"""Training gives the memory of large areas back: what it takes stays in the
stream-ordered pool only up to a bound."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import despeckcl_b200 as dcl  # noqa: E402
from despeckcl_b200 import synthetic  # noqa: E402

RESERVED = 5  # CU_MEMPOOL_ATTR_RESERVED_MEM_CURRENT


# pairs of 1 x 1 patches: 0.07 GiB, 0.5 GiB and (3 x 3 patches) 0.2 GiB
@pytest.mark.parametrize("size,patch", [(78, 1), (128, 1), (300, 3)])
def test_training_leaves_little_in_the_pool(size, patch):
    torch.cuda.synchronize()
    cu = ctypes.CDLL("libcuda.so.1")
    pool = ctypes.c_void_p()
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    assert cu.cuMemPoolTrimTo(pool, ctypes.c_size_t(0)) == 0

    def reserved():
        v = ctypes.c_uint64()
        assert cu.cuMemPoolGetAttribute(pool, RESERVED, ctypes.byref(v)) == 0
        return v.value

    before = reserved()
    st = dcl.nlsar_train_insar(*synthetic.training_area(size, seed=3), [patch], [1])
    assert list(st) == [(patch, 1)] and st[(patch, 1)].dissims_max > st[(patch, 1)].dissims_min
    assert reserved() - before <= (300 << 20)
