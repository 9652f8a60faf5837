"""What mpzmm_matmul_noalloc says when a product does not fit its static
scratch: the figure it names exceeds the limit it names."""
import ctypes as C
import re

import numpy as np
import pytest

from rforest_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,n,limbs", [(180, 1, 180, 1), (300, 3, 300, 1), (8, 8, 8, 4096)])
def test_refusal_names_what_is_exceeded(gpu, m, k, n, limbs):
    import torch
    buf = torch.zeros(8, dtype=torch.int64, device="cuda")  # refused before it is read
    a = [np.zeros(m * k, np.int64), np.full(m * k, limbs, np.int32),
         np.zeros(k * n, np.int64), np.full(k * n, limbs, np.int32),
         np.zeros(m * n, np.int64), np.full(m * n, 1 << 40, np.int64)]
    dev = C.c_void_p(buf.data_ptr())
    i64, i32 = _lib.i64p, _lib.i32p
    with pytest.raises(_lib.MpzmmError) as e:
        _lib.check(_lib.lib().mpzmm_matmul_noalloc(
            m, k, n, dev, a[0].ctypes.data_as(i64), a[1].ctypes.data_as(i32),
            dev, a[2].ctypes.data_as(i64), a[3].ctypes.data_as(i32),
            dev, a[4].ctypes.data_as(i64), a[5].ctypes.data_as(i64), dev,
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    wants, holds = (int(x) for x in re.findall(r"\d{4,}", str(e.value)))
    assert wants > holds
