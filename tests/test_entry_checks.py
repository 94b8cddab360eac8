"""What the entry points refuse before they touch a device: no GPU is needed, and none is used where there is one."""
import ctypes as C

import pytest


@pytest.mark.parametrize("elt_bytes", [-1, 0, 3, 6, 16, 32])
@pytest.mark.parametrize("shape,perm", [((2, 3, 5, 8), (2, 1, 0, 3)), ((2, 3, 5, 8), (3, 1, 2, 0)), ((4, 6), (1, 0)), ((7, 4, 6), (0, 2, 1))])
def test_permute_refuses_other_element_sizes(shape, perm, elt_bytes):
    from byteir_b200 import _native as N
    n = len(shape)
    rc = N.lib().b200_permute(elt_bytes, 0x10000, 0x20000, n, (C.c_int64 * n)(*shape), (C.c_int64 * n)(*perm), None)
    assert rc == -2  # B200_ERR_UNSUPPORTED
