"""Calls on a device that is nearly full: memory that the library uses for speed
(rows padded to whole pieces of 32 columns, blocks kept between adjoint runs) is
given up before a call that needs the room fails."""
import contextlib
import ctypes as C
import gc

import numpy as np
import pytest

from multicomponent_color_gradient_b200 import Solver, _lib, derive

pytestmark = pytest.mark.gpu

MB = 1 << 20
# 97 columns are padded to 128: 0.34 GB of 1.4 GB, far above what the allocator
# rounds (2 MB a buffer, fifteen buffers)
CASE = dict(NX=97, NY=160, NZ=160, boundary="periodic", tau=0.7, sigma=0.01, bubble_radius=20.0,
            NSTATS_START_STEP=10 ** 9)
PADDING = 2 * 216 * 160 * 160 * (128 - 97)


@contextlib.contextmanager
def only_free(bytes_free):
    """All but about `bytes_free` of the device's free memory taken."""
    import torch

    gc.collect()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - int(bytes_free), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del filler
        torch.cuda.empty_cache()


def device_bytes(S):
    out = C.c_uint64()
    S._c("mcg_device_bytes", C.byref(out))
    return out.value


def walk(S):
    S.init_bubble()
    S.step(3)
    return S.get_fields()


def assert_same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def test_create_without_room_for_padded_rows():
    """A handle whose padded rows do not fit is made with the rows as they are,
    and gives the same results."""
    case = derive(CASE)
    with Solver(case) as S:
        padded = device_bytes(S)
        want = walk(S)
    plain = padded - PADDING
    with only_free((plain + padded) // 2):
        with Solver(case) as S:
            assert device_bytes(S) == plain
            got = walk(S)
    assert_same(got, want)
    # the padding it did without is there for the next handle
    with Solver(case) as S:
        assert device_bytes(S) == padded


def test_out_of_memory_does_not_reach_the_next_call():
    """A call that found no memory leaves nothing behind that a later launch
    would report as its own failure."""
    with only_free(64 * MB):
        with pytest.raises(_lib.McgError) as err:
            Solver(derive(CASE))
        assert err.value.status == 2  # MCG_ERR_OOM
        with Solver(derive(dict(CASE, NX=24, NY=20, NZ=20, bubble_radius=5.0))) as S:
            walk(S)
