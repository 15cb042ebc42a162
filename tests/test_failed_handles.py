"""Handles whose open failed refuse every call with an error code (both with
and without a GPU): nothing is launched, nothing divides by their zero SMs."""
import ctypes as C

import numpy as np
import pytest


def _u32(n):
    return (C.c_uint32 * n)()


def test_a_pool_that_failed_to_open(lx):
    L = lx.lib()
    p = C.c_void_p()
    assert L.lxmfv_pool_open(C.byref(lx.PoolOptions(0, 0, 0, 100, 0, 0, None)), C.byref(p)) == lx.ERR_ARG
    n, ids = C.c_uint32(), _u32(1)
    d = lx.SearchDesc()
    d.lanes = 32
    scal, _ = lx.seeded_scalars(1, 0, 32)
    sp = scal.ctypes.data_as(C.POINTER(C.c_uint8))
    assert L.lxmfv_pool_submit(p, C.byref(d), sp, ids) != lx.OK
    assert L.lxmfv_pool_submit_many(p, C.byref(d), 1, sp, ids, C.byref(n)) != lx.OK
    assert L.lxmfv_pool_step(p, 1) == lx.ERR_CUDA
    assert L.lxmfv_pool_poll(p, None, 0, C.byref(n)) != lx.OK
    L.lxmfv_pool_close(p)


def test_a_handle_that_failed_to_open(lx):
    L = lx.lib()
    h = C.c_void_p()
    assert L.lxmfv_open(C.byref(lx.Options(0, 64, 7, 0, 0, 0, None)), C.byref(h)) == lx.ERR_ARG
    n = C.c_uint32()
    a = np.ones((4, 8), np.uint32)
    out = np.zeros_like(a)
    ap, op = a.ctypes.data_as(C.POINTER(C.c_uint32)), out.ctypes.data_as(C.POINTER(C.c_uint32))
    scal, _ = lx.seeded_scalars(1, 0, 4)
    sp = scal.ctypes.data_as(C.POINTER(C.c_uint8))
    assert L.lxmfv_collect(h, None, 0, C.byref(n), None, None) == lx.ERR_CUDA
    assert L.lxmfv_init_from_scalars(h, sp, 128) == lx.ERR_STATE
    assert L.lxmfv_first_public_keys(h, sp, 4, _u32(64)) == lx.ERR_STATE
    for op_kind in range(4):
        assert L.lxmfv_fe_op(h, op_kind, ap, ap, op, 4, 2) == lx.ERR_CUDA
    L.lxmfv_close(h)


@pytest.mark.gpu
def test_the_same_beside_a_device(lx):
    test_a_pool_that_failed_to_open(lx)
    test_a_handle_that_failed_to_open(lx)
