"""The library's host code over a CUDA runtime without a device
(fake_cudart.c, linked with the library's own objects): what an allocation
that fails leaves open, and what stays behind in device memory.  No GPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def fake(lx, tmp_path_factory):
    import build as lxbuild

    lxbuild.build()
    so = str(tmp_path_factory.mktemp("fake") / "liblxmfv_fake.so")
    objs = [os.path.join(lxbuild.OBJ, s + ".o") for s in lxbuild.CU_SOURCES + lxbuild.CXX_SOURCES]
    obj = so + ".o"
    subprocess.run(["gcc", "-O1", "-fPIC", "-I", CUDA_INCLUDE, "-c", os.path.join(HERE, "fake_cudart.c"), "-o", obj], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, obj] + objs + ["-lcrypto"], check=True)
    L = C.CDLL(so)
    for name in ("fake_used",):
        getattr(L, name).restype = C.c_size_t
    L.fake_set_capacity.argtypes = [C.c_size_t]
    L.fake_holds.argtypes = [C.c_char_p, C.c_size_t]
    L.lxmfv_pool_keys_per_lane.restype = C.c_uint64
    for name in ("lxmfv_close", "lxmfv_pool_close"):
        getattr(L, name).restype = None
    L.fake_reset()
    yield L
    L.fake_reset()


def _u8(a):
    return a.ctypes.data_as(C.POINTER(C.c_uint8))


def _u32(a):
    return a.ctypes.data_as(C.POINTER(C.c_uint32))


def _handle_calls(lx, L, h, lanes):
    """Every entry point that works on a handle, with arguments that an open
    one accepts."""
    scal, _ = lx.seeded_scalars(3, 0, lanes)
    words = np.ones((lanes, 16), np.uint32)
    a, out = np.ones((64, 8), np.uint32), np.zeros((64, 8), np.uint32)
    pks, addr = np.zeros((64, 64), np.uint8), np.zeros((64, 16), np.uint8)
    args = lx.make_launch_args(1, bytes(32), lx.prefix_parse("b0"))
    n, d = C.c_uint32(), C.c_double()
    nh = (C.c_uint8 * 10)()
    yield "init", lambda: L.lxmfv_init(h, _u32(words), C.c_size_t(words.size))
    yield "init_from_scalars", lambda: L.lxmfv_init_from_scalars(h, _u8(scal), C.c_size_t(32 * lanes))
    yield "first_public_keys", lambda: L.lxmfv_first_public_keys(h, _u8(scal), C.c_size_t(lanes), _u32(words))
    yield "launch_async", lambda: L.lxmfv_launch_async(h, C.byref(args))
    yield "collect", lambda: L.lxmfv_collect(h, None, 0, C.byref(n), None, None)
    yield "launch", lambda: L.lxmfv_launch(h, C.byref(args), None, 0, C.byref(n), None, None)
    for op in range(4):
        yield f"fe_op {op}", lambda op=op: L.lxmfv_fe_op(h, op, _u32(a), _u32(a), _u32(out), C.c_uint64(64), 8)
    yield "address_chain", lambda: L.lxmfv_address_chain(h, _u8(pks), nh, _u8(addr), C.c_uint64(64))
    yield "peak_probe", lambda: L.lxmfv_peak_probe(h, 0, C.c_float(1.0), C.byref(d))


@pytest.mark.parametrize("walk,batch", [(0, 64), (0, 1024), (1, 64)])
def test_a_handle_whose_open_failed_at_any_allocation(lx, fake, walk, batch):
    """Every allocation of lxmfv_open fails in turn: open says so, every call
    on the handle is refused before any launch, and close leaves nothing."""
    lanes = 96
    for at in range(64):
        fake.fake_reset()
        fake.fake_fail_after(at)
        h = C.c_void_p()
        rc = fake.lxmfv_open(C.byref(lx.Options(0, lanes, batch, 0, walk, 0, None)), C.byref(h))
        if fake.fake_pending():  # open made fewer allocations than that
            assert rc == lx.OK
            fake.fake_reset()
            for name, call in _handle_calls(lx, fake, h, lanes):
                assert call() == lx.OK, name
            fake.lxmfv_close(h)
            assert fake.fake_used() == 0
            break
        assert rc == lx.ERR_CUDA, at
        before = fake.fake_launches()
        for name, call in _handle_calls(lx, fake, h, lanes):
            assert call() != lx.OK, (at, name)
            assert fake.fake_launches() == before, (at, name)
        fake.lxmfv_close(h)
        assert fake.fake_used() == 0, at
    else:
        pytest.fail("open never succeeded")
    assert at > 5


def test_a_handle_refused_before_its_device_is_known(lx, fake):
    """As above for options that lxmfv_open refuses."""
    fake.fake_reset()
    h = C.c_void_p()
    assert fake.lxmfv_open(C.byref(lx.Options(0, 96, 7, 0, 0, 0, None)), C.byref(h)) == lx.ERR_ARG
    for name, call in _handle_calls(lx, fake, h, 96):
        assert call() != lx.OK, name
    assert fake.fake_launches() == 0
    fake.lxmfv_close(h)
    assert fake.fake_used() == 0


def _pool_calls(lx, L, p):
    scal, _ = lx.seeded_scalars(4, 0, 64)
    d = lx.SearchDesc()
    d.lanes = 64
    ids, n = (C.c_uint32 * 1)(), C.c_uint32()
    yield "submit", lambda: L.lxmfv_pool_submit(p, C.byref(d), _u8(scal), ids)
    yield "step", lambda: L.lxmfv_pool_step(p, 1)
    yield "poll", lambda: L.lxmfv_pool_poll(p, None, 0, C.byref(n))
    yield "retire", lambda: L.lxmfv_pool_retire(p, 0)
    yield "submit_many", lambda: L.lxmfv_pool_submit_many(p, C.byref(d), 1, _u8(scal), ids, C.byref(n))


@pytest.mark.parametrize("batch", [64, 1024])
def test_a_pool_whose_open_failed_at_any_allocation(lx, fake, batch):
    for at in range(64):
        fake.fake_reset()
        fake.fake_fail_after(at)
        p = C.c_void_p()
        rc = fake.lxmfv_pool_open(C.byref(lx.PoolOptions(0, 256, 0, batch, 8, 0, None)), C.byref(p))
        if fake.fake_pending():
            assert rc == lx.OK
            fake.fake_reset()
            for name, call in _pool_calls(lx, fake, p):
                assert call() == lx.OK, name
            fake.lxmfv_pool_close(p)
            assert fake.fake_used() == 0
            break
        assert rc == lx.ERR_CUDA, at
        before = fake.fake_launches()
        assert fake.lxmfv_pool_keys_per_lane(p, 0) == 0, at
        for name, call in _pool_calls(lx, fake, p):
            assert call() != lx.OK, (at, name)
            assert fake.fake_launches() == before, (at, name)
        fake.lxmfv_pool_close(p)
        assert fake.fake_used() == 0, at
    else:
        pytest.fail("open never succeeded")
    assert at > 9


def test_start_scalars_leave_device_memory(lx, fake):
    """Start scalars are private keys: no copy of them stays in the handle's
    device memory after the call that used them."""
    fake.fake_reset()
    lanes = 96
    for walk in (0, 1):
        h = C.c_void_p()
        assert fake.lxmfv_open(C.byref(lx.Options(0, lanes, 64, 0, walk, 0, None)), C.byref(h)) == lx.OK
        scal, _ = lx.seeded_scalars(5 + walk, 0, lanes)
        out = np.zeros((lanes, 16), np.uint32)
        for call in (lambda: fake.lxmfv_init_from_scalars(h, _u8(scal), C.c_size_t(32 * lanes)),
                     lambda: fake.lxmfv_first_public_keys(h, _u8(scal), C.c_size_t(lanes), _u32(out))):
            assert call() == lx.OK
            for t in range(lanes):
                assert not fake.fake_holds(bytes(scal[t]), 32), t
        fake.lxmfv_close(h)


def test_kept_buffers_are_given_back_when_memory_is_short(lx, fake):
    """What a handle keeps for its array calls never stands in the way of an
    allocation: of a dump, of hit slots, of a larger array call.  A call that
    runs out of memory all the same fails alone."""
    lanes, rows = 96, 1 << 18
    nh = (C.c_uint8 * 10)()
    big_rows = 2 * rows  # 40 MiB
    pks, addr = np.zeros((big_rows, 64), np.uint8), np.zeros((big_rows, 16), np.uint8)
    n = C.c_uint32()

    def chain(h, count):
        return fake.lxmfv_address_chain(h, _u8(pks), nh, _u8(addr), C.c_uint64(count))

    def launch(h, **kw):
        args = lx.make_launch_args(64, bytes(32), lx.prefix_parse("b0"), **kw)
        return fake.lxmfv_launch(h, C.byref(args), None, 0, C.byref(n), None, None)

    for what in ("dump", "hits", "array"):
        fake.fake_reset()
        h = C.c_void_p()
        assert fake.lxmfv_open(C.byref(lx.Options(0, lanes, 1024, 0, 0, 0, None)), C.byref(h)) == lx.OK
        opened = fake.fake_used()
        scal, _ = lx.seeded_scalars(6, 0, lanes)
        assert fake.lxmfv_init_from_scalars(h, _u8(scal), C.c_size_t(32 * lanes)) == lx.OK
        assert chain(h, rows) == lx.OK
        assert fake.fake_used() >= opened + 80 * rows  # kept
        fake.fake_set_capacity(opened + 41 * (1 << 20))  # room for what comes next, but not beside the kept buffer
        if what == "dump":
            assert launch(h, dump_threads=8, dump_keys=1 << 16) == lx.OK  # 24 MiB
        elif what == "hits":
            assert launch(h, max_hits=3 << 19) == lx.OK  # 24 MiB
        else:
            assert chain(h, big_rows) == lx.OK
        fake.fake_set_capacity(0)
        assert launch(h, max_hits=1 << 28) == lx.ERR_CUDA
        assert launch(h) == lx.OK
        fake.lxmfv_close(h)
        assert fake.fake_used() == 0
