"""sppm_reduce_texture keeps its scratch per CUDA context: the device's memory in use stays the same over
calls that alternate between contexts, between a thread with a context and fresh threads whose first
CUDA call this is, and over contexts that come and go; every call still gives the fold's values."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
R = 64
USED_MEM_CURRENT = 7  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT


@pytest.fixture
def driver():
    cu = C.CDLL("libcuda.so.1")
    assert cu.cuInit(0) == 0
    return cu


def used(cu):
    """Bytes that the allocations of device 0's default pool hold, and the device's free bytes."""
    import torch
    pool, n = C.c_void_p(), C.c_uint64()
    assert cu.cuDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert cu.cuMemPoolGetAttribute(pool, USED_MEM_CURRENT, C.byref(n)) == 0
    torch.cuda.synchronize()
    return n.value, torch.cuda.mem_get_info()[0]


def no_more(before, now):
    """(less is what an object of another test gives back when it is collected)"""
    assert now[0] <= before[0] and now[1] >= before[1], (before, now)


def reduce(ptr, want):
    from glslppm_gb300 import native as N
    out = (C.c_float * 4)()
    assert N.lib.sppm_reduce_texture(ptr, R, 1, out, None) == N.OK, N.last_error()
    assert list(out) == want


def texture():
    t = np.arange(R * R * 4, dtype=np.float32)
    return t, [float(x) for x in t.reshape(-1, 4).max(0)]


def test_fresh_threads(driver):
    torch = pytest.importorskip("torch")
    t, want = texture()
    d = torch.from_numpy(t).cuda()
    torch.cuda.synchronize()
    bad = []

    def fresh():
        try:
            reduce(d.data_ptr(), want)
        except BaseException as e:
            bad.append(e)

    def both():
        reduce(d.data_ptr(), want)
        th = threading.Thread(target=fresh)
        th.start()
        th.join()

    both()
    before = used(driver)
    for _ in range(8):
        both()
    assert not bad, bad
    no_more(before, used(driver))


def test_two_contexts(driver):
    torch = pytest.importorskip("torch")
    t, want = texture()
    d = torch.from_numpy(t).cuda()
    torch.cuda.synchronize()
    first, second, own = C.c_void_p(), C.c_void_p(), C.c_uint64()
    assert driver.cuCtxGetCurrent(C.byref(first)) == 0 and first.value
    assert driver.cuCtxCreate_v2(C.byref(second), 0, 0) == 0  # and makes it current
    try:
        assert driver.cuMemAlloc_v2(C.byref(own), C.c_size_t(t.nbytes)) == 0
        assert driver.cuMemcpyHtoD_v2(own, t.ctypes.data_as(C.c_void_p), C.c_size_t(t.nbytes)) == 0

        def both():
            assert driver.cuCtxSetCurrent(second) == 0
            reduce(own.value, want)
            assert driver.cuCtxSetCurrent(first) == 0
            reduce(d.data_ptr(), want)

        both()
        before = used(driver)
        for _ in range(8):
            both()
        no_more(before, used(driver))
    finally:
        driver.cuCtxDestroy_v2(second)
        assert driver.cuCtxSetCurrent(first) == 0


def test_contexts_that_come_and_go(driver):
    torch = pytest.importorskip("torch")
    t, want = texture()
    reduce(torch.from_numpy(t).cuda().data_ptr(), want)
    first = C.c_void_p()
    assert driver.cuCtxGetCurrent(C.byref(first)) == 0 and first.value

    def one():
        ctx, own = C.c_void_p(), C.c_uint64()
        assert driver.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0
        try:
            assert driver.cuMemAlloc_v2(C.byref(own), C.c_size_t(t.nbytes)) == 0
            assert driver.cuMemcpyHtoD_v2(own, t.ctypes.data_as(C.c_void_p), C.c_size_t(t.nbytes)) == 0
            reduce(own.value, want)
        finally:
            driver.cuCtxDestroy_v2(ctx)
            assert driver.cuCtxSetCurrent(first) == 0

    one()
    before = used(driver)
    for _ in range(6):
        one()
    no_more(before, used(driver))


def test_larger_sizes_replace_the_buffers(driver):
    torch = pytest.importorskip("torch")
    from glslppm_gb300 import renderer
    t = torch.ones((8192, 8192, 4), device="cuda")

    def sizes():
        for n in (64, 8192, 256, 4096, 8192):
            assert renderer.reduce_texture(t.data_ptr(), n, 2).tolist() == [float(n * n)] * 4

    sizes()
    before = used(driver)
    for _ in range(4):
        sizes()
    no_more(before, used(driver))


def test_more_threads_than_buffers():
    """Eight threads at once, four buffers: the others allocate their own."""
    torch = pytest.importorskip("torch")
    bad = []

    def work(seed):
        try:
            stream = torch.cuda.Stream()
            t = np.random.default_rng(seed).permutation(R * R * 4).astype(np.float32)
            with torch.cuda.stream(stream):
                d = torch.from_numpy(t).cuda()
            stream.synchronize()
            from glslppm_gb300 import renderer
            for _ in range(50):
                got = renderer.reduce_texture(d.data_ptr(), R, 1, stream.cuda_stream)
                assert np.array_equal(got, t.reshape(-1, 4).max(0))
        except BaseException as e:
            bad.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(8)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad, bad


def test_a_capturing_stream_keeps_nothing(driver):
    """A stream under capture cannot be waited for: the call fails and holds no memory."""
    torch = pytest.importorskip("torch")
    from glslppm_gb300 import native as N
    t, want = texture()
    d = torch.from_numpy(t).cuda()
    s = torch.cuda.Stream()

    def one():
        reduce(d.data_ptr(), want)
        graph = torch.cuda.CUDAGraph()
        failed = False
        try:
            with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
                out = (C.c_float * 4)()
                failed = N.lib.sppm_reduce_texture(d.data_ptr(), R, 1, out, s.cuda_stream) != N.OK
        except RuntimeError:
            pass  # the capture was invalidated
        assert failed

    one()
    before = used(driver)
    for _ in range(6):
        one()
    no_more(before, used(driver))
