"""The bulk host transfers and the snapshots over them, on the CPU: the library's own sources against a stand-in for the CUDA
runtime (fake_cuda.cpp) whose copies can be made to fail."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ternary-bonsai-inference_b200", "csrc")
BK_ERR_OOM, BK_ERR_CUDA = 3, 2
SLOT = 512 << 10


@pytest.fixture(scope="module", params=[[], ["-U__SSE2__"]], ids=["sse2", "portable"])
def fake(request, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "host_transfers.so")
    cuda = next(d for d in ("/usr/local/cuda/include", "/usr/include") if os.path.exists(os.path.join(d, "cuda_runtime.h")))
    subprocess.run(["g++", *request.param, "-std=c++20", "-O1", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-Wno-changes-meaning", "-I", cuda,
                    "-I", os.path.join(ROOT, "include"), "-I", CSRC, os.path.join(ROOT, "tests", "fake_cuda.cpp"),
                    os.path.join(CSRC, "bk_hostpipe.cpp"), os.path.join(CSRC, "bk_snapshot.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    lib.fake_ctx.restype = lib.fake_cache.restype = C.c_void_p
    lib.fake_in_flight.restype = lib.fake_advice.restype = C.c_long
    lib.bk_cache_snapshot_bytes.restype = C.c_size_t
    return lib


@pytest.fixture
def ctx(fake):
    c = C.c_void_p(fake.fake_ctx())
    fake.fake_plan(C.c_long(-1), C.c_long(-1), C.c_long(-1))
    yield c
    fake.fake_plan(C.c_long(-1), C.c_long(-1), C.c_long(-1))
    fake.fake_ctx_free(c)


def plan(fake, copy=-1, sync=-1, alloc=-1):
    fake.fake_plan(C.c_long(copy), C.c_long(sync), C.c_long(alloc))


def transfer(fake, ctx, to_host, host, dev, cuts):
    """Move `dev` to `host` (or back) as the ranges between the cuts."""
    edges = [0, *cuts, host.size]
    sizes = [b - a for a, b in zip(edges, edges[1:])]
    n = len(sizes)
    hp = (C.c_void_p * n)(*(host.ctypes.data + a for a in edges[:-1]))
    dp = (C.c_void_p * n)(*(dev.ctypes.data + a for a in edges[:-1]))
    return fake.fake_transfer(ctx, int(to_host), C.c_size_t(n), hp, dp, (C.c_size_t * n)(*sizes))


@pytest.mark.parametrize("n,cuts", [(1, []), (SLOT - 1, [5]), (SLOT, []), (SLOT + 1, [SLOT]), (17 * SLOT, [1, 3 * SLOT, 3 * SLOT + 7]),
                                    (40 * SLOT + 12345, [100, 70000, 5 * SLOT + 1, 39 * SLOT])])
@pytest.mark.parametrize("pin", [False, True])
def test_transfers_move_every_byte(fake, ctx, n, cuts, pin):
    rng = np.random.default_rng(n)
    dev, host = rng.integers(0, 256, n, dtype=np.uint8), np.zeros(n, np.uint8)
    if pin:
        fake.fake_pin(C.c_void_p(host.ctypes.data), C.c_size_t(n))
    assert transfer(fake, ctx, True, host, dev, cuts) == 0 and fake.fake_in_flight() == 0
    assert np.array_equal(host, dev)
    back = np.zeros(n, np.uint8)
    assert transfer(fake, ctx, False, host, back, cuts) == 0 and fake.fake_in_flight() == 0
    assert np.array_equal(back, dev)


@pytest.mark.parametrize("to_host", [True, False])
@pytest.mark.parametrize("bad", [0, 3, 16, 25, 39])
def test_failed_copy_leaves_nothing_behind(fake, ctx, to_host, bad):
    """The bad-th copy cannot be issued: the call reports it, nothing is in flight when it returns, no byte of an earlier
    transfer turns up in the caller's memory, and the next transfer is whole."""
    n = 40 * SLOT
    old = np.full(n, 0x77, np.uint8)
    assert transfer(fake, ctx, True, np.zeros(n, np.uint8), old, []) == 0  # the slots hold 0x77 now
    rng = np.random.default_rng(bad)
    src, dst = rng.integers(0, 0x70, n, dtype=np.uint8), np.full(n, 0xaa, np.uint8)
    plan(fake, copy=bad)
    host, dev = (dst, src) if to_host else (src, dst)
    assert transfer(fake, ctx, to_host, host, dev, []) == BK_ERR_CUDA
    assert fake.fake_in_flight() == 0
    arrived = dst != 0xaa
    assert np.array_equal(dst[arrived], src[arrived])
    plan(fake)
    assert transfer(fake, ctx, to_host, host, dev, []) == 0 and np.array_equal(dst, src)


@pytest.mark.parametrize("bad", [0, 20])
def test_failed_wait_and_failed_copy_are_reported_once(fake, ctx, bad):
    n = 40 * SLOT
    dev, host = np.random.default_rng(1).integers(0, 256, n, dtype=np.uint8), np.zeros(n, np.uint8)
    plan(fake, copy=30, sync=bad)
    assert transfer(fake, ctx, True, host, dev, []) == BK_ERR_CUDA and fake.fake_in_flight() == 0
    plan(fake)
    assert transfer(fake, ctx, True, host, dev, []) == 0 and np.array_equal(host, dev)


@pytest.mark.parametrize("to_host", [True, False])
def test_failed_copy_of_pinned_memory_leaves_nothing_in_flight(fake, ctx, to_host):
    host, dev = np.zeros(1 << 20, np.uint8), np.ones(1 << 20, np.uint8)
    fake.fake_pin(C.c_void_p(host.ctypes.data), C.c_size_t(host.size))
    plan(fake, copy=2)
    assert transfer(fake, ctx, to_host, host, dev, [1000, 2000, 3000]) == BK_ERR_CUDA
    assert fake.fake_in_flight() == 0


def caches(fake, ctx, n_pos, n_ctx, bits=4):
    """Two caches of the same geometry with other contents; positions per layer of sequence 0."""
    n = (C.c_int * len(n_pos))(*n_pos)
    return [C.c_void_p(fake.fake_cache(ctx, len(n_pos), 2, n_ctx, bits, n, seed)) for seed in (1, 2)]


def save(fake, cache, seq, layout):
    n = fake.bk_cache_snapshot_bytes(cache, seq)
    buf, written = np.zeros(n, np.uint8), C.c_size_t(0)
    assert fake.bk_cache_snapshot_save(cache, seq, layout, C.c_void_p(buf.ctypes.data), C.c_size_t(n), C.byref(written)) == 0 and written.value == n
    return buf


@pytest.mark.parametrize("n_pos", [[7000, 0, 1, 9000, 257, 0], [0, 0], [40000]])
def test_snapshot_of_unequal_layers(fake, ctx, n_pos):
    """Snapshots of up to 20 MB with empty and short layers: the rows come back into another cache, and the row-by-row layout
    that does not use the bulk transfer agrees."""
    a, b = caches(fake, ctx, n_pos, 40000 if len(n_pos) == 1 else 9000)
    blob, rows = save(fake, a, 0, 0), save(fake, a, 0, 1)
    assert fake.bk_cache_snapshot_load(b, 1, C.c_void_p(blob.ctypes.data), C.c_size_t(blob.size)) == 0
    assert [fake.fake_n_pos(b, il, 1) for il in range(len(n_pos))] == n_pos
    assert np.array_equal(save(fake, b, 1, 0), blob) and np.array_equal(save(fake, b, 1, 1), rows)
    assert fake.fake_advice() == 0  # the buffers are the caller's: how they are paged is not the library's business
    for c in (a, b):
        fake.fake_cache_free(c)


def test_snapshot_without_memory_for_its_lists(fake, ctx):
    """Whichever allocation of a save or a load fails, the call says so; no exception passes the C boundary."""
    a, b = caches(fake, ctx, [3000] * 9, 3000)
    for layout in (0, 1):
        blob = save(fake, a, 0, layout)
        for call in (lambda: fake.bk_cache_snapshot_save(a, 0, layout, C.c_void_p(blob.ctypes.data), C.c_size_t(blob.size), None),
                     lambda: fake.bk_cache_snapshot_load(b, 0, C.c_void_p(blob.ctypes.data), C.c_size_t(blob.size))):
            failed = 0
            for k in range(200):
                plan(fake, alloc=k)
                st = call()
                plan(fake)
                assert st in (0, BK_ERR_OOM), (layout, k, st)
                failed += st != 0
                if st == 0:
                    break
            assert st == 0 and failed > 0
    for c in (a, b):
        fake.fake_cache_free(c)


def test_kernels_are_set_up_once_per_device(fake):
    """A kernel's attribute is set once on a device, again after a failure, and with every launch on devices beyond the table, which are not refused."""
    devices = [0, 0, 63, 63, 0, 64, 64, 200]
    failed = (C.c_int * len(devices))()
    assert fake.fake_set_ups((C.c_int * len(devices))(*devices), len(devices), -1, failed) == 5 and not any(failed)
    assert fake.fake_set_ups((C.c_int * len(devices))(*devices), len(devices), 0, failed) == 6 and list(failed) == [1] + [0] * 7
