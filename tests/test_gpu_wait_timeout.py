"""A bounded device wait that runs out: the kernel returns, the host is told, the context stays usable.

The context-split exchange waits for the other ranks' rows with a poll limit.  Here two ranks are
played by ONE process on ONE GPU (two contexts; mailboxes of the same process are opened directly),
and they never run at the same time: first rank 0 calls alone - nothing ever sets the arrival words
it waits for, so its wait gives up after the (shortened) limit, the output is zeros and the next
synchronising call reports BK_ERR_CUDA; a second lone call fails the same way (the error word was
re-armed).  Then rank 1 calls alone (it sends its rows, then gives up waiting for rank 0's), and
finally rank 0 calls again with the same sequence number: rank 1's rows are there, the wait is
satisfied at once and the merged output equals the whole-cache attention.  No kernel traps, faults
or spins without a limit, and no two kernels that wait for one another are ever in flight together.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NH, NKV, HD = 24, 4, 256


def _mailbox(ctx, world, rank):
    handle = (C.c_ubyte * 64)()
    mb = C.c_void_p()
    ctx.check(ctx.lib.bk_mailbox_create(ctx.h, world, rank, NH, HD, C.byref(mb), handle))
    return mb, bytes(handle)


def test_exchange_wait_gives_up_reports_and_recovers(bk, monkeypatch):
    monkeypatch.setenv("BONSAI_KV_XCH_POLLS", "3000")     # a few milliseconds instead of about a second
    abi = bk._abi
    ctx = [bk.Context(0), bk.Context(0)]
    lib = ctx[0].lib
    rng = np.random.default_rng(17)
    n = [2500, 700]                                        # rank 0: tensor-core kernel, rank 1: generic kernel
    total = sum(n)
    k = rng.standard_normal((total, NKV, HD), dtype=np.float32)
    v = rng.standard_normal((total, NKV, HD), dtype=np.float32)
    k[:, :, [7, 70, 170]] *= np.float32(20.0)
    v[:, :, [7, 70, 170]] *= np.float32(20.0)
    q = rng.standard_normal((NH, HD), dtype=np.float32)
    mode = bk.parse_mode("planar4")
    part = [bk.AttnCache(ctx[r], mode, n_layers=1, n_ctx=n[r], rope_positions=total) for r in range(2)]
    part[0].append(0, k[:n[0]], v[:n[0]], pos=0)
    part[1].append(0, k[n[0]:], v[n[0]:], pos=n[0])
    whole = bk.AttnCache(ctx[0], mode, n_layers=1, n_ctx=total)
    whole.append(0, k, v)
    want = whole.attend(0, q)[0]

    boxes = [_mailbox(ctx[r], 2, r) for r in range(2)]
    blob = (C.c_ubyte * 128).from_buffer_copy(boxes[0][1] + boxes[1][1])
    for r in range(2):
        ctx[r].check(lib.bk_mailbox_open_peers(boxes[r][0], blob))
    d_q = [ctx[r].to_device(q) for r in range(2)]
    d_out = [ctx[r].alloc(NH * HD * 4) for r in range(2)]

    def call(r, seqno):
        ctx[r].check(lib.bk_decode_attn_split(part[r].h, 0, 0, n[r], total - 1, d_q[r].ptr, d_out[r].ptr, boxes[r][0], seqno))
        return lib.bk_synchronize(ctx[r].h)

    for seqno in (1, 2):                                   # rank 0 alone: the wait runs out, twice
        d_out[0].upload(np.ones((NH, HD), np.float32))
        assert call(0, seqno) == abi.BK_ERR_CUDA
        msg = lib.bk_last_error(ctx[0].h)
        assert b"bounded wait" in msg and b"code 3" in msg, msg
        assert lib.bk_synchronize(ctx[0].h) == abi.BK_OK   # reported once, then clear
        assert np.all(d_out[0].download((NH, HD), np.float32) == 0.0)
    assert call(1, 3) == abi.BK_ERR_CUDA                   # rank 1 alone: sends, then gives up on rank 0
    assert call(0, 3) == abi.BK_OK                         # rank 0 again: everything it waits for is there
    got = d_out[0].download((NH, HD), np.float32)
    err = float(np.max(np.abs(got - want)))
    assert err <= 5e-4, err   # two GPU results over different splits, each about 1e-4 from the oracle
    # the ordinary path still works on the context that saw the time-outs
    again = part[0].attend(0, q, q_pos=[total - 1])[0]
    assert np.isfinite(again).all()
    for r in range(2):
        lib.bk_mailbox_destroy(boxes[r][0])
    for c in part + [whole]:
        c.close()
    for c in ctx:
        c.close()


def test_exchange_of_several_layers_rows_in_one_call(bk, monkeypatch):
    """bk_exchange_merge: the partial rows of two layers (48 rows, a mailbox with more arrival words than the
    per-layer one) cross in one call per rank and merge to the whole-cache attention.  The two ranks are played
    by one process and never run together: rank 1 sends and gives up waiting (reported), then rank 0 finds
    everything it waits for."""
    monkeypatch.setenv("BONSAI_KV_XCH_POLLS", "3000")
    abi = bk._abi
    ctx = [bk.Context(0), bk.Context(0)]
    lib = ctx[0].lib
    rng = np.random.default_rng(23)
    n_layers, n = 2, [2300, 900]
    total = sum(n)
    k = rng.standard_normal((n_layers, total, NKV, HD), dtype=np.float32)
    v = rng.standard_normal((n_layers, total, NKV, HD), dtype=np.float32)
    q = rng.standard_normal((n_layers, NH, HD), dtype=np.float32)
    mode = bk.parse_mode("planar4")
    part = [bk.AttnCache(ctx[r], mode, n_layers=n_layers, n_ctx=n[r], rope_positions=total) for r in range(2)]
    whole = bk.AttnCache(ctx[0], mode, n_layers=n_layers, n_ctx=total)
    for il in range(n_layers):
        part[0].append(il, k[il, :n[0]], v[il, :n[0]], pos=0)
        part[1].append(il, k[il, n[0]:], v[il, n[0]:], pos=n[0])
        whole.append(il, k[il], v[il])
    want = np.stack([whole.attend(il, q[il])[0] for il in range(n_layers)])

    boxes = []
    for r in range(2):
        handle = (C.c_ubyte * 64)()
        mb = C.c_void_p()
        ctx[r].check(lib.bk_mailbox_create(ctx[r].h, 2, r, n_layers * NH, HD, C.byref(mb), handle))
        boxes.append((mb, bytes(handle)))
    blob = (C.c_ubyte * 128).from_buffer_copy(boxes[0][1] + boxes[1][1])
    for r in range(2):
        ctx[r].check(lib.bk_mailbox_open_peers(boxes[r][0], blob))
    d_q = [ctx[r].to_device(q) for r in range(2)]
    d_part = [ctx[r].alloc(n_layers * NH * (HD + 2) * 4) for r in range(2)]
    d_out = [ctx[r].alloc(n_layers * NH * HD * 4) for r in range(2)]

    def call(r, seqno):
        for il in range(n_layers):
            part[r].decode_device(il, d_q[r].ptr + il * NH * HD * 4, d_part[r].ptr + il * NH * (HD + 2) * 4,
                                  q_pos=[total - 1], partial=True)
        ctx[r].check(lib.bk_exchange_merge(boxes[r][0], NH // NKV, d_part[r].ptr, d_out[r].ptr, seqno))
        return lib.bk_synchronize(ctx[r].h)

    assert call(1, 1) == abi.BK_ERR_CUDA                   # rank 1 alone: sends its 48 rows, gives up on rank 0
    assert call(0, 1) == abi.BK_OK                         # rank 0: rank 1's rows are there
    got = d_out[0].download((n_layers, NH, HD), np.float32)
    err = float(np.max(np.abs(got - want)))
    assert err <= 5e-4, err
    # bad arguments are refused
    assert lib.bk_exchange_merge(boxes[0][0], 5, d_part[0].ptr, d_out[0].ptr, 2) == abi.BK_ERR_INVALID   # 48 % 5 != 0
    assert lib.bk_exchange_merge(boxes[0][0], NH // NKV, d_part[0].ptr, d_out[0].ptr, 0) == abi.BK_ERR_INVALID
    for r in range(2):
        lib.bk_mailbox_destroy(boxes[r][0])
    for c in part + [whole]:
        c.close()


def test_exchange_of_slices(bk, monkeypatch):
    """The same with the slice form of the split-K combine in rank 0's launches (next to another context they take the
    last-arriver form unless told that the two never run together)."""
    monkeypatch.setenv("BONSAI_KV_DIST", "1")
    test_exchange_wait_gives_up_reports_and_recovers(bk, monkeypatch)


def test_exchange_of_more_chunks_than_one_round(bk, oracle, monkeypatch):
    """A rank whose slices come from as many chunks as SMs (one kv head, 32 rows each), more than a thread of the slice combine takes
    in one round when slices lie on the mailbox's grid of eight coordinates."""
    monkeypatch.setenv("BONSAI_KV_XCH_POLLS", "3000")
    monkeypatch.setenv("BONSAI_KV_DIST", "1")
    from oracle_lib import MODE_F16
    abi = bk._abi
    ctx = [bk.Context(0), bk.Context(0)]
    lib = ctx[0].lib
    rng = np.random.default_rng(37)
    n = [4731, 700]
    total = sum(n)
    k, v = (rng.standard_normal((total, 1, HD), dtype=np.float32) for _ in range(2))
    q = rng.standard_normal((6, HD), dtype=np.float32)
    ref = oracle.cache(MODE_F16, 0, False, n_head=6, n_kv=1)
    for p in range(total):
        ref.append(0, k[p], v[p], p)
    want = ref.attend(0, q, total - 1, total, threads=8)
    part = [bk.AttnCache(ctx[r], bk.parse_mode("f16"), n_layers=1, n_ctx=n[r], n_head=6, n_kv=1, rope_positions=total) for r in range(2)]
    part[0].append(0, k[:n[0]], v[:n[0]], pos=0)
    part[1].append(0, k[n[0]:], v[n[0]:], pos=n[0])
    boxes = []
    for r in range(2):
        handle = (C.c_ubyte * 64)()
        mb = C.c_void_p()
        ctx[r].check(lib.bk_mailbox_create(ctx[r].h, 2, r, 6, HD, C.byref(mb), handle))
        boxes.append((mb, bytes(handle)))
    blob = (C.c_ubyte * 128).from_buffer_copy(boxes[0][1] + boxes[1][1])
    for r in range(2):
        ctx[r].check(lib.bk_mailbox_open_peers(boxes[r][0], blob))
    d_q = [ctx[r].to_device(q) for r in range(2)]
    d_out = [ctx[r].alloc(q.nbytes) for r in range(2)]

    def call(r):
        ctx[r].check(lib.bk_decode_attn_split(part[r].h, 0, 0, n[r], total - 1, d_q[r].ptr, d_out[r].ptr, boxes[r][0], 1))
        return lib.bk_synchronize(ctx[r].h)

    assert call(1) == abi.BK_ERR_CUDA                      # rank 1 alone: sends, then gives up on rank 0
    assert call(0) == abi.BK_OK
    got = d_out[0].download(q.shape, np.float32)
    assert float(np.max(np.abs(got - want))) <= 1e-5
    for r in range(2):
        lib.bk_mailbox_destroy(boxes[r][0])
    for c in part:
        c.close()
    for c in ctx:
        c.close()


@pytest.mark.parametrize("tag", ["f16", "planar4"])
def test_combine_wait_gives_up_and_nothing_stale_is_handed_out(bk, monkeypatch, tag):
    """The wait of the split-K combine runs out (a limit of no polls, read when a cache is made): the error is reported once;
    launches that were already queued behind it, with the ordinary limit, neither take the words that it left behind as
    results nor write anything; after the report the same launches give what a context that saw no error gives."""
    monkeypatch.setenv("BONSAI_KV_DIST", "1")   # (whatever other contexts the session holds)
    abi = bk._abi
    rng = np.random.default_rng(29)
    n = 2500
    k, v = (rng.standard_normal((n, NKV, HD), dtype=np.float32) for _ in range(2))
    q = rng.standard_normal((2, NH, HD), dtype=np.float32)
    mode = bk.parse_mode(tag)

    def make(ctx):
        c = bk.AttnCache(ctx, mode, n_layers=1, n_ctx=n)
        c.append(0, k, v)
        return c
    ctx = bk.Context(0)
    cache = make(ctx)
    want = cache.attend(0, q[1])[0]
    cache.close()
    ctx.close()

    ctx = bk.Context(0)
    monkeypatch.setenv("BONSAI_KV_BOX_POLLS", "0")
    hasty = make(ctx)
    monkeypatch.delenv("BONSAI_KV_BOX_POLLS")
    cache = make(ctx)
    ones = np.ones((NH, HD), np.float32)
    d_q, d_out = [ctx.to_device(x) for x in q], [ctx.to_device(ones) for _ in range(3)]
    for _ in range(2):
        hasty.decode_device(0, d_q[0].ptr, d_out[0].ptr)
        cache.decode_device(0, d_q[1].ptr, d_out[1].ptr)
        cache.decode_device(0, d_q[1].ptr, d_out[2].ptr)
        assert ctx.lib.bk_synchronize(ctx.h) == abi.BK_ERR_CUDA
        msg = ctx.lib.bk_last_error(ctx.h)
        assert b"bounded wait" in msg and b"code 6" in msg, msg
        assert ctx.lib.bk_synchronize(ctx.h) == abi.BK_OK       # reported once, then clear
        for o in d_out:
            assert np.array_equal(o.download((NH, HD), np.float32), ones)
        cache.decode_device(0, d_q[1].ptr, d_out[1].ptr)
        got = d_out[1].download((NH, HD), np.float32)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
        d_out[1].upload(ones)
    for c in (hasty, cache):
        c.close()
    ctx.close()
