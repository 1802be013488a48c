"""CPU-side checks of the C ABI: the library loads, exports every declared symbol, and its
host-side pieces (mode parser, environment readers, set-up tables) agree with the oracle.
No compute entry point is called here."""
import ctypes as C
import os
import re

import numpy as np
import pytest

from oracle_lib import MODE_F16, MODE_F32, MODE_PLANAR

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "bonsai_kv.h")).read()
    return sorted(set(re.findall(r"BK_API[^;(]*?\b(bk_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol(bk):
    lib = C.CDLL(bk.library_path())
    names = declared_symbols()
    assert len(names) >= 50
    for n in names:
        assert hasattr(lib, n), f"{n} is declared in include/bonsai_kv.h but not exported"


def test_ctypes_table_covers_the_header(bk):
    assert sorted(bk._abi.SIGNATURES) == declared_symbols()


def test_version_and_status_strings(bk):
    lib = bk._abi.load()
    assert b"sm_100a" in lib.bk_version()
    assert lib.bk_status_string(0) == b"ok" and lib.bk_status_string(4).startswith(b"position")


def test_parse_mode_matches_reference_table(bk, oracle):
    """src/kvquant.rs:670-720 through the ABI, cross-checked with the oracle on more strings."""
    kinds = {MODE_F32: "f32", MODE_F16: "f16", MODE_PLANAR: "planar"}
    cases = ["", "f32", "f16", "fp16", "half", "planar4", "planar4k", "iso3", "iso8k", "planar9", "planar0",
             "garbage", "planark", "planar", "iso", "isok", "planar1", "planar8", "iso1k", "planar+4",
             "planar04", "planar4kk", "PLANAR4", "planar 4", "planar4 ", "k", "f16k", "planar-1", "iso99999999999"]
    for s in cases:
        kind, bits, vq = oracle.parse_mode(s)
        m = bk.parse_mode(s)
        assert (m.kind, m.bits, m.v_quant) == (kinds[kind], bits, vq), s
    assert bk.parse_mode("planar4") == bk.Planar(4, True)
    assert bk.parse_mode("iso8k") == bk.Planar(8, False)


def test_quantizers_follow_the_mode(bk):
    """src/kvquant.rs:711-719 (construction only; no GPU call)."""
    class FakeCtx:  # quantizers_for only stores the context
        pass
    k, v = bk.quantizers_for(bk.parse_mode("planar4"), 256, FakeCtx())
    assert k is not None and v is not None
    k, v = bk.quantizers_for(bk.parse_mode("planar4k"), 256, FakeCtx())
    assert k is not None and v is None
    assert bk.quantizers_for(bk.parse_mode("f16"), 256, FakeCtx()) == (None, None)
    assert bk.quantizers_for(bk.parse_mode("f32"), 256, FakeCtx()) == (None, None)
    with pytest.raises(AssertionError):
        bk.PlanarQuant(256, 9, FakeCtx())
    assert bk.PlanarQuant(256, 3, FakeCtx()).packed_len() == 96


def test_env_readers(bk, monkeypatch):
    """BONSAI_KV (src/kvquant.rs:546-550) and BONSAI_CTX (src/gdev.rs:39-48)."""
    monkeypatch.delenv("BONSAI_KV", raising=False)
    monkeypatch.delenv("BONSAI_CTX", raising=False)
    assert bk.mode_from_env() == bk.F32 and bk.n_ctx_env() == 2048
    monkeypatch.setenv("BONSAI_KV", "planar3k")
    assert bk.mode_from_env() == bk.Planar(3, False)
    for val, want in [("16", 16), ("262144", 262144), ("15", 2048), ("262145", 2048), ("abc", 2048), ("4096", 4096)]:
        monkeypatch.setenv("BONSAI_CTX", val)
        assert bk.n_ctx_env() == want, val


@pytest.mark.parametrize("bits", range(1, 9))
def test_setup_tables_equal_the_oracle(bk, oracle, bits):
    """The library's own host set-up code (not the oracle) builds the codebook and the
    Givens table; both must equal the oracle's bit for bit."""
    assert np.array_equal(bk.codebook(256, bits).view(np.uint32), oracle.codebook(256, bits).view(np.uint32))
    assert np.array_equal(bk.givens_table(256).view(np.uint32), oracle.givens(256).view(np.uint32))
    assert bk.packed_bytes(256, bits) == 32 * bits == bk._abi.load().bk_kvq_packed_len(256, bits)


@pytest.mark.parametrize("bits", [1, 2, 3, 4])
def test_threshold_cells_give_the_reference_scan(bk, oracle, bits):
    """The decision thresholds in 512 cells, for programs that find the nearest centroid with one table read and one
    comparison, against the reference's scan (src/kvquant.rs:357-370: ascending, strict '<', f32 differences) on the
    values where the two could part: centroids, exact midpoints, the decision thresholds themselves, cell edges, each with
    their neighbouring floats, and a dense random sample.  (The kernels' own table: the next test.)"""
    lib = bk._abi.load()
    cells = np.zeros((512, 2), np.uint32)
    assert lib.bk_kvq_threshold_cells(bits, cells.ctypes.data) == 0
    count, thr = cells[:, 0].astype(np.int64), cells[:, 1].copy().view(np.float32)
    book = oracle.codebook(256, bits).astype(np.float32)
    n = 1 << bits
    assert count[0] == 0 and count[-1] + np.isfinite(thr[-1]) <= n - 1 and np.all(np.diff(count) >= 0)
    assert int(np.isfinite(thr).sum()) == n - 1            # every threshold sits in a cell of its own

    def neighbours(x, k=3):
        out = [np.float32(x)]
        lo = hi = np.float32(x)
        for _ in range(k):
            lo, hi = np.nextafter(lo, np.float32(-np.inf)), np.nextafter(hi, np.float32(np.inf))
            out += [lo, hi]
        return out
    probes = []
    for c in book:
        probes += neighbours(c)
    for a, b in zip(book[:-1], book[1:]):
        probes += neighbours(np.float32(0.5) * (a + b)) + neighbours(np.float32((np.float64(a) + np.float64(b)) / 2))
    for t in thr[np.isfinite(thr)]:
        probes += neighbours(t, 5)
    for k in range(0, 513):
        probes += neighbours(np.float32(k) / np.float32(1024) - np.float32(0.25))
    probes += [np.float32(x) for x in (-3.9, -1.0, -0.26, -0.25, 0.0, -0.0, 0.25, 0.26, 1.0, 3.9)]
    rng = np.random.default_rng(bits)
    v = np.concatenate([np.array(probes, np.float32), (rng.standard_normal(200000) / 16).astype(np.float32),
                        rng.uniform(-0.3, 0.3, 200000).astype(np.float32)])
    want = np.argmin(np.abs(v[:, None] - book[None, :]), axis=1)       # f32 differences; first minimum = lowest index
    cell = np.clip(np.floor((v + np.float32(0.25)) * np.float32(1024)).astype(np.int64), 0, 511)
    got = count[cell] + (v >= thr[cell])
    bad = np.flatnonzero(got != want)
    assert bad.size == 0, (v[bad[:5]], got[bad[:5]], want[bad[:5]])


@pytest.mark.parametrize("bits", [1, 2, 3, 4])
def test_lane_cells_give_the_reference_scan(bk, oracle, bits):
    """The table that the append and quantize kernels read: 32 cells of floor(31.999998 clamp(v scale + 1/2)), the sum rounded
    once to f32.  Checked against the reference's scan on centroids, midpoints, thresholds and cell edges, each with their
    neighbouring floats, and on a dense random sample."""
    lib = bk._abi.load()
    words = np.zeros(65, np.uint32)
    assert lib.bk_kvq_lane_cells(bits, words.ctypes.data) == 0
    below, thr, scale = words[0:64:2].astype(np.int64), words[1:64:2].copy().view(np.float32), words[64:].view(np.float32)[0]
    book = oracle.codebook(256, bits).astype(np.float32)
    assert int(np.isfinite(thr).sum()) == (1 << bits) - 1 and np.all(np.diff(below) >= 0) and scale > 0
    edges = [(np.float64(c) / np.float64(np.float32(31.999998)) - 0.5) / np.float64(scale) for c in range(33)]
    at = np.array([*book, *(0.5 * (book[:-1].astype(np.float64) + book[1:])), *thr[np.isfinite(thr)], *edges, 0.0, 0.25, -0.25], np.float32)
    probes = [at]
    for towards in (np.float32(-np.inf), np.float32(np.inf)):
        x = at
        for _ in range(6):
            x = np.nextafter(x, towards)
            probes.append(x)
    rng = np.random.default_rng(bits)
    probes += [(rng.standard_normal(300000) / 16).astype(np.float32), rng.uniform(-0.3, 0.3, 300000).astype(np.float32),
               np.array([1.5, -1.5, -0.0, 1e-30, -1e-30, 1e-45], np.float32)]   # (rotated unit vectors stay below 1.5)
    v = np.concatenate(probes)
    want = np.argmin(np.abs(v[:, None].astype(np.float32) - book[None, :]), axis=1)
    u = np.clip((v.astype(np.longdouble) * np.longdouble(scale) + np.longdouble(0.5)).astype(np.float32), np.float32(0), np.float32(1))
    cell = np.floor(u.astype(np.float64) * np.float64(np.float32(31.999998))).astype(np.int64)   # (24 + 24 bits: exact)
    assert cell.min() == 0 and cell.max() == 31
    got = below[cell] + (v >= thr[cell])
    bad = np.flatnonzero(got != want)
    assert bad.size == 0, (v[bad[:5]], got[bad[:5]], want[bad[:5]])


@pytest.mark.parametrize("n_head,n_kv", [(24, 4), (6, 1), (4, 4), (8, 4), (8, 8)])
def test_prefill_plan_covers_every_tile_once(bk, n_head, n_kv):
    """The pieces of a prompt block: every tile that an item sees in exactly one of them, a place of the scratch (two a processor, up to 160
    processors) for every piece of a cut item, one item's places side by side in the order of its tiles."""
    lib = bk._abi.load()
    tq = 128 // (n_head // n_kv)
    rng = np.random.default_rng(n_head + n_kv)
    shapes = [(0, 4), (0, 512), (0, 777), (4096, 512), (262000, 100), (20000, 5), (0, 3100), (0, 3400), (0, 9000), (2097000, 300)]
    shapes += [(int(rng.integers(0, 9000)) * (i % 3 > 0), int(rng.integers(4, 2000))) for i in range(60)]
    for n_sms in (148, 1, 2, 200):
        for pos0, n_tok in shapes:
            words = np.full((768, 4), -7, np.int32)
            n = lib.bk_hook_prefill_plan(n_sms, pos0, n_tok, n_head, n_kv, 768, C.c_void_p(words.ctypes.data))
            if n == 0:
                continue
            blocks = -(-n_tok // tq)
            assert blocks * n_kv <= n <= 768
            words = words[:n]
            parts = words[words[:, 3] >= 0, 3]
            assert len(set(parts)) == len(parts) and (len(parts) == 0 or parts.max() < 2 * min(n_sms, 160))
            words = words[np.lexsort((words[:, 1], words[:, 0]))]
            assert np.array_equal(np.unique(words[:, 0]), np.arange(blocks * n_kv))
            for item in range(blocks * n_kv):
                w = words[words[:, 0] == item]
                tiles = -(-(pos0 + min((blocks - item // n_kv) * tq, n_tok)) // 32)
                assert w[0, 1] == 0 and w[-1, 2] == tiles and np.array_equal(w[1:, 1], w[:-1, 2]) and (w[:, 2] > w[:, 1]).all()
                assert np.array_equal(w[:, 3], w[0, 3] + np.arange(len(w))) and (w[0, 3] >= 0 or len(w) == 1)


def test_prefill_plan_cuts_where_it_gains(bk):
    """A plan of pieces, each handed to the processor that is free first at seven tiles a piece beside its own, ends before whole items would, within
    a fifth and a piece's seven tiles of an even spread; and blocks that go out whole would not have gained more than the cutting costs."""
    import heapq
    lib = bk._abi.load()

    def end(lengths, n_sms):
        free = [0] * n_sms
        for n in lengths:
            heapq.heapreplace(free, free[0] + n + 7)
        return max(free)

    seen = {True: 0, False: 0}
    for n_sms in (148, 132, 16):
        for n_head, n_kv in ((24, 4), (48, 8), (8, 8), (6, 1)):
            tq = 128 // (n_head // n_kv)
            for pos0 in (0, 500, 1024, 4096, 30000):
                for n_tok in (4, 50, 130, 300, 400, 512, 600, 777, 1000, 1500, 2500):
                    blocks = -(-n_tok // tq)
                    if blocks * n_kv > 608:
                        continue
                    words = np.zeros((768, 4), np.int32)
                    n = lib.bk_hook_prefill_plan(n_sms, pos0, n_tok, n_head, n_kv, 768, C.c_void_p(words.ctypes.data))
                    items = [-(-(pos0 + min((blocks - i // n_kv) * tq, n_tok)) // 32) for i in range(blocks * n_kv)]
                    whole, even = end(items, n_sms), sum(t + 7 for t in items) / n_sms
                    what = (n_sms, n_head, n_kv, pos0, n_tok)
                    if n:
                        cut = end((words[:n, 2] - words[:n, 1]).tolist(), n_sms)
                        assert cut < whole, (what, cut, whole)
                        spread = (sum(items) + 7 * n) / n_sms
                        assert cut <= 1.2 * max(spread, 11) + 7, (what, cut, spread)
                    else:
                        assert whole <= 1.05 * max(1.25 * even + 7, 11) + 3 + 320 / 45, (what, whole, even)
                    seen[n > 0] += 1
    assert min(seen.values()) > 50
    for shape in ((0, 400, 24, 4), (4096, 512, 24, 4), (30000, 4, 6, 1)):
        assert lib.bk_hook_prefill_plan(148, *shape, 0, None) > 0
    for shape in ((0, 4, 24, 4), (0, 1000, 24, 4), (0, 600, 48, 8), (0, 3400, 24, 4)):
        assert lib.bk_hook_prefill_plan(148, *shape, 0, None) == 0


def test_read_only_loads_are_of_constants():
    """A kernel that is launched under the end of another one (it has a griddepcontrol.wait) may use the read-only path, which takes it for granted
    that nobody writes the data while the kernel lives, only for tables and weights: its other inputs may still be on their way when it starts."""
    csrc = os.path.join(ROOT, "ternary-bonsai-inference_b200", "csrc")
    sources = {f: open(os.path.join(csrc, f)).read() for f in sorted(os.listdir(csrc)) if f.endswith((".cu", ".cuh"))}
    early = [f for f in sources if "griddepcontrol.wait" in sources[f] or f == "bk_decode_common.cuh"]
    assert {"bk_append.cu", "bk_decode.cu", "bk_prefill_umma.cu"} <= set(early)
    found = [(f, line.strip()) for f in early for line in sources[f].splitlines() if re.search(r"__ldg\(|global\.nc|__restrict__", line)]
    assert len(found) > 3
    for f, line in found:
        for arg in re.split(r"__ldg\(", line)[1:]:
            assert re.match(r"(reinterpret_cast<[^>]*>\()?(a\.rope|a\.givens|a\.book|a\.k_norm_w|rope_row|weights)\b", arg), (f, line)
        assert "global.nc" not in line and "__restrict__" not in line, (f, line)


def test_default_config_is_qwen35(bk):
    cfg = bk._abi.CacheConfig()
    bk._abi.load().bk_default_config(C.byref(cfg))
    assert (cfg.n_layers, cfg.n_head, cfg.n_kv, cfg.hd, cfg.n_rot) == (16, 24, 4, 256, 64)
    assert list(cfg.sections) == [11, 11, 10, 0] and cfg.freq_base == np.float32(1e7)


def test_null_arguments_are_rejected_without_a_device(bk):
    lib = bk._abi.load()
    assert lib.bk_synchronize(None) == bk._abi.BK_ERR_INVALID
    assert lib.bk_cache_n_pos(None, 0, 0) == -1
    assert lib.bk_kvq_packed_len(256, 0) == 0 and lib.bk_kvq_packed_len(256, 9) == 0
    assert lib.bk_parse_mode(None, None) == bk._abi.BK_ERR_INVALID
    assert lib.bk_ctx_create(0, None) == bk._abi.BK_ERR_INVALID
    assert lib.bk_lse_merge(None, 1, 1, 256, None, None) == bk._abi.BK_ERR_INVALID


def test_no_cpu_fallback(bk):
    """Without a GPU the context cannot be created and says why; nothing computes on the CPU."""
    import shutil
    if shutil.which("nvidia-smi"):
        pytest.skip("a GPU is present")
    with pytest.raises(bk.BonsaiKvError) as e:
        bk.Context(0)
    assert e.value.status in (bk._abi.BK_ERR_CUDA, bk._abi.BK_ERR_INVALID)
