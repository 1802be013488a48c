"""PQ2_0 ternary rows: the oracle pinned to the reference's known answers (CPU), and the CUDA
matvec, through the C ABI, against the oracle (GPU).

Bar for the product (floating point): |y - y_oracle| <= 2e-5 * sum_j |x_j| |w_j| per output.  The
reference ships three summation orders for this product (decoded-row dot, scalar block dot, AVX2)
and bounds their mutual difference by 1e-4 relative in its own test (src/kernels.rs:855-906);
the norm-wise form used here is the same bound without the blow-up on outputs that cancel to ~0.
"""
import ctypes

import numpy as np
import pytest

TOL = 2e-5


def synth(bk, seed, n_rows, ne0, n_tok, x_scale=1.0):
    rng = np.random.default_rng(seed)
    nb = -(-ne0 // 128)
    codes = rng.integers(0, 4, size=(n_rows, ne0), dtype=np.uint8)
    scales = (0.01 + rng.random((n_rows, nb)) * 2.0).astype(np.float16)
    payload = bk.pack_pq2(codes, scales)
    x = (rng.standard_normal((n_tok, ne0)) * x_scale).astype(np.float32)
    return payload, codes, scales, x


def dense(codes, scales, ne0):
    w = codes.astype(np.float64) - 1.0
    return w * np.repeat(scales.astype(np.float64), 128, axis=1)[:, :ne0]


# ---- CPU: the oracle against the reference's own tests -------------------------------------------

def test_pq2_decode_known_row(oracle):
    # src/kernels.rs:774-787: scale 0x4000 = 2.0; code 3 at j = 0, code 1 at j = 4, code 2 at j = 5
    raw = np.zeros(34, np.uint8)
    raw[1] = 0x40
    raw[2] = 0b11
    raw[3] = 0b1001
    v = oracle.pq2_decode_row(raw, 128)
    assert v[0] == 4.0 and v[1] == -2.0 and v[4] == 0.0 and v[5] == 2.0
    assert v.size == 128 and np.all(v[6:] == -2.0)


def test_pq2_row_bytes(oracle, bk):
    for ne0, want in ((128, 34), (129, 68), (256, 68), (5120, 1360), (6144, 1632), (1, 34)):
        assert oracle.pq2_row_bytes(ne0) == want == bk.pq2_row_bytes(ne0)


def test_pq2_matmul_n_matches_per_token_matvec(oracle, bk):
    # src/kernels.rs:909-947: the N-column product equals the per-token matvec exactly
    payload, _, _, x = synth(bk, 1, 12, 256, 3)
    y_n = oracle.pq2_matmul(payload, 256, 0, 12, x, 3)
    for t in range(3):
        assert np.array_equal(y_n[t], oracle.pq2_matmul(payload, 256, 0, 12, x[t], 1)[0])


def test_pq2_scalar_dot_matches_decoded_dot_and_f64(oracle, bk):
    ne0, n_rows = 5120, 8  # the model's row width (src/kernels.rs:864)
    payload, codes, scales, x = synth(bk, 2, n_rows, ne0, 1)
    w = dense(codes, scales, ne0)
    y = oracle.pq2_matmul(payload, ne0, 0, n_rows, x, 1)[0]
    norm = np.abs(w) @ np.abs(x[0].astype(np.float64))
    truth = w @ x[0].astype(np.float64)
    assert np.all(np.abs(y - truth) <= TOL * norm)
    for r in range(n_rows):
        assert abs(oracle.pq2_dot_row(payload, ne0, r, x[0]) - y[r]) <= TOL * norm[r]
        assert np.array_equal(oracle.pq2_decode_row(payload[r * 1360:(r + 1) * 1360], ne0), w[r].astype(np.float32))


def test_pq2_ragged_row_ignores_codes_past_ne0(oracle, bk):
    ne0 = 200
    payload, codes, scales, x = synth(bk, 3, 5, ne0, 1)
    dirty = payload.copy().reshape(5, 2, 34)
    dirty[:, 1, 2 + (ne0 - 128) // 4:] = 0xFF  # codes past ne0 in the last block
    y0 = oracle.pq2_matmul(payload, ne0, 0, 5, x, 1)
    y1 = oracle.pq2_matmul(dirty.reshape(-1), ne0, 0, 5, x, 1)
    assert np.array_equal(y0, y1)
    assert oracle.pq2_decode_row(payload[:68], ne0).size == ne0


def test_pq2_range_errors(oracle, bk):
    payload, _, _, x = synth(bk, 4, 4, 128, 1)
    with pytest.raises(ValueError):
        oracle.pq2_matmul(payload, 128, 2, 3, x, 1)  # rows 2..5 of 4 (src/kernels.rs:288-299)
    with pytest.raises(ValueError):
        oracle.pq2_matmul(payload, 128, 0, 4, x[0, :100], 1)  # x length (src/kernels.rs:282-284)
    with pytest.raises(ValueError):
        oracle.pq2_dot_row(payload, 128, 4, x[0])


# ---- GPU: the CUDA matvec against the oracle -------------------------------------------------------

SHAPES = [(5120, 1024, 1), (5120, 1000, 1), (6144, 512, 1), (256, 12, 3), (200, 37, 2), (5120, 64, 4), (5120, 33, 7),
          (128, 1, 1), (17408, 48, 1), (5120, 16 * 300, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("ne0,n_rows,n_tok", SHAPES)
def test_gpu_pq2_matvec_matches_oracle(oracle, bk, gpu_ctx, ne0, n_rows, n_tok):
    payload, codes, scales, x = synth(bk, ne0 + n_rows + n_tok, n_rows, ne0, n_tok)
    t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
    got = t.matmul_n(x, n_tok)
    gpu_ctx.synchronize()
    want = oracle.pq2_matmul(payload, ne0, 0, n_rows, x, n_tok)
    w = dense(codes, scales, ne0)
    norm = np.abs(x.astype(np.float64)) @ np.abs(w).T
    truth = x.astype(np.float64) @ w.T
    assert np.all(np.abs(got - want) <= TOL * norm + 1e-30), f"max {np.max(np.abs(got - want) / (norm + 1e-30)):.3e}"
    assert np.max(np.abs(got - truth) / (norm + 1e-30)) <= 2e-6  # exact block sums of 25-bit fixed-point x, f32 sums across blocks
    t.free()


@pytest.mark.gpu
def test_gpu_pq2_row_ranges_aligned_and_not(oracle, bk, gpu_ctx):
    # ne0 = 128: rows of 34 bytes, so most base rows start off a 16-byte boundary (plain-load path)
    for ne0, n_all in ((128, 70), (5120, 90)):
        payload, _, _, x = synth(bk, 11 + ne0, n_all, ne0, 1)
        t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
        for base, n in ((0, n_all), (3, 40), (8, 33), (16, 16), (n_all - 1, 1), (5, 0)):
            got = t.matvec(x[0], base_row=base, n_rows=n)
            want = oracle.pq2_matmul(payload, ne0, base, n, x, 1)[0]
            full = oracle.pq2_matmul(payload, ne0, 0, n_all, x, 1)[0]
            assert np.array_equal(want, full[base:base + n])
            assert np.all(np.abs(got - want) <= TOL * np.abs(x[0]).sum() * 2.0)
        t.free()


@pytest.mark.gpu
def test_gpu_pq2_errors_like_the_reference(bk, gpu_ctx):
    payload, _, _, x = synth(bk, 5, 4, 128, 1)
    t = bk.Pq2Tensor(gpu_ctx, payload, 128)
    with pytest.raises(bk.BonsaiKvError) as e:
        t.matvec(x[0], base_row=2, n_rows=3)
    assert e.value.status == bk._abi.BK_ERR_RANGE and "payload is" in str(e.value)
    with pytest.raises(bk.BonsaiKvError):
        t.matvec(x[0, :100])
    t.free()


@pytest.mark.gpu
def test_gpu_pq2_properties_at_model_size(bk, gpu_ctx):
    """wq of a full-attention layer (12288 x 5120): exact behaviour that needs no oracle."""
    ne0, n_rows = 5120, 12288
    rng = np.random.default_rng(99)
    nb = ne0 // 128
    x = rng.standard_normal((1, ne0)).astype(np.float32)
    # weight 0 everywhere (code 1): exactly zero; weight +1 with scale 1 (code 2): the sum of x
    zeros = bk.Pq2Tensor(gpu_ctx, bk.pack_pq2(np.ones((64, ne0), np.uint8), np.ones((64, nb))), ne0)
    assert np.all(np.abs(zeros.matvec(x[0])) <= 1e-6 * np.abs(x).sum())
    ones = bk.Pq2Tensor(gpu_ctx, bk.pack_pq2(np.full((64, ne0), 2, np.uint8), np.ones((64, nb))), ne0)
    assert np.allclose(ones.matvec(x[0]), x.astype(np.float64).sum(), rtol=0, atol=2e-6 * np.abs(x).sum())
    zeros.free()
    ones.free()
    codes = rng.integers(0, 4, size=(n_rows, ne0), dtype=np.uint8)
    scales = (0.01 + rng.random((n_rows, nb))).astype(np.float16)
    t = bk.Pq2Tensor(gpu_ctx, bk.pack_pq2(codes, scales), ne0)
    y = t.matvec(x[0])
    # a power-of-two factor on x passes through exactly (the kernel normalises every block of x by a power of two)
    assert np.array_equal(t.matvec(x[0] * np.float32(1024.0)), y * np.float32(1024.0))
    assert np.array_equal(t.matvec(x[0] * np.float32(2.0 ** -20)), y * np.float32(2.0 ** -20))
    # rows are independent: any row range equals the slice of the whole product
    assert np.array_equal(t.matvec(x[0], base_row=4096, n_rows=1024), y[4096:5120])
    # against float64 on a sample of rows
    rows = rng.choice(n_rows, 64, replace=False)
    w = dense(codes[rows], scales[rows], ne0)
    assert np.max(np.abs(y[rows] - w @ x[0].astype(np.float64)) / (np.abs(w) @ np.abs(x[0]).astype(np.float64))) <= 2e-6
    t.free()


@pytest.mark.gpu
def test_gpu_pq2_multi_equals_separate_calls(bk, gpu_ctx):
    """attn_q, attn_k, attn_v shapes on one x in one launch: bit-equal to three launches."""
    ne0 = 5120
    rng = np.random.default_rng(7)
    tensors = []
    for n_rows in (12288, 1024, 1000):
        payload, _, _, _ = synth(bk, n_rows, n_rows, ne0, 1)
        tensors.append(bk.Pq2Tensor(gpu_ctx, payload, ne0))
    for n_tok in (1, 2, 3):
        x = rng.standard_normal((n_tok, ne0)).astype(np.float32)
        dx = gpu_ctx.to_device(x)
        ys = [gpu_ctx.alloc(n_tok * t.n_rows * 4) for t in tensors]
        bk.pq2_matvec_multi_device(gpu_ctx, tensors, dx.ptr, [y.ptr for y in ys], n_tok)
        for t, y in zip(tensors, ys):
            got = y.download((n_tok, t.n_rows), np.float32)
            assert np.array_equal(got, t.matmul_n(x, n_tok))
            y.free()
        dx.free()
    for t in tensors:
        t.free()


@pytest.mark.gpu
@pytest.mark.parametrize("ne0,n_rows,n_tok,base", [(128, 1, 5, 0), (128, 130, 6, 3), (200, 129, 15, 1), (512, 128, 16, 0), (640, 257, 17, 1), (5120, 300, 33, 2),
                                                   (1280, 2000, 128, 0), (768, 255, 129, 0), (384, 40, 1025, 1), (128, 40000, 100, 0), (5120, 40, 512, 5),
                                                   (1024, 300, 20, 0), (1152, 300, 128, 0), (1280, 20000, 512, 0), (1408, 300, 90, 0), (2432, 140, 40, 0)])
def test_gpu_pq2_token_block_product(bk, gpu_ctx, ne0, n_rows, n_tok, base):
    """The tensor-core product at the edges of its tiles (128 rows, 16..128 tokens, segments of four and groups of eight blocks,
    1024 tokens a pass, rows off a word boundary).  Bound: f16 pairs hold x to 2^-22 of each element and the per-block sums are
    rounded to f32 (2^-24 of sum |x||w|, up to 16 times a block, then once a block): 2e-6 of sum |x||w|."""
    payload, codes, scales, x = synth(bk, 7 * ne0 + n_rows + n_tok, n_rows + base, ne0, n_tok)
    t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
    got = t.matmul_n(x, n_tok, base_row=base)
    w = dense(codes[base:], scales[base:], ne0)
    truth = x.astype(np.float64) @ w.T
    norm = np.abs(x.astype(np.float64)) @ np.abs(w).T
    assert np.max(np.abs(got - truth) / (norm + 1e-30)) <= 2e-6
    t.free()


@pytest.mark.gpu
def test_gpu_pq2_row_length_limit(bk, gpu_ctx):
    """Rows of 157 blocks fit the product of one token and not that of two: whatever the number of tokens from two on,
    the call is refused."""
    payload, _, _, x = synth(bk, 5, 3, 157 * 128, 6)
    t = bk.Pq2Tensor(gpu_ctx, payload, 157 * 128)
    assert t.matmul_n(x[:1], 1).shape == (1, 3)
    for n_tok in (2, 4, 5, 6):
        with pytest.raises(bk.BonsaiKvError, match="rows too long"):
            t.matmul_n(x[:n_tok], n_tok)
    t.free()


def product(bk, ctx, t, x, base=0, n_rows=None, x_shift=0):
    """The product on device buffers, with x placed x_shift floats behind a 256-byte boundary."""
    n_tok, ne0 = x.shape
    n_rows = t.n_rows - base if n_rows is None else n_rows
    dx = ctx.to_device(np.concatenate([np.zeros(x_shift, np.float32), x.ravel()]))
    dy = ctx.alloc(max(n_tok * n_rows * 4, 4))
    t.matvec_device(dx.ptr + 4 * x_shift, dy.ptr, n_tok, base, n_rows)
    y = dy.download((n_tok, n_rows), np.float32)
    dx.free()
    dy.free()
    return y


@pytest.mark.gpu
@pytest.mark.parametrize("n_tok", [4, 5, 70])
def test_gpu_pq2_blocks_of_unlike_size(bk, gpu_ctx, n_tok):
    """A block of x a factor of 1e13 above the others, and rows whose weights there are zero: the other blocks count in full.
    Bound: x is held to 2^-25 of its own block's largest element (about 4 times its mean size: 2^-23 of |x||w|) and the f32 sums of
    ten blocks round by 2^-24 each: 2e-6 of sum |x||w|."""
    rng = np.random.default_rng(n_tok)
    _, codes, scales, x = synth(bk, 11, 200, 1280, n_tok)
    codes[::2, :128] = 1
    x[:, :128] *= 1e13
    x[:, 256:512] *= 2.0 ** rng.integers(-40, 1, (n_tok, 1))
    t = bk.Pq2Tensor(gpu_ctx, bk.pack_pq2(codes, scales), 1280)
    w = dense(codes, scales, 1280)
    got, x64 = product(bk, gpu_ctx, t, x), x.astype(np.float64)
    assert np.max(np.abs(got - x64 @ w.T) / (np.abs(x64) @ np.abs(w).T)) <= 2e-6
    t.free()


@pytest.mark.gpu
@pytest.mark.parametrize("n_tok", [4, 64])
def test_gpu_pq2_sums_are_not_biased(bk, gpu_ctx, n_tok):
    """Products of one sign: exact block sums and sums rounded to nearest leave no mean error.  The errors of 300 x n_tok outputs are about 5e-8
    each and cancel to 2e-9 or less; truncated sums showed 5e-8."""
    _, _, scales, x = synth(bk, 12, 300, 5120, n_tok)
    codes, x = np.full((300, 5120), 2, np.uint8), np.abs(x) + np.float32(0.5)
    t = bk.Pq2Tensor(gpu_ctx, bk.pack_pq2(codes, scales), 5120)
    truth = x.astype(np.float64) @ dense(codes, scales, 5120).T
    assert abs(np.mean((product(bk, gpu_ctx, t, x) - truth) / truth)) <= 1e-8
    t.free()


@pytest.mark.gpu
def test_gpu_pq2_zero_and_non_finite_tokens(bk, gpu_ctx):
    """A token of zeros gives zeros, one with an infinity or a NaN in it gives NaN, and neither touches the others."""
    payload, _, _, x = synth(bk, 13, 130, 640, 20)
    t = bk.Pq2Tensor(gpu_ctx, payload, 640)
    clean = product(bk, gpu_ctx, t, x)
    x[3], x[7, 5], x[8, 639], x[9, 130] = 0, np.nan, np.inf, -np.inf
    got = product(bk, gpu_ctx, t, x)
    assert not got[3].any() and np.isnan(got[7:10]).all()
    rest = [i for i in range(20) if i not in (3, 7, 8, 9)]
    assert np.array_equal(got[rest], clean[rest])
    t.free()


@pytest.mark.gpu
@pytest.mark.parametrize("ne0,shift,off", [(1026, 0, 0), (1027, 0, 0), (1024, 1, 0), (1024, 2, 0), (1024, 0, 4), (1024, 3, 2), (2048, 0, 8)])
def test_gpu_pq2_token_block_alignment(bk, gpu_ctx, ne0, shift, off):
    """x off a 16-byte boundary, rows of an odd length, weights off 16- and 4-byte boundaries: bit for bit the aligned call's result."""
    payload, codes, scales, x = synth(bk, 14, 150, ne0, 21)
    t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
    want = product(bk, gpu_ctx, t, x)
    w, x64 = dense(codes, scales, ne0), x.astype(np.float64)
    assert np.max(np.abs(want - x64 @ w.T) / (np.abs(x64) @ np.abs(w).T + 1e-30)) <= 2e-6  # as in the token-block test
    moved = gpu_ctx.to_device(np.concatenate([np.zeros(off, np.uint8), payload]))
    dx, dy = gpu_ctx.to_device(np.concatenate([np.zeros(shift, np.float32), x.ravel()])), gpu_ctx.alloc(want.nbytes)
    gpu_ctx.check(gpu_ctx.lib.bk_pq2_matvec(gpu_ctx.h, moved.ptr + off, payload.size, ne0, 0, 150, dx.ptr + 4 * shift, 21, dy.ptr))
    assert np.array_equal(dy.download(want.shape, np.float32), want)
    for b in (moved, dx, dy):
        b.free()
    t.free()


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 2, 4, 5, 8, 9, 12, 13, 16, 17, 20, 33, 40])
def test_gpu_pq2_tiling_does_not_show(bk, gpu_ctx, nb):
    """One or two row tiles a CTA, 16 to 64 tokens a tile, rows handed to a second launch: the first tokens of a long block
    come out bit for bit as in a short one.  14336 rows x 512 tokens take the split launch, 300 rows single row tiles."""
    rng = np.random.default_rng(nb)
    n_rows, ne0 = 14336 + 3, nb * 128
    payload = rng.integers(0, 256, (n_rows, nb, 34), dtype=np.uint8)
    payload[..., :2] = rng.uniform(0.01, 2.0, (n_rows, nb, 1)).astype(np.float16).view(np.uint8)
    x = rng.standard_normal((512, ne0)).astype(np.float32)
    t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
    whole = product(bk, gpu_ctx, t, x)
    for n_tok in (5, 40, 130):
        assert np.array_equal(product(bk, gpu_ctx, t, x[:n_tok]), whole[:n_tok]), n_tok
    for base in (0, 14039):
        assert np.array_equal(product(bk, gpu_ctx, t, x[:33], base, 300), whole[:33, base:base + 300]), base
    t.free()


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [16, 17, 33, 36, 48, 49, 129])
def test_gpu_pq2_clusters_on_a_tile_do_not_show(bk, gpu_ctx, nb):
    """Few row tiles and few tokens: clusters share a tile's units (none with 16 blocks, which are one pair), up to eight CTAs of them with 129
    blocks, which have nine pairs.  The same bits as among so many tokens that nothing is shared, with rows that do not fill their tile."""
    ne0, n_rows, n_all = nb * 128 - 40, 1000, 1024
    payload, _, _, x = synth(bk, nb, n_rows, ne0, n_all)
    t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
    want = t.matmul_n(x, n_all)
    for n_tok in (5, 17, 33, 64):
        assert np.array_equal(t.matmul_n(x[:n_tok], n_tok), want[:n_tok]), n_tok
    assert np.array_equal(t.matmul_n(x[:9], 9, base_row=130, n_rows=150), want[:9, 130:280])
    t.free()


def pq2_plan(bk, n_sms, clusters, n_rows, nb, n_tok):
    """(row tiles a CTA, token tile / 16, CTAs that share a tile, tiles of the first launch)"""
    out = (ctypes.c_int32 * 4)()
    bk._abi.load().bk_hook_pq2_plan(n_sms, (ctypes.c_int32 * 9)(*clusters), n_rows, nb, n_tok, out)
    return tuple(out)


def test_pq2_plan_keeps_to_the_clusters_that_fit(bk):
    """A launch never has more clusters than the device takes at once, a tile's CTAs all have work, and the device decides: with room for none,
    none are made.  The counts are a B200's, then fewer."""
    b200 = [0, 0, 74, 45, 33, 26, 22, 15, 15]
    assert pq2_plan(bk, 148, b200, 5120, 48, 16)[:3] == (1, 1, 3)
    assert pq2_plan(bk, 148, b200, 3072, 40, 32)[:3] == (1, 2, 3)  # (48 clusters of three for tiles of 16 tokens)
    forms = set()
    for clusters in (b200, [0, 0, 9, 6, 4, 3, 3, 2, 2], [0] * 9):
        for n_rows in (1, 150, 640, 1000, 2304, 3072, 5120, 5760, 9472, 14336):
            for nb in (1, 16, 17, 33, 40, 48, 49, 72, 88, 104, 113, 120, 128, 129, 140):
                for n_tok in (5, 16, 17, 33, 48, 49, 64, 100, 130, 256, 512):
                    mt, nc, split, _ = pq2_plan(bk, 148, clusters, n_rows, nb, n_tok)
                    if split > 1:
                        assert mt == 1 and -(-n_rows // 128) * -(-n_tok // (16 * nc)) <= clusters[split]
                        assert split <= (-(-(-(-nb // 4)) // 2) + 1) // 2
                        forms.add((nc, split))
    assert {nc for nc, _ in forms} == {1, 2, 3, 4} and {split for _, split in forms} == set(range(2, 9))


@pytest.mark.gpu
@pytest.mark.parametrize("nb,n_rows,forms", [
    (48, 5120, {(1, 3), (2, 3), (3, 3), (4, 3)}),  # the output projection
    (17, 1000, {(1, 2)}), (64, 5100, {(1, 2), (2, 2)}), (49, 1000, {(1, 4), (2, 4), (3, 4)}), (72, 1000, {(1, 5), (2, 5)}), (88, 1000, {(1, 6), (2, 6), (4, 6)}),
    (104, 1000, {(1, 7), (2, 7), (3, 7), (4, 7)}), (120, 1000, {(1, 8), (2, 8), (3, 8)})])
def test_gpu_pq2_every_form_of_clusters(bk, gpu_ctx, nb, n_rows, forms):
    """Tiles of 16, 32, 48 and 64 tokens in clusters of 2 to 8: bit for bit a block of so many tokens that no tile is shared, and that within
    the bound of the token-block test.  Which forms a B200 gets is part of the test."""
    ne0, n_all, counts = nb * 128 - 40, 1024, (5, 17, 33, 48, 50, 64, 100, 130)
    clusters = (ctypes.c_int32 * 9)()
    fn = bk._abi.load().bk_hook_pq2_clusters
    fn.restype = ctypes.POINTER(ctypes.c_int32)
    clusters[:] = [0, 0, *fn(gpu_ctx.h)[2:9]]
    plans = {n: pq2_plan(bk, 148, clusters, n_rows, nb, n) for n in (*counts, n_all)}
    assert plans[n_all][2] == 1
    if list(clusters) == [0, 0, 74, 45, 33, 26, 22, 15, 15]:  # (a device with other groups of SMs has other forms)
        assert {p[1:3] for p in plans.values() if p[2] > 1} >= forms
    payload, codes, scales, x = synth(bk, nb, n_rows, ne0, n_all)
    t = bk.Pq2Tensor(gpu_ctx, payload, ne0)
    want = t.matmul_n(x, n_all)
    w, x64 = dense(codes[:200], scales[:200], ne0), x[:130].astype(np.float64)
    assert np.max(np.abs(want[:130, :200] - x64 @ w.T) / (np.abs(x64) @ np.abs(w).T + 1e-30)) <= 2e-6  # as in the token-block test
    for n_tok in counts:
        assert np.array_equal(t.matmul_n(x[:n_tok], n_tok), want[:n_tok]), (n_tok, plans[n_tok])
    t.free()


@pytest.mark.gpu
@pytest.mark.parametrize("n_tok", [5, 17, 200])
def test_gpu_pq2_multi_token_block_equals_separate_calls(bk, gpu_ctx, n_tok):
    """Ranges of odd row counts, one of them off a 16-byte boundary, in one launch: bit for bit the separate calls."""
    ne0 = 1280
    payload, _, _, x = synth(bk, 15, 1000, ne0, n_tok)
    buf = gpu_ctx.to_device(np.concatenate([np.zeros(6, np.uint8), payload]))
    dx = gpu_ctx.to_device(x)
    ranges = [(6, 0, 333), (0, 0, 1), (6, 400, 257), (0, 0, 0)]  # (offset, base row, rows); row bytes 340, so offset 0 holds other rows
    multi = [gpu_ctx.alloc(max(n_tok * n, 1) * 4) for _, _, n in ranges]
    segs = (bk.pq2._Seg * len(ranges))()
    for sg, y, (off, base, n) in zip(segs, multi, ranges):
        sg.payload_dev, sg.payload_bytes, sg.base_row, sg.n_rows, sg.y_dev = buf.ptr + off, payload.size, base, n, y.ptr
    gpu_ctx.check(gpu_ctx.lib.bk_pq2_matvec_multi(gpu_ctx.h, len(ranges), ctypes.cast(segs, ctypes.c_void_p), ne0, dx.ptr, n_tok))
    for y, (off, base, n) in zip(multi, ranges):
        if n:
            one = gpu_ctx.alloc(n_tok * n * 4)
            gpu_ctx.check(gpu_ctx.lib.bk_pq2_matvec(gpu_ctx.h, buf.ptr + off, payload.size, ne0, base, n, dx.ptr, n_tok, one.ptr))
            assert np.array_equal(y.download((n_tok, n), np.float32).view(np.uint32), one.download((n_tok, n), np.float32).view(np.uint32)), (off, base)
            one.free()
    for b in (buf, dx, *multi):
        b.free()


@pytest.mark.gpu
@pytest.mark.parametrize("n_tok", [2, 5, 100])
def test_gpu_pq2_first_call_can_be_captured(bk, n_tok):
    """The first product of a context goes into a CUDA graph: no call allocates or waits for the stream."""
    import torch
    ctx = bk.Context(0)
    payload, _, _, x = synth(bk, 16, 300, 640, n_tok)
    t = bk.Pq2Tensor(ctx, payload, 640)
    dx, dy = ctx.to_device(x), ctx.to_device(np.zeros((n_tok, 300), np.float32))
    ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    stream = torch.cuda.ExternalStream(ctx.lib.bk_ctx_stream(ctx.h))
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
        t.matvec_device(dx.ptr, dy.ptr, n_tok)
    with torch.cuda.stream(stream):
        graph.replay()
    ctx.synchronize()
    assert np.array_equal(dy.download((n_tok, 300), np.float32), product(bk, ctx, t, x))
    del graph
    t.free()
    dx.free()
    dy.free()
    ctx.close()
