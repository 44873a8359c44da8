"""Prefill GEMM (csrc/gemm_tc.cu) in the modes whose promote reads a scale per token and group: every tile width
of two row blocks, with an odd number of row blocks (the last tile's second one does not exist), and the one of a
single row block, with a ragged last token block and more steps than step slots. The operands are e4m3
numbers that stand for the codes exactly, an int8 activation as the sum of two: the codes here are drawn from all
their values, -128 and -8 too, and the weights have every zero point. Every output word is compared with the
oracle; all sums up to the promote are exact integers, so no tolerance is needed."""
import numpy as np
import pytest

# tokens a tile -> rows, tokens
SIZES = {32: (384, 688), 48: (7552, 136), 64: (9600, 152), 80: (9600, 200), 96: (9600, 248), 112: (9600, 296),
         128: (9600, 344), 256: (4736, 1000)}
K = 1088                # 17 steps on 4 to 8 slots
SMS = 148


@pytest.mark.parametrize("width", SIZES)
def test_sizes_reach_every_width(lib_host, width):
    M, T = SIZES[width]
    assert lib_host.qwn_dbg_prefill_tile(M, T, 0, SMS) == width and M % 256 == 128 and T % width
    assert lib_host.qwn_choose_gemm_splits(M // 16, T // 8, K // 32) == 1


def test_widths_of_ordinary_calls(lib_host):
    tile = lib_host.qwn_dbg_prefill_tile
    assert [tile(M, T, 0, SMS) for M, T in ((10240, 136), (5120, 1000), (17408, 4096))] == [48, 80, 128]
    # one round of 256 tokens x 128 rows where pairs of row blocks need two, pairs where they need one as well
    assert tile(4736, 1024, 0, SMS) == tile(1664, 2728, 0, SMS) == tile(1152, 4056, 0, SMS) == 256
    assert tile(9472, 512, 0, SMS) == 128
    assert {tile(M, T, 1, SMS) for M in (128, 5120, 17408) for T in (128, 256, 1000, 2048)} <= {128, 192, 256}
    assert tile(100, 128, 0, SMS) == tile(128, 120, 0, SMS) == tile(128, 132, 0, SMS) == -1


@pytest.fixture(scope="module")
def lib_host(pkg):
    return pkg.load()


@pytest.mark.gpu
@pytest.mark.parametrize("wrong_sums", [False, True])
@pytest.mark.parametrize("mode", ["block_k32", "block_k64", "w4a4"])
@pytest.mark.parametrize("width", SIZES)
def test_all_codes_at_every_width(lib, pkg, orc, wl, width, mode, wrong_sums):
    M, T = SIZES[width]
    int4, ksh = mode == "w4a4", int(mode != "block_k32")
    codes, scales = wl.random_packed_weight(M, K, seed=width, ksh=ksh)
    w = pkg.PackedWeight(codes, scales, M, K, k64=bool(ksh))
    rng = np.random.default_rng(width)
    n = K // (64 if int4 else 32) * T
    q = rng.integers(0, 256, size=n * 32, dtype=np.uint8)
    if int4:
        values = (np.stack((q & 15, q >> 4), -1).astype(np.int32) ^ 8) - 8
    else:
        q = q.view(np.int8)
        values = q.astype(np.int32)
    sm = values.reshape(n, -1).sum(1, dtype=np.int32)
    if wrong_sums:
        sm[rng.random(n) < 1e-3] += 5
        sm[-1] -= 3
    s = (rng.random(n, dtype=np.float32) * 0.05).astype(np.float32)
    if int4:
        rc, want = orc.gemm_w4a4(codes, scales, M, K, q, s, sm, T, fma=1)
    else:
        rc, want = orc.gemm_w4a8(codes, scales, M, K, ksh, q, s, sm, T, fma=1)
    assert rc == 0
    dq, ds, dsm = (pkg.DevBuf.from_numpy(np.ascontiguousarray(v)) for v in (q, s, sm))
    y = pkg.DevBuf(T * M * 4)
    for _ in range(2):
        y.fill(0xA5)
        if int4:
            assert lib.qwn_x_gemm_w4a4(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr, T) == 0
        else:
            assert lib.qwn_x_gemm_w4a8(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr, T, None, 0) == 0
        lib.tq_sync()
        assert lib.tq_last_error() == 0
        assert y.to_numpy(np.float32).tobytes() == np.ascontiguousarray(want, dtype=np.float32).tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["block_k32", "block_k64", "token_k32", "token_k64", "w4a4"])
def test_largest_sums_are_exact(lib, pkg, mode):
    """The largest sums that a group can have (weights of -15 or 15, activations of -128, in 4 bits -8) with a few terms of
    1 among them: an accumulator that dropped a bit of theirs would show, for with scales of 1 every result is an
    integer below 2^24."""
    M, K, T = 2048, 192, 136
    int4, ksh = mode == "w4a4", int(not mode.endswith("k32"))
    if mode.startswith("block"):
        assert pkg.load().qwn_choose_gemm_splits(M // 16, T // 8, K // 32) == 1
    rows, toks, ks = np.arange(M)[:, None], np.arange(T)[:, None], np.arange(K)[None, :]
    # even rows: zero point 7, codes -8 (-15) and 6 (-1); odd rows: zero point -8, codes 7 (15) and -7 (1)
    z = np.where(rows % 2 == 0, 7, -8)
    one_w = (rows + ks) % 61 == 0
    q = np.where(rows % 2 == 0, np.where(one_w, 6, -8), np.where(one_w, -7, 7))
    one_a = (3 * toks + ks) % 37 == 0
    a = np.where(one_a, np.where(ks % 2 == 0, 1, -1), -8 if int4 else -128)
    want = a.astype(np.int64) @ (q - z).astype(np.int64).T
    assert np.abs(want).max() > K * 15 * (8 if int4 else 128) * 0.9 and np.abs(want).max() < 2 ** 24
    n = (q & 15).astype(np.uint8).reshape(M // 16, 16, K // 32, 16, 2).transpose(0, 2, 1, 3, 4)
    codes = n[..., 0] | (n[..., 1] << 4)
    grp = 64 if ksh else 32
    word = (0x3C00 | (z & 15)).astype(np.uint16)          # fp16 1.0 with the zero point in its low nibble
    scales = np.broadcast_to(word.reshape(M // 16, 1, 16), (M // 16, K // grp, 16))
    w = pkg.PackedWeight(codes, np.ascontiguousarray(scales), M, K, k64=bool(ksh))
    blk = 64 if int4 else 32
    ab = a.reshape(T, K // blk, blk).transpose(1, 0, 2)
    sm = ab.sum(2).astype(np.int32)
    if int4:
        nib = (ab & 15).astype(np.uint8).reshape(K // 64, T, 32, 2)
        staged = nib[..., 0] | (nib[..., 1] << 4)
    else:
        staged = ab.astype(np.int8)
    dq, ds, dsm, dat = (pkg.DevBuf.from_numpy(np.ascontiguousarray(v))
                        for v in (staged, np.ones(sm.size, np.float32), sm, np.ones(T, np.float32)))
    y = pkg.DevBuf(T * M * 4)
    if int4:
        assert lib.qwn_x_gemm_w4a4(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr, T) == 0
    elif mode.startswith("token"):
        assert lib.qwn_x_gemm_w4a8_pertoken(w.ref, dq.ptr, dat.ptr, dsm.ptr, y.ptr, T, 0) == 0
    else:
        assert lib.qwn_x_gemm_w4a8(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr, T, None, 0) == 0
    lib.tq_sync()
    assert lib.tq_last_error() == 0
    assert np.array_equal(y.to_numpy(np.float32).reshape(T, M), want.astype(np.float32))
