"""Prefill GEMM (csrc/gemm_tc.cu) in the modes whose tiles are two row blocks high: every tile width, with
an odd number of row blocks (the last tile's second one does not exist), a ragged last token block and
more steps than step slots. The operands are e4m3 numbers that stand for the codes exactly, an int8
activation as the sum of two: the codes here are drawn from all their values, -128 and -8 too, and
the weights have every zero point. Every output word is compared with the oracle; all sums up to the
promote are exact integers, so no tolerance is needed."""
import numpy as np
import pytest

# tokens a tile -> rows, tokens
SIZES = {32: (384, 688), 48: (7552, 136), 64: (9600, 152), 80: (9600, 200), 96: (9600, 248), 112: (9600, 296),
         128: (9600, 344)}
K = 1088                # 17 steps on 6 to 8 slots
SMS = 148


def tile_tokens(M, T):
    """The kernel's choice: rounds of tiles of 256 rows over the SMs, a round counted as tokens + 26."""
    def cost(tn):
        tiles = (M + 255) // 256 * ((T + tn - 1) // tn)
        return (tiles + SMS - 1) // SMS * (tn + 26)
    return min(range(128, 31, -16), key=cost)


@pytest.mark.parametrize("width", SIZES)
def test_sizes_reach_every_width(lib_host, width):
    M, T = SIZES[width]
    assert tile_tokens(M, T) == width and M % 256 == 128 and T % width
    assert lib_host.qwn_choose_gemm_splits(M // 16, T // 8, K // 32) == 1


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
