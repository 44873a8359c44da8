"""Prefill GEMM (csrc/gemm_tc.cu): every tile width it chooses between, and a caller whose code sums
are not the sums of its codes.

The kernel takes 128, 192 or 256 tokens a tile, by the rounds that M / 128 row blocks x token
blocks make on 148 SMs; the sizes below select each of them, with a ragged last block, a full one
and more than one round of tiles. Zero points are taken off the weights before the dot, so that
z * asum enters as z * sum(codes); an asum that is something else takes a kernel of its own. Every
output word is compared with the oracle, which reads asum as given: all terms up to the promote are
integers below 2^24 in either association, so no tolerance is needed."""
import numpy as np
import pytest

SIZES = [
    (128, 64, 136),        # one row block
    (5120, 128, 136),      # few row blocks
    (9472, 128, 248),      # 128 a tile, exactly one round
    (10240, 128, 136),     # 192 a tile, one ragged block
    (128, 192, 1000),      # one row block, three steps: an odd number of slot uses
    (17408, 128, 256),     # 256 a tile, one full block
    (17408, 64, 320),      # several rounds: a CTA walks from tile to tile
]


def _buf(pkg, a):
    return pkg.DevBuf.from_numpy(np.ascontiguousarray(a))


@pytest.mark.gpu
@pytest.mark.parametrize("wrong_sums", [False, True])
@pytest.mark.parametrize("M,K,T", SIZES)
@pytest.mark.parametrize("mode", ["block_k32", "block_k64", "token_k32", "token_k64", "w4a4"])
def test_prefill_tile_widths(lib, pkg, orc, wl, mode, M, K, T, wrong_sums):
    ksh = 0 if mode.endswith("k32") else 1
    if mode.startswith("block") and lib.qwn_choose_gemm_splits(M // 16, T // 8, K // 32) != 1:
        pytest.skip("the call is split: not the prefill kernel's")
    codes, scales = wl.random_packed_weight(M, K, seed=M + K + T, ksh=ksh)
    w = pkg.PackedWeight(codes, scales, M, K, k64=bool(ksh))
    x = wl.activations_normal(T, K, seed=T, outlier_frac=0.01)
    rng = np.random.default_rng(T)
    if mode == "w4a4":
        q, s, sm = orc.quantize_act_chunk_s4(x)
    else:
        q, s, sm = orc.quantize_act_chunk(x, per_token=mode.startswith("token"))
    if wrong_sums:         # one block in a thousand carries another sum
        sm = sm + np.where(rng.random(sm.shape) < 1e-3, 7, 0).astype(np.int32)
        sm.reshape(-1)[-1] += 3
    dq, ds, dsm = _buf(pkg, q), _buf(pkg, s), _buf(pkg, sm)
    # a result buffer whose rows start off 16 bytes in half of the cases
    off = 4 if wrong_sums else 0
    y = pkg.DevBuf(T * M * 4 + 16)
    y.fill(0xA5)
    if mode == "w4a4":
        assert lib.qwn_x_gemm_w4a4(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr + off, T) == 0
        rc, want = orc.gemm_w4a4(codes, scales, M, K, q, s, sm, T, fma=1)
    elif mode.startswith("token"):
        at = np.ascontiguousarray(s.reshape(K // 32, T)[0])
        dat = _buf(pkg, at)
        assert lib.qwn_x_gemm_w4a8_pertoken(w.ref, dq.ptr, dat.ptr, dsm.ptr, y.ptr + off, T, 0) == 0
        rc, want = orc.gemm_w4a8_pertoken(codes, scales, M, K, ksh, q, at, sm, T)
    else:
        assert lib.qwn_x_gemm_w4a8(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr + off, T, None, 0) == 0
        rc, want = orc.gemm_w4a8(codes, scales, M, K, ksh, q, s, sm, T, fma=1)
    lib.tq_sync()
    assert rc == 0 and lib.tq_last_error() == 0
    raw = y.to_numpy(np.uint8)
    assert raw[off:off + T * M * 4].tobytes() == np.ascontiguousarray(want, dtype=np.float32).tobytes()
    assert (raw[:off] == 0xA5).all() and (raw[off + T * M * 4:] == 0xA5).all()      # nothing beyond y
