"""int8 output head on decode batches (csrc/w8a8.cu): the kernel that stages a window's activations in
shared memory, in all its forms (8, 16 or 32 tokens a warp, 16 or 28 warps), at tails of its register
batches, in several rounds of row-groups and with a last window that is not full, and the general kernel where the
activations do not fit or do not allow the copies, or where it is the faster one. Every output word equals the oracle's: the dots are exact integers and the
fp32 sums keep the order of the k-tiles."""
import ctypes as C

import numpy as np
import pytest

CASES = [
    (16, 32, 8, 0), (48, 160, 8, 0), (272, 416, 16, 0), (1040, 288, 32, 0), (1040, 288, 40, 0), (80, 96, 64, 0),
    (38400, 96, 8, 0), (38400, 160, 16, 0), (38400, 224, 32, 0),       # 17 row-groups per SM: 28 warps
    (66320, 96, 24, 0), (80000, 64, 16, 0),                            # several rounds
    (1040, 288, 600, 0),                                               # more tokens than a decode batch
    (32, 25856, 8, 0), (32, 12960, 16, 0),                             # too long to stage; staged one group at a time
    (272, 416, 16, 4),                                                 # activations off 16 bytes
    (66320, 96, 8, 0),                                                 # two rounds against one of the general kernel
]
# M, K, tokens: groups of 8 tokens a warp, windows, CTAs a window, warps, rounds on 148 SMs, where the last window
# is not full
RAGGED = {
    (38400, 96, 24): (4, 1, 148, 17, 1), (20000, 224, 56): (4, 2, 74, 17, 1), (66320, 160, 40): (4, 2, 74, 19, 3),
    (32000, 160, 24): (4, 1, 148, 14, 1), (8192, 416, 104): (4, 4, 37, 14, 1),
    (8192, 288, 40): (2, 3, 49, 11, 1), (20000, 96, 40): (2, 3, 49, 26, 1),
}


def plan(pkg, M, K, T, sms=148):
    out = (C.c_int * 5)()
    assert pkg.load().qwn_dbg_head_plan(M, K, T, sms, out) == 0
    return tuple(out)


def test_plans(pkg):
    for case, want in RAGGED.items():
        assert plan(pkg, *case) == want and case[2] // 8 % want[0]
    # an odd number of token groups is no reason for windows of one group, nor many windows for idle SMs
    for T in range(16, 2048, 8):
        ntg, windows, ctas, warps, rounds = plan(pkg, 65536, 5120, T)
        assert ntg > 1 and windows == -(-T // (8 * ntg)) and windows * ctas > 148 / 2 and warps <= 28
    # 8 tokens: one round of the general kernel's tasks against two rounds of the staged one
    assert plan(pkg, 65536, 5120, 8) == (1, 1, 148, 28, 1)
    assert plan(pkg, 66320, 5120, 8) == plan(pkg, 75776, 5120, 8) == (0, 0, 0, 0, 0)
    assert plan(pkg, 75792, 5120, 8) == (1, 1, 148, 17, 2)


@pytest.mark.gpu
@pytest.mark.parametrize("M,K,T,off", CASES + [(*c, 0) for c in RAGGED])
def test_head_equals_the_oracle(lib, pkg, orc, M, K, T, off):
    rng = np.random.default_rng(M + K + T)
    codes = rng.integers(-127, 128, size=M * K, dtype=np.int8)
    scales = (rng.random(M * (K // 32)) * 0.01).astype(np.float16)
    q = rng.integers(-127, 128, size=K * T, dtype=np.int8)
    s = (rng.random(K // 32 * T) * 0.1).astype(np.float32)
    rc, want = orc.gemm_w8a8(codes.view(np.uint8), scales.view(np.uint16), M, K, q, s, T, fma=1)
    assert rc == 0
    dc, dsc, ds = (pkg.DevBuf.from_numpy(v) for v in (codes, scales, s))
    dq = pkg.DevBuf.from_numpy(np.concatenate([np.zeros(off, np.int8), q]))
    w = pkg.TqWeight()
    w.M, w.K, w.Mt, w.Kt = M, K, M // 16, K // 32
    w.d_s8, w.d_s8_scale, w.s8_ready = dc.ptr, dsc.ptr, 1
    y = pkg.DevBuf(T * M * 4 + 4)
    y.fill(0xA5)
    assert lib.qwn_x_gemm_w8a8(C.byref(w), dq.ptr + off, ds.ptr, y.ptr, T) == 0
    lib.tq_sync()
    assert lib.tq_last_error() == 0
    raw = y.to_numpy(np.uint8)
    assert raw[:T * M * 4].tobytes() == np.ascontiguousarray(want, dtype=np.float32).tobytes()
    assert (raw[T * M * 4:] == 0xA5).all()
