"""Decode batches of 16 to 64 tokens in the reference's arithmetic (csrc/gemm_batch.cu): two to eight token
groups a warp, activations of a split in one piece and in phases, split and unsplit sums, ranges of
tasks that end inside a row-group, K ranges that are no multiple of a chunk of eight k-tiles, several
weights, and buffers that do not allow 16-byte copies (the other kernels). Every output word equals
the oracle's: dots are exact integers, the fp32 sums keep their order."""
import ctypes as C

import numpy as np
import pytest

# rows of each weight, K, tokens, K64 groups, offset of the activation buffers in bytes
CASES = [
    ([4112], 2784, 64, 0, 0),            # unsplit, three phases
    ([17424], 2816, 64, 1, 0),           # eight groups a warp
    ([1040], 1056, 64, 0, 0), ([16], 256, 64, 0, 0), ([2048, 2048], 1024, 64, 1, 0),
    ([5120], 416, 56, 0, 0), ([528], 1056, 56, 0, 0), ([3008], 4032, 56, 1, 0),
    ([17424], 192, 48, 1, 0), ([1040, 1040], 1056, 48, 0, 0), ([10240], 3040, 48, 0, 0),
    ([272], 2080, 40, 0, 0), ([3008], 1504, 40, 0, 0),
    ([8192], 2048, 32, 0, 0), ([4096, 4096], 608, 32, 0, 0), ([17408], 64, 32, 1, 0),
    ([2064, 2064, 2064], 1056, 24, 0, 0), ([10928], 7392, 24, 0, 0), ([64], 512, 24, 1, 0),
    ([5120], 1088, 16, 1, 0), ([4096], 992, 16, 0, 0), ([10240], 1184, 16, 0, 0),
    ([1040], 1056, 64, 0, 8), ([2064, 2064], 1056, 24, 0, 8),
]


@pytest.mark.gpu
@pytest.mark.parametrize("rows,K,T,ksh,off", CASES, ids=lambda v: str(v).replace(" ", ""))
def test_batch_equals_the_oracle(lib, pkg, orc, wl, rows, K, T, ksh, off):
    rng = np.random.default_rng(sum(rows) + K + T)
    q = rng.integers(-127, 128, size=K * T, dtype=np.int8)
    s = (rng.random(K // 32 * T) * 0.05).astype(np.float32)
    sm = q.reshape(-1, 32).sum(1, dtype=np.int32)
    pad = np.zeros(off, np.uint8)
    dq, ds, dsm = (pkg.DevBuf.from_numpy(np.concatenate([pad, v.view(np.uint8)])) for v in (q, s, sm))
    weights, wants, ys = [], [], []
    for i, M in enumerate(rows):
        codes, scales = wl.random_packed_weight(M, K, seed=M + K + i, ksh=ksh)
        weights.append(pkg.PackedWeight(codes, scales, M, K, k64=bool(ksh)))
        rc, want = orc.gemm_w4a8(codes, scales, M, K, ksh, q, s, sm, T, fma=1)
        assert rc == 0
        wants.append(np.ascontiguousarray(want, dtype=np.float32).tobytes())
        ys.append(pkg.DevBuf(T * M * 4 + 4))
    out = (C.c_void_p * len(rows))(*[y.ptr for y in ys])
    for _ in range(2):      # the second call finds the split counters as the first one left them
        for y in ys:
            y.fill(0xA5)
        assert lib.qwn_x_gemm_w4a8_fanout(pkg.weight_array(weights), out, len(rows), dq.ptr + off, ds.ptr + off,
                                          dsm.ptr + off, T, None, 0) == 0
        lib.tq_sync()
        assert lib.tq_last_error() == 0
        for y, want in zip(ys, wants):
            raw = y.to_numpy(np.uint8)
            assert raw[:-4].tobytes() == want and (raw[-4:] == 0xA5).all()
