"""Decode batches of 16 to 64 tokens in the reference's arithmetic (csrc/gemm_batch.cu): two to eight token
groups a warp, up to 12 and up to 16 warps, activations of a split in one piece and in phases, split and unsplit sums,
several rounds of tasks, ranges of tasks that end inside a row-group, K ranges that are no multiple of a chunk of
eight k-tiles, a split whose last phase is empty, several weights, and buffers that do not allow 16-byte copies (the
other kernels). Every case states the plan that it runs by, and test_plans() that the plans reach every form. Every
output word equals the oracle's: dots are exact integers, the fp32 sums keep their order."""
import ctypes as C

import numpy as np
import pytest

SMS = 148
# (rows of each weight, K, tokens, K64 groups, offset of the activation buffers in bytes): token groups a warp, 16
# warps, warps, rounds, splits, phases, k-tiles of a phase, with aligned buffers; None: another kernel's call
CASES = {
    ((4112,), 2784, 64, 0, 0): (2, 0, 7, 1, 1, 1, 88),
    ((17424,), 2816, 64, 1, 0): None,
    ((1040,), 1056, 64, 0, 0): (2, 0, 8, 1, 4, 1, 16),
    ((16,), 256, 64, 0, 0): (2, 0, 4, 1, 8, 1, 8),
    ((2048, 2048), 1024, 64, 1, 0): (4, 0, 7, 1, 2, 1, 16),
    ((5120,), 416, 56, 0, 0): None,
    ((528,), 1056, 56, 0, 0): (7, 0, 4, 1, 16, 1, 8),
    ((3008,), 4032, 56, 1, 0): None,
    ((17424,), 192, 48, 1, 0): (6, 0, 8, 1, 1, 1, 8),
    ((1040, 1040), 1056, 48, 0, 0): (6, 0, 8, 1, 8, 1, 8),
    ((10240,), 3040, 48, 0, 0): None,
    ((272,), 2080, 40, 0, 0): None,
    ((3008,), 1504, 40, 0, 0): (5, 0, 6, 1, 4, 1, 16),
    ((8192,), 2048, 32, 0, 0): (2, 0, 7, 1, 1, 1, 64),
    ((4096, 4096), 608, 32, 0, 0): (4, 0, 7, 1, 2, 1, 16),
    ((17408,), 64, 32, 1, 0): (4, 0, 8, 1, 1, 1, 8),
    ((2064, 2064, 2064), 1056, 24, 0, 0): (3, 0, 11, 2, 8, 1, 8),
    ((10928,), 7392, 24, 0, 0): None,
    ((64,), 512, 24, 1, 0): None,
    ((5120,), 1088, 16, 1, 0): (2, 0, 9, 1, 4, 1, 16),
    ((4096,), 992, 16, 0, 0): (2, 0, 7, 1, 4, 1, 8),
    ((10240,), 1184, 16, 0, 0): (2, 0, 9, 1, 2, 1, 24),
    ((1040,), 1056, 64, 0, 8): (2, 0, 8, 1, 4, 1, 16),
    ((2064, 2064), 1056, 24, 0, 8): (3, 1, 15, 1, 8, 1, 8),
    # in phases
    ((1024,), 11328, 64, 0, 0): (2, 0, 7, 1, 4, 3, 40),
    ((1408,), 14400, 48, 1, 0): (2, 0, 8, 1, 4, 3, 56),
    ((4096,), 2944, 64, 0, 0): (2, 0, 7, 1, 1, 3, 40),
    ((10672,), 14368, 24, 0, 0): (3, 0, 10, 1, 2, 3, 112),
    ((6336, 6336, 6336), 14912, 24, 0, 0): (3, 0, 9, 2, 2, 3, 112),
    ((15744,), 7488, 24, 0, 0): (3, 0, 7, 1, 1, 3, 112),
    ((8288, 8288), 14368, 24, 0, 0): (3, 1, 14, 1, 2, 3, 112),
    ((2160, 2160), 5152, 64, 0, 0): (4, 0, 8, 1, 2, 3, 40),
    ((12832, 12832, 12832), 5472, 32, 0, 0): (4, 0, 9, 2, 1, 3, 80),
    ((4800, 4800, 4800), 11264, 32, 0, 0): (4, 1, 13, 1, 2, 3, 80),
    ((3472, 3472), 12320, 40, 0, 0): (5, 0, 6, 1, 2, 4, 64),
    ((4800, 4800, 4800), 8960, 40, 1, 0): (5, 0, 7, 2, 2, 3, 64),
    ((4288, 4288), 7200, 48, 0, 0): (6, 0, 8, 1, 2, 3, 56),
    ((5152, 5152, 5152), 7360, 48, 1, 0): (6, 0, 7, 2, 2, 3, 56),
    ((1344, 1344), 12352, 56, 1, 0): (7, 0, 5, 1, 4, 3, 48),
    ((9616, 9616, 9616), 3136, 56, 1, 0): (7, 0, 7, 2, 1, 3, 48),
    ((2512, 2512, 2512), 7712, 64, 0, 0): (8, 0, 7, 1, 2, 4, 40),
    ((11936, 11936, 11936), 2688, 64, 1, 0): (8, 0, 8, 2, 1, 3, 40),
    # few k-tiles: rounds of tasks, 16 warps
    ((2320, 2320, 2320), 256, 24, 0, 0): (3, 1, 13, 2, 8, 1, 8),
    ((14224, 14224), 64, 24, 0, 0): None,
    ((1936, 1936, 1936), 256, 16, 1, 0): (2, 0, 11, 2, 8, 1, 8),
    ((16384, 16384), 64, 16, 1, 0): (2, 0, 7, 2, 1, 1, 8),
    ((9488, 9488, 9488), 64, 32, 1, 0): (4, 1, 13, 1, 1, 1, 8),
    ((1744, 1744), 256, 32, 0, 0): (4, 1, 13, 1, 8, 1, 8),
    ((784, 784, 784), 256, 64, 0, 0): (8, 0, 9, 1, 8, 1, 8),
    # few row-groups, long K: the windows of the other kernels are as fast or faster
    ((11456,), 16960, 24, 1, 0): None,
    ((912,), 6464, 40, 1, 0): None,
    ((14880,), 7008, 16, 0, 0): None,
}


def plan(pkg, rows, K, T, ksh, sms=SMS):
    out = (C.c_int * 7)()
    rc = pkg.load().qwn_dbg_batch_plan((C.c_int * len(rows))(*rows), len(rows), K, T, ksh, sms, out)
    assert rc in (0, 1)
    return tuple(out) if rc else None


def last_phase_empty(K, splits, phases, P):
    kt = K // 32
    spans = [kt * (s + 1) // splits - kt * s // splits for s in range(splits)]
    return phases > 1 and min(-(-n // P) for n in spans) < phases


def test_plans(pkg):
    forms, seen = {(2, 0), (3, 0), (3, 1), (4, 0), (4, 1), (5, 0), (6, 0), (7, 0), (8, 0)}, set()
    for (rows, K, T, ksh, off), want in CASES.items():
        got = plan(pkg, rows, K, T, ksh)
        assert got == want, (rows, K, T, ksh, got)
        if got is None or off:
            continue
        ntg, wide, warps, rounds, splits, phases, P = got
        kind = "phases" if phases > 1 else "whole"
        seen |= {(ntg, wide, kind), (kind, "split" if splits > 1 else "unsplit"), (kind, "one" if rounds == 1 else "rounds"),
                 ("form", wide, rounds > 1), ("splits and rounds", kind, splits > 1 and rounds > 1)}
        if last_phase_empty(K, splits, phases, P):
            seen |= {(ntg, "empty")}
    for form in forms:
        assert {(*form, "whole"), (*form, "phases")} <= seen, form
    for kind in ("whole", "phases"):
        assert {(kind, "split"), (kind, "unsplit"), (kind, "one"), (kind, "rounds"), ("splits and rounds", kind, True)} <= seen
    assert {(n, "empty") for n in range(2, 9)} <= seen
    assert plan(pkg, [5120], 17408, 64, 0)[5] > 1 and plan(pkg, [17408], 17408, 64, 0)[0] == 8
    assert plan(pkg, [5120], 17408, 8, 0) is None and plan(pkg, [5120], 17408, 72, 0) is None


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
