"""Prefill GEMM (csrc/gemm_tc.cu): the tile widths of the per-token mode, the other modes at the same sizes, and a
caller whose code sums are not the sums of its codes.

With per-token scales the kernel takes 128, 192 or 256 tokens a tile, by the rounds that M / 128 row blocks x token
blocks make on 148 SMs; the sizes below select each of them, with a ragged last block, a full one
and more than one round of tiles. (The other modes take tiles of their own at these sizes; test_prefill_widths.py goes
through those.) A tile is K / 64 steps; the step slots (8, 6 and 5 at the three widths per token, 4 to 8 in the other
modes) and the accumulator buffers are used in turn, so REFILL has more steps than slots, odd step counts, within one tile and
from tile to tile. Zero points are taken off the weights before the dot, so that
z * asum enters as z * sum(codes); an asum that is something else takes a form of its own. Every
output word is compared with the oracle, which reads asum as given: all terms up to the promote are
integers below 2^24 in either association, so no tolerance is needed."""
import os
import re

import numpy as np
import pytest

SIZES = [
    (5120, 128, 136),      # few row blocks
    (9472, 128, 248),      # 128 a tile per token, exactly one round
    (10240, 128, 136),     # 192 a tile, one ragged block
    (17408, 128, 256),     # 256 a tile, one full block
    (17408, 64, 320),      # several rounds: a CTA walks from tile to tile
]
# one row block; block scales need 2048 tokens and more there, or the call is split and goes elsewhere
ONE_ROW_BLOCK = {
    "block": [(128, 64, 2048), (128, 192, 2056)],
    "other": [(128, 64, 136), (128, 192, 1000)],
}
REFILL = [
    (1024, 1600, 256),     # 128 a tile, 25 steps: every slot refilled three times
    (19200, 320, 128),     # 128 a tile, two tiles of 5 steps on a CTA
    (9600, 1088, 136),     # 192 a tile, 17 steps on 6 slots
    (20480, 320, 136),     # 192 a tile, two tiles of 5 steps on a CTA
    (9600, 832, 200),      # 256 a tile, 13 steps on 5 slots
    (28544, 320, 200),     # 256 a tile, two tiles of 5 steps on a CTA
]
MODES = ["block_k32", "block_k64", "token_k32", "token_k64", "w4a4"]
CASES = [(m, s) for m in MODES for s in SIZES + ONE_ROW_BLOCK["block" if m.startswith("block") else "other"] + REFILL]


def _buf(pkg, a):
    return pkg.DevBuf.from_numpy(np.ascontiguousarray(a))


def _unfenced_releases(source):
    """Releases of a step slot in the workers (arrives on `ebar`) that no proxy fence of their own branch precedes, behind
    the last read of the slot; and the number of releases."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", source, flags=re.S)
    workers = text[text.index("if (warp < kWorkWarps)"):text.index("reg_dealloc<kRoleRegs>();")]
    reads = [m.end() for m in re.finditer(r"\bchunk\(std::integral_constant|\blds_\w+\(", workers)]
    bad, releases = [], list(re.finditer(r"mbar_arrive_if\([^;]*\bebar\b[^;]*;", workers))
    for m in releases:
        behind = workers[max(r for r in reads if r < m.start()):m.start()]
        if max(reads) > m.start():
            bad.append(m.group())                      # a read behind the release
        elif "abar" in m.group():                      # one arrive for both barriers: a group per step
            if not re.search(r"if \(kOneArrive\) fence_proxy_async_smem\(\);.*__syncwarp\(\);", behind, re.S):
                bad.append(m.group())
        else:                                          # the innermost block of the release
            if not re.search(r"fence_proxy_async_smem\(\);\s*__syncwarp\(\);\s*$", behind[behind.rindex("{"):]):
                bad.append(m.group())
    return bad, len(releases)


def test_slots_are_released_behind_a_proxy_fence():
    """The next bulk copy into a slot writes through the async proxy, so the workers' reads of it are
    fenced before the arrive that allows it (read from the source: a copy that comes too early shows
    only in the timing of some runs). Without either fence the check fails."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with open(os.path.join(root, "knivesysl-xe_b200", "csrc", "gemm_tc.cu")) as f:
        source = f.read()
    assert _unfenced_releases(source) == ([], 2)
    fences = [m.span() for m in re.finditer(r"fence_proxy_async_smem\(\);", source)]
    assert len(fences) == 2
    for a, b in fences:
        bad, n = _unfenced_releases(source[:a] + ";" + source[b:])
        assert n == 2 and len(bad) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("wrong_sums", [False, True])
@pytest.mark.parametrize("mode,size", CASES, ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_prefill_tile_widths(lib, pkg, orc, wl, mode, size, wrong_sums):
    M, K, T = size
    ksh = 0 if mode.endswith("k32") else 1
    if mode.startswith("block"):       # unsplit: the prefill kernel's
        assert lib.qwn_choose_gemm_splits(M // 16, T // 8, K // 32) == 1
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
    at = np.ascontiguousarray(s.reshape(K // 32, T)[0]) if mode.startswith("token") else None
    dat = _buf(pkg, at) if at is not None else None
    if mode == "w4a4":
        rc, want = orc.gemm_w4a4(codes, scales, M, K, q, s, sm, T, fma=1)
    elif at is not None:
        rc, want = orc.gemm_w4a8_pertoken(codes, scales, M, K, ksh, q, at, sm, T)
    else:
        rc, want = orc.gemm_w4a8(codes, scales, M, K, ksh, q, s, sm, T, fma=1)
    assert rc == 0
    want = np.ascontiguousarray(want, dtype=np.float32).tobytes()
    for _ in range(3):
        y.fill(0xA5)
        if mode == "w4a4":
            assert lib.qwn_x_gemm_w4a4(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr + off, T) == 0
        elif at is not None:
            assert lib.qwn_x_gemm_w4a8_pertoken(w.ref, dq.ptr, dat.ptr, dsm.ptr, y.ptr + off, T, 0) == 0
        else:
            assert lib.qwn_x_gemm_w4a8(w.ref, dq.ptr, ds.ptr, dsm.ptr, y.ptr + off, T, None, 0) == 0
        lib.tq_sync()
        assert lib.tq_last_error() == 0
        raw = y.to_numpy(np.uint8)
        assert raw[off:off + T * M * 4].tobytes() == want
        assert (raw[:off] == 0xA5).all() and (raw[off + T * M * 4:] == 0xA5).all()      # nothing beyond y
