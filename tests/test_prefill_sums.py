"""Which variant of the prefill GEMM does a call (csrc/gemm_tc.cu): the one that applies
z * (sum of codes - asum) only where that term enters the result, decided by each call's own data.
Callers whose weights are symmetric may leave the code sums unset, and a captured call follows the
sums of each replay."""
import numpy as np
import pytest

M, K, T = 1024, 256, 256        # unsplit, 16 tiles


def _call(lib, pkg, mode, w, d, y):
    if mode == "w4a4":
        return lib.qwn_x_gemm_w4a4(w.ref, d["q"].ptr, d["s"].ptr, d["sum"].ptr, y.ptr, T)
    if mode == "token":
        return lib.qwn_x_gemm_w4a8_pertoken(w.ref, d["q"].ptr, d["at"].ptr, d["sum"].ptr, y.ptr, T, 0)
    return lib.qwn_x_gemm_w4a8(w.ref, d["q"].ptr, d["s"].ptr, d["sum"].ptr, y.ptr, T, None, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("zp", [False, True])
@pytest.mark.parametrize("mode", ["block", "token", "w4a4"])
def test_variant_follows_the_data_of_each_call(lib, pkg, orc, wl, mode, zp):
    codes, scales = wl.random_packed_weight(M, K, seed=7, ksh=1)
    if not zp:
        scales = (scales & 0xFFF0).astype(np.uint16)
    w = pkg.PackedWeight(codes, scales, M, K, k64=True)
    x = wl.activations_normal(T, K, seed=8, outlier_frac=0.01)
    q, s, sm = orc.quantize_act_chunk_s4(x) if mode == "w4a4" else orc.quantize_act_chunk(x, per_token=mode == "token")
    at = np.ascontiguousarray(s.reshape(-1, T)[0])
    unset = np.full_like(sm, 1 << 19)
    one_off = sm.copy()
    one_off.reshape(-1)[-1] += 1
    d = {k: pkg.DevBuf.from_numpy(np.ascontiguousarray(v)) for k, v in (("q", q), ("s", s), ("sum", sm), ("at", at))}
    y = pkg.DevBuf(T * M * 4)

    def check(sums):
        got = y.to_numpy(np.float32)
        if mode == "w4a4":
            rc, want = orc.gemm_w4a4(codes, scales, M, K, q, s, sums, T, fma=1)
        elif mode == "token":
            rc, want = orc.gemm_w4a8_pertoken(codes, scales, M, K, 1, q, at, sums, T)
        else:
            rc, want = orc.gemm_w4a8(codes, scales, M, K, 1, q, s, sums, T, fma=1)
        assert rc == 0 and got.tobytes() == np.ascontiguousarray(want, dtype=np.float32).tobytes()
        differs = not np.array_equal(sums, sm)
        assert lib.qwn_dbg_prefill_sums_variant() == int(differs and zp)
        assert lib.tq_last_error() == 0

    order = (sm, one_off, sm, sm, unset, unset, sm)
    for sums in order:
        d["sum"] = pkg.DevBuf.from_numpy(np.ascontiguousarray(sums))
        y.fill(0xA5)
        assert _call(lib, pkg, mode, w, d, y) == 0
        lib.tq_sync()
        check(sums)
    assert lib.tq_graph_capture_begin() == 0
    assert _call(lib, pkg, mode, w, d, y) == 0
    g = lib.tq_graph_capture_end()
    assert g
    for sums in order:
        host = np.ascontiguousarray(sums)
        lib.tq_h2d(d["sum"].ptr, host.ctypes.data, host.nbytes)
        y.fill(0xA5)
        lib.tq_sync()
        lib.tq_graph_launch(g)
        lib.tq_sync()
        check(sums)
    lib.tq_graph_destroy(g)
