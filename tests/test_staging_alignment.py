"""Per-token staging of decode batches from buffers that do not take vector accesses (rows that start
4 bytes off, codes that start 1 byte off, bf16 weights 2 bytes off): the same words as from aligned
ones, with guard bytes around the codes."""
import numpy as np
import pytest


def _off(pkg, a, nbytes):
    raw = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
    buf = pkg.DevBuf.from_numpy(np.concatenate([np.full(nbytes, 0xA5, np.uint8), raw, np.full(16, 0xA5, np.uint8)]))
    return buf, buf.ptr + nbytes


class _Staged:
    def __init__(self, pkg, K, T, code_off):
        n = K // 32 * T
        self.n, self.off = n, code_off
        self.q, self.s, self.sm, self.at = pkg.DevBuf(n * 32 + 32), pkg.DevBuf(n * 4), pkg.DevBuf(n * 4), pkg.DevBuf(T * 4)
        self.q.fill(0xA5)
        self.args = (self.q.ptr + code_off, self.s.ptr, self.sm.ptr, self.at.ptr)

    def check(self, want, T):
        oq, os_, osm = want
        raw = self.q.to_numpy(np.uint8)
        assert raw[self.off:self.off + self.n * 32].tobytes() == np.ascontiguousarray(oq, dtype=np.int8).tobytes()
        assert (raw[:self.off] == 0xA5).all() and (raw[self.off + self.n * 32:] == 0xA5).all()
        assert self.s.to_numpy(np.float32).tobytes() == os_.tobytes()
        assert np.array_equal(self.sm.to_numpy(np.int32), osm)
        assert self.at.to_numpy(np.float32).tobytes() == os_.reshape(-1, T)[0].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("row_off,code_off", [(4, 0), (0, 1), (8, 2)])
@pytest.mark.parametrize("K,T", [(64, 8), (352, 3), (5120, 8), (17408, 8), (5120, 40), (17408, 64)])
def test_pertoken_staging_of_unaligned_buffers(lib, pkg, orc, wl, K, T, row_off, code_off):
    x = wl.activations_normal(T, K, seed=K + T, outlier_frac=0.01)
    keep, ptr = _off(pkg, x, row_off)
    st = _Staged(pkg, K, T, code_off)
    lib.qwn_x_quantize_act_chunk_pertoken(ptr, K, T, *st.args)
    lib.tq_sync()
    assert lib.tq_last_error() == 0
    st.check(orc.quantize_act_chunk(x, per_token=True), T)


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["in", "out", "w", "codes"])
def test_fused_pertoken_stagings_of_unaligned_buffers(lib, pkg, orc, which):
    K, T = 1280, 8
    rng = np.random.default_rng(1)
    x, up = (rng.standard_normal((T, K)).astype(np.float32) for _ in range(2))
    w = ((rng.standard_normal(K) * 0.1).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    (kx, px), (ku, pu), (kw, pw) = _off(pkg, x, 4 if which == "in" else 0), _off(pkg, up, 4 if which == "w" else 0), \
        _off(pkg, w, 2 if which == "w" else 0)
    out_off = 4 if which == "out" else 0
    for norm in (True, False):
        out = pkg.DevBuf(T * K * 4 + 16)
        st = _Staged(pkg, K, T, 1 if which == "codes" else 0)
        if norm:
            lib.qwn_x_rmsnorm_quant_chunk_pertoken(out.ptr + out_off, px, pw, K, T, 1e-6, *st.args, 0)
            want = orc.rmsnorm_chunk(x, w, 1e-6)
        else:
            lib.qwn_x_silu_mul_quant_chunk_pertoken(out.ptr + out_off, px, pu, K, T, *st.args)
            want = orc.silu_mul(x, up).reshape(T, K)
        lib.tq_sync()
        assert lib.tq_last_error() == 0
        assert out.to_numpy(np.uint8)[out_off:out_off + T * K * 4].tobytes() == want.tobytes()
        st.check(orc.quantize_act_chunk(want, per_token=True), T)
