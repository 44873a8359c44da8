"""RMSNorm + quantiser of one row: the cluster kernel at every cluster size, its longest row, the
first row that the two-kernel path takes, and a call in place. Bit-identical to the oracle."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("in_place", [False, True])
@pytest.mark.parametrize("H", [32, 256, 288, 1024, 1056, 2048, 5120, 8192, 8224, 17408])
def test_rmsnorm_quant_rows(lib, pkg, orc, H, in_place):
    rng = np.random.default_rng(H)
    x = (rng.standard_normal(H) * 3).astype(np.float32)
    w = ((rng.standard_normal(H) * 0.1).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
    dx, dw = pkg.DevBuf.from_numpy(x), pkg.DevBuf.from_numpy(w)
    out = dx if in_place else pkg.DevBuf(H * 4)
    lib.qwn_x_rmsnorm_quant(out.ptr, dx.ptr, dw.ptr, H, 1e-6)
    dq, ds, dsm = pkg.DevBuf(H), pkg.DevBuf(H // 32 * 4), pkg.DevBuf(H // 16 * 4)
    assert lib.qwn_dbg_prepared_act(H, dq.ptr, ds.ptr, dsm.ptr) == 0
    lib.tq_sync()
    q, s, sm = dq.to_numpy(np.int8), ds.to_numpy(np.float32), dsm.to_numpy(np.int32)
    oo, oq, os_, osm = orc.rmsnorm_quant(x, w, 1e-6)
    assert out.to_numpy(np.float32).tobytes() == oo.tobytes()
    assert np.array_equal(q, oq) and s.tobytes() == os_.tobytes() and np.array_equal(sm, osm)
    assert lib.tq_last_error() == 0
