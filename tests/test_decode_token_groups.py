"""Per-token decode batches of 3, 5, 6 and 7 eight-token groups: all of a call's tokens on one warp
(gemm_w4a8_ring_kernel) where a call has many row groups, windows of tokens on CTA columns where it
has few. Bit-identical to the oracle: integer dots, then the same fp32 operations in the same order."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("T", [24, 40, 48, 56])
@pytest.mark.parametrize("Ms,K,ksh", [
    ([5120], 1088, 0),          # many row groups: more tasks than warps
    ([5120], 1088, 1),
    ([1040, 1040, 1040], 1088, 0),   # 16 splits of 2 or 3 k-tiles; 48 tokens in windows of 24
    ([16], 64, 1),              # one row group, one K64 group: windows of 8 or 16
    ([272], 2112, 0),           # windows, 4 or 5 k-tiles a split
    ([48, 16], 4160, 1),        # windows, splits of unequal length
    ([2064, 48], 4160, 1),      # one warp, splits of unequal length
    ([40976], 64, 1),           # one warp, one K64 group
])
def test_pertoken_token_groups(lib, pkg, orc, wl, Ms, K, ksh, T):
    host = [wl.random_packed_weight(M, K, seed=M + K + T + i, ksh=ksh) for i, M in enumerate(Ms)]
    ws = [pkg.PackedWeight(c, s, M, K, k64=bool(ksh)) for (c, s), M in zip(host, Ms)]
    x = wl.activations_normal(T, K, seed=T + K, outlier_frac=0.01)
    oq, os_, osm = orc.quantize_act_chunk(x, per_token=True)
    at = np.ascontiguousarray(os_.reshape(K // 32, T)[0])
    aq, dat, dsm = (pkg.DevBuf.from_numpy(np.ascontiguousarray(a)) for a in (oq, at, osm))
    ys = [pkg.DevBuf(T * M * 4) for M in Ms]
    for rep in range(2):        # the arrival counters are back at zero after a call
        for yb in ys:
            yb.fill(0xA5)
        assert lib.qwn_x_gemm_w4a8_fanout_pertoken(pkg.weight_array(ws), pkg.ptr_array(ys), len(Ms), aq.ptr,
                                                   dat.ptr, dsm.ptr, T) == 0
        lib.tq_sync()
        S = max(lib.qwn_choose_pertoken_splits(M // 16, T // 8, K // 32, ksh) for M in Ms)
        for (c, s), M, yb in zip(host, Ms, ys):
            _, want = orc.gemm_w4a8_pertoken(c, s, M, K, ksh, oq, at, osm, T, splits=S)
            assert yb.to_numpy(np.float32).tobytes() == np.ascontiguousarray(want, dtype=np.float32).tobytes()
    assert lib.tq_last_error() == 0
