"""Kernels that store into the shared memory of other CTAs of their cluster: the store waits for a
cluster barrier that every CTA passes at its entry (a CTA's shared memory exists only once it has
started). The order is read from the source; on the GPU, calls of every cluster size queued without
a pause between them are compared word by word with the oracle."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "knivesysl-xe_b200", "csrc")


def _kernels_with_peer_stores():
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for body in re.split(r"__global__", text)[1:]:
            body = body[:body.index("\n}")]
            if "st_cluster_f32(" in body:
                head = re.sub(r"void|__launch_bounds__\([^)]*\)", "", body)
                yield name, re.search(r"\w+", head).group(0), body


def test_peer_stores_follow_a_cluster_barrier():
    found = list(_kernels_with_peer_stores())
    assert len(found) >= 3
    for name, kernel, body in found:
        arrive, wait, store = (body.find(s) for s in ("cluster_arrive()", "cluster_wait()", "st_cluster_f32("))
        assert 0 <= arrive < wait < store, f"{name}: {kernel} stores into its peers before the cluster has started"
        assert "return" not in body[:wait], f"{name}: {kernel} can leave before the cluster barrier"


@pytest.mark.gpu
def test_queued_cluster_calls(lib, pkg, orc, wl):
    """Clusters of 1, 2, 4 and 8 CTAs (RMSNorm + quantiser) and of 2, 4 and 8 (per-token staging),
    each call's own outputs, 20 rounds queued back to back."""
    rows, chunks = [], []
    for H in (32, 288, 1056, 5120, 8192):
        rng = np.random.default_rng(H)
        x = (rng.standard_normal(H) * 3).astype(np.float32)
        w = ((rng.standard_normal(H) * 0.1).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)
        rows.append((H, pkg.DevBuf.from_numpy(x), pkg.DevBuf.from_numpy(w), pkg.DevBuf(H * 4), orc.rmsnorm_quant(x, w, 1e-6)[0]))
    for K, T in ((64, 3), (128, 8), (1280, 8), (5120, 8), (17408, 5)):
        x = wl.activations_normal(T, K, seed=K, outlier_frac=0.01)
        n = K // 32 * T
        bufs = [pkg.DevBuf(n * 32), pkg.DevBuf(n * 4), pkg.DevBuf(n * 4), pkg.DevBuf(T * 4)]
        chunks.append((K, T, pkg.DevBuf.from_numpy(x), bufs, orc.quantize_act_chunk(x, per_token=True)))
    for _ in range(20):
        for H, x, w, out, _want in rows:
            lib.qwn_x_rmsnorm_quant(out.ptr, x.ptr, w.ptr, H, 1e-6)
        for K, T, x, bufs, _want in chunks:
            lib.qwn_x_quantize_act_chunk_pertoken(x.ptr, K, T, *(b.ptr for b in bufs))
    lib.tq_sync()
    for H, x, w, out, want in rows:
        assert out.to_numpy(np.float32).tobytes() == want.tobytes(), H
    for K, T, x, (aq, as_, asum, _at), (oq, os_, osm) in chunks:
        assert np.array_equal(aq.to_numpy(np.int8), oq), (K, T)
        assert as_.to_numpy(np.float32).tobytes() == os_.tobytes(), (K, T)
        assert np.array_equal(asum.to_numpy(np.int32), osm), (K, T)
    assert lib.tq_last_error() == 0
