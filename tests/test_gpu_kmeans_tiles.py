"""k-means at the edges of the pruned assign, the block scan and the scatter: centroid counts
around the warps' words of 32 and beyond the shared candidate list (1024), point counts around
the 256-point tiles and 512-point blocks, flat and one-cell clouds, and values outside FP32's
range -- against the oracle, bit for bit, in both precisions."""
import numpy as np
import pytest

import oracle
from thcpp_gb300 import capi

pytestmark = pytest.mark.gpu


def _cloud(ng, kind, seed):
    r = np.random.default_rng(seed)
    g = r.uniform(-3.0, 5.0, size=(ng, 3))
    if kind == "flat":
        g[:, 2] = 0.25
    elif kind == "line":
        g[:, :2] = 1.0
    elif kind == "lattice":              # exact ties
        n = int(np.ceil(ng ** (1 / 3)))
        ax = np.arange(n, dtype=np.float64)
        g = np.stack(np.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)[:ng]
    elif kind == "huge":
        g = g * 1e25                     # squared distances overflow FP32
    elif kind == "small":
        g = g * 1e-25                    # and underflow it
    return np.ascontiguousarray(g), r.uniform(0.5, 2.0, size=ng)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("ng,nmu,kind", [
    (255, 7, "cube"), (256, 8, "cube"), (257, 9, "cube"), (511, 31, "cube"), (513, 32, "flat"),
    (1000, 33, "line"), (4097, 63, "cube"), (5000, 64, "lattice"), (5000, 255, "cube"),
    (9000, 257, "flat"), (3000, 1023, "cube"), (3000, 1100, "cube"), (20000, 1500, "lattice"),
    (2000, 48, "huge"), (2000, 48, "small"), (12000, 1100, "small")])
def test_kmeans_tile_edges(request, prec, ng, nmu, kind):
    ctx = request.getfixturevalue("gpu_ctx_fp64" if prec == "fp64" else "gpu_ctx_mixed")
    g, rho = _cloud(ng, kind, ng + nmu)
    init = oracle.initial_indices(ng, nmu, 11)
    ref = oracle.kmeans(g, rho, nmu, init, 12, 1e-9)
    idx, st, status = ctx.kmeans(g, rho, nmu, init, 12, 1e-9, raise_on_error=False)
    # The oracle's status 2 is the reference's exit on an empty cluster.
    assert status == {0: capi.THC_OK, 2: capi.THC_ERR_EMPTY_CLUSTER}[ref.status]
    if status == 0:
        assert np.array_equal(idx, ref.idx)
        assert st.iterations == ref.iters and st.final_diff == ref.diff
        diff, pct = ctx.kmeans_history(ref.iters)
        assert np.array_equal(pct, ref.pct)


@pytest.mark.parametrize("ng,nmu,clump", [
    (2048, 8, 0.0), (2500, 8, 0.9), (7500, 9, 0.95),     # members around a block's windows
    (70000, 80, 0.0), (140000, 140, 0.5),                # index ranges over 65,536
    (150000, 150, 0.98),                                 # a cluster over more than 512 tiles
    (7168, 8, 0.0), (7169, 8, 0.0),                      # mean members at the rules' two sides
    (2560, 8, 0.0), (2561, 8, 0.0)])
def test_kmeans_cluster_stretches(gpu_ctx_fp64, ng, nmu, clump):
    """Clusters at and over the buffers of the one-kernel sums: members, index range, tiles."""
    r = np.random.default_rng(ng)
    g = r.uniform(-1.0, 1.0, size=(ng, 3))
    near = r.random(ng) < clump
    g[near] = 0.9 + 0.01 * g[near]
    init = np.sort(r.choice(np.flatnonzero(~near), nmu, replace=False)).astype(np.int32)
    g = np.ascontiguousarray(g)
    rho = r.uniform(0.5, 2.0, size=ng)
    ref = oracle.kmeans(g, rho, nmu, init, 4, 1e-9)
    idx, st, status = gpu_ctx_fp64.kmeans(g, rho, nmu, init, 4, 1e-9, raise_on_error=False)
    assert status == {0: capi.THC_OK, 2: capi.THC_ERR_EMPTY_CLUSTER}[ref.status]
    if status == 0:
        assert np.array_equal(idx, ref.idx)
        assert st.iterations == ref.iters and st.final_diff == ref.diff
        diff, pct = gpu_ctx_fp64.kmeans_history(ref.iters)
        assert np.array_equal(pct, ref.pct)
