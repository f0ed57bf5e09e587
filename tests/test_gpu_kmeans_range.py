"""k-means where FP32, which filters the candidates, runs out: squared distances that underflow it
in part or overflow it, cells far from the origin, coordinates and densities that are not finite --
against the oracle, bit for bit, in both precisions."""
import numpy as np
import pytest

import oracle
from thcpp_gb300 import capi

pytestmark = pytest.mark.gpu


def _check(ctx, g, rho, nmu, max_it, seed):
    init = oracle.initial_indices(len(g), nmu, seed)
    ref = oracle.kmeans(g, rho, nmu, init, max_it, 1e-9)
    idx, st, status = ctx.kmeans(g, rho, nmu, init, max_it, 1e-9, raise_on_error=False)
    # The oracle's status 2 is the reference's exit on an empty cluster.
    assert status == {0: capi.THC_OK, 2: capi.THC_ERR_EMPTY_CLUSTER}[ref.status]
    if status == 0:
        assert np.array_equal(idx, ref.idx)
        assert st.iterations == ref.iters
        assert st.final_diff == ref.diff or (np.isnan(st.final_diff) and np.isnan(ref.diff))


# From 8 centroids on the assign and the map prune; 5 take the exhaustive kernels.
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nmu", [5, 9, 40, 64, 300])
@pytest.mark.parametrize("scale,offset", [
    (1e-19, 0), (1e-20, 0), (3e-21, 0), (1e-21, 0), (3e-22, 0), (1e-22, 0), (3e-23, 0), (1e-23, 0),
    (1e18, 0), (1e19, 0), (1.0, 1e2), (1.0, -1e5), (1.0, 1e8), (1e-21, 1e-19)])
def test_scales_and_places(request, prec, nmu, scale, offset):
    ctx = request.getfixturevalue("gpu_ctx_fp64" if prec == "fp64" else "gpu_ctx_mixed")
    r = np.random.default_rng(nmu)
    g = np.ascontiguousarray(r.uniform(-3.0, 5.0, size=(6000, 3)) * scale + offset)
    _check(ctx, g, r.uniform(0.5, 2.0, size=6000), nmu, 4, 11)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nmu", [5, 40, 64])
@pytest.mark.parametrize("what,value", [("point", np.inf), ("density", np.inf), ("density", np.nan),
                                        ("density", -0.5)])
def test_values_out_of_the_ordinary(request, prec, nmu, what, value):
    ctx = request.getfixturevalue("gpu_ctx_fp64" if prec == "fp64" else "gpu_ctx_mixed")
    r = np.random.default_rng(nmu)
    g, rho = r.uniform(-3.0, 5.0, size=(3000, 3)), r.uniform(0.5, 2.0, size=3000)
    if what == "point":
        g[1500, 1] = value
    else:
        rho[1000] = value
    for max_it in (1, 6):
        _check(ctx, g, rho, nmu, max_it, 5)
