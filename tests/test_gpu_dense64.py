"""The FP64 dense kernels at the edges of their tiles: products on the tensor cores
(csrc/dgemm_tc.cu) against the oracle and the FMA route (option gemm_tc), an orbital value that
is not finite, and the Cholesky (csrc/dense64.cu) with a breakdown at every kind of position."""
import numpy as np
import pytest

import oracle
from thcpp_gb300 import capi, synth

pytestmark = pytest.mark.gpu

_SYS = {}


def _system(mesh):
    if mesh not in _SYS:
        lat, atoms = synth.diamond_supercell(1)
        s = synth.make_system(f"edge{mesh}", lat, atoms, mesh, 32, 8, 4321, 55)
        _SYS[mesh] = (s, oracle.kmeans_system(s).idx)
    return _SYS[mesh]


def _cplx(a):
    return a[..., 0] + 1j * a[..., 1]


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# Points on either side of the 128-row and 64-column tile edges; meshes whose N_g and half
# spectrum are odd, below and above a multiple of the tiles.
@pytest.mark.parametrize("mesh", [(24, 24, 24), (23, 25, 27)])
@pytest.mark.parametrize("nmu", [63, 127, 128, 129, 193, 256])
def test_isdf_tile_edges(gpu_ctx_fp64, mesh, nmu):
    s, idx_all = _system(mesh)
    idx = np.ascontiguousarray(np.sort(np.random.default_rng(nmu).permutation(idx_all)[:nmu]))
    pm = s.phi[idx]
    # A relative perturbation eps of Z and C moves zeta, and with it M, by cond(C) eps.
    tol = np.linalg.cond((pm @ pm.T) ** 2) * np.finfo(float).eps
    ref = oracle.isdf_real(s.phi, idx, s.mesh, s.coulG)
    got = {}
    for tc in (1, 0):
        gpu_ctx_fp64.set_option("gemm_tc", tc)
        try:
            got[tc] = gpu_ctx_fp64.isdf(s.phi, idx, s.mesh, s.coulG)
        finally:
            gpu_ctx_fp64.set_option("gemm_tc", 1)
        assert got[tc]["status"] == 0
        L = _cplx(got[tc]["L"])
        # The factor's backward error: n eps, for the blocked loop as for the plain one.
        assert _rel(L @ L.conj().T, _cplx(got[tc]["M"])) < nmu * np.finfo(float).eps
        assert _rel(_cplx(got[tc]["M"]), ref["M"]) < tol
    assert _rel(_cplx(got[1]["M"]), _cplx(got[0]["M"])) < tol


def test_negative_weights_and_symmetry(gpu_ctx_fp64):
    """A Coulomb kernel with both signs: the product keeps its weights on one side."""
    s, idx = _system((24, 24, 24))
    v = s.coulG * np.where(np.arange(s.ng) % 7 == 3, -0.5, 1.0)
    r = gpu_ctx_fp64.isdf(s.phi, idx, s.mesh, v, raise_on_error=False)
    ref = oracle.isdf_real(s.phi, idx, s.mesh, v)
    pm = s.phi[idx]
    tol = np.linalg.cond((pm @ pm.T) ** 2) * np.finfo(float).eps
    assert _rel(_cplx(r["M"]), ref["M"]) < tol


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_orbital(gpu_ctx_fp64, value):
    """A value that is not finite, at a point that is no interpolating point, spoils every
    interpolating vector there and so M, on either route."""
    s, idx = _system((24, 24, 24))
    phi = s.phi.copy()
    g = int(np.setdiff1d(np.arange(s.ng), idx)[100])
    phi[g, 5] = value
    for tc in (1, 0):
        gpu_ctx_fp64.set_option("gemm_tc", tc)
        try:
            r = gpu_ctx_fp64.isdf(phi, idx, s.mesh, s.coulG, raise_on_error=False)
            z = gpu_ctx_fp64.interpolating_vectors(s.ng, s.nmu) if r["status"] == 0 else None
        finally:
            gpu_ctx_fp64.set_option("gemm_tc", 1)
        assert r["status"] == capi.THC_ERR_NOT_PD and r["stats"].chol_m_info == 1
        assert z is None and not np.isfinite(r["M"][..., 0]).any()


# Positions at the edges of the Cholesky's panels (4 columns), of the warp that owns the rows
# (32) and of its blocks (64).
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("pos", [1, 3, 4, 31, 32, 36, 63, 64, 67, 127, 129])
def test_breakdown_position(gpu_ctx_fp64, gpu_ctx_mixed, prec, pos):
    """A repeated interpolating point makes C singular at that pivot, in any block."""
    ctx = gpu_ctx_fp64 if prec == "fp64" else gpu_ctx_mixed
    s, idx_all = _system((24, 24, 24))
    idx = np.ascontiguousarray(np.random.default_rng(7).permutation(idx_all)[:130])
    idx[pos] = idx[pos - 1]
    r = ctx.isdf(s.phi, idx, s.mesh, s.coulG)
    assert r["stats"].chol_c_info == pos + 1 and r["stats"].rank_deficient == 1


@pytest.mark.parametrize("kind", ["real", "half", "complex"])
def test_c_keeps_the_fma_kernels_rounding(gpu_ctx_fp64, kind):
    """C = Z[:, idx] at a size whose other products are on the tensor cores: its factor, and so the
    pivots, are the FMA route's to the last bit."""
    r = np.random.default_rng(8)
    mesh, no, nmu = (16, 16, 20), 64, 640
    phi = r.standard_normal((int(np.prod(mesh)), no))
    idx = np.sort(r.choice(len(phi), nmu, replace=False)).astype(np.int32)
    v = np.ones(len(phi))
    pivot = {}
    for tc in (1, 0):
        gpu_ctx_fp64.set_option("gemm_tc", tc)
        try:
            if kind == "half":
                got = gpu_ctx_fp64.isdf_half(phi, np.ascontiguousarray(phi[:, :40]), idx, mesh, v)
            elif kind == "complex":
                pc = phi + 1j * np.roll(phi, 7, axis=0)
                got = gpu_ctx_fp64.isdf_complex(np.ascontiguousarray(pc), idx, mesh, v)
            else:
                got = gpu_ctx_fp64.isdf(phi, idx, mesh, v)
        finally:
            gpu_ctx_fp64.set_option("gemm_tc", 1)
        assert got["status"] == 0
        pivot[tc] = got["stats"].c_min_pivot
    assert pivot[1] == pivot[0] > 0
