"""Error paths of the C ABI on the GPU, made without faulting anything.

* A bounded device wait that runs out: the context option "spin_limit" = 0 makes every
  mbarrier wait of the tensor-core GEMM give up at once (before any copy or MMA is issued);
  the call returns THC_ERR_TIMEOUT and the next call on the same context is exact again.
* Cholesky breakdowns reported the way the reference reports them: THC_ERR_NOT_PD for M
  (the reference prints the failed minor and still writes Luv,
  src/interpolating_vectors.cpp:296-304) and for a singular C solved without a shift.
"""
import numpy as np
import pytest

import oracle
from thcpp_gb300 import capi
from tests.conftest import system

pytestmark = pytest.mark.gpu


def _cplx(a):
    return a[..., 0] + 1j * a[..., 1]


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def test_device_wait_timeout_is_reported_and_context_stays_usable(gpu_ctx_mixed):
    s = system("tiny")
    idx = oracle.kmeans_system(s).idx
    gpu_ctx_mixed.set_option("spin_limit", 0)
    try:
        r = gpu_ctx_mixed.isdf(s.phi, idx, s.mesh, s.coulG, raise_on_error=False)
        assert r["status"] == capi.THC_ERR_TIMEOUT
        assert "timed out" in gpu_ctx_mixed.lib.thc_ctx_last_error(gpu_ctx_mixed.h).decode()
    finally:
        gpu_ctx_mixed.set_option("spin_limit", 1 << 24)
    r = gpu_ctx_mixed.isdf(s.phi, idx, s.mesh, s.coulG)
    assert r["status"] == capi.THC_OK
    ref = oracle.isdf_real(s.phi, idx, s.mesh, s.coulG)
    assert _rel(_cplx(r["M"]), ref["M"]) < 1e-6


def _noise(mesh, norb, nmu, cplx=False):
    r = np.random.default_rng(norb + nmu)
    ng = int(np.prod(mesh))
    phi = r.standard_normal((ng, norb))
    if cplx:
        phi = phi + 1j * r.standard_normal((ng, norb))
    idx = np.sort(r.choice(ng, nmu, replace=False)).astype(np.int32)
    return phi, idx, np.ones(ng)


# The products on the tensor cores: from C's on (2 N_mu^2 N_o >= 4e7, the one whose result the
# call judges half-way), from Z's on, and with the transforms (N_g N_mu >= 1e6) as products too.
@pytest.mark.parametrize("kind,mesh,norb,nmu", [
    ("real", (16, 16, 20), 64, 640), ("real", (16, 16, 18), 24, 96), ("real", (20, 24, 25), 24, 96),
    ("half", (16, 16, 20), 64, 640), ("complex", (16, 16, 20), 40, 640),
    ("half_complex", (20, 24, 25), 24, 96)])
def test_fp64_device_wait_timeout(gpu_ctx_fp64, kind, mesh, norb, nmu):
    ctx = gpu_ctx_fp64
    phi, idx, v = _noise(mesh, norb, nmu, "complex" in kind)
    occ = np.ascontiguousarray(phi[:, :norb // 2])
    call = {"real": lambda: ctx.isdf(phi, idx, mesh, v),
            "half": lambda: ctx.isdf_half(phi, occ, idx, mesh, v),
            "complex": lambda: ctx.isdf_complex(phi, idx, mesh, v),
            "half_complex": lambda: ctx.isdf_half_complex(phi, occ, idx, mesh, v)}[kind]
    before = call()["M"].copy()
    # Stale workspace: another call's C, Z and zeta, which the next one must not take for its own.
    ctx.isdf(*_noise(mesh, 8, 30)[:2], mesh, v)
    ctx.set_option("spin_limit", 0)
    try:
        with pytest.raises(capi.ThcError, match="timed out") as e:
            call()
        assert e.value.status == capi.THC_ERR_TIMEOUT
    finally:
        ctx.set_option("spin_limit", 1 << 24)
    assert np.array_equal(call()["M"], before)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_m_not_positive_definite(gpu_ctx_fp64, gpu_ctx_mixed, prec):
    """A negative Coulomb kernel makes M negative definite: THC_ERR_NOT_PD with the failed
    leading minor, and M and Luv are still written."""
    ctx = gpu_ctx_fp64 if prec == "fp64" else gpu_ctx_mixed
    s = system("tiny")
    idx = oracle.kmeans_system(s).idx
    r = ctx.isdf(s.phi, idx, s.mesh, -s.coulG, raise_on_error=False)
    assert r["status"] == capi.THC_ERR_NOT_PD
    assert r["stats"].chol_m_info == 1
    ref = oracle.isdf_real(s.phi, idx, s.mesh, -s.coulG)
    assert _rel(_cplx(r["M"]), ref["M"]) < 1e-6
    assert np.isfinite(r["L"]).all()
    ok = ctx.isdf(s.phi, idx, s.mesh, s.coulG)
    assert ok["status"] == capi.THC_OK


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_singular_c_without_shift(gpu_ctx_fp64, gpu_ctx_mixed, prec):
    """C1's C is singular (N_mu 64 > 36 pair products); shift_rel = 0 forbids the shift, so
    the Cholesky of C breaks down: THC_ERR_NOT_PD, and the automatic policy still works."""
    ctx = gpu_ctx_fp64 if prec == "fp64" else gpu_ctx_mixed
    s = system("c1")
    idx = oracle.kmeans_system(s).idx
    r = ctx.isdf(s.phi, idx, s.mesh, s.coulG, 0.0, raise_on_error=False)
    assert r["status"] == capi.THC_ERR_NOT_PD
    assert "Cholesky of C failed" in ctx.lib.thc_ctx_last_error(ctx.h).decode()
    r = ctx.isdf(s.phi, idx, s.mesh, s.coulG)
    assert r["status"] == capi.THC_OK and r["stats"].rank_deficient == 1


@pytest.mark.parametrize("bad", [-1, 1000])
def test_index_outside_the_grid(gpu_ctx_fp64, bad):
    """An interpolating index that is no grid point is reported, and never used as an address."""
    r = np.random.default_rng(1)
    phi = r.standard_normal((1000, 6)) + 1j * r.standard_normal((1000, 6))
    idx = np.array([3, 500, bad, 800], dtype=np.int32)
    with pytest.raises(capi.ThcError, match="interpolating index out of range") as e:
        gpu_ctx_fp64.isdf_half_complex(phi, np.ascontiguousarray(phi[:, :3]), idx, (10, 10, 10),
                                       np.ones(1000))
    assert e.value.status == capi.THC_ERR_ARG


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nmu", [5, 40])
@pytest.mark.parametrize("bad", [-1, 2000])
def test_initial_index_outside_the_grid(request, prec, nmu, bad):
    ctx = request.getfixturevalue("gpu_ctx_fp64" if prec == "fp64" else "gpu_ctx_mixed")
    r = np.random.default_rng(2)
    g, rho = r.uniform(size=(2000, 3)), r.uniform(0.5, 2.0, size=2000)
    init = np.arange(nmu, dtype=np.int32) * 3
    init[nmu // 2] = bad
    with pytest.raises(capi.ThcError, match="initial index out of range") as e:
        ctx.kmeans(g, rho, nmu, init, 5, 1e-9)
    assert e.value.status == capi.THC_ERR_ARG
    init[nmu // 2] = 1999
    idx, _, status = ctx.kmeans(g, rho, nmu, init, 5, 1e-9)
    assert status == capi.THC_OK and len(idx) == nmu
