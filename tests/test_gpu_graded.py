"""Interpolating points of very different weight: two groups of orbitals and points, the second's
amplitude s times smaller, so that C's diagonal spans s^4.  Cholesky's error bound does not see
that scaling (Demmel: with C = D K D, K of unit diagonal, D zeta is off by kappa(K) u, whatever
D), and the products of the solve, cut relative to the largest entry of a row, must not either."""
import numpy as np
import pytest

from thcpp_gb300 import capi

pytestmark = pytest.mark.gpu

MESH, NO, NMU = (20, 18, 24), 32, 128


def _fragments(s, seed):
    """phi, idx and the points' weights d = diag(C)^(1/2); d spans about 5 s^2."""
    r = np.random.default_rng(seed)
    ng = int(np.prod(MESH))
    fg = (np.arange(ng) % MESH[2]) >= MESH[2] // 2
    fo = np.arange(NO) >= NO // 2
    amp = np.where(fg[:, None] == fo[None], 1.0, 1e-3) * np.where(fo, 1.0 / s, 1.0)
    phi = r.standard_normal((ng, NO)) * amp
    idx = np.sort(np.concatenate([r.choice(np.flatnonzero(fg == f), NMU // 2, replace=False)
                                  for f in (False, True)])).astype(np.int32)
    return phi, idx, (phi[idx] ** 2).sum(1)


def _solve(c, z):
    """C X = Z by Cholesky in long double."""
    n, a, x = len(c), c.copy(), z.copy()
    for j in range(n):
        a[j:, j] /= np.sqrt(a[j, j])
        a[j + 1:, j + 1:] -= np.outer(a[j + 1:, j], a[j + 1:, j])
    for j in range(n):
        x[j] /= a[j, j]
        x[j + 1:] -= np.outer(a[j + 1:, j], x[j])
    for j in range(n - 1, -1, -1):
        x[j] /= a[j, j]
        x[:j] -= np.outer(a[j, :j], x[j])
    return x


def _tolerance(phi, idx, d):
    """kappa(K) sqrt(n) roundings."""
    k = (phi[idx] @ phi[idx].T) ** 2 / np.outer(d, d)
    return np.linalg.cond(k) * np.sqrt(NMU) * np.finfo(float).eps


# s = 1 and 30 stay on the tensor cores, balanced; at 100 and 200 the FP64 FMAs take the solve.
@pytest.mark.parametrize("s", [1, 30, 100, 200])
@pytest.mark.parametrize("seed", [0, 1])
def test_solve_is_independent_of_the_points_weights(gpu_ctx_fp64, s, seed):
    phi, idx, d = _fragments(s, seed)
    ng = len(phi)
    r = gpu_ctx_fp64.isdf(phi, idx, MESH, np.ones(ng), 0.0)
    assert r["status"] == capi.THC_OK
    zeta = gpu_ctx_fp64.interpolating_vectors(ng, NMU)
    cols = np.random.default_rng(2).choice(ng, 64, replace=False)
    pm = phi[idx].astype(np.longdouble)
    ref = _solve((pm @ pm.T) ** 2, (pm @ phi[cols].astype(np.longdouble).T) ** 2)
    err = np.linalg.norm((d[:, None] * (zeta[:, cols] - ref)).astype(float), axis=0)
    err /= np.linalg.norm((d[:, None] * ref).astype(float), axis=0)
    assert err.max() < _tolerance(phi, idx, d)


@pytest.mark.parametrize("s", [1, 30, 100])
def test_complex_half_rotated_solve(gpu_ctx_fp64, s):
    """The same system through the complex half-rotated form, all orbitals occupied: Z and C are
    the real ones, and M = sum v zeta_mu(-G) zeta_nu(G) with v = 1 is N_g zeta zeta^T.  Its
    elimination with partial pivoting does see D, so the measure is the FMA route's error."""
    phi, idx, d = _fragments(s, 3)
    pm = phi[idx]
    k, y = (pm @ pm.T) ** 2 / np.outer(d, d), (pm @ phi.T) ** 2 / d[:, None]
    y = np.linalg.solve(k, y)                       # D zeta
    ref = len(phi) * (y @ y.T)
    err = {}
    for tc in (0, 1):
        gpu_ctx_fp64.set_option("gemm_tc", tc)
        try:
            got = gpu_ctx_fp64.isdf_half_complex(phi.astype(complex), phi.astype(complex), idx,
                                                 MESH, np.ones(len(phi)))
        finally:
            gpu_ctx_fp64.set_option("gemm_tc", 1)
        assert got["status"] == capi.THC_OK
        m = got["M"][..., 0] + 1j * got["M"][..., 1]
        err[tc] = np.linalg.norm(m * np.outer(d, d) - ref) / np.linalg.norm(ref)
    assert err[1] < 2 * err[0] + 2 * _tolerance(phi, idx, d)


@pytest.mark.parametrize("binades", [-220, -100, 100, 220])
def test_orbitals_of_any_size(gpu_ctx_fp64, binades):
    """zeta does not change when all orbitals are scaled (C as the fourth power, Z with it)."""
    phi, idx, d = _fragments(30, 5)
    ng = len(phi)
    zeta = []
    for f in (1.0, 2.0 ** binades):
        r = gpu_ctx_fp64.isdf(phi * f, idx, MESH, np.ones(ng), 0.0)
        assert r["status"] == capi.THC_OK
        zeta.append(gpu_ctx_fp64.interpolating_vectors(ng, NMU))
    err = np.linalg.norm(d[:, None] * (zeta[1] - zeta[0]), axis=0)
    err /= np.linalg.norm(d[:, None] * zeta[0], axis=0)
    assert err.max() < 2 * _tolerance(phi, idx, d)
