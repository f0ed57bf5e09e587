"""The FP64 tensor-core products and transforms where their digits do not fit: panels of N and of K
and chunks of fields under a small "digits_mb", the FMA and cuFFT routes with none, and a device
with too little memory left -- against the oracle and the FMA route (option gemm_tc)."""
import subprocess
import sys
import textwrap

import numpy as np
import pytest

import oracle
from thcpp_gb300 import capi

pytestmark = pytest.mark.gpu

MESH = (20, 21, 22)          # three edges, one odd; N_c 5040 is over the long rows' 4096


def _noise(nmu, norb, seed):
    r = np.random.default_rng(seed)
    ng = int(np.prod(MESH))
    phi = r.standard_normal((ng, norb))
    return phi, np.sort(r.choice(ng, nmu, replace=False)).astype(np.int32), r


def _kernel(r, kind):
    """v(G): v(-G) = v(G), no symmetry at all, or both signs."""
    v = r.uniform(0.2, 2.0, MESH)
    if kind != "any":
        flip = v
        for ax in range(3):
            flip = np.roll(np.flip(flip, ax), 1, ax)
        v = 0.5 * (v + flip)
    if kind == "signed":
        n = [np.arange(m) for m in MESH]
        sign = [np.minimum(a, m - a) for a, m in zip(n, MESH)]
        v = v * np.where((sign[0][:, None, None] + sign[1][:, None] + sign[2]) % 5 == 2, -1.0, 1.0)
    return np.ascontiguousarray(v.reshape(-1))


def _rel(a, b):
    a, b = (x[..., 0] + 1j * x[..., 1] if x.dtype == float else x for x in (a, b))
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _with(ctx, opts, call):
    for k, v in opts.items():
        ctx.set_option(k, v)
    try:
        return call()
    finally:
        ctx.set_option("digits_mb", 3072)
        ctx.set_option("gemm_tc", 1)
        ctx.set_option("refine", 0)


# 3072: one panel.  2: ten panels of N for zeta, six of K for M (one side cut, or two where the
# weights have both signs), and chunks of a few fields.  0.25: less than the smallest panels of
# some products, which stay on the FMAs.  0: none.
@pytest.mark.parametrize("kind", ["even", "any", "signed"])
@pytest.mark.parametrize("mb", [3072, 2, 0.25, 0])
def test_panels(gpu_ctx_fp64, kind, mb):
    nmu = 200
    phi, idx, r = _noise(nmu, 24, 11)
    v = _kernel(r, kind)
    pm = phi[idx]
    tol = np.sqrt(nmu) * np.linalg.cond((pm @ pm.T) ** 2) * np.finfo(float).eps
    call = lambda: gpu_ctx_fp64.isdf(phi, idx, MESH, v, raise_on_error=False)
    got = _with(gpu_ctx_fp64, {"digits_mb": mb}, call)
    fma = _with(gpu_ctx_fp64, {"gemm_tc": 0}, call)
    assert got["status"] == fma["status"] == (capi.THC_OK if kind == "even" else fma["status"])
    assert got["stats"].n_anti == fma["stats"].n_anti and (got["stats"].n_anti > 0) == (kind == "any")
    assert _rel(got["M"], fma["M"]) < tol
    assert _rel(got["M"], oracle.isdf_real(phi, idx, np.array(MESH), v)["M"]) < tol


@pytest.mark.parametrize("mb", [3072, 2])
def test_non_finite_value_in_a_late_panel(gpu_ctx_fp64, mb):
    phi, idx, r = _noise(200, 24, 12)
    g = int(np.setdiff1d(np.arange(len(phi)), idx)[-1])
    phi[g, 3] = np.nan
    got = _with(gpu_ctx_fp64, {"digits_mb": mb}, lambda: gpu_ctx_fp64.isdf(
        phi, idx, MESH, np.ones(len(phi)), raise_on_error=False))
    assert got["status"] == capi.THC_ERR_NOT_PD and not np.isfinite(got["M"][..., 0]).any()
    zeta_ok = _with(gpu_ctx_fp64, {"gemm_tc": 0}, lambda: gpu_ctx_fp64.isdf(
        phi, idx, MESH, np.ones(len(phi)), raise_on_error=False))
    assert zeta_ok["status"] == got["status"]


@pytest.mark.parametrize("mb", [3072, 2])
def test_refined_shifted_solve(gpu_ctx_fp64, mb):
    """More points than pair products: the shift, and two refinement steps, whose products have a
    factor and add to a matrix (alpha, beta)."""
    nmu = 300
    phi, idx, _ = _noise(nmu, 16, 13)
    call = lambda: gpu_ctx_fp64.isdf(phi, idx, MESH, np.ones(len(phi)), raise_on_error=False)
    got = _with(gpu_ctx_fp64, {"digits_mb": mb, "refine": 2}, call)
    fma = _with(gpu_ctx_fp64, {"gemm_tc": 0, "refine": 2}, call)
    assert got["stats"].rank_deficient == fma["stats"].rank_deficient == 1
    # The shift is 1e-10 of the mean of C's diagonal, whose largest eigenvalue is below N_mu of it.
    assert _rel(got["M"], fma["M"]) < 1e10 * nmu * np.finfo(float).eps


@pytest.mark.parametrize("mb", [3072, 2, 0])
def test_complex_forms(gpu_ctx_fp64, mb):
    nmu = 150
    phi, idx, r = _noise(nmu, 20, 14)
    phi = phi + 1j * r.standard_normal(phi.shape)
    occ = np.ascontiguousarray(phi[:, :12])
    v = _kernel(r, "any")
    pm, po = phi[idx], occ[idx]
    cond = np.linalg.cond((po.conj() @ po.T) * (pm.conj() @ pm.T).conj())
    tol = np.sqrt(nmu) * cond * np.finfo(float).eps
    call = lambda: gpu_ctx_fp64.isdf_half_complex(phi, occ, idx, MESH, v)
    got = _with(gpu_ctx_fp64, {"digits_mb": mb}, call)
    fma = _with(gpu_ctx_fp64, {"gemm_tc": 0}, call)
    assert _rel(got["M"], fma["M"]) < 2 * tol
    assert _rel(got["M"], oracle.isdf_half_reference(phi, occ, idx, np.array(MESH), v)) < 2 * tol
    tol = np.sqrt(nmu) * np.linalg.cond(np.abs(pm.conj() @ pm.T) ** 2) * np.finfo(float).eps
    call = lambda: gpu_ctx_fp64.isdf_complex(phi, idx, MESH, v)
    got = _with(gpu_ctx_fp64, {"digits_mb": mb}, call)
    fma = _with(gpu_ctx_fp64, {"gemm_tc": 0}, call)
    assert _rel(got["M"], fma["M"]) < tol


_SHORT = """
    import numpy as np, torch
    from thcpp_gb300 import capi
    mesh, nmu, norb = (48, 48, 48), 256, 32
    ng = 48 ** 3
    gen = torch.Generator(device="cuda").manual_seed(5)
    phi = torch.randn(ng, norb, dtype=torch.float64, device="cuda", generator=gen)
    idx = torch.arange(nmu, dtype=torch.int32, device="cuda") * 431
    v = torch.ones(ng, dtype=torch.float64, device="cuda")
    M = torch.zeros(nmu, nmu, 2, dtype=torch.float64, device="cuda")
    ctx = capi.Context(0, capi.THC_PREC_FP64)
    # Enough for Z, zeta, its spectrum and cuFFT's work area (0.8 GB), not for the transforms' chunk.
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (MB << 20), dtype=torch.uint8, device="cuda")
    r = ctx.isdf(phi, idx, mesh, v, out_M=M, want=())
    short = M.clone()
    ctx.close()
    del hold
    torch.cuda.empty_cache()
    ctx = capi.Context(0, capi.THC_PREC_FP64)
    ctx.set_option("gemm_tc", 0)
    ctx.isdf(phi, idx, mesh, v, out_M=M, want=())
    pm = phi[idx.long()]
    tol = nmu ** 0.5 * float(torch.linalg.cond((pm @ pm.T) ** 2)) * 2.2e-16
    err = float((short - M).norm() / M.norm())
    assert r["status"] == 0 and err < tol, (r["status"], err, tol)
    print("done")
"""


# 1400 and 1100 MB leave some digits for the products, 950 the call's own arrays and little else.
@pytest.mark.parametrize("mb", [1400, 1100, 950])
def test_little_memory_left(lib, mb):
    """In a process of its own, where nothing is kept from earlier calls."""
    code = textwrap.dedent(_SHORT).replace("MB", str(mb))
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "done" in out.stdout, out.stderr[-2000:]
