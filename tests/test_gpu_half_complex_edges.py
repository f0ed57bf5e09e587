"""The complex half-rotated form's elimination (csrc/halfc.cu, gj_step) at the edges of its
blocks of 64 columns and 4 R rows, R = 1, 2, 4, 8 by size, against the oracle's literal form, and
a singular C at its column."""
import numpy as np
import pytest

import oracle
from thcpp_gb300 import capi

pytestmark = pytest.mark.gpu


def _cplx(a):
    return a[..., 0] + 1j * a[..., 1]


def _orbitals(ng, no, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal((ng, no)) + 1j * r.standard_normal((ng, no))


@pytest.mark.parametrize("nmu", [1, 2, 5, 31, 32, 33, 65, 396, 561, 800])
def test_half_complex_sizes(gpu_ctx_fp64, nmu):
    mesh = (8, 9, 12)
    ng = int(np.prod(mesh))
    r = np.random.default_rng(nmu)
    pc = _orbitals(ng, 40, nmu)
    po = np.ascontiguousarray(pc[:, :32])
    idx = np.sort(r.choice(ng, nmu, replace=False)).astype(np.int32)
    coulG = r.uniform(0.1, 2.0, ng)
    got = gpu_ctx_fp64.isdf_half_complex(pc, po, idx, mesh, coulG)
    assert got["status"] == capi.THC_OK
    ref = oracle.isdf_half_reference(pc, po, idx, np.array(mesh), coulG)
    P, Q = pc[idx].conj() @ pc[idx].T, po[idx].conj() @ po[idx].T
    cond = np.linalg.cond(Q * P.conj())
    # Each of M's two factors carries the elimination's error, N_mu u cond(C) at most.
    err = np.linalg.norm(_cplx(got["M"]) - ref) / np.linalg.norm(ref)
    assert err < 2 * 1.2e-16 * nmu * cond + 1e-13


@pytest.mark.parametrize("nmu,col", [(1, 1), (70, 1), (70, 37), (70, 70)])
def test_half_complex_singular_column(gpu_ctx_fp64, nmu, col):
    """A point where every orbital vanishes: its row and column of C are zero."""
    mesh = (8, 9, 12)
    ng = int(np.prod(mesh))
    pc = _orbitals(ng, 24, 5)
    idx = np.arange(nmu, dtype=np.int32) * 7
    pc[idx[col - 1]] = 0.0
    with pytest.raises(capi.ThcError, match=f"singular at column {col} ") as e:
        gpu_ctx_fp64.isdf_half_complex(pc, np.ascontiguousarray(pc[:, :8]), idx, mesh, np.ones(ng))
    assert e.value.status == capi.THC_ERR_NOT_PD
