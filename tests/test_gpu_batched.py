"""thc_factorize_batched against one-at-a-time thc_kmeans + thc_isdf (the C4 workload)."""
import numpy as np
import pytest

from thcpp_gb300 import batch, capi, synth
from tests.conftest import system

pytestmark = pytest.mark.gpu

_C4 = {}


def c4(s):
    if s not in _C4:
        _C4[s] = synth.c4_system(s)
    return _C4[s]


@pytest.mark.parametrize("prec", [capi.THC_PREC_FP64, capi.THC_PREC_MIXED])
def test_batched_matches_sequential(prec):
    import torch
    systems = [system("tiny"), c4(0), c4(1)]
    dev = torch.device("cuda", 0)
    seq = [batch.system_arrays(s, dev) for s in systems]
    bat = [batch.system_arrays(s, dev) for s in systems]
    with capi.Context(0, prec) as ctx:
        st_seq = batch.run_sequential(ctx, systems, seq)
    st, st_bat = batch.run_batched(systems, bat, prec, nstreams=2)
    torch.cuda.synchronize()
    # THC_ERR_NOT_PD (the reference's Cholesky warning on M; L is still written) is a result,
    # not a failure: an M with eigenvalues below its mixed-precision error can report it.
    assert all(x in (capi.THC_OK, capi.THC_ERR_NOT_PD) for x in st_seq)
    assert st == capi.THC_OK and st_bat == st_seq
    for s, a, b in zip(systems, seq, bat):
        assert torch.equal(a["out_idx"], b["out_idx"]), s.name
        m_a, m_b = a["out_M"].cpu().numpy(), b["out_M"].cpu().numpy()
        d = np.linalg.norm(m_a - m_b) / np.linalg.norm(m_a)
        assert d <= 1e-12, (s.name, d)
        assert torch.equal(a["out_orbitals"], b["out_orbitals"]), s.name


def test_batched_reports_per_system_errors():
    """An empty cluster in one system fails that system only."""
    import torch
    good = system("tiny")
    dev = torch.device("cuda", 0)
    a_good = batch.system_arrays(good, dev)
    bad_s = synth.config("tiny")
    bad_s.density = np.zeros_like(bad_s.density)   # every centroid weight 0
    a_bad = batch.system_arrays(bad_s, dev)
    st, per = batch.run_batched([good, bad_s], [a_good, a_bad], capi.THC_PREC_MIXED, nstreams=2)
    assert per[0] == capi.THC_OK
    assert per[1] == capi.THC_ERR_EMPTY_CLUSTER
    assert st == capi.THC_ERR_EMPTY_CLUSTER


@pytest.mark.parametrize("prec", [capi.THC_PREC_FP64, capi.THC_PREC_MIXED])
def test_batched_look_ahead(prec):
    """N_mu 600: the Cholesky looks ahead (from 512 on), in a batch on the worker's one stream with
    the same results to the last bit."""
    import torch
    r = np.random.default_rng(3)
    mesh, norb, nmu = (16, 18, 20), 40, 600
    ng = int(np.prod(mesh))
    grid = np.stack(np.meshgrid(*[np.arange(float(m)) for m in mesh], indexing="ij"), -1).reshape(-1, 3)
    dev = torch.device("cuda", 0)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    systems = []
    for _ in range(2):
        phi = r.standard_normal((ng, norb))
        systems.append(dict(
            grid=cu(grid), rho=cu((phi ** 2).sum(1)), ng=ng, nmu=nmu, max_it=4, threshold=1e-9,
            init_idx=np.sort(r.choice(ng, nmu, replace=False)).astype(np.int32), phi=cu(phi),
            norb=norb, mesh=np.array(mesh, np.int32), coulG=cu(np.ones(ng)), shift_rel=-1.0,
            out_idx=np.zeros(nmu, np.int32), out_orbitals=np.zeros((norb, nmu, 2)),
            out_M=np.zeros((nmu, nmu, 2)), out_L=np.zeros((nmu, nmu, 2))))
    torch.cuda.synchronize()
    status, done = capi.factorize_batched(systems, precision=prec, nstreams=2)
    assert status == capi.THC_OK
    with capi.Context(0, prec) as ctx:
        for s in systems:
            got = ctx.isdf(s["phi"], s["out_idx"], mesh, s["coulG"])
            assert got["status"] == capi.THC_OK
            assert np.array_equal(got["M"], s["out_M"]) and np.array_equal(got["L"], s["out_L"])
