"""The workloads this library is used for, as timed cases.

Each case is one call of the public Python binding (``thcpp_gb300.capi``) on a synthetic
periodic cell: interpolating points by k-means or QRCP, the ISDF factorisation in FP64 (the
default precision of the C ABI and of the C++ classes) and in mixed precision, the
half-rotated pass and the complex (k-point) forms, and a batch of independent small systems.

The cells are those of the library's configurations: diamond-like atom density (38.3 cubic
bohr an atom), four s/p Gaussians per atom, periodised, mixed by a random matrix and
Loewdin-orthonormalised.  The exponents come from U[0.3, 0.8], the smooth part of the
configurations' range, so that the least-squares problem is well conditioned (C between 1e4
and 1e7) and results can be compared to many digits; the atoms are displaced from their sites
so that no two grid points are equivalent.  Cells are orthorhombic, so every function is a
product of three one-dimensional ones and the inputs are made on the GPU in milliseconds.

Mixed-precision factorisations run with the documented option ``autotune`` = 0: a program
whose results are compared between processes turns the timed kernel choice off, because the
choice decides the last bits of the sliced products.
"""
import math

import numpy as np
import torch

from thcpp_gb300 import capi

EDGE_PER_ATOM = 3.37        # bohr: 8 atoms in the 6.74-bohr cubic diamond cell
MAX_IT = 100                # the k-means limits of the library's configurations
THRESHOLD = 1e-6

_CONTEXTS = {}


def _device():
    return torch.device("cuda")


def _context(precision):
    """The context a program keeps for all its calls in one precision."""
    if precision not in _CONTEXTS:
        c = capi.Context(0, capi.THC_PREC_MIXED if precision == "mixed" else capi.THC_PREC_FP64)
        if precision == "mixed":
            c.set_option("autotune", 0)
        _CONTEXTS[precision] = c
    return _CONTEXTS[precision]


def listed():
    return [
        # The smallest call: points of a unit-test-sized cell, where launches and the
        # convergence checks count (ragged mesh, FP64).
        dict(name="points_small", kind="points", precision="fp64", n0=15, n1=16, n2=18, norb=12, nmu=48),
        # Points of the 8-atom benchmark cell (48^3, 8 N_o points).
        dict(name="points_mid", kind="points", precision="mixed", n0=48, n1=48, n2=48, norb=32, nmu=256),
        # Points of the 64-atom benchmark cell.
        dict(name="points_large", kind="points", precision="mixed", n0=72, n1=72, n2=72, norb=256, nmu=2048),
        # A screening run: six small independent systems from host arrays, points and
        # factorisation each, on four streams; ragged sizes.
        dict(name="batch_small", kind="batch", precision="fp64", n0=24, n1=25, n2=27, norb=20, nmu=97, nsys=6, nstreams=4),
        # The factorisation as the C++ classes call it by default (FP64), 8-atom cell.
        dict(name="vectors_mid", kind="vectors", precision="fp64", n0=48, n1=48, n2=48, norb=32, nmu=256),
        # The largest FP64 factorisation here: 32 atoms, a mesh with three different edges.
        dict(name="vectors_large", kind="vectors", precision="fp64", n0=60, n1=64, n2=54, norb=128, nmu=1024),
        # The mixed-precision factorisation, 8-atom and 64-atom benchmark cells.
        dict(name="vectors_mixed_mid", kind="vectors", precision="mixed", n0=48, n1=48, n2=48, norb=32, nmu=256),
        dict(name="vectors_mixed_large", kind="vectors", precision="mixed", n0=72, n1=72, n2=72, norb=256, nmu=2048),
        # The second pass of a half_rotated input.
        dict(name="half_mid", kind="half", precision="fp64", n0=45, n1=48, n2=40, norb=40, nmu=240, nocc=20),
        # k-point (complex) orbitals, plain and half-rotated pass.
        dict(name="complex_mid", kind="complex", precision="fp64", n0=40, n1=36, n2=45, norb=24, nmu=168),
        dict(name="half_complex_mid", kind="half_complex", precision="fp64", n0=30, n1=32, n2=36, norb=24, nmu=144, nocc=12),
        # Points by QR with column pivoting, 8-atom cell.
        dict(name="qrcp_mid", kind="qrcp", precision="fp64", n0=48, n1=48, n2=48, norb=32, nmu=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


#: Per kind: most N_g, smallest and largest N_o, and the most a drawn case may cost (see
#: work()); the limits are those of the largest listed case of the kind's precision.
_RANGES = {
    "points": (373248, 12, 256, 1e12),
    "batch": (32768, 16, 32, 2e10),
    "vectors": (207360, 16, 128, 7e11),
    "vectors_mixed": (373248, 16, 256, 5e12),
    "half": (110592, 16, 64, 2e11),
    "complex": (110592, 16, 48, 2e11),
    "half_complex": (65536, 16, 40, 1e11),
    "qrcp": (110592, 12, 48, 2e10),
}


def draw(rng):
    while True:
        kind = rng.choice(sorted(_RANGES))
        most, no_lo, no_hi, cost = _RANGES[kind]
        precision = "mixed" if kind == "vectors_mixed" else "fp64"
        if kind == "points":
            precision = rng.choice(["fp64", "mixed"])
        ng = _log_int(rng, 4096, most)
        edge = ng ** (1.0 / 3.0)
        # Three edges near the cube root, odd ones as often as even ones.
        n0, n1, n2 = (max(12, int(round(edge * rng.uniform(0.85, 1.15)))) for _ in range(3))
        norb = _log_int(rng, no_lo, no_hi)
        # 4 to 7 points per orbital, not always a multiple of N_o.
        nmu = int(norb * rng.uniform(4.0, 7.0))
        case = dict(kind="vectors" if kind == "vectors_mixed" else kind, precision=precision,
                    n0=n0, n1=n1, n2=n2, norb=norb, nmu=nmu)
        if kind in ("half", "half_complex"):
            case["nocc"] = max(8, int(norb * rng.uniform(0.35, 0.6)))
            case["nmu"] = nmu = int(norb * rng.uniform(3.0, 5.0))
        if kind == "batch":
            case["nsys"] = rng.randint(3, 8)
            case["nstreams"] = rng.choice([1, 2, 4, 8])
        ng = n0 * n1 * n2
        # At least 90 grid points for each interpolating point and a mesh spacing below
        # 0.85 bohr, as the configurations have.
        edge_bohr = EDGE_PER_ATOM * ((norb + 3) // 4) ** (1.0 / 3.0)
        if ng > most or ng < 90 * nmu or edge_bohr > 0.85 * min(n0, n1, n2):
            continue
        if work(case)["flops"] <= cost:
            return case


# ---------------------------------------------------------------------------- inputs

def _sites(natom, rs):
    """natom fractional positions spread over the cell, displaced from a cubic arrangement."""
    k = 1
    while k ** 3 < natom:
        k += 1
    cells = [(i, j, l) for i in range(k) for j in range(k) for l in range(k)]
    keep = [cells[(q * len(cells)) // natom] for q in range(natom)]
    pos = (np.array(keep, dtype=np.float64) + 0.5) / k
    return (pos + rs.uniform(-0.06, 0.06, size=pos.shape) / k) % 1.0


def _cell(case, seed, device, nfunc=None):
    """grid, mesh, phi (N_g x N_o), edge lengths and coulG of one cell (FP64 tensors)."""
    rs = np.random.RandomState(seed % (1 << 31))
    mesh = (case["n0"], case["n1"], case["n2"])
    no = case["norb"]
    natom = (no + 3) // 4
    edge = EDGE_PER_ATOM * natom ** (1.0 / 3.0)
    mean = (mesh[0] * mesh[1] * mesh[2]) ** (1.0 / 3.0)
    # The same mesh spacing along the three axes.
    box = [edge * n / mean for n in mesh]
    sites = _sites(natom, rs)
    alphas = rs.uniform(0.3, 0.8, size=4 * natom)[:no]
    mix = torch.from_numpy(rs.standard_normal((no, no))).to(device)
    al = torch.from_numpy(alphas).to(device)
    axes, plain, times = [], [], []
    for d in range(3):
        x = torch.arange(mesh[d], dtype=torch.float64, device=device) * (box[d] / mesh[d])
        axes.append(x)
        centre = torch.from_numpy(np.repeat(sites[:, d], 4)[:no] * box[d]).to(device)
        reach = int(math.ceil(math.sqrt(40.0 / alphas.min()) / box[d])) + 1
        t = torch.arange(-reach, reach + 1, dtype=torch.float64, device=device) * box[d]
        dist = x[:, None, None] - centre[None, :, None] - t[None, None, :]
        g = torch.exp(-al[None, :, None] * dist * dist)
        plain.append(g.sum(-1))
        times.append((dist * g).sum(-1))
    kind = torch.arange(no, device=device) % 4
    one = [torch.where(kind[None, :] == d + 1, times[d], plain[d]) for d in range(3)]
    raw = torch.einsum("xf,yf,zf->xyzf", *one).reshape(-1, no)
    del plain, times, one
    vol = box[0] * box[1] * box[2]
    ng = raw.shape[0]
    phi = raw @ mix
    s = (vol / ng) * (phi.T @ phi)
    w, u = torch.linalg.eigh(s)
    phi = (phi @ (u * w.rsqrt()) @ u.T).contiguous()
    grid = torch.stack(torch.meshgrid(*axes, indexing="ij"), dim=-1).reshape(-1, 3).contiguous()
    g2 = 0.0
    for d in range(3):
        k = torch.fft.fftfreq(mesh[d], 1.0 / mesh[d], dtype=torch.float64, device=device)
        shape = [1, 1, 1]
        shape[d] = -1
        g2 = g2 + (k * (2.0 * math.pi / box[d])).square().reshape(shape)
    g2 = g2.reshape(-1)
    coul = torch.where(g2 > 1e-12, 4.0 * math.pi / g2.clamp_min(1e-12), torch.zeros_like(g2))
    coul = (coul * (vol / float(ng) ** 2)).contiguous()
    return dict(mesh=np.asarray(mesh, np.int32), grid=grid, phi=phi, coul=coul, ng=ng, rs=rs)


def _points(ctx, cell, nmu, nocc, seed):
    """k-means points of the occupied density, as the driver selects them before the
    factorisation; another initial draw where two of them fall on one grid point."""
    rho = cell["phi"][:, :nocc].square().sum(1).contiguous()
    torch.cuda.synchronize()
    for k in range(8):
        init = capi.initial_indices(cell["ng"], nmu, (seed + 7919 * k) & 0x7FFFFFFF)
        idx, st, status = ctx.kmeans(cell["grid"], rho, nmu, init, MAX_IT, THRESHOLD,
                                     raise_on_error=False)
        if status == 0 and st.duplicates == 0:
            return idx
    raise RuntimeError("no interpolating points for this cell")


def _complex_orbitals(cell, device):
    """Complex orbitals of the same span: the real ones under a random unitary matrix."""
    no = cell["phi"].shape[1]
    q = cell["rs"].standard_normal((no, no)) + 1j * cell["rs"].standard_normal((no, no))
    q = np.linalg.qr(q)[0]
    return (cell["phi"].to(torch.complex128) @ torch.from_numpy(q).to(device)).contiguous()


def prepare(case, seed):
    dev = _device()
    kind, nmu = case["kind"], case["nmu"]
    ctx = _context(case["precision"])
    if kind == "batch":
        return _prepare_batch(case, seed, ctx, dev)
    cell = _cell(case, seed, dev)
    no, ng = case["norb"], cell["ng"]
    st = dict(case=case, ctx=ctx, **cell)
    if kind == "points":
        st["rho"] = cell["phi"][:, :no // 2].square().sum(1).contiguous()
        st["init"] = torch.from_numpy(capi.initial_indices(ng, nmu, seed & 0x7FFFFFFF)).to(dev)
        st["idx"] = torch.zeros(nmu, dtype=torch.int32, device=dev)
        del st["phi"], st["coul"]
    elif kind == "vectors":
        st["idx"] = torch.from_numpy(_points(ctx, cell, nmu, no // 2, seed)).to(dev)
        for name, shape in (("M", (nmu, nmu, 2)), ("L", (nmu, nmu, 2)), ("orbitals", (no, nmu, 2))):
            st["out_" + name] = torch.zeros(shape, dtype=torch.float64, device=dev)
    elif kind == "half":
        st["idx"] = torch.from_numpy(_points(ctx, cell, nmu, case["nocc"], seed)).to(dev)
        st["occ"] = cell["phi"][:, :case["nocc"]].contiguous()
    elif kind in ("complex", "half_complex"):
        nocc = case.get("nocc", no // 2)
        st["idx"] = torch.from_numpy(_points(ctx, cell, nmu, nocc, seed)).to(dev)
        st["phi"] = _complex_orbitals(cell, dev)
        st["occ"] = st["phi"][:, :nocc].contiguous()
    torch.cuda.synchronize()   # the library's stream does not wait for torch's
    return st


def _prepare_batch(case, seed, ctx, dev):
    """Systems of the batch: the case's sizes and smaller, all in host memory."""
    systems, nmu = [], case["nmu"]
    for s in range(case["nsys"]):
        c = dict(case, n0=case["n0"] - s % 3, n1=case["n1"] - s % 2, n2=case["n2"], nmu=nmu - 3 * s)
        cell = _cell(c, seed + 101 * s, dev)
        rho = cell["phi"][:, :c["norb"] // 2].square().sum(1).contiguous()
        # An initial draw whose points are distinct, as for a single system.
        for k in range(8):
            init = capi.initial_indices(cell["ng"], c["nmu"], (seed + s + 7919 * k) & 0x7FFFFFFF)
            torch.cuda.synchronize()
            _, st, status = ctx.kmeans(cell["grid"], rho, c["nmu"], init, MAX_IT, THRESHOLD,
                                       raise_on_error=False)
            if status == 0 and st.duplicates == 0:
                break
        n, no = c["nmu"], c["norb"]
        systems.append(dict(
            grid=cell["grid"].cpu().numpy(), rho=rho.cpu().numpy(), ng=cell["ng"], nmu=n,
            init_idx=init, max_it=MAX_IT, threshold=THRESHOLD, phi=cell["phi"].cpu().numpy(),
            norb=no, mesh=cell["mesh"], coulG=cell["coul"].cpu().numpy(), shift_rel=-1.0,
            out_idx=np.zeros(n, np.int32), out_orbitals=np.zeros((no, n, 2)),
            out_M=np.zeros((n, n, 2)), out_L=np.zeros((n, n, 2))))
    return dict(case=case, systems=systems)


# ---------------------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        status, done = capi.factorize_batched(state["systems"], precision=capi.THC_PREC_FP64,
                                              nstreams=case["nstreams"])
        return dict(status=status, systems=[
            dict(idx=s["out_idx"], M=s["out_M"], L=s["out_L"], orbitals=s["out_orbitals"],
                 iterations=int(done[i].kmeans_stats.iterations))
            for i, s in enumerate(state["systems"])])
    ctx = state["ctx"]
    if kind == "points":
        idx, st, _ = ctx.kmeans(state["grid"], state["rho"], case["nmu"], state["init"], MAX_IT,
                                THRESHOLD, out_idx=state["idx"])
        return dict(idx=idx, iterations=int(st.iterations), diff=float(st.final_diff))
    if kind == "vectors":
        r = ctx.isdf(state["phi"], state["idx"], state["mesh"], state["coul"],
                     out_M=state["out_M"], out_L=state["out_L"], out_orbitals=state["out_orbitals"])
        return dict(M=r["M"], L=r["L"], orbitals=r["orbitals"], status=int(r["status"]))
    if kind == "half":
        r = ctx.isdf_half(state["phi"], state["occ"], state["idx"], state["mesh"], state["coul"])
        return dict(M=r["M"], orbitals=r["orbitals"], occ_orbitals=r["occ_orbitals"])
    if kind == "complex":
        r = ctx.isdf_complex(state["phi"], state["idx"], state["mesh"], state["coul"])
        return dict(M=r["M"], L=r["L"], orbitals=r["orbitals"], status=int(r["status"]))
    if kind == "half_complex":
        r = ctx.isdf_half_complex(state["phi"], state["occ"], state["idx"], state["mesh"],
                                  state["coul"])
        return dict(M=r["M"], orbitals=r["orbitals"], occ_orbitals=r["occ_orbitals"])
    r = ctx.qrcp(state["phi"], case["nmu"])
    return dict(idx=r["idx"], order=r["order"], diag=r["diag"])


# ---------------------------------------------------------------------------- its cost

def work(case):
    """Bytes of the inputs and outputs, and the operations of the products, the transforms
    and the factorisations (k-means: one distance and four sums per point and iteration)."""
    ng, no, nmu = case["n0"] * case["n1"] * case["n2"], case["norb"], case["nmu"]
    kind = case["kind"]
    if kind == "batch":
        one = work(dict(case, kind="vectors"))
        two = work(dict(case, kind="points"))
        return {k: case["nsys"] * (one[k] + two[k]) for k in one}
    if kind == "points":
        return {"bytes": 32.0 * ng + 8.0 * nmu, "flops": 16.0 * MAX_IT * ng}
    if kind == "qrcp":
        return {"bytes": 8.0 * ng * no + 16.0 * nmu, "flops": 2.0 * ng * nmu * (no + 0.5 * nmu)}
    cplx = kind in ("complex", "half_complex")
    rot = kind in ("half", "half_complex")
    w = 2.0 if cplx else 1.0
    nocc = case.get("nocc", 0) if rot else 0
    nbytes = 8.0 * w * ng * (no + nocc) + 8.0 * ng + 16.0 * nmu * (no + nocc)
    nbytes += 16.0 * nmu * nmu * (1 if rot else 2)
    lg = math.log2(ng)
    if kind == "half_complex":
        flops = 8.0 * ng * nmu * (no + nocc) + 8.0 * nmu * nmu * ng + 8.0 / 3.0 * nmu ** 3
        flops += 2 * 5.0 * ng * lg * nmu + 8.0 * nmu * nmu * ng
    else:
        pairs = 4.0 if cplx else 1.0
        flops = pairs * 2.0 * ng * nmu * (no + nocc) + 2.0 * nmu * nmu * ng + nmu ** 3 / 3.0
        flops += 2.5 * ng * lg * nmu + nmu * nmu * ng + (0 if rot else nmu ** 3 / 3.0)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------- 64-bit values

def _pairs(x):
    return torch.view_as_real(x.to(torch.complex128).contiguous())


def _coulomb(zeta_hat, coul, left=None):
    """sum_G conj(left) v zeta_hat over the full spectrum, rows mu (left: zeta_hat)."""
    left = zeta_hat.conj() if left is None else left
    return (left * coul) @ zeta_hat.T


def _fields(x, mesh, inverse=False):
    f = x.reshape(x.shape[0], *[int(m) for m in mesh])
    y = torch.fft.ifftn(f, dim=(1, 2, 3), norm="forward") if inverse else torch.fft.fftn(f, dim=(1, 2, 3))
    return y.reshape(x.shape[0], -1)


def _exact_plain(phi, idx, mesh, coul, occ=None):
    """Z = P o conj(P) or P_occ o P, C X = Z, M over the half spectrum (real fields, v even)."""
    pm = phi[idx]
    z = pm.conj() @ phi.T
    z = (z.real.square() + z.imag.square()) if z.is_complex() else z.square() if occ is None else z * (occ[idx] @ occ.T)
    c = z[:, idx]
    zeta = torch.cholesky_solve(z, torch.linalg.cholesky(0.5 * (c + c.T)))
    del z
    n0, n1, n2 = (int(m) for m in mesh)
    nc = n2 // 2 + 1
    v = coul.reshape(n0, n1, n2)[:, :, :nc].clone()
    v[:, :, 1:nc - 1 if n2 % 2 == 0 else nc] *= 2.0
    m = torch.zeros((pm.shape[0],) * 2, dtype=torch.float64, device=phi.device)
    zh = torch.fft.rfftn(zeta.reshape(-1, n0, n1, n2), dim=(1, 2, 3)).reshape(pm.shape[0], -1)
    del zeta
    a = torch.view_as_real(zh * v.reshape(-1).sqrt()).reshape(pm.shape[0], -1)
    m = a @ a.T
    return pm, m


def exact(case, seed):
    """The factorisations' matrices, the orbitals at the points and the QRCP diagonal in plain
    64-bit torch; the k-means results are compared as they are (whole numbers)."""
    kind = case["kind"]
    if kind == "points":
        return None
    if kind == "batch":
        st = prepare(case, seed)
        run(st)            # the points, which are whole numbers; all else is formed here
        out = []
        for s in st["systems"]:
            phi = torch.from_numpy(s["phi"]).to(_device())
            coul = torch.from_numpy(s["coulG"]).to(_device())
            pm, m = _exact_plain(phi, torch.from_numpy(s["out_idx"]).to(_device()).long(), s["mesh"], coul)
            out.append(dict(idx=None, M=_pairs(m), L=_pairs(torch.linalg.cholesky(m)),
                            orbitals=_pairs(pm.T), iterations=None))
        return dict(status=None, systems=out)
    st = prepare(case, seed)
    phi, coul, mesh = st["phi"], st["coul"], st["mesh"]
    if kind == "qrcp":
        g = (phi * phi).sum(1).square()
        low, diag = [], []
        for k in range(case["nmu"]):
            p = int(torch.argmax(g))
            d = float(g[p].sqrt())
            col = (phi @ phi[p]).square()
            if low:
                lk = torch.stack(low)
                col = col - lk[:, p] @ lk
            col = col / d
            low.append(col)
            diag.append(d)
            g = g - col * col
            g[p] = -1.0
        return dict(idx=None, order=None, diag=np.array(diag))
    idx = st["idx"].long()
    if kind == "half_complex":
        pm, po = phi[idx], st["occ"][idx]
        z = (po.conj() @ st["occ"].T) * (pm.conj() @ phi.T).conj()
        zeta = torch.linalg.solve(z[:, idx], z).conj()
        m = _coulomb(_fields(zeta, mesh), coul, _fields(zeta, mesh, inverse=True))
        return dict(M=_pairs(m), orbitals=_pairs(pm.T), occ_orbitals=_pairs(po.T))
    pm, m = _exact_plain(phi, idx, mesh, coul, st["occ"] if kind == "half" else None)
    if kind == "half":
        return dict(M=_pairs(m), orbitals=_pairs(pm.T), occ_orbitals=_pairs(st["occ"][idx].T))
    return dict(M=_pairs(m), L=_pairs(torch.linalg.cholesky(m)), orbitals=_pairs(pm.T), status=None)
