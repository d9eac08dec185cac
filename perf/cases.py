"""Timed workloads of the projected-HF framework, through the calls a user's program makes.

Kinds of call (``case["kind"]``):

* ``buildhsg``  the f2py-signature calls of one optimiser step of the reference's driver: phftools.buildhsg
                with a dense HTwo on host arrays, then phftools.localg
* ``host``      Plan.buildhsg: the same step with the Hamiltonian kept on the GPU (Cholesky vectors), host in and out
* ``step``      optimizer.DeviceEandG: energy and gradient of a device-resident parameter vector
* ``eval``      Plan.eval_device: the accumulated H, S and gradient sums for a device-resident determinant
* ``grad``      autograd.projected_energy, forward and backward
* ``batch``     api.eval_batch: many instances of uneven size together
* ``pcc``       fpucc.pbarhbarolap: the projected-CCSD grid kernel (host arrays)
* ``buildsc``   phftools.buildsc: the grid-projected product of the linear-dependency solver (host arrays)

Sizes: n spatial orbitals, N electrons, L Cholesky vectors, a Lebedev x trapezoid grid times the operations
of a point group.  Problems are those of phf_pcc_b200.synth (seeded Hamiltonians and determinants).
"""
import math

import numpy as np
import torch

from phf_pcc_b200 import api, synth
from phf_pcc_b200.PHFTools_F import phftools
from phf_pcc_b200.PUCC_X2 import fpucc
from phf_pcc_b200.autograd import projected_energy
from phf_pcc_b200.grid import make_grid
from phf_pcc_b200.optimizer import DeviceEandG

phftools.on_not_hermitian = "return"  # random determinants on finite grids: H is Hermitian only to the grid's error


def _case(name, kind, n, N, L, grid, pg="None", precision="ozaki_i8", **more):
    return dict(name=name, kind=kind, n=n, N=N, L=L, nl=grid[0], ny=grid[1], pg=pg, precision=precision, **more)


def listed():
    return [
        # smallest: an optimiser step of a 20-orbital molecule, every array on the device; launches and latency
        _case("step_n20_fp64", "step", 20, 10, 120, (14, 8), precision="fp64"),
        # the reference's driver unedited: dense integrals passed from the host in every call
        _case("buildhsg_n20_dense", "buildhsg", 20, 10, 120, (14, 8), precision="fp64"),
        # odd sizes, exact gradient (what autograd users differentiate with), tensor-core form
        _case("grad_n37_exact_i8", "grad", 37, 19, 150, (14, 8), "C2v", gradient="exact"),
        # optimiser step at a middle size, tensor-core form
        _case("step_n48_i8", "step", 48, 24, 240, (26, 10)),
        # the plain FP64 form (the default precision) on the 800-point grid
        _case("eval_n64_fp64", "eval", 64, 32, 400, (50, 16), precision="fp64"),
        # energy and gradient on the 3200-point grid with point-group projection
        _case("grad_n64_c2v_i8", "grad", 64, 32, 400, (50, 16), "C2v", gradient="reference"),
        # host-driven step, odd orbital and electron counts above one tile of the tensor-core kernels
        _case("host_n101_i8", "host", 101, 51, 405, (26, 12)),
        # large basis, stored exchange matrix
        _case("eval_n128_i8", "eval", 128, 64, 800, (50, 16)),
        # largest: no n^4 tensor, exchange rows streamed from the Cholesky vectors
        _case("eval_n200_c2v_i8", "eval", 200, 100, 1000, (38, 16), "C2v"),
        # many independent instances of uneven size, grids of 112 and 800 points in turn
        dict(name="batch_16_i8", kind="batch", count=16, nmin=16, nmax=96, precision="ozaki_i8"),
        # projected-CCSD grid kernel, one Broyden iteration's call
        _case("pcc_n20", "pcc", 20, 10, 120, (14, 8), precision="fp64"),
        # grid-projected product of the linear-dependency solver
        _case("buildsc_n16", "buildsc", 16, 8, 32, (14, 8), precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["buildhsg", "host", "step", "eval", "eval", "grad", "batch", "pcc", "buildsc"])
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 16), nmin=16, nmax=rng.choice([48, 64, 96]),
                    precision=rng.choice(["ozaki_i8", "ozaki_i8", "fp64"]))
    grid = rng.choice([(6, 6), (14, 8), (26, 10), (26, 12), (38, 16), (50, 16)])
    pg = rng.choice(["None", "None", "C2v"])
    if kind == "buildhsg":
        n, precision = rng.randint(8, 22), "fp64"
        grid, pg = rng.choice([(6, 6), (14, 8), (26, 10)]), rng.choice(["None", "C2v"])
    elif kind == "pcc":
        n, precision, pg = rng.randint(8, 20), "fp64", "None"
        grid = rng.choice([(6, 6), (14, 8)])
    elif kind == "buildsc":
        n, precision, pg = rng.randint(5, 16), "fp64", "None"
        grid = rng.choice([(6, 6), (14, 8)])
    else:
        precision = rng.choice(["ozaki_i8", "ozaki_i8", "fp64"])
        n = _log_int(rng, 14, 180 if precision == "ozaki_i8" and kind == "eval" else 128 if precision == "ozaki_i8" else 72)
        if n > 128:
            grid = rng.choice([(14, 8), (26, 12)])
    N = max(2, min(n, int(round(n * rng.uniform(0.3, 0.6)))))
    case = _case("", kind, n, N, int(round(n * rng.uniform(4, 6))), grid, pg, precision)
    case.pop("name")
    if kind == "grad":
        case["gradient"] = rng.choice(["exact", "reference"])
    return case


# ---------------------------------------------------------------- inputs


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _problem(c, seed):
    return synth.make_problem(c["n"], c["N"], c["L"], ngrid=(c["nl"], c["ny"]), seed=seed, pg=c["pg"])


def _start_z(p, seed):
    """A Thouless matrix some way from the reference determinant, as within an optimisation."""
    rng = np.random.default_rng(seed + 101)
    s = (p.M - p.N, p.N)
    return 0.1 * (rng.normal(size=s) + 1j * rng.normal(size=s))


def _grid_args(g, N):
    return dict(ngrid=list(g.ngrid), nci=g.nci, cmplxconj=g.CmplxConj, ncisp=g.ncisp, nocc=N, r1=g.R1, r2=g.R2,
                rpg=g.Rpg, weightsp=g.weightsp, weightpg=g.weightpg, roota=g.roota, rootb=g.rootb, rooty=g.rooty,
                qj=g.J, sp=g.SP)


def _plan(p, precision, gradient="reference"):
    return api.Plan(h=p.h, B=p.B, ref=p.Qfull, precision=precision, gradient=gradient, **_grid_args(p.grid, p.N))


def _dense(p):
    """HOne and the antisymmetrised HTwo in the Ref-MO basis, as the driver's ao2mo makes them."""
    U = torch.from_numpy(p.Qfull).to(_device())
    B = torch.from_numpy(p.B).to(U)
    n = p.n
    Bm = torch.zeros((p.L, p.M, p.M), dtype=U.dtype, device=U.device)
    Bm[:, :n, :n] = B
    Bm[:, n:, n:] = B
    Bm = U.conj().T @ Bm @ U
    m = torch.einsum("Lik,Ljl->ijkl", Bm, Bm)
    H1 = U.conj().T @ torch.from_numpy(p.hone_ao()).to(U) @ U
    H2 = m - m.transpose(2, 3)
    return np.asfortranarray(H1.cpu().numpy()), np.asfortranarray(H2.cpu().numpy())


def _batch_problems(c, seed):
    rng = np.random.default_rng(seed)
    shapes = np.random.default_rng(c["count"] * 1000 + c["nmax"])  # the sizes belong to the case, the data to the seed
    out = []
    for i in range(c["count"]):
        n = int(shapes.choice(np.arange(c["nmin"], c["nmax"] + 1, 8)))
        out.append(synth.make_problem(n, n // 2, 4 * n, ngrid=(14, 8) if i % 2 == 0 else (50, 16),
                                      seed=int(rng.integers(1 << 30))))
    return out


def _pcc_problem(c, seed):
    return synth.make_pcc_problem(c["n"], c["N"], c["L"], ngrid=(c["nl"], c["ny"]), seed=seed)


def _sc_problem(c, seed):
    g = make_grid(c["n"], ngrid=(c["nl"], c["ny"]), pg=c["pg"])
    rng = np.random.default_rng(seed)
    M = 2 * c["n"]
    U = synth.random_unitary(M, rng)
    cz = lambda *s: rng.normal(size=s) + 1j * rng.normal(size=s)
    mo = lambda R: np.asfortranarray(U.conj().T @ R @ U)
    vec = (complex(cz(1)[0]), np.asfortranarray(0.3 * cz(M, M)), np.asfortranarray(0.1 * cz(M, M, M, M)))
    return vec, g, mo(g.R1), mo(g.R2), mo(g.Rpg)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        ps = _batch_problems(case, seed)
        s["plans"] = [_plan(p, case["precision"]) for p in ps]
        s["C"] = [torch.from_numpy(p.C).to(_device()) for p in ps]
        s["outs"] = None
        return s
    if kind == "pcc":
        p = _pcc_problem(case, seed)
        M, o = 2 * case["n"], p["NOcc"]
        f = lambda a: np.asfortranarray(a, dtype=np.complex128)
        s["args"] = (f(p["HOne"]), f(p["HTwo"]), None, f(p["T1"]), f(p["T2"]), o, M // 2, M, p["ENuc"], p["QJ"], p["SP"],
                     p["NPoints"], p["Npg"], len(p["fsp"]), len(p["fpg"]), p["ncik"], f(p["R1"]), f(p["R2"]),
                     f(p["Rpg"]), f(p["Rk"]), p["Roota"], p["Rootb"], p["Rooty"], p["Weightsp"], p["Weightpg"],
                     p["fsp"], p["fpg"], p["fk"], p["TrunODE"])
        return s
    if kind == "buildsc":
        vec, g, R1, R2, Rpg = _sc_problem(case, seed)
        rk = np.eye(2 * case["n"], dtype=complex)[None]
        one = np.ones(1, complex)
        s["args"] = (*vec, case["N"], list(g.ngrid), g.J, R1, R2, Rpg, rk, g.roota, g.rootb, g.rooty, g.weightsp,
                     g.weightpg, one, one, one)
        return s
    p = _problem(case, seed)
    if kind == "buildhsg":
        H1, H2 = _dense(p)
        g = p.grid
        s["args"] = (H1, H2, np.asfortranarray(p.Qfull), np.asfortranarray(_start_z(p, seed)), list(g.ngrid), g.nci,
                     g.CmplxConj, g.ncisp, p.N, np.asfortranarray(g.R1), np.asfortranarray(g.R2),
                     np.asfortranarray(g.Rpg), g.weightsp, g.weightpg, g.roota, g.rootb, g.rooty, g.J, g.SP)
        return s
    s["plan"] = _plan(p, case["precision"], case.get("gradient", "reference"))
    if kind == "host":
        s["z"] = np.asfortranarray(_start_z(p, seed))
    elif kind == "step":
        s["fun"] = DeviceEandG(s["plan"])
        z = _start_z(p, seed).reshape(-1)
        s["x"] = torch.from_numpy(np.concatenate([z.real, z.imag])).to(_device())
    else:
        s["C"] = torch.from_numpy(p.C).to(_device()).requires_grad_(kind == "grad")
    return s


def run(s):
    kind = s["kind"]
    if kind == "eval":
        return s["plan"].eval_device(s["C"])
    if kind == "grad":
        s["C"].grad = None
        E = projected_energy(s["C"], s["plan"])
        E.backward()
        return E.detach(), s["C"].grad
    if kind == "step":
        return s["fun"](s["x"])
    if kind == "host":
        return s["plan"].buildhsg(s["z"], check_hermitian=False)
    if kind == "buildhsg":
        H, S, G, R = phftools.buildhsg(*s["args"])
        one = np.ones(1, complex)
        E = H[0, 0].real / abs(S[0, 0].real)
        return H, S, G, R, phftools.localg(G, R, S, E, one, one, one, s["args"][6])
    if kind == "batch":
        s["outs"] = api.eval_batch(s["plans"], s["C"], s["outs"])
        return s["outs"]
    if kind == "pcc":
        return [np.asarray(x) for x in fpucc.pbarhbarolap(*s["args"])]
    return [np.asarray(x) for x in phftools.buildsc(*s["args"])]


# ---------------------------------------------------------------- least work of one pass


def _hf_work(n, N, L, pts, rot, dense=False):
    """Exchange over index pairs (8 n^4 real operations a point), Coulomb over the Cholesky vectors, density, F X,
    the N-wide products and the inverse; inputs and outputs once."""
    M = 2 * n
    per = (8.0 * M ** 4 if dense else 8.0 * n ** 4 + 4.0 * L * n * n) + 16.0 * M * M * N + 32.0 * M * N * N + 8.0 * N ** 3
    ham = 16.0 * M ** 4 if dense else 8.0 * (L * n * n + n * n)
    return {"flops": per * pts, "bytes": ham + 16.0 * M * M * rot + 48.0 * M * N}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ws = [_hf_work(p.n, p.N, p.L, p.grid.npoints, 0) for p in _batch_problems(case, 0)]
        return {k: sum(w[k] for w in ws) for k in ("flops", "bytes")}
    n, N, npg = case["n"], case["N"], 4 if case["pg"] == "C2v" else 1
    M, pts, rot = 2 * n, case["nl"] * case["ny"] * npg, case["nl"] + case["ny"] + npg
    if kind == "pcc":
        o, v = N, M - N
        # four one-index transforms that start from the vvoo block, and the particle-particle, hole-hole and ring terms
        per = 8.0 * (M * v * v * o * o + M * M * v * o * o + M ** 3 * o * o + M ** 4 * o) + \
            8.0 * (v ** 4 * o * o + v * v * o ** 4 + 2 * v ** 3 * o ** 3)
        return {"flops": per * pts, "bytes": 16.0 * (M ** 4 + 3 * v * v * o * o + M * M * rot)}
    if kind == "buildsc":
        return {"flops": 8.0 * 9 * M ** 5 * pts, "bytes": 16.0 * (2 * M ** 4 + M * M * rot)}
    return _hf_work(n, N, case["L"], pts, rot, dense=kind == "buildhsg")


# ---------------------------------------------------------------- the same values in plain 64-bit torch


def _hf_sums(p, C, exact_gradient=False):
    """(hs, yg, yr) of eval_device for one projection channel, straight from the definitions: rho = X C^H,
    Gamma = J - K, F = h + Gamma, and per point N [(1 - rho) F X + h X]."""
    dev = _device()
    n, N, M, g = p.n, p.N, p.M, p.grid
    C = torch.as_tensor(C).to(dev)
    B = torch.from_numpy(p.B).to(dev).reshape(p.L, n * n)
    ek = (B.T @ B).reshape(n, n, n, n).permute(0, 2, 1, 3).reshape(n * n, n * n)  # [(i, k), (l, j)] = (il|kj)
    h = torch.from_numpy(p.hone_ao()).to(dev)
    R1, R2, Rpg = (torch.from_numpy(np.ascontiguousarray(r)).to(dev) for r in (g.R1, g.R2, g.Rpg))
    hs = torch.zeros(2, dtype=C.dtype, device=dev)
    sums = torch.zeros((4, M, N), dtype=C.dtype, device=dev)
    step = max(1, int(2e9 / (16 * 8 * M * M)))
    pts = [(il, iy, ig) for il in range(R1.shape[0]) for iy in range(R2.shape[0]) for ig in range(Rpg.shape[0])]
    for a in range(0, len(pts), step):
        il, iy, ig = (torch.tensor(t, device=dev) for t in zip(*pts[a:a + step]))
        wt = torch.from_numpy(np.array([g.weightsp[x, y] * g.weightpg[z, 0, 0] for x, y, z in pts[a:a + step]])).to(dev)
        R = R1[il] @ R2[iy] @ Rpg[ig]
        Y = R @ C
        S = C.conj().T @ Y
        Si, det = torch.linalg.inv(S), torch.linalg.det(S)
        X = Y @ Si
        b = X.shape[0]
        rho = (X @ C.conj().T).reshape(b, 2, n, 2, n)
        P = (rho[:, 0, :, 0] + rho[:, 1, :, 1]).reshape(b, n * n)
        cols = torch.view_as_real(rho.permute(2, 4, 0, 1, 3).reshape(n * n, -1).contiguous()).reshape(n * n, -1)
        K = torch.view_as_complex((ek @ cols).reshape(n * n, b * 4, 2).contiguous()).reshape(n, n, b, 2, 2)
        del cols
        F = -K.permute(2, 3, 0, 4, 1).reshape(b, M, M)
        J = torch.complex((P.real @ B.T) @ B, (P.imag @ B.T) @ B).reshape(b, n, n)
        F[:, :n, :n] += J
        F[:, n:, n:] += J
        GX, HX = F @ X, h @ X
        e1 = torch.einsum("ij,bij->b", C.conj(), HX)
        ew = e1 + 0.5 * torch.einsum("ij,bij->b", C.conj(), GX)
        F += h
        W = C.conj().T @ (GX + HX)
        c = wt * det
        hs[0] += (c * ew).sum()
        hs[1] += c.sum()
        sums[0] += torch.einsum("b,bij->ij", c, GX + HX - X @ W + ew[:, None, None] * X)
        sums[1] += torch.einsum("b,bij->ij", c, X)
        if exact_gradient:
            V = F.mH @ C - C @ W.mH + ew.conj()[:, None, None] * C
            A = R.mH @ torch.cat([V, C.expand(b, M, N)], 2)
            sums[2] += torch.einsum("b,bij->ij", c.conj(), A[:, :, :N] @ Si.mH)
            sums[3] += torch.einsum("b,bij->ij", c.conj(), A[:, :, N:] @ Si.mH)
    if exact_gradient:
        return hs, (sums[0] + sums[2]) / 2, (sums[1] + sums[3]) / 2
    return hs, sums[0], sums[1]


def _exact_hf(case, seed):
    kind = case["kind"]
    p = _problem(case, seed)
    if kind in ("eval", "grad"):
        hs, yg, yr = _hf_sums(p, p.C, case.get("gradient") == "exact")
        if kind == "eval":
            return hs[None], yg[None], yr[None]
        E = hs[0].real / hs[1].real.abs()
        by = hs[1].real if case["gradient"] == "exact" else hs[1]
        return E, 2 * (yg - E * yr) / by if case["gradient"] != "exact" else 2 * (yg - E * by.sign() * yr) / by.abs()
    z = torch.from_numpy(_start_z(p, seed)).to(_device())
    U = torch.from_numpy(p.Qfull).to(z)
    mo = torch.cat([torch.eye(p.N, dtype=z.dtype, device=z.device), z], 0)
    hs, yg, yr = _hf_sums(p, U @ mo)
    if kind == "step":
        E = hs[0].real / hs[1].real.abs()
        G = (U.mH @ ((yg - E * yr) / hs[1]))[p.N:]
        return E, torch.cat([G.real.reshape(-1), G.imag.reshape(-1)])
    grad, rdm = ((U.mH @ y @ mo.mH) for y in (yg, yr))
    out = [hs[0].reshape(1, 1), hs[1].reshape(1, 1), grad[None, None], rdm[None, None]]
    if kind == "buildhsg":
        out.append((grad - hs[0].real / hs[1].real.abs() * rdm) / hs[1])
    return tuple(x.cpu().numpy() for x in out)


def _perm(t, p):
    """t - t with the two indices that p names exchanged."""
    return t - t.transpose(*p)


def _exact_pcc(case, seed):
    """Olap0, OlapEx1, OlapEx2, EOlap0, EOlapEx1, EOlapEx2: per point the Thouless form of R [1; T1], the similarity
    transform of T2 to second order, the CCSD energy and residuals and the disconnected terms, summed with the weights."""
    p, dev, e = _pcc_problem(case, seed), _device(), torch.einsum
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    h, H, T1, T2, R1, R2, Rpg = (t(p[k]) for k in ("HOne", "HTwo", "T1", "T2", "R1", "R2", "Rpg"))
    o, M = p["NOcc"], h.shape[0]
    O, V = slice(0, o), slice(o, M)
    F = h + e("piqi->pq", H[:, O, :, O])
    scf = e("ii->", h[O, O]) + e("ijij->", H[O, O, O, O]) / 2
    Hoovv, Hooov, Hvovv = H[O, O, V, V], H[O, O, O, V], H[V, O, V, V]
    acc = [0, 0, 0, 0, 0, 0]
    for il in range(R1.shape[0]):
        for iy in range(R2.shape[0]):
            for ig in range(Rpg.shape[0]):
                R = R1[il] @ R2[iy] @ Rpg[ig]
                A = torch.cat([torch.eye(o, dtype=h.dtype, device=dev), T1], 0)
                A = R @ A
                U0, U1 = torch.linalg.det(A[:o]), A[o:] @ torch.linalg.inv(A[:o])
                W = torch.eye(M, dtype=h.dtype, device=dev)
                W[o:, :o] = -U1
                W = W @ R
                I = torch.linalg.inv(W)
                u = e("pa,abij->pbij", W[:, V], T2)
                u = e("qb,pbij->pqij", W[:, V], u)
                u = e("pqij,ir->pqrj", u, I[O])
                u = e("pqrj,js->pqrs", u, I[O])
                f = e("piqi->pq", u[:, O, :, O])
                E0 = e("ijij->", u[O, O, O, O]) / 2
                fov, fvo, foo, fvv = f[O, V], f[V, O], f[O, O], f[V, V]
                vvoo = u[V, V, O, O]
                C0 = 1 + E0 + E0 ** 2 / 2 + (fov * fvo.T).sum() / 2 + e("ijab,abij->", u[O, O, V, V], vvoo) / 8
                C1 = fvo + E0 * fvo - fvo @ foo / 2 + fvv @ fvo / 2
                C1 = C1 - e("abij,ijkb->ak", vvoo, u[O, O, O, V]) / 4 - e("jabc,bckj->ak", u[O, V, V, V], vvoo) / 4
                C1 = C1 + e("abij,jb->ai", vvoo, fov) / 2 - e("jaib,bj->ai", u[O, V, O, V], fvo) / 2
                C2 = vvoo / 4 + E0 / 4 * vvoo - e("aj,bi->abij", fvo, fvo) / 2
                C2 = C2 + e("acjk,kbic->abij", vvoo, u[O, V, O, V]) / 2
                C2 = C2 + e("cdij,abcd->abij", vvoo, u[V, V, V, V]) / 16 + e("klij,abkl->abij", u[O, O, O, O], vvoo) / 16
                C2 = C2 - e("abik,kj->abij", vvoo, foo) / 4 + e("cbij,ac->abij", vvoo, fvv) / 4
                C2 = C2 - e("kbij,ak->abij", u[O, V, O, O], fvo) / 4 + e("abic,cj->abij", u[V, V, O, V], fvo) / 4
                w1 = C1 / C0
                t2 = _perm(_perm(C2 / C0 - e("ai,bj->abij", w1, w1) / 2, (2, 3)), (0, 1))
                t1, lam = w1 + U1, C0 * U0
                tt = e("ai,bj->abij", t1, t1)
                at = _perm(tt, (0, 1))
                tau, tb, half = t2 + at, t2 + at / 2, t2 / 2 + tt
                Ene = (F[O, V] * t1.T).sum() + e("ijab,abij->", Hoovv, tau) / 4 + scf
                Fvv = F[V, V] - t1 @ F[O, V] / 2 + e("ci,aibc->ab", t1, Hvovv) - e("abij,ijcb->ac", tb, Hoovv) / 2
                Foo = F[O, O] + F[O, V] @ t1 / 2 + e("ak,ikja->ij", t1, Hooov) + e("ikcb,cbjk->ij", Hoovv, tb) / 2
                Fov = F[O, V] + e("bj,ijab->ia", t1, Hoovv)
                Woo = H[O, O, O, O] + e("ijab,abkl->ijkl", Hoovv, tau) / 4 + _perm(e("ijka,al->ijkl", Hooov, t1), (2, 3))
                Wvv = H[V, V, V, V] + e("cdij,ijab->cdab", tau, Hoovv) / 4 - _perm(e("aicd,bi->abcd", Hvovv, t1), (0, 1))
                Wov = H[O, V, V, O] + e("iabc,cj->iabj", H[O, V, V, V], t1) - e("ikcj,bk->ibcj", H[O, O, V, O], t1)
                Wov = Wov - e("dbjk,ikcd->ibcj", half, Hoovv)
                r1 = F[V, O] + Fvv @ t1 - t1 @ Foo + e("jb,abij->ai", Fov, t2) + e("bj,ajib->ai", t1, H[V, O, O, V])
                r1 = r1 - e("abjk,jkib->ai", t2, Hooov) / 2 + e("ajcb,cbij->ai", Hvovv, t2) / 2
                r2 = H[V, V, O, O] + _perm(e("acij,bc->abij", t2, Fvv - t1 @ Fov / 2), (0, 1))
                r2 = r2 - _perm(e("abik,kj->abij", t2, Foo + Fov @ t1 / 2), (2, 3))
                ring = e("acik,kbcj->abij", t2, Wov) - e("ci,kbcj,ak->abij", t1, H[O, V, V, O], t1)
                r2 = r2 + _perm(_perm(ring, (0, 1)), (2, 3))
                r2 = r2 + e("cdij,abcd->abij", tau, Wvv) / 2 + e("klij,abkl->abij", Woo, tau) / 2
                r2 = r2 + _perm(e("ci,abcj->abij", t1, H[V, V, V, O]), (2, 3)) - _perm(e("kbij,ak->abij", H[O, V, O, O], t1), (0, 1))
                l2 = t2 + at
                x = e("ai,bj->abij", t1, r1)
                x = _perm(_perm(x, (0, 1)), (2, 3))
                wt = p["Weightsp"][il, iy] * p["Weightpg"][ig, 0, 0] * lam
                new = (1, t1, l2, Ene, r1 + t1 * Ene, r2 + l2 * Ene + x)
                acc = [q + wt * y for q, y in zip(acc, new)]
    return tuple(torch.as_tensor(q).cpu().numpy() for q in acc)


def _exact_buildsc(case, seed):
    """t0, t1, t2: per point the transition density Y of [I; 0], the vector in the rotated basis, the contractions of
    its doubles with Y, and the weighted sums over the projected overlap."""
    (c0, c1, c2), g, R1, R2, Rpg = _sc_problem(case, seed)
    dev, e, N = _device(), torch.einsum, case["N"]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
    c1, c2, R1, R2, Rpg = t(c1), t(c2), t(R1), t(R2), t(Rpg)
    out, ovl = [0, 0, 0], 0
    for il in range(R1.shape[0]):
        for iy in range(R2.shape[0]):
            for ig in range(Rpg.shape[0]):
                R = R1[il] @ R2[iy] @ Rpg[ig]
                Y = torch.zeros_like(R)
                Y[:, :N] = R[:, :N] @ torch.linalg.inv(R[:N, :N])
                U = R.mH
                a1 = R @ c1 @ U
                d = e("pa,abcd->pbcd", R, c2)
                d = e("qb,pbcd->pqcd", R, d)
                d = e("pqcd,cr->pqrd", d, U)
                d = e("pqrd,ds->pqrs", d, U)
                tau0 = d - d.transpose(0, 1)
                k1, k5 = e("cd,dabc->ab", Y, tau0), e("cd,adcb->ab", Y, tau0)
                s8 = -e("ab,ba->", Y, k1)
                m = -k1 - k5
                a14 = Y @ m
                a15 = e("ca,bc->ab", Y, a14)
                a21 = e("ca,bc->ab", Y, m)
                a2 = a1 - k1
                t3 = e("ab,ba->", Y, a2)
                t1 = t3 * Y
                a7 = k1 + k5 + Y @ (m + a1) - a1
                t1 = t1 - e("cb,ac->ab", Y, a7)
                b9 = e("ea,bcde->abcd", Y, d)
                b10 = e("ea,bcde->abcd", Y, b9)
                b12 = e("ae,bcde->abcd", Y, e("ae,bcde->abcd", Y, b10))
                x = b12 - e("ac,db->abcd", Y, a15)
                t2 = s8 * (e("ac,bd->abcd", Y, Y) - e("ad,bc->abcd", Y, Y))
                t2 = t2 + x - x.transpose(2, 3) - x.transpose(0, 1) + x.transpose(0, 1).transpose(2, 3)
                b19 = b10.transpose(2, 3) - b10
                b22 = e("ab,cd->abcd", Y, a21) - e("ae,bcde->abcd", Y, b19)
                t2 = t2 + e("acdb->abcd", b22) - e("adcb->abcd", b22) - e("bcda->abcd", b22) + e("bdca->abcd", b22)
                t2 = t2 + e("cdab->abcd", b10) - e("cdba->abcd", b10) - e("dcab->abcd", b10) + e("dcba->abcd", b10)
                a17 = e("ca,bc->ab", Y, a1)
                a18 = e("ac,bc->ab", Y, a17)
                t2 = t2 - e("ac,bd->abcd", Y, a18) + e("bc,ad->abcd", Y, a18) + e("ac,db->abcd", Y, a17) - e("bc,da->abcd", Y, a17)
                a27 = e("ba,ab->", Y, a1) * Y.T - e("ca,bc->ab", Y, Y @ a1 - a1) + c0 * Y.T
                t2 = t2 + e("bd,ca->abcd", Y, a27) - e("ad,cb->abcd", Y, a27)
                s = g.weightsp[il, iy] * g.weightpg[ig, 0, 0] * torch.linalg.det(R[:N, :N])
                out = [q + s * y for q, y in zip(out, (t3 + c0, t1 + c0 * Y, t2))]
                ovl = ovl + s
    return tuple((q / ovl).cpu().numpy() for q in out)


def exact(case, seed):
    if case["kind"] == "batch":
        sums = [_hf_sums(p, p.C) for p in _batch_problems(case, seed)]
        return [tuple(x[None] for x in s) for s in sums]
    if case["kind"] == "pcc":
        return _exact_pcc(case, seed)
    if case["kind"] == "buildsc":
        return _exact_buildsc(case, seed)
    return _exact_hf(case, seed)
