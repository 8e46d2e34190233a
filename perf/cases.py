"""The calls that a user of this library makes, as cases to be timed.

Every case is one call of a public entry point of the Python mirror (or, where the
caller's arrays live on the device, of the C ABI) with a resident Hops handle, as a
program that calls it in a loop holds it:

  bands   ``bandmatrix``: eigenvalues on a list of k-points
  bdr     ``bands_dos_rho``: bands, DOS and rho_R from one eigen pass
  rho     ``lqm_densitymatrix_dev``: rho_R and the band energy into device arrays
  mu      ``chemicalpotential`` at T = 0 or T > 0
  vjp     ``densitymatrix_vjp``: the reverse pass of rho_R
  kubo    ``opticalconductivity``: chi_xx(omega)
  scf     ``solvehartreefock``: a fixed number of Hartree-Fock iterations

Models are the repository's own (honeycomb supercells, the kagome and triangular
cells of the batched workload, the triangular Hubbard cell, twisted bilayers), with
on-site disorder from the seed; orders in between come from the next larger
supercell with vacancies.  k-points: the regular grid with a random offset (a Monkhorst
shift), or random points of the zone for a list of odd length.
"""
import ctypes
import functools
import math
import os
import sys
import warnings

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "latticeqm.jl_b200", "python")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lqm_cuda as Q  # noqa: E402
from lqm_workloads import lattice as L  # noqa: E402
from lqm_workloads import models as M  # noqa: E402

TWISTED = {4 * (3 * m * m + 3 * m + 1): m for m in range(1, 16)}  # orders of the twisted bilayers
LARGEST = 6.0e10  # n^3 nk of a drawn case; the largest listed one has 8.6e11


def listed():
    return [
        # the reference benchmark's smallest entry: a k-path of the graphene cell; launches and latency
        {"name": "path_n2_k128", "kind": "bands", "model": "cell", "n": 2, "nk": 128},
        # its dense twisted bilayers, the 32-point path of n = 364
        {"name": "path_n364_k32", "kind": "bands", "model": "cell", "n": 364, "nk": 32},
        # the k-path of the m = 10 twisted bilayer
        {"name": "path_n1324_k100", "kind": "bands", "model": "cell", "n": 1324, "nk": 100},
        # the batched workload's kagome cell on its 256 x 256 grid
        {"name": "bdr_n24_k65536", "kind": "bdr", "model": "kagome", "n": 24, "nk": 65536, "nw": 500},
        # its spin-orbit triangular cell, on a 90 x 90 grid
        {"name": "rho_n96_k8100", "kind": "rho", "model": "triangular", "n": 96, "nk": 8100, "T": 0.01},
        # spinful honeycomb 6 x 6 with on-site disorder, 48 x 48 grid (every level twofold)
        {"name": "rho_n144_k2304", "kind": "rho", "model": "honeycomb", "n": 144, "nk": 2304, "T": 0.01},
        # the m = 10 twisted bilayer on a 12 x 12 grid
        {"name": "rho_n1324_k144", "kind": "rho", "model": "cell", "n": 1324, "nk": 144, "T": 0.01},
        # the largest configuration, m = 15, on a 6 x 6 grid
        {"name": "rho_n2884_k36", "kind": "rho", "model": "cell", "n": 2884, "nk": 36, "T": 0.01},
        # chemical potential of a mid-size cell: one eigen pass, then the search
        {"name": "mu_n51_k1024", "kind": "mu", "model": "cell", "n": 51, "nk": 1024, "T": 0.02},
        # the reverse pass of rho on the triangular Hubbard cell, 36 x 36 grid
        {"name": "vjp_n72_k1296", "kind": "vjp", "model": "hubbard", "n": 72, "nk": 1296, "T": 0.02},
        # optical conductivity of the honeycomb cell, 48 x 48 grid, 64 frequencies
        {"name": "kubo_n144_k2304", "kind": "kubo", "model": "honeycomb", "n": 144, "nk": 2304, "nw": 64},
        # Hartree-Fock on the triangular Hubbard cell, 36 x 36 grid
        {"name": "scf_n72_k1296", "kind": "scf", "model": "hubbard", "n": 72, "nk": 1296, "T": 0.02, "iterations": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: orders between 2 and about 1300, lists of 16 to 65536 k-points.  Odd
    orders are among them; the passes with eigenvectors take them from 113 on only, because
    below that the one-CTA kernel as it was first timed faulted on them."""
    kind = rng.choice(["bands", "bands", "bdr", "rho", "rho", "mu", "vjp", "kubo", "scf"])
    top = {"bands": 1300, "rho": 1300, "bdr": 700, "mu": 400, "vjp": 300, "kubo": 300, "scf": 100}[kind]
    n = _log(rng, 2, top)
    if kind not in ("bands", "mu") and n < 112:
        n += n % 2
    most = {"vjp": 3000, "kubo": 3000, "scf": 1500}.get(kind, 65536)
    nk = _log(rng, 16, max(20, min(most, int(LARGEST / n ** 3))))
    if rng.random() < 0.4:
        nk = max(4, math.isqrt(nk)) ** 2  # a square grid
    case = {"kind": kind, "model": "cell", "n": n, "nk": nk}
    if kind in ("rho", "mu", "vjp"):
        case["T"] = rng.choice([0.01, 0.02, 0.1])
    if kind == "rho" and rng.random() < 0.2:
        case["T"] = 0.0
    if kind in ("bdr", "kubo"):
        case["nw"] = rng.randint(16, 500 if kind == "bdr" else 100)
    if kind == "scf":
        side = rng.randint(2, 7)
        case.update(model="hubbard", n=2 * side * side, T=rng.choice([0.02, 0.1]), iterations=rng.randint(4, 8))
    return case


# ----------------------------------------------------------------------------- models
@functools.lru_cache(maxsize=None)
def _twisted(m):
    return M.tbg_slater_koster(m)


@functools.lru_cache(maxsize=None)
def _honeycomb_cell(side):
    lat = L.superlattice(L.honeycomb(), [side, side])
    return lat, M.graphene(lat, tz=0.0, tmin=1e-3)


@functools.lru_cache(maxsize=None)
def _spinful_honeycomb():
    return M.honeycomb_disorder(6, sigma=0.0)


@functools.lru_cache(maxsize=None)
def _hubbard(side):
    return M.triangular_hubbard(L_super=side)


def _model(case, seed):
    """(positions, primitive vectors, Hops) of a case's model with the seed's disorder."""
    n, rng = case["n"], np.random.default_rng(seed)
    kind = case["model"]
    if kind in ("kagome", "triangular"):
        return None, None, M.batch_models(seed)[1 if kind == "kagome" else 2][1]
    if kind == "hubbard":
        lat, h, _ = _hubbard(math.isqrt(n // 2))
        eps = np.repeat(rng.normal(0.0, 0.1, n // 2), 2)
        keep = np.arange(n)
    elif kind == "honeycomb":
        lat, h = _spinful_honeycomb()
        eps = np.repeat(rng.normal(0.0, 0.1, n // 2), 2)
        keep = np.arange(n)
    else:
        if n > 224 or n in TWISTED:
            parent = min(p for p in TWISTED if p >= n)
            lat, h = _twisted(TWISTED[parent])
            sigma = 0.05
        else:
            lat, h = _honeycomb_cell(math.isqrt((n + 1) // 2 - 1) + 1)
            parent = lat.norb
            sigma = 0.1
        keep = np.sort(rng.permutation(parent)[:n])  # the others are vacancies
        eps = rng.normal(0.0, sigma, n)
    h = {R: (B if len(keep) == len(B) else B[np.ix_(keep, keep)]) for R, B in h.items()}
    h[(0, 0)] = h[(0, 0)] + np.diag(eps)
    return lat, keep, h


def _kpoints(case, seed):
    rng = np.random.default_rng(1000003 * (seed % 1000) + 17)
    nk = case["nk"]
    side = math.isqrt(nk)
    if side * side == nk and case["kind"] != "bands":
        return np.asfortranarray(L.regulargrid(nk) + rng.uniform(0.0, 1.0 / side, (2, 1)))
    if case["kind"] == "bands":  # a straight piece of a path
        a, b = rng.uniform(-0.5, 0.5, 2), rng.uniform(-0.5, 0.5, 2)
        return np.asfortranarray(a[:, None] + (b - a)[:, None] * np.linspace(0.0, 1.0, nk))
    return np.asfortranarray(rng.uniform(-0.5, 0.5, (2, nk)))


def _cotangent(case, seed):
    rng = np.random.default_rng(seed + 5)
    n = case["n"]
    return {R: rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)) for R in ((0, 0), (1, 0))}


def _frequencies(case):
    return np.linspace(0.0, 3.0, case["nw"]) if case["kind"] == "kubo" else np.linspace(-6.0, 6.0, case["nw"])


def _width(case):
    return 0.05


# ----------------------------------------------------------------------------- the calls
_CTX = None


def _context():
    global _CTX
    if _CTX is None:
        _CTX = Q.Context(0, timeout=600)
    return _CTX


def prepare(case, seed):
    ctx = _context()
    lat, keep, h = _model(case, seed)
    s = {"case": case, "ctx": ctx, "H": Q.DeviceHops(h, ctx), "ks": _kpoints(case, seed), "keys": list(h)}
    kind = case["kind"]
    if kind == "rho":
        n, nL = case["n"], len(h)
        s["d_ks"] = torch.from_numpy(np.ascontiguousarray(s["ks"].T)).cuda()
        s["Lk"] = np.asfortranarray(np.array(s["keys"], dtype=np.int64).T)
        s["rho"] = torch.zeros(nL, n, n, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
    elif kind == "vjp":
        s["G"] = _cotangent(case, seed)
    elif kind == "kubo":
        s["J"] = Q.DeviceHops(_current(lat, keep, h), ctx)
    elif kind == "scf":
        n = case["n"]
        v = _hubbard(math.isqrt(n // 2))[2]
        s["V"] = Q.DeviceHops(v, ctx)
        s["rho0"] = {R: np.zeros((n, n), complex) for R in v}
        s["rho0"][(0, 0)] = M.random_local_magnetization(n // 2, seed=seed)
    return s


def _current(lat, keep, h):
    """The x current operator of the kept orbitals (``currentoperators``, alpha = 0)."""
    r, A = lat.positions(), lat.basis[:, :2]
    x = np.repeat(r[0], max(1, len(keep) // r.shape[1]))[keep]
    return {R: B * (-1j * (x[:, None] + (A @ np.array(R, float))[0] - x[None, :])) for R, B in h.items()}


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "bands":
        return Q.bandmatrix(s["H"], s["ks"], ctx=ctx)[0]
    if kind == "bdr":
        rho = {R: None for R in s["keys"]}
        bands, dos, energy = Q.bands_dos_rho(rho, s["H"], s["ks"], _frequencies(case), _width(case), ctx=ctx)
        return {"bands": bands, "dos": dos, "energy": np.float64(energy), "rho": np.stack(list(rho.values()))}
    if kind == "rho":
        energy = ctypes.c_double()
        ctx.check(Q.lib().lqm_densitymatrix_dev(
            ctx.handle, s["H"].handle, case["nk"], Q._ptr(s["d_ks"]), None, 0.0, case["T"], len(s["keys"]),
            Q._ptr(s["Lk"]), Q._ptr(s["rho"]), ctypes.byref(energy), 0))
        return {"rho": s["rho"], "energy": np.float64(energy.value)}
    if kind == "mu":
        return np.array([Q.chemicalpotential(s["H"], s["ks"], 0.37, T=T, ctx=ctx) for T in (0.0, case["T"])])
    if kind == "vjp":
        return np.stack(list(Q.densitymatrix_vjp(s["H"], s["ks"], s["G"], mu=0.0, T=case["T"], ctx=ctx).values()))
    if kind == "kubo":
        return Q.opticalconductivity(_frequencies(case), s["H"], s["J"], s["J"], s["ks"], Gamma=_width(case),
                                     T=0.01, ctx=ctx)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # a fixed number of iterations, converged or not
        r = Q.solvehartreefock(s["H"], s["V"], s["rho0"], 0.5, s["ks"], T=case["T"], beta=0.3, tol=0.0,
                               iterations=case["iterations"], ctx=ctx)
    return {"rho": np.stack(list(r.rho.values())), "energy": np.float64(r.energy), "mu": np.float64(r.mf.mu)}


# ----------------------------------------------------------------------------- what it takes
def _keys(case):
    return {"kagome": 9, "triangular": 9, "honeycomb": 9}.get(case["model"], 7)


def work(case):
    """Reduction to a tridiagonal (16/3 n^3), eigenvectors (8 n^3) and rho_k (4 n^3) per
    k-point as real operations, and the sums over the keys; bytes: H, k-points and results."""
    n, nk, nR, kind = case["n"], case["nk"], _keys(case), case["kind"]
    per = 8.0 * nR * n * n + 16.0 / 3.0 * n ** 3
    byte = 16.0 * nR * n * n + 16.0 * nk
    if kind in ("bdr", "rho"):
        per += 12.0 * n ** 3 + 8.0 * nR * n * n
        byte += 16.0 * nR * n * n
    if kind in ("bands", "bdr"):
        byte += 8.0 * n * nk
    if kind == "bdr":
        per += 6.0 * case["nw"] * n
        byte += 16.0 * case["nw"]
    if kind == "mu":
        per *= 2  # two calls
        byte = 2 * byte + 16
    if kind == "vjp":
        per += 8.0 * n ** 3 + 32.0 * n ** 3 + 8.0 * (2 + nR) * n * n
        byte += 16.0 * (2 + nR) * n * n
    if kind == "kubo":
        per += 8.0 * n ** 3 + 16.0 * n ** 3 + 8.0 * nR * n * n + 10.0 * case["nw"] * n * n
        byte += 16.0 * nR * n * n + 24.0 * case["nw"]
    if kind == "scf":
        return {"bytes": 2 * byte, "flops": case["iterations"] * nk * (per + 12.0 * n ** 3)}
    return {"bytes": byte, "flops": per * nk}


# ----------------------------------------------------------------------------- 64-bit values
def _blocks(h):
    return (torch.tensor(np.array(list(h)), dtype=torch.float64, device="cuda"),
            torch.from_numpy(np.stack([np.asarray(B, dtype=complex) for B in h.values()])).cuda())


def _eigen(h, ks, vectors=True):
    """Chunks (k0, k1, phases e^{i 2 pi k.R}, eigenvalues, eigenvectors) of H(k)."""
    keys, blocks = _blocks(h)
    n = blocks.shape[1]
    kt = torch.from_numpy(np.ascontiguousarray(ks.T)).cuda()
    step = max(1, int(2.0e8 / (16 * n * n)))
    for k0 in range(0, kt.shape[0], step):
        ph = torch.exp(2j * math.pi * (kt[k0:k0 + step] @ keys.T))
        Hk = torch.einsum("kr,rij->kij", ph, blocks)
        up = torch.triu(Hk, 1)
        Hk = up + up.mH + torch.diag_embed(torch.diagonal(Hk, dim1=-2, dim2=-1).real.to(Hk.dtype))
        if vectors:
            e, U = torch.linalg.eigh(Hk)
        else:
            e, U = torch.linalg.eigvalsh(Hk), None
        yield k0, min(k0 + step, kt.shape[0]), ph, e, U


def _occupation(x, T):
    return torch.special.expit(-x / T) if T > 0 else torch.heaviside(-x, torch.full((), 0.5, dtype=x.dtype, device=x.device))


def _gemm_order(x):
    """(keys, n, n) row-major blocks -> the column-major device layout of the library."""
    return x.transpose(-1, -2).contiguous()


def _root(bands, filling, T):
    """The chemical potential of a uniform k-sum."""
    x = bands.reshape(-1)
    if T == 0:
        s, i = torch.sort(x).values, int(math.floor(filling * (x.numel() - 1)))
        return float((s[i] + s[i + 1]) / 2)
    lo, hi = float(x.min()), float(x.max())
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        if float(_occupation(x - mid, T).mean()) < filling:
            lo = mid
        else:
            hi = mid
    return 0.5 * (lo + hi)


def _seconds(case):
    """A dense eigensolve of each k-point takes about this long (a loop over them beyond n = 32)."""
    n = case["n"]
    return case["nk"] * case.get("iterations", 1) * (2e-6 if n <= 32 else 1.5e-3 + 1.2e-8 * n * n)


def exact(case, seed):
    kind, n, nk = case["kind"], case["n"], case["nk"]
    if _seconds(case) > 18.0:
        return None
    lat, keep, h = _model(case, seed)
    ks = _kpoints(case, seed)
    if kind in ("bands", "mu"):
        bands = torch.cat([e for _, _, _, e, _ in _eigen(h, ks, vectors=False)])
        if kind == "bands":
            return bands.T.contiguous().cpu().numpy()
        return np.array([_root(bands, 0.37, T) for T in (0.0, case["T"])])
    if kind in ("bdr", "rho"):
        T = case.get("T", 0.01)
        rho, energy, bands = 0.0, 0.0, []
        for k0, k1, ph, e, U in _eigen(h, ks):
            f = _occupation(e, T)
            rho = rho + torch.einsum("kr,kij->rij", ph.conj() / nk, (U * f[:, None, :]) @ U.mH)
            energy += float((f * e).sum()) / nk
            bands.append(e)
        if kind == "rho":
            return {"rho": _gemm_order(rho), "energy": np.float64(energy)}
        e = torch.cat(bands)
        om = torch.from_numpy(_frequencies(case)).cuda()
        g = _width(case)
        dos = torch.stack([(g / ((w - e) ** 2 + g * g)).sum() / nk for w in om])
        return {"bands": e.T.contiguous().cpu().numpy(), "dos": dos.cpu().numpy(),
                "energy": np.float64(energy), "rho": rho.cpu().numpy()}
    if kind == "vjp":
        G = _cotangent(case, seed)
        gk, gb = _blocks(G)
        kt = torch.from_numpy(np.ascontiguousarray(ks.T)).cuda()
        out, T = 0.0, case["T"]
        for k0, k1, ph, e, U in _eigen(h, ks):
            # rho_L = sum_k w e^{-i 2 pi k.L} rho_k, so the cotangent of rho_k is sum_L w e^{+i 2 pi k.L} G_L
            Gk = torch.einsum("kl,lij->kij", torch.exp(2j * math.pi * (kt[k0:k1] @ gk.T)) / nk, gb)
            f = _occupation(e, T)
            d = e[:, :, None] - e[:, None, :]
            mid = (e[:, :, None] + e[:, None, :]) / 2
            # (f_i - f_j) / (e_i - e_j) = -sinh(d/2T) / (d (cosh(mid/T) + cosh(d/2T))), with the limit at d = 0
            a = (mid / T).abs()
            b = (d / (2 * T)).abs()
            top = torch.where(b > 1e-8, -torch.expm1(-2 * b) / torch.where(b > 1e-8, b, torch.ones_like(b)),
                              torch.full_like(b, 2.0))
            big = torch.maximum(a, b)
            F = -top * torch.exp(b - big) / (2 * T) / (torch.exp(a - big) + torch.exp(-a - big)
                                                       + torch.exp(b - big) + torch.exp(-b - big))
            Hb = U @ ((U.mH @ Gk @ U) * F) @ U.mH
            out = out + torch.einsum("kr,kij->rij", ph.conj(), Hb)
        return out.cpu().numpy()
    if kind == "scf":
        return _scf(case, seed, h, ks)
    jk, jb = _blocks(_current(lat, keep, h))
    kt = torch.from_numpy(np.ascontiguousarray(ks.T)).cuda()
    om, g = torch.from_numpy(_frequencies(case)).cuda(), _width(case)
    chi = torch.zeros(len(om), dtype=torch.complex128, device="cuda")
    for k0, k1, ph, e, U in _eigen(h, ks):
        Jk = torch.einsum("kr,rij->kij", torch.exp(2j * math.pi * (kt[k0:k1] @ jk.T)), jb)
        # sum_{i != j} (f_i - f_j) (U^H J U)_ij (U^H J^H U)_ji / (e_i - e_j - omega - i Gamma)
        m = (U.mH @ Jk @ U).abs() ** 2
        f = _occupation(e, 0.01)
        wt = ((f[:, :, None] - f[:, None, :]) * m).to(torch.complex128)
        d = e[:, :, None] - e[:, None, :]
        for i, w in enumerate(om):
            chi[i] += (wt / (d - w - 1j * g)).sum()
    return (chi * (-1j / nk)).cpu().numpy()


def _scf(case, seed, h, ks):
    """Hartree-Fock with an on-site v: hMF = h - v .* rho + diag(v diag rho), linear mixing."""
    n, nk, T, beta = case["n"], case["nk"], case["T"], 0.3
    (v,) = _hubbard(math.isqrt(n // 2))[2].values()
    rho = M.random_local_magnetization(n // 2, seed=seed)
    rho = (rho + rho.conj().T) / 2

    def field(rho):
        d = np.diag(rho)
        energy = 0.5 * np.real(d @ v @ d) - 0.5 * np.real(np.sum(rho * rho.conj() * v))
        return {R: (B - v * rho + np.diag(v @ d) if R == (0, 0) else B) for R, B in h.items()}, energy

    for _ in range(case["iterations"]):
        parts = [(e, U) for _, _, _, e, U in _eigen(field(rho)[0], ks)]
        mu = _root(torch.cat([e for e, _ in parts]), 0.5, T)
        new, band = 0.0, 0.0
        for e, U in parts:
            f = _occupation(e - mu, T)
            new = new + ((U * f[:, None, :]) @ U.mH).sum(0) / nk
            band += float((f * e).sum()) / nk
        rho = beta * new.cpu().numpy() + (1 - beta) * rho
    energy = band - field(rho)[1]
    return {"rho": (rho + rho.conj().T)[None] / 2, "energy": np.float64(energy), "mu": np.float64(mu)}
