"""The work a user has this library do, as cases that can be timed and checked one by one.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same ranges; ``prepare`` makes
what a program holds before the call (a context with its gauge field, sources, weights), ``run`` is
one pass through the public entry points, ``work`` the bytes and operations the pass cannot do
without, and ``exact`` the same results from plain torch in 64 bits.

Gauge fields are hot starts U = exp(i eps H), periodic in space and antiperiodic in time; sources
are those the callers use (spin-colour points for propagators, Gaussian or Z2 noise on the odd
sites for the rest).  Solves go to a fixed true residual, as a caller sets it.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
DEV = "cuda" if torch.cuda.is_available() else "cpu"
WEIGHTS16 = os.path.join(ROOT, "chroma_gb300", "weights", "cnn_16x16x16x32_k0.115_csw1.0.gbcw")


def _case(kind, dims, nrhs=1, kappa=0.125, csw=1.6, **kw):
    return dict(kind=kind, dims=dims, nrhs=nrhs, kappa=kappa, csw=csw, **kw)


def listed():
    return [
        # the benchmark's propagator: 12 point sources as one batch, full system, resident on the GPU
        dict(name="propagator_32", **_case("propagator", "32x32x32x64", 12)),
        # the same call on an ordinary test-sized configuration
        dict(name="propagator_16", **_case("propagator", "16x16x16x32", 12)),
        # a propagator's twelve calls as a factory-only Chroma input makes them: one right-hand side,
        # odd-site system, the default solver, host buffers
        dict(name="linop_24", **_case("linop", "24x24x24x48", solver="mixed", prec="half")),
        # one molecular-dynamics step of a smeared-link HMC: smear, load the links, solve M~^dag M~
        dict(name="hmc_16", **_case("hmc", "16x16x16x32", kappa=0.12, csw=1.2, n_stout=2, prec="single")),
        # the rational approximation's shifted systems of RHMC
        dict(name="rhmc_16", **_case("rhmc", "16x16x16x32", kappa=0.12, csw=1.2, shifts=8, prec="half")),
        # the symmetric operator (SEOPREC_CLOVER) with full links: a few sources, FP32, ragged extents
        dict(name="symmetric_12", **_case("symmetric", "12x12x10x22", 3, kappa=0.12, csw=1.4, prec="single")),
        # plain FP64 CG on a small lattice: what tests and tuning runs call all the time
        dict(name="cg_8", **_case("cg", "8x8x8x16", kappa=0.12, csw=1.2)),
        # independent configurations of uneven extents solved together
        dict(name="batch_4", **_case("batch", "8x8x8x16,12x12x12x24,16x16x16x32,20x20x20x40", kappa=0.124, csw=1.5)),
        # the flexible GMRES with the trained network on the lattice it was trained for
        dict(name="learned_16", **_case("learned", "16x16x16x32", kappa=0.115, csw=1.0)),
        # the network by itself on a propagator's sources (building pairs, checking weights)
        dict(name="network_16", **_case("network", "16x16x16x32", 12, kappa=0.115, csw=1.0)),
        # one training step's loss and gradient, forward and backward
        dict(name="training_16", **_case("training", "16x16x16x32", 4, kappa=0.115, csw=1.0)),
        # one FP64 operator application on the caller's own device buffers: the smallest call
        dict(name="operator_8", **_case("operator", "8x8x8x8", kappa=0.115, csw=1.0)),
    ]


# kind -> (smallest, largest number of sites) that draw() takes
RANGE = {
    "propagator": (4096, 32 ** 3 * 64), "linop": (4096, 24 ** 3 * 48), "hmc": (4096, 20 ** 3 * 40),
    "rhmc": (4096, 20 ** 3 * 40), "symmetric": (2048, 20 ** 3 * 40), "cg": (1024, 16 ** 3 * 32),
    "batch": (1024, 20 ** 3 * 40), "learned": (8192, 20 ** 3 * 40), "network": (4096, 20 ** 3 * 40),
    "training": (4096, 16 ** 3 * 32), "operator": (1024, 2 * 65536),
}


def _draw_dims(rng, lo, hi):
    """Even extents, the volume spread over its logarithm, the time extent up to twice the others."""
    for _ in range(10000):
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        s = (v / 2) ** 0.25
        d = [max(4, 2 * round(s * rng.uniform(0.7, 1.4) / 2)) for _ in range(3)]
        d.append(max(4, 2 * round(v / (d[0] * d[1] * d[2]) / 2)))
        n = d[0] * d[1] * d[2] * d[3]
        if lo <= n <= hi and d[3] <= 96:
            return "x".join(map(str, d))
    raise RuntimeError("no lattice in range")


def draw(rng):
    kind = rng.choice(sorted(RANGE))
    lo, hi = RANGE[kind]
    c = _case(kind, _draw_dims(rng, lo, hi), kappa=round(rng.uniform(0.115, 0.125), 4), csw=round(rng.uniform(1.0, 1.6), 2))
    if kind == "propagator":
        c["nrhs"] = rng.choice([3, 4, 6, 8, 12, 12])
    elif kind == "linop":
        c["solver"], c["prec"] = rng.choice(["mixed", "bicgstab", "fgmres"]), rng.choice(["half", "single"])
    elif kind == "hmc":
        c["n_stout"], c["prec"] = rng.randint(1, 3), rng.choice(["half", "single"])
    elif kind == "rhmc":
        c["shifts"], c["prec"] = rng.randint(3, 12), rng.choice(["half", "single", "double"])
    elif kind == "symmetric":
        c["nrhs"], c["prec"] = rng.randint(1, 7), rng.choice(["half", "single"])
    elif kind == "batch":
        c["dims"] = ",".join([c["dims"]] + [_draw_dims(rng, lo, hi // 4) for _ in range(rng.randint(1, 4))])
    elif kind in ("learned", "network", "training"):
        c["kappa"], c["csw"] = 0.115, 1.0
        if kind != "learned":
            c["nrhs"] = rng.randint(1, 12 if kind == "network" else 4)
    return c


# ---- inputs -----------------------------------------------------------------------------------
def _dims(text):
    return tuple(int(x) for x in text.split("x"))


def _parity(dims):
    """(x + y + z + t) mod 2 of every site, site index x fastest."""
    t, z, y, x = torch.meshgrid(*[torch.arange(n, device=DEV) for n in reversed(dims)], indexing="ij")
    return ((x + y + z + t) % 2).reshape(-1)


def _links(dims, eps, seed, boundary=True):
    """U = exp(i eps H), H traceless Hermitian with unit Gaussian entries, as (V, 4, 3, 3)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    V = math.prod(dims)
    a = torch.randn(V * 4, 3, 3, 2, dtype=torch.float64, device=DEV, generator=g)
    a = torch.view_as_complex(a)
    h = 0.5 * (a + a.mH)
    eye = torch.eye(3, dtype=h.dtype, device=DEV)
    h = h - eye * (h.diagonal(dim1=-2, dim2=-1).sum(-1) / 3)[:, None, None]
    h = h * (1j * eps / 8)
    u = eye + h / 12
    for k in range(11, 0, -1):
        u = eye + torch.matmul(h, u) / k
    for _ in range(3):
        u = torch.matmul(u, u)
    u = u.reshape(V, 4, 3, 3)
    if boundary:
        _antiperiodic(u, dims)
    return u


def _antiperiodic(u, dims):
    n = dims[0] * dims[1] * dims[2]
    u[u.shape[0] - n:, 3] *= -1


def _noise(dims, n, seed, odd=True):
    g = torch.Generator(device=DEV).manual_seed(seed + 77)
    v = torch.randn(n, math.prod(dims), 12, 2, dtype=torch.float64, device=DEV, generator=g)
    v = torch.view_as_complex(v)
    return v * _parity(dims)[None, :, None] if odd else v


def _z2(dims, n, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 99)
    v = torch.randint(0, 2, (n, math.prod(dims), 12, 2), device=DEV, generator=g).double() * 2 - 1
    return torch.view_as_complex(v / math.sqrt(2.0)) * _parity(dims)[None, :, None]


def _points(dims, n, seed):
    """n of the 12 spin-colour sources at a seeded origin, in the order colour * 4 + spin."""
    r = np.random.default_rng(seed)
    x = [int(r.integers(0, k)) for k in dims]
    site = x[0] + dims[0] * (x[1] + dims[1] * (x[2] + dims[2] * x[3]))
    v = torch.zeros(n, math.prod(dims), 12, dtype=torch.complex128, device=DEV)
    for k in range(n):
        v[k, site, (k % 4) * 3 + k // 4] = 1.0
    return v


def _shifts(n):
    """Shifts of a rational approximation: spread over their logarithm."""
    return [float(x) for x in np.geomspace(1e-3, 2.0, n)]


def _weights(seed, hidden=12, layers=4):
    """Network weights near a trained network's: close to the identity map, small hops."""
    r = np.random.default_rng(seed + 5)
    out = []
    for l in range(layers):
        ci, co = 4 if l == 0 else hidden, 4 if l == layers - 1 else hidden
        w = (r.standard_normal((9, co, ci)) + 1j * r.standard_normal((9, co, ci))) * 0.05
        for o in range(co):
            for i in range(ci):
                if o % ci == i or (ci > co and i % co == o):
                    w[0, o, i] += 1.0 if ci <= co else co / ci
        out.append(w.astype(np.complex64))
    return out


def _inputs(case, seed):
    """Gauge fields (with the boundary sign unless they are smeared first) and sources of a case."""
    kind, n = case["kind"], case["nrhs"]
    if kind == "batch":
        lats = [_dims(t) for t in case["dims"].split(",")]
        return [_links(d, 0.3, seed * 16 + k) for k, d in enumerate(lats)], [_z2(d, 1, seed * 16 + k)[0] for k, d in enumerate(lats)]
    dims = _dims(case["dims"])
    u = _links(dims, 0.2 if kind == "hmc" else 0.3, seed, boundary=kind != "hmc")
    if kind == "propagator":
        return u, _points(dims, n, seed)
    if kind == "linop":
        return u, _z2(dims, n, seed)
    return u, _noise(dims, n, seed, odd=kind != "operator")


# ---- the passes -------------------------------------------------------------------------------
def _mass(case):
    return 1 / (2 * case["kappa"]) - 4


def prepare(case, seed):
    from chroma_gb300 import gbclover as G
    kind = case["kind"]
    u, src = _inputs(case, seed)
    st = {"case": case, "G": G}
    prec = {"half": G.PREC_HALF, "single": G.PREC_SINGLE, "double": G.PREC_DOUBLE}.get(case.get("prec"), G.PREC_HALF)
    st["prec"] = prec
    if kind == "batch":
        st["ctxs"] = []
        for k, t in enumerate(case["dims"].split(",")):
            c = G.Context(_dims(t), _mass(case), case["csw"], max_rhs=1)
            c.load_gauge(u[k].cpu().numpy())
            st["ctxs"].append(c)
        st["batch"] = G.Batch(st["ctxs"])
        st["src"] = [s.cpu().numpy() for s in src]
        return st
    dims = _dims(case["dims"])
    links = u.cpu().numpy()
    ctx = st["ctx"] = G.Context(dims, _mass(case), case["csw"], max_rhs=max(1, case["nrhs"], case.get("shifts", 1)),
                                sloppy_precision=G.PREC_SINGLE if kind == "symmetric" else prec,
                                sloppy_reconstruct=G.RECON_18 if kind == "symmetric" else G.RECON_12)
    ctx.load_gauge(links)
    if kind == "hmc":
        st["links"] = links
    if kind == "propagator":
        st["chi"], st["psi"] = src, torch.zeros_like(src)
        return st
    if kind == "operator":
        clov, inv, _, _ = ctx.get_clover()
        st["geom"] = G.Geom((ctypes.c_int * 4)(*dims), -1)
        st["act"] = G.Action(_mass(case), case["csw"], case["csw"], 0, 1.0, 1.0, 3, 0, 0.0)
        lib = G.load()
        lib.gbc_apply_meo_noalloc.argtypes = [ctypes.POINTER(G.Geom), ctypes.POINTER(G.Action)] + [ctypes.c_void_p] * 3 + [ctypes.c_int] + [ctypes.c_void_p] * 3
        st["dev"] = [u, torch.from_numpy(clov).to(DEV), torch.from_numpy(inv).to(DEV)]
        st["in"], st["out"] = src[0], torch.zeros_like(src[0])
        st["call"] = lib.gbc_apply_meo_noalloc
        st["args"] = [ctypes.byref(st["geom"]), ctypes.byref(st["act"])] + [t.data_ptr() for t in st["dev"]] + [
            1, st["out"].data_ptr(), st["in"].data_ptr()]
        return st
    st["src"] = src.cpu().numpy()
    if kind == "learned":
        ctx.load_precond(WEIGHTS16)
    elif kind in ("network", "training"):
        ctx.precond_init(hidden=12, layers=4, seed=1)
        w = np.concatenate([x.reshape(-1) for x in _weights(seed)])
        ctx.precond_set_weights(w.view(np.float32))
    if kind == "training":
        st["target"] = (src + 0.3 * _noise(dims, case["nrhs"], seed + 1)).cpu().numpy()
    return st


def _converged(status):
    if status:
        raise RuntimeError("the solve did not converge: status %d" % status)


def run(st):
    G, case = st["G"], st["case"]
    kind, ctx = case["kind"], st.get("ctx")
    if kind == "propagator":
        _, rc = ctx.solve_device(st["psi"].data_ptr(), st["chi"].data_ptr(), case["nrhs"], solver=G.SOLVER_BICGSTAB,
                                 system=G.SYS_FULL, rsd_target=1e-10, delta=0.01, sloppy_precision=G.PREC_HALF,
                                 inner_tol=1e-5)
        _converged(rc)
        return st["psi"]
    if kind == "linop":
        kw = {"mixed": dict(solver=G.SOLVER_MIXED, inner_tol=1e-6),
              "bicgstab": dict(solver=G.SOLVER_BICGSTAB, delta=0.01, inner_tol=1e-5),
              "fgmres": dict(solver=G.SOLVER_FGMRES, nkrylov=16)}[case["solver"]]
        return ctx.solve(st["src"], system=G.SYS_MEO, rsd_target=1e-10, sloppy_precision=st["prec"], **kw)[0]
    if kind == "hmc":
        dims = _dims(case["dims"])
        u = G.stout_smear(dims, st["links"], case["n_stout"], 0.1)
        _antiperiodic(u, dims)
        ctx.load_gauge(u)
        psi = ctx.solve(st["src"], solver=G.SOLVER_MIXED, system=G.SYS_MDAGM, rsd_target=1e-11,
                        sloppy_precision=st["prec"])[0]
        return [u, psi]
    if kind == "rhmc":
        return ctx.solve_multishift(st["src"], _shifts(case["shifts"]), rsd_target=1e-11,
                                    sloppy_precision=st["prec"])[0]
    if kind == "symmetric":
        return ctx.solve(st["src"], solver=G.SOLVER_BICGSTAB, system=G.SYS_SYM, rsd_target=1e-10, delta=0.01,
                         inner_tol=1e-5, sloppy_precision=st["prec"])[0]
    if kind == "cg":
        return ctx.solve(st["src"], solver=G.SOLVER_CG, system=G.SYS_MEO, rsd_target=1e-10)[0]
    if kind == "batch":
        return st["batch"].solve(st["src"], rsd_target=1e-10)[0]
    if kind == "learned":
        return ctx.solve(st["src"], solver=G.SOLVER_FGMRES, system=G.SYS_MEO, rsd_target=1e-10, nkrylov=16,
                         use_precond=1, sloppy_precision=G.PREC_SINGLE)[0]
    if kind == "network":
        return ctx.precond_apply(st["src"])
    if kind == "training":
        loss, grad = ctx.precond_loss_grad(st["src"], st["target"])
        return {"loss": loss, "grad": grad}
    if kind == "operator":
        _converged(st["call"](*st["args"], torch.cuda.current_stream().cuda_stream))
        return st["out"]
    raise ValueError(kind)


# ---- what a pass cannot do without ----------------------------------------------------------------
# floating-point operations of M~ per odd site: two hopping terms of 1320 and two clover blocks of 504
MEO_FLOPS = 2 * 1320 + 2 * 504 + 48
# applications of M~ that a solve to these targets takes on these fields (Krylov counts in FP64)
APPLICATIONS = {"propagator": 90, "linop": 100, "hmc": 110, "rhmc": 120, "symmetric": 80, "cg": 220, "batch": 200,
                "learned": 20, "operator": 1}


def work(case):
    kind, n = case["kind"], case["nrhs"]
    V = sum(math.prod(_dims(t)) for t in case["dims"].split(","))
    links, spinor = 576.0 * V, 192.0 * V
    if kind in ("network", "training"):
        # per site and right-hand side: 8 transports and 9 channel mixings of the 4-12-12-12-4 layers
        pairs = 4 * 12 + 12 * 12 + 12 * 12 + 12 * 4
        fwd = V * n * (8.0 * 66 * (4 + 12 + 12 + 12) + 9 * 3 * 8 * pairs)
        if kind == "network":
            return {"bytes": links + 2 * n * spinor, "flops": fwd}
        return {"bytes": links + 2 * n * spinor + 8 * 9 * pairs, "flops": 3 * fwd}
    flops = V / 2 * n * MEO_FLOPS * APPLICATIONS[kind]
    byts = links + 2 * n * spinor
    if kind == "rhmc":
        byts = links + (1 + case["shifts"]) * spinor
    if kind == "hmc":
        byts += links
        flops += case["n_stout"] * V * 4 * 6 * 4 * 198.0
    if kind == "operator":
        byts = links + V / 2 * 2 * 576 + spinor
    if kind == "learned":
        flops *= 1 + 6
    return {"bytes": byts, "flops": flops}


# ---- the same results in 64 bits --------------------------------------------------------------
# DeGrand-Rossi gamma matrices, (gamma_mu psi)[s] = PHASE[mu][s] psi[PERM[mu][s]]
PERM = [[3, 2, 1, 0], [3, 2, 1, 0], [2, 3, 0, 1], [2, 3, 0, 1]]
PHASE = [[1j, 1j, -1j, -1j], [-1, 1, 1, -1], [1j, -1j, -1j, 1j], [1, 1, 1, 1]]


def _roll(f, mu, step):
    """f at x + step in direction mu; the sites are the leading dimensions (t, z, y, x)."""
    return torch.roll(f, -step, dims=3 - mu)


class _Wilson:
    """The clover operator on fields of shape (t, z, y, x, colour, spin, n)."""

    def __init__(self, dims, links, mass, csw):
        self.dims = dims
        self.shape = tuple(reversed(dims))
        self.u = [links[:, m].reshape(*self.shape, 3, 3) for m in range(4)]
        self.phase = torch.tensor(PHASE, dtype=torch.complex128, device=DEV)
        self.odd = _parity(dims).reshape(*self.shape, 1, 1, 1).bool()
        self.A = self._clover(mass, csw)
        self.Ainv = torch.linalg.inv(self.A)

    def _clover(self, mass, csw):
        """A = (4 + m) - csw/4 sigma.F as a dense (colour, spin) x (colour, spin) matrix per site."""
        gam = torch.zeros(4, 4, 4, dtype=torch.complex128, device=DEV)
        for m in range(4):
            for s in range(4):
                gam[m, s, PERM[m][s]] = PHASE[m][s]
        A = torch.zeros(*self.shape, 3, 4, 3, 4, dtype=torch.complex128, device=DEV)
        for m in range(4):
            for n in range(m + 1, 4):
                U, W = self.u[m], self.u[n]
                q = 0
                for sm, sn in ((1, 1), (-1, 1), (-1, -1), (1, -1)):
                    a = U if sm > 0 else _roll(U, m, -1).mH
                    b = W if sn > 0 else _roll(W, n, -1).mH
                    # the leaf x -> x+sm m -> +sn n -> back, its orientation that of the (m, n) plane
                    leaf = a @ _roll(b, m, sm) @ _roll(a, n, sn).mH @ b.mH
                    q = q + (leaf if sm * sn > 0 else leaf.mH)
                f = (q - q.mH) / 8
                s_mn = 0.5 * (gam[m] @ gam[n] - gam[n] @ gam[m])
                A += torch.einsum("tzyxab,SR->tzyxaSbR", f, s_mn) * (-csw / 2)
        A = A.reshape(*self.shape, 12, 12)
        return A + (4 + mass) * torch.eye(12, dtype=torch.complex128, device=DEV)

    def gamma(self, f, mu):
        return f[..., PERM[mu], :] * self.phase[mu][:, None]

    def g5(self, f):
        s = torch.tensor([1.0, 1.0, -1.0, -1.0], dtype=torch.float64, device=DEV)
        return f * s[:, None]

    def mul(self, u, f):
        return torch.matmul(u, f.reshape(*f.shape[:5], -1)).reshape(f.shape)

    def D(self, f):
        """sum_mu (1 - gamma_mu) U f(x + mu) + (1 + gamma_mu) U^dag f(x - mu)"""
        out = torch.zeros_like(f)
        for mu in range(4):
            h = _roll(f, mu, 1)
            out += self.mul(self.u[mu], h - self.gamma(h, mu))
            h = self.mul(self.u[mu].mH, f + self.gamma(f, mu))
            out += _roll(h, mu, -1)
        return out

    def block(self, A, f):
        return torch.matmul(A, f.reshape(*f.shape[:4], 12, -1)).reshape(f.shape)

    def even(self, f):
        return f.masked_fill(self.odd, 0)

    def odds(self, f):
        return f.masked_fill(~self.odd, 0)

    def meo(self, f, dag=False):
        if dag:
            return self.g5(self.meo(self.g5(f)))
        t = self.block(self.Ainv, self.even(self.D(f)))
        return self.block(self.A, f) - 0.25 * self.odds(self.D(t))

    def sym(self, f, dag=False):
        if dag:
            t = self.block(self.Ainv, self.even(self.g5(self.D(self.g5(self.block(self.Ainv, f))))))
            return f - 0.25 * self.odds(self.g5(self.D(self.g5(t))))
        t = self.block(self.Ainv, self.even(self.D(f)))
        return f - 0.25 * self.block(self.Ainv, self.odds(self.D(t)))

    def to(self, v):
        """(n, V, 12) with component spin * 3 + colour -> the layout of this class"""
        n = v.shape[0]
        return v.reshape(n, *self.shape, 4, 3).permute(1, 2, 3, 4, 6, 5, 0).contiguous()

    def back(self, f):
        return f.permute(6, 0, 1, 2, 3, 5, 4).reshape(f.shape[-1], math.prod(self.dims), 12)


def _cg(op, b, shift=0.0, tol=1e-14):
    """(op^dag op + shift) x = b on fields with the right-hand sides last, restarted once."""
    def mul(v):
        w = op(op(v), True)
        return w + shift * v if shift else w

    def dot(x, y):
        return (x.conj() * y).real.reshape(-1, x.shape[-1]).sum(0)

    x = torch.zeros_like(b)
    nb = dot(b, b)
    for _ in range(2):
        r = b - mul(x) if x.any() else b.clone()
        p, c = r.clone(), dot(r, r)
        for k in range(2000):
            if k % 10 == 0 and bool((c <= tol * tol * nb).all()):
                break
            q = mul(p)
            a = torch.where(c > 0, c / dot(p, q).clamp_min(1e-300), torch.zeros_like(c))
            x += a * p
            r -= a * q
            d = dot(r, r)
            p = r + torch.where(c > 0, d / c.clamp_min(1e-300), torch.zeros_like(c)) * p
            c = d
    return x


def _stout(u, dims, steps, rho):
    """Stout links exp(-rho/2 (W - W^dag - trace)) U, W = sum of staples times U^dag."""
    shape = tuple(reversed(dims))
    u = [u[:, m].reshape(*shape, 3, 3) for m in range(4)]
    eye = torch.eye(3, dtype=torch.complex128, device=DEV)
    for _ in range(steps):
        new = []
        for m in range(4):
            c = 0
            for n in range(4):
                if n == m:
                    continue
                c = c + u[n] @ _roll(u[m], n, 1) @ _roll(u[n], m, 1).mH
                c = c + _roll(u[n].mH @ u[m] @ _roll(u[n], m, 1), n, -1)
            w = rho * c @ u[m].mH
            w = 0.5 * (w - w.mH)
            w = (w - eye * (w.diagonal(dim1=-2, dim2=-1).sum(-1) / 3)[..., None, None]) / 8
            e = eye + w / 14
            for k in range(13, 0, -1):
                e = eye + w @ e / k
            for _ in range(3):
                e = e @ e
            new.append(e @ u[m])
        u = new
    return torch.stack([x.reshape(-1, 3, 3) for x in u], dim=1)


def _network(dims, links, w, x, odd):
    """The network's layers on (n, V, 12) in complex128; w: a tensor (9, out, in) per layer."""
    shape = tuple(reversed(dims))
    u = [links[:, m].reshape(*shape, 3, 3) for m in range(4)]
    h = x.reshape(-1, *shape, 4, 3).permute(1, 2, 3, 4, 6, 5, 0)  # (t, z, y, x, colour, channel, n)
    for W in w:
        terms = [h]
        for m in range(4):
            f = _roll(h, m, 1)
            terms.append((u[m] @ f.reshape(*shape, 3, -1)).reshape(f.shape))
            b = (u[m].mH @ h.reshape(*shape, 3, -1)).reshape(h.shape)
            terms.append(_roll(b, m, -1))
        h = sum(torch.einsum("oi,tzyxcin->tzyxcon", W[d], terms[d]) for d in range(9))
    return h.permute(6, 0, 1, 2, 3, 5, 4).reshape(x.shape) * odd[None, :, None]


def exact(case, seed):
    kind, n = case["kind"], case["nrhs"]
    if sum(math.prod(_dims(t)) for t in case["dims"].split(",")) * max(n, case.get("shifts", 1)) > 1_700_000:
        return None
    if kind == "batch":
        lats = [_dims(t) for t in case["dims"].split(",")]
        u, src = _inputs(case, seed)
        return [_solve(_Wilson(d, a, _mass(case), case["csw"]), "linop", s[None])[0] for d, a, s in zip(lats, u, src)]
    dims = _dims(case["dims"])
    u, src = _inputs(case, seed)
    odd = _parity(dims).bool()
    if kind in ("network", "training"):
        ws = [torch.from_numpy(x).to(DEV).to(torch.complex128) for x in _weights(seed)]
        if kind == "network":
            return _network(dims, u, ws, src, odd)
        target = src + 0.3 * _noise(dims, n, seed + 1)
        grads = [torch.zeros_like(w) for w in ws]
        loss = 0.0
        for k in range(n):
            leaf = [w.clone().requires_grad_(True) for w in ws]
            d = _network(dims, u, leaf, src[k:k + 1], odd) - target[k:k + 1]
            part = (d.abs() ** 2).sum() / (target[k].abs() ** 2).sum()
            for g, x in zip(grads, torch.autograd.grad(part, leaf)):
                g += x
            loss += float(part.detach())
        return {"loss": loss, "grad": torch.view_as_real(torch.cat([g.reshape(-1) for g in grads])).reshape(-1)}
    if kind == "hmc":
        s = _stout(u, dims, case["n_stout"], 0.1)
        _antiperiodic(s, dims)
        return [s, _solve(_Wilson(dims, s, _mass(case), case["csw"]), "mdagm", src)]
    W = _Wilson(dims, u, _mass(case), case["csw"])
    if kind == "operator":
        return W.back(W.odds(W.meo(W.odds(W.to(src)))))[0]
    if kind == "rhmc":
        return torch.cat([_solve(W, "mdagm", src, s) for s in _shifts(case["shifts"])])
    if kind == "propagator":
        f = W.to(src)
        chi = W.odds(f) + 0.5 * W.odds(W.D(W.block(W.Ainv, W.even(f))))
        odd_x = _cg(W.meo, W.odds(W.meo(chi, True)))
        return W.back(odd_x + W.block(W.Ainv, W.even(f + 0.5 * W.D(odd_x))))
    return _solve(W, "sym" if kind == "symmetric" else "linop", src)


def _solve(W, system, src, shift=0.0):
    b = W.to(src)
    op = W.sym if system == "sym" else W.meo
    return W.back(_cg(op, b if system == "mdagm" else op(b, True), shift))
