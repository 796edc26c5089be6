"""The calls that a user of this framework makes, as cases that can be timed.

Every case is one of six kinds of call through the package's public entry
points:

  event         maps in, initial conditions, evolution, observables out
                (the loop body of the reference's executable)
  restart       the same from Wilson lines that another program made
                (readInitialWilsonLines): tau = 0 links, evolution, observables
  batch         events of different sizes advanced together, maps in and
                observables out for each
  adjoint       one gradient step: initial conditions, forward, backward to the
                tau = 0 fields, the g2mu maps and the colour charges
  multiplicity  an event with gauge fixing and the gluon spectrum after the
                first step and after the last (computeGluonMultiplicity)
  ipsat         the g2mu maps from nucleon positions and the Q_s^2 table

Lattice sizes, sheet counts, boxes, nuclei, time grids and Newton modes are
those of the benchmark, the tests and the reference's input files: 64^2 to
1024^2, the benchmark's spacing a = 0.078125 fm where the box follows from the
size. The plain FP64 form solves its tau = 0 links by the reference's
iteration, the FP32 form by Newton on the group, as the benchmark does.

exact() evaluates the same event with plain torch and numpy in 64 bits: exp of
the sheets, Newton on the group, the leapfrog on full 3x3 matrices, T^{mu nu}
and the eigenvectors; gradients come from torch's autograd.
"""
import math

import numpy as np
import torch

import ipglasma_b200 as ipg

HBARC = 0.1973269718
A_FM = 0.078125  # the benchmark's lattice spacing
NUCLEI = {"O": (16, 2.61, 0.513), "Au": (197, 6.38, 0.535), "Pb": (208, 6.62, 0.546)}


# ---- cases --------------------------------------------------------------------

def listed():
    return [
        # a small system on a small lattice: every stage is a few launches that
        # do not fill the GPU
        event("event64", 64, "O", prec="fp64", Ny=50, b=1.5, maxtime=0.4),
        # the plain form at the benchmark's O+O size
        event("event256", 256, "O", prec="fp64", Ny=50, b=2.0, maxtime=0.4),
        # the benchmark's single event, in both forms
        event("event512", 512, "Pb", prec="fp64", Ny=50, b=6.0, maxtime=0.6),
        event("event512_fp32", 512, "Pb", prec="fp32", Ny=50, b=6.0, maxtime=0.6),
        # the production lattice: 1024^2, 100 sheets, dtau = 0.05 a
        event("event1024_fp32", 1024, "Pb", prec="fp32", Ny=100, b=7.0, maxtime=0.4, L=40.0,
              dtau=0.05),
        # Wilson lines read from files
        {"name": "restart256", "kind": "restart", "prec": "fp64", "N": 256, "L": 30.0,
         "nucleus": "Au", "b": 4.0, "Ny": 50, "maxtime": 0.4, "dtau": 0.0},
        # the benchmark's batch in its proportions (4 O+O 256^2 to 1 Pb+Pb 512^2)
        batch("batch_fp32", "fp32", 50, 0.4, (256, "O", 16), (512, "Pb", 4)),
        # a min-bias run of small events in the plain form; sheets not a
        # multiple of anything
        batch("batch_fp64_small", "fp64", 37, 0.33, (64, "O", 8), (128, "O", 5)),
        # gradients, every state kept, through to the colour charges
        {"name": "adjoint128", "kind": "adjoint", "prec": "fp64", "N": 128, "L": 10.0,
         "nucleus": "O", "b": 2.0, "Ny": 25, "maxtime": 0.6, "dtau": 0.0, "keep": 1,
         "rho": True},
        # gradients of the FP32 form, checkpointed
        {"name": "adjoint256_fp32", "kind": "adjoint", "prec": "fp32", "N": 256, "L": 30.0,
         "nucleus": "Au", "b": 5.0, "Ny": 50, "maxtime": 1.0, "dtau": 0.0, "keep": 11,
         "rho": False},
        # gluon spectra of a plain event
        {"name": "multiplicity256", "kind": "multiplicity", "prec": "fp64", "N": 256, "L": 20.0,
         "nucleus": "O", "b": 2.0, "Ny": 50, "maxtime": 0.4, "dtau": 0.0, "rapidity": 0.3,
         "pseudo": True},
        # the maps of a Pb+Pb event from its nucleons
        {"name": "ipsat256", "kind": "ipsat", "prec": "fp64", "N": 256, "L": 30.0,
         "nucleus": "Pb", "b": 4.0, "roots": 5020.0, "fluctuating": True},
    ]


def event(name, N, nucleus, prec, Ny, b, maxtime, L=None, dtau=0.0):
    return {"name": name, "kind": "event", "prec": prec, "N": N,
            "L": N * A_FM if L is None else L, "nucleus": nucleus, "b": b, "Ny": Ny,
            "maxtime": maxtime, "dtau": dtau}


def batch(name, prec, Ny, maxtime, small, large):
    return {"name": name, "kind": "batch", "prec": prec, "Ny": Ny, "maxtime": maxtime,
            "N1": small[0], "nucleus1": small[1], "count1": small[2],
            "N2": large[0], "nucleus2": large[1], "count2": large[2]}


def draw(rng):
    kind = rng.choice(["event", "event", "event", "event", "restart", "batch", "adjoint",
                       "multiplicity", "ipsat"])
    prec = rng.choice(["fp64", "fp32"])
    Ny = round(8 * 10 ** rng.uniform(0.0, 1.0))
    maxtime = round(rng.uniform(0.15, 0.6), 3)
    if kind == "batch":
        logn = rng.choice([5, 6, 7])
        c = {"kind": kind, "prec": prec, "Ny": Ny, "maxtime": maxtime,
             "N1": 2 ** logn, "nucleus1": "O", "count1": rng.randint(2, 12),
             "N2": 2 ** (logn + rng.randint(1, 2)), "nucleus2": rng.choice(["O", "Au", "Pb"]),
             "count2": rng.randint(1, 4)}
        return c
    N = 2 ** rng.choice({"adjoint": [6, 6, 7], "multiplicity": [6, 7, 8], "ipsat": [6, 7, 8, 9],
                         "restart": [6, 7, 8]}.get(kind, [6, 6, 7, 7, 8, 8, 9]))
    a = rng.uniform(0.06, 0.12)
    nucleus = rng.choice(["O", "Au", "Pb"]) if N * a > 14 else "O"
    c = {"kind": kind, "prec": prec, "N": N, "L": round(N * a, 3), "nucleus": nucleus,
         "b": round(rng.uniform(0.0, 0.9) * NUCLEI[nucleus][1], 3)}
    if kind == "ipsat":
        # a table for protons at the energies of RHIC and of the LHC
        c.update(prec="fp64", L=round(max(N * a, 12.0), 3),
                 roots=float(rng.choice([200, 2760, 5020])), fluctuating=rng.random() < 0.75)
        return c
    c.update(Ny=Ny, maxtime=maxtime, dtau=0.0)
    if kind == "adjoint":
        c.update(Ny=min(Ny, 40), keep=rng.choice([1, 1, 5, 9]), rho=rng.random() < 0.3)
    if kind == "multiplicity":
        c.update(rapidity=round(rng.uniform(0.0, 1.0), 2), pseudo=rng.random() < 0.5)
    return c


# ---- inputs -------------------------------------------------------------------

def nucleus(rng, name, shift):
    """Nucleon positions (A, 3) of a Woods-Saxon nucleus, moved along x."""
    A, R, d = NUCLEI[name]
    r = np.empty(0)
    while r.size < A:
        s = (R + 10 * d) * rng.random(8 * A) ** (1 / 3)
        r = np.concatenate([r, s[rng.random(s.size) <= 1 / (1 + np.exp((s - R) / d))]])
    z = rng.standard_normal((A, 3))
    z *= (r[:A] / np.linalg.norm(z, axis=1))[:, None]
    z -= z.mean(axis=0)
    z[:, 0] += shift
    return z


def thickness_map(xyz, N, L):
    """g^2 mu^2 a^2 of one nucleus with Q_s^2 = (1.5 GeV)^2 T / max T."""
    a = L / N
    x = -L / 2 + a * np.arange(N)
    B = 4.0 * HBARC ** 2
    T = (np.exp(-(x[None] - xyz[:, :1]) ** 2 / (2 * B)).T
         @ np.exp(-(x[None] - xyz[:, 1:2]) ** 2 / (2 * B)))
    return (1.5 ** 2 * T / T.max() / 0.8 ** 2 * a * a / HBARC ** 2 / 4.0).ravel()


def maps(seed, k, name, N, L, b):
    rng = np.random.default_rng([seed, k])
    return np.stack([thickness_map(nucleus(rng, name, s * b / 2), N, L) for s in (-1, 1)])


def pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def config(c, seed, N=None, L=None, **more):
    p = c["prec"] == "fp32"
    return ipg.Config(size=N or c["N"], L=L or c["L"], Ny=c.get("Ny", 2),
                      maxtime=c.get("maxtime", 0.1), dtau=c.get("dtau", 0.0),
                      precision=ipg.FP32 if p else ipg.FP64, seed=int(seed) * 1000 + 1,
                      newton_mode=more.pop("newton_mode", int(p)), **more)


class Outputs:
    """Page-locked arrays that one event's observables are copied into: the
    rows of `all` are e, u (4), pi (10) and T (10)."""

    def __init__(self, n):
        self.all = pinned(25, n)
        self.eps, self.u4, self.pi10, self.T10 = np.split(self.all, [1, 5, 15])

    def start(self, ev):
        ev.observables_async(self.eps, self.u4, self.pi10, self.T10)

    def dict(self, res):
        return {"eps": self.eps[0], "u4": self.u4, "pi10": self.pi10, "T10": self.T10,
                "scalars": scalars(res)}


def scalars(r):
    return np.array([r.E_T, r.sum_Ttautau, r.sum_eps, *r.eccentricity, *r.psi])


def qs_table():
    T = 1e-4 * (9.44 / 1e-4) ** (np.arange(200) / 199)
    y = 0.25 * np.arange(44)
    return T, (2.2 * T[:, None] ** 0.92 * np.exp(0.28 * y) * (1 + 0.05 * np.sin(3 * y)))


def wilson_lines(c, seed, k):
    """V of one nucleus as (n, 3, 3): the ordered product over the sheets."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(device=dev).manual_seed(int(seed) * 2 + k)
    N, n = c["N"], c["N"] ** 2
    g2 = torch.from_numpy(maps(seed, 0, c["nucleus"], N, c["L"], c["b"])[k]).to(dev)

    def noise(s):
        return torch.randn(n, 8, dtype=torch.float64, device=dev, generator=gen)

    return sheets(c, g2, noise)


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"kind": kind, "case": c}
    if kind == "batch":
        s["events"], s["maps"], s["out"] = [], [], []
        for k in range(c["count1"] + c["count2"]):
            one = "1" if k < c["count1"] else "2"
            N, name = c["N" + one], c["nucleus" + one]
            rng = np.random.default_rng([seed, k, 1])
            m = pinned(2, N * N)
            m[:] = maps(seed, k, name, N, N * A_FM,
                        min(2 * NUCLEI[name][1], 0.5 * N * A_FM) * rng.random())
            ev = ipg.Event(config(c, seed * 100 + k, N=N, L=N * A_FM))
            ev.use_device_noise()
            s["events"].append(ev)
            s["maps"].append(m)
            s["out"].append(Outputs(N * N))
        s["batch"] = ipg.Batch(s["events"])
        return s
    if kind == "ipsat":
        rng = np.random.default_rng([seed, 7])
        s["nuclei"] = [nucleus(rng, c["nucleus"], 0.0) for _ in range(2)]
        s["table"] = qs_table()
        s["ev"] = ipg.Event(config(c, seed))
        return s
    if kind == "restart":
        s["ev"] = ipg.Event(config(c, seed))
        for k, f in enumerate((ipg.VA, ipg.VB)):
            s["ev"].set_field(f, wilson_lines(c, seed, k).cpu().numpy())
    else:
        s["maps"] = pinned(2, c["N"] ** 2)
        s["maps"][:] = maps(seed, 0, c["nucleus"], c["N"], c["L"], c["b"])
        more = {"newton_mode": 0, "newton_tolerance": 1e-12} if kind == "adjoint" else {}
        s["ev"] = ipg.Event(config(c, seed, **more))
        s["ev"].use_device_noise()
    if kind == "adjoint":
        n = c["N"] ** 2
        s["out"] = {"state": pinned(108 * n), "g2mu": pinned(2 * n)}
        if c["rho"]:
            s["out"]["rho"] = pinned(16 * c["Ny"] * n)
    else:
        s["out"] = Outputs(c["N"] ** 2)
    return s


def run(state):
    c, kind = state["case"], state["kind"]
    if kind == "batch":
        for ev, m in zip(state["events"], state["maps"]):
            ev.set_g2mu(m[0], m[1])
        state["batch"].init_fields(allow_nonconverged=True)
        res = state["batch"].run()
        for ev, o in zip(state["events"], state["out"]):
            o.start(ev)
        for ev in state["events"]:
            ev.wait_observables()
        # one array of each event and the scalars of all
        return {"observables": [o.all for o in state["out"]],
                "scalars": np.stack([scalars(r) for r in res])}
    ev = state["ev"]
    if kind == "ipsat":
        rep = ev.set_nuclei_ipsat(*state["nuclei"], c["b"], state["table"], roots=c["roots"],
                                  use_fluctuating_x=c["fluctuating"])
        return {"g2mu": ev.g2mu(), "thickness": ev.thickness(),
                "counts": np.array([rep["Npart"], rep["Ncoll"], rep["overlap_cells"]]),
                "averages": np.array([rep["Tpp"], rep["average_Qs"], rep["average_Qs_avg"],
                                      rep["average_Qs_min"]])}
    if kind == "restart":
        ev.init_from_wilson_lines(allow_nonconverged=True)
    else:
        ev.set_g2mu(state["maps"][0], state["maps"][1])
        ev.init_fields(allow_nonconverged=True)
    if kind == "adjoint":
        et, e2 = ev.forward(c["keep"])
        g = ev.backward(1.0, 1.0, inputs=True, rho=c["rho"], out=state["out"])
        return {"E_T": et, "eps2": e2, **{"grad_" + str(k): v for k, v in g.items()}}
    if kind == "multiplicity":
        res, first, last = ev.run_multiplicity(use_pseudorapidity=c["pseudo"],
                                               rapidity=c["rapidity"])
        state["out"].start(ev)
        ev.wait_observables()
        spec = {k: [np.concatenate([m["n_kt"], m["E_kt"]]), m["count_kt"],
                    np.array([m["dNdy"], m["dEdy"], m["dNdy_binned"], m["dEdy_binned"],
                              m["mean_pt"]])]
                for k, m in (("first", first), ("last", last))}
        return {**state["out"].dict(res), **spec}
    res = ev.run()
    state["out"].start(ev)
    ev.wait_observables()
    return state["out"].dict(res)


# ---- what a pass cannot do without --------------------------------------------

MUL = 198.0  # real operations of a 3x3 complex product


def steps_of(c, L, N):
    a = L / N
    dtau = c.get("dtau", 0.0)
    if not dtau > 0:
        dtau = c["maxtime"] / ((int(10 * c["maxtime"] / a) + 1) * a)
    return int(c["maxtime"] / (a * dtau) + 0.1), dtau


def event_flops(c, N, L, init=True):
    n, lg = float(N * N), math.log2(N)
    steps, _ = steps_of(c, L, N)
    f = n * steps * 15 * MUL             # staples, transports, commutators, link update
    f += n * 110 * MUL                   # T^{mu nu}, Landau matching
    f += 2 * n * 4 * 8 * MUL             # tau = 0 links: a few Newton steps of two links
    if init:
        # per sheet and nucleus: 4 complex transforms there and back, exp, product
        f += 2 * n * c["Ny"] * (4 * 2 * 10 * lg + 250 + MUL)
    return f


def work(case):
    c, kind = case, case["kind"]
    if kind == "ipsat":
        n, A = float(c["N"] ** 2), NUCLEI[c["nucleus"]][0]
        return {"bytes": 8 * 4 * n + 48 * A, "flops": 2 * n * A * 12}
    if kind == "batch":
        w = {"bytes": 0.0, "flops": 0.0}
        for k in "12":
            N, m = c["N" + k], c["count" + k]
            w["bytes"] += m * 27 * 8.0 * N * N
            w["flops"] += m * event_flops(c, N, N * A_FM)
        return w
    n = float(c["N"] ** 2)
    flops = event_flops(c, c["N"], c["L"], kind != "restart")
    if kind == "adjoint":
        out = 108 + 2 + (16 * c["Ny"] if c["rho"] else 0)
        return {"bytes": 8 * n * (2 + out), "flops": 3 * flops}
    if kind == "multiplicity":  # two gauge fixings of some tens of iterations
        flops += 2 * 40 * n * (8 * 10 * math.log2(c["N"]) + 20 * MUL)
    return {"bytes": 8 * n * ((36 if kind == "restart" else 2) + 25), "flops": flops}


# ---- the same in 64 bits with plain torch -------------------------------------

def generators(like):
    t = torch.zeros(8, 3, 3, dtype=torch.complex128, device=like.device)
    for a, (i, j, v) in {0: (0, 1, 1), 1: (0, 1, -1j), 3: (0, 2, 1), 4: (0, 2, -1j),
                         5: (1, 2, 1), 6: (1, 2, -1j)}.items():
        t[a, i, j], t[a, j, i] = 0.5 * v, 0.5 * complex(v).conjugate()
    t[2] = torch.diag(torch.tensor([0.5, -0.5, 0.0], dtype=t.dtype))
    t[7] = torch.diag(torch.tensor([1.0, 1.0, -2.0], dtype=t.dtype)) / (2 * math.sqrt(3))
    return t


def sheets(c, g2, noise):
    """prod_k exp(-i A_k.t), A_k = (k~^2 + m^2)^-1 rho_k, newest sheet leftmost."""
    N, Ny = c["N"], c["Ny"]
    dev = g2.device
    m = 0.2 * c["L"] / N / HBARC
    s = torch.sin(math.pi * torch.arange(N, dtype=torch.float64, device=dev) / N) ** 2
    green = 1 / (4 * (s[:, None] + s[None]) + m * m)
    t = generators(g2)
    amp = 2.0 * torch.sqrt(g2 / Ny)
    V = torch.eye(3, dtype=torch.complex128, device=dev).repeat(N * N, 1, 1)
    for k in range(Ny):
        rho = (amp[:, None] * noise(k)).reshape(N, N, 8)
        A = torch.fft.ifft2(torch.fft.fft2(rho, dim=(0, 1)) * green[:, :, None], dim=(0, 1)).real
        V = torch.linalg.matrix_exp(torch.einsum("pa,aij->pij", -1j * A.reshape(-1, 8), t)) @ V
    return V


def device_noise(seed, nuc, n, dev):
    """The documented draw: Philox4x32-10 with key `seed` and counter (site,
    sheet, 2 nucleus + half, 0), Box-Muller of 24-bit uniforms."""
    mask = 0xFFFFFFFF

    def mulhilo(a, x):  # 32 x 32 -> 64 bits without overflowing int64
        lo, hi = x * (a & 0xFFFF), x * (a >> 16)
        mid = (lo >> 16) + hi
        return ((mid & 0xFFFF) << 16) | (lo & 0xFFFF), mid >> 16

    def uni(x):
        return ((x >> 8).double() + 1) / 16777216.0

    def noise(k):
        pos = torch.arange(n, device=dev)
        out = []
        for half in range(2):
            x, y = pos, torch.full_like(pos, k)
            z, w = torch.full_like(pos, 2 * nuc + half), torch.zeros_like(pos)
            k0, k1 = seed & mask, seed >> 32
            for _ in range(10):
                lo0, hi0 = mulhilo(0xD2511F53, x)
                lo1, hi1 = mulhilo(0xCD9E8D57, z)
                x, y, z, w = hi1 ^ y ^ k0, lo1, hi0 ^ w ^ k1, lo0
                k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
            for u, v in ((x, y), (z, w)):
                r, ph = torch.sqrt(-2 * torch.log(uni(u))), 2 * math.pi * uni(v)
                out += [r * torch.cos(ph), r * torch.sin(ph)]
        return torch.stack(out, dim=-1)

    return noise


def xp(f, k=1):  # neighbours, clamped at the edges
    return xp(torch.cat([f[1:], f[-1:]]), k - 1) if k else f


def xm(f):
    return torch.cat([f[:1], f[:-1]])


def yp(f, k=1):
    return yp(torch.cat([f[:, 1:], f[:, -1:]], dim=1), k - 1) if k else f


def ym(f):
    return torch.cat([f[:, :1], f[:, :-1]], dim=1)


def tr(a):
    return torch.einsum("...ii->...", a)


def tl(a):
    return a - tr(a)[..., None, None] / 3 * torch.eye(3, dtype=a.dtype, device=a.device)


def tau0(V, N):
    """Links and pi at tau = 0 from the Wilson lines of both nuclei."""
    VA, VB = (v.reshape(N, N, 3, 3) for v in V)
    t = generators(VA)
    tab = torch.einsum("bij,ajk->abik", t, t)
    links, diffs = [], []
    for sh in (xp, yp):
        U1, U2 = VA @ sh(VA).mH, VB @ sh(VB).mH
        S, U = U1 + U2, U1 @ U2

        def miss(U):
            W = S @ U.mH
            F = -torch.einsum("aij,...ji->...a", t, S - S.mH + W - W.mH).imag
            return W, F, F.abs().sum(-1)

        W, F, best = miss(U)
        for _ in range(12):
            J = 2 * torch.einsum("abij,...ji->...ab", tab, W).real
            d = torch.linalg.solve(J, -F)
            new = torch.linalg.matrix_exp(torch.einsum("...a,aij->...ij", 1j * d, t)) @ U
            W1, F1, e1 = miss(new)
            ok = (e1 < best)[..., None, None]
            U = torch.where(ok, new, U)
            W, F = torch.where(ok, W1, W), torch.where(ok[..., 0], F1, F)
            best = torch.minimum(best, e1)
        links.append(U)
        diffs.append(U1 - U2)
    (ux, uy), (dx, dy) = links, diffs

    def fwd(D, U):
        return D @ U.mH - D - U @ D.mH + D.mH

    def bwd(D, U):
        return -U.mH @ D + D + D.mH @ U - D.mH

    e = (fwd(dx, ux) + bwd(xm(dx), xm(ux)) + fwd(dy, uy) + bwd(ym(dy), ym(uy))) / 8
    zero = torch.zeros_like(ux)
    return [ux, uy, zero, zero, zero, -1j * e]  # g = 2


def kick(f, tau, dtau):
    """pi and E (g = 2)."""
    ux, uy, e1, e2, phi, pi = f
    px, py = ux @ xp(phi) @ ux.mH, uy @ yp(phi) @ uy.mH
    mx, my = xm(ux.mH @ phi @ ux), ym(uy.mH @ phi @ uy)
    pi = pi + dtau / tau * (px + py + mx + my - 4 * phi)
    U12 = ux @ xp(uy) @ yp(ux).mH @ uy.mH
    U1m2 = (ux @ ym(xp(uy)).mH) @ ym(ux.mH @ uy)
    U2m1 = (uy @ xm(yp(ux)).mH) @ xm(uy.mH @ ux)
    ca, cb = 1j * tau * dtau / 8, 1j * dtau / tau
    s1, s2 = U12 + U1m2, U12.mH + U2m1
    e1 = tl(e1 + ca * tl(s1 - s1.mH) + cb * (px @ phi - phi @ px))
    e2 = tl(e2 + ca * tl(s2 - s2.mH) + cb * (py @ phi - phi @ py))
    return [ux, uy, e1, e2, phi, pi]


def drift(f, tau, dtau):
    ux, uy, e1, e2, phi, pi = f
    one = torch.eye(3, dtype=ux.dtype, device=ux.device)
    c = 4j * dtau / (tau + dtau / 2)

    def turn(e, u):
        X = c * e
        return (one + X + X @ X / 2) @ u

    return [turn(e1, ux), turn(e2, uy), e1, e2, phi + (tau + dtau / 2) * dtau * pi, pi]


def evolved(f, steps, dtau):
    f = drift(f, 0.0, dtau)
    for it in range(1, steps):
        f = drift(kick(f, it * dtau, dtau), it * dtau, dtau)
    return f


def fwd(u, a):
    return u @ a @ u.mH


def re2(a, b=None):
    return tr(a @ (a if b is None else b)).real


def diagonal(f, tau, a):
    """T^{tau tau}, T^{xx}, T^{yy}, T^{eta eta} in fm^-4 (fm^-6), g = 2."""
    ux, uy, e1, e2, phi, pi = f
    ge = 4 / tau ** 2
    E1, E2, P = re2(e1), re2(e2), re2(pi)
    E1, E2 = E1 + yp(E1), E2 + xp(E2)
    P = P + xp(P) + yp(P) + xp(yp(P))
    pl = ux @ xp(uy) @ yp(ux).mH @ uy.mH
    B = 0.5 * (3 - tr(pl).real)
    B = torch.cat([B[:-1], torch.zeros_like(B[-1:])])
    d1, d3 = phi - fwd(ux, xp(phi)), phi - fwd(uy, yp(phi))
    d2, d4 = yp(phi) - fwd(yp(ux), xp(yp(phi))), xp(phi) - fwd(xp(uy), xp(yp(phi)))
    P12, P34 = re2(d1) + re2(d2), re2(d3) + re2(d4)
    h = 0.5 / tau ** 2
    return [(ge * (E1 + E2) / 2 + P / 4 + B + h * (P12 + P34)) / a ** 4,
            (ge * (E2 - E1) / 2 + P / 4 + B + h * (P12 - P34)) / a ** 4,
            (ge * (E1 - E2) / 2 + P / 4 + B + h * (P34 - P12)) / a ** 4,
            (ge * (E1 + E2) / 2 - P / 4 - B + h * (P12 + P34)) / tau ** 2 / a ** 6]


def off_diagonal(f, tau, a):
    """T^{tau x}, tau y, tau eta, xy, x eta, y eta."""
    ux, uy, e1, e2, phi, pi = f
    g = 2.0

    def ah(p):
        return tl(p - p.mH)

    def back(u, q):
        return u.mH @ q @ u

    P = ux @ xp(uy) @ yp(ux).mH @ uy.mH
    Q1 = xm(ux).mH @ xm(uy) @ yp(xm(ux)) @ uy.mH
    R1 = xp(uy) @ xp(yp(ux)) @ xp(uy, 2).mH @ xp(ux).mH
    S1 = ux.mH @ uy @ yp(ux) @ xp(uy).mH
    Q3 = ym(uy).mH @ ym(ux) @ xp(ym(uy)) @ ux.mH
    R3 = yp(ux) @ xp(yp(uy)) @ yp(ux, 2).mH @ yp(uy).mH
    S3 = uy.mH @ ux @ xp(uy) @ yp(ux).mH
    e1p, e2p = yp(e1), xp(e2)
    pX, pY, pXY = xp(pi), yp(pi), xp(yp(pi))
    fX, fY, fXY = xp(phi), yp(phi), xp(yp(phi))
    K, Kp = -ah(P) + ah(Q1), ah(R1) + ah(S1)
    mag = (tr(e2 @ K) + tr(e2p @ Kp)).imag
    el = re2(pi, fwd(ux, fX) - back(xm(ux), xm(phi)))
    el = el + re2(pY, fwd(yp(ux), fXY) - back(yp(xm(ux)), yp(xm(phi))))
    el = el + re2(pX, fwd(xp(ux), xp(phi, 2)) - back(ux, phi))
    el = el + re2(pXY, fwd(xp(yp(ux)), xp(yp(phi), 2)) - back(yp(ux), fY))
    out = [(mag - el) / (4 * tau) / a ** 4]
    K, Kp = ah(P) + ah(Q3), ah(R3) + ah(S3)
    mag = (tr(e1 @ K) + tr(e1p @ Kp)).imag
    el = re2(pi, fwd(uy, fY) - back(ym(uy), ym(phi)))
    el = el + re2(pX, fwd(xp(uy), fXY) - back(xp(ym(uy)), xp(ym(phi))))
    el = el + re2(pY, fwd(yp(uy), yp(phi, 2)) - back(uy, phi))
    el = el + re2(pXY, fwd(xp(yp(uy)), yp(xp(phi), 2)) - back(xp(uy), fX))
    out += [(mag - el) / (4 * tau) / a ** 4]
    dX, dY = fwd(ux, fX) - phi, fwd(uy, fY) - phi
    dXY1, dXY2 = fwd(yp(ux), fXY) - fY, fwd(xp(uy), fXY) - fX
    out += [g / tau ** 3 * (re2(e1, dX) + re2(e1p, dXY1) + re2(e2, dY) + re2(e2p, dXY2)) / a ** 5]
    wy, wx = fwd(uy, dXY1), fwd(ux, dXY2)
    t = -0.25 * g * g * re2(e1 + fwd(uy, e1p), e2 + fwd(ux, e2p)) + 0.25 * re2(dX + wy, dY + wx)
    out += [2 / tau ** 2 * t / a ** 4]
    e = re2(e1, pi + fwd(ux, pX)) + re2(e1p, pY + fwd(yp(ux), pXY))
    m = tr((ah(P) - ah(Q1)) @ dY + (-ah(S1) - ah(R1)) @ dXY2).imag
    out += [-2 / tau ** 2 * (0.25 * g * e + m / (8 * g)) / a ** 5]
    e = re2(e2, pi + fwd(uy, pY)) + re2(e2p, pX + fwd(xp(uy), pXY))
    m = tr((-ah(P) - ah(Q3)) @ dX + (-ah(S3) - ah(R3)) @ dXY1).imag
    out += [-2 / tau ** 2 * (0.25 * g * e + m / (8 * g)) / a ** 5]
    return out


def landau(T, tau_fm, N):
    """e, u^mu, pi^{mu nu} from T (10, n)."""
    tt, xx, yy, ee, tx, ty, te, xy, xe, ye = T
    t2 = tau_fm ** 2
    M = np.stack([tt, -tx, -ty, -t2 * te, tx, -xx, -xy, -t2 * xe, ty, -xy, -yy, -t2 * ye,
                  te, -xe, -ye, -t2 * ee], axis=-1).reshape(-1, 4, 4)
    w, v = np.linalg.eig(M)
    v = v.transpose(0, 2, 1)  # [cell][vector][component]
    met = np.array([1, -1, -1, -t2])
    size = (v ** 2 * met).sum(-1).real
    k, n = size.argmax(1), np.arange(len(size))
    found = size[n, k] > 0
    v = v[n, k].real / np.sqrt(np.where(found, np.abs(size[n, k]), 1))[:, None]
    v *= np.sign(v[:, :1])
    # without a real timelike vector: T^{tau tau} at rest, but at the border
    e = np.where(found & ((np.abs(w[n, k].imag) <= 0.001) | border(N, 1, 5)), w[n, k].real, tt)
    real = (np.abs(w[n, k].imag) <= 0.001) | border(N, 11, 10)
    u = np.where((found & (e > 0.1) & real)[:, None], v, [1.0, 0, 0, 0])
    c, (a, b, d, h) = e, u.T
    P = np.stack([tt - 4 / 3 * c * a * a + c / 3, xx - 4 / 3 * c * b * b - c / 3,
                  yy - 4 / 3 * c * d * d - c / 3, ee - 4 / 3 * c * h * h - c / 3 / t2,
                  tx - 4 / 3 * c * a * b, ty - 4 / 3 * c * a * d, te - 4 / 3 * c * a * h,
                  xy - 4 / 3 * c * b * d, xe - 4 / 3 * c * b * h, ye - 4 / 3 * c * d * h])
    P[:, a == 1] = 0
    return e, np.ascontiguousarray(u.T), P


def border(N, low, high):
    i = np.arange(N)
    i = (i < low) | (i >= N - high)
    return (i[:, None] | i[None]).ravel()


def eccentricities(e, ut, N, L):
    a = L / N
    x = -L / 2 + a * np.arange(N)
    w = (np.maximum(e, 0) * ut).reshape(N, N)
    X = x[:, None] - (w.sum(1) @ x) / w.sum()
    Y = x[None, :] - (w.sum(0) @ x) / w.sum()
    r, ph, w = np.hypot(X, Y)[2:-2, 2:-2], np.arctan2(Y, X + 0 * Y)[2:-2, 2:-2], w[2:-2, 2:-2]
    ecc, psi = [], []
    for k in range(1, 7):
        rp = r ** (3 if k == 1 else k)
        cs, sn = (w * rp * np.cos(k * ph)).sum(), (w * rp * np.sin(k * ph)).sum()
        ecc.append(math.hypot(cs, sn) / (w * rp).sum())
        psi.append((math.atan(sn / cs) + math.pi) / k)
    return ecc + psi


def exact(case, seed):
    c = case
    if c["kind"] not in ("event", "restart", "adjoint") or c["N"] > 256 or \
            (c["kind"] == "adjoint" and c["N"] > 128):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    N, L = c["N"], c["L"]
    a = L / N
    steps, dtau = steps_of(c, L, N)
    if c["kind"] == "restart":
        V = [wilson_lines(c, seed, k) for k in range(2)]
    else:
        g2 = torch.from_numpy(maps(seed, 0, c["nucleus"], N, L, c["b"])).to(dev)
        V = [sheets(c, g2[k], device_noise(int(seed) * 1000 + 1, k, N * N, dev))
             for k in range(2)]
    f = tau0(V, N)
    tau = steps * dtau
    unit = tau * a ** 3 * HBARC  # E_T of the sum of T^{tau tau}
    if c["kind"] == "adjoint":
        start = [x.clone().requires_grad_() for x in f]
        T = diagonal(evolved(start, steps, dtau), tau, a)[0]
        et, w = unit * T.sum(), T[2:-2, 2:-2]
        x = -L / 2 + a * torch.arange(N, dtype=torch.float64, device=dev)[2:-2]
        W = w.sum()
        X, Y = (w.sum(1) * x).sum() / W, (w.sum(0) * x).sum() / W
        cxx = (w.sum(1) * (x - X) ** 2).sum()
        cyy = (w.sum(0) * (x - Y) ** 2).sum()
        cxy = (w * (x - X)[:, None] * (x - Y)[None]).sum()
        e2 = torch.sqrt((cxx - cyy) ** 2 + 4 * cxy ** 2) / (cxx + cyy)
        (et + e2).backward()
        out = {"E_T": et.item(), "eps2": e2.item(), "grad_g2mu": None}
        for k, s in enumerate(start):
            g = s.grad if k < 2 else 0.5 * (s.grad + s.grad.mH)
            g = tl(g) if k in (2, 3) else g
            out["grad_%d" % k] = g.reshape(N * N, 3, 3).cpu().numpy()
        if c["rho"]:
            out["grad_rho"] = None
        return out
    f = evolved(f, steps, dtau)
    T = torch.stack(diagonal(f, tau, a) + off_diagonal(f, tau, a)).reshape(10, -1).cpu().numpy()
    e, u, P = landau(T, tau * a, N)
    return {"eps": e, "u4": u, "pi10": P, "T10": T,
            "scalars": np.array([unit * T[0].sum(), T[0].sum(), e.sum(),
                                 *eccentricities(e, u[0], N, L)])}
