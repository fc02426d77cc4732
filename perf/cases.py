"""Workloads of the CCD + (T) engine, through its public entry points.

Each case is one call, or one short run of calls, that a program driving the engine makes:
amplitude solves in both precisions, the call-by-call loop of a Fortran host, a batch of
twists, the generation and the hand-over of an interaction, the triples sum, the energy on
caller-owned buffers and the training pass of the learned start.  Lattices are the closed
shells of pure neutron matter (pnm, Minnesota, real) and symmetric matter (snm,
chiral-like, complex) that the tests and the benchmark use.  A seed moves the density by a
few per cent, as a scan of the equation of state does, or draws the inputs that are arrays,
so that sizes stay and values change.
"""
import ctypes
import importlib.util
import itertools
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "coupled-cluster-nuclearmatter_gb300")


def engine_package():
    """The engine package (its directory name is not a Python identifier)."""
    if "ccnm_gb300" not in sys.modules:
        spec = importlib.util.spec_from_file_location("ccnm_gb300", os.path.join(PKG, "__init__.py"),
                                                      submodule_search_locations=[PKG])
        sys.modules["ccnm_gb300"] = m = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(m)
    return sys.modules["ccnm_gb300"]


def listed():
    return [
        # a host that owns its device buffers asks for the energy of a small lattice: launches only
        dict(name="energy-pnm14", kind="energy", nmax=2, A=14, snm=False),
        # one point of an equation of state on the smallest lattice that is used, plain FP64
        dict(name="solve64-pnm14", kind="solve", nmax=2, A=14, snm=False, mixed=False),
        # the same with a complex interaction
        dict(name="solve64-snm28", kind="solve", nmax=2, A=28, snm=True, mixed=False),
        # the loop of a Fortran host, call by call, in FP64 on the production neutron lattice
        dict(name="steps-pnm66", kind="steps", nmax=4, A=66, snm=False, steps=2),
        # production solve of neutron matter: tensor-core corrections, digit-product re-bases
        dict(name="solve-pnm66", kind="solve", nmax=4, A=66, snm=False, mixed=True),
        # the headline: the largest lattice that one GPU holds
        dict(name="solve-snm132n4", kind="solve", nmax=4, A=132, snm=True, mixed=True),
        # twist averaging: a few random twists of symmetric matter in lockstep
        dict(name="batch-snm76", kind="batch", nmax=2, A=76, snm=True, twists=3),
        # set-up of a production point: every block of the interaction, and the MP2 start
        dict(name="setup-pnm66", kind="setup", nmax=4, A=66, snm=False),
        dict(name="setup-snm132n3", kind="setup", nmax=3, A=132, snm=True),
        # the triples correction in its default arithmetic
        dict(name="triples-snm76", kind="triples", nmax=2, A=76, snm=True, fp32=True),
        # a host hands over every block of its interaction and reads the amplitudes back
        dict(name="handover-pnm38", kind="handover", nmax=3, A=38, snm=False, pinned=True),
        # one training pass of the learned start (loss and gradients of a batch)
        dict(name="learn-8192", kind="learn", batch=8192),
    ]


#: closed shells (particles) that fit the lattices of each nmax with room for particle states
PNM = {1: (2, 14, 38), 2: (14, 38, 54, 66), 3: (14, 38, 54, 66, 114), 4: (14, 38, 54, 66)}
SNM = {1: (4, 28), 2: (4, 28, 76, 108), 3: (28, 76, 108, 132)}


def draw(rng):
    kind = rng.choice(["energy", "solve", "steps", "solve", "batch", "setup", "triples", "handover", "learn"])
    if kind == "learn":
        return dict(kind=kind, batch=int(round(2 ** rng.uniform(5, 16))))
    snm = rng.random() < 0.5
    shells = SNM if snm else PNM
    nmax = rng.choice(sorted(shells))
    if kind == "handover":  # the host blocks grow as the fourth power of the basis
        nmax = min(nmax, 2 if snm else 3)
    if kind == "triples":  # and the triples as its sixth
        nmax = min(nmax, 2)
    if kind == "batch":
        nmax = min(nmax, 3 if not snm else 2)
    A = rng.choice(shells[nmax])
    if kind == "triples":
        A = max(min(A, 76 if snm else 54), 4 if snm else 14)
    case = dict(kind=kind, nmax=nmax, A=A, snm=snm)
    if kind == "solve":
        case["mixed"] = rng.random() < 0.6
    elif kind == "steps":
        case["steps"] = rng.randint(1, 4)
    elif kind == "batch":
        case["A"], case["twists"] = max(A, 14), rng.randint(2, 6)
    elif kind == "triples":
        case["fp32"] = rng.random() < 0.6
    elif kind == "handover":
        case["pinned"] = rng.random() < 0.5
    return case


def density(case, seed):
    return (0.08 if case["A"] == 14 else 0.16) * (1.0 + 0.03 * random.Random(seed).uniform(-1.0, 1.0))


def layout_of(case, seed, theta=(0.0, 0.0, 0.0)):
    ccx = engine_package()
    return ccx.Layout.from_basis(case["nmax"], case["A"], density(case, seed), snm=case["snm"], theta=theta)


def engine_of(case, layout, generate=True):
    ccx = engine_package()
    e = ccx.Engine(layout, real=not case["snm"])
    if generate:
        e.generate(potential_of(case))
    return e


def potential_of(case):
    ccx = engine_package()
    return ccx.POT_CHIRAL_LIKE if case["snm"] else ccx.POT_MINNESOTA


def solve_options(case):
    ccx = engine_package()
    if not case.get("mixed", True):
        return dict(mode=ccx.MODE_STANDARD, precision=ccx.PREC_FP64, max_iter=200, tol=1e-10)
    return dict(mode=ccx.MODE_STANDARD, precision=ccx.PREC_MIXED, max_iter=200, tol=1e-10, rebase=ccx.REBASE_DIGITS)


def prepare_solve(e, opts):
    e.setup_t_amplitudes()
    e.prepare(mode=opts["mode"], precision=opts["precision"], rebase=opts.get("rebase", 0))


def twists(case):
    """Twists of the batch: generic ones, the same for every seed (a twist picks the hole
    states, and with them the sizes)."""
    r = random.Random(1)
    return [tuple(r.uniform(-math.pi, math.pi) for _ in range(3)) for _ in range(case["twists"])]


def pinned(n):
    """Page-locked host memory of n doubles."""
    return torch.empty(max(n, 1), dtype=torch.float64, pin_memory=True)


def read_t2(e, buf):
    """All amplitudes into page-locked host memory, as a host that keeps them does."""
    ccx = engine_package()
    rc = ccx.lib().ccx_get_t2_all(e._h, ctypes.c_void_p(buf.data_ptr()))
    if rc:
        raise RuntimeError("ccx_get_t2_all: %d" % rc)
    return buf


def prepare(case, seed):
    ccx = engine_package()
    kind = case["kind"]
    if kind == "learn":
        X, y, p = learn_data(case, seed)
        m = ccx.Learner()
        m.set_params(p)
        return dict(case=case, learner=m, X=X, y=y)
    if kind == "energy":
        dims, t, v = energy_data(case, seed)
        return dict(case=case, nch=len(dims), dims=torch.tensor(dims, dtype=torch.int32, device="cuda"), t=t, v=v,
                    out=torch.zeros(2, dtype=torch.float64, device="cuda"))
    if kind == "batch":
        es = [engine_of(case, layout_of(case, seed, th)) for th in twists(case)]
        for e in es:
            prepare_solve(e, solve_options(case))
        return dict(case=case, engines=es, t2=[pinned(2 * e.layout.counts()["amps"]) for e in es])
    L = layout_of(case, seed)
    if kind == "handover":
        src = engine_of(case, L)
        c = L.counts()
        fams = {ccx.CH_HHPP: c["hhpp"], ccx.V_PPPP: c["hhpp"], ccx.CH_HHHH: c["hhhh"], ccx.CH_HPHP: c["hphp"]}
        blocks, keep = {}, []
        for k, n in fams.items():
            got = [src.vblock(k, ch) for ch in range(n)]
            if case["pinned"]:
                keep.append(pinned(2 * sum(b.size for b in got)))
                flat, at, views = keep[-1].numpy().view(np.complex128), 0, []
                for b in got:
                    to = flat[at:at + b.size].reshape(b.shape, order="F")
                    to[...] = b
                    views.append(to)
                    at += b.size
                got = views
            blocks[k] = dict(enumerate(got))
        fock, e0 = src.fock(), src.e0()
        src.close()
        return dict(case=case, engine=engine_of(case, L, generate=False), blocks=blocks, keep=keep, fock=fock, e0=e0,
                    t2=pinned(2 * c["amps"]))
    e = engine_of(case, L, generate=kind != "setup")
    state = dict(case=case, engine=e, t2=pinned(2 * L.counts()["amps"]))
    if kind == "solve":
        prepare_solve(e, solve_options(case))
    if kind == "triples":
        e.set_triples_precision(case["fp32"])
        e.setup_t_amplitudes()
    return state


def run(state):
    ccx = engine_package()
    case = state["case"]
    kind = case["kind"]
    if kind == "learn":
        loss, grad = state["learner"].loss_grad(state["X"], state["y"])
        return dict(loss=np.float32(loss), grad=grad)
    if kind == "energy":
        ccx.ccd_energy_noalloc(state["nch"], state["dims"].data_ptr(), state["t"].data_ptr(), state["v"].data_ptr(),
                               state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return dict(e=state["out"])
    if kind == "batch":
        for e in state["engines"]:
            e.setup_t_amplitudes()
        rs, _ = ccx.ccd_iter_batch(state["engines"], **solve_options(case))
        return dict(e_mbpt2=[np.complex128(r["e_mbpt2"]) for r in rs], e_ccd=[np.complex128(r["e_ccd"]) for r in rs],
                    t2=[read_t2(e, b) for e, b in zip(state["engines"], state["t2"])])
    e = state["engine"]
    if kind == "triples":
        return dict(e_t=np.complex128(e.pert_triples()))
    if kind == "setup":
        e.generate(potential_of(case))
    if kind == "handover":
        e.set_fock(state["fock"], state["e0"])
        for k, blocks in state["blocks"].items():
            e.set_vblocks(k, blocks)
    e.setup_t_amplitudes()
    if kind in ("setup", "handover"):
        return dict(e0=np.complex128(e.e0()), e_mbpt2=np.complex128(e.ccd_energy()), t2=read_t2(e, state["t2"]))
    if kind == "steps":
        e.diis_setup(6, 6)
        out, count = [np.complex128(e.ccd_energy())], 0
        for _ in range(case["steps"]):
            e.t2_intermediate()
            count = e.diis_t1t2(count + 1)
            out.append(np.complex128(e.ccd_energy()))
        return dict(energies=out, t2=read_t2(e, state["t2"]))
    r = e.ccd_iter(**solve_options(case))
    return dict(e_mbpt2=np.complex128(r["e_mbpt2"]), e_ccd=np.complex128(r["e_ccd"]), t2=read_t2(e, state["t2"]))


# ---------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "learn":
        n, p = case["batch"], 35585
        return dict(bytes=4 * (19 * n + 2 * p), flops=6 * n * (18 * 128 + 2 * 128 * 128 + 128))
    ccx = engine_package()
    L = layout_of(case, 0, (0.1, 0.2, 0.3) if kind == "batch" else (0.0, 0.0, 0.0))
    c = L.counts()
    es, f = (16, 8) if case["snm"] else (8, 2)  # scalar bytes, flops of a multiply-add
    if kind == "energy":  # the caller's arrays are complex in either case
        return dict(bytes=32 * c["amps"], flops=8 * c["amps"])
    dims = np.array(L.hhpp_dims(), dtype=np.float64)
    H, P = 0.5 * dims[:, 0], 0.5 * dims[:, 1]  # pairs i < j and a < b
    ring = np.array([L.channel(ccx.CH_PH_PHHP, q)[1:] for q in range(c["ph_phhp"])], dtype=np.float64)
    amps, vpp, vhh, w = (P * H).sum(), (P * P).sum(), (H * H).sum(), (ring[:, 1] ** 2).sum()
    t2 = 16 * c["amps"]  # the amplitudes in the host's ordered complex layout
    if kind == "triples":
        n, blocks = triple_sizes(case)
        return dict(bytes=es * (amps + blocks), flops=n * 18 * 2 * f)
    if kind == "setup":
        return dict(bytes=es * (amps + vpp + vhh + w) + t2, flops=60 * (amps + 0.5 * vpp + vhh + w))
    if kind == "handover":
        return dict(bytes=(16 + es) * (amps + vpp + vhh + w) + t2, flops=4 * amps)
    once = f * ((P * P * H).sum() + 2 * (P * H * H).sum() + 2 * (ring[:, 0] * ring[:, 1] ** 2).sum())
    n = {"steps": case.get("steps", 0), "solve": 20 if case["snm"] else 13, "batch": 20}[kind]
    m = case["twists"] if kind == "batch" else 1
    return dict(bytes=m * (es * (2 * amps + vpp + vhh + w) + t2), flops=m * n * once)


def triple_sizes(case):
    """Number of (abc, ijk) pairs of equal momentum and isospin, and of the elements
    <ab|V|id> and <ij|V|ka> with a < b and i < j that they read."""
    n, tz, _, holes = orbitals(case, 0.16, (0.0, 0.0, 0.0))[:4]
    size = [2 * 3 + 3] + [6 * case["nmax"] + 1] * 3

    def powers(sel):
        """Transformed histogram of the totals of m times one state, m = 1, 2, 3."""
        out = []
        for m in (1, 2, 3):
            h = np.zeros(size)
            at = np.concatenate([((tz[sel] + 1) // 2 * m)[:, None], (n[sel] + case["nmax"]) * m], axis=1)
            np.add.at(h, tuple(at.T), 1.0)
            out.append(np.fft.fftn(h))
        return out

    def count(x):
        return np.rint(np.real(np.fft.ifftn(x)))

    (h1, h2, h3), (p1, p2, p3) = powers(holes), powers(~holes)
    pairs = (count((h1 ** 3 - 3 * h1 * h2 + 2 * h3) / 6) * count((p1 ** 3 - 3 * p1 * p2 + 2 * p3) / 6)).sum()
    return float(pairs), float((count(h1 * p1) * (count((p1 * p1 - p2) / 2) + count((h1 * h1 - h2) / 2))).sum())


# ---------------------------------------------------------------- inputs that are arrays
def learn_data(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    X = r.standard_normal((case["batch"], 18)).astype(np.float32)
    y = (0.3 * r.standard_normal(case["batch"])).astype(np.float32)
    parts = []
    for fan, n, gain in ((18, 128, 1.0), (128, 128, 1.0), (128, 128, 1.0), (128, 1, 0.3)):
        parts += [gain * math.sqrt(6.0 / fan) * r.uniform(-1, 1, n * fan), 0.1 * r.uniform(-1, 1, n)]
    return X, y, np.concatenate(parts).astype(np.float32)


def energy_data(case, seed):
    """Dimensions, amplitudes (n_pp x n_hh) and interaction (n_hh x n_pp) of every channel, concatenated."""
    dims = layout_of(case, 0).hhpp_dims()
    n = sum(h * p for h, p in dims)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    t = torch.randn(2 * n, dtype=torch.float64, device="cuda", generator=g) * 3e-3
    v = torch.randn(2 * n, dtype=torch.float64, device="cuda", generator=g) * 0.5
    return dims, t, v


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """Energies of the MP2 amplitudes (and the triples sum on small lattices) from the
    matrix elements themselves; the amplitudes of a converged solve have no closed form."""
    kind = case["kind"]
    if kind == "learn":
        return exact_learn(case, seed)
    if kind == "energy":
        dims, t, v = energy_data(case, seed)
        at, e = 0, 0.0
        for h, p in dims:
            a = torch.view_as_complex(t[2 * at:2 * (at + h * p)].view(-1, 2)).view(h, p)
            b = torch.view_as_complex(v[2 * at:2 * (at + h * p)].view(-1, 2)).view(p, h)
            e = e + 0.25 * (a * b.T).sum()
            at += h * p
        return dict(e=torch.view_as_real(e))
    if kind == "batch":
        es = [Matter(case, density(case, seed), th).mp2() for th in twists(case)]
        return dict(e_mbpt2=[np.complex128(x) for x in es], e_ccd=[None] * len(es), t2=[None] * len(es))
    m = Matter(case, density(case, seed), (0.0, 0.0, 0.0))
    if kind == "triples":
        return dict(e_t=np.complex128(m.triples())) if triple_sizes(case)[0] < 3e6 else None
    if kind in ("setup", "handover"):
        return dict(e0=np.complex128(m.e0()), e_mbpt2=np.complex128(m.mp2()), t2=None)
    if kind == "steps":
        return dict(energies=[np.complex128(m.mp2())] + [None] * case["steps"], t2=None)
    return dict(e_mbpt2=np.complex128(m.mp2()), e_ccd=None, t2=None)


def exact_learn(case, seed):
    X, y, p = (torch.tensor(a, dtype=torch.float64, device="cuda") for a in learn_data(case, seed))
    p.requires_grad_(True)
    at, h = 0, X
    for i, o in ((18, 128), (128, 128), (128, 128), (128, 1)):
        W, b = p[at:at + i * o].view(o, i), p[at + i * o:at + i * o + o]
        at += i * o + o
        h = h @ W.T + b
        if o > 1:
            h = torch.nn.functional.silu(h)
    loss = ((h[:, 0] - y) ** 2).mean()
    loss.backward()
    return dict(loss=loss.detach(), grad=p.grad)


HBARC, PI, MASS = 197.326968, 3.14159265358979, float(np.float32(939.565))


def orbitals(case, rho, theta):
    """Quantum numbers, momenta (fm^-1) and hole mask of the lattice's states."""
    box = (case["A"] / rho) ** (1.0 / 3.0)
    r = range(-case["nmax"], case["nmax"] + 1)
    q = np.array(list(itertools.product(r, r, r, (-1, 1), (-1, 1) if case["snm"] else (1,))))
    n, sz, tz = q[:, :3], q[:, 3], q[:, 4]
    k = (2.0 * PI * n + np.array(theta)) / box
    holes = np.zeros(len(q), dtype=bool)
    holes[np.argsort(np.round((k * k).sum(1), 9), kind="stable")[:case["A"]]] = True
    return n, tz, sz, holes, k, box


class Matter:
    """A lattice with its synthetic interaction, element by element in 64 bits."""

    def __init__(self, case, rho, theta):
        n, tz, sz, holes, k, self.box = orbitals(case, rho, theta)
        at = dict(device="cuda" if torch.cuda.is_available() else "cpu")
        self.chiral, self.nmax = case["snm"], case["nmax"]
        self.n, self.tz, self.sz = (torch.tensor(x, **at) for x in (n, tz, sz))
        self.k = torch.tensor(k, dtype=torch.float64, **at)
        self.h = torch.tensor(np.nonzero(holes)[0], **at)
        self.p = torch.tensor(np.nonzero(~holes)[0], **at)
        ext = 2 * self.nmax + 1
        self.of = torch.full((ext, ext, ext, 2, 2), -1, dtype=torch.int64, **at)
        i = self.n + self.nmax
        self.of[i[:, 0], i[:, 1], i[:, 2], (self.sz + 1) // 2, (self.tz + 1) // 2] = torch.arange(len(n), **at)
        self.hole = torch.tensor(holes, **at)
        self.kin = (self.k ** 2).sum(1) * HBARC ** 2 / MASS / 2.0
        f = self.kin.to(torch.complex128)
        for x in self.h:
            f = f + self.anti(x, torch.arange(len(n), **at), x, torch.arange(len(n), **at))
        self.f = f

    def e0(self):
        i, j = self.h[:, None], self.h[None, :]
        return complex(self.kin[self.h].sum() + 0.5 * self.anti(i, j, i, j).sum())

    def closing(self, total, t, spin):
        """The orbital of momentum `total`, isospin t and the spin, or -1."""
        i = total + self.nmax
        ok = ((i >= 0) & (i <= 2 * self.nmax)).all(-1) & (t.abs() == 1)
        i, t = i.clamp(0, 2 * self.nmax), t.clamp(-1, 1)
        return torch.where(ok, self.of[i[..., 0], i[..., 1], i[..., 2], (spin + 1) // 2, (t + 1) // 2], -1)

    def anti(self, p, q, r, s):
        return self.bare(p, q, r, s) - self.bare(p, q, s, r)

    def bare(self, p, q, r, s):
        p, q, r, s = torch.broadcast_tensors(p, q, r, s)
        m, t = ([x[y] for y in (p, q, r, s)] for x in (self.sz, self.tz))
        ok = (self.n[p] + self.n[q] == self.n[r] + self.n[s]).all(-1) & (t[0] + t[1] == t[2] + t[3])

        def same(x):
            return ((x[0] == x[2]) & (x[1] == x[3])).double()

        def dot(x):  # sigma1 . sigma2
            swap = (x[0] == x[3]) & (x[1] == x[2]) & (x[0] != x[1])
            return torch.where(same(x) > 0, (x[0] * x[1]).double(), 2.0 * swap.double())

        dm, dt, ss, tt = same(m), same(t), dot(m), dot(t)
        pi, pf = 0.5 * (self.k[p] - self.k[q]), 0.5 * (self.k[r] - self.k[s])
        if not self.chiral:
            q2 = ((pi - pf) ** 2).sum(-1)

            def gauss(v, kappa):
                kappa = float(np.float32(kappa))
                return float(np.float32(v)) * (PI / kappa) ** 1.5 * torch.exp(-q2 / (4.0 * kappa))

            v = gauss(200.0, 1.487) * (3 * dm * dt - tt * dm - ss * dt - tt * ss) / 8.0
            v = v + -gauss(91.85, 0.465) * (3 * dm * dt + tt * dm - 3 * ss * dt - tt * ss) / 16.0
            v = v + -gauss(178.0, 0.639) * (3 * dm * dt - 3 * tt * dm + ss * dt - tt * ss) / 16.0
            return torch.where(ok, v, 0.0).to(torch.complex128) / self.box ** 3
        pi, pf = pi * HBARC, pf * HBARC
        km, qt = 0.5 * (pi + pf), pi - pf
        q2, k2, a2, b2 = ((x ** 2).sum(-1) for x in (qt, km, pi, pf))

        def sigma(x, a, b):  # <a| sigma . x |b>
            z, up = torch.where(a > 0, x[..., 2], -x[..., 2]), (a > 0).double()
            off = torch.complex(x[..., 0], x[..., 1] * (1.0 - 2.0 * up))
            return torch.where(a == b, z.to(torch.complex128), off)

        def both(x):
            return sigma(x, m[0], m[2]) * sigma(x, m[1], m[3])

        qxk = torch.linalg.cross(qt, km)
        ls = -0.5j * (sigma(qxk, m[0], m[2]) * (m[1] == m[3]) + sigma(qxk, m[1], m[3]) * (m[0] == m[2]))
        c = contacts()
        v = -(1.27 / 92.4) ** 2 / 4.0 / (q2 + 138.0 ** 2) * tt * both(qt)
        v = v + c[0] * dm * dt + c[1] * ss * dt + (c[2] * q2 + c[3] * k2) * dm * dt + (c[4] * q2 + c[5] * k2) * ss * dt
        v = v + dt * (c[6] * ls + c[7] * both(qt) + c[8] * both(km))
        tot = torch.div(t[0] + t[1], 2, rounding_mode="trunc")
        mass = torch.tensor([938.272046, 938.918267117927371, 939.565379], dtype=torch.float64, device=tot.device)
        mass = mass[tot.sign() + 1]
        v = v * mass / ((mass ** 2 + a2) * (mass ** 2 + b2)) ** 0.25 * torch.exp(-(a2 ** 3 + b2 ** 3) / 450.0 ** 6)
        return torch.where(ok, v, 0.0) * HBARC ** 3 / self.box ** 3

    def amplitude(self, a, b, i, j):
        """MP2 amplitude of the pairs."""
        return self.anti(i, j, a, b).conj() / (self.f[i] + self.f[j] - self.f[a] - self.f[b])

    def mp2(self):
        i, j = torch.combinations(self.h, 2).unbind(1)
        e, step = 0.0, max(1, 2_000_000 // len(self.p))
        for at in range(0, len(i), step):
            x, y, a = i[at:at + step, None], j[at:at + step, None], self.p[None, :]
            for spin in (-1, 1):
                b = self.closing(self.n[x] + self.n[y] - self.n[a], self.tz[x] + self.tz[y] - self.tz[a], spin)
                u, w = torch.nonzero((b > a) & ~self.hole[b.clamp(0)], as_tuple=True)
                v = self.anti(x[u, 0], y[u, 0], a[0, w], b[u, w])
                d = self.f[x[u, 0]] + self.f[y[u, 0]] - self.f[a[0, w]] - self.f[b[u, w]]
                e = e + (v * v.conj() / d).sum()
        return complex(e)

    def triples(self):
        """E(T) of the MP2 amplitudes: sum over i < j < k, a < b < c of |W|^2 / D."""
        hhh = torch.combinations(self.h, 3)
        ab = torch.combinations(self.p, 2)
        e, step = 0.0, max(1, 4_000_000 // len(ab))
        for at in range(0, len(hhh), step):
            x = hhh[at:at + step, None, :]
            n = self.n[x].sum(2) - self.n[ab].sum(1)[None]
            t = self.tz[x].sum(2) - self.tz[ab].sum(1)[None]
            for spin in (-1, 1):
                c = self.closing(n, t, spin)
                u, w = torch.nonzero((c > ab[None, :, 1]) & ~self.hole[c.clamp(0)], as_tuple=True)
                if len(u):
                    e = e + self.triple_terms(hhh[at + u], torch.cat([ab[w], c[u, w][:, None]], 1))
        return complex(e)

    def triple_terms(self, ijk, abc):
        w = 0.0
        for ph, (i, j, k) in ((1, (0, 1, 2)), (-1, (2, 1, 0)), (-1, (0, 2, 1))):
            for pp, (a, b, c) in ((1, (0, 1, 2)), (-1, (1, 0, 2)), (-1, (2, 1, 0))):
                w = w + ph * pp * self.through_particle(*abc[:, [a, b, c]].T, *ijk[:, [i, j, k]].T)
        for ph, (i, j, k) in ((1, (0, 1, 2)), (-1, (2, 1, 0)), (-1, (1, 0, 2))):
            for pp, (a, b, c) in ((1, (0, 1, 2)), (-1, (0, 2, 1)), (-1, (2, 1, 0))):
                w = w - ph * pp * self.through_hole(*abc[:, [a, b, c]].T, *ijk[:, [i, j, k]].T)
        return (w * w.conj() / (self.f[ijk].sum(1) - self.f[abc].sum(1))).sum()

    def through_particle(self, a, b, c, i, j, k):
        out = 0.0
        for spin in (-1, 1):
            d = self.closing(self.n[i] + self.n[j] - self.n[a], self.tz[i] + self.tz[j] - self.tz[a], spin)
            ok, d = (d >= 0) & ~self.hole[d.clamp(0)], d.clamp(0)
            out = out + torch.where(ok, self.anti(c, b, k, d).conj() * self.amplitude(a, d, i, j), 0.0)
        return out

    def through_hole(self, a, b, c, i, j, k):
        out = 0.0
        for spin in (-1, 1):
            m = self.closing(self.n[k] + self.n[j] - self.n[c], self.tz[k] + self.tz[j] - self.tz[c], spin)
            ok, m = (m >= 0) & self.hole[m.clamp(0)], m.clamp(0)
            out = out + torch.where(ok, self.anti(j, k, m, c).conj() * self.amplitude(a, b, i, m), 0.0)
        return out


def contacts():
    """Contact strengths of the chiral-like interaction: a splitmix64 stream within half of their centres."""
    state, out, mask = 20261203, [], (1 << 64) - 1
    for i, c in enumerate((-0.1, 0.01) + (0.1,) * 7):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        u = ((z ^ (z >> 31)) >> 11) * 2.0 ** -53
        out.append(c * (0.5 + u) * (1e-2 if i < 2 else 1e-8) / (16.0 * PI))
    return out
