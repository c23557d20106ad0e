"""What a user of this framework has it do, as cases to time: each through the public entry point a program
would call, on inputs made from a seed.

Precision.  The engine returns every result in FP64 arrays whatever it computed in.  Where a case asks for
the mixed path (FP32 terms and transforms), the program keeps the result in FP32, the precision it asked
for; results of the FP64 path stay FP64.

`exact` restates each result in FP64 with torch and numpy alone, from the definitions: the dense sums
instead of the separable expansion, closed-form Bessel functions, plain matrix products.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from sgl_analytic_gb300 import Lam, Population, invert
from sgl_analytic_gb300 import cfbatch, cosmology, planes, surrogate, workloads
from sgl_analytic_gb300._lib import SGL_FP64, SGL_MIXED, Engine
from sgl_analytic_gb300.cells import Cells

# the CLI's ln mu grid (1601 points of the body, 1600 of the tail)
XI_OUT = np.concatenate([np.linspace(-1.0, 1.0, 1601), np.linspace(1.005, 9.0, 1600)])
F64 = torch.float64


def listed():
    return [
        # generate_pdf_lnmu(1.0) on a resident population, FP32 arithmetic: the headline benchmark
        dict(name="pdf_mixed", kind="pdf", precision="mixed", cells=1.0, shells=67, n_x=3201),
        # the same in the default precision, the one results are published from
        dict(name="pdf_fp64", kind="pdf", precision="fp64", cells=1.0, shells=67, n_x=3201),
        # the drop-in call with a new population in host memory every time (Lam, then invert)
        dict(name="dropin_mixed", kind="dropin", precision="mixed", cells=1.0, shells=67, n_x=3201),
        # the smallest PDF: a thousand broad cells without clustering, a short ln mu grid
        dict(name="pdf_few_cells", kind="few", precision="mixed", cells=1000, n_x=161),
        # a PDF with the positive (vp) closure over 24 shells
        dict(name="pdf_vp", kind="vp", precision="mixed", shells=24, n_x=3201),
        # one-dimensional compound-Poisson CF over a long list of cells, ragged sizes
        dict(name="cf_sweep", kind="sweep", precision="mixed", nz=32, nm=64, nb=509, nk=5003),
        # uneven (cosmology, z_s, closure) instances in one call, dP/dln mu of each
        dict(name="cf_batch", kind="batch", precision="mixed", n=41, nm=12, nb=12, n_x=2048),
        # plain solver in node form over z_s = 1 instances of 64 planes x 131072 cells
        dict(name="node_pdfs", kind="nodes", precision="mixed", n=6, zs=1.0, n_x=2048),
        # one training step of a surrogate member: forward, loss, backward, AdamW
        dict(name="surrogate_train", kind="train", batch=16384),
        # inference of a trained member at every node of a sweep, a ragged number of rows
        dict(name="surrogate_infer", kind="infer", rows=700001),
        # one lens-redshift node of the population build deposited and compressed
        dict(name="deposit_node", kind="cells", n_host=512, n_fil=128, nx=260, nu=119),
        # the chain's cosmology tables for the cosmologies of a small grid
        dict(name="cosmo_tables", kind="cosmo", n=24, nz=65, nm=48, nzm=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pdf", "pdf", "dropin", "few", "vp", "sweep", "batch", "nodes", "train", "infer", "cells", "cosmo"])
    prec = rng.choice(["mixed", "fp64"])
    nx = rng.randrange(101, 3201)
    if kind in ("pdf", "dropin"):
        return dict(kind=kind, precision=prec if kind == "pdf" else "mixed", cells=round(rng.uniform(0.15, 1.0), 3),
                    shells=rng.randrange(1, 68), n_x=nx)
    if kind == "few":
        return dict(kind=kind, precision=prec, cells=rng.randrange(300, 1001), n_x=nx)
    if kind == "vp":
        return dict(kind=kind, precision="mixed", shells=rng.randrange(3, 25), n_x=nx)
    if kind == "sweep":
        return dict(kind=kind, precision="mixed", nz=rng.randrange(1, 33), nm=rng.randrange(16, 65), nb=rng.randrange(64, 510),
                    nk=_log_int(rng, 17, 5003))
    if kind == "batch":
        return dict(kind=kind, precision="mixed", n=_log_int(rng, 2, 41), nm=rng.randrange(6, 13), nb=rng.randrange(6, 13), n_x=nx // 2 + 51)
    if kind == "nodes":
        return dict(kind=kind, precision="mixed", n=rng.randrange(1, 7), zs=round(rng.uniform(0.2, 1.0), 3), n_x=nx // 2 + 51)
    if kind == "train":
        return dict(kind=kind, batch=_log_int(rng, 1024, 16384))
    if kind == "infer":
        return dict(kind=kind, rows=_log_int(rng, 257, 700001))
    if kind == "cells":
        return dict(kind=kind, n_host=_log_int(rng, 8, 512), n_fil=_log_int(rng, 4, 128), nx=rng.randrange(100, 261),
                    nu=rng.randrange(40, 120))
    return dict(kind=kind, n=_log_int(rng, 1, 24), nz=rng.randrange(5, 66), nm=rng.randrange(8, 49), nzm=rng.randrange(1, 6))


# ---------------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _fixture(name):
    """Arrays of one of the repository's own population files, read once per process."""
    d = np.load(workloads.GOLDEN / name)
    return {k: d[k] for k in d.files}


def _population(case, seed):
    """The reference's z_s = 1 cells (a random part of them, the weights scaled up to keep the population's
    width) with the clustering groups of `shells` shells, every weight and shell amplitude jittered."""
    rng = np.random.default_rng(seed)
    b, st = _fixture("pop_zs1_sub.npz"), _fixture("zs1_xi_shell_stats.npz")
    n = b["w0"].size
    take = np.arange(n) if case["cells"] >= 1.0 else np.sort(rng.choice(n, int(n * case["cells"]), replace=False))
    w0 = b["w0"][take] * np.exp(0.05 * rng.standard_normal(take.size)) * (n / take.size)
    rows, off = [], 0
    for r, i in zip(b["xg_nrow"], b["xg_nidx"]):
        rows.append(b["xg_rows"][off:off + int(r) * (int(i) + 1)])
        off += int(r) * (int(i) + 1)
    shells = case["shells"]
    f = st["norms"][:shells] / st["norms"][workloads.BASE_SHELL] * np.exp(0.05 * rng.standard_normal((shells, 1)))
    pop = Population(w0=w0, k0=b["k0"][take], g0=b["g0"][take], ig=b["ig"][take], fe_g=b["fe_g"], V=float(b["V"]),
                     xg_m=np.tile(b["xg_m"], shells), xg_nrow=np.tile(b["xg_nrow"], shells),
                     xg_nidx=np.tile(b["xg_nidx"], shells), xg_idx=np.tile(b["xg_idx"], shells),
                     xg_rows=np.concatenate([rows[g] * f[s, b["xg_m"][g]] for s in range(shells) for g in range(3)]),
                     ce_k=b["ce_k"], ce_g=b["ce_g"], xg_s0=float(st["s0"]))
    return pop, f


def _few(case, seed):
    rng = np.random.default_rng(seed)
    b = _fixture("pop_window.npz")
    take = np.sort(rng.choice(b["w0"].size, case["cells"], replace=False))
    w0 = b["w0"][take] * np.exp(0.05 * rng.standard_normal(take.size)) * (b["w0"].size / take.size)
    return Population(w0=w0, k0=b["k0"][take], g0=b["g0"][take], ig=b["ig"][take], fe_g=b["fe_g"], V=float(b["V"]))


def _vp(case, seed):
    """The z_s = 1 cells, one shell's clustering groups (they set sigma) and the positive closure of the first
    shells repeated up to `shells`, its weights shared out so that the closure keeps its strength."""
    rng = np.random.default_rng(seed)
    pop, f = _population(dict(cells=1.0, shells=1), seed)
    b, n = _fixture("vp_zs1_sub.npz"), case["shells"]
    ns = b["sh_g"].size - 1
    cw = b["cw"] * np.exp(0.05 * rng.standard_normal(b["cw"].size))
    d = {k: b[k] for k in ("u", "w", "ku", "gu", "shear_var")}
    parts = {k: [] for k in ("cu", "cw", "ga", "gb", "gc", "glo", "ghi")}
    gstart, sh_g, K, nc = [np.zeros(1, np.int64)], [0], [], 0
    for s in range(n):
        r = s % ns
        g0, g1 = int(b["sh_g"][r]), int(b["sh_g"][r + 1])
        c0, c1 = int(b["gstart"][g0]), int(b["gstart"][g1])
        parts["cu"].append(b["cu"][c0:c1])
        parts["cw"].append(cw[c0:c1] * (ns / n))
        for k in ("ga", "gb", "gc", "glo", "ghi"):
            parts[k].append(b[k][g0:g1])
        gstart.append(b["gstart"][g0 + 1:g1 + 1] - c0 + nc)
        nc += c1 - c0
        sh_g.append(sh_g[-1] + g1 - g0)
        if s:
            K.append(b["K"][(s - 1) % (ns - 1)])
    d.update({k: np.concatenate(v) for k, v in parts.items()})
    d.update(gstart=np.concatenate(gstart), sh_g=np.array(sh_g, np.int32), K=np.array(K))
    return pop, f, d


def _sweep(case, seed):
    return workloads.cf_sweep_problem(seed=seed, nz=case["nz"], nm=case["nm"], nb=case["nb"], nk=case["nk"])


def _batch(case, seed):
    return cfbatch.make_batch(case["n"], seed=seed, nm=case["nm"], nb=case["nb"])


def _tables(case, seed):
    th, zs = surrogate.sample_instances(case["n"], seed, zs=case["zs"])
    return surrogate.SweepTables(planes.PlaneModel(), th, zs)


def _rows(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return 2 * torch.rand((n, 8), generator=g, device="cuda") - 1


def _member(seed):
    """A member in the middle of its training: weights, and AdamW moments of the size its gradients have."""
    m = surrogate.MLP(Engine(0), seed=seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    for w, b in zip(m.W, m.b):
        b += 0.1 * torch.randn(b.shape, generator=g, device="cuda")
    for lst, s in ((m.mW, 1e-3), (m.mb, 1e-3)):
        for t in lst:
            t += s * torch.randn(t.shape, generator=g, device="cuda")
    for lst in (m.vW, m.vb):
        for t in lst:
            t += 1e-4
    m.step_count = 1000
    torch.cuda.synchronize()
    return m


def _targets(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 1)
    return torch.randn((n, 2), generator=g, device="cuda")


def _xi_nodes():
    b = _fixture("cells_ref.npz")
    return dict(kp=b["xi_kp"], c=b["xi_c"], mmax=2)


def _node(case, seed):
    return workloads.deposit_node(seed=seed, n_host=case["n_host"], n_fil=case["n_fil"], nx=case["nx"], nu=case["nu"])


def _cosmo(case, seed):
    """Cosmologies around the default one, all with curvature and a CPL dark energy, and table axes."""
    rng = np.random.default_rng(seed)
    d = cosmology.DEFAULT
    u = rng.uniform(-1, 1, (case["n"], 9))
    width = dict(h=0.05, Om=0.05, Ob=0.004, s8=0.08, ns=0.03, zeq=60.0, Ok=0.04, w0=0.15, wa=0.2)
    p = np.array([[d[k] + width[k] * v for k, v in zip(cosmology.PARAM_KEYS, row)] for row in u])
    z = np.sort(np.expm1(rng.uniform(0.01, math.log(11.0), case["nz"])))
    return p, z, np.geomspace(1e8, 1e15, case["nm"]) * math.exp(0.1 * u[0, 0]), np.sort(rng.uniform(0.05, 6.0, case["nzm"]))


def _x(case):
    n = case["n_x"]
    if case["kind"] in ("batch", "nodes"):
        return np.linspace(-0.5, 2.0, n)
    return XI_OUT if n == XI_OUT.size else np.linspace(-1.0, 3.0, n)


def prepare(case, seed):
    kind, prec = case["kind"], case.get("precision")
    s = dict(case=case)
    if "n_x" in case:
        s["x"] = _x(case)
    if kind in ("pdf", "dropin"):
        pop, _ = _population(case, seed)
        s["engine"] = Engine(0)
        if kind == "pdf":
            s["lam"] = Lam(pop, xi=True, engine=s["engine"], precision=prec)
        else:
            s["pop"] = pop
    elif kind == "few":
        s["lam"] = Lam(_few(case, seed), precision=prec)
    elif kind == "vp":
        pop, _, d = _vp(case, seed)
        s["lam"] = Lam(pop, xi=True, precision=prec)
        s["lam"].install_vp(d)
    elif kind == "sweep":
        kap, w, s["kk"] = _sweep(case, seed)
        s["engine"] = Engine(0)
        s["engine"].sweep_set_cells(kap, w)
    elif kind == "batch":
        s["engine"] = Engine(0)
        s["engine"].cfb_set(_batch(case, seed).arrays())
    elif kind == "nodes":
        s["engine"], s["tables"] = Engine(0), _tables(case, seed)
    elif kind == "train":
        s["mlp"], s["X"], s["Y"] = _member(seed), _rows(case["batch"], seed), _targets(case["batch"], seed)
    elif kind == "infer":
        s["mlp"], s["X"] = _member(seed), _rows(case["rows"], seed)
    elif kind == "cells":
        s["engine"], (s["objects"], s["dchi"]), s["xi"] = Engine(0), _node(case, seed), _xi_nodes()
        # where the build collects its nodes' row groups: room for every coarse bin and every k_perp node
        bins = 340 * 110
        s["idx"], s["rows"], s["sizes"] = np.zeros(3 * bins, np.int32), np.zeros(3 * 42 * (bins + 1)), np.zeros(9, np.int64)
    else:
        s["engine"], s["args"] = Engine(0), _cosmo(case, seed)
    return s


# ---------------------------------------------------------------------------------------- one pass
def _kept(a, precision):
    """The result in the precision that was asked for."""
    if precision != "mixed":
        return a
    return a.astype(np.complex64 if np.iscomplexobj(a) else np.float32)


def _pdf(lam, x, **kw):
    prec = "mixed" if lam.precision == SGL_MIXED else "fp64"
    _, P, m = invert(lam, lam.sigma(), xi_out=x, phi_tol=1e-8, **kw)
    return dict(P=_kept(P, prec), moments=_kept(np.array([m["mean"], m["var"], m["skew"], m["norm"]]), prec))


def run(s):
    case = s["case"]
    kind, prec = case["kind"], case.get("precision")
    if kind in ("pdf", "few"):
        return _pdf(s["lam"], s["x"])
    if kind == "dropin":
        return _pdf(Lam(s["pop"], xi=True, engine=s["engine"], precision=prec), s["x"])
    if kind == "vp":
        return _pdf(s["lam"], s["x"], window="auto", n_xi_wide=4000)
    if kind == "sweep":
        return _kept(s["engine"].sweep(s["kk"], SGL_MIXED if prec == "mixed" else SGL_FP64), prec)
    if kind == "batch":
        return _kept(s["engine"].cfb_pdf(s["x"], SGL_MIXED if prec == "mixed" else SGL_FP64)[0], prec)
    if kind == "nodes":
        return _kept(surrogate.plain_node_pdfs(s["engine"], s["tables"], s["x"])[0], prec)
    if kind == "train":
        m = s["mlp"]
        pred = m.forward(s["X"], keep=True)
        loss, dY = m.loss_grad(pred, s["Y"])
        grads = m.backward_step(dY, 1e-3)
        return dict(pred=pred, loss=loss, grads=[[dW, db] for _, dW, db in grads], W=m.W, b=m.b)
    if kind == "infer":
        return s["mlp"].infer(s["X"])
    if kind == "cells":
        c = Cells(1, 1, xi=s["xi"], engine=s["engine"])
        c.xi_begin(s["dchi"])
        c.add_many(s["objects"])
        c.xi_end(0)
        ni = nr = 0
        for j, g in enumerate(c.xi_groups):
            s["sizes"][3 * j:3 * j + 3] = g["m"], g["idx"].size, g["rows"].shape[0]
            s["idx"][ni:ni + g["idx"].size] = g["idx"]
            s["rows"][nr:nr + g["rows"].size] = g["rows"].ravel()
            ni, nr = ni + g["idx"].size, nr + g["rows"].size
        return dict(H0=c.H0, H0k=c.H0k, H0g=c.H0g, Hc=c.Hc, totals=np.array([c.N, c.dropped]), sizes=s["sizes"],
                    idx=s["idx"], rows=s["rows"])
    p, z, M, zm = s["args"]
    return s["engine"].cosmo_tables(p, z, M, zm)


# ---------------------------------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once, and the operations of the shortest known way: a (k, cell)
    term of a CF is one sine, one cosine and two multiply-adds (about 30 operations)."""
    kind = case["kind"]
    if kind in ("pdf", "dropin", "vp"):
        # the z_s = 1 grid: 1683 x 2687 k-points onto 2400 x 796 output points
        nc = 79574 * case.get("cells", 1.0)
        rows = 564277 * 8 * (case["shells"] if kind != "vp" else 1) + (193341 / 6 * case["shells"] * 20 if kind == "vp" else 0)
        sep = 2.0 * 2 * 1683 * 6384 * 580
        tr = 2.0 * 2 * 1683 * 2687 * 796 + 2.0 * 2400 * 2 * 1683 * 798
        xi = 2.0 * 2 * 101 * 101 * 8 * 341 * 3 * 8 * case["shells"] / 3 if kind != "vp" else 405 * 101 * 193341 / 6 * case["shells"] * 12.0
        return dict(bytes=nc * 32 + rows + 8 * case["n_x"], flops=30.0 * 1683 * nc + sep + tr + xi)
    if kind == "few":
        return dict(bytes=32.0 * case["cells"] + 8 * case["n_x"], flops=1e10)
    if kind == "sweep":
        nc = case["nz"] * case["nm"] * case["nb"]
        return dict(bytes=16.0 * nc + 24.0 * case["nk"], flops=30.0 * nc * case["nk"])
    if kind == "batch":
        k, c = case["n"] * 18432.0, 144.0 * case["nm"] * case["nb"]
        return dict(bytes=16.0 * case["n"] * c + 8.0 * case["n"] * case["n_x"], flops=30.0 * k * c + 8.0 * k * case["n_x"])
    if kind == "nodes":
        pl = sum(planes.n_planes(case["zs"]) for _ in range(case["n"]))
        return dict(bytes=pl * 256 * 16.0 + 8.0 * case["n"] * case["n_x"], flops=30.0 * pl * 131072 * 128)
    per_row = 2.0 * (8 * 256 + 5 * 256 * 256 + 256 * 2)
    if kind == "train":
        return dict(bytes=case["batch"] * 40.0 + 6 * 4.0 * 330000, flops=case["batch"] * per_row * 3)
    if kind == "infer":
        return dict(bytes=case["rows"] * 40.0 + 4.0 * 330000, flops=case["rows"] * per_row)
    if kind == "cells":
        n = case["n_host"] * 12 * case["nx"] + case["n_fil"] * 12 * case["nu"]
        return dict(bytes=32.0 * n + 3 * 8 * 960 * 300 + 8 * 42.0 * 3 * 12000, flops=2.0 * 42 * 3 * n)
    return dict(bytes=case["n"] * 8.0 * (9 + 4 * case["nz"] + 2 * case["nm"] + 2 * case["nzm"] * case["nm"]),
                flops=case["n"] * (500 * 4000 * 10.0 + 32768 * 4 * 40.0))


# ---------------------------------------------------------------------------------------- exact values
def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device="cuda")


def _bessel(n, x, less=0.0):
    """J_n(x) - less for n = 0, 1, 2: below 25 Bessel's integral by the 64-point rule on the circle (its error
    is of the size of J_64; for n = 0 and less = 1 the small parts are kept), from 25 on Hankel's asymptotic
    expansion."""
    out = torch.zeros_like(x)
    for j in range(16):
        t = (j + 0.5) * math.pi / 32
        y = x * math.sin(t)
        if n == 0:
            out += -2 * torch.sin(0.5 * y) ** 2 + (1 - less) if less else torch.cos(y)
        else:
            out += torch.sin(y) * math.sin(t) if n == 1 else torch.cos(y) * math.cos(2 * t)
    out /= 16
    z = x.clamp_min(25.0)
    term, p, q = torch.ones_like(z), torch.ones_like(z), torch.zeros_like(z)
    for k in range(1, 21):
        term = term * ((4 * n * n - (2 * k - 1) ** 2) / (8.0 * k)) / z
        if k % 2:
            q = q + (1 if k % 4 == 1 else -1) * term
        else:
            p = p + (1 if k % 4 == 0 else -1) * term
    w = z - (0.5 * n + 0.25) * math.pi
    return torch.where(x < 25, out, torch.sqrt(2 / (math.pi * z)) * (p * torch.cos(w) - q * torch.sin(w)) - less)


def _j0m1(x):
    return _bessel(0, x, less=1.0)


def _comp(ph):
    """e^{i ph} - 1 - i ph as (re, im)."""
    h = torch.sin(0.5 * ph)
    p2 = ph * ph
    ser = -ph * p2 / 6 * (1 - p2 / 20 * (1 - p2 / 42 * (1 - p2 / 72 * (1 - p2 / 110))))
    return -2 * h * h, torch.where(ph.abs() < 0.3, ser, torch.sin(ph) - ph)


def _psi1(pop, kk, kg, chunk=8192):
    """sum_c w (e^{i kk kap} J0(kg gam) - 1 - i kk kap), dense, in pieces that keep their small parts."""
    kk, kg = _t(kk), _t(kg)
    re = torch.zeros((kk.numel(), kg.numel()), dtype=F64, device="cuda")
    im = torch.zeros_like(re)
    for a in range(0, pop.w0.size, chunk):
        k0, g0, w = (_t(v[a:a + chunk]) for v in (pop.k0, pop.g0, pop.w0))
        B = _j0m1(torch.outer(g0, kg))
        ph = torch.outer(kk, k0)
        c, s = _comp(ph)
        re += (c * w) @ B + (c @ w)[:, None] + (w @ B)[None, :]
        im += (torch.sin(ph) * w) @ B + (s @ w)[:, None]
    return torch.complex(re, im)


def _groups(f):
    """(m, row sums' amplitude over the shells, up, uq, dense rows (r, nP, nQ), residuals) of the three base
    groups: every shell's groups are one of them times f, so the shells' squares add up to one factor."""
    b = _fixture("pop_zs1_sub.npz")
    out, ro, io = [], 0, 0
    ngc = b["ce_g"].size - 1
    for m, r, n in zip(b["xg_m"], b["xg_nrow"], b["xg_nidx"]):
        m, r, n = int(m), int(r), int(n)
        rows = b["xg_rows"][ro:ro + r * (n + 1)].reshape(r, n + 1)
        idx = b["xg_idx"][io:io + n].astype(np.int64)
        ro, io = ro + r * (n + 1), io + n
        up, pi = np.unique(idx // ngc, return_inverse=True)
        uq, qi = np.unique(idx % ngc, return_inverse=True)
        H = np.zeros((r, up.size, uq.size))
        H[:, pi, qi] = rows[:, :-1]
        out.append((m, float(np.sum(f[:, m] ** 2)), up, uq, _t(H), _t(rows[:, -1])))
    return out


def _centres():
    b = _fixture("pop_zs1_sub.npz")
    e, g = b["ce_k"], b["ce_g"]
    p = e[:-1] * e[1:]
    return np.where(p > 0, np.sign(e[1:]) * np.sqrt(np.abs(p)), 0.0), np.sqrt(g[:-1] * g[1:])


def _psi2(f, kk, kg):
    """The gauss two-point term, 1/2 sum over rows of the squared amplitudes."""
    kc, gc = _centres()
    kk, kg = _t(kk), _t(kg)
    out = torch.zeros((kk.numel(), kg.numel()), dtype=torch.complex128, device="cuda")
    for m, amp, up, uq, H, res in _groups(f):
        x = torch.outer(_t(gc[uq]), kg)
        J = _bessel(m, x)
        T = torch.einsum("rpq,qk->rpk", H, J)
        ph = torch.outer(kk, _t(kc[up]))
        Gr, Gi = torch.einsum("np,rpk->rnk", torch.cos(ph), T), torch.einsum("np,rpk->rnk", torch.sin(ph), T)
        if m == 0:
            Gr = Gr - H.sum((1, 2))[:, None, None]
            Gi = Gi + kk[None, :, None] * res[:, None, None]
        elif m == 1:
            Gr = Gr + 0.5 * kg[None, None, :] * res[:, None, None]
        G = torch.complex(Gr, Gi)
        out += 0.5 * (1.0 if m == 0 else 2.0 * (-1) ** m) * amp * (G * G).sum(0)
    return out


def _sigma(pop, f):
    v = float(np.sum(pop.w0 * pop.k0 ** 2)) + pop.V
    if f is not None:
        kc, _ = _centres()
        for m, amp, up, uq, H, res in _groups(f):
            if m == 0:
                v += amp * float(((H.sum(2) @ _t(kc[up]) + res) ** 2).sum())
    return math.sqrt(v)


def _vp_lnR(d, kk, kg):
    """ln R of the positive closure: the shells' rate-weighted sums, then the chain over the shells."""
    kk, kg, u, w = _t(kk), _t(kg), _t(d["u"]), _t(d["w"])
    nk, nq, ns = kk.numel(), kg.numel(), u.numel()
    lin = _t(d["gc"]) == 0
    lo, hi = (torch.as_tensor(d[k].astype(np.int64), device="cuda") for k in ("glo", "ghi"))
    anchor = torch.where(hi == ns - 1, u[lo], u[hi])
    j = torch.arange(ns, device="cuda")
    on = (j[None, :] >= lo[:, None]) & (j[None, :] <= hi[:, None])
    ga, gb, gc = (_t(d[k])[:, None] for k in ("ga", "gb", "gc"))
    D = torch.where(lin[:, None], ga * u + gb, gc + torch.where(on, (u - anchor[:, None]) * ga + gb, 0.0))
    size = torch.as_tensor(np.diff(d["gstart"]), device="cuda")
    grp = torch.repeat_interleave(torch.arange(D.shape[0], device="cuda"), size)
    cw, cu = _t(d["cw"]), torch.as_tensor(d["cu"].astype(np.int64), device="cuda")
    ku, gu = _t(d["ku"]), _t(d["gu"])
    a, scale, kept = None, torch.zeros((nk, nq), dtype=F64, device="cuda"), {}
    n_sh = d["sh_g"].size - 1
    for s in range(n_sh):
        if s % 6 not in kept:                              # the shells repeat with a period of six
            z = torch.zeros((ns, nk, nq), dtype=torch.complex128, device="cuda")
            c0, c1 = int(d["gstart"][d["sh_g"][s]]), int(d["gstart"][d["sh_g"][s + 1]])
            for c in range(c0, c1, 4096):
                i = cu[c:min(c + 4096, c1)]
                A = (D[grp[c:min(c + 4096, c1)]] * cw[c:min(c + 4096, c1), None]).T.contiguous()
                B = _j0m1(torch.outer(gu[i], kg))
                z += (A @ B)[:, None, :]
                for n0 in range(0, nk, 64):
                    ph = torch.outer(kk[n0:n0 + 64], ku[i])
                    er, ei = -2 * torch.sin(0.5 * ph) ** 2, torch.sin(ph)
                    z[:, n0:n0 + 64] += torch.complex(*(torch.matmul((A[:, None, :] * e[None]).reshape(-1, i.numel()), B + 1)
                                                        .reshape(ns, -1, nq) for e in (er, ei)))
            kept[s % 6] = z
        z = kept[s % 6]
        K = w[:, None, None].to(torch.complex128).expand(ns, nk, nq) if s == 0 else \
            torch.einsum("ij,ikq->jkq", _t(d["K"][s - 1]).to(torch.complex128), a)
        mx = z.real.amax(0)
        a = K * torch.exp(z - mx)
        nrm = a.abs().amax(0)
        a = a / nrm
        scale += mx + torch.log(nrm)
    t = a.sum(0)
    return torch.complex(scale + torch.log(t.abs()), torch.angle(t))


def _vp_term(d, kk, kg):
    v = _vp_lnR(d, kk, kg).cpu().numpy()
    im = v.imag.copy()
    im[:, 0] = np.unwrap(im[:, 0])
    im = np.unwrap(im, axis=1)
    return _t(v.real - 0.25 * float(d["shear_var"]) * np.asarray(kg)[None, :] ** 2) + 1j * _t(im)


def _spline(n, s):
    """Matrix (len(s), n) of the not-a-knot cubic interpolant on n uniform nodes of [0, 1]."""
    h = 1.0 / (n - 1)
    A, B = np.zeros((n, n)), np.zeros((n, n))              # A (second derivatives) = B (values)
    for i in range(1, n - 1):
        A[i, i - 1:i + 2] = h / 6, 2 * h / 3, h / 6
        B[i, i - 1:i + 2] = 1 / h, -2 / h, 1 / h
    A[0, :3] = A[-1, -3:] = 1, -2, 1
    S2 = np.linalg.solve(A, B)
    i = np.minimum((s * (n - 1)).astype(int), n - 2)
    b = s * (n - 1) - i
    a = 1 - b
    M = (((a ** 3 - a) * h * h / 6)[:, None] * S2[i] + ((b ** 3 - b) * h * h / 6)[:, None] * S2[i + 1])
    M[np.arange(s.size), i] += a
    M[np.arange(s.size), i + 1] += b
    return _t(M)


def _path(P3, kap, gam, xs, g_def, n_int=2400):
    """Constant-mu path integrals of the bilinear P3, trapezoid rule."""
    dk, dg = kap[1] - kap[0], gam[1] - gam[0]
    k_lo, k_hi, g_hi = float(kap[0]), float(kap[-1]), float(gam[-1])

    def at(k, g):
        ok = (k >= k_lo) & (k <= k_hi) & (g >= 0) & (g <= g_hi)
        i = ((k - k_lo) / dk).floor().long().clamp(0, kap.numel() - 2)
        j = (g / dg).floor().long().clamp(0, gam.numel() - 2)
        a, b = (k - kap[i]) / (kap[i + 1] - kap[i]), (g - gam[j]) / (gam[j + 1] - gam[j])
        v = (1 - a) * ((1 - b) * P3[i, j] + b * P3[i, j + 1]) + a * ((1 - b) * P3[i + 1, j] + b * P3[i + 1, j + 1])
        return torch.where(ok, v, 0.0)

    out = torch.zeros(xs.size, dtype=F64, device="cuda")
    for q, xi in enumerate(xs):
        mu = math.exp(xi)
        rm = 1 / math.sqrt(mu)
        hi, lo = 1 - rm, max(k_lo, 1 - math.sqrt(1 / mu + g_def ** 2))
        if hi <= lo:
            continue
        ke = _line(lo, hi, n_int)
        out[q] = math.pi / mu ** 2 * torch.trapezoid(at(ke, ((hi - ke) * (1 - ke + rm)).clamp_min(0).sqrt()), ke)
        if g_hi > g_def and lo > k_lo:
            gb = min(g_hi, math.sqrt(max((hi - k_lo) * (1 - k_lo + rm), 0.0)))
            if gb > g_def:
                gx = _line(g_def, gb, int(math.ceil((gb - g_def) / (0.5 * float(dg)))) + 1)
                r = (1 / mu + gx ** 2).sqrt()
                out[q] += math.pi / mu ** 2 * torch.trapezoid(at((1 - r).clamp(k_lo, k_hi), gx) * gx / r, gx)
    return out.cpu().numpy()


def _line(a, b, n):
    v = a + (b - a) * torch.arange(n, dtype=F64, device="cuda") / (n - 1)
    v[-1] = b
    return v


def _exact_pdf(pop, f, x, vp=None, n_wide=500):
    """The inversion to P_s(ln mu): box and reach from sigma and |Phi|, ln Phi on the k grid, the Hankel and
    kappa transforms with the endpoint term, the path integrals, the normalisation."""
    sig = _sigma(pop, f)

    def direct(kk, kg):
        L = _psi1(pop, kk, kg) - 0.5 * pop.V * (_t(kk) ** 2)[:, None]
        if vp is not None:
            return L + _vp_term(vp, kk, kg)
        return L if f is None else L + _psi2(f, kk, kg)

    xi_max = 48.0 * sig
    k_hi, k_lo, g_def = 1 - math.exp(-0.5 * xi_max), -6.0 * sig, 6.0 * sig
    kap_max, gam_max = max(k_hi, 0.99), max(g_def, 0.8)
    dk = 2 * math.pi / (18.0 * max(abs(k_lo), k_hi))
    dg = min(2 * math.pi / (96.0 * g_def), 2 * math.pi / (12.0 * gam_max))
    probes = 12.0 / sig * 1.25 ** np.arange(int(math.ceil(math.log(64.0) / math.log(1.25))) + 1)
    top = []
    for L in (direct(probes, np.zeros(1))[:, 0], direct(np.zeros(1), probes)[0]):
        phi = np.exp(L.real.cpu().numpy())
        ok = np.nonzero(phi <= 1e-8)[0]
        i = int(ok[0]) if ok.size else int(np.argmin(phi))
        top.append((float(probes[i]), float(phi[i])))
    (kmax, pk), (gmax, pg) = top
    kk = np.linspace(0, kmax, int(math.ceil(kmax / dk)) + 1)
    kg = np.linspace(0, gmax, int(math.ceil(gmax / dg)) + 1)
    kap = np.linspace(k_lo, kap_max, int(math.ceil((kap_max - k_lo) / (sig / 72.0))) + 1)
    gam = np.linspace(0, gam_max, int(math.ceil(gam_max / (sig / 36.0))) + 1)
    L = _psi1(pop, kk, kg) - 0.5 * pop.V * (_t(kk) ** 2)[:, None]
    if f is not None:
        ng = nk = 101
        if vp is not None:
            ng = int(min(401, max(101, 1 + math.ceil(12.65 * math.sqrt(gmax * sig)))))
            nk = int(min(4001, max(ng, 1 + math.ceil(66.7 * math.sqrt(kmax * sig)))))
        sk, sg = np.linspace(0, 1, nk), np.linspace(0, 1, ng)
        Q = _vp_term(vp, kmax * sk ** 2, gmax * sg ** 2) if vp is not None else _psi2(f, kmax * sk ** 2, gmax * sg ** 2)
        A, B = _spline(nk, np.sqrt(np.clip(kk / kmax, 0, 1))), _spline(ng, np.sqrt(np.clip(kg / gmax, 0, 1)))
        L += torch.complex(A @ Q.real @ B.T, A @ Q.imag @ B.T)
    Phi = torch.exp(L)
    if vp is not None and max(pk, pg) > 1e-8:
        xk = 2 * kk / kmax
        wk = np.where(xk < 1, 2 / 3 - xk ** 2 + xk ** 3 / 2, np.clip(2 - xk, 0, None) ** 3 / 6) / (2 / 3)
        r = np.clip(kg / gmax, 0, 1)
        Phi = Phi * _t(wk)[:, None] * _t((1 - r) ** 4 * (4 * r + 1))[None, :]
    tk, tg, ka, ga = _t(kk), _t(kg), _t(kap), _t(gam)
    hk, hg = kk[1] - kk[0], kg[1] - kg[0]
    wk, wg = torch.full_like(tk, hk), torch.full_like(tg, hg)
    for w in (wk, wg):
        w[0] *= 0.5
        w[-1] *= 0.5
    M = (tg * wg)[:, None] * (_j0m1(torch.outer(tg, ga)) + 1)
    two = (Phi[:, 1] - Phi[:, 0]) / hg ** 2
    va, vb = hg ** 2 / 12 * Phi[:, 0] - hg ** 4 / 120 * two, hg ** 4 / 480 * Phi[:, 0]
    Fr = torch.cat([Phi.real @ M, va.real[:, None], vb.real[:, None]], 1) * wk[:, None]
    Fi = torch.cat([Phi.imag @ M, va.imag[:, None], vb.imag[:, None]], 1) * wk[:, None]
    ph = torch.outer(ka, tk)
    P = (torch.cos(ph) @ Fr + torch.sin(ph) @ Fi) / (2 * math.pi ** 2)
    P3 = P[:, :-2] + P[:, -2:-1] + P[:, -1:] * (ga ** 2)[None, :]
    xw = np.linspace(-12.0 * sig, xi_max, n_wide)
    pw = _path(P3, ka, ga, xw, g_def)
    norm = np.trapezoid(pw, xw)
    pw = pw / norm
    mean = np.trapezoid(xw * pw, xw)
    var = np.trapezoid((xw - mean) ** 2 * pw, xw)
    skew = np.trapezoid((xw - mean) ** 3 * pw, xw) / var ** 1.5
    return dict(P=_path(P3, ka, ga, x, g_def) / norm, moments=np.array([mean, var, skew, norm]))


def _exact_sums(k, kap, w, chunk=1 << 25):
    """sum_c w (e^{i k kap} - 1 - i k kap) at the points k."""
    k, out = _t(k), []
    kap, w = _t(kap), _t(w)
    step = max(1, chunk // kap.numel())
    for a in range(0, k.numel(), step):
        c, s = _comp(torch.outer(k[a:a + step], kap))
        out.append(torch.complex(c @ w, s @ w))
    return torch.cat(out)


def _dlnmu(L, dk, x):
    """dP/dln mu of a log-CF on a uniform grid."""
    n = L.numel()
    wt = torch.full((n,), dk / math.pi, dtype=F64, device="cuda")
    wt[0] *= 0.5
    wt[-1] *= 0.5
    cf, kap = torch.exp(L) * wt, 1 - torch.exp(-0.5 * _t(x))
    out = []
    for a in range(0, kap.numel(), 512):
        ph = torch.outer(kap[a:a + 512], dk * torch.arange(n, dtype=F64, device="cuda"))
        out.append(torch.cos(ph) @ cf.real + torch.sin(ph) @ cf.imag)
    return (torch.cat(out) * (1 - kap) * 0.5).cpu().numpy()


def _exact_batch(b, x):
    P, vp = [], 0
    for i in range(b.n_inst):
        p0, p1, k = b.instance(i)
        if b.closure[i] == 0:
            c0, c1 = b.plane_cells[p0], b.plane_cells[p1]
            L = _exact_sums(k, b.kap[c0:c1], b.w[c0:c1]) - 0.5 * b.V[i] * _t(k) ** 2
        else:
            K, w, a = _t(b.vp_K[vp]), _t(b.vp_w[vp]), None
            vp += 1
            L = torch.zeros(k.size, dtype=torch.complex128, device="cuda")
            for p in range(p0, p1):
                S = _exact_sums(k, b.kap[b.plane_cells[p]:b.plane_cells[p + 1]], b.w[b.plane_cells[p]:b.plane_cells[p + 1]])
                z = _t(b.vp_D[p])[:, None] * S[None, :]
                mx = z.real.amax(0)
                a = (w[:, None] + 0j if a is None else K.T.to(torch.complex128) @ a) * torch.exp(z - mx)
                nrm = a.abs().amax(0)
                a = a / nrm
                L = L + S + mx + torch.log(nrm)
            L = L + torch.log(a.sum(0))
        P.append(_dlnmu(L, float(b.dk[i]), x))
    return np.array(P)


def _exact_nodes(t, x):
    """Every plane's H at its nodes, ln H minus its two-moment form interpolated onto the instance's k grid."""
    P = []
    for i in range(t.zs.size):
        p0, p1, nk, dk = int(t.inst_plane0[i]), int(t.inst_plane0[i + 1]), int(t.nk[i]), float(t.dk[i])
        k = dk * torch.arange(1, nk, dtype=F64, device="cuda")
        L = torch.zeros(nk, dtype=torch.complex128, device="cuda")
        for p in range(p0, p1):
            S, w = t.model.cells(t.bg, i, t.zl[p])
            m1, m2 = float(t.mu1[p]), float(t.mu2[p])
            form = lambda lq: (math.log(0.5 * m2) + 2 * lq - 0.5 * torch.log1p((torch.exp(lq) * m2 / (2 * m1)) ** 2),
                               torch.atan(torch.exp(lq) * m2 / (2 * m1)))
            ln = t.lnq0[p] + t.hq[p] * torch.arange(t.nq, dtype=F64, device="cuda")
            H, (b0, b1) = _exact_sums(torch.exp(ln).cpu().numpy(), S, w), form(ln)
            r = torch.stack([torch.log(H.abs()) - b0, torch.angle(-H) - b1])
            lq = torch.log(float(t.s[p]) * k)
            xx = (lq - t.lnq0[p]) / t.hq[p]
            j = xx.floor().long().clamp(1, t.nq - 3)
            u = xx - j
            v = (-u * (u - 1) * (u - 2) / 6 * r[:, j - 1] + (u + 1) * (u - 1) * (u - 2) / 2 * r[:, j]
                 - (u + 1) * u * (u - 2) / 2 * r[:, j + 1] + (u + 1) * u * (u - 1) / 6 * r[:, j + 2])
            v = torch.where(xx < 0, r[:, :1] * torch.exp((lq - t.lnq0[p]).clamp_max(0)), v)
            c0, c1 = form(lq)
            L[1:] += float(t.dz[p]) * -torch.exp(torch.complex(v[0] + c0, v[1] + c1))
        P.append(_dlnmu(L, dk, x))
    return np.array(P)


def _forward(m, X):
    """Activations and pre-activations of a member, its weights rounded to BF16 as the model has them."""
    acts, pre = [X.double()], []
    for i, (w, b) in enumerate(zip(m.W, m.b)):
        z = acts[-1] @ w.bfloat16().double() + b.double()
        pre.append(z)
        acts.append(z if i == len(m.W) - 1 else z * torch.sigmoid(z))
    return acts, pre


def _exact_train(case, seed):
    m, X, Y = _member(seed), _rows(case["batch"], seed), _targets(case["batch"], seed)
    acts, pre = _forward(m, X)
    d = acts[-1] - Y.double()
    dA, grads, W, B = 2 * d / d.numel(), [], list(m.W), list(m.b)

    def adamw(w, g, mo, v, t=m.step_count + 1, lr=1e-3):
        mo, v = 0.9 * mo.double() + 0.1 * g, 0.999 * v.double() + 0.001 * g * g
        return w.double() - lr * (mo / (1 - 0.9 ** t) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8) + 1e-4 * w.double())

    for i in range(len(m.W) - 1, -1, -1):
        if i < len(m.W) - 1:
            s = torch.sigmoid(pre[i])
            dA = dA * s * (1 + pre[i] * (1 - s))
        gW, gb = acts[i].T @ dA, dA.sum(0)
        grads.append([gW, gb])
        dA = dA @ m.W[i].bfloat16().double().T
        W[i], B[i] = adamw(m.W[i], gW, m.mW[i], m.vW[i]), adamw(m.b[i], gb, m.mb[i], m.vb[i])
    return dict(pred=acts[-1], loss=float((d * d).mean()), grads=grads, W=W, b=B)


def _exact_infer(case, seed):
    m, X = _member(seed), _rows(case["rows"], seed)
    return torch.cat([_forward(m, X[a:a + 65536])[0][-1] for a in range(0, X.shape[0], 65536)])


def _exact_cells(case, seed):
    """The lattices as plain histograms.  The compressed rows are fixed only up to a rotation of near-equal
    modes, so they have no value of their own."""
    objs, _ = _node(case, seed)
    log = lambda lo, hi, n: np.geomspace(lo, hi, n + 1)
    sl = lambda e: np.concatenate([-e[::-1], e])
    fk, fg, ck, cg = sl(log(1e-7, 30.0, 480)), log(1e-9, 30.0, 300), sl(log(1e-7, 30.0, 170)), log(1e-9, 30.0, 110)
    K, G, W = (np.concatenate([np.ravel(o[k]) for o in objs]) for k in "KGW")
    B = np.concatenate([np.full(np.size(o["K"]), o["beta"]) for o in objs])
    G = np.maximum(G, 1.0000001e-9)

    def where(v, e):
        i = np.searchsorted(e, v, side="right")
        i[v == e[-1]] -= 1
        return i - 1, (i >= 1) & (i < e.size)

    def hist(ek, eg, w):
        (i, a), (j, b) = where(K, ek), where(G, eg)
        ok, n = a & b, eg.size - 1
        return [np.bincount(i[ok] * n + j[ok], v[ok], (ek.size - 1) * n).reshape(-1, n) for v in w], ok

    (H0, H0k, H0g), ok = hist(fk, fg, [W, W * K, W * G])
    Hc, _ = hist(ck, cg, [W, W * B])
    return dict(H0=H0, H0k=H0k, H0g=H0g, Hc=np.array(Hc)[None], totals=np.array([W.sum(), W.sum() - W[ok].sum()]), rows=None)


def _exact_cosmo(p, z, M, zm):
    """Background, distances, growth, EH98 sigma(M), Sheth-Tormen and concentration tables."""
    h, Om, Ob, s8, ns, zeq, Ok, w0, wa = p.T[:, :, None]
    Or = Om / (1 + zeq)
    OL = 1 - Om - Ok - Or
    c, H0 = 299792.458, 100 * h
    de = lambda a: OL * np.exp(-3 * (1 + w0 + wa) * np.log(a) - 3 * wa * (1 - a))
    E = lambda zz: np.sqrt(Om * (1 + zz) ** 3 + Or * (1 + zz) ** 4 + Ok * (1 + zz) ** 2 + de(1 / (1 + zz)))
    xg, wg = np.polynomial.legendre.leggauss(16)
    edge = np.concatenate([[0.0], z])
    fine = np.concatenate([np.linspace(a, b, 9)[:-1] for a, b in zip(edge[:-1], edge[1:])] + [z[-1:]])
    mid, half = 0.5 * (fine[1:] + fine[:-1]), 0.5 * np.diff(fine)
    seg = sum(wg[q] / E((mid + half * xg[q])[None, :]) for q in range(16)) * half
    chi = np.cumsum(seg.reshape(p.shape[0], z.size, 8).sum(2), 1) * c / H0
    t = np.sqrt(np.abs(Ok)) * chi * H0 / c
    DM = chi * np.where(Ok > 0, np.sinh(t) / t, np.sin(t) / t)

    def rhs(x, y):
        a = np.exp(x)
        m, r, k, d = Om / a ** 3, Or / a ** 4, Ok / a ** 2, de(a)
        tot = m + r + k + d
        dh = -0.5 * (3 * m + 4 * r + 2 * k + 3 * (1 + w0 + wa * (1 - a)) * d) / tot
        return np.concatenate([y[:, 1:], -(2 + dh) * y[:, 1:] + 1.5 * m / tot * y[:, :1]], 1)

    x0, n = math.log(1e-6), 1 << 14
    xs = np.concatenate([x0 + (0 - x0) * np.arange(n) / n, -np.log1p(z), -np.log1p(zm), [0.0]])
    order = np.argsort(xs, kind="stable")
    y = np.concatenate([np.exp(x0) + 2 / 3 * Or / Om, np.full_like(Om, np.exp(x0))], 1)
    got, at = np.empty((xs.size, p.shape[0])), x0
    for o in order:
        hs = xs[o] - at
        if hs > 0:
            a = rhs(at, y)
            b = rhs(at + hs / 2, y + hs / 2 * a)
            d = rhs(at + hs / 2, y + hs / 2 * b)
            y = y + hs / 6 * (a + 2 * b + 2 * d + rhs(at + hs, y + hs * d))
            at = xs[o]
        got[o] = y[:, 0]
    D = (got[n:] / got[-1]).T
    # Eisenstein & Hu (1998) transfer function
    wm, wb, fb = Om * h * h, Ob * h * h, Ob / Om
    keq = H0 / c * np.sqrt(2 * Om) * np.sqrt(1 + zeq)
    silk = 0.0016 * wb ** 0.52 * wm ** 0.73 * (1 + (10.4 * wm) ** -0.95)
    a1 = (46.9 * wm) ** 0.67 * (1 + (32.1 * wm) ** -0.532)
    a2 = (12.0 * wm) ** 0.424 * (1 + (45.0 * wm) ** -0.582)
    b1, b2 = 0.944 / (1 + (458 * wm) ** -0.708), (0.395 * wm) ** -0.026
    ac, bc = a1 ** -fb * a2 ** -fb ** 3, 1 / (1 + b1 * ((1 - fb) ** b2 - 1))
    ss = 44.5 * np.log(9.83 / wm) / np.sqrt(1 + 10 * wb ** 0.75)
    zd = 1291 * wm ** 0.251 / (1 + 0.659 * wm ** 0.828) * (1 + 0.313 * wm ** -0.419 * (1 + 0.607 * wm ** 0.674) * wb ** (0.238 * wm ** 0.223))
    R, yy = 31.5 * wb * (2.7255 / 2.7) ** -4 / (zd / 1000), (1 + zeq) / (1 + zd)
    g2 = yy * (-6 * np.sqrt(1 + yy) + (2 + 3 * yy) * np.log((np.sqrt(1 + yy) + 1) / (np.sqrt(1 + yy) - 1)))
    ab = 2.07 * keq * ss * (1 + R) ** -0.75 * g2
    bb, bn = 0.5 + fb + (3 - 2 * fb) * np.sqrt(1 + (17.2 * wm) ** 2), 8.41 * wm ** 0.435
    k = np.logspace(-5, 3, 4000)[None, :]
    q = k / (13.41 * keq)

    def To(al, be):
        v = np.log(np.e + 1.8 * be * q)
        return v / (v + (14.2 / al + 386 / (1 + 69.9 * q ** 1.08)) * q * q)

    f = 1 / (1 + (k * ss / 5.4) ** 4)
    Tc = f * To(1.0, bc) + (1 - f) * To(ac, bc)
    xx = k * ss / np.cbrt(1 + (bn / (k * ss)) ** 3)
    Tb = (To(1.0, 1.0) / (1 + (k * ss / 5.2) ** 2) + ab / (1 + (bb / (k * ss)) ** 3) * np.exp(-(k / silk) ** 1.4)) * np.sin(xx) / xx
    kP = k * k * k ** ns * (fb * Tb + (1 - fb) * Tc) ** 2
    r8 = k * 8 / h
    A = s8[:, 0] / np.sqrt(np.trapezoid(kP * (3 * (np.sin(r8) - r8 * np.cos(r8)) / r8 ** 3) ** 2, k, axis=1) / (2 * math.pi ** 2))
    rho = (Om * 2.77536627e11 * h * h)[:, 0]
    Mn = np.logspace(4, 17, 500)
    lns = np.empty((p.shape[0], 500))
    for i in range(500):
        W = 1 / (1 + (0.43 * k * np.cbrt(3 * Mn[i] / (4 * math.pi * rho))[:, None]) ** 6)
        lns[:, i] = np.log(A * np.sqrt(np.trapezoid(kP * W * W, k, axis=1) / (2 * math.pi ** 2)))
    # the not-a-knot spline of ln sigma in ln M (uniform nodes), its value and slope
    u, eps = (np.log(M) - math.log(1e4)) / math.log(1e13), 1.0 / 499
    i = np.minimum((u / eps).astype(int), 498)
    Sp = lambda s: _spline(500, s).cpu().numpy()
    left, right = np.linspace(0, 1, 500)[i], np.linspace(0, 1, 500)[i + 1]
    quarter = [Sp(left + (right - left) * v) @ lns.T for v in (0.0, 1 / 3, 2 / 3, 1.0 - 1e-15)]
    v = (u - left) / (right - left)
    lag, dlag = _cubic(v)
    lnsig = sum(l[:, None] * y_ for l, y_ in zip(lag, quarter)).T
    dls = (sum(l[:, None] * y_ for l, y_ in zip(dlag, quarter)) / (eps * math.log(1e13))).T
    sig = np.exp(lnsig)
    Dm = D[:, z.size:z.size + zm.size]
    nu = 0.8 * (1.686 / (sig[:, None, :] * Dm[:, :, None])) ** 2
    Ast = 1 / (1 + 2 ** -0.3 * math.gamma(0.2) / math.sqrt(math.pi))
    dn = (rho[:, None] / M)[:, None, :] * Ast * (1 + nu ** -0.3) * np.sqrt(nu / (2 * math.pi)) * np.exp(-nu / 2) * (-2 * dls[:, None, :])
    ap = 1 + np.minimum(zm, 7.0)
    poly = 4.135 - 0.564 * ap - 0.210 * ap ** 2 + 0.0557 * ap ** 3 - 0.00348 * ap ** 4
    qc = 1.686 / (sig[:, None, :] * poly[None, :, None])
    ap = ap[None, :, None]
    c0, be, g1, g2 = 3.395 * ap ** -0.215, 0.307 * ap ** 0.540, 0.628 * ap ** -0.047, 0.317 * ap ** -0.893
    conc = c0 * qc ** -g1 * (1 + qc ** (1 / be)) ** (-be * (g2 - g1))
    return dict(E=E(z[None, :]), chi=chi, DM=DM, D=D[:, :z.size], sigmaM=sig, dlnsig=dls, dndlnM=dn, conc=conc)


def _cubic(v):
    """Lagrange basis on 0, 1/3, 2/3, 1 at v, and its derivative."""
    n = (0.0, 1 / 3, 2 / 3, 1.0)
    val, der = [], []
    for a in range(4):
        o = [n[b] for b in range(4) if b != a]
        s = np.prod([n[a] - x for x in o])
        val.append((v - o[0]) * (v - o[1]) * (v - o[2]) / s)
        der.append(((v - o[0]) * (v - o[1]) + (v - o[0]) * (v - o[2]) + (v - o[1]) * (v - o[2])) / s)
    return val, der


def exact(case, seed):
    kind = case["kind"]
    if kind in ("pdf", "dropin"):
        return _exact_pdf(*_population(case, seed), _x(case))
    if kind == "few":
        return _exact_pdf(_few(case, seed), None, _x(case))
    if kind == "vp":
        pop, f, d = _vp(case, seed)
        return _exact_pdf(pop, f, _x(case), vp=d, n_wide=4000)
    if kind == "sweep":
        kap, w, kk = _sweep(case, seed)
        return _exact_sums(kk, kap, w).cpu().numpy()
    if kind == "batch":
        return _exact_batch(_batch(case, seed), _x(case))
    if kind == "nodes":
        return _exact_nodes(_tables(case, seed), _x(case))
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "infer":
        return _exact_infer(case, seed)
    if kind == "cells":
        return _exact_cells(case, seed)
    return _exact_cosmo(*_cosmo(case, seed))
