"""The work that is timed: what a user has the framework do, through its public entry points.

Five kinds of call, each over its range of sizes, axis lengths (powers of two, products of
2, 3, 5 and 7, odd ones) and both precisions (float64, and float32 grids with float64 sums):

  ev       one energy + potential evaluation of a total functional on a density, the call
           that every density optimisation and every OE-SCF step is made of
  adjoint  the differentiable total energy forward and backward (potential fitting)
  ionstep  what a molecular-dynamics or relaxation step pays besides the density solve:
           ions moved, local pseudopotential and Ewald sum rebuilt, energy, potential, forces
  batch    one evaluation of many small independent systems in one launch
  opt      a few L-BFGS iterations of the density optimiser

``exact`` restates each call's mathematics in float64 with torch alone (smooth PME with the
same B-splines, the same kernel tables and k_F nodes).
"""
import math

import numpy as np
import torch

import dftpy_gb300 as D
from dftpy_gb300.autograd import total_energy
from dftpy_gb300.batch import BatchEvaluator

A_FCC = 7.6          # Bohr, conventional fcc cell of 4 atoms
DENSITY_AMP = 0.6    # log-amplitude of the trial density: max/min about 3.3, as in a bulk metal
AB_WGC = ((5 + 5 ** 0.5) / 6, (5 - 5 ** 0.5) / 6)
Z = {"Al": 3.0, "Mg": 2.0}
RC = {"Al": 1.0, "Mg": 1.2}
ORDER = 10           # B-spline order of the smooth PME (the framework's default)
FRAC = np.array([[0.0, 0.0, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5], [0.5, 0.5, 0.0]])


def listed():
    return [
        # a 4-atom cell: the smallest real calculation, all latency
        dict(name="ev_tfvw_f64_32", kind="ev", kedf="TFVW", dtype="f64", n0=32, n1=32, n2=32, nsp=0, interp=""),
        # 256 atoms with Wang-Teter, the ordinary production functional, in float64
        dict(name="ev_wt_f64_128", kind="ev", kedf="WT", dtype="f64", n0=128, n1=128, n2=128, nsp=0, interp=""),
        # the same functional in float32 on a cell whose axes differ (one of them odd)
        dict(name="ev_wt_f32_ragged", kind="ev", kedf="WT", dtype="f32", n0=150, n1=160, n2=135, nsp=0, interp=""),
        # 2048 atoms with the density-dependent kernel on 64 nodes: the benchmark's configuration
        dict(name="ev_lwt_f32_256", kind="ev", kedf="LWT", dtype="f32", n0=256, n1=256, n2=256, nsp=64,
             interp="linear"),
        # the same kernel on a grid that an energy cutoff gives (not powers of two)
        dict(name="ev_lwt_f32_ragged", kind="ev", kedf="LWT", dtype="f32", n0=96, n1=108, n2=120, nsp=64,
             interp="linear"),
        # the continuously differentiable interpolation, which ground states need
        dict(name="ev_lwt_hermite_f32_128", kind="ev", kedf="LWT", dtype="f32", n0=128, n1=128, n2=128, nsp=64,
             interp="hermite"),
        # float64 reference evaluations of the density-dependent kernel
        dict(name="ev_lwt_f64_ragged", kind="ev", kedf="LWT", dtype="f64", n0=64, n1=72, n2=80, nsp=64,
             interp="linear"),
        # pseudopotential fitting on a 500-atom two-species alloy: forward and backward
        dict(name="adjoint_wt_f32_160", kind="adjoint", dtype="f32", n0=160, n1=160, n2=160),
        # the geometry part of an MD step: 256 atoms in float64, 2048 in float32
        dict(name="ionstep_f64_128", kind="ionstep", dtype="f64", n0=128, n1=128, n2=128),
        dict(name="ionstep_f32_256", kind="ionstep", dtype="f32", n0=256, n1=256, n2=256),
        # 16 small cells of uneven size together, as a high-throughput screening does
        dict(name="batch_f32_16", kind="batch", dtype="f32", systems=16),
        # the optimiser itself (directions, rotations, line searches) on 32 atoms
        dict(name="opt_lbfgs_wt_f64_60", kind="opt", dtype="f64", n0=60, n1=60, n2=60),
    ]


def _axis(rng, lo, hi):
    """An axis length an energy cutoff gives: a product of 2, 3, 5, 7, log-uniform in [lo, hi]."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    n = max(lo, min(hi, int(round(want))))
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n = n - 1 if n > lo else hi


def draw(rng):
    kind = rng.choice(["ev", "ev", "ev", "ev", "adjoint", "ionstep", "batch", "opt"])
    dtype = rng.choice(["f64", "f32"])
    if kind == "batch":
        return dict(kind=kind, dtype=dtype, systems=rng.randint(2, 20 if dtype == "f32" else 8))
    kedf = rng.choice(["TFVW", "WT", "LWT", "LWT"]) if kind == "ev" else ""
    lo, hi = 20, 180
    if kind == "opt":
        lo, hi = 20, 72
    elif dtype == "f64":
        hi = 80 if kedf == "LWT" else 128
    n = [_axis(rng, lo, hi) for _ in range(3)]
    if kind == "ev" and rng.random() < 0.3:  # grids are often chosen as powers of two
        n = [rng.choice([32, 64, 128, 256]) if dtype == "f32" else rng.choice([32, 64]) for _ in range(3)]
    c = dict(kind=kind, dtype=dtype, n0=n[0], n1=n[1], n2=n[2])
    if kind == "ev":
        c.update(kedf=kedf, nsp=0, interp="")
        if kedf == "LWT":
            c.update(nsp=rng.randint(8, 64), interp=rng.choice(["linear", "hermite"]))
    return c


# ------------------------------------------------------------------ inputs
def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _table(sp, npts=4096, gmax=40.0):
    g = np.linspace(0.0, gmax, npts)
    e = np.exp(-g[1:] ** 2 * RC[sp] ** 2 / 4.0)
    v = np.empty(npts)
    v[1:] = -4.0 * np.pi * Z[sp] / g[1:] ** 2 * e + 15.0 * e
    v[0] = 15.0 + np.pi * Z[sp] * RC[sp] ** 2
    return g, v


def _crystal(nr, rng, a=A_FCC, sigma=0.1, reps=None):
    reps = np.array(reps if reps else [max(1, round(n / 32)) for n in nr])
    cells = np.stack(np.meshgrid(*[np.arange(r) for r in reps], indexing="ij"), -1).reshape(-1, 1, 3)
    pos = ((cells + FRAC[None]).reshape(-1, 3)) * a
    return np.diag(reps * float(a)), pos + rng.normal(0.0, sigma, pos.shape)


def _density(nr, volume, nelec, rng, amp=DENSITY_AMP):
    """rho0 exp(s) with s a sum of low plane waves: positive, smooth, periodic; float64."""
    x = [torch.arange(n, dtype=torch.float64, device="cuda") * (2 * math.pi / n) for n in nr]
    s = torch.zeros(tuple(nr), dtype=torch.float64, device="cuda")
    for _ in range(12):
        k, ph = rng.integers(-3, 4, size=3), rng.uniform(0, 2 * math.pi)
        s += torch.cos((k[0] * x[0] + ph)[:, None, None] + (k[1] * x[1])[None, :, None] + (k[2] * x[2])[None, None, :])
    s *= amp / max(1e-12, float(s.abs().max()))
    rho = torch.exp(s)
    return rho * (nelec / (float(rho.sum()) * volume / rho.numel()))


def _system(case, seed):
    """Geometry, species, tables and density of a case, without the framework."""
    rng = np.random.default_rng(seed)
    nr = (case["n0"], case["n1"], case["n2"])
    kind = case["kind"]
    if kind == "adjoint":
        lat, pos = _crystal(nr, rng, a=9.0, sigma=0.3)
        sym = ["Al" if i % 2 == 0 else "Mg" for i in range(len(pos))]
        tables = {s: _table(s, npts=256) for s in ("Al", "Mg")}
    else:
        lat, pos = _crystal(nr, rng)
        sym = ["Al"] * len(pos)
        tables = {"Al": _table("Al")}
    q = np.array([Z[s] for s in sym])
    rho = _density(nr, abs(np.linalg.det(lat)), q.sum(), rng).to(_dtype(case))
    return dict(nr=nr, lat=lat, pos=pos, sym=sym, q=q, tables=tables, rho=rho)


def _batch_systems(case, seed):
    rng, size = np.random.default_rng(seed), np.random.default_rng(case["systems"])
    out = []
    for _ in range(case["systems"]):
        r, n = int(size.integers(1, 4)), int(size.choice([48, 64, 72, 80, 96]))
        lat, pos = _crystal((n,) * 3, rng, a=float(rng.uniform(7.3, 7.9)), reps=(r, r, r))
        q = np.full(len(pos), 3.0)
        rho = _density((n,) * 3, abs(np.linalg.det(lat)), q.sum(), rng).to(_dtype(case))
        out.append(dict(nr=(n,) * 3, lat=lat, pos=pos, sym=["Al"] * len(pos), q=q, tables={"Al": _table("Al")}, rho=rho))
    return out


def _kedf(case):
    if case.get("kedf") == "LWT":
        return D.Functional(type="KEDF", name="LWT", nsp=case["nsp"], kdd=3, interp=case["interp"], alpha=AB_WGC[0],
                            beta=AB_WGC[1])
    return D.Functional(type="KEDF", name=case["kedf"])


def _total(s, kedf):
    grid = D.DirectGrid(s["lat"], s["nr"])
    ions = D.Ions(symbols=list(s["sym"]), positions=s["pos"], cell=s["lat"])
    pp_list = {k: D.functional.RECPOT(r=g, v=v, zval=Z[k]) for k, (g, v) in s["tables"].items()}
    pp = D.LocalPseudo(grid=grid, ions=ions, PP_list=pp_list, PME=True)
    total = D.TotalFunctional(KineticEnergyFunctional=kedf, XCFunctional=D.Functional(type="XC", name="LDA"),
                              HARTREE=D.Functional(type="HARTREE"), PSEUDO=pp)
    return grid, pp, total


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems = _batch_systems(case, seed)
        parts = [_total(s, D.Functional(type="KEDF", name="TFVW")) for s in systems]
        rhos = [D.DirectField(g, data=s["rho"], dtype=_dtype(case)) for s, (g, _, _) in zip(systems, parts)]
        ev = BatchEvaluator([t for _, _, t in parts], [g for g, _, _ in parts], dtype=_dtype(case))
        return dict(kind=kind, ev=ev, rhos=rhos, keep=parts)
    s = _system(case, seed)
    if kind == "ev":
        grid, _, total = _total(s, _kedf(case))
        return dict(kind=kind, total=total, rho=D.DirectField(grid, data=s["rho"], dtype=_dtype(case)))
    if kind == "adjoint":
        _, pp, total = _total(s, D.Functional(type="KEDF", name="WT"))
        tables = torch.tensor(np.concatenate([s["tables"][k][1] for k in pp.species_keys]), requires_grad=True)
        return dict(kind=kind, total=total, rho=s["rho"].requires_grad_(True), tables=tables,
                    pos=torch.tensor(s["pos"], requires_grad=True))
    if kind == "ionstep":
        grid, pp, total = _total(s, D.Functional(type="KEDF", name="TFVW"))
        return dict(kind=kind, total=total, pp=pp, pos=s["pos"],
                    rho=D.DirectField(grid, data=s["rho"], dtype=_dtype(case)))
    grid, _, total = _total(s, D.Functional(type="KEDF", name="WT"))
    opt = D.Optimization(optimization_method="LBFGS", EnergyEvaluator=total,
                         optimization_options={"maxiter": 6, "econv": 1e-14})
    return dict(kind=kind, opt=opt, rho=D.DirectField(grid, data=s["rho"], dtype=_dtype(case)))


def run(state):
    kind = state["kind"]
    if kind == "ev":
        out = state["total"](state["rho"], calcType={"E", "V"})
        return {"energy": out.energy, "potential": out.potential}
    if kind == "adjoint":
        E = total_energy(state["total"], state["rho"], state["pos"], state["tables"])
        g = torch.autograd.grad(E, (state["rho"], state["pos"], state["tables"]))
        return {"energy": E.detach(), "rho": g[0], "positions": g[1], "tables": g[2]}
    if kind == "ionstep":
        state["pp"].set_positions(state["pos"])
        out = state["total"](state["rho"], calcType={"E", "V"})
        return {"energy": out.energy, "potential": out.potential, "forces": state["total"].get_forces(state["rho"])}
    if kind == "batch":
        res = state["ev"](state["rhos"])
        return {"energy": np.array([r.energy for r in res]), "potential": [r.potential for r in res]}
    rho = state["opt"].optimize_rho(guess_rho=state["rho"])
    f = state["opt"].functional
    return {"energy": f.energy, "rho": rho, "potential": f.potential}


# -------------------------------------------------------------------- work
def work(case):
    """Density and pseudopotential read, potential written; 2.5 N log2 N per real transform."""
    s = 8 if case["dtype"] == "f64" else 4
    kind = case["kind"]
    if kind == "batch":
        N = case["systems"] * 72 ** 3
        return {"bytes": 3.0 * s * N, "flops": 4 * 2.5 * N * 3 * math.log2(72)}
    N = case["n0"] * case["n1"] * case["n2"]
    fft = 2.5 * N * math.log2(N)
    if kind == "ev":
        nfft = {"TFVW": 4, "WT": 6, "LWT": 6}[case["kedf"]]
        if case["kedf"] == "LWT":
            nfft += case["nsp"] * (4 if case["interp"] == "hermite" else 3)
        return {"bytes": 3.0 * s * N, "flops": nfft * fft}
    if kind == "adjoint":
        return {"bytes": 4.0 * s * N, "flops": 14 * fft}
    if kind == "ionstep":
        return {"bytes": 2.0 * s * N, "flops": 10 * fft}
    return {"bytes": 3.0 * s * N, "flops": 12 * 6 * fft}


# ------------------------------------------------- the same in 64 bits, torch only
class _Grid:
    def __init__(self, lat, nr):
        self.nr, self.N, self.V = nr, nr[0] * nr[1] * nr[2], abs(np.linalg.det(lat))
        self.dV, self.lat = self.V / self.N, lat
        b = torch.tensor(2 * math.pi * np.linalg.inv(lat).T, dtype=torch.float64, device="cuda")
        f = [torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda") for n in nr[:2]]
        f.append(torch.arange(nr[2] // 2 + 1, dtype=torch.float64, device="cuda"))
        g = [f[0][:, None, None] * b[0, c] + f[1][None, :, None] * b[1, c] + f[2][None, None, :] * b[2, c] for c in range(3)]
        self.gg = g[0] * g[0] + g[1] * g[1] + g[2] * g[2]
        self.q = self.gg.sqrt()
        self.inv = torch.where(self.gg > 0, 1.0 / self.gg.clamp_min(1e-300), torch.zeros_like(self.gg))

    def fft(self, x):
        return torch.fft.rfftn(x)

    def ifft(self, X):
        return torch.fft.irfftn(X, s=self.nr)


def _spline(x, y):
    """Not-a-knot cubic spline on a uniform grid: coefficients (n - 1, 4)."""
    n, h = len(x), (x[-1] - x[0]) / (len(x) - 1)
    r = np.zeros(n)
    r[1:-1] = 6.0 * (y[:-2] - 2.0 * y[1:-1] + y[2:]) / (h * h)
    M = np.zeros(n)
    M[1], M[-2] = r[1] / 6.0, r[-2] / 6.0
    rhs = r[2:-2].copy()
    rhs[0] -= M[1]
    rhs[-1] -= M[-2]
    c, d = [0.0] * len(rhs), rhs.tolist()  # Thomas with 1, 4, 1
    c[0], d[0] = 0.25, d[0] / 4.0
    for i in range(1, len(rhs)):
        w = 1.0 / (4.0 - c[i - 1])
        c[i], d[i] = w, (d[i] - d[i - 1]) * w
    for i in range(len(rhs) - 2, -1, -1):
        d[i] -= c[i] * d[i + 1]
    M[2:-2] = d
    M[0], M[-1] = 2 * M[1] - M[2], 2 * M[-2] - M[-3]
    co = np.empty((n - 1, 4))
    co[:, 0] = y[:-1]
    co[:, 1] = (y[1:] - y[:-1]) / h - h * (2 * M[:-1] + M[1:]) / 6.0
    co[:, 2] = M[:-1] / 2.0
    co[:, 3] = (M[1:] - M[:-1]) / (6.0 * h)
    return co


def _spline_matrix(x):
    """The same spline's coefficients as a linear map of its values, (n - 1, 4, n)."""
    return np.stack([_spline(x, e) for e in np.eye(len(x))], -1)


def _eval(co, x0, h, q):
    i = ((q - x0) / h).floor().clamp(0, co.shape[0] - 1).long()
    u = q - (x0 + i.double() * h)
    c = co[i]
    return c[..., 0] + u * (c[..., 1] + u * (c[..., 2] + u * c[..., 3]))


def _lindhard(eta, lbda=1.0):
    """1 / Lindhard(eta) - 3 eta^2 - lbda, with the usual large-eta expansion above 3.65."""
    e = torch.where((eta - 1.0).abs() < 1e-11, torch.full_like(eta, 0.5), eta).clamp_min(1e-10)
    out = 1.0 / (0.5 + 0.25 * (1.0 - e * e) * torch.log((1.0 + e) / (1.0 - e).abs()) / e) - 3.0 * e * e - lbda
    out = torch.where((eta - 1.0).abs() < 1e-11, torch.full_like(eta, 2.0 - lbda - 3.0), out)
    out = torch.where(eta < 1e-10, 1.0 - lbda + eta * eta * (1.0 / 3.0 - 3.0), out)
    c = [-0.13714285714285712, -6.4e-2, -3.77825602968460128e-2, -2.51824061652633074e-2, -1.80879839616166146e-2,
         -1.36715733124818332e-2, -1.07236045520990083e-2, -8.65192783339199453e-3, -7.1372762502456763e-3,
         -5.9945117538835746e-3, -5.10997527675418131e-3, -4.41060829979912465e-3, -3.84763737842981233e-3,
         -3.38745061493813488e-3, -3.00624946457977689e-3]
    i2, acc = 1.0 / (e * e), torch.zeros_like(e)
    for v in reversed(c):
        acc = i2 * (v + acc)
    return torch.where(eta > 3.65, -lbda - 0.6 + acc, out)


def _mn(x, order):
    """B-spline values M_order(x + n - 1), n = 0..order (column n), recursively."""
    M = [torch.zeros_like(x) for _ in range(order + 1)]
    M[1], M[2] = x, 1.0 - x
    for i in range(3, order + 1):
        for n in range(i, 0, -1):
            M[n] = ((x + n - 1) * M[n] + (i - n + 1 - x) * M[n - 1]) / (i - 1)
    return torch.stack(M[1:], -1)


def _spread(G, pos, w):
    """Charges w on the PME mesh, differentiable in pos."""
    inv = torch.tensor(np.linalg.inv(G.lat), dtype=torch.float64, device="cuda")
    fr = pos @ inv
    fr = fr - fr.detach().floor()
    wt, idx = [], []
    for d in range(3):
        u = fr[:, d] * G.nr[d]
        fl = u.detach().floor()
        wt.append(_mn(u - fl, ORDER))
        idx.append((fl.long()[:, None] + 1 - torch.arange(ORDER, device="cuda")) % G.nr[d])
    val = wt[0][:, :, None, None] * wt[1][:, None, :, None] * wt[2][:, None, None, :] * w[:, None, None, None]
    lin = (idx[0][:, :, None, None] * G.nr[1] + idx[1][:, None, :, None]) * G.nr[2] + idx[2][:, None, None, :]
    Q = torch.zeros(G.N, dtype=torch.float64, device="cuda")
    return Q.index_add(0, lin.reshape(-1), val.reshape(-1)).reshape(G.nr)


def _euler(G):
    """Product of the B-spline Euler factors of the three axes on the half grid."""
    M = _mn(torch.ones(1, dtype=torch.float64), ORDER)[0].numpy()
    b = []
    for d, m in enumerate((G.nr[0], G.nr[1], G.nr[2] // 2 + 1)):
        x = 2 * np.pi * np.arange(m) / G.nr[d]
        f = sum(M[k - 1] * np.exp(-1j * k * x) for k in range(1, ORDER))
        b.append(torch.tensor(np.exp(-1j * (ORDER - 1) * x) / f, device="cuda"))
    return b[0][:, None, None] * b[1][None, :, None] * b[2][None, None, :]


def _vline(G, g, v, matrix=None):
    """Radial potential on the half grid: the spline of the table, a quartic below its first point."""
    v = v if torch.is_tensor(v) else torch.tensor(v, device="cuda")
    if matrix is None:
        co = torch.tensor(_spline(g[1:], v.detach().cpu().numpy()[1:]), device="cuda")
    else:
        co = matrix @ v[1:]
    h = g[1] - g[0]
    out = _eval(co, g[1], h, G.q)
    f = [v[2], v[1], v[0], v[1], v[2]]
    t = [2 * f[0] - 16 * f[1] + 16 * f[3] - 2 * f[4], -f[0] + 16 * f[1] - 30 * f[2] + 16 * f[3] - f[4],
         -2 * f[0] + 4 * f[1] - 4 * f[3] + 2 * f[4], f[0] - 4 * f[1] + 6 * f[2] - 4 * f[3] + f[4]]
    x = G.q / h
    low = f[2] + x * (t[0] + x * (t[1] + x * (t[2] + x * t[3]))) / 24.0
    out = torch.where(G.q < g[1], low, out)
    return torch.where(G.q < g[-1], out, torch.zeros_like(out))


def _vloc(G, s, pos, tables, matrix=None):
    X = 0
    for k, (g, _) in s["tables"].items():
        sel = torch.tensor([i for i, e in enumerate(s["sym"]) if e == k], device="cuda")
        X = X + _vline(G, g, tables[k], matrix) * G.fft(_spread(G, pos[sel], torch.ones(len(sel), dtype=torch.float64, device="cuda")))
    return G.ifft(X * _euler(G)) * (G.N / G.V)


def _ewald(G, s, pos):
    """Ewald energy (PME reciprocal part), differentiable in pos."""
    q = torch.tensor(s["q"], device="cuda")
    L = np.sqrt((G.lat ** 2).sum(1))
    sp = max(0.5 * (L[d] / G.nr[d] + L[d] / (G.nr[d] - 1)) for d in range(3))
    gmax, q2, eta = math.pi / sp, float((q * q).sum()), 1.6
    while 4 * math.pi * len(q) * q2 * math.sqrt(eta / math.pi) * math.erfc(gmax / 2 * math.sqrt(1 / eta)) >= 1e-8:
        eta -= 0.01
    lo, hi = 0.0, 10.0
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if math.erfc(mid) > 1e-8 / 3 else (lo, mid)
    rc = hi / math.sqrt(eta)
    E = -math.sqrt(eta / math.pi) * q2 - math.pi / (2 * eta * G.V) * float(q.sum()) ** 2
    lat = torch.tensor(G.lat, device="cuda")
    R = pos - torch.floor(pos.detach() @ torch.linalg.inv(lat)) @ lat
    K = [int(math.ceil(rc / L[d])) for d in range(3)]
    for n0 in range(-K[0], K[0] + 1):
        for n1 in range(-K[1], K[1] + 1):
            for n2 in range(-K[2], K[2] + 1):
                t = torch.tensor([n0, n1, n2], dtype=torch.float64, device="cuda") @ lat
                d = (R[:, None, :] - (R + t)[None, :, :])
                i, j = torch.nonzero(((d.detach() ** 2).sum(-1) < rc * rc) & ((d.detach() ** 2).sum(-1) > 1e-6), as_tuple=True)
                r = (R[i] - R[j] - t).norm(dim=-1)
                E = E + 0.5 * (q[i] * q[j] * torch.erfc(math.sqrt(eta) * r) / r).sum()
    S = G.fft(_spread(G, pos, q)) * _euler(G)
    w = torch.full((G.nr[2] // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    w[0] = 1.0
    if G.nr[2] % 2 == 0:
        w[-1] = 1.0
    return E + 2 * math.pi / G.V * (w * (S.real ** 2 + S.imag ** 2) * torch.exp(-G.gg / (4 * eta)) * G.inv).sum()


def _local(G, rho, vloc):
    """TF + vW + LDA + Hartree + local pseudopotential: energy and potential."""
    p2 = 3.0 * math.pi ** 2
    c = rho.pow(1.0 / 3.0)
    E = (0.3 * p2 ** (2 / 3) * c ** 5).sum()
    V = 0.5 * p2 ** (2 / 3) * c * c
    s = rho.sqrt()
    w = 0.5 * G.ifft(G.gg * G.fft(s)) / s
    E, V = E + (rho * w).sum(), V + w
    h = G.ifft(4 * math.pi * G.inv * G.fft(rho))
    E, V = E + 0.5 * (rho * h).sum(), V + h
    rs = (3 / (4 * math.pi)) ** (1 / 3) / c
    l, r2 = rs.log(), rs.sqrt()
    a, b, cc, d, ga, b1, b2 = 0.0311, -0.048, 0.0020, -0.0116, -0.1423, 1.0529, 0.3334
    den = 1 + b1 * r2 + b2 * rs
    ex = -0.75 * (3 / math.pi) ** (1 / 3) * c + torch.where(rs < 1, a * l + b + cc * rs * l + d * rs, ga / den)
    vx = -(3 / math.pi) ** (1 / 3) * c + torch.where(
        rs < 1, l * (a + 2 / 3 * cc * rs) + b - a / 3 + (2 * d - cc) / 3 * rs,
        (ga + 7 / 6 * ga * b1 * r2 + 4 / 3 * ga * b2 * rs) / den ** 2)
    return (E + (ex * rho).sum() + (vloc * rho).sum()) * G.dV, V + vx + vloc


def _wt(G, rho):
    r0 = float(rho.mean())
    K = _lindhard(G.q / (2 * (3 * r0 * math.pi ** 2) ** (1 / 3))) * (0.8 * 0.3 * (3 * math.pi ** 2) ** (2 / 3))
    rb = rho ** (5 / 6)
    v = G.ifft(K * G.fft(rb))
    return (rb * v).sum() * G.dV, 5 / 3 * rb / rho * v


def _lwt(G, rho, nsp, hermite):
    """The k_F-node kernel: nodes spread evenly over the density's own k_F range."""
    al, be = AB_WGC
    kf = 2.0 * (3 * math.pi ** 2 * rho).pow(1 / 3)
    lo, hi = float(kf.min()), float(kf.max())
    k = lo + (hi - lo) / (nsp - 1) * np.arange(nsp)
    eta = np.linspace(0, 50.0, 50000)
    y = _lindhard(torch.tensor(eta)).numpy() * (0.8 * 0.3 * (3 * math.pi ** 2) ** (2 / 3))
    c0 = _spline(eta, y)
    dy = np.append(c0[:, 1], 0.0)
    h = eta[1]
    dy[-1] = c0[-1, 1] + h * (2 * c0[-1, 2] + 3 * h * c0[-1, 3])
    c1 = _spline(eta, -eta * dy)
    co, cd = torch.tensor(c0, device="cuda"), torch.tensor(c1, device="cuda")

    def kernel(c, kj):
        e = (G.q / kj).clamp_max(50.0)
        out = _eval(c, 0.0, h, e)
        out[0, 0, 0] = 0.0
        return out

    kn = torch.tensor(k, device="cuda")
    i = (torch.searchsorted(kn, kf) - 1).clamp(0, nsp - 2)
    inside = (kf > lo) & (kf < hi)
    dk = (kn[i + 1] - kn[i])
    t = (kf - kn[i]) / dk
    rA, rB = rho ** al, rho ** be
    B = G.fft(rB)
    p1, p3, p2 = torch.zeros_like(rho), torch.zeros_like(rho), torch.zeros_like(B)
    zero = torch.zeros_like(rho)
    for j in range(nsp):
        K, KD = kernel(co, k[j]), kernel(cd, k[j]) / k[j]
        P, M = G.ifft(K * B), G.ifft(KD * B)
        a, b = inside & (i == j), inside & (i == j - 1)
        if not hermite:
            w = torch.where(a, 1 - t, torch.where(b, t, zero))
            p1 += w * P
            p3 += w * M
            p2 += K * G.fft(rA * w)
        else:
            h00, h10 = 2 * t ** 3 - 3 * t ** 2 + 1, t ** 3 - 2 * t ** 2 + t
            h01, h11 = 1 - h00, t ** 3 - t ** 2
            w, wd = torch.where(a, h00, torch.where(b, h01, zero)), dk * torch.where(a, h10, torch.where(b, h11, zero))
            d00 = (6 * t * t - 6 * t) / dk
            v, vd = torch.where(a, d00, torch.where(b, -d00, zero)), torch.where(
                a, 3 * t * t - 4 * t + 1, torch.where(b, 3 * t * t - 2 * t, zero))
            p1 += w * P + wd * M
            p3 += v * P + vd * M
            p2 += K * G.fft(rA * w) + KD * G.fft(rA * wd)
    pot2 = G.ifft(p2)
    return (rA * p1).sum() * G.dV, al * rA / rho * p1 + be * rB / rho * pot2 + kf / 3 * rA / rho * p3


def _exact_ev(s, kedf, case):
    G = _Grid(s["lat"], s["nr"])
    pos = torch.tensor(s["pos"], device="cuda")
    tables = {k: v for k, (_, v) in s["tables"].items()}
    rho = s["rho"].detach().double()
    E, V = _local(G, rho, _vloc(G, s, pos, tables))
    if kedf in ("WT", "LWT"):
        e, v = _wt(G, rho) if kedf == "WT" else _lwt(G, rho, case["nsp"], case["interp"] == "hermite")
        E, V = E + e, V + v
    return float(E + _ewald(G, s, pos)), V


def exact(case, seed):
    kind = case["kind"]
    if kind == "opt":
        return None
    if kind == "batch":
        got = [_exact_ev(s, "TFVW", case) for s in _batch_systems(case, seed)]
        return {"energy": np.array([e for e, _ in got]), "potential": [v for _, v in got]}
    s = _system(case, seed)
    if kind == "ev":
        E, V = _exact_ev(s, case["kedf"], case)
        return {"energy": E, "potential": V}
    G = _Grid(s["lat"], s["nr"])
    rho = s["rho"].detach().double()
    pos = torch.tensor(s["pos"], device="cuda", requires_grad=True)
    if kind == "ionstep":
        tables = {k: v for k, (_, v) in s["tables"].items()}
        v = _vloc(G, s, pos, tables)
        ion = (v * rho).sum() * G.dV + _ewald(G, s, pos)
        F = -torch.autograd.grad(ion, pos)[0]
        E, V = _local(G, rho, v.detach())
        return {"energy": float(E + _ewald(G, s, pos.detach())), "potential": V, "forces": F}
    keys = sorted(s["tables"])
    flat = {k: torch.tensor(s["tables"][k][1], device="cuda", requires_grad=True) for k in keys}
    matrix = torch.tensor(_spline_matrix(s["tables"][keys[0]][0][1:]), device="cuda")
    v = _vloc(G, s, pos, flat, matrix)
    ion = (v * rho).sum() * G.dV + _ewald(G, s, pos)
    g = torch.autograd.grad(ion, [pos] + [flat[k] for k in keys])
    E, V = _local(G, rho, v.detach())
    e, w = _wt(G, rho)
    return {"energy": float(E + e + _ewald(G, s, pos.detach())), "rho": (V + w) * G.dV, "positions": g[0],
            "tables": torch.cat(g[1:])}
