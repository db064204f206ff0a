"""What the performance of this package is measured on: surveys run through its public entry points.

A case is one of five uses, each over the grids it is used on:

* ``run``       every step of each transmitter of one survey (``Simulation.run``), the product's main use;
* ``batch``     several surveys of different sizes set up, advanced together and collected (``Batch``);
* ``stages``    a host program that drives the time loop itself, one call per stage of a step;
* ``snapshot``  some steps of a run, then the six field volumes on the host.

The grids go from 40 x 36 x 24 to 256 x 256 x 160 cells, odd sizes among them, in FP32 (the production
precision) and FP64 (the reference's), on land and at sea, on the reference's continuation plane and on
the padded one.  Models are seeded and synthetic.  ``exact`` restates the whole path in 64 bits with torch.
"""
import copy
import math
import os
import tempfile

import numpy as np
import torch

from tcsem_fdtd_gb300 import Batch, Simulation, inputs

MU0 = 4e-7 * math.pi


# ------------------------------------------------------------------------------------------- the cases


def _case(name, use, L, M, N, **kw):
    c = dict(name=name, use=use, kind="marine", L=L, M=M, N=N, strip=20, growth=1.08, cell=25.0, sfa1=2.0, Tn=1.0, Nt=61,
             nrx=40, ntx=1, precision=32, plane=0, surveys=1, steps=0)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest: a towline, several transmitters over one small model, a launch-bound step loop
        _case("towline_44x38x27", "run", 44, 38, 27, strip=10, growth=1.15, cell=40.0, Tn=0.05, Nt=24, nrx=12, ntx=4),
        # a land survey over a half-space, in both precisions
        _case("land_64x64x48", "run", 64, 64, 48, kind="land", growth=1.15, sfa1=1.5, nrx=15),
        _case("land_64x64x48_fp64", "run", 64, 64, 48, kind="land", growth=1.15, sfa1=1.5, nrx=15, Tn=0.1, precision=64),
        # a long thin grid: an odd continuation plane with large prime factors
        _case("land_160x56x40", "run", 160, 56, 40, kind="land", growth=1.2, cell=12.5, sfa1=1.5, Tn=0.1, Nt=41, nrx=8),
        # marine surveys of ordinary size
        _case("marine_128x128x96", "run", 128, 128, 96, growth=1.12, cell=20.0),
        _case("marine_187x121x101", "run", 187, 121, 101, strip=25, nrx=60),
        # the padded continuation plane (smooth transform lengths), odd grid
        _case("smooth_133x130x95", "run", 133, 130, 95, kind="land", strip=29, growth=1.075, Tn=0.3, Nt=41, plane=2),
        # the largest: the 3-D marine survey, in both precisions
        _case("marine_256x256x160", "run", 256, 256, 160, strip=40, nrx=441),
        _case("marine_256x256x160_fp64", "run", 256, 256, 160, strip=40, nrx=441, Tn=0.02, Nt=21, precision=64),
        # surveys of different sizes as one batch, from their input files
        _case("batch_8", "batch", 152, 131, 112, surveys=8, Tn=0.3, Nt=41),
        # a host that calls the stages of each step itself and samples the receivers
        _case("stages_64x64x48", "stages", 64, 64, 48, kind="land", growth=1.1, steps=32, nrx=20),
        # field volumes for inspection
        _case("snapshot_128x128x96", "snapshot", 128, 128, 96, growth=1.06, cell=20.0, steps=256),
    ]


def draw(rng):
    use = rng.choice(["run"] * 6 + ["batch", "stages", "snapshot"])
    precision = 64 if use == "run" and rng.random() < 0.25 else 32
    kind = rng.choice(["land", "marine"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    top = {"run": (256, 256, 160), "batch": (152, 131, 112), "stages": (128, 128, 96), "snapshot": (128, 128, 96)}[use]
    L, M, N = size(40, top[0]), size(36, top[1]), size(24, top[2])
    if rng.random() < 0.5:
        L, M, N = L | 1, M | 1, N | 1
    L, M, N = min(L, top[0]), min(M, top[1]), min(N, top[2])
    strip = max(6, min(40, (min(L, M) - 20) // 2, (N - 10), rng.randint(8, 40)))
    growth = rng.choice([1.06, 1.08]) if strip > 24 else rng.choice([1.06, 1.08, 1.1, 1.15])
    c = _case("", use, L, M, N, kind=kind, strip=strip, growth=growth, cell=rng.choice([20.0, 25.0, 40.0]),
              sfa1=2.0 if kind == "marine" else 1.5, Nt=rng.randint(20, 81), nrx=rng.randint(4, 120), precision=precision)
    del c["name"]
    if use == "run":
        c["plane"] = rng.choice([0, 0, 0, 2])
        c["ntx"] = rng.randint(1, 4) if L * M * N < 200_000 else 1
        c["Tn"] = float("%.3g" % math.exp(rng.uniform(math.log(0.02), math.log(1.0))))
        # no more work than the largest listed case of the precision
        most = 2.0e10 if precision == 32 else 3e9
        while c["Tn"] > 0.012 and L * M * N * c["ntx"] * _nsteps(c) > most:
            c["Tn"] = float("%.3g" % (0.6 * c["Tn"]))
    elif use == "batch":
        c["surveys"], c["Tn"] = rng.randint(2, 8), 0.3
    else:  # stages on land, where the source reaches the air plane within the steps; volumes at sea
        c["kind"], c["steps"] = ("land", rng.randint(8, 32)) if use == "stages" else ("marine", rng.randint(64, 256))
    return c


# ------------------------------------------------------------------------------------------ the surveys


def _survey(case, seed, q=0):
    """Survey q of the case as the values of inputs.write_case / inputs.memory_case, drawn from the seed."""
    rng = np.random.default_rng([int(seed), q])
    L, M, N = case["L"], case["M"], case["N"]
    if case["use"] == "batch":  # surveys of different sizes, fixed by the case
        f = 1.0 - 0.045 * q
        L, M, N = max(40, int(L * f)), max(36, int(M * (1.12 - f * 0.12) * f)), max(24, int(N * (0.5 + 0.5 * f)))
    s = min(case["strip"], (min(L, M) - 20) // 2)
    sz = min(case["strip"], N // 2)
    d, nx, ny, nz = case["cell"], L - 2 * s, M - 2 * s, N - sz
    hx, hy, depth = 0.5 * nx * d, 0.5 * ny * d, nz * d
    marine = case["kind"] == "marine"
    floor = round(0.4 * nz) * d if marine else 0.0
    c = dict(sfa1=case["sfa1"], sfa2=2.0, n1=200, sita_t=1e-4, origin=(0.0, 0.0, 0.0), dmin=(d, d, d), arg1=case["growth"],
             arg2=case["growth"], xsplit=(0, s, nx, s, 0), ysplit=(0, s, ny), zsplit=(0, sz, nz), T0=1e-3, Tn=case["Tn"],
             Nt=case["Nt"], islog=1, comps=(1, 1, 0, 1, 1, 1) if marine else (1, 1, 0, 0, 1, 1))
    rows = max(1, int(math.sqrt(case["nrx"] / 4.0)))
    cols = -(-case["nrx"] // rows)
    c["receivers"] = [(0.83 * hx * (2.0 * (i + 0.53) / cols - 1.0), 0.71 * hy * ((2.0 * j + 1.1) / rows - 1.0), floor)
                      for j in range(rows) for i in range(cols)][: case["nrx"]]
    x0 = float(rng.uniform(-0.3, 0.3)) * hx
    c["transmitters"] = [dict(ort=1, len=2 * d, x=x0 + 0.37 * hx * (t / max(1, case["ntx"] - 1) - 0.5) * (case["ntx"] > 1),
                              y=float(rng.uniform(-0.2, 0.2)) * hy, z=max(0.0, floor - 2 * d)) for t in range(case["ntx"])]
    # layers, a smooth lateral and vertical variation, a resistive block
    g = inputs.grid_axes(c)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    z = np.asarray(g["Z"])
    layer = np.where(z < floor, 3.2, float(rng.uniform(0.5, 1.5)))
    layer = np.where(z > floor + float(rng.uniform(0.3, 0.6)) * (depth - floor), float(rng.uniform(0.3, 2.0)), layer)
    ax = [torch.as_tensor(np.asarray(g[a]), dtype=torch.float64, device=dev) for a in "ZYX"]
    noise = torch.zeros(N, M, L, dtype=torch.float64, device=dev)
    for _ in range(4):
        k = rng.uniform(0.2, 1.0, 3) * 2 * math.pi / np.array([depth, hy, hx])
        p = rng.uniform(0, 2 * math.pi, 3)
        w = [torch.cos(a * float(kk) + float(pp)) for a, kk, pp in zip(ax, k, p)]
        noise += 0.15 * w[0][:, None, None] * w[1][None, :, None] * w[2][None, None, :]
    con = torch.as_tensor(layer, dtype=torch.float64, device=dev)[:, None, None] * 10.0 ** noise
    if marine:
        con[torch.as_tensor(z < floor, device=dev)] = 3.2
        b = [(ax[0] > floor + 0.3 * (depth - floor)) & (ax[0] < floor + 0.3 * (depth - floor) + 4 * d), ax[1].abs() < 0.4 * hy,
             ax[2].abs() < 0.4 * hx]
        con = torch.where(b[0][:, None, None] & b[1][None, :, None] & b[2][None, None, :], torch.full_like(con, 0.02), con)
    return c, con.cpu().numpy()


def _model(c, con):
    """The (model, survey) values of the in-memory open."""
    m = dict(sfa1=c["sfa1"], sfa2=c["sfa2"], n1=c["n1"], sita_t=c["sita_t"], x0=0.0, y0=0.0, z0=0.0, dxmin=c["dmin"][0],
             dymin=c["dmin"][1], dzmin=c["dmin"][2], arg1=c["arg1"], arg2=c["arg2"], con=con)
    m.update(zip(("ALx2", "ALx1", "Nx", "ARx1", "ARx2"), c["xsplit"]))
    m.update(zip(("Ay2", "Ay1", "Ny"), c["ysplit"]))
    m.update(zip(("Az2", "Az1", "Nz"), c["zsplit"]))
    s = dict(T0=c["T0"], Tn=c["Tn"], Nt=c["Nt"], IsLog=c["islog"], comps=list(c["comps"]), rx_xyz=np.array(c["receivers"]),
             tx=[dict(t, rx=list(range(1, len(c["receivers"]) + 1))) for t in c["transmitters"]])
    return m, s


def prepare(case, seed):
    if case["use"] == "batch":  # the input files of the surveys, as the batch reads them
        root = tempfile.TemporaryDirectory(prefix="tcsem_cases_")
        dirs = []
        for q in range(case["surveys"]):
            c, con = _survey(case, seed, q)
            dirs.append(os.path.join(root.name, "s%d" % q))
            inputs.write_case(dict(copy.deepcopy(c), model=dict(kind="uniform", sigma=1.0)), dirs[-1])
            con.astype("<f8").tofile(os.path.join(dirs[-1], "Cond.bin"))
        return dict(case=case, dirs=dirs, root=root)
    model, survey = _model(*_survey(case, seed))
    sim = Simulation(model=model, survey=survey, precision=case["precision"], padded_plane=case["plane"])
    return dict(case=case, sim=sim, sched=sim.schedule())


FIELDS = ("Ex", "Ey", "Ez", "Bx", "By", "Bz")


def run(state):
    case = state["case"]
    # the package hands FP32 results over as doubles: give them back their own type
    out = np.float32 if case["precision"] == 32 else np.float64
    if case["use"] == "batch":
        with Batch(precision=case["precision"]) as b:
            slots = [b.add(d) for d in state["dirs"]]
            while b.stats()["running"]:
                b.advance(1024)
            return [b.traces(s).astype(out) for s in slots]
    sim = state["sim"]
    if case["use"] == "run":
        return [sim.run(t).astype(out) for t in range(case["ntx"])]
    sim.begin(0)
    if case["use"] == "snapshot":
        sim.advance(case["steps"])
        return {n: sim.get(n).astype(out) for n in FIELDS}
    sc, nr, ne, e, b = state["sched"], case["nrx"], 2, [], []  # two E components are recorded
    for n in range(case["steps"]):
        sim.upcontinuation()
        sim.electric_field(sc["lam"][n], sc["dt1"][n], sc["wave"][n])
        sim.bderivate(0.5 * (sc["dt1"][n] + sc["dt2"][n]))
        e.append(sim.rx_sample(True, 0, nr)[:ne].astype(out))
        b.append(sim.rx_sample(False, 0, nr)[ne:].astype(out))
    return dict(e=np.stack(e), b=np.stack(b), bxair=sim.get("BxAir").astype(out), byair=sim.get("ByAir").astype(out))


def work(case):
    """Per step and cell: six field components and the conductivity read, six components written; about 60 operations."""
    word = case["precision"] // 8
    if case["use"] == "batch":
        cells = 0
        for q in range(case["surveys"]):
            f = 1.0 - 0.045 * q
            cells += max(40, int(case["L"] * f)) * max(36, int(case["M"] * (1.12 - f * 0.12) * f)) * max(24, int(case["N"] * (0.5 + 0.5 * f)))
    else:
        cells = case["L"] * case["M"] * case["N"]
    steps = case["steps"] or case["ntx"] * _nsteps(case)
    return {"bytes": 13.0 * word * cells * steps, "flops": 60.0 * cells * steps}


# ---------------------------------------------------------------- the same path in 64 bits, for comparison


def _source_wave(sita, nsrc):
    """Gaussian pulse sampled at steps of equal area, and the time steps between the samples."""
    t, dt = np.zeros(2 * nsrc + 1), np.zeros(2 * nsrc + 2)
    for i in range(nsrc):
        a = t[i] - 3 * sita
        dt[i] = -sita * sita * (1 - math.exp(-4.5)) / nsrc / a / math.exp(-a * a / (2 * sita * sita))
        t[i + 1] = t[i] + dt[i]
    t[nsrc] = min(t[nsrc], 3 * sita) if 3 * sita < t[nsrc] else t[nsrc]
    for i in range(nsrc + 1, 2 * nsrc + 1):
        t[i] = 6 * sita - t[2 * nsrc - i]
        dt[i - 1] = t[i] - t[i - 1]
    wave = np.exp(-((t - 3 * sita) ** 2) / 2 / sita / sita) / (math.sqrt(2 * math.pi) * sita)
    dt[2 * nsrc] = 0.0
    mid = np.zeros(2 * nsrc + 2)
    mid[2 * nsrc + 1] = 0.5 * (dt[2 * nsrc] ** 2 / dt[2 * nsrc - 1] + dt[2 * nsrc])
    mid[0] = 0.5 * (dt[0] * dt[0] / dt[1] + dt[0])
    mid[1: 2 * nsrc + 1] = 0.5 * (dt[: 2 * nsrc] + dt[1: 2 * nsrc + 1])
    return mid, wave


def _steps(c, nefcmp, has_b):
    """Per step (dt1, dt2, gamma, amplitude) and which receiver samples it completes; per sample its weight."""
    nsrc, d = c["n1"] // 2, min(c["dmin"])
    mid, wave = _source_wave(c["sita_t"], nsrc)
    T = 10.0 ** (np.log10(c["T0"]) + np.arange(c["Nt"]) * (np.log10(c["Tn"]) - np.log10(c["T0"])) / (c["Nt"] - 1))
    Nt, n, to, dt1, dt2 = c["Nt"], 0, 0.0, mid[0], mid[1]
    tp = [[0.0, dt1, 0.0], [0.0, dt1 + 0.5 * dt2, 0.0]]
    done, weight, steps = [0, 0 if has_b else Nt], [np.zeros(Nt), np.zeros(Nt)], []
    while min(done) < Nt:
        s = [dt1, dt2, 7.5 * c["sfa2"] * dt2 * dt1 / MU0 / d / d, wave[n] if n < 2 * nsrc else 0.0]
        to, dt1, n = to + dt1, dt2, n + 1
        dt2 = mid[n + 1] if n < 2 * nsrc else min(0.15 * c["sfa1"] * math.sqrt(MU0 * to * 0.1 / 8.0) * d, 1.2 * dt1)
        for f in (0, 1):
            act, m = None, done[f]
            if m < Nt:
                p = tp[f]
                p[2] = to + dt1 + (0.5 * dt2 if f else 0.0)
                while m < Nt and T[m] <= p[0]:
                    m += 1
                if m < Nt and p[1] < T[m] <= p[2]:
                    act = (0, m, m)
                elif m < Nt and p[0] < T[m] <= p[1]:
                    first = m
                    while m < Nt and T[m] <= p[1]:
                        weight[f][m] = (T[m] - p[0]) / (p[1] - p[0])
                        m += 1
                    act = (1, first, m)
                done[f] = m
                p[0], p[1] = p[1], p[2]
            s.append(act)
        steps.append(s)
    return steps, weight


_COUNTS = {}


def _nsteps(case):
    """Steps of one transmitter run of the case (the number depends on the times and the smallest cell alone)."""
    key = (case["sfa1"], case["cell"], case["Tn"], case["Nt"], case["kind"])
    if key not in _COUNTS:
        c = dict(sfa1=case["sfa1"], sfa2=2.0, n1=200, sita_t=1e-4, dmin=(case["cell"],) * 3, T0=1e-3, Tn=case["Tn"], Nt=case["Nt"])
        _COUNTS[key] = len(_steps(c, 2, True)[0])
    return _COUNTS[key]


def _axis(d, lead, core, tail, growth, centred):
    size = np.array([d * growth ** (lead - i) for i in range(lead)] + [d] * core + [d * growth ** (i + 1) for i in range(tail)])
    x = np.zeros(len(size))
    if not centred:
        x[0] = 0.5 * size[0]
        start = 0
    else:
        start = core // 2 + lead if core % 2 == 0 else (core - 1) // 2 + lead
        x[start] = 0.5 * size[start] if core % 2 == 0 else 0.0
    for i in range(start + 1, len(size)):
        x[i] = x[i - 1] + 0.5 * size[i - 1] + 0.5 * size[i]
    for i in range(start - 1, -1, -1):
        x[i] = x[i + 1] - 0.5 * size[i + 1] - 0.5 * size[i]
    return size, x


def _strip(d, x, new, rows):
    """Natural cubic spline from the nodes x to the points new as a matrix; the end slopes continue beyond the nodes."""
    n, h = len(x), 0.5 * (d[:-1] + d[1:])
    A, R = np.eye(n) * 2.0, np.zeros((n, n))
    for i in range(1, n - 1):
        A[i, i - 1], A[i, i], A[i, i + 1] = h[i - 1] / 3, 2.0 / 3 * (h[i - 1] + h[i]), h[i] / 3
        R[i, i - 1], R[i, i], R[i, i + 1] = 1 / h[i - 1], -1 / h[i - 1] - 1 / h[i], 1 / h[i]
    y, m = np.eye(n), np.linalg.solve(A, R)
    out = np.zeros((len(new), n))
    for p, (t, r) in enumerate(zip(new, rows)):
        i = max(r - 1, 0)
        if i < n - 1:
            a, b = (m[i + 1] - m[i]) / h[i] / 3, (y[i + 1] - y[i]) / h[i] - (2 * m[i] + m[i + 1]) * h[i] / 3
        else:
            a, b = (m[i] - m[i - 1]) / h[i - 1] / 3, (y[i] - y[i - 1]) / h[i - 1] - (2 * m[i - 1] + m[i]) * h[i - 1] / 3
            b, a = b + 3 * a * h[i - 1] ** 2 + 2 * m[i - 1] * h[i - 1], 0 * a
        u = t - x[i]
        out[p] = ((a * u if 0 <= r - 1 < n - 1 else 0) + m[i]) * u * u + b * u + y[i]
    return out


def _plane_axis(d, x, lead, core, tail, cell):
    """Uniform line under the grid's line: its nodes, the remap onto it, and the two samplings back (faces, centres)."""
    nl = math.ceil((x[lead - 1] - x[0] + d[lead - 1] / 2 + d[0] / 2) / cell)
    nr = math.ceil((x[-1] - x[len(x) - tail] + d[-1] / 2 + d[len(x) - tail] / 2) / cell)
    new = np.zeros(nl + core + nr)
    new[nl: nl + core] = x[lead: lead + core]
    for i in range(nl - 1, -1, -1):
        new[i] = new[i + 1] - cell
    for i in range(nl + core, len(new)):
        new[i] = new[i - 1] + cell
    P = np.zeros((len(new), len(x)))
    P[nl: nl + core, lead: lead + core] = np.eye(core)
    at = np.searchsorted(x, new)
    P[:nl, : lead + 4] = _strip(d[: lead + 4], x[: lead + 4], new[:nl], at[:nl])
    o = lead + core - 4
    P[nl + core:, o:] = _strip(d[o:], x[o:], new[nl + core:], at[nl + core:] - o)

    def back(pos):
        B = np.zeros((len(pos), len(new)))
        i = np.clip(np.searchsorted(new, pos), 1, len(new) - 1)
        w = (pos - new[i - 1]) / (new[i] - new[i - 1])
        B[np.arange(len(pos)), i - 1], B[np.arange(len(pos)), i] = 1 - w, w
        return B

    return new, P, back(np.append(x - 0.5 * d, x[-1] + 0.5 * d[-1])), back(x)


def _padded(P, n):
    """The remap onto a line of n points whose points beyond the grid taper from its edge values to zero."""
    u = P.shape[0]
    lo = (n - u) // 2
    hi = n - u - lo
    out = np.zeros((n, P.shape[1]))
    out[lo: lo + u] = P
    for i in range(lo):
        out[i] = 0.5 * (1 - math.cos(math.pi * i / lo)) * P[0]
    for i in range(lo + u, n):
        out[i] = 0.5 * (1 - math.cos(math.pi * (n - i) / (hi + 1))) * P[-1]
    return out, lo


def _smooth_length(n):
    while True:
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1:
            return n
        n += 1


def _spline4(x, t):
    """Weights of four nodes in their natural cubic spline at t, between the middle two."""
    w = []
    for q in range(4):
        y = np.eye(4)[q]
        h, v1, v2 = x[2] - x[1], 2 * (x[2] - x[0]), 2 * (x[3] - x[1])
        u1 = 6 * ((y[2] - y[1]) / h - (y[1] - y[0]) / (x[1] - x[0]))
        u2 = 6 * ((y[3] - y[2]) / (x[3] - x[2]) - (y[2] - y[1]) / h)
        z1, z2 = (v2 * u1 - h * u2) / (v1 * v2 - h * h), (v1 * u2 - h * u1) / (v1 * v2 - h * h)
        w.append(z2 / 6 / h * (t - x[1]) ** 3 + z1 / 6 / h * (x[2] - t) ** 3 + (y[2] / h - z2 / 6 * h) * (t - x[1]) +
                 (y[1] / h - z1 / 6 * h) * (x[2] - t))
    return w


class _Path:
    """The survey's whole time loop in 64 bits."""

    def __init__(self, c, con, plane):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        d = c["dmin"][0]
        s, (nx, ny, nz), sz, gr = c["xsplit"][1], (c["xsplit"][2], c["ysplit"][2], c["zsplit"][2]), c["zsplit"][1], c["arg1"]
        self.c, self.con = c, con
        self.d = [_axis(d, s, nx, s, gr, True), _axis(d, s, ny, s, gr, True), _axis(d, 0, nz, sz, gr, False)]
        (dx, X), (dy, Y), (dz, Z) = self.d
        self.L, self.M, self.N = len(X), len(Y), len(Z)
        self.T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)
        self.steps, self.weight = _steps(c, 2, any(c["comps"][3:]))
        r = lambda a: self.T(1.0 / a)  # noqa: E731
        self.rdx, self.rdy, self.rdz, self.dz = r(dx), r(dy)[:, None], r(dz)[:, None, None], self.T(dz)[:, None, None]
        self.rdx2, self.rdy2 = r(dx[1:] + dx[:-1]), r(dy[1:] + dy[:-1])[:, None]
        self.rdzs = r(dz + np.append(dz[0], dz[:-1]))[:, None, None]
        k = self.T(con)
        up = torch.cat([torch.zeros_like(k[:1]), k[:-1]])
        self.sx = 0.25 * (k[:, :-1] + k[:, 1:] + up[:, :-1] + up[:, 1:])
        self.sy = 0.25 * (k[:, :, :-1] + k[:, :, 1:] + up[:, :, :-1] + up[:, :, 1:])
        self.sz = 0.25 * (k[:, :-1, :-1] + k[:, 1:, :-1] + k[:, :-1, 1:] + k[:, 1:, 1:])
        # air plane: remap, transform, continuation filters, sampling back
        px, py = _plane_axis(dx, X, s, nx, s, d), _plane_axis(dy, Y, s, ny, s, d)
        Px, Py, fx, cx, fy, cy = px[1], py[1], px[2], px[3], py[2], py[3]
        if plane:
            ln, mn = _smooth_length(Px.shape[0]), _smooth_length(Py.shape[0])
            Px, lx = _padded(Px, ln)
            Py, ly = _padded(Py, mn)
            fx, cx = (np.pad(a, ((0, 0), (lx, ln - lx - a.shape[1]))) for a in (fx, cx))
            fy, cy = (np.pad(a, ((0, 0), (ly, mn - ly - a.shape[1]))) for a in (fy, cy))
        L1, M1 = Px.shape[0], Py.shape[0]
        u = (np.pi * np.arange(L1 // 2 + 1) / L1)[None, :]
        ky = np.arange(M1)
        v = (np.pi * np.where(ky < M1 // 2 + 1, ky, ky - M1) / M1)[:, None]
        w = np.sqrt(u * u + v * v)
        w[0, 0] = 1.0
        e = np.exp(-w) / w
        gx, gy = u * e, v * e
        gx[0, 0] = gy[0, 0] = 1.0
        self.Px, self.Py = self.T(Px.T), self.T(Py)
        self.gx, self.gy = 1j * self.T(gx), 1j * self.T(gy)
        self.size = (M1, L1)
        self.bxy, self.bxx, self.byy, self.byx = self.T(cy), self.T(fx.T), self.T(fy), self.T(cx.T)

    def begin(self, itx):
        L, M, N = self.L, self.M, self.N
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=self.rdx.device)  # noqa: E731
        self.ex, self.ey, self.ez = z(N + 1, M + 1, L), z(N + 1, M, L + 1), z(N, M + 1, L + 1)
        self.bx, self.by, self.bz = z(N + 1, M, L + 1), z(N + 1, M + 1, L), z(N + 1, M, L)  # plane 0 of bx, by: the air
        t, (dx, X), (dy, Y), (dz, Z) = self.c["transmitters"][itx], *self.d
        a, b = np.searchsorted(X, t["x"] - t["len"] / 2), np.searchsorted(X, t["x"] + t["len"] / 2) - 1
        j, k = np.searchsorted(Y, t["y"]), np.searchsorted(Z, t["z"])
        gain = 1.0 / (X[b] - X[a] + dx[b] / 2 + dx[a] / 2)
        lo, n = min(a, b), abs(b - a) + 1
        sg = self.con[k, j, lo: lo + n] + self.con[k, j - 1, lo: lo + n]
        if k:
            sg = sg + self.con[k - 1, j, lo: lo + n] + self.con[k - 1, j - 1, lo: lo + n]
        self.src = (k, j, slice(lo, lo + n), self.T(gain * 2.0 / (0.25 * sg * dy[j] * dz[k])))
        self.rx = [self._receivers(q) for q in range(6) if self.c["comps"][q]]
        self.ne = sum(1 for q in range(3) if self.c["comps"][q])

    def _receivers(self, comp):
        """Four nodes and weights per axis of every receiver for one component."""
        face = (comp in (1, 2, 3), comp in (0, 2, 4), comp in (0, 1, 5))
        idx, wgt = [], []
        for a, ((d, x), f) in enumerate(zip(self.d, face)):
            pos = np.array([r[a] for r in self.c["receivers"]])
            n = np.searchsorted(x, pos)
            at = np.where(x[np.maximum(n - 1, 0)] + 0.5 * d[np.maximum(n - 1, 0)] > pos, n - 2, n - 1) if f else n - 2
            at = np.maximum(np.where(n >= 1, at, -1) if f else at, 0)
            node = x[at[:, None] + np.arange(4)] - (0.5 * d[at[:, None] + np.arange(4)] if f else 0.0)
            idx.append(torch.as_tensor(at[:, None] + np.arange(4), device=self.rdx.device))
            wgt.append(self.T([_spline4(q, p) for q, p in zip(node, pos)]))
        return comp, idx, wgt

    def sample(self, p):
        comp, (i, j, k), (wx, wy, wz) = self.rx[p]
        f = (self.ex, self.ey, self.ez, self.bx[1:], self.by[1:], self.bz)[comp]
        return torch.einsum("rkji,rk,rj,ri->r", f[k[:, :, None, None], j[:, None, :, None], i[:, None, None, :]], wz, wy, wx)

    def air(self):
        F = torch.fft.rfft2(self.Py @ self.bz[0] @ self.Px)
        self.bx[0] = self.bxy @ torch.fft.irfft2(self.gx * F, s=self.size) @ self.bxx
        self.by[0] = self.byy @ torch.fft.irfft2(self.gy * F, s=self.size) @ self.byx

    def step(self, s):
        dt, dtb, lam, wave = s[0], 0.5 * (s[0] + s[1]), 2 * s[2], s[3]
        N = self.N
        self.air()
        bx, by, bz = self.bx, self.by, self.bz
        for e, sg, curl in ((self.ex[:N, 1:-1], self.sx, torch.diff(bz[:N], dim=1) * self.rdy2 - torch.diff(by, dim=0)[:, 1:-1] * self.rdzs),
                            (self.ey[:N, :, 1:-1], self.sy, torch.diff(bx, dim=0)[:, :, 1:-1] * self.rdzs - torch.diff(bz[:N], dim=2) * self.rdx2),
                            (self.ez[:, 1:-1, 1:-1], self.sz, torch.diff(by[1:, 1:-1], dim=2) * self.rdx2 - torch.diff(bx[1:, :, 1:-1], dim=1) * self.rdy2)):
            q = sg * dt
            e.mul_(lam - q).add_(curl, alpha=4 * dt / MU0).div_(q.add_(lam))
        if wave:
            k, j, i, coef = self.src
            self.ex[k, j, i] -= wave * coef
        bx[1:, :, 1:-1] += (torch.diff(self.ey, dim=0) * self.rdz - torch.diff(self.ez, dim=1) * self.rdy)[:, :, 1:-1] * dtb
        by[1:, 1:-1] += (torch.diff(self.ez, dim=2) * self.rdx - torch.diff(self.ex, dim=0) * self.rdz)[:, 1:-1] * dtb
        div = (torch.diff(bx[1:], dim=2) * self.rdx + torch.diff(by[1:], dim=1) * self.rdy) * self.dz
        bz[:N] = div.flip(0).cumsum(0).flip(0)

    def traces(self, itx):
        self.begin(itx)
        Nt, nr, n = self.c["Nt"], len(self.c["receivers"]), len(self.rx)
        out, held = np.zeros((nr, n, Nt)), [None] * n
        for s in self.steps:
            self.step(s)
            for p in range(n):
                f = 0 if p < self.ne else 1
                act = s[4 + f]
                if act is None:
                    continue
                v = self.sample(p).cpu().numpy()
                if act[0] == 0:
                    held[p] = v
                else:
                    v0 = held[p] if held[p] is not None else np.zeros(nr)
                    w = self.weight[f][act[1]: act[2]]
                    out[:, p, act[1]: act[2]] = (1 - w) * v0[:, None] + w * v[:, None]
        return out


def exact(case, seed):
    if case["use"] == "batch":
        return [_Path(*_survey(case, seed, q), 0).traces(0) for q in range(case["surveys"])]
    p = _Path(*_survey(case, seed), case["plane"])
    if case["use"] == "run":
        return [p.traces(t) for t in range(case["ntx"])]
    p.begin(0)
    e, b = [], []
    for s in p.steps[: case["steps"]]:
        p.step(s)
        if case["use"] == "stages":
            v = [p.sample(q).cpu().numpy() for q in range(len(p.rx))]
            e.append(v[: p.ne])
            b.append(v[p.ne:])
    if case["use"] == "stages":
        return dict(e=np.array(e), b=np.array(b), bxair=p.bx[0].cpu().numpy(), byair=p.by[0].cpu().numpy())
    return {n: a.cpu().numpy() for n, a in zip(FIELDS, (p.ex, p.ey, p.ez, p.bx[1:], p.by[1:], p.bz))}
