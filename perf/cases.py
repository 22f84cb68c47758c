"""Performance cases of the walker-propagation library.

What a program does with this library, through its public Python view
(2degas_b200.Handle and Batch over the C-ABI): evaluate configurations
(compute_properties), run a block of VMC or DMC generations or of reptation
moves on a device-resident population, sweep single electrons, and advance a
batch of populations together. A pass of a chain case is one block, as the
method loops of 2degas_b200/drivers.py run it: reset the block sums, move,
read the block sums back; the population itself comes out as walker records
packed on the device (what a multi-rank run sends to its peers).

Decks are those of 2degas_b200/tables.py (the benchmark's u2, u3, backflow
and Ewald forms) at closed shells of 26 to 162 electrons, unpolarised and
polarised; walkers start from the seed and are equilibrated by a few VMC
steps. Launch choices stay at their defaults, as the serving loop leaves
them, so that a block depends on its inputs alone.

    kind    pass
    eval    compute_properties of `walkers` configurations; host buffers
            with host=True, else device buffers
    vmc     `steps` all-electron VMC steps of the population
    dmc     `steps` DMC generations (one move, weights, comb) of the population
    single  `steps` single-electron sweeps (plain determinants: bf=False)
    rmc     `steps` reptation moves of `walkers` reptiles of `beads` beads
    batch   `steps` DMC generations of four populations of different shells
"""
import importlib
import math
import os
import tempfile

import numpy as np
import torch

q = importlib.import_module("2degas_b200")
tables = importlib.import_module("2degas_b200.tables")

UNPOLARISED = (13, 21, 25, 29, 37, 45, 49, 57, 61, 69, 81)
POLARISED = (25, 29, 37, 45, 49, 57, 61, 69, 81, 89, 97, 101, 109, 113, 121, 129, 137, 145, 149,
             161)
# the shells that a batch case advances together: (up, down)
BATCH_SHELLS = ((13, 13), (29, 29), (45, 0), (37, 37))
EQUIL = 20  # VMC steps before the timed work


def _case(name, kind, up, down, rs, walkers, steps, u3=False, bf=True, mixed=False, host=False,
          beads=0):
    return dict(name=name, kind=kind, up=up, down=down, rs=rs, walkers=walkers, steps=steps,
                u3=u3, bf=bf, mixed=mixed, host=host, beads=beads)


def listed():
    return [
        # a host program (the reference's Fortran caller) that evaluates a few
        # configurations at a time from its own arrays
        _case("eval_host_n26_u3_w64", "eval", 13, 13, 10.0, 64, 1, u3=True, host=True),
        # properties of a whole population, as reading configurations back does
        _case("eval_n58_w4096", "eval", 29, 29, 5.0, 4096, 1),
        # the plain Slater-Jastrow VMC benchmark configuration
        _case("vmc_n26_rs1_w256", "vmc", 13, 13, 1.0, 256, 20, bf=False),
        # the same state point with single-electron sweeps
        _case("single_n26_rs1_w256", "single", 13, 13, 1.0, 256, 10, bf=False),
        # VMC with every Jastrow and backflow term, an odd number of walkers
        _case("vmc_n74_u3_w1001", "vmc", 37, 37, 3.0, 1001, 4, u3=True),
        # the headline DMC population
        _case("dmc_n58_rs5_w4096", "dmc", 29, 29, 5.0, 4096, 6),
        # a small mixed-precision DMC request
        _case("dmc_n42_mixed_w700", "dmc", 21, 21, 5.0, 700, 6, mixed=True),
        # the largest shells held in shared memory, and beyond, as the batch
        # and serving workloads run them
        _case("dmc_n90_rs10_w1024", "dmc", 45, 45, 10.0, 1024, 4),
        _case("dmc_n122_rs2_w1024", "dmc", 61, 61, 2.0, 1024, 3),
        _case("dmc_n161p_rs5_w768", "dmc", 161, 0, 5.0, 768, 2),
        # the reptation benchmark configuration
        _case("rmc_n58_rs10_r512", "rmc", 29, 29, 10.0, 512, 12, u3=True, beads=200),
        # populations of different shells and polarisations in one graph
        _case("batch_dmc_4pops_w512", "batch", 0, 0, 5.0, 512, 4),
    ]


def draw(rng):
    kind = rng.choice(("eval", "vmc", "dmc", "dmc", "rmc", "single", "batch"))
    c = _case("", kind, 0, 0, rng.choice((1.0, 2.0, 3.0, 5.0, 10.0, 20.0)),
              int(round(math.exp(rng.uniform(math.log(64), math.log(4096))))),
              1 if kind == "eval" else rng.randint(2, 8))
    del c["name"]
    if kind != "batch":
        if rng.random() < 0.3:
            c["up"], c["down"] = rng.choice(POLARISED), 0
        elif rng.random() < 0.25:  # partly polarised: two neighbouring shells
            k = rng.randrange(1, len(UNPOLARISED))
            c["up"], c["down"] = UNPOLARISED[k], UNPOLARISED[k - 1]
        else:
            c["up"] = c["down"] = rng.choice(UNPOLARISED)
        c["u3"] = rng.random() < 0.3
        c["mixed"] = kind in ("eval", "vmc", "dmc") and rng.random() < 0.25
        c["host"] = kind == "eval" and rng.random() < 0.5
    if kind == "single":  # shells whose inverses stay in shared memory
        c.update(up=rng.choice((13, 21, 25, 29)), u3=False, bf=False)
        c["down"] = rng.choice((0, c["up"]))
    elif kind == "vmc":
        c["bf"] = rng.random() < 0.7
    elif kind == "rmc":
        c["beads"] = rng.randint(20, 200)
        c["walkers"] = min(c["walkers"], 768)
    elif kind == "batch":
        c["walkers"], c["steps"] = min(c["walkers"], 1024), 2 * rng.randint(1, 4)
    # no dearer than the largest listed case, in work and in set-up
    most = max(work(x)["flops"] for x in listed())
    while work(c)["flops"] > most and c["walkers"] > 64:
        c["walkers"] = c["walkers"] * 3 // 4
    while c["steps"] > 2 and work(c)["flops"] > most:
        c["steps"] -= 2 if kind == "batch" else 1
    while c["walkers"] * c["beads"] * (c["up"] + c["down"]) > 512 * 200 * 58:
        c["beads"] = c["beads"] * 3 // 4
        c["walkers"] = max(64, c["walkers"] * 3 // 4)
    return c


# ------------------------------------------------------------- set-up
def _deck(directory, case):
    rs = case["rs"]
    return tables.make_run(directory, "c", case["up"], case["down"], rs,
                           backflow=(0.2 if case["bf"] else 0.0, rs, 0.6 * rs), u3=case["u3"])


def _start(case, seed):
    """Configurations away from each other's electrons and from the nodes, as
    sampled ones are: jittered square lattices, their sites dealt to the
    electrons at random, and of four such per walker the one with the largest
    determinants."""
    n, nw = case["up"] + case["down"], case["walkers"]
    side = math.sqrt(n * math.pi)
    rng = np.random.default_rng(seed)
    m = math.ceil(math.sqrt(n))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    best, top = None, None
    for _ in range(4):
        site = rng.permuted(np.tile(np.arange(m * m), (nw, 1)), axis=1)[:, :n]
        x = np.stack((site // m, site % m), axis=2) + rng.uniform(0.1, 0.9, (nw, n, 2))
        x = torch.as_tensor(x * (side / m) - 0.5 * side, device=dev)
        qx = x.clone()
        if case["bf"]:
            r = x[:, :, None] - x[:, None]
            r -= side * torch.round(r / side)
            d = torch.sqrt((r * r).sum(-1, keepdim=True))
            qx += (0.2 * torch.exp(-((d - 1.0) / 0.6) ** 2) * r).sum(2)
        val, f0 = 0.0, 0
        for k in (case["up"], case["down"]):
            if k:
                g = torch.as_tensor(_waves(k), device=dev) * (2.0 * math.pi / side)
                a = torch.exp(1j * torch.einsum("kd,wjd->wkj", g, qx[:, f0:f0 + k]))
                val = val + torch.linalg.slogdet(a)[1]
                f0 += k
        if best is None:
            best, top = x, val
        else:
            best = torch.where((val > top)[:, None, None], x, best)
            top = torch.maximum(val, top)
    return best.reshape(nw, 2 * n).cpu().numpy()


def _waves(k):
    """The k shortest vectors of the square lattice (a closed shell)."""
    v = [(a * a + b * b, a, b) for a in range(-12, 13) for b in range(-12, 13)]
    return np.array([w[1:] for w in sorted(v)[:k]], dtype=np.float64)


def _tau(case):
    """Time steps that accept most moves: shorter the more electrons move
    together; a twentieth of that for the methods that need a small bias."""
    n = max(26, case["up"] + case["down"])
    t = 0.02 * case["rs"] ** 2 * 26.0 / n
    return t if case["kind"] in ("vmc", "single") else 0.05 * t


def _population(case, seed):
    """A handle with an equilibrated population, and its mean energy."""
    with tempfile.TemporaryDirectory(prefix="qmc2d_cases_") as tmp:
        system = q.System.read(_deck(os.path.join(tmp, "c"), case), "c")
    h = q.Handle(system, capacity=case["walkers"], seed=seed)
    if case["mixed"]:
        h.set_precision("mixed")
    h.population_set(_start(case, seed))
    h.vmc(EQUIL, _tau(dict(case, kind="vmc")), 50)
    h.block_reset()
    h.vmc(4, _tau(dict(case, kind="vmc")), 50)
    blk, norm = h.block_get()
    return h, float(blk[0] / norm)


def prepare(case, seed):
    s = dict(case)
    nw = case["walkers"]
    if case["kind"] == "eval":
        with tempfile.TemporaryDirectory(prefix="qmc2d_cases_") as tmp:
            system = q.System.read(_deck(os.path.join(tmp, "c"), case), "c")
        s["h"] = q.Handle(system, capacity=nw, seed=seed)
        if case["mixed"]:
            s["h"].set_precision("mixed")
        s["x"] = _start(case, seed)
        if not case["host"]:
            s["x"] = torch.from_numpy(s["x"]).cuda()
            s["out"] = [torch.empty(nw, k, dtype=torch.float64, device="cuda")
                        for k in (2 * system.N, system.ntypes, system.nprops, 1)]
            torch.cuda.synchronize()  # the handle's stream does not wait for torch's
    elif case["kind"] == "batch":
        pops = [dict(case, up=u, down=d) for u, d in BATCH_SHELLS]
        got = [_population(p, seed + 1000 * k) for k, p in enumerate(pops)]
        s["hs"], s["etrial"] = [g[0] for g in got], [g[1] for g in got]
        s["tau"] = [_tau(p) for p in pops]
        for h, p, tau in zip(s["hs"], pops, s["tau"]):
            h.set_dmc_ecut(_ecut(p, tau))
        s["batch"] = q.Batch(s["hs"])
    else:
        s["h"], s["etrial"] = _population(case, seed)
        s["tau"] = _tau(case)
        if case["kind"] == "dmc":
            s["h"].set_dmc_ecut(_ecut(case, s["tau"]))
        elif case["kind"] == "rmc":
            # reptiles: random walks of the propagator's link variance
            x = torch.from_numpy(s["h"].population_get()["x"]).cuda()
            gen = torch.Generator(device="cuda").manual_seed(seed)
            step = torch.randn(nw, case["beads"], x.shape[1], dtype=torch.float64, device="cuda",
                               generator=gen) * math.sqrt(2.0 * s["tau"] / case["rs"] ** 2)
            step[:, 0] = x
            paths = step.cumsum(1).reshape(nw * case["beads"], -1).cpu().numpy()
            s["h"].rmc_init(nw, paths, case["beads"], 1, 1, s["tau"], s["etrial"], 10 ** 9, 50)
    if case["kind"] in ("vmc", "dmc", "single", "batch"):
        s["slots"] = np.arange(nw, dtype=np.int32)
        s["rec"] = [torch.empty(nw, h.record_len(), dtype=torch.float64, device="cuda")
                    for h in s.get("hs", [s.get("h")])]
        torch.cuda.synchronize()
    return s


def _ecut(case, tau):
    """The serving loop's local-energy cutoff, per electron."""
    return 0.2 / math.sqrt((case["up"] + case["down"]) * tau)


# ----------------------------------------------------------- one pass
def run(s):
    kind, nw = s["kind"], s["walkers"]
    if kind == "eval":
        if s["host"]:
            return list(s["h"].compute_properties(s["x"]))
        s["h"].compute_properties_dev(nw, s["x"].data_ptr(), *(o.data_ptr() for o in s["out"]))
        s["h"].compute_properties_dev_status(nw)
        return s["out"]
    if kind == "batch":
        for h in s["hs"]:
            h.block_reset()
        s["batch"].dmc(s["steps"], s["tau"], s["etrial"])
        return [_block(h) + _records(h, s["slots"], r) for h, r in zip(s["hs"], s["rec"])]
    h = s["h"]
    h.block_reset()
    if kind == "vmc":
        h.vmc(s["steps"], s["tau"], 50)
    elif kind == "dmc":
        h.dmc(s["steps"], 1, s["tau"], s["etrial"], 2.0, 50)
    elif kind == "single":
        h.vmc_single(s["steps"], s["tau"], 50)
    else:  # the reptiles stay on the device; a block reads its sums
        h.rmc(s["steps"])
        return _block(h) + [h.counters()]
    return _block(h) + _records(h, s["slots"], s["rec"][0])


def _block(h):
    blk, norm = h.block_get()
    return [blk, norm]


def _records(h, slots, rec):
    h.records_pack(slots, rec.data_ptr())
    return [rec]


# ----------------------------------------------- what a pass cannot do without
def _pair_flops(case):
    """Pair sums of one configuration: geometry, the u2 and v2 splines, the
    u3 sums and their second pass, the backflow sums; and rho_k."""
    n = case["up"] + case["down"]
    k = max(60, n // 2)
    per = 16 + 32 + 12 + (110 if case["u3"] else 0) + (40 if case["bf"] else 0)
    return 0.5 * n * (n - 1) * per + 7.0 * n * k


def _det_flops(case):
    """Determinants of one configuration, per spin of m orbitals: the inverse
    (8 m^3), and either the drift and Laplacian from its diagonals, or with
    backflow F_x and F_y (16 m^3), the symmetric cross term (8 n m^2) and the
    Jacobian columns (60 n m)."""
    n = case["up"] + case["down"]
    f = 0.0
    for m in (case["up"], case["down"]):
        f += 8.0 * m ** 3 + 12.0 * m * m
        f += 16.0 * m ** 3 + 8.0 * n * m * m + 60.0 * n * m if case["bf"] else 20.0 * m * m
    return f


def work(case):
    if case["kind"] == "batch":
        parts = [work(dict(case, kind="dmc", up=u, down=d)) for u, d in BATCH_SHELLS]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, nw = case["up"] + case["down"], case["walkers"]
    nt = 2 if case["down"] else 1
    props = 8 + 3 * nt + 2 * nt * max(60, n // 2)
    record = 8.0 * (4 * n + nt + props + 2)
    if case["kind"] == "eval":
        return {"bytes": nw * (record + 16.0 * n), "flops": nw * (_pair_flops(case) + _det_flops(case))}
    moves = float(nw) * case["steps"]
    if case["kind"] == "single":
        # per move: orbitals, drifts, ratio and rank-one update, partners;
        # per sweep: the measurement from the resident inverse
        per = sum(m * (16.0 * m * m + 80.0 * m + 24.0 * n) for m in (case["up"], case["down"]))
        per += _pair_flops(case) + 40.0 * (case["up"] ** 2 + case["down"] ** 2)
        return {"bytes": 2 * nw * record, "flops": moves * per}
    flops = moves * (_pair_flops(case) + _det_flops(case))
    if case["kind"] == "rmc":  # a grown bead reads its neighbour and is written
        return {"bytes": 2 * moves * record, "flops": flops}
    return {"bytes": 2 * nw * record, "flops": flops}


# ------------------------------------------------- the evaluation in 64 bits
def _rows(path):
    """A spline table file: its rows, knot spacing and k-space list."""
    with open(path) as fh:
        lines = fh.read().splitlines()
    nt, drt = int(lines[0].split()[0]), float(lines[0].split()[1])
    rows = np.array([[float(v) for v in ln.split()] for ln in lines[1:nt + 2]])
    vk = []
    if any(ln.strip() == "kspace" for ln in lines):
        at = [ln.strip() for ln in lines].index("kspace")
        vk = [float(v) for v in lines[at + 2:at + 2 + int(lines[at + 1])]]
    return rows, drt, vk


def exact(case, seed):
    """compute_properties of the configurations in plain torch, FP64: -ln psi
    of u2, u3 and the backflow determinants, its gradient and Laplacian, the
    Ewald energy and rho_k. Chains have no such value: which moves are made
    is drawn from the library's own random streams."""
    if case["kind"] != "eval":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def dbl(a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)

    ns = [m for m in (case["up"], case["down"]) if m]
    n, rs = sum(ns), case["rs"]
    side = math.sqrt(n * math.pi)
    with tempfile.TemporaryDirectory(prefix="qmc2d_cases_") as tmp:
        d = _deck(os.path.join(tmp, "c"), case)
        tab = {k: _rows(os.path.join(d, "c." + k))
               for k in ("u2", "b", "v") + (("u3",) if case["u3"] else ())}
        kv = dbl(np.loadtxt(os.path.join(d, "c.k")))
        with open(os.path.join(d, "c.sy")) as fh:
            v0 = [float(ln.split()[1]) for ln in fh if ln.split()[:1] == ["v0"]][0]
    drt = tab["u2"][1]
    vk = dbl(tab["v"][2])
    coef = {k: dbl(v[0]) for k, v in tab.items()}
    # plane waves: k = 0 and +-k, the shells in order
    g = torch.cat((torch.zeros(1, 2, dtype=torch.float64, device=dev), kv, -kv))
    g = g[torch.argsort((g * g).sum(1).round(decimals=9), stable=True)]
    spin = torch.cat([torch.full((m,), float(t), device=dev) for t, m in enumerate(ns)])
    out = [[], [], [], []]
    eye = torch.eye(n, dtype=torch.bool, device=dev)
    chunk = max(1, int(2e8 / (32 * n * n * (2 + n // 8))))
    for x in dbl(_start(case, seed)).reshape(-1, n, 2).split(chunk):
        w = x.shape[0]
        r = x[:, :, None] - x[:, None]
        r = r - side * torch.round(r / side)
        dist = torch.sqrt((r * r).sum(-1)).masked_fill(eye, 1.0)
        knot = (dist / drt).long()
        rm = dist / drt - knot

        def spline(kind):
            c = coef[kind][knot.clamp(0, coef[kind].shape[0] - 1)].masked_fill(
                eye[None, :, :, None], 0.0)
            f = c[..., 0] + rm * (c[..., 1] + rm * (c[..., 2] + rm * c[..., 3]))
            df = (c[..., 1] + rm * (2 * c[..., 2] + rm * 3 * c[..., 3])) / drt
            return f, df, (2 * c[..., 2] + 6 * rm * c[..., 3]) / drt ** 2

        u, du, ddu = spline("u2")
        ltf = 0.5 * u.sum((1, 2))
        grad = ((du / dist)[..., None] * r).sum(2)
        lap = (ddu + du / dist).sum(2)
        if case["u3"]:  # -1/2 sum_i |G_i|^2 and its pair part, G_i = sum_j xi r_ij
            t, dt, ddt = spline("u3")
            s, ds = (t * dist) ** 2, 2 * t * dist * (t + dist * dt)
            dds = 2 * (t + dist * dt) ** 2 + 2 * t * dist * (2 * dt + dist * ddt)
            ltf = ltf + 0.5 * s.sum((1, 2))
            grad = grad + ((ds / dist)[..., None] * r).sum(2)
            lap = lap + (dds + ds / dist).sum(2)
            big = (t[..., None] * r).sum(2)  # G
            eye2 = torch.eye(2, dtype=torch.float64, device=dev)
            mm = t[..., None, None] * eye2 + (dt / dist)[..., None, None] * (
                r[..., :, None] * r[..., None, :])
            dg = big[:, :, None] - big[:, None]
            ltf = ltf - 0.5 * (big * big).sum((1, 2))
            grad = grad - torch.einsum("wkjab,wkjb->wka", mm, dg)
            sk = mm.sum(2)
            lap = lap - ((ddt + 3 * dt / dist) * (r * dg).sum(-1)).sum(2) \
                - (sk * sk).sum((-1, -2)) - (mm * mm).sum((2, 3, 4))
        # backflow coordinates q_j and J[j, a, i, b] = d q_ja / d x_ib
        t, dt, ddt = spline("b")
        qx = x + (t[..., None] * r).sum(2)
        eye2 = torch.eye(2, dtype=torch.float64, device=dev)
        mm = t[..., None, None] * eye2 + (dt / dist)[..., None, None] * (
            r[..., :, None] * r[..., None, :])
        jac = -mm
        jac[:, torch.arange(n), torch.arange(n)] = eye2 + mm.sum(2)
        w2 = (3 * dt / dist + ddt)[..., None] * r  # second derivatives of eta r, summed
        lq = w2.clone()  # [j, i] = nabla_i^2 q_j
        lq[:, torch.arange(n), torch.arange(n)] = w2.sum(2)
        dgrad, dlap = torch.zeros_like(grad), torch.zeros_like(lap)
        logdet = torch.zeros_like(ltf)
        f0 = 0
        for m in ns:
            sl = slice(f0, f0 + m)
            gm = g[:m]
            a = torch.exp(1j * torch.einsum("kd,wjd->wkj", gm, qx[:, sl]))
            inv = torch.linalg.inv(a)
            logdet = logdet + torch.linalg.slogdet(a)[1]
            f = torch.stack([inv @ ((1j * gm[:, d])[:, None] * a) for d in (0, 1)], 1)  # w a l j
            d2 = torch.stack([-torch.einsum("wjk,k,wkj->wj", inv, (gm[:, p] * gm[:, o]).to(a.dtype),
                                            a).real for p in (0, 1) for o in (0, 1)], -1)
            fd = f.diagonal(dim1=-2, dim2=-1).real  # w a j
            js = jac[:, sl].movedim(3, 2)  # w j a i b
            dgrad = dgrad - torch.einsum("waj,wjaib->wib", fd, js)
            tmp = torch.einsum("wjac,wjcib->wjaib", d2.reshape(w, m, 2, 2), js)
            lpart = torch.einsum("waj,wjia->wi", fd, lq[:, sl]) + torch.einsum(
                "wjaib,wjaib->wi", js, tmp)
            # sum_{jk} Re[F_a(k,j) F_c(j,k)] J_ja J_kc
            mat = torch.einsum("wakj,wcjk->wajck", f, f).real.reshape(w, 2 * m, 2 * m)
            cols = js.movedim(2, 1).reshape(w, 2 * m, 2 * n)
            cross = (cols * (mat @ cols)).sum(1).reshape(w, n, 2).sum(2)
            dlap = dlap - (lpart - cross)
            f0 += m
        ltf = ltf - logdet
        on = (torch.exp(-2.0 * ltf) > 0.0).to(torch.float64)  # the reference's underflow return
        grad = grad + on[:, None, None] * dgrad
        lap = lap + on[:, None] * dlap
        rho = []
        for t in range(len(ns)):
            ph = torch.einsum("kd,wjd->wkj", kv, x[:, spin == t])
            rho.append(torch.stack((torch.cos(ph).sum(2), torch.sin(ph).sum(2)), 2))
        vs, _, _ = spline("v")
        pair = 0.5 * (vs / dist).sum(2)
        hl, pot, kin, un = [], [], [], []
        for t, m in enumerate(ns):
            pick = spin == t
            hl.append(lap[:, pick].sum(1))
            g2 = (grad[:, pick] ** 2).sum((1, 2))
            kin.append((hl[-1] - g2) / rs ** 2 / m)
            un.append(1.0 / torch.sqrt(g2))
            kpart = sum((vk * (rho[t] * o).sum(2)).sum(1) for o in rho)
            pot.append(pair[:, pick].sum(1) + kpart)
        pot0 = (sum(pot) + v0) / n
        kin0 = sum(k * m for k, m in zip(kin, ns)) / n
        e, one = pot0 + kin0, torch.ones_like(pot0)
        props = [e, ltf, 0 * one, pot0, kin0, e * e, one] + [p / m for p, m in zip(pot, ns)] \
            + kin + un + [0 * one]
        out[0].append(grad.reshape(w, -1))
        out[1].append(torch.stack(hl, 1))
        out[2].append(torch.cat([torch.stack(props, 1)] + [o.reshape(w, -1) for o in rho], 1))
        out[3].append(one[:, None])
    got = [torch.cat(o).cpu() for o in out]
    if case["host"]:
        got[3] = got[3][:, 0]
    return got
