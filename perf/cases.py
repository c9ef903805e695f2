"""Workloads whose speed is tracked, through the package's public entry points.

Three kinds of case, over the sizes of the test suite, the benchmark
configurations (workloads.py) and the range between them:
  forward   one shot on host arrays, `Context.forward` (what solve1D/2D/3D call);
  batch     many 2D shots over several models, `Batch` (what solve2D_batch runs);
  gradient  misfit and dJ/d(c²) of one or more shots of one model,
            `adjoint.misfit_gradient` / `misfit_gradient_shots`.
`exact` restates them in plain torch in float64 on dense arrays.
"""
import importlib
import math

import numpy as np
import torch

SPACING = 10.0  # m, every axis


def _pkg():
    return importlib.import_module("__graft_entry__").load_package()


def listed():
    return [
        # a 1D line: the smallest call, all launch latency
        dict(name="line_f64_1001", kind="forward", ndim=1, nx=1001, ny=1, nz=1, halo=20,
             freetop=False, prec="f64", nt=1500, nsrc=1, nrec=5, surface=False),
        # the reference's CPU-runnable 2D size, double precision, CPML on all sides
        dict(name="plane_f64_241", kind="forward", ndim=2, nx=241, ny=241, nz=1, halo=20,
             freetop=False, prec="f64", nt=1000, nsrc=1, nrec=21, surface=False),
        # the reference's surface-source test size: sources that snap onto the
        # Dirichlet row of the free top
        dict(name="plane_f64_surface", kind="forward", ndim=2, nx=422, ny=242, nz=1, halo=20,
             freetop=True, prec="f64", nt=1200, nsrc=6, nrec=40, surface=True),
        # an ordinary 2D survey line in single precision, ragged sizes
        dict(name="plane_f32_1573x787", kind="forward", ndim=2, nx=1573, ny=787, nz=1, halo=20,
             freetop=True, prec="f32", nt=1000, nsrc=1, nrec=384, surface=False),
        # a 2D grid larger than the GPU's on-chip memories
        dict(name="plane_f32_5210x2604", kind="forward", ndim=2, nx=5210, ny=2604, nz=1, halo=30,
             freetop=True, prec="f32", nt=300, nsrc=1, nrec=1000, surface=False),
        # the reference's 3D test size in double precision: mostly CPML nodes
        dict(name="volume_f64_101", kind="forward", ndim=3, nx=101, ny=101, nz=101, halo=20,
             freetop=False, prec="f64", nt=300, nsrc=1, nrec=4, surface=False),
        # an ordinary 3D model with ragged sizes in double precision
        dict(name="volume_f64_203x187x171", kind="forward", ndim=3, nx=203, ny=187, nz=171,
             halo=20, freetop=True, prec="f64", nt=300, nsrc=1, nrec=900, surface=False),
        # the headline benchmark's grid and receiver count
        dict(name="volume_f32_296", kind="forward", ndim=3, nx=296, ny=276, nz=296, halo=20,
             freetop=True, prec="f32", nt=600, nsrc=1, nrec=4096, surface=False),
        # the largest configuration's CPML grid
        dict(name="volume_f32_424", kind="forward", ndim=3, nx=424, ny=404, nz=424, halo=20,
             freetop=True, prec="f32", nt=300, nsrc=1, nrec=4096, surface=False),
        # a batch of shots over the six models of uneven size
        dict(name="batch_f32_six_models", kind="batch", models=6, shots_per_model=2, scale=1.0,
             halo=20, freetop=True, prec="f32", nt=500),
        # a 2D waveform-inversion gradient
        dict(name="gradient2d_f32_540x296", kind="gradient", ndim=2, nx=540, ny=296, nz=1,
             halo=20, freetop=True, prec="f32", nt=600, nsrc=1, nrec=120, surface=False,
             every=50, shots=1),
        # a 3D waveform-inversion gradient over two shots of one model
        dict(name="gradient3d_f32_232", kind="gradient", ndim=3, nx=232, ny=212, nz=232, halo=20,
             freetop=True, prec="f32", nt=150, nsrc=1, nrec=2304, surface=False, every=50,
             shots=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes over their logarithm, ragged, every kind, both
    precisions, free top on and off, interior and surface sources."""
    kind = rng.choice(["line", "plane", "plane", "plane", "volume", "volume", "volume", "batch",
                       "gradient2d", "gradient3d"])
    prec = rng.choice(["f32", "f64"])
    halo = rng.choice([10, 20, 20, 30])
    freetop = rng.random() < 0.7
    if kind == "line":
        return dict(kind="forward", ndim=1, nx=_log(rng, 120, 12000), ny=1, nz=1, halo=halo,
                    freetop=False, prec=prec, nt=_log(rng, 300, 3000), nsrc=rng.randint(1, 2),
                    nrec=rng.randint(1, 20), surface=False)
    if kind == "plane":
        nx = _log(rng, 100, 4000)
        ny = max(90, min(2060, int(nx * rng.uniform(0.4, 1.1))))
        return dict(kind="forward", ndim=2, nx=nx, ny=ny, nz=1, halo=halo, freetop=freetop,
                    prec=prec, nt=_log(rng, 150, 400 if nx > 1600 else 1500),
                    nsrc=rng.choice([1, 1, 2, 6]), nrec=_log(rng, 1, 400),
                    surface=freetop and rng.random() < 0.3)
    if kind == "volume":
        n = _log(rng, 90, 300 if prec == "f32" else 210)
        nx, ny, nz = (max(80, int(n * rng.uniform(0.85, 1.1))) for _ in range(3))
        return dict(kind="forward", ndim=3, nx=nx, ny=ny, nz=nz, halo=halo, freetop=freetop,
                    prec=prec, nt=rng.randint(100, 300), nsrc=rng.choice([1, 1, 4]),
                    nrec=_log(rng, 4, 4096), surface=freetop and rng.random() < 0.2)
    if kind == "batch":
        return dict(kind="batch", models=rng.randint(1, 6), shots_per_model=rng.randint(1, 4),
                    scale=round(rng.uniform(0.4, 1.0), 3), halo=halo, freetop=freetop, prec=prec,
                    nt=rng.randint(100, 500))
    if kind == "gradient2d":
        nx = _log(rng, 120, 1100)
        return dict(kind="gradient", ndim=2, nx=nx, ny=max(100, int(nx * rng.uniform(0.4, 1.0))),
                    nz=1, halo=halo, freetop=freetop, prec=prec, nt=rng.randint(200, 800),
                    nsrc=1, nrec=_log(rng, 20, 300), surface=False, every=rng.choice([25, 50]),
                    shots=rng.choice([1, 2]))
    n = _log(rng, 84, 210)
    nx, ny, nz = (max(80, int(n * rng.uniform(0.9, 1.1))) for _ in range(3))
    return dict(kind="gradient", ndim=3, nx=nx, ny=ny, nz=nz, halo=halo, freetop=freetop,
                prec="f32", nt=rng.randint(60, 150), nsrc=1, nrec=_log(rng, 100, 2304),
                surface=False, every=rng.choice([25, 50]), shots=rng.choice([1, 2]))


# ---- inputs -------------------------------------------------------------------

def _pinned(n):
    return torch.empty(max(int(n), 1), dtype=torch.float64,
                       pin_memory=torch.cuda.is_available()).numpy()


def _velocity(shape, rng):
    """1500 m/s plus a depth gradient (depth is the second axis), times
    1 + 5 % of a smooth random field (a few plane waves), in a pinned
    column-major array."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ndim = len(shape)
    depth_axis = min(1, ndim - 1)
    axes = [torch.arange(n, dtype=torch.float64, device=dev) for n in shape]
    view = [[1] * ndim for _ in range(ndim)]
    for a in range(ndim):
        view[a][a] = shape[a]
    noise = torch.zeros(shape, dtype=torch.float64, device=dev)
    for _ in range(4):
        term = torch.ones([1] * ndim, dtype=torch.float64, device=dev)
        for a in range(ndim):
            k, ph = 2 * math.pi / rng.uniform(30.0, 120.0), rng.uniform(0, 2 * math.pi)
            term = term * torch.sin(k * axes[a] + ph).reshape(view[a])
        noise += term / 4
    depth = (axes[depth_axis] * SPACING).reshape(view[depth_axis])
    slope = 2000.0 / (shape[depth_axis] * SPACING)
    vel = (1500.0 + slope * depth) * (1.0 + 0.05 * noise)
    flat = _pinned(vel.numel())
    torch.from_numpy(flat).copy_(vel.permute(*reversed(range(ndim))).reshape(-1))
    return flat.reshape(shape, order="F")


def _positions(case, rng, shot=0):
    """Source and receiver positions [m] on the nodes: sources spread along
    the first axis, receivers on a line (2D) or a square grid (3D) near the
    top, both inside the CPML."""
    ndim = case["ndim"]
    n = [case["nx"], case["ny"], case["nz"]][:ndim]
    h = case["halo"]
    lo, hi = h + 2, [x - h - 3 for x in n]
    top = 0 if case["freetop"] else h
    mid = [(lo + b) // 2 for b in hi]
    shift = int(rng.integers(-6, 7)) + 7 * shot
    src, rec = [], []
    for s in range(case["nsrc"]):
        x = lo + (hi[0] - lo) * (s + 1) // (case["nsrc"] + 1) + shift
        x = min(max(x, lo), hi[0])
        if ndim == 1:
            src.append([x])
        elif ndim == 2:
            src.append([x, 0 if case["surface"] else top + 9])
        else:
            src.append([x, 0 if case["surface"] else top + 9, mid[2]])
    m = case["nrec"]
    if ndim == 1:
        rec = [[min(max(src[0][0] + 5 * (r + 1), 1), n[0] - 2)] for r in range(m)]
    elif ndim == 2:
        rec = [[lo + (hi[0] - lo) * r // max(m - 1, 1), top + 5] for r in range(m)]
    else:
        side = max(1, math.isqrt(m - 1) + 1)
        for r in range(m):
            rec.append([lo + (hi[0] - lo) * (r % side) // max(side - 1, 1), top + 5,
                        lo + (hi[2] - lo) * (r // side) // max(side - 1, 1)])
    to_m = lambda q: [[SPACING * c for c in p] for p in q]  # noqa: E731
    return to_m(src), to_m(rec)


F0 = 12.0


def _setup(pkg, case, vel, rng, shot=0):
    src, rec = _positions(case, rng, shot)
    n = vel.shape
    srcs = pkg.Sources(src, [1.2 / F0] * len(src), [pkg.rickersource1D] * len(src), F0)
    return pkg.prepare([(x - 1) * SPACING for x in n], None, vel, srcs, pkg.Receivers(rec),
                       halo=case["halo"], freetop=case["freetop"], precision=case["prec"],
                       ppw=5.0, nt=case["nt"])


def _observed(s, rng):
    """Recorded data to fit: a direct arrival of each source at each receiver,
    slightly late, scaled to the amplitude of a modelled one."""
    p = s["problem"]
    t = np.arange(p.nt)[:, None] * p.dt
    d = np.linalg.norm((s["posrecs"] - s["possrcs"][:1]) * SPACING, axis=1)[None, :]
    x = (math.pi * F0 * (t - 1.2 / F0 - 1.02 * d / 1600.0)) ** 2
    amp = 2e-7 if p.ndim == 2 else 1e-9
    noise = rng.standard_normal((p.nt, p.nrec))
    return np.asfortranarray(amp * ((1 - 2 * x) * np.exp(-x) * 50.0 / (d + 50.0) + 0.01 * noise))


INTERIORS = ((512, 256), (768, 384), (1024, 512), (1536, 768), (2048, 1024), (1024, 1024))


def _batch_inputs(case, seed):
    pkg = _pkg()
    rng = np.random.default_rng(seed)
    models, shots = [], []
    h = case["halo"]
    for m in range(case["models"]):
        ix, iy = (max(64, int(v * case["scale"])) for v in INTERIORS[m])
        nx, ny = ix + 2 * h, iy + (h if case["freetop"] else 2 * h)
        models.append(((nx - 1) * SPACING, (ny - 1) * SPACING, _velocity((nx, ny), rng)))
        top = 0 if case["freetop"] else h
        rec = [[i * SPACING, (top + 3) * SPACING] for i in range(h + 1, nx - h, 8)]
        for k in range(case["shots_per_model"]):
            f0 = float(rng.uniform(8.0, 14.0))
            i = h + 1 + int((k + 0.5) * ix / case["shots_per_model"])
            shots.append((m, pkg.Sources([[i * SPACING, (top + 2) * SPACING]], [1.2 / f0],
                                         [pkg.rickersource1D], f0), pkg.Receivers(rec)))
    return pkg.prepare_batch(models, shots, nt=case["nt"], halo=h, freetop=case["freetop"],
                             precision=case["prec"], ppw=5.0)


def _inputs(case, seed):
    """Shot set-ups (prepare() dicts) and observed data of a forward or
    gradient case."""
    pkg = _pkg()
    rng = np.random.default_rng(seed)
    vel = _velocity(tuple((case["nx"], case["ny"], case["nz"])[:case["ndim"]]), rng)
    setups = [_setup(pkg, case, vel, rng, k) for k in range(case.get("shots", 1))]
    obs = [_observed(s, rng) for s in setups] if case["kind"] == "gradient" else None
    return setups, obs


def prepare(case, seed):
    pkg = _pkg()
    ctx = pkg.default_context(0)
    if case["kind"] == "batch":
        probs, vels, setups, idx = _batch_inputs(case, seed)
        b = pkg.Batch(ctx, probs, vels, setups, idx)
        if case["nt"] >= 100:
            b.autotune(20)
        return dict(case=case, batch=b, traces=[np.zeros((case["nt"], n), order="F")
                                                for n in b.shot_nrec])
    setups, obs = _inputs(case, seed)
    state = dict(case=case, ctx=ctx, setups=setups, obs=obs)
    if case["kind"] == "forward":
        p = setups[0]["problem"]
        shape = setups[0]["vel"].shape
        state["traces"] = _pinned(p.nt * p.nrec).reshape((p.nt, p.nrec), order="F")
        state["field"] = _pinned(math.prod(shape)).reshape(shape, order="F")
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.reset()
        b.run()
        return [b.traces(k, state["traces"][k]) for k in range(b.nshots)]
    if case["kind"] == "forward":
        s = state["setups"][0]
        state["ctx"].forward(s["problem"], s["vel"], s["coeffs"], s["possrcs"], s["dt2srctf"],
                             s["posrecs"], state["traces"], state["field"])
        return dict(traces=state["traces"], field=state["field"])
    adj = _pkg().adjoint
    if case["shots"] == 1:
        J, grad, traces = adj.misfit_gradient(state["setups"][0], state["obs"][0], case["every"],
                                              state["ctx"])
        return dict(misfit=J, grad=grad, traces=traces)
    J, grad = adj.misfit_gradient_shots(state["setups"], state["obs"], case["every"],
                                        state["ctx"])
    return dict(misfit=J, grad=grad)


# ---- the least work -----------------------------------------------------------

ON_CHIP = 126e6 + 148 * 227e3  # L2 and shared memory of one B200 [bytes]


def _step_work(n, ndim, halo, freetop, word):
    """(bytes, flops, bytes of state) of one time step of a grid of n nodes
    per axis: each field node read and written once per step (read p_t,
    p_{t-1}, fact; write p_{t+1}), each ψ and ξ entry read and written once."""
    nodes = math.prod(n[:ndim])
    band = 0
    for a in range(ndim):
        sides = 1 if (a == 1 and freetop) else 2
        band += sides * halo * nodes // n[a]
    return ((4 * nodes + 4 * band) * word, (4 * ndim + 3) * nodes + 14 * band,
            (3 * nodes + 2 * band) * word)


def work(case):
    """Inputs read once and outputs written once, on the device in the working
    precision; plus, for a grid whose state exceeds the on-chip memories, one
    pass over the state per time step. A gradient also steps the adjoint
    (λ_{t+1}, λ_{t+2}, fact, the stored p_t and the double gradient, read and
    written) and stores the forward fields once."""
    word = 8 if case["prec"] == "f64" else 4
    nt = case["nt"]
    if case["kind"] == "batch":
        tot_b = tot_f = 0.0
        h = case["halo"]
        for m in range(case["models"]):
            ix, iy = (max(64, int(v * case["scale"])) for v in INTERIORS[m])
            n = (ix + 2 * h, iy + (h if case["freetop"] else 2 * h))
            b, f, st = _step_work(n, 2, h, case["freetop"], word)
            nrec = len(range(h + 1, n[0] - h, 8))
            k = case["shots_per_model"]
            tot_f += k * nt * f
            tot_b += math.prod(n) * 8 + k * nt * (nrec + 1) * 8
            if st > ON_CHIP:
                tot_b += k * nt * b
        return dict(bytes=tot_b, flops=tot_f)
    n = (case["nx"], case["ny"], case["nz"])
    nodes = math.prod(n)
    b, f, st = _step_work(n, case["ndim"], case["halo"], case["freetop"] and case["ndim"] > 1,
                          word)
    shots = case.get("shots", 1)
    io = 2 * nodes * 8 + shots * nt * (case["nrec"] + case["nsrc"]) * 8
    if case["kind"] == "forward":
        return dict(bytes=io + (nt * b if st > ON_CHIP else 0), flops=nt * f)
    back = b + (word + 16) * nodes  # the step's transpose, p_t read, gradient read and written
    both = nt * (b + back) + 2 * nt * nodes * word if st > ON_CHIP else 2 * nt * nodes * word
    return dict(bytes=io + shots * both, flops=shots * nt * 3 * f)


# ---- the same in plain torch, float64 -----------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Exact:
    """The CPML time step on dense float64 arrays (nx, ny, nz)[:ndim]."""

    def __init__(self, s):
        p = self.p = s["problem"]
        self.dev, self.nd, self.h = _device(), p.ndim, p.halo
        self.shape = tuple((p.nx, p.ny, p.nz)[:p.ndim])
        self.d = (p.dx, p.dy, p.dz)[:p.ndim]
        to = lambda a, **k: torch.as_tensor(np.ascontiguousarray(a), device=self.dev, **k)  # noqa: E731
        self.stf = to(s["dt2srctf"])
        flat = lambda pos: to(np.ravel_multi_index(tuple((pos - 1).T), self.shape))  # noqa: E731
        self.src, self.rec = flat(s["possrcs"]), flat(s["posrecs"])
        h, self.sides = self.h, []
        for a in range(self.nd):
            blk = s["coeffs"][a * (8 * h + 4):(a + 1) * (8 * h + 4)]
            on, half = blk[:4 * h].reshape(4, h), blk[4 * h:].reshape(4, h + 1)
            view = [1] * self.nd
            view[a] = -1
            for side in range(2 if h > 0 else 0):
                c = [to(v).reshape(view) for v in (on[side], on[2 + side], half[side],
                                                   half[2 + side])]
                start = 0 if side == 0 else self.shape[a] - h - 2  # the band's first face
                self.sides.append((a, start, c))

    def zero_state(self):
        z = lambda a, m: torch.zeros([m if b == a else self.shape[b] for b in range(self.nd)],  # noqa: E731
                                     dtype=torch.float64, device=self.dev)
        psi = [z(a, self.h + 1) for a, _, _ in self.sides]
        xi = [z(a, self.h) for a, _, _ in self.sides]
        f = [torch.zeros(self.shape, dtype=torch.float64, device=self.dev) for _ in range(3)]
        return f, psi, xi

    def step(self, it, fact, before, pold, pcur, psi, xi):
        """(p_{t+1}, ψ, ξ); `before` is p_{t-2}, whose rim values p_{t+1} keeps."""
        nd = self.nd
        inner = tuple(slice(1, -1) for _ in range(nd))
        acc = torch.zeros([n - 2 for n in self.shape], dtype=torch.float64, device=self.dev)
        d2 = []
        for a in range(nd):
            q = pcur[tuple(slice(None) if b == a else slice(1, -1) for b in range(nd))]
            n = self.shape[a]
            d2.append((q.narrow(a, 2, n - 2) - 2 * q.narrow(a, 1, n - 2) + q.narrow(a, 0, n - 2))
                      / self.d[a] ** 2)
            acc = acc + d2[a]
        psi_new, xi_new = [], []
        for (a, start, (ao, bo, ah, bh)), ps, x in zip(self.sides, psi, xi):
            h, d = self.h, self.d[a]
            jump = (pcur.narrow(a, start + 1, h + 1) - pcur.narrow(a, start, h + 1)) / d
            ps = bh * ps + ah * jump
            # band nodes start + 1 .. start + h, between faces q - 1 and q
            dps = (ps.narrow(a, 1, h) - ps.narrow(a, 0, h)) / d
            cut = tuple(slice(None) if b == a else slice(1, -1) for b in range(nd))
            dd = torch.zeros_like(x)
            dd[cut] = d2[a].narrow(a, start, h)
            x = bo * x + ao * (dd + dps)
            acc.narrow(a, start, h).add_((dps + x)[cut])
            psi_new.append(ps)
            xi_new.append(x)
        new = before.clone()
        new[inner] = 2 * pcur[inner] - pold[inner] + fact[inner] * acc
        new = new.reshape(-1).index_add(0, self.src, self.stf[it]).reshape(self.shape)
        return new, psi_new, xi_new


def _exact_forward(s):
    E = _Exact(s)
    p = E.p
    fact = p.dt ** 2 * torch.as_tensor(np.ascontiguousarray(s["vel"]), device=E.dev) ** 2
    (before, old, cur), psi, xi = E.zero_state()
    traces = torch.zeros((p.nt, p.nrec), dtype=torch.float64, device=E.dev)
    with torch.no_grad():
        for it in range(p.nt):
            new, psi, xi = E.step(it, fact, before, old, cur, psi, xi)
            traces[it] = new.reshape(-1)[E.rec]
            before, old, cur = old, cur, new
    return traces.cpu().numpy(), cur.cpu().numpy()


def _exact_gradient(s, observed, segment):
    """(J, dJ/dc², traces) by autograd, segment by segment."""
    from torch.utils.checkpoint import checkpoint

    E = _Exact(s)
    p = E.p
    c2 = torch.as_tensor(np.ascontiguousarray(s["vel"]), device=E.dev) ** 2
    c2.requires_grad_(True)
    obs = torch.as_tensor(np.ascontiguousarray(observed), device=E.dev)
    f, psi, xi = E.zero_state()
    ns = len(psi)

    def advance(it0, it1, c2, *state):
        f, psi, xi = list(state[:3]), list(state[3:3 + ns]), list(state[3 + ns:])
        fact = p.dt ** 2 * c2
        rows = []
        for it in range(it0, it1):
            new, psi, xi = E.step(it, fact, *f, psi, xi)
            rows.append(new.reshape(-1)[E.rec])
            f = [f[1], f[2], new]
        return (torch.stack(rows), *f, *psi, *xi)

    state, rows = (*f, *psi, *xi), []
    for it in range(0, p.nt, segment):
        out = checkpoint(advance, it, min(it + segment, p.nt), c2, *state, use_reentrant=False)
        rows.append(out[0])
        state = out[1:]
    traces = torch.cat(rows)
    J = 0.5 * ((traces - obs) ** 2).sum()
    J.backward()
    grad = c2.grad.clone()
    edge = torch.ones_like(grad, dtype=torch.bool)
    edge[tuple(slice(1, -1) for _ in E.shape)] = False
    grad[edge] = 0.0
    return float(J), grad.cpu().numpy(), traces.detach().cpu().numpy()


def exact(case, seed):
    if not torch.cuda.is_available():
        return None
    if case["kind"] == "batch":
        if case["models"] * case["shots_per_model"] * case["nt"] > 6000:
            return None
        return [_exact_forward(s)[0] for s in _batch_inputs(case, seed)[2]]
    setups, obs = _inputs(case, seed)
    if case["kind"] == "forward":
        traces, field = _exact_forward(setups[0])
        return dict(traces=traces, field=field)
    nodes = case["nx"] * case["ny"] * case["nz"]
    segment = max(2, min(50, int(2e8 / nodes)))
    parts = [_exact_gradient(s, o, segment) for s, o in zip(setups, obs)]
    out = dict(misfit=sum(q[0] for q in parts), grad=sum(q[1] for q in parts))
    if case["shots"] == 1:
        out["traces"] = parts[0][2]
    return out
