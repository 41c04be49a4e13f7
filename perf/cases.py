"""Timed workloads of the framework, through its public Python entry points.

A case is a dict of plain values.  prepare() makes what a user's program holds
before the call (seeded fields on the GPU, the model, batch, string or
updater), run() makes one pass, exact() restates the same pass with torch's
complex128 FFTs, work() counts the bytes and operations a pass cannot do
without.

Kinds:
  model   a Model_AB solve started from given fields and run for `iters` SCFT
          iterations (the work of scft::relax between two records), then H and
          the residual are read
  grad    the adjoint: gradient of a density-target loss with respect to wA, wB
  stress  the adjoint: derivative of -ln Q with respect to the cell lengths
  solve   one propagator through the Updater interface (RQM4 / OS2 / ETDRK4)
  string  one string iteration of all images (SCFT of each, re-sampling)
  batch   one SCFT iteration of independent solves of uneven grids and Ns
"""
import math

import numpy as np
import torch

import polystring_b200 as ps

# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------


def _model(name, dim, grid, lengths, sA, sB, chiN, scft, iters, mde="RQM4", system=None, n_anderson=10,
           compressible=False, lam=0.1, lam_eta=5.0, pattern="waves", noise=0.1):
    Lx, Ly, Lz = grid
    a, b, c = (tuple(lengths) + (0.0, 0.0))[:3]
    if system is None:
        system = {1: "LAMELLAR", 2: "RECTANGULAR", 3: "ORTHORHOMBIC"}[dim]
    case = dict(kind="model", dim=dim, Lx=Lx, Ly=Ly, Lz=Lz, system=system, a=a, b=b, c=c, sA=sA, sB=sB, chiN=chiN,
                scft=scft, iters=iters, mde=mde, n_anderson=n_anderson, compressible=compressible, lam=lam,
                lam_eta=lam_eta, pattern=pattern, noise=noise)
    if name:
        case["name"] = name
    return case


def _as(case, kind, name=None):
    case = dict(case, kind=kind)
    case.pop("name", None)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest call: one SCFT iteration of the 1D lamellar melt of the
        # example configurations (64 points, Ms [51, 51], simple mixing)
        _model("lamella_1d", 1, (64, 1, 1), (4.0,), 51, 51, 30.0, "EM", 1),
        # 2D hexagonal melt on 64^2, Ns 100, simple mixing (benchmark configuration C1)
        _model("disk_2d", 2, (64, 64, 1), (4.0, 4.0), 31, 71, 20.0, "EM", 4, system="SQUARE"),
        # the string driver's own 128 x 352 grid with its compressible model, Ms [21, 21]
        _model("defect_2d", 2, (128, 352, 1), (8.0, 22.0), 21, 21, 18.0, "EM", 2, compressible=True, lam=0.05,
               lam_eta=20.0),
        # the 3D example with second-order splitting and Anderson mixing, 32^3
        _model("os2_3d", 3, (32, 32, 32), (4.0, 4.0, 4.0), 51, 51, 30.0, "Anderson", 2, mde="OS2", system="CUBIC"),
        # exponential time differencing on the 2D example, 32^2
        _model("etd_2d", 2, (32, 32, 1), (4.0, 4.0), 51, 51, 30.0, "Anderson", 1, mde="ETDRK4", system="SQUARE"),
        # an uneven 3D grid and cell, Ns 128 (configuration C4 is 48^3 of this cell)
        _model("cell_3d", 3, (48, 48, 48), (3.8, 4.0, 4.2), 39, 91, 22.0, "Anderson", 2, n_anderson=20, lam=0.05),
        # the headline solve: gyroid on 64^3, Ns 200, Anderson mixing over 20 fields (configuration C2)
        _model("gyroid_3d", 3, (64, 64, 64), (4.2, 4.2, 4.2), 71, 131, 25.0, "Anderson", 2, system="CUBIC",
               n_anderson=20, lam=0.05, pattern="gyroid"),
        # backward: loss gradient on the C4 cell, and the stress that a cell optimisation reads every solve
        _as(_model(None, 3, (48, 48, 48), (3.8, 4.0, 4.2), 39, 91, 22.0, "Anderson", 1), "grad", "gradient_3d"),
        _as(_model(None, 3, (32, 32, 32), (3.8, 4.0, 4.2), 31, 71, 22.0, "Anderson", 1), "stress", "stress_3d"),
        # one chain through the Updater interface, device tensors, an uneven grid
        _as(_model(None, 3, (48, 64, 32), (4.4, 4.8, 3.6), 51, 51, 20.0, "EM", 1), "solve", "propagator_3d"),
        # string method: 40 images of 128^2, Ns 128, three SCFT iterations each (configuration C3)
        dict(name="string_2d", kind="string", Lx=128, Ly=128, a=8.0, b=8.0, sA=46, sB=84, chiN=18.0, images=40,
             iters=3, mde="RQM4"),
        # twelve independent solves, diblocks and triblocks of three grids and three Ns (a sample of configuration C5)
        dict(name="batch_3d", kind="batch", diblocks=9, triblocks=3, grid0=32, grid1=48, grid2=64, scale=64,
             n_anderson=10),
    ]


def _pick(rng, values):
    return values[rng.randrange(len(values))]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


LINES_1D = (32, 48, 64, 96, 128, 192, 256)
LINES_2D = (16, 24, 32, 48, 64, 96, 128)
LINES_3D = (16, 24, 32, 48, 64)


def _drawn_model(rng, dims, mdes):
    dim = _pick(rng, dims)
    if dim == 1:
        grid = (_pick(rng, LINES_1D), 1, 1)
    elif dim == 2:
        grid = (_pick(rng, LINES_2D), _pick(rng, LINES_2D), 1)
    else:
        while True:
            grid = tuple(_pick(rng, LINES_3D) for _ in range(3))
            if rng.random() < 0.4:
                grid = (grid[0],) * 3
            if grid[0] * grid[1] * grid[2] >= 16 ** 3:
                break
    lengths = tuple(round(rng.uniform(3.5, 5.0) * max(1.0, n / 64.0), 3) for n in grid[:dim])
    mde = _pick(rng, mdes)
    # contour points of each block; Ms odd or even (Simpson or the closed fourth-order rule)
    Ns = _log_int(rng, 30, 200 if dim < 3 else 140)
    LA = max(8, min(Ns - 8, int(round(rng.uniform(0.2, 0.5) * Ns))))
    if mde == "ETDRK4":
        Ns, LA = min(Ns, 60), min(LA, 30)
    scft = _pick(rng, ("EM", "Anderson"))
    return _model(None, dim, grid, lengths, LA + 1, Ns - LA + 1, round(rng.uniform(12.0, 30.0), 3), scft,
                  rng.randint(1, 3), mde=mde, n_anderson=_pick(rng, (5, 10, 20)),
                  compressible=rng.random() < 0.25, lam=round(rng.uniform(0.05, 0.2), 3),
                  lam_eta=round(rng.uniform(2.0, 10.0), 3))


def draw(rng):
    u = rng.random()
    if u < 0.55:
        return _drawn_model(rng, (1, 2, 2, 3, 3), ("RQM4", "RQM4", "RQM4", "RQM4", "OS2", "ETDRK4"))
    if u < 0.72:
        return _as(_drawn_model(rng, (1, 2, 3, 3), ("RQM4", "RQM4", "OS2")), "solve")
    if u < 0.80:
        return _as(_drawn_model(rng, (2, 3), ("RQM4",)), "grad")
    if u < 0.88:
        return _as(_drawn_model(rng, (2, 3), ("RQM4",)), "stress")
    if u < 0.95:
        while True:
            Lx, Ly = _pick(rng, LINES_2D), _pick(rng, LINES_2D)
            images = _log_int(rng, 5, 40)
            if Lx * Ly * images <= 128 * 128 * 40:
                break
        Ns = rng.randint(40, 128)
        LA = int(round(rng.uniform(0.3, 0.5) * Ns))
        return dict(kind="string", Lx=Lx, Ly=Ly, a=round(rng.uniform(4.0, 8.0), 3), b=round(rng.uniform(4.0, 8.0), 3),
                    sA=LA + 1, sB=Ns - LA + 1, chiN=round(rng.uniform(14.0, 20.0), 3), images=images,
                    iters=rng.randint(1, 3), mde="RQM4")
    return dict(kind="batch", diblocks=rng.randint(2, 9), triblocks=rng.randint(0, 3), grid0=_pick(rng, (16, 24, 32)),
                grid1=_pick(rng, (32, 48)), grid2=_pick(rng, (32, 48, 64)), scale=rng.randint(40, 64),
                n_anderson=_pick(rng, (5, 10)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _shape(case):
    return (case["Lx"], case["Ly"], case["Lz"])


def _waves(shape, rng, pattern):
    """An ordered field of order one with one period per cell axis."""
    ax = [2.0 * np.pi * (np.arange(n) / n + rng.uniform()) for n in shape]
    x, y, z = np.meshgrid(*ax, indexing="ij")
    if pattern == "gyroid":
        return np.sin(x) * np.cos(y) + np.sin(y) * np.cos(z) + np.sin(z) * np.cos(x)
    f = np.cos(x)
    if shape[1] > 1:
        f = f + np.cos(y)
    if shape[2] > 1:
        f = f + np.cos(z)
    return f


def _fields(case, seed):
    shape = _shape(case)
    rng = np.random.default_rng(seed)
    g = _waves(shape, rng, case["pattern"])
    n = case["noise"] * rng.standard_normal((2,) + shape)
    return g + n[0], -g + n[1]


def _cell(case):
    return ps.make_cell(case["dim"], case["system"], case["a"], case["b"], case["c"])


def _lengths(case):
    return [case["a"], case["b"], case["c"]][:case["dim"]]


def _ds(case):
    return 1.0 / (case["sA"] - 1 + case["sB"] - 1)


def _string_fields(case, seed):
    """Images between a lamellar and a hexagonal field, each end with noise."""
    shape, m = (case["Lx"], case["Ly"], 1), case["images"]
    rng = np.random.default_rng(seed)
    x = (2.0 * np.pi * (np.arange(shape[0]) / shape[0] + rng.uniform()))[:, None, None]
    y = (2.0 * np.pi * (np.arange(shape[1]) / shape[1] + rng.uniform()))[None, :, None]
    lam = 2.0 * np.cos(x) + 0.0 * y
    hexa = (2.0 / 3.0) * (np.cos(x) + np.cos(y) + np.cos(x - y))
    t = (np.arange(m) / (m - 1.0))[:, None, None, None]
    n = 0.05 * rng.standard_normal((4,) + shape)
    wa = (1 - t) * (lam + n[0]) + t * (hexa + n[1])
    wb = (1 - t) * (-lam + n[2]) + t * (-hexa + n[3])
    return wa, wb


def _batch_specs(case, seed):
    """Plain parameters and fields of the batch's solves: the sizes follow from
    the case, block fractions, chi N and cells from the seed."""
    rng = np.random.default_rng(seed)
    grids = (case["grid0"], case["grid1"], case["grid2"])
    di, tri = [], []
    for k in range(case["diblocks"]):
        L, Ns = grids[k % 3], case["scale"] * (1, 2, 4)[(k // 3) % 3]
        LA = int(round(rng.uniform(0.25, 0.5) * Ns))
        di.append(dict(shape=(L, L, L), a=rng.uniform(3.5, 5.0), Ms=(LA + 1, Ns - LA + 1),
                       chiN=rng.uniform(12.0, 30.0), w=0.1 * rng.standard_normal((2, L, L, L))))
    for k in range(case["triblocks"]):
        L, Ns = grids[k % 3], 2 * case["scale"]
        LA, LB = int(round(rng.uniform(0.25, 0.4) * Ns)), int(round(rng.uniform(0.25, 0.4) * Ns))
        tri.append(dict(shape=(L, L, L), a=rng.uniform(3.5, 5.0), Ms=(LA + 1, LB + 1, Ns - LA - LB + 1),
                        chi=tuple(rng.uniform(12.0, 30.0, 3)), w=0.1 * rng.standard_normal((3, L, L, L))))
    return di, tri


class _View:
    """Device memory of a context as a CUDA array, for torch.as_tensor (which
    keeps the view, and with it the context that owns the memory, alive)."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3, "strides": None}


def _views(obj, names, shape):
    return {n: torch.as_tensor(_View(obj, obj.device_ptr(n), shape), device="cuda") for n in names}


def _new_model(case):
    return ps.ModelAB(case["dim"], _shape(case), _cell(case), (case["sA"], case["sB"]), case["chiN"],
                      lam=(case["lam"], case["lam"], case["lam_eta"]), mde=case["mde"], scft=case["scft"],
                      n_anderson=case["n_anderson"], compressible=case["compressible"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "string":
        shape, m = (case["Lx"], case["Ly"], 1), case["images"]
        wa, wb = _string_fields(case, seed)
        g = ps.StringAB(m, 2, shape, ps.make_cell(2, "RECTANGULAR", case["a"], case["b"]), (case["sA"], case["sB"]),
                        case["chiN"], mde=case["mde"], max_iter=case["iters"])
        g.set_images(wa, wb)
        return dict(kind=kind, obj=g, out=_views(g, ("wa", "wb", "phiA", "phiB"), (m,) + shape),
                    wa=torch.from_numpy(wa).cuda(), wb=torch.from_numpy(wb).cuda(),
                    stream=torch.cuda.ExternalStream(g.stream()))
    if kind == "batch":
        di, tri = _batch_specs(case, seed)
        na = case["n_anderson"]
        b = ps.BatchAB([dict(dim=3, shape=s["shape"], cell=ps.make_cell(3, "CUBIC", s["a"]), Ms=s["Ms"],
                             chiN=s["chiN"], scft="Anderson", n_anderson=na) for s in di],
                       [dict(dim=3, shape=s["shape"], cell=ps.make_cell(3, "CUBIC", s["a"]), Ms=s["Ms"],
                             chi=s["chi"], scft="Anderson", n_anderson=na) for s in tri])
        for k, s in enumerate(di + tri):
            b.set_fields(k, *s["w"])
        return dict(kind=kind, obj=b, diblocks=len(di), triblocks=len(tri))
    wA, wB = _fields(case, seed)
    if kind == "solve":
        n = case["sA"] + case["sB"] - 1
        cls = {"RQM4": ps.RQM4, "OS2": ps.PseudoSpectral}[case["mde"]]
        qs = torch.empty((n,) + _shape(case), dtype=torch.float64, device="cuda")
        qs[0] = 1.0
        return dict(kind=kind, obj=cls(_cell(case), *_shape(case), _ds(case)), w=torch.from_numpy(wA).cuda(), qs=qs)
    m = _new_model(case)
    s = dict(kind=kind, obj=m, wA=torch.from_numpy(wA).cuda(), wB=torch.from_numpy(wB).cuda(), iters=case["iters"],
             out=_views(m, ("wA", "wB", "phiA", "phiB"), _shape(case)))
    if kind == "grad":
        rng = np.random.default_rng(seed + 1000)
        s["gA"], s["gB"] = 0.1 * rng.standard_normal((2,) + _shape(case))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    kind, obj = state["kind"], state["obj"]
    if kind == "model":
        obj.set_fields(state["wA"], state["wB"])
        obj.update(state["iters"])
        return dict(state["out"], H=obj.H()[0], residual=obj.residual_error())
    if kind == "grad":
        obj.set_fields(state["wA"], state["wB"])
        gA, gB = obj.grad_w(state["gA"], state["gB"], 0.5)
        return dict(gA=gA, gB=gB, phiA=state["out"]["phiA"], phiB=state["out"]["phiB"])
    if kind == "stress":
        obj.set_fields(state["wA"], state["wB"])
        s = obj.stress()
        return dict(stress=s, phiA=state["out"]["phiA"], phiB=state["out"]["phiB"])
    if kind == "solve":
        return obj.solve(state["qs"], state["w"], stream=torch.cuda.current_stream().cuda_stream)
    if kind == "string":
        with torch.cuda.stream(state["stream"]):
            state["out"]["wa"].copy_(state["wa"])
            state["out"]["wb"].copy_(state["wb"])
        obj.iterate(1)
        return dict(state["out"], H=obj.H(), S=obj.S())
    # a batch goes on from its own fields, iteration after iteration
    obj.update(1)
    n, nd = state["diblocks"] + state["triblocks"], state["diblocks"]
    out = dict(H=np.array([obj.H(k)[0] for k in range(n)]))
    for k in range(n):
        out["phiA%d" % k] = obj.get(k, "phiA")
    for k in range(nd):
        out["wA%d" % k] = obj.get(k, "wA")
    for k in range(nd, n):
        out["wC%d" % k] = obj.get(k, "wC")
    return out


# ---------------------------------------------------------------------------
# the least work of one pass
# ---------------------------------------------------------------------------
def _sweep_work(M, Ns, chains, mde="RQM4"):
    """A propagator slice is written once and read once; a contour step takes
    three (RQM4), one (OS2) or four (ETDRK4) pairs of transforms of M points,
    5 M log2 M / 2 operations each for a real field, and a few operations a
    point."""
    pairs = {"RQM4": 3, "OS2": 1, "ETDRK4": 4}[mde]
    steps = chains * Ns * float(M)
    return 16.0 * steps, steps * (pairs * 5.0 * math.log2(M) + 6.0 * pairs + 2.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        di, tri = _batch_specs(case, 0)
        nb = nf = 0.0
        for s in di + tri:
            M, Ns = s["shape"][0] ** 3, sum(x - 1 for x in s["Ms"])
            b, f = _sweep_work(M, Ns, 2)
            nb, nf = nb + b + 40.0 * len(s["Ms"]) * M, nf + f + 4.0 * Ns * M
        return {"bytes": nb, "flops": nf}
    Ns = case["sA"] + case["sB"] - 2
    if kind == "string":
        M = case["Lx"] * case["Ly"] * case["images"]
        b, f = _sweep_work(case["Lx"] * case["Ly"], Ns, 2)
        n = case["images"] * case["iters"]
        return {"bytes": n * b + 48.0 * M, "flops": n * f + case["iters"] * 4.0 * Ns * M}
    M = case["Lx"] * case["Ly"] * case["Lz"]
    if kind == "solve":
        b, f = _sweep_work(M, Ns, 1, case["mde"])
        return {"bytes": b / 2 + 8.0 * M, "flops": f}
    b, f = _sweep_work(M, Ns, 2, case["mde"])
    if kind == "model":
        return {"bytes": case["iters"] * b + 48.0 * M, "flops": case["iters"] * (f + 4.0 * Ns * M)}
    # the reverse step advances the adjoint and needs the forward slice's
    # intermediate results: the forward chains, then a reverse sweep of each
    # (the stress: of one)
    back = 2.0 if kind == "grad" else 1.0
    return {"bytes": b + back * b / 2, "flops": f * (1.0 + back) + 4.0 * Ns * M}


# ---------------------------------------------------------------------------
# the same pass in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=_dev())


def _k2(shape, lengths):
    """|k|^2 on an orthogonal cell; lengths: tensors or numbers."""
    out = 0.0
    for d, l in enumerate(lengths):
        n = shape[d]
        i = torch.arange(n, dtype=torch.float64, device=_dev())
        r = torch.where(i < n // 2 + 1, i, n - i)
        view = [1, 1, 1]
        view[d] = n
        out = out + (2.0 * math.pi / l * r).square().reshape(view)
    return out


def _split(q, e, L):
    return torch.fft.ifftn(torch.fft.fftn(e * q, dim=(-3, -2, -1)) * L, dim=(-3, -2, -1)).real * e


def _step_fn(mde, w, k2, ds):
    """One contour step q -> q' of a block with field w."""
    if mde == "ETDRK4":
        return None
    e1 = torch.exp(-0.5 * ds * w)
    L1 = torch.exp(-ds * k2)
    if mde == "OS2":
        return lambda q: _split(q, e1, L1)
    e2, L2 = torch.exp(-0.25 * ds * w), torch.exp(-0.5 * ds * k2)
    return lambda q: (4.0 * _split(_split(q, e2, L2), e2, L2) - _split(q, e1, L1)) / 3.0


def _etd_tables(k2, ds, n=32):
    L = (-k2)[..., None].to(torch.complex128)
    r = torch.exp(1j * math.pi * (torch.arange(n, dtype=torch.float64, device=k2.device) + 0.5) / n)
    x = ds * L + r
    ex = torch.exp(x)
    mean = lambda f: ds * f.mean(-1).real  # noqa: E731
    return (torch.exp(-ds * k2), torch.exp(-0.5 * ds * k2), mean((torch.exp(x / 2.0) - 1.0) / x),
            mean((ex * (x * x - 3.0 * x + 4.0) - x - 4.0) / x ** 3), mean((ex * (x - 2.0) + x + 2.0) / x ** 3),
            mean((ex * (4.0 - x) - x * x - 3.0 * x - 4.0) / x ** 3))


def _propagate(mde, q0, w, k2, ds, n):
    """n + 1 slices of a block of n steps from its head."""
    qs = [q0]
    if mde == "ETDRK4":
        E, E2, Q, f1, f2, f3 = _etd_tables(k2, ds)
        F = lambda x: torch.fft.fftn(x, dim=(-3, -2, -1))  # noqa: E731
        R = lambda x: torch.fft.ifftn(x, dim=(-3, -2, -1)).real  # noqa: E731
        v = F(q0)
        for _ in range(n):
            Nv = F(-w * qs[-1])
            a = E2 * v + Q * Nv
            Na = F(-w * R(a))
            Nb = F(-w * R(E2 * v + Q * Na))
            Nc = F(-w * R(E2 * a + Q * (2.0 * Nb - Nv)))
            v = E * v + f1 * Nv + 2.0 * f2 * (Na + Nb) + f3 * Nc
            qs.append(R(v))
        return qs
    step = _step_fn(mde, w, k2, ds)
    for _ in range(n):
        qs.append(step(qs[-1]))
    return qs


def _weights(n):
    """Contour weights of a block of n steps: Simpson for an odd number of
    slices, else the closed fourth-order rule."""
    c = np.ones(n + 1)
    if n % 2 == 0:
        c[1:n:2], c[2:n - 1:2] = 4.0, 2.0
        return c / 3.0
    c[0] = c[n] = 9.0 / 24.0
    c[1] = c[n - 1] = 28.0 / 24.0
    c[2] = c[n - 2] = 23.0 / 24.0
    return c


def _densities(mde, ws, Ls, k2, ds):
    """Densities of the blocks and Q (per leading batch index)."""
    one = torch.ones_like(ws[0])
    head, fwd = one, []
    for w, n in zip(ws, Ls):
        fwd.append(_propagate(mde, head, w, k2, ds, n))
        head = fwd[-1][-1]
    Q = head.mean(dim=(-3, -2, -1), keepdim=True)
    head, phis = one, [None] * len(ws)
    for x in reversed(range(len(ws))):
        bwd = _propagate(mde, head, ws[x], k2, ds, Ls[x])
        head = bwd[-1]
        acc = 0.0
        for s, c in enumerate(_weights(Ls[x])):
            acc = acc + float(c) * fwd[x][s] * bwd[Ls[x] - s]
        phis[x] = acc * ds / Q
    return phis, Q


class _Mixer:
    """Anderson mixing of several fields with one set of coefficients."""

    def __init__(self, ws, n, lams):
        self.n, self.lams, self.k = n, lams, 0
        self.w, self.d = [[w] for w in ws], [[] for _ in ws]   # newest first

    def mix(self, targets):
        nf = len(targets)
        for x in range(nf):
            self.d[x].insert(0, targets[x] - self.w[x][0])
        nn = min(self.k, self.n)
        U, V = np.zeros((nn, nn)), np.zeros(nn)
        for x in range(nf):
            d0 = self.d[x][0]
            diffs = [d0 - self.d[x][j] for j in range(1, nn + 1)]
            for i in range(nn):
                V[i] += float((diffs[i] * d0).mean())
                for j in range(nn):
                    U[i, j] += float((diffs[i] * diffs[j]).mean())
        C = np.linalg.solve(U, V) if nn else []
        for x in range(nf):
            W, D = self.w[x][0].clone(), self.d[x][0].clone()
            for j in range(nn):
                W += float(C[j]) * (self.w[x][j + 1] - self.w[x][0])
                D += float(C[j]) * (self.d[x][j + 1] - self.d[x][0])
            self.w[x].insert(0, W + (1.0 - self.lams[x] ** (self.k + 1)) * D)
            del self.w[x][self.n + 1:], self.d[x][self.n + 1:]
        self.k += 1
        return [w[0] for w in self.w]


def _mean(x):
    return float(x.mean())


def _exact_model(case, wA, wB):
    shape, ds = _shape(case), _ds(case)
    k2 = _k2(shape, _lengths(case))
    Ls, chiN, le = (case["sA"] - 1, case["sB"] - 1), case["chiN"], case["lam_eta"]
    comp, lam = case["compressible"], case["lam"]
    eta = torch.zeros_like(wA)
    mixer = _Mixer([wA, wB], case["n_anderson"], [lam, lam]) if case["scft"] == "Anderson" else None
    for _ in range(case["iters"]):
        (pA, pB), Q = _densities(case["mde"], (wA, wB), Ls, k2, ds)
        if mixer:
            eta = le * (pA + pB - 1.0) if comp else 0.5 * (wA + wB - chiN)
            wA0, wB0 = wA, wB
            wA, wB = mixer.mix([chiN * pB + eta, chiN * pA + eta])
            dA, dB = mixer.d[0][0], mixer.d[1][0]
            res = math.sqrt((_mean(dA * dA) + _mean(dB * dB)) / (_mean(wA0 * wA0) + _mean(wB0 * wB0)))
        else:
            eta = le * (pA + pB - 1.0) + (0.0 if comp else eta)
            tA, tB = chiN * pB + eta, chiN * pA + eta
            wA, wB = wA * (1.0 - lam) + lam * tA, wB * (1.0 - lam) + lam * tB
            res = _mean((tA - wA).abs()) / (_mean(wA.abs()) + _mean(tA.abs()))
            res += _mean((tB - wB).abs()) / (_mean(wB.abs()) + _mean(tB.abs()))
            s = pA + pB
            res = res / 2.0 if comp else (res + _mean((s - 1.0).abs()) / (1.0 + _mean(s.abs()))) / 3.0
    h = chiN * pA * pB - wA * pA - wB * pB
    if comp:
        h = h + 0.5 * le * (pA + pB - 1.0) ** 2
    return dict(wA=wA, wB=wB, phiA=pA, phiB=pB, H=_mean(h) - math.log(float(Q)), residual=res)


def _spline(y, S):
    """Natural cubic spline through (S, y) (images first), at z / (m - 1)."""
    m = len(S)
    h = np.diff(S)
    A = np.zeros((m, m))
    A[0, 0] = A[m - 1, m - 1] = 1.0
    R = np.zeros((m, m))
    for j in range(1, m - 1):
        A[j, j - 1], A[j, j], A[j, j + 1] = h[j - 1] / 3.0, 2.0 * (h[j - 1] + h[j]) / 3.0, h[j] / 3.0
        R[j, j - 1], R[j, j], R[j, j + 1] = 1.0 / h[j - 1], -1.0 / h[j - 1] - 1.0 / h[j], 1.0 / h[j]
    flat = y.reshape(m, -1)
    b = torch.linalg.solve(_t(A), _t(R) @ flat)
    out = torch.empty_like(flat)
    for z in range(m):
        t = z / (m - 1.0)
        k = min(max(int(np.searchsorted(S, t, side="left")) - 1, 0), m - 2)
        u, hk = t - S[k], h[k]
        a = (b[k + 1] - b[k]) / (3.0 * hk)
        c = (flat[k + 1] - flat[k]) / hk - (2.0 * b[k] + b[k + 1]) * hk / 3.0
        out[z] = ((a * u + b[k]) * u + c) * u + flat[k]
    return out.reshape(y.shape)


def _exact_string(case, wa0, wb0):
    k2 = _k2((case["Lx"], case["Ly"], 1), (case["a"], case["b"]))
    Ls, chiN, lam, le, ds = (case["sA"] - 1, case["sB"] - 1), case["chiN"], 0.05, 5.0, _ds(case)
    wa, wb, eta = wa0, wb0, torch.zeros_like(wa0)
    for _ in range(case["iters"]):
        (pA, pB), Q = _densities(case["mde"], (wa, wb), Ls, k2, ds)
        eta = eta + le * (pA + pB - 1.0)
        wa = wa * (1.0 - lam) + lam * (chiN * pB + eta)
        wb = wb * (1.0 - lam) + lam * (chiN * pA + eta)
    H = (chiN * pA * pB - wa * pA - wb * pB).mean(dim=(1, 2, 3)) - torch.log(Q.reshape(-1))
    step = (wa[1:] - wa[:-1]).square().mean(dim=(1, 2, 3)).sqrt().cpu().numpy()
    S = np.concatenate([[0.0], np.cumsum(step)])
    S /= S[-1]
    na, nb = _spline(wa, S), _spline(wb, S)
    na[0], na[-1], nb[0], nb[-1] = wa0[0], wa0[-1], wb0[0], wb0[-1]
    return dict(wa=na, wb=nb, phiA=pA, phiB=pB, H=H.cpu().numpy(), S=S)


def _exact_batch(case, seed):
    di, tri = _batch_specs(case, seed)
    out, Hs = {}, []
    for k, s in enumerate(di + tri):
        ws = [_t(w) for w in s["w"]]
        Ls = [x - 1 for x in s["Ms"]]
        phi, Q = _densities("RQM4", ws, Ls, _k2(s["shape"], (s["a"],) * 3), 1.0 / sum(Ls))
        if len(ws) == 2:
            eta = 0.5 * (ws[0] + ws[1] - s["chiN"])
            tgt = [s["chiN"] * phi[1] + eta, s["chiN"] * phi[0] + eta]
            h = s["chiN"] * phi[0] * phi[1]
        else:
            ab, bc, ac = s["chi"]
            mix = [ab * phi[1] + ac * phi[2], ab * phi[0] + bc * phi[2], ac * phi[0] + bc * phi[1]]
            eta = (ws[0] + ws[1] + ws[2] - mix[0] - mix[1] - mix[2]) / 3.0
            tgt = [x + eta for x in mix]
            h = ab * phi[0] * phi[1] + bc * phi[1] * phi[2] + ac * phi[0] * phi[2]
        # the first Anderson step has no history: w + (1 - lambda) d, lambda 0.05
        ws = [w + 0.95 * (t - w) for w, t in zip(ws, tgt)]
        for w, p in zip(ws, phi):
            h = h - w * p
        Hs.append(_mean(h) - math.log(float(Q)))
        out["phiA%d" % k] = phi[0].cpu().numpy()
        if len(ws) == 2:
            out["wA%d" % k] = ws[0].cpu().numpy()
        else:
            out["wC%d" % k] = ws[2].cpu().numpy()
    out["H"] = np.array(Hs)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "string":
        return _exact_string(case, *[_t(w) for w in _string_fields(case, seed)])
    wA, wB = [_t(w) for w in _fields(case, seed)]
    shape, ds, n = _shape(case), _ds(case), case["sA"] + case["sB"] - 2
    if kind == "solve":
        return torch.stack(_propagate(case["mde"], torch.ones_like(wA), wA, _k2(shape, _lengths(case)), ds, n))
    if kind == "model":
        return _exact_model(case, wA, wB)
    Ls = (case["sA"] - 1, case["sB"] - 1)
    lengths = [torch.tensor(float(l), dtype=torch.float64, device=_dev(), requires_grad=kind == "stress")
               for l in _lengths(case)]
    wA.requires_grad_(kind == "grad")
    wB.requires_grad_(kind == "grad")
    (pA, pB), Q = _densities("RQM4", (wA, wB), Ls, _k2(shape, lengths), ds)
    if kind == "grad":
        rng = np.random.default_rng(seed + 1000)
        gA, gB = 0.1 * rng.standard_normal((2,) + shape)
        ((pA * _t(gA)).sum() + (pB * _t(gB)).sum() + 0.5 * Q.sum()).backward()
        return dict(gA=wA.grad, gB=wB.grad, phiA=pA.detach(), phiB=pB.detach())
    (-torch.log(Q.sum())).backward()
    g = [float(l.grad) for l in lengths]
    return dict(stress=np.array(g + [0.0] * (3 - len(g))), phiA=pA.detach(), phiB=pB.detach())
