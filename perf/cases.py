"""The work users give this framework, as cases whose passes can be timed.

A case is one call sequence of a user's program on one solver context:

* "forward": one forward step of a batch of teleseismic events -- solve,
  receiver times, rays and Frechet rows -- through ``Solver.forward_device``
  (api "device": everything stays in HBM, the tomography loop) or
  ``Solver.forward_into`` (api "host": the program's own host arrays in and
  out, as the file driver calls it); with "update", the velocity model is set
  anew first, as every tomography iteration does;
* "times": plane-wave requests of one grid and their receiver times, what
  the serving loop does for a batch of teleseismic requests;
* "point": local point sources with a refined source grid and their receiver
  times, the serving loop's other kind of request;
* "rays": rays and Frechet rows through fields solved before, as a study
  that moves its receivers calls them.

Inputs are synthetic and made from the seed: a 400 km x 10 deg x 10 deg
section with a 5.8 to 8.9 km/s gradient and node perturbations, plane waves of
distance 30 to 90 degrees from all azimuths, surface receivers.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parallel-fast-marching-method_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

PI = float(np.float32(3.1415926535898))      # the program's angles are converted with this value
EARTH = 6371.0
ROW_ENTRIES_PER_LAYER = 20                   # Frechet entries of a row, per velocity layer (about)


def _case(name, kind, nn, nv, model, nev, nrc, precision="f32", **more):
    c = {"name": name, "kind": kind, "nnr": nn[0], "nnx": nn[1], "nnz": nn[2], "nvr": nv[0], "nvx": nv[1],
         "nvz": nv[2], "model": model, "nev": nev, "nrc": nrc, "precision": precision}
    c.update(more)
    return c


def listed():
    small, large = (12, 14, 14), (16, 20, 20)
    return [
        # a service's smallest teleseismic request, alone on its grid
        _case("request 64", "times", (64, 64, 64), small, "gauss", 1, 100),
        # a few requests that came while the grid was busy; odd edge
        _case("requests 97", "times", (97, 97, 97), small, "gauss", 3, 100),
        # the service's largest grid, a full batch
        _case("requests 256", "times", (256, 256, 256), small, "gauss", 8, 100),
        # local earthquakes with the 5x refined source grid
        _case("local 96", "point", (96, 96, 96), small, "gauss", 2, 100, refine=5, extent=4),
        # the plain drop-in of the reference program: one event, double precision, host arrays
        _case("plain 64 f64", "forward", (64, 64, 64), small, "checker", 1, 100, "f64", api="host"),
        # the same on the tomography grid: an oblique event and one along a grid axis
        _case("plain 192x224x224 f64", "forward", (192, 224, 224), large, "checker", 2, 100, "f64", api="host"),
        # a double-precision batch
        _case("batch 128 f64", "forward", (128, 128, 128), small, "gauss", 32, 300, "f64", api="device"),
        # a single-precision batch, the throughput workload on a smooth model
        _case("batch 128", "forward", (128, 128, 128), small, "gauss", 256, 300, api="device"),
        # a model with a sharp slow slab on the largest grid, one of a set of models that are tried
        _case("slab 256", "forward", (256, 256, 256), large, "slab", 8, 300, api="device", update=True),
        # first order on an odd grid whose rows are no multiple of 16 bytes, with gaps in the boundary times
        _case("first order 75x91x83", "forward", (75, 91, 83), small, "gauss", 12, 60, api="device", fom=0,
              holes=0.02),
        # a full tomography iteration's forward step, the checkerboard partly recovered (the schedule tuned as for
        # such models)
        _case("tomography 192x224x224", "forward", (192, 224, 224), large, "checker", 500, 300, api="device",
              update=True, contrast=0.03, shape=1, tie_sweeps=6, tie_ratio=0.2),
        # rays alone, through double-precision fields
        _case("rays 96x112x112 f64", "rays", (96, 112, 112), large, "checker", 8, 300, "f64"),
    ]


def _splits_evenly(nnr):
    """Whether every power-of-two number of height segments down to eight
    layers each is used in full: a sweep may split the height so, and no
    grid on which a segment would be left empty stands for real use."""
    n, ok = 1, True
    while n <= max(1, nnr // 8):
        size = -(-nnr // n)
        ok = ok and -(-nnr // size) == n
        n *= 2
    return ok


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def height(lo, hi):
        while True:
            n = logint(lo, hi)
            if _splits_evenly(n):
                return n

    kind = rng.choice(["times", "times", "point", "forward", "forward", "forward", "forward", "rays"])
    f64 = kind in ("forward", "rays") and rng.random() < 0.4
    model = rng.choice(["checker", "gauss", "slab"]) if kind == "forward" else "gauss"
    if kind in ("times", "point"):
        n = height(64, 256) if kind == "times" else height(64, 128)
        nn, nv = (n, n, n), (12, 14, 14)
    else:
        nn = (height(40, 224), logint(40, 224), logint(40, 224))
        nv = rng.choice([(12, 14, 14), (16, 20, 20), (9, 11, 13)])
    nodes = nn[0] * nn[1] * nn[2]
    # (well within the listed tomography step's nodes; double precision and
    # rough models cost more for each)
    room = {"times": 2e8, "point": 1e7, "rays": 3e7}.get(kind, {"gauss": 1.2e9, "checker": 1e9, "slab": 1e8}[model])
    if f64:
        room = min(room, 2e7 if model != "gauss" else 6e7)
    nev = max(1, min(logint(1, 500 if kind == "forward" else 32), int(room / nodes), 4 if kind == "point" else 500))
    nrc = logint(20, 400 if kind != "point" else 200)
    c = _case("drawn", kind, nn, nv, model, nev, nrc, "f64" if f64 else "f32")
    del c["name"]
    if model == "checker":
        c["contrast"] = rng.choice([0.03, 0.05]) if f64 else 0.03
    if kind == "forward":
        c["api"] = rng.choice(["device", "device", "host"]) if nev * nrc <= 2000 else "device"
        c["update"] = rng.random() < 0.5
        c["fom"] = 0 if rng.random() < 0.2 else 1
        c["holes"] = 0.02 if rng.random() < 0.2 else 0.0
    if kind == "point":
        c.update(refine=rng.choice([0, 3, 5]), extent=rng.choice([3, 4]))
    return c


# --- inputs -----------------------------------------------------------------

def _inputs(case, seed):
    """Geometry, velocity nodes, events and receivers of a case (numpy)."""
    rng = np.random.default_rng([int(seed), case["nnr"], case["nnx"], case["nnz"], case["nev"]])
    nn = (case["nnr"], case["nnx"], case["nnz"])
    nv = (case["nvr"], case["nvx"], case["nvz"])
    step = (400.0 / (nn[0] - 1), 10.0 / (nn[1] - 1), 10.0 / (nn[2] - 1))
    orig = (0.0, -30.0, 140.0)               # height km, latitude, longitude of the first node
    # the velocity nodes' splines cover the grid and its ghost layer
    m = 2.05
    vorig = (orig[0] + m * step[0], orig[1] + m * step[1], orig[2] - m * step[2])
    vstep = tuple((n + m) * d / (v - 1.5) for n, d, v in zip(nn, step, nv))
    depth = (np.arange(nv[0] + 2) - 1.0) * vstep[0] - vorig[0]
    iz, ix, ir = np.meshgrid(np.arange(nv[2] + 2), np.arange(nv[1] + 2), np.arange(nv[0] + 2), indexing="ij")
    v = np.broadcast_to(5.8 + 3.1 * depth / 400.0, ix.shape).copy()
    if case["model"] == "checker":
        v *= (1.0 + case.get("contrast", 0.05) * np.where((iz // 3 + ix // 3 + ir // 3) % 2 == 0, 1.0, -1.0)
              + rng.normal(0.0, 1e-3, v.shape))
    elif case["model"] == "gauss":
        v *= 1.0 + np.clip(rng.normal(0.0, 0.015, v.shape), -0.03, 0.03)
    else:                                    # a slow slab dipping 45 degrees, and node noise
        x = (ix - 0.5 * (nv[1] + 1)) * vstep[1] * math.pi / 180.0 * EARTH
        v *= 1.0 - 0.10 * (np.abs(depth[ir] - x - 100.0) < 42.0)
        v *= 1.0 + np.clip(rng.normal(0.0, 0.01, v.shape), -0.02, 0.02)
    nev = case["nev"]
    dist = rng.uniform(30.0, 90.0, nev)
    # All round the circle, but for the four degrees either side of the grid's
    # axes: there the mixed-order update can end in a cycle of last bits,
    # which the solver reports as no convergence (about one event in 10,000).
    if nev <= 2:                             # an oblique event, and one near an axis
        baz = np.array([45.0, 276.0])[:nev] + rng.uniform(-2.0, 2.0, nev)
    else:
        quarter, deg = np.divmod((np.arange(nev) + rng.uniform(0.0, 1.0, nev)) * 360.0 / nev, 90.0)
        baz = 90.0 * quarter + 4.0 + deg * 82.0 / 90.0
    rb = EARTH + orig[0] - (nn[0] - 1) * step[0]
    az = np.radians(baz + 180.0)
    params = np.stack([150.0 + 10.0 * dist - 0.025 * dist ** 2, (10.0 - 0.05 * dist) / math.radians(rb),
                       np.cos(az), np.sin(az)], axis=1)
    nrc = case["nrc"]
    lat = rng.uniform(orig[1] - (nn[1] - 2) * step[1], orig[1] - step[1], nrc)
    lon = rng.uniform(orig[2] + step[2], orig[2] + (nn[2] - 2) * step[2], nrc)
    rec = (np.zeros(nrc), (90.0 - lat) * PI / 180.0, lon * PI / 180.0)
    src = np.stack([-rng.uniform(5.0, 30.0, nev),
                    (90.0 - orig[1] + rng.uniform(6, nn[1] - 7, nev) * step[1]) * PI / 180.0,
                    (orig[2] + rng.uniform(6, nn[2] - 7, nev) * step[2]) * PI / 180.0], axis=1)
    unset = rng.uniform(0.0, 1.0, (nev, nn[1], nn[2])) < case.get("holes", 0.0)
    return {"nn": nn, "nv": nv, "orig": orig, "step": step, "vorig": vorig, "vstep": vstep,
            "velv": np.ascontiguousarray(v.reshape(-1)), "params": params, "rec": rec, "src": src, "unset": unset}


def _frames(inp, device):
    """Boundary frames of the plane waves (float64, nev x nnx x nnz): times at
    the bottom nodes from their tangent-plane distances; 0 where unset."""
    nn, orig, step = inp["nn"], inp["orig"], inp["step"]
    th0, ph0 = (90.0 - orig[1]) * PI / 180.0, orig[2] * PI / 180.0
    dx, dz = step[1] * PI / 180.0, step[2] * PI / 180.0
    rb = EARTH + (orig[0] - (nn[0] - 1) * step[0])
    thc, phc = th0 + (nn[1] - 1) * dx * 0.5, ph0 + (nn[2] - 1) * dz * 0.5
    f = dict(dtype=torch.float64, device=device)
    dn = rb * (thc - (th0 + torch.arange(nn[1], **f) * dx))
    de = rb * math.sin(thc) * (ph0 + torch.arange(nn[2], **f) * dz - phc)
    p = torch.tensor(inp["params"], **f)[:, :, None, None]
    t = p[:, 0] + p[:, 1] * (dn[None, :, None] * p[:, 2] + de[None, None, :] * p[:, 3])
    return torch.where(torch.from_numpy(inp["unset"]).to(device), torch.zeros_like(t), t).contiguous()


def prepare(case, seed):
    import fm3dt
    from fm3dt.synth import Header
    inp = _inputs(case, seed)
    nn, nv, nev, nrc = inp["nn"], inp["nv"], case["nev"], case["nrc"]
    h = Header(nv, inp["vorig"], inp["vstep"], nn, inp["orig"], inp["step"], EARTH)
    solver = fm3dt.Solver(h, fom=case.get("fom", 1), max_events=nev,
                          precision=fm3dt.FP64 if case["precision"] == "f64" else fm3dt.FP32_OFFSET)
    if "shape" in case:
        solver.set_tuning(case["shape"])
    if "tie_sweeps" in case:
        solver.set_schedule(case["tie_sweeps"], case["tie_ratio"])
    solver.set_velocity(inp["velv"])
    state = {"case": case, "solver": solver, "velv": inp["velv"], "rec": inp["rec"]}
    if case["kind"] == "times":
        state["params"] = inp["params"]
    elif case["kind"] == "point":
        state["src"] = inp["src"]
    else:
        rows = nev * nrc
        host = case.get("api") == "host"
        dev = "cpu" if host else "cuda"
        cap = rows * ROW_ENTRIES_PER_LAYER * (nv[0] + 2) * 2
        # (the rows' arrays are larger than the rows; what no row fills stays 0)
        state.update(frames=_frames(inp, "cuda").to(dev), cap=cap,
                     times=torch.zeros((nev, nrc), dtype=torch.float32, device=dev),
                     row_ptr=torch.zeros(rows + 1, dtype=torch.int64, device=dev),
                     cols=torch.zeros(cap, dtype=torch.int32, device=dev),
                     vals=torch.zeros(cap, dtype=torch.float32, device=dev))
        if not host:
            state["d_rec"] = torch.tensor(np.stack(inp["rec"]), device=dev)
            state["ends"] = torch.zeros((rows, 3), dtype=torch.float64, device=dev)
        torch.cuda.synchronize()             # (the solver's stream does not wait for torch's)
        if case["kind"] == "rays":
            solver.solve_ptr(nev, state["frames"].data_ptr(), True)
    return state


def run(state):
    case, s = state["case"], state["solver"]
    if case["kind"] == "times":
        s.solve_planewave(state["params"])
        return {"times": s.receiver_times(*state["rec"])}
    if case["kind"] == "point":
        s.solve_point(state["src"], case["refine"], case["extent"])
        return {"times": s.receiver_times(*state["rec"])}
    if case.get("update"):
        s.set_velocity(state["velv"])
    out = [state[k].data_ptr() for k in ("row_ptr", "cols", "vals")] + [state["cap"]]
    rec = [x.data_ptr() for x in state["d_rec"]] if "d_rec" in state else state["rec"]
    names = ["row_ptr", "cols", "vals"]
    if case["kind"] == "rays":
        n = s.rays_frechet_device(case["nrc"], *rec, *out, state["ends"].data_ptr())
        names += ["ends"]
    elif case["api"] == "host":
        n = s.forward_into(case["nev"], state["frames"].data_ptr(), *rec, state["times"].data_ptr(), *out)
        names += ["times"]
    else:
        _, n = s.forward_device(case["nev"], state["frames"].data_ptr(), case["nrc"], *rec,
                                state["times"].data_ptr(), *out, state["ends"].data_ptr())
        names += ["times", "ends"]
    return {"entries": n, **{k: state[k] for k in names}}


def work(case):
    """What a pass cannot do without: each node solved once (its slowness read
    once, its time written), the boundary in, receiver times and rows out."""
    nodes = case["nnr"] * case["nnx"] * case["nnz"]
    nev, rows = case["nev"], case["nev"] * case["nrc"]
    size = 8 if case["precision"] == "f64" else 4
    b = 4.0 * rows
    fl = 30.0 * rows
    if case["kind"] != "rays":
        # an update of the three upwind terms: the causal solves of their
        # seven subsets (four quadratics)
        b += size * nodes * (nev + 1)
        fl += 110.0 * nodes * nev
        if case["kind"] == "forward":
            b += 8.0 * nev * case["nnx"] * case["nnz"]
    if case["kind"] in ("forward", "rays"):
        b += rows * (8.0 * ROW_ENTRIES_PER_LAYER * case["nvr"] + 32.0)
        # a ray's steps: gradient, velocity, and the weights of 64 nodes
        fl += rows * case["nnr"] * 600.0
    if case.get("update"):
        b += 8.0 * nodes
        fl += 16.0 * nodes
    return {"bytes": b, "flops": fl}


# --- the same results in plain 64-bit torch --------------------------------

class _Grid:
    """A grid in solver units: node (r, theta, phi) i at org + i * step (r
    counted downward as a height)."""

    def __init__(self, nn, org, step):
        self.nn, self.org, self.step = nn, org, step

    def axes(self, dev):
        f = dict(dtype=torch.float64, device=dev)
        return (self.org[0] - torch.arange(self.nn[0], **f) * self.step[0],
                self.org[1] + torch.arange(self.nn[1], **f) * self.step[1],
                self.org[2] + torch.arange(self.nn[2], **f) * self.step[2])


def _rad(origin, step):
    return ((origin[0], (90.0 - origin[1]) * PI / 180.0, origin[2] * PI / 180.0),
            (step[0], step[1] * PI / 180.0, step[2] * PI / 180.0))


def _velocity(inp, grid, dev):
    """Cubic B-spline velocity at a grid's nodes (nnr, nnx, nnz)."""
    org, step = _rad(inp["vorig"], inp["vstep"])
    mats = []
    for a, x in enumerate(grid.axes(dev)):
        u = ((org[0] - x) if a == 0 else (x - org[a])) / step[a]
        i = torch.floor(u)
        u, i = u - i, i.long()
        w = [(1 - u) ** 3 / 6, (4 - 6 * u ** 2 + 3 * u ** 3) / 6, (1 + 3 * u + 3 * u ** 2 - 3 * u ** 3) / 6, u ** 3 / 6]
        m = torch.zeros((len(x), inp["nv"][a] + 2), dtype=torch.float64, device=dev)
        for k in range(4):
            m[torch.arange(len(x), device=dev), (i + k).clamp(0, inp["nv"][a] + 1)] += w[k]
        mats.append(m)
    v = torch.tensor(inp["velv"], device=dev).reshape(inp["nv"][2] + 2, inp["nv"][1] + 2, inp["nv"][0] + 2)
    v = torch.einsum("cba,kc->kba", v, mats[2])
    v = torch.einsum("kba,jb->kja", v, mats[1])
    return torch.einsum("kja,ia->ijk", v, mats[0]).contiguous()


def _octants(T, s, hx, hz, hr, order2):
    """One node update of every node from its neighbours (T padded by two
    unset nodes): the least over octants of the causal upwind solve."""
    n = s.shape
    inf = math.inf

    def at(a, k):
        o = [2, 2, 2]
        o[a] += k
        return T[o[0]:o[0] + n[0], o[1]:o[1] + n[1], o[2]:o[2] + n[2]]

    nb = [(at(a, d), at(a, 2 * d)) for a in range(3) for d in (-1, 1)]
    tmin = nb[0][0]
    for t1, _ in nb[1:]:
        tmin = torch.minimum(tmin, t1)
    h = (hr, hx, hz)
    term = []
    for d, (t1, t2) in enumerate(nb):
        a, side = d // 2, d % 2
        o2 = t2 < t1 if order2 else torch.zeros_like(t1, dtype=torch.bool)
        k = t1 - tmin
        g = torch.where(o2, h[a] * (2.0 / 3.0), h[a])
        inside = torch.ones(n[a], dtype=torch.bool, device=T.device)
        inside[0 if side == 0 else -1] = False
        shape = [1, 1, 1]
        shape[a] = n[a]
        term.append((k, torch.where(o2, k + (t1 - t2) / 3.0, k), g, inside.reshape(shape)))
    best = torch.full(n, inf, dtype=T.dtype, device=T.device)
    s2 = s * s
    for q in range(8):
        oct_ = [term[0 + (q & 1)], term[2 + ((q >> 1) & 1)], term[4 + ((q >> 2) & 1)]]
        inside = oct_[0][3] & oct_[1][3] & oct_[2][3]
        t = [list(o[:3]) for o in oct_]
        for i, j in ((0, 1), (1, 2), (0, 1)):
            p = t[j][0] < t[i][0]
            for c in range(3):
                t[i][c], t[j][c] = torch.where(p, t[j][c], t[i][c]), torch.where(p, t[i][c], t[j][c])
        x = t[0][1] + s * t[0][2]
        on = torch.ones_like(p)
        A, B, C = 1.0 / t[0][2] ** 2, t[0][1] / t[0][2] ** 2, (t[0][1] / t[0][2]) ** 2 - s2
        for k, e, g in t[1:]:
            on = on & (k < x)
            A, B, C = A + 1.0 / g ** 2, B + e / g ** 2, C + (e / g) ** 2
            x = torch.where(on, (B + torch.sqrt((B * B - A * C).clamp(min=0.0))) / A, x)
        best = torch.where(inside & (x < best), x, best)
    return torch.where(tmin < inf, tmin + best, inf)


def _fixed_point(grid, s, start, fixed, order2, upward, deadline):
    """The field whose every free node is its own update (start: given times,
    +inf unset); None past the deadline.  upward: a wave from below, slab by
    slab first."""
    import time
    r, th, _ = grid.axes(s.device)
    nnr = grid.nn[0]
    hx = ((r + EARTH) * grid.step[1])[:, None, None]
    hz = ((r + EARTH)[:, None] * torch.sin(th) * grid.step[2])[:, :, None]
    T = torch.full([n + 4 for n in grid.nn], math.inf, dtype=torch.float64, device=s.device)
    T[2:-2, 2:-2, 2:-2] = start

    def relax(lo, hi, stop, most):
        for k in range(most):
            # (a slab's own edges in r count as inside unless they are the grid's)
            a, b = max(0, lo - 1), min(nnr, hi + 1)
            v = _octants(T[a:b + 4], s[a:b], hx[a:b], hz[a:b], torch.full_like(hx[:1], grid.step[0]), order2)
            v = v[lo - a:v.shape[0] - (b - hi)]
            core = T[lo + 2:hi + 2, 2:-2, 2:-2]
            v = torch.where(fixed[lo:hi], core, v)
            off = torch.where(v == core, 0.0, (v - core).abs())
            T[lo + 2:hi + 2, 2:-2, 2:-2] = v
            if k % 8 == 7 and float(off.max()) < stop:
                return True
            if k % 8 == 7 and time.monotonic() > deadline:
                return False
        return True

    for top in range(nnr - 8, -8, -8) if upward else ():
        relax(max(0, top), min(nnr, max(0, top) + 16), 1e-9, 64)
    done = relax(0, nnr, 1e-11, 20000) and time.monotonic() < deadline
    return T[2:-2, 2:-2, 2:-2] if done else None


def _at_receivers(grid, T, rec):
    out = torch.zeros(len(rec[0]), dtype=torch.float64, device=T.device)
    pos = []
    for a in range(3):
        x = torch.tensor(rec[a], dtype=torch.float64, device=T.device)
        u = ((grid.org[0] - x) if a == 0 else (x - grid.org[a])) / grid.step[a]
        i = torch.floor(u).clamp(0, grid.nn[a] - 2)
        pos.append((i.long(), u - i))
    for q in range(8):
        w = torch.ones_like(out)
        ix = []
        for a in range(3):
            b = (q >> a) & 1
            ix.append(pos[a][0] + b)
            w = w * (pos[a][1] if b else 1 - pos[a][1])
        out += w * T[ix[0], ix[1], ix[2]]
    return out


def _ray_ends(grid, T, rec):
    """End points of the rays that follow the field's gradient down from the
    receivers, a layer's height at a step, clipped at the grid's faces."""
    n, dev = grid.nn, T.device
    x = [torch.tensor(c, dtype=torch.float64, device=dev) for c in rec]

    def cell(p):
        return [torch.floor(((grid.org[0] - p[0]) if a == 0 else (p[a] - grid.org[a])) / grid.step[a]) for a in range(3)]

    c = [torch.minimum(i, torch.tensor(float(n[a] - 2), device=dev)).long() for a, i in enumerate(cell(x))]
    live = torch.ones_like(x[0], dtype=torch.bool)
    for _ in range(20 * sum(n)):
        t = {(i, j, k): T[c[0] + i, c[1] + j, c[2] + k] for i in (0, 1) for j in (0, 1) for k in (0, 1)}
        down = torch.stack([t[1, j, k] - t[0, j, k] for j in (0, 1) for k in (0, 1)])
        neg = down < 0
        num = neg.sum(0)
        dr = torch.where(num > 0, torch.where(neg, down, 0.0).sum(0) / (num.clamp(min=1) * grid.step[0]), 0.0)
        rc = EARTH + grid.org[0] - c[0] * grid.step[0]
        sx = torch.sin(x[1])
        dx = sum(t[i, 1, k] - t[i, 0, k] for i in (0, 1) for k in (0, 1)) / (4 * rc * grid.step[1])
        dz = sum(t[i, j, 1] - t[i, j, 0] for i in (0, 1) for j in (0, 1)) / (4 * rc * sx * grid.step[2])
        norm, cr, d = torch.sqrt(dr * dr + dx * dx + dz * dz), EARTH + x[0], grid.step[0]
        y = [x[0] + d * dr / norm, x[1] - d * dx / (cr * norm), x[2] - d * dz / (cr * sx * norm)]
        m = cell(y)
        part = torch.ones_like(norm)
        for a in range(3):
            low, high = m[a] < 0, m[a] >= n[a] - 1
            sign = -1.0 if a == 0 else 1.0
            face = grid.org[a] + sign * torch.where(low, 0.0, float(n[a] - 1)) * grid.step[a]
            part = torch.where(low | high, torch.minimum(part, (face - x[a]) / (y[a] - x[a])), part)
        out = torch.zeros_like(live)
        for a in range(3):
            out |= (m[a] < 0) | (m[a] >= n[a] - 1)
        for a in range(3):
            x[a] = torch.where(live, torch.where(out, x[a] + part * (y[a] - x[a]), y[a]), x[a])
            c[a] = torch.where(live & ~out, m[a].long(), c[a])
        live = live & ~out
        if not bool(live.any()):
            break
    return torch.stack(x, dim=1)


def _chord(grid, v, p):
    """Straight-ray times from point p to every node: chord length times the
    mean of the slowness at both ends."""
    dev = v.device
    u = [(grid.org[0] - p[0]) / grid.step[0]] + [(p[a] - grid.org[a]) / grid.step[a] for a in (1, 2)]
    i = [min(max(int(math.floor(q)), 0), n - 2) for q, n in zip(u, grid.nn)]
    ss = 0.0
    for q in range(8):
        b = ((q >> 2) & 1, (q >> 1) & 1, q & 1)
        w = math.prod((u[a] - i[a]) if b[a] else 1 - (u[a] - i[a]) for a in range(3))
        ss += w / float(v[i[0] + b[0], i[1] + b[1], i[2] + b[2]])
    r, th, ph = grid.axes(dev)
    r, th, ph = (r + EARTH)[:, None, None], th[None, :, None], ph[None, None, :]
    rs = EARTH + p[0]
    d2 = ((r * torch.sin(th) * torch.cos(ph) - rs * math.sin(p[1]) * math.cos(p[2])) ** 2
          + (r * torch.sin(th) * torch.sin(ph) - rs * math.sin(p[1]) * math.sin(p[2])) ** 2
          + (r * torch.cos(th) - rs * math.cos(p[1])) ** 2)
    return torch.sqrt(d2) * 0.5 * (ss + 1.0 / v)


def _point_start(inp, grid, v, p, refine, extent, order2, deadline):
    """Start and fixed nodes of a point source on the grid."""
    dev = v.device
    u = [(grid.org[0] - p[0]) / grid.step[0]] + [(p[a] - grid.org[a]) / grid.step[a] for a in (1, 2)]
    lo = [max(0, int(math.floor(q)) - extent + 1) for q in u]
    hi = [min(n - 1, int(math.floor(q)) + extent) for q, n in zip(u, grid.nn)]
    start = torch.full(grid.nn, math.inf, dtype=torch.float64, device=dev)
    fixed = torch.zeros(grid.nn, dtype=torch.bool, device=dev)
    box = tuple(slice(a, b + 1) for a, b in zip(lo, hi))
    if not refine:
        start[box] = _chord(grid, v, p)[box]
        fixed[box] = True
        return start, fixed
    sign = (-1.0, 1.0, 1.0)
    fine = _Grid(tuple((b - a) * refine + 1 for a, b in zip(lo, hi)),
                 tuple(grid.org[a] + sign[a] * lo[a] * grid.step[a] for a in range(3)),
                 tuple(q / refine for q in grid.step))
    vf = _velocity(inp, fine, dev)
    uf = [(fine.org[0] - p[0]) / fine.step[0]] + [(p[a] - fine.org[a]) / fine.step[a] for a in (1, 2)]
    cf = [min(max(int(math.floor(q)), 0), n - 2) for q, n in zip(uf, fine.nn)]
    near = tuple(slice(max(0, c - 1), min(n - 1, c + 2) + 1) for c, n in zip(cf, fine.nn))
    fs = torch.full(fine.nn, math.inf, dtype=torch.float64, device=dev)
    ff = torch.zeros(fine.nn, dtype=torch.bool, device=dev)
    fs[near] = _chord(fine, vf, p)[near]
    ff[near] = True
    Tf = _fixed_point(fine, 1.0 / vf, fs, ff, order2, False, deadline)
    if Tf is None:
        return None
    start[box] = Tf[::refine, ::refine, ::refine]
    fixed[tuple(slice(a + 1 if a > 0 else a, b if b < n - 1 else b + 1) for a, b, n in zip(lo, hi, grid.nn))] = True
    return start, fixed


def exact(case, seed):
    """Receiver times and ray end points in 64 bits, by iterating the node
    update over the whole grid; None where that takes too long."""
    import time
    if case["nnr"] * case["nnx"] * case["nnz"] * case["nev"] > 2e7:
        return None
    deadline = time.monotonic() + 18.0
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    inp = _inputs(case, seed)
    grid = _Grid(inp["nn"], *_rad(inp["orig"], inp["step"]))
    v = _velocity(inp, grid, dev)
    order2 = case.get("fom", 1) == 1
    frames = _frames(inp, dev)
    times, ends = [], []
    for e in range(case["nev"]):
        if case["kind"] == "point":
            got = _point_start(inp, grid, v, inp["src"][e], case["refine"], case["extent"], order2, deadline)
            if got is None:
                return None
            start, fixed = got
        else:
            start = torch.full(grid.nn, math.inf, dtype=torch.float64, device=dev)
            fixed = torch.zeros(grid.nn, dtype=torch.bool, device=dev)
            fixed[-1] = frames[e] > 0
            start[-1] = torch.where(fixed[-1], frames[e], math.inf)
        T = _fixed_point(grid, 1.0 / v, start, fixed, order2, case["kind"] != "point", deadline)
        if T is None:
            return None
        times.append(_at_receivers(grid, T, inp["rec"]))
        if case["kind"] == "rays" or case.get("api") == "device":
            ends.append(_ray_ends(grid, T, inp["rec"]))
    out = {"entries": None, "row_ptr": None, "cols": None, "vals": None}
    if case["kind"] != "rays":
        out["times"] = torch.stack(times)
    if case["kind"] in ("times", "point"):
        out = {"times": out["times"]}
    elif case.get("api") != "host":
        out["ends"] = torch.cat(ends)
    return out
