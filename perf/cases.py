"""The work a user of this framework has it do, as cases that can be timed.

Every case is one call, or one short sequence of calls, of the public Python class
``sunset_viscoelastic_b200.labfm.Sunset`` on a node set made from a seed:

* ``steps``: a host code that owns its fields hands them over, has them stepped and takes them
  back (``run_host``, pinned host buffers both ways): 2-D and 3-D, periodic, walled and
  inflow/outflow node sets, the three conformation forms, orders 4 to 8, FP64 and mixed.
* ``setup``: neighbour lists and LABFM weights of a new node set, exported to the host in the
  reference's layout, with or without the stencil adaptation that runs by default there.
* ``first_step``: from a node set to the first stepped field: create, build, set up, step.
* ``operators``: gradient, Laplacian and filter of one field held by the host.
* ``adjoint``: gradients of the final kinetic energy with respect to Wi, beta and the initial
  state (the backward direction of ``steps``).

``exact`` restates the periodic 2-D path in torch in 64 bits: the weights by an LU solve of the
moment systems, the step from the equations, the adjoint by automatic differentiation.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from sunset_viscoelastic_b200 import labfm
from sunset_viscoelastic_b200.nodesets import NodeSet, cylinder_channel, inflow_channel, reader_nodes

# stencil radius in spacings of the periodic sets (the repository's measured workloads)
RADIUS = {4: 3.0, 6: 4.2, 8: 5.4}
# links a node the host code's own arrays hold (ij_link(nplink, npfb)), by order
NPLINK = {4: 48, 6: 80, 8: 128}
# fluid parameters of the periodic sets, and of the walled channel (body force 50 in x)
FLUID = {"di": dict(Re=1.0, Wi=1.0, beta=0.5, epsPTT=0.0), "lc": dict(Re=1.0, Wi=1.0, beta=0.5, epsPTT=0.25),
         "chl": dict(Re=1.0, Wi=2.0, beta=0.1, epsPTT=0.0)}
CHANNEL = dict(Re=0.01, Wi=0.5, beta=0.59, Ma=0.05, grav=(50.0, 0.0, 0.0), kolmogorov_forcing=0)
INFLOW = dict(Re=10.0, Wi=0.5, beta=0.59, Ma=0.1, kolmogorov_forcing=0)
MA = 0.1
FIELDS = ("ro", "rou", "rov", "q0", "q1", "q2", "q3")
FIELDS_3D = ("ro", "rou", "rov", "row", "xx", "xy", "yy", "xz", "yz", "zz")


def listed():
    return [
        # the node count of the reference's own case at its default order, one step a call: what a
        # host code that couples every step waits for
        dict(name="chl-o8-4k-step", kind="steps", geometry="periodic", form="chl", order=8, nside=64, layers=0,
             precision="fp64", steps=1),
        # the small direct-form configuration, twenty steps a call
        dict(name="di-o4-16k", kind="steps", geometry="periodic", form="di", order=4, nside=128, layers=0,
             precision="fp64", steps=20),
        # the confined-cylinder benchmark of viscoelastic flow: walls, uneven node set, 35k nodes
        dict(name="cylinder-di-o8", kind="steps", geometry="cylinder", form="di", order=8, nside=64, layers=0,
             precision="fp64", steps=20),
        # the log-conformation configuration, 262,144 nodes
        dict(name="lc-o6-262k", kind="steps", geometry="periodic", form="lc", order=6, nside=512, layers=0,
             precision="fp64", steps=10),
        # the benchmark's configuration and the largest 2-D one, 1,048,576 nodes
        dict(name="chl-o8-1m", kind="steps", geometry="periodic", form="chl", order=8, nside=1024, layers=0,
             precision="fp64", steps=10),
        # the mixed-precision step where a long production run uses it
        dict(name="chl-o8-590k-mixed", kind="steps", geometry="periodic", form="chl", order=8, nside=768, layers=0,
             precision="mixed", steps=10),
        # 3-D: the benchmark's layered set, 2,097,152 nodes
        dict(name="di-o4-3d-2m", kind="steps", geometry="periodic", form="di", order=4, nside=128, layers=128,
             precision="fp64", steps=4),
        # 3-D log-conformation with an odd number of layers
        dict(name="lc-o6-3d-600k", kind="steps", geometry="periodic", form="lc", order=6, nside=96, layers=65,
             precision="fp64", steps=4),
        # a new node set as the reference sets it up by default: lists, adapted stencils, lists again,
        # weights, taken back by the host code
        dict(name="setup-o8-9k-adapt", kind="setup", order=8, nside=96, adapt=True),
        # from a new node set to the first field, as each run of a parameter study starts
        dict(name="first-step-o6-262k", kind="first_step", form="lc", order=6, nside=512, steps=1),
        # a gradient evaluation of an inverse problem: forward and reverse sweep
        dict(name="adjoint-o6-65k", kind="adjoint", order=6, nside=256, steps=40, checkpoint=20),
        # single operators on a field the host holds (diagnostics, coupling)
        dict(name="operators-o6-90k", kind="operators", order=6, nside=301),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: odd sides, every form, order, precision and node set."""
    kind = rng.choice(["steps"] * 6 + ["setup", "first_step", "adjoint", "operators"])
    order = rng.choice([4, 6, 8])
    if kind == "setup":
        return dict(kind="setup", order=order, nside=_log_uniform(rng, 41, 110), adapt=False)
    if kind == "first_step":
        return dict(kind="first_step", form=rng.choice(["di", "chl", "lc"]), order=order,
                    nside=_log_uniform(rng, 64, 300), steps=rng.randint(1, 4))
    if kind == "adjoint":
        return dict(kind="adjoint", order=6, nside=_log_uniform(rng, 48, 200), steps=rng.randint(10, 40),
                    checkpoint=rng.choice([7, 10, 20]))
    if kind == "operators":
        return dict(kind="operators", order=order, nside=_log_uniform(rng, 50, 400))
    form = rng.choice(["di", "chl", "lc"])
    shape = rng.choice(["periodic", "periodic", "periodic", "mixed", "3d", "cylinder", "inflow"])
    if shape == "3d":
        return dict(kind="steps", geometry="periodic", form=form, order=rng.choice([4, 6]),
                    nside=_log_uniform(rng, 30, 110), layers=rng.randint(24, 100), precision="fp64",
                    steps=rng.randint(1, 4))
    if shape == "cylinder":
        return dict(kind="steps", geometry="cylinder", form=form, order=rng.choice([6, 8]), nside=rng.randint(32, 64),
                    layers=0, precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(1, 20))
    if shape == "inflow":
        return dict(kind="steps", geometry="inflow", form=form, order=rng.choice([6, 8]),
                    nside=_log_uniform(rng, 40, 200), layers=0, precision="fp64", steps=rng.randint(1, 20))
    return dict(kind="steps", geometry="periodic", form=form, order=order, nside=_log_uniform(rng, 45, 600), layers=0,
                precision="mixed" if shape == "mixed" else "fp64", steps=rng.randint(1, 20))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _lattice(nside, seed):
    """Positions of the jittered lattice on the periodic unit square (+-0.3 spacings)."""
    s = 1.0 / nside
    rng = np.random.default_rng([seed, nside])
    j, i = np.divmod(np.arange(nside * nside), nside)
    x = (i + 0.5) * s + rng.uniform(-0.3 * s, 0.3 * s, nside * nside)
    y = (j + 0.5) * s + rng.uniform(-0.3 * s, 0.3 * s, nside * nside)
    return x, y


def _periodic_nodes(nside, seed):
    x, y = _lattice(nside, seed)
    n = len(x)
    return NodeSet(x=x, y=y, node_type=np.full(n, 999, np.int32), nx=np.zeros(n), ny=np.zeros(n),
                   s=np.full(n, 1.0 / nside), xmin=0.0, xmax=1.0, ymin=0.0, ymax=1.0, bcond=(1, 1, 1, 1))


def _amplitudes(seed):
    return np.random.default_rng([seed, 7]).uniform(0.5, 1.0, 12)


def _flow(x, y, a):
    """A smooth doubly periodic velocity of order 1, density near 1 and log-conformation."""
    t = 2.0 * np.pi
    ro = 1.0 + 0.004 * a[0] * np.sin(t * x + 1.0) * np.cos(t * y)
    u = a[1] * np.sin(t * x) * np.cos(t * y) + 0.2 * a[2] * np.cos(t * (x + 2 * y))
    v = -a[1] * np.cos(t * x) * np.sin(t * y) + 0.2 * a[3] * np.sin(t * (2 * x - y))
    psi = (0.2 + 0.1 * a[4] * np.sin(t * x), 0.15 * a[5] * np.cos(t * y) + 0.05 * a[6] * np.sin(t * x),
           -0.3 + 0.05 * a[7] * np.sin(t * (x + y)))
    return ro, u, v, psi


def _expm2(p0, p1, p2):
    m, d = 0.5 * (p0 + p2), 0.5 * (p0 - p2)
    r = np.sqrt(d * d + p1 * p1)
    ch, sh = np.exp(m) * np.cosh(r), np.exp(m) * np.sinh(r) / np.where(r > 0, r, 1.0)
    return ch + sh * d, sh * p1, ch - sh * d


def _variables(form, psi, czz):
    """The evolved conformation variables of a form (q0..q3) and c, from log c."""
    cxx, cxy, cyy = _expm2(*psi)
    one = np.ones_like(cxx)
    if form == "di":
        return (cxx, cxy, cyy, czz), (cxx, cxy, cyy, czz)
    if form == "lc":
        return (psi[0], psi[1], psi[2], 0.0 * one), (cxx, cxy, cyy, one)
    lxx = np.sqrt(cxx)
    lxy = cxy / lxx
    return (np.log(lxx), lxy, 0.5 * np.log(cyy - lxy * lxy), 0.0 * one), (cxx, cxy, cyy, one)


def _initial_2d(x, y, form, seed):
    a = _amplitudes(seed)
    ro, u, v, psi = _flow(x, y, a)
    q, c = _variables(form, psi, 1.0 + 0.05 * a[8] * np.cos(2.0 * np.pi * x))
    return ro, u, v, q, c


def _dt(s, visc=1.0, sound=10.0):
    """A quarter of the smaller of the viscous and acoustic limits of the step."""
    return 0.25 * min(2.0 / 3.0 * s * s / visc, s / (1.3 + sound))


def _pinned(arrays):
    t = torch.empty(sum(len(a) for a in arrays), dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.copy_(torch.from_numpy(np.concatenate(arrays)))
    return t


def _periodic_handle(form, order, ns, precision="fp64", **over):
    g = labfm.Sunset(form=form, order=order, h_over_s=RADIUS[order] / 2.0, Ma=MA, precision=precision,
                     **dict(FLUID[form], **over))
    return g.build_domain(ns)


def _prepare_steps_2d(case, seed):
    form, order, nside = case["form"], case["order"], case["nside"]
    a = _amplitudes(seed)
    if case["geometry"] == "periodic":
        ns = _periodic_nodes(nside, seed)
        g = _periodic_handle(form, order, ns, case["precision"])
        x, y, dt, walls = ns.x, ns.y, _dt(1.0 / nside), None
        ro, u, v, q, c = _initial_2d(x, y, form, seed)
    elif case["geometry"] == "cylinder":
        # spacing R/nside on the cylinder, a quarter of the default channel length at half that
        ns = cylinder_channel(s_min_frac=1.0 / nside, half_length=15.0 * nside / 64.0, seed=seed)
        x, y, t = reader_nodes(ns)
        g = labfm.Sunset(form=form, order=order, precision=case["precision"], **CHANNEL).build_domain(ns)
        dt, walls = _dt(ns.smin, visc=100.0, sound=20.0), (t == 0)
        ro, u, v, psi = _flow(x / 8.0, y / 8.0, a)
        bump = (1.0 - 0.25 * y * y) * (1.0 - 1.0 / np.maximum(x * x + y * y, 1.0))
        u, v = 0.5 * bump * (1.0 + 0.2 * u), 0.2 * bump * v
        q, c = _variables(form, psi, np.ones(len(x)))
    else:
        ns = inflow_channel(nside, ybc=1, seed=seed)
        x, y, t = reader_nodes(ns)
        g = labfm.Sunset(form=form, order=order, precision=case["precision"], **INFLOW).build_domain(ns)
        dt, walls = _dt(ns.smin, visc=0.1), None
        ro, u, v, psi = _flow(0.5 * x, y, a)
        u, v = 1.0 + 0.05 * u, 0.05 * v
        q, c = _variables(form, psi, np.ones(len(x)))
    g.setup()
    if walls is not None:
        u, v = np.where(walls, 0.0, u), np.where(walls, 0.0, v)
    g.set_state(ro, u, v, *c)
    g.set_time(0.0, dt, 10, [1e-5] * 3)  # a run that is under way
    return dict(g=g, dt=dt, steps=case["steps"], n=len(x), keys=FIELDS,
                inp=_pinned((ro, ro * u, ro * v) + tuple(q)), out=_pinned([np.zeros(7 * len(x))]))


def _prepare_steps_3d(case, seed):
    form, nside, a = case["form"], case["nside"], _amplitudes(seed)
    ns = _periodic_nodes(nside, seed)
    g = _periodic_handle(form, case["order"], ns)
    nz, dz = g.set_layers((case["layers"] - 0.5) / nside)
    g.setup()
    t = 2.0 * np.pi
    z = (np.arange(nz) + 0.5) / nz
    x, y, z = np.tile(ns.x, nz), np.tile(ns.y, nz), np.repeat(z, ns.n)
    ro, u, v, psi = _flow(x, y, a)
    u, v = u * (1.0 + 0.3 * np.cos(t * z)), v * (1.0 - 0.2 * np.sin(t * z))
    w = 0.3 * a[9] * np.cos(t * x) * np.sin(t * z)
    pxz, pyz = 0.05 * a[10] * np.sin(t * (x + z)), 0.04 * a[11] * np.cos(t * (y - z))
    pzz = 0.1 + 0.03 * np.cos(t * z)
    if form == "di":  # c itself, diagonally dominant
        q = (1.0 + psi[0], 0.5 * psi[1], 1.5 + psi[2], pxz, pyz, 1.0 + pzz)
    else:             # Cholesky or log-conformation variables
        q = (psi[0], psi[1], psi[2], pxz, pyz, pzz)
    g.set_state_3d(ro, u, v, w)
    dt = _dt(min(1.0 / nside, dz))
    g.set_time(0.0, dt, 10, [1e-5] * 3)
    return dict(g=g, dt=dt, steps=case["steps"], n=len(x), keys=FIELDS_3D,
                inp=_pinned((ro, ro * u, ro * v, ro * w) + q), out=_pinned([np.zeros(10 * len(x))]))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        return dict((_prepare_steps_3d if case["layers"] else _prepare_steps_2d)(case, seed), kind=kind)
    ns = _periodic_nodes(case["nside"], seed)
    if kind == "setup":
        nplink = NPLINK[case["order"]]
        host = dict(w_grad=np.zeros((ns.n, nplink, 2)), w_lap=np.zeros((ns.n, nplink)), w_hyp=np.zeros((ns.n, nplink)),
                    links=np.zeros((ns.n, nplink), np.int32))
        return dict(kind=kind, ns=ns, order=case["order"], adapt=case["adapt"], host=host)
    if kind == "first_step":
        form = case["form"]
        ro, u, v, q, c = _initial_2d(ns.x, ns.y, form, seed)
        return dict(kind=kind, ns=ns, form=form, order=case["order"], steps=case["steps"], dt=_dt(1.0 / case["nside"]),
                    n=ns.n, c=(ro, u, v) + tuple(c), inp=_pinned((ro, ro * u, ro * v) + tuple(q)),
                    out=_pinned([np.zeros(7 * ns.n)]))
    if kind == "adjoint":
        g = _periodic_handle("lc", case["order"], ns, epsPTT=0.0).setup()
        ro, u, v, q, c = _initial_2d(ns.x, ns.y, "lc", seed)
        return dict(kind=kind, g=g, dt=_dt(1.0 / case["nside"]), steps=case["steps"], checkpoint=case["checkpoint"],
                    c=(ro, u, v) + tuple(c))
    g = _periodic_handle("di", case["order"], ns).setup()
    ro, u, v, q, c = _initial_2d(ns.x, ns.y, "di", seed)
    return dict(kind=kind, g=g, phi=u)


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def _fields(st, keys):
    return {k: st["out"][f * st["n"]:(f + 1) * st["n"]] for f, k in enumerate(keys)}


def run(st):
    kind = st["kind"]
    if kind == "steps":
        st["g"].run_host(st["inp"].data_ptr(), st["dt"], st["steps"], st["out"].data_ptr())
        return _fields(st, st["keys"])
    if kind == "operators":
        g, phi = st["g"], st["phi"]
        return dict(gradient=g.gradient(phi), laplacian=g.laplacian(phi), filtered=g.filtered(phi),
                    filter_term=g.filter_term(phi))
    if kind == "adjoint":
        g = st["g"]
        g.set_state(*st["c"])
        g.set_time(0.0, st["dt"], 10, [1e-5] * 3)
        J, dparams, dstate = g.adjoint_run(st["dt"], st["steps"], st["checkpoint"])
        return dict(J=J, dWi=dparams[0], dbeta=dparams[1], dstate=dstate)
    if kind == "setup":
        g = labfm.Sunset(form="chl", order=st["order"], Ma=MA, **FLUID["chl"],
                         h_over_s=0.0 if st["adapt"] else RADIUS[st["order"]] / 2.0).build_domain(st["ns"])
        if st["adapt"]:
            g.find_neighbours()
            g.adapt_stencils()
            g.calc_labf_weights()
            g.calc_boundary_weights()
            g.calc_labf_sums()
            g.filter_coefficients()
        else:
            g.setup()
        count, count_small, links = g.neighbours()
        out = dict(g.weights(), count=count, count_small=count_small, links=links)
        for key, a in st["host"].items():
            a[:, :out[key].shape[1]] = out[key]
            out[key] = a
        if st["adapt"]:
            out["h"], out["h_small"] = g.lengths()
        g.close()
        return out
    g = _periodic_handle(st["form"], st["order"], st["ns"]).setup()
    g.set_state(*st["c"])
    g.set_time(0.0, st["dt"], 10, [1e-5] * 3)
    g.run_host(st["inp"].data_ptr(), st["dt"], st["steps"], st["out"].data_ptr())
    g.close()
    return _fields(st, FIELDS)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _nodes_and_links(case):
    """Nodes and mean links a node."""
    nside, order = case["nside"], case["order"]
    k = math.pi * RADIUS[order] ** 2
    if case.get("geometry") == "cylinder":
        return int(34853 * (nside / 64.0)), math.pi * (2 * {6: 2.2, 8: 2.7}[order]) ** 2
    if case.get("geometry") == "inflow":
        return 2 * nside * nside, math.pi * (2 * {6: 2.2, 8: 2.7}[order]) ** 2
    if case.get("adapt"):
        k = math.pi * (2 * 2.4) ** 2
    return nside * nside, k


def _step_work(case, form, n, k, nz, mixed):
    """One RK3 step.  The link streams exceed the caches on the larger sets and every stage needs
    every node's neighbours, so each stage reads its links (three weights and an index) and
    reads and writes the state and the two RK registers once; the filter likewise."""
    wide = 4.0 if mixed else 8.0
    nf = 10 if nz > 1 else 7
    sums = {"di": 14, "chl": 14, "lc": 20}[form] + (16 if nz > 1 else 0)
    stage = k * (12.0 if mixed else 26.0) + nz * (nf * 16.0 + nf * 4.0 * wide)
    filt = k * (6.0 if mixed else 10.0) + nz * nf * 16.0
    return n * (4.0 * stage + filt), n * nz * (4.0 * (2.0 * k * sums + 250.0) + 2.0 * k * nf)


def _setup_work(n, k, order):
    """Moment matrices, one factorisation each, the weights; links and four weights written."""
    m = (order * order + 3 * order) // 2
    return n * k * 36.0, n * (2.0 * k * m * m + 12.0 * m ** 3 + 12.0 * k * m)


def work(case):
    n, k = _nodes_and_links(case)
    kind = case["kind"]
    if kind == "operators":  # gradient, Laplacian and two filters: links and a field in and out
        return {"bytes": n * (k * (18.0 + 10.0 + 10.0 + 10.0) + 8.0 * 9), "flops": n * k * 10.0}
    if kind == "setup":
        b, f = _setup_work(n, k, case["order"])
        return {"bytes": b, "flops": f}
    nz = max(1, case.get("layers", 0))
    b, f = _step_work(case, case.get("form", "lc"), n, k, nz, case.get("precision") == "mixed")
    b, f = b * case["steps"], f * case["steps"]
    if kind == "adjoint":  # the forward run, and a reverse sweep over the same links
        return {"bytes": 2.0 * b, "flops": 2.0 * f}
    io = n * nz * 8.0 * 2.0 * (10 if nz > 1 else 7)
    if kind == "first_step":
        sb, sf = _setup_work(n, k, case["order"])
        b, f = b + sb, f + sf
    return {"bytes": b + io, "flops": f}


# ---------------------------------------------------------------------------------------
# the same in plain torch, 64 bits (periodic 2-D sets)
# ---------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _exponents(order):
    return [(d - q, q) for d in range(1, order + 1) for q in range(d + 1)]


def _hermites(order, z):
    h = [torch.ones_like(z), z]
    for m in range(1, order):
        h.append(z * h[m] - m * h[m - 1])
    return h


class _Stencils:
    """Neighbours in order of distance, weights, row sums and volumes of a periodic set."""

    def __init__(self, nside, order, seed):
        dev, s = _device(), 1.0 / nside
        xs, ys = (torch.from_numpy(a).to(dev) for a in _lattice(nside, seed))
        hh = RADIUS[order] / 2.0 * s
        reach = int(math.ceil(RADIUS[order] + 0.6))
        if nside < 2 * reach + 1:
            raise ValueError("the set is smaller than a stencil")
        off = torch.arange(-reach, reach + 1, device=dev)
        oj, oi = (t.reshape(-1) for t in torch.meshgrid(off, off, indexing="ij"))
        n, ex = nside * nside, _exponents(order)
        m = len(ex)
        fact = [math.factorial(p) * math.factorial(q) for p, q in ex]
        rhs = torch.zeros(m, 4, dtype=torch.float64, device=dev)
        rhs[0, 0] = rhs[1, 1] = rhs[2, 2] = rhs[4, 2] = 1.0
        # the hyperviscous operator (-1)^(order/2 - 1) (d2/dx2 + d2/dy2)^(order/2)
        half = order // 2
        for c in range(half + 1):
            rhs[ex.index((order - 2 * c, 2 * c)), 3] = (-1.0) ** (half + 1) * math.comb(half, c)
        parts = []
        step = max(1, 60_000_000 // (len(oi) * m))
        for b in range(0, n, step):
            node = torch.arange(b, min(n, b + step), device=dev)
            i, j = node % nside, node // nside
            ci, cj = i[:, None] + oi[None], j[:, None] + oj[None]
            nb = (cj % nside) * nside + ci % nside
            dx = xs[nb] + torch.div(ci, nside, rounding_mode="floor") - xs[node][:, None]
            dy = ys[nb] + torch.div(cj, nside, rounding_mode="floor") - ys[node][:, None]
            r2 = dx * dx + dy * dy
            inside = r2 <= (2.0 * hh) ** 2
            cnt = inside.sum(1)
            k = int(cnt.max())
            r2, at = torch.where(inside, r2, torch.inf).sort(1)
            at, ok = at[:, :k], torch.isfinite(r2[:, :k])
            nb, dx, dy = (t.gather(1, at) for t in (nb, dx, dy))
            x, y, qq = dx / hh, dy / hh, torch.where(ok, r2[:, :k], 0.0).sqrt() / hh
            ker = 7.0 / (4.0 * math.pi * hh * hh) * (2.0 * qq + 1.0) * (1.0 - 0.5 * qq) ** 4
            ker = torch.where(ok & (qq > 0), ker, 0.0)
            hx, hy = _hermites(order, x), _hermites(order, y)
            G = torch.stack([hx[p] * hy[q] for p, q in ex], 2) * ker[:, :, None]
            X = torch.stack([x ** p * y ** q / f for (p, q), f in zip(ex, fact)], 2)
            sol = torch.linalg.solve(X.transpose(1, 2) @ G, rhs.expand(len(node), m, 4))
            w = G @ sol
            w = torch.where(ok[:, :, None], w, 0.0) / torch.tensor([hh, hh, hh * hh, 1.0], device=dev, dtype=torch.float64)
            ls = 2.0 * hh * torch.sqrt(math.pi / cnt.double())
            t = (2.0 / 3.0 * math.pi / ls)[:, None]
            fc = 2.0 / 3.0 / ((1.0 - torch.cos(t * dx) * torch.cos(t * dy)) * w[:, :, 3]).sum(1)
            w[:, :, 3] *= fc[:, None]
            vol = 1.0 / torch.where(ok, 9.0 / math.pi * torch.exp(-9.0 * qq * qq) / hh ** 2, 0.0).sum(1)
            parts.append((torch.where(ok, nb, 0), w, vol, cnt))
        k = max(p[0].shape[1] for p in parts)
        pad = torch.nn.functional.pad
        self.nb = torch.cat([pad(p[0], (0, k - p[0].shape[1])) for p in parts])
        self.w = torch.cat([pad(p[1], (0, 0, 0, k - p[1].shape[1])) for p in parts])
        self.vol = torch.cat([p[2] for p in parts])
        self.y = ys
        self.sums = self.w.sum(1)

    def apply(self, phi, ops):
        """[op] of each column of phi (n, f): (len(ops), n, f), in the difference form."""
        out = [[] for _ in ops]
        step = max(1, 40_000_000 // self.nb.shape[1])
        for c in range(phi.shape[1]):
            rows = [[] for _ in ops]
            for b in range(0, phi.shape[0], step):
                d = phi[self.nb[b:b + step], c] - phi[b:b + step, c, None]
                for r, o in zip(rows, ops):
                    r.append((d * self.w[b:b + step, :, o]).sum(1))
            for o, r in zip(out, rows):
                o.append(torch.cat(r))
        return torch.stack([torch.stack(o, 1) for o in out])


A21, A32, A43 = 11847461282814.0 / 36547543011857.0, 3943225443063.0 / 7078155732230.0, -346793006927.0 / 4029903576067.0
B1, B2, B3, B4 = (1017324711453.0 / 9774461848756.0, 8237718856693.0 / 13685301971492.0,
                  57731312506979.0 / 19404895981398.0, -101169746363290.0 / 37734290219643.0)


def _conformation(form, q):
    if form == "di":
        return q[0], q[1], q[2]
    if form == "chl":
        lxx = torch.exp(q[0])
        return lxx * lxx, lxx * q[1], q[1] * q[1] + torch.exp(2.0 * q[2])
    m, d = 0.5 * (q[0] + q[2]), 0.5 * (q[0] - q[2])
    r = torch.sqrt(d * d + q[1] * q[1])
    ch, sh = torch.exp(m) * torch.cosh(r), torch.exp(m) * torch.sinh(r) / r
    return ch + sh * d, sh * q[1], ch - sh * d


def _rhs(form, S, U, Re, Wi, beta, eps):
    ro, rou, rov, q = U[0], U[1], U[2], U[3:7]
    u, v = rou / ro, rov / ro
    c = _conformation(form, q)
    conf = list(q[:3]) + (list(c) if form == "lc" else [])
    D = S.apply(torch.stack([ro, u, v] + conf, 1), (0, 1))
    lap = S.apply(torch.stack([u, v], 1), (2,))[0]
    (rx, ux, vx), (ry, uy, vy) = D[0].T[:3], D[1].T[:3]
    qx, qy = D[0].T[3:], D[1].T[3:]
    csq, lam = (1.0 / MA) ** 2, Wi
    poly = (1.0 - beta) / Re / lam
    if form == "chl":
        exx, eyy, l = torch.exp(q[0]), torch.exp(q[2]), q[1]
        divx = 2.0 * exx * exx * qx[0] + exx * (qy[1] + l * qy[0])
        divy = exx * (qx[1] + l * qx[0]) + 2.0 * l * qy[1] + 2.0 * eyy * eyy * qy[2]
    else:
        o = 0 if form == "di" else 3
        divx, divy = qx[o] + qy[o + 1], qx[o + 1] + qy[o + 2]
    dro = -ro * (ux + vy) - (u * rx + v * ry)
    force = torch.cos(S.y) / Re if form == "chl" else 0.0
    drou = -(ro * (u * ux + v * uy) - u * dro) - csq * rx + beta / Re * lap[:, 0] + poly * divx + force
    drov = -(ro * (u * vx + v * vy) - v * dro) - csq * ry + beta / Re * lap[:, 1] + poly * divy
    adv = [u * qx[k] + v * qy[k] for k in range(3)]
    zero = torch.zeros_like(ro)
    if form == "di":
        cxx, cxy, cyy, czz = q
        f = -((1.0 - 2.0 * eps) + eps * (cxx + cyy + czz)) / lam
        return [dro, drou, drov, -adv[0] + 2.0 * (ux * cxx + uy * cxy) + f * (cxx - 1.0),
                -adv[1] + ux * cxy + uy * cyy + vx * cxx + vy * cxy + f * cxy,
                -adv[2] + 2.0 * (vx * cxy + vy * cyy) + f * (cyy - 1.0), f * (czz - 1.0)]
    if form == "chl":
        f = -((1.0 - 3.0 * eps) + eps * (c[0] + c[2] + 1.0)) / lam
        sxx, sxy, syy = f * (c[0] - 1.0), f * c[1], f * (c[2] - 1.0)
        return [dro, drou, drov, -adv[0] + ux + uy * l / exx + 0.5 * sxx / exx ** 2,
                -adv[1] + vy * l + uy * eyy ** 2 / exx + vx * exx + sxy / exx - 0.5 * sxx * l / exx ** 2,
                -adv[2] + vy - uy * l / exx + 0.5 * syy / eyy ** 2 - sxy * l / (exx * eyy ** 2)
                + 0.5 * sxx * l * l / (exx * eyy) ** 2, zero]
    # log-conformation: the velocity gradient in the eigenframe of psi
    th = 0.5 * torch.atan2(2.0 * q[1], q[0] - q[2])
    co, si = torch.cos(th), torch.sin(th)
    r = torch.sqrt(0.25 * (q[0] - q[2]) ** 2 + q[1] ** 2)
    l1, l2 = torch.exp(0.5 * (q[0] + q[2]) + r), torch.exp(0.5 * (q[0] + q[2]) - r)
    m11 = co * (ux * co + uy * si) + si * (vx * co + vy * si)
    m12 = co * (-ux * si + uy * co) + si * (-vx * si + vy * co)
    m21 = -si * (ux * co + uy * si) + co * (vx * co + vy * si)
    m22 = -si * (-ux * si + uy * co) + co * (-vx * si + vy * co)
    om = (l2 * m12 + l1 * m21) / (l2 - l1)
    f = (1.0 - 2.0 * eps) + eps * (l1 + l2)
    d1, d2 = 2.0 * m11 + (f / l1 - f) / lam, 2.0 * m22 + (f / l2 - f) / lam
    return [dro, drou, drov, -adv[0] + 2.0 * om * q[1] + co * co * d1 + si * si * d2,
            -adv[1] + om * (q[2] - q[0]) + co * si * (d1 - d2),
            -adv[2] - 2.0 * om * q[1] + si * si * d1 + co * co * d2, zero]


def _step(form, S, U, dt, par):
    T = U
    for a, b in ((A21, B1), (A32, B2), (A43, B3), (None, B4)):
        R = _rhs(form, S, U, *par)
        if a is None:
            U = [t + dt * b * r for t, r in zip(T, R)]
        else:
            U, T = [t + dt * a * r for t, r in zip(T, R)], [t + dt * b * r for t, r in zip(T, R)]
    nf = 7 if form == "di" else 6
    F = S.apply(torch.stack(U[:nf], 1), (3,))[0]
    U = [U[f] + F[:, f] if f < nf else U[f] for f in range(7)]
    dro = ((U[0] - 1.0) * S.vol).sum() / S.vol.sum()
    return [U[0] - dro] + U[1:]


def _exact_steps(case, form, seed):
    S = _Stencils(case["nside"], case["order"], seed)
    x, y = _lattice(case["nside"], seed)
    ro, u, v, q, c = _initial_2d(x, y, form, seed)
    U = [torch.from_numpy(a).to(S.vol.device) for a in (ro, ro * u, ro * v) + tuple(q)]
    fl = FLUID[form]
    for _ in range(case["steps"]):
        U = _step(form, S, U, _dt(1.0 / case["nside"]), (fl["Re"], fl["Wi"], fl["beta"], fl["epsPTT"]))
    return {k: t.cpu() for k, t in zip(FIELDS, U)}


def _exact_adjoint(case, seed):
    S = _Stencils(case["nside"], case["order"], seed)
    x, y = _lattice(case["nside"], seed)
    ro, u, v, q, c = _initial_2d(x, y, "lc", seed)
    dev = S.vol.device
    U0 = [torch.from_numpy(a).to(dev).requires_grad_(k < 6) for k, a in enumerate((ro, ro * u, ro * v) + tuple(q))]
    par = [torch.tensor(p, dtype=torch.float64, device=dev, requires_grad=True) for p in (FLUID["lc"]["Wi"], FLUID["lc"]["beta"])]
    U, dt = U0, _dt(1.0 / case["nside"])
    for _ in range(case["steps"]):
        U = torch.utils.checkpoint.checkpoint(
            lambda *V: tuple(_step("lc", S, list(V), dt, (FLUID["lc"]["Re"], par[0], par[1], 0.0))), *U, use_reentrant=False)
    J = (0.5 * (U[1] ** 2 + U[2] ** 2) / U[0] * S.vol).sum()
    grads = torch.autograd.grad(J, U0[:6] + par)
    keys = ("ro", "rou", "rov", "psixx", "psixy", "psiyy")
    return dict(J=float(J), dWi=float(grads[6]), dbeta=float(grads[7]),
                dstate=dict({k: t.cpu() for k, t in zip(keys, grads)}, psizz=None))


def exact(case, seed):
    kind, nodes = case["kind"], case["nside"] ** 2
    if kind == "steps" and (case["geometry"] != "periodic" or case["layers"]):
        return None  # boundary closures and layers: not restated here
    if case.get("adapt") or nodes * case["order"] ** 4 > 600_000 * 8 ** 4:
        return None
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind in ("steps", "first_step"):
        return _exact_steps(case, case["form"], seed)
    S = _Stencils(case["nside"], case["order"], seed)
    if kind == "setup":
        sums = S.sums.cpu()
        w = torch.nn.functional.pad(S.w, (0, 0, 0, NPLINK[case["order"]] - S.w.shape[1])).cpu()
        return dict(w_grad=w[:, :, :2].contiguous(), w_lap=w[:, :, 2].contiguous(), w_hyp=w[:, :, 3].contiguous(),
                    w_grad_sum=sums[:, :2].contiguous(), w_lap_sum=sums[:, 2].contiguous(), w_hyp_sum=sums[:, 3].contiguous(),
                    vol=S.vol.cpu(), count=None, count_small=None, links=None)
    phi = torch.from_numpy(_initial_2d(*_lattice(case["nside"], seed), "di", seed)[1]).to(S.vol.device)
    D = S.apply(phi[:, None], (0, 1, 2, 3))[:, :, 0]
    return dict(gradient=torch.stack([D[0], D[1]], 1).cpu(), laplacian=D[2].cpu(), filtered=(phi + D[3]).cpu(),
                filter_term=D[3].cpu())
