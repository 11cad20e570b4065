"""The routes of the FP64 time step on periodic and symmetric sets of more than 75,776 nodes, which
take whole tiles of 256 nodes (smaller ones split them, 8 n_SM slices on 148 SMs): every form with FENE-P
and polymer diffusion, with the stage's link ring two and three pairs deep, against the CPU
restatement.  Each case states the route it is there for, and the library is asked for it.

The ring is three pairs deep where the last wave of blocks is at most half full and the third pair
costs no resident block (338^2 nodes with eight gathered fields are 64 bytes a block over): 298 tiles (276^2 nodes) fit one wave of three blocks a SM (444) and begin a
second one of two blocks, which the wide stencils (halos of 868 nodes) leave; 447 tiles (338^2)
begin a second wave of 444; the Newtonian form has four blocks a SM, 625 tiles (400^2) begin its
second wave, and with the wide stencil it gives one of them up.  With FENE-P and ten or eleven
gathered fields the ring stays at two pairs.

The sums' rounding, eps * 20 |u| / s^2 = 5e-10 in the viscous terms, is 1e-11 of the largest
right-hand side; 1e-10 of it is allowed, as in the set-up's tests.

The same for channels with walls, which keep whole tiles at every size: up to one tile a SM the ring
is two or four pairs deep by the fields, the lists and the tiles, above two or three as without walls.

And the tile halos of a stencil that reaches more than 2048 nodes from a tile, where the hash set
that gathers them takes its larger size (mixed precision keeps whole tiles on small sets)."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from sunset_viscoelastic_b200 import labfm
from sunset_viscoelastic_b200.nodesets import channel, initial_state, jittered_lattice, poiseuille_state
import oracle as O

pytestmark = pytest.mark.gpu


def tiles(g):
    """slices a tile, tiles, largest halo, pairs in the stage's ring"""
    out = (C.c_int * 4)()
    assert labfm.load_library().sunset_check_tiles(g.h, out) == 0
    return tuple(out)


def pair(ns, **kw):
    O.set_pow_mode(True)
    try:
        okw = {k: v for k, v in kw.items() if k != "precision"}
        ref = O.Oracle(**okw).build_domain(ns).setup()
    finally:
        O.set_pow_mode(False)
    return ref, labfm.Sunset(**kw).build_domain(ns).setup()


def fields(ns, form):
    st = initial_state(ns)
    x, y = ns.x, ns.y
    st["ro"] = 1.0 + 0.01 * np.cos(2 * np.pi * x)
    st["cxx"] = 1.5 + 0.4 * np.sin(2 * np.pi * y) ** 2
    st["cxy"] = 0.3 * np.sin(2 * np.pi * x) * np.cos(2 * np.pi * y)
    st["cyy"] = 1.2 + 0.2 * np.cos(2 * np.pi * x)
    st["czz"] = np.ones(ns.n) if form == "lc" else 1.1 + 0.1 * np.sin(2 * np.pi * (x + y))
    return st


FENEP, MDIFF = dict(fenep=True, fenep_l2=100.0), dict(Mdiff=1e-3)
BOTH = dict(FENEP, **MDIFF)
# form, options, nodes a side, radius over spacing, pairs in the ring
CASES = [("di", FENEP, 276, 3.0, 2), ("di", FENEP, 338, 3.0, 3), ("di", MDIFF, 276, 3.0, 2), ("di", MDIFF, 338, 3.0, 3),
         ("di", BOTH, 276, 3.0, 2), ("di", BOTH, 338, 3.0, 2), ("di", BOTH, 276, 5.0, 3),
         ("chl", FENEP, 276, 3.0, 2), ("chl", FENEP, 338, 3.0, 3), ("chl", MDIFF, 276, 3.0, 2), ("chl", MDIFF, 276, 5.0, 3),
         ("chl", BOTH, 338, 3.0, 2), ("chl", BOTH, 276, 3.0, 2),
         ("lc", {}, 276, 5.0, 3), ("lc", FENEP, 276, 3.0, 2), ("lc", FENEP, 276, 5.0, 2),
         ("newt", {}, 276, 3.0, 2), ("newt", {}, 338, 3.0, 2), ("newt", {}, 400, 3.0, 3), ("newt", {}, 400, 5.0, 3)]


def check(ns, form, kw, ring):
    ref, gpu = pair(ns, form=form, **kw)
    route = tiles(gpu)
    assert route[0] == 8 and route[3] == ring, route
    st = fields(ns, form)
    for g in (ref, gpu):
        g.set_state(**st)
    a, b = gpu.rhs(), ref.rhs()
    for k in b:
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * max(1.0, np.abs(b[k]).max()), k
    dt = 0.1 / ns.n
    for g in (ref, gpu):
        g.step(dt, 3)
    a, b = gpu.state(), ref.state()
    for k in ("ro", "u", "v") + (() if form == "newt" else ("cxx", "cxy", "cyy", "czz")):  # no polymer: no c
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * max(1.0, np.abs(b[k]).max()), k
    gpu.close()


@pytest.mark.parametrize("form,options,nside,radius,ring", CASES,
                         ids=[f"{f}{'-fenep' if 'fenep' in o else ''}{'-mdiff' if 'Mdiff' in o else ''}-{n}-r{r:g}"
                              for f, o, n, r, _ in CASES])
def test_whole_tiles(form, options, nside, radius, ring):
    check(jittered_lattice(nside), form, dict(options, order=4, h_over_s=radius / 2), ring)


@pytest.mark.parametrize("form,ring", [("di", 2), ("chl", 2), ("lc", 2), ("newt", 2)])
def test_whole_tiles_symmetric(form, ring):
    ns = dataclasses.replace(jittered_lattice(276), bcond=(1, 1, 2, 2))
    check(ns, form, dict(order=4, h_over_s=1.5), ring)


# form, order, cells across, options, pairs in the ring: 10, 89, 158, 308 and 453 tiles on 148 SMs
WALLS = [("di", 6, 48, {}, 4), ("newt", 6, 48, {}, 4), ("chl", 6, 48, FENEP, 4), ("di", 6, 48, BOTH, 2), ("chl", 6, 48, MDIFF, 2),
         ("chl", 6, 150, MDIFF, 4), ("lc", 6, 48, {}, 2), ("lc", 6, 150, {}, 4), ("lc", 6, 150, FENEP, 4), ("lc", 4, 150, FENEP, 2),
         ("chl", 6, 48, BOTH, 4), ("chl", 4, 48, BOTH, 2), ("di", 6, 200, BOTH, 2), ("chl", 6, 280, BOTH, 2),
         ("di", 6, 200, {}, 2), ("chl", 6, 200, {}, 2), ("lc", 6, 200, {}, 2), ("di", 6, 200, MDIFF, 2), ("chl", 6, 200, FENEP, 2),
         ("di", 4, 340, {}, 3), ("chl", 4, 340, {}, 3), ("lc", 6, 280, {}, 3), ("lc", 6, 280, FENEP, 2), ("newt", 4, 340, {}, 3)]


@pytest.mark.parametrize("form,order,ny,options,ring", WALLS,
                         ids=[f"{f}-o{o}-{n}{'-fenep' if 'fenep' in k else ''}{'-mdiff' if 'Mdiff' in k else ''}"
                              for f, o, n, k, _ in WALLS])
def test_walled_tiles(form, order, ny, options, ring):
    grav = 8.0
    ns = channel(ny)
    ref, gpu = pair(ns, form=form, order=order, Re=1.0, Wi=0.5, beta=0.59, Ma=0.1, grav=(grav, 0.0, 0.0),
                    kolmogorov_forcing=0, **options)
    route = tiles(gpu)
    assert route[0] == 8 and route[3] == ring, route
    nd, npfb = ref.nodes(), ref.sizes()[1]
    x, y, t = nd["x"][:npfb], nd["y"][:npfb], nd["node_type"][:npfb]
    st = poiseuille_state(type("P", (), {"y": y, "n": npfb}), grav, 1.0, 0.5)
    st["u"] = st["u"] + 0.3 * np.sin(2 * np.pi * x) * y * (1.0 - y)
    st["v"] = 0.2 * np.cos(2 * np.pi * x) * y * (1.0 - y)
    st["ro"] = 1.0 + 0.01 * np.sin(2 * np.pi * x) * np.cos(np.pi * y)
    st["cxx"] = st["cxx"] + 0.1 * np.sin(2 * np.pi * x) ** 2
    st["cyy"] = st["cyy"] + 0.05 * np.cos(np.pi * y) ** 2
    for g in (ref, gpu):
        g.set_state(**st)
    a, b = gpu.rhs(), ref.rhs()
    # 1e-10 of the terms, as on the small channels, and eight roundings of the viscous sums, whose
    # terms are 20 |u| / s^2 (the weights of the rows next to walls agree to rounding only)
    gu = np.abs(ref.gradient(st["u"])).max()
    scale = max(gu, *(np.abs(b[k]).max() for k in ("rou", "rov"))) * max(1.0, *(np.abs(st[k]).max() for k in ("cxx", "cyy")))
    bound = 1e-10 * scale + 8 * 2.2e-16 * 20 * ny * ny
    for k in b:
        assert np.abs(a[k] - b[k]).max() <= bound, k
    dt = 0.3 * min(ref.set_tstep())
    for g in (ref, gpu):
        g.step(dt, 3)
    a, b = gpu.state(), ref.state()
    for k in ("ro", "u", "v") + (() if form == "newt" else ("cxx", "cxy", "cyy")):
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * max(1.0, np.abs(b[k]).max()), k
    assert np.all(a["rou"][t == 0] == 0.0)
    gpu.close()


def test_halos_of_more_than_2048_nodes():
    ns = jittered_lattice(64)
    ref, gpu = pair(ns, form="di", order=4, h_over_s=17.0 / 2, precision="mixed")
    assert tiles(gpu)[0] == 8 and tiles(gpu)[2] > 2048
    st = fields(ns, "di")
    for g in (ref, gpu):
        g.set_state(**st)
        g.step(0.1 / ns.n, 3)
    a, b = gpu.state(), ref.state()
    for k in ("ro", "u", "v", "cxx", "cxy", "cyy"):  # the tolerance mixed fields keep over 100 steps
        assert np.abs(a[k] - b[k]).max() <= 1e-6 * max(1.0, np.abs(b[k]).max()), k
    gpu.close()
