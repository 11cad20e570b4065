"""The set-up kernels at the sizes where they can go wrong: the device's bank-aware link order
against the host's, the weight build over several batches and at order 10, the tile halos of a
stencil too wide for the smaller hash set, and the tiles of small sets, whose nodes' links
several threads share.

The link order is compared entry by entry; the weights bit for bit with the restatement (both
round every operation alike, with its correctly rounded x^4), except the filter's, which CUDA's
and glibc's cos separate in the last bit (1e-13, as in the parity tests); the right-hand
sides of the wide stencil, whose sums run in another order, within 1e-10 of their terms.
"""
import ctypes as C
import os

import numpy as np
import pytest

from sunset_viscoelastic_b200 import labfm
from sunset_viscoelastic_b200.nodesets import initial_state, jittered_lattice
import oracle as O

pytestmark = pytest.mark.gpu
HOSTCHECK = os.path.join(os.path.dirname(labfm.library_path()), "libsunset_hostcheck.so")


def sell_at(base, k, lane):
    return base + ((k >> 1) << 6) + (lane << 1) + (k & 1)


# (links a lane at most, slices, lanes without links, share of small links)
@pytest.mark.parametrize("group", [8, 16])
@pytest.mark.parametrize("most,slices,empty,small", [(1, 3, 0, 1.0), (2, 5, 31, 0.5), (37, 7, 5, 0.6), (92, 6, 0, 1.0),
                                                     (92, 5, 3, 0.0), (333, 2, 1, 0.8)])
def test_link_order_equals_the_hosts(group, most, slices, empty, small):
    rng = np.random.default_rng(most + group)
    cnt = rng.integers(max(1, most // 2), most + 1, (slices, 32)).astype(np.int32)
    cnt[-1, 32 - empty:] = 0
    cs = np.floor(cnt * np.minimum(1.0, small + 0.1 * rng.random(cnt.shape) * (small not in (0.0, 1.0)))).astype(np.int32)
    w = ((cnt.max(1) + 1) & ~1).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum(32 * w.astype(np.int64))])
    pos = rng.integers(0, 900, int(ptr[-1])).astype(np.uint16)
    pos[rng.random(pos.size) < 0.2] |= np.uint16(1 << 14)  # reflection codes ride in the top bits
    lib, host = labfm.load_library(), C.CDLL(HOSTCHECK)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    got = np.full(int(ptr[-1]), -7, np.int32)
    assert lib.sunset_check_deal(group, slices, p(ptr), p(w), p(cnt), p(cs), p(pos), int(w.max()), p(got)) == 0
    for s in range(slices):
        lists = [[[sell_at(int(ptr[s]), k, r) for k in range(*rng_)] for r, rng_ in enumerate(rows)]
                 for rows in ([(0, int(cs[s, r])) for r in range(32)], [(int(cs[s, r]), int(cnt[s, r])) for r in range(32)])]
        flat = [np.array([e for row in rows for e in row] or [0], np.int32) for rows in lists]
        off = [np.concatenate([[0], np.cumsum([len(row) for row in rows])]).astype(np.int32) for rows in lists]
        want = np.full(int(w[s]) * 32, -7, np.int32)
        host.sunset_hostcheck_deal(group, p(pos), p(flat[0]), p(off[0]), p(flat[1]), p(off[1]), int(w[s]), p(want))
        mine = np.array([[got[sell_at(int(ptr[s]), k, r)] for r in range(32)] for k in range(int(w[s]))])
        assert np.array_equal(mine, want.reshape(-1, 32))


def pair(ns, order, h_over_s, **kw):
    O.set_pow_mode(True)
    try:
        ref = O.Oracle(form="di", order=order, h_over_s=h_over_s, **kw).build_domain(ns).setup()
    finally:
        O.set_pow_mode(False)
    return ref, labfm.Sunset(form="di", order=order, h_over_s=h_over_s, **kw).build_domain(ns).setup()


# 183^2 nodes are one batch of 32,768 and a ragged one; the record of order 4 does not hold every
# node's rotations, so some take a second round
@pytest.mark.parametrize("order,nside,radius", [(4, 183, 3.0), (10, 31, 7.0)])
def test_weights_equal_the_restatements(order, nside, radius):
    ref, gpu = pair(jittered_lattice(nside), order, radius / 2)
    a, b = gpu.weights(), ref.weights()
    for k in ("w_grad", "w_lap", "w_grad_sum", "w_lap_sum"):
        assert np.array_equal(a[k], b[k]), k
    assert np.abs(a["w_hyp"] - b["w_hyp"]).max() <= 1e-13 * np.abs(b["w_hyp"]).max()


def test_wide_stencil_halos():
    ns = jittered_lattice(64)
    ref, gpu = pair(ns, 4, 15.5 / 2)
    st = initial_state(ns)
    st["cxx"] = 1.0 + 0.2 * np.sin(2 * np.pi * ns.x)
    for g in (ref, gpu):
        g.set_state(**st)
    a, b = gpu.rhs(), ref.rhs()
    # the largest term: the viscous force, (1 / s^2) |u|, and the pressure gradient, c^2 |grad rho|
    for k in ("ro", "rou", "rov", "xx", "xy", "yy"):
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * max(1.0, np.abs(b[k]).max()), k


# 2 n_SM = 296 tiles at most: tiles of 1, 1 (the largest such set), 2, 4 and 8 slices on 148 SMs
@pytest.mark.parametrize("form,order", [("di", 4), ("lc", 4), ("chl", 6)])
@pytest.mark.parametrize("nside", [17, 97, 98, 150, 201])
def test_small_set_tiles(nside, form, order):
    ns = jittered_lattice(nside)
    O.set_pow_mode(True)
    try:
        ref = O.Oracle(form=form, order=order, h_over_s={4: 1.5, 6: 2.1}[order]).build_domain(ns).setup()
    finally:
        O.set_pow_mode(False)
    gpus = [labfm.Sunset(form=form, order=order, h_over_s={4: 1.5, 6: 2.1}[order], precision=p).build_domain(ns).setup()
            for p in ("fp64", "mixed")]
    st = initial_state(ns)
    st["ro"] = 1.0 + 0.01 * np.cos(2 * np.pi * ns.x)
    st["cxx"] = 1.3 + 0.2 * np.sin(2 * np.pi * ns.x)
    st["cxy"] = 0.1 * np.cos(2 * np.pi * ns.y)
    for g in [ref] + gpus:
        g.set_state(**st)
    a, b = gpus[0].rhs(), ref.rhs()
    for k in ("ro", "rou", "rov", "xx", "xy", "yy"):
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * max(1.0, np.abs(b[k]).max()), k
    dt = 0.1 / (nside * nside)
    for g in [ref] + gpus:
        g.step(dt, 3)
    want = ref.state()
    for g, tol in zip(gpus, (1e-10, 1e-6)):  # mixed: the tolerance its fields keep over 100 steps
        got = g.state()
        for k in ("ro", "u", "v", "cxx", "cxy", "cyy"):
            assert np.abs(got[k] - want[k]).max() <= tol * max(1.0, np.abs(want[k]).max()), k


# Whole tiles on either side of a full wave (444 tiles on 148 SMs at three blocks each): 337^2
# nodes fill it with the ring two pairs deep, 338^2 begin another with the ring three deep.  The
# sums' rounding, eps * 20 |u| / s^2 = 5e-10, is 1e-11 of the largest right-hand side.
@pytest.mark.parametrize("form,order", [("di", 4), ("chl", 6), ("lc", 4)])
@pytest.mark.parametrize("nside", [337, 338])
def test_ring_depths(nside, form, order):
    ns = jittered_lattice(nside)
    kw = dict(form=form, order=order, h_over_s={4: 1.5, 6: 2.1}[order])
    O.set_pow_mode(True)
    try:
        ref = O.Oracle(**kw).build_domain(ns).setup()
    finally:
        O.set_pow_mode(False)
    gpu = labfm.Sunset(**kw).build_domain(ns).setup()
    st = initial_state(ns)
    st["cxx"] = 1.3 + 0.2 * np.sin(2 * np.pi * ns.x)
    for g in (ref, gpu):
        g.set_state(**st)
    a, b = gpu.rhs(), ref.rhs()
    for k in ("ro", "rou", "rov", "xx", "xy", "yy"):
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * max(1.0, np.abs(b[k]).max()), k
