"""Distinct handles are independent: two handles of different configurations (log-conformation
at order 6 and the direct form at order 4, different Wi and epsPTT), stepped at the same time
from two host threads, end bit for bit where each ends when stepped alone.  The library's
calls release the interpreter lock (ctypes), so the two threads' launches interleave on the
device; each kernel takes its run's constants as a launch parameter.
"""
import dataclasses
import threading

import numpy as np
import pytest

from sunset_viscoelastic_b200 import labfm
from sunset_viscoelastic_b200.nodesets import WORKLOADS, initial_state, jittered_lattice

pytestmark = pytest.mark.gpu


def make(name, **over):
    wl = dataclasses.replace(WORKLOADS[name], nside=48)
    ns = wl.nodes()
    g = labfm.for_workload(wl, ns, **over).setup()
    st = initial_state(ns)
    return g, wl, st


def run(g, st, dt, n, out, key):
    g.set_state(**st)
    for _ in range(n):
        g.step(dt, 5)
    out[key] = g.state()


def test_two_configurations_from_two_threads():
    a, wa, sa = make("periodic-lc-o6-262k", Wi=1.0, epsPTT=0.25)
    b, wb, sb = make("periodic-di-o4-16k", Wi=0.5, epsPTT=0.1)
    for g, st in ((a, sa), (b, sb)):
        g.set_state(**st)
    dta = 0.3 * min(a.set_tstep())
    dtb = 0.3 * min(b.set_tstep())
    alone = {}
    run(a, sa, dta, 8, alone, "a")
    run(b, sb, dtb, 8, alone, "b")
    together = {}
    ta = threading.Thread(target=run, args=(a, sa, dta, 8, together, "a"))
    tb = threading.Thread(target=run, args=(b, sb, dtb, 8, together, "b"))
    ta.start()
    tb.start()
    ta.join(300)
    tb.join(300)
    assert set(together) == {"a", "b"}
    for key in ("a", "b"):
        for f in ("ro", "rou", "rov", "cxx", "cxy", "cyy"):
            assert np.array_equal(together[key][f], alone[key][f]), (key, f)
    a.close()
    b.close()


def test_wide_and_narrow_lists_from_two_threads():
    """Set-ups in several threads: lists whose halos need the larger hash set in shared memory
    (900 links a node; mixed precision keeps whole tiles) in one, ordinary ones in the others.  A
    kernel's limit of dynamic shared memory is the process's, so no set-up may lower it between
    another's call and launch."""
    ns = jittered_lattice(64)
    errors, stop = [], threading.Event()

    def build(radius, n):
        try:
            for _ in range(n):
                if stop.is_set():
                    return
                g = labfm.Sunset(form="di", order=4, h_over_s=radius / 2, precision="mixed").build_domain(ns)
                g.find_neighbours()
                g.close()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append((radius, str(e)))
        finally:
            if radius > 10.0:
                stop.set()

    narrow = [threading.Thread(target=build, args=(3.0, 100000)) for _ in range(3)]
    wide = threading.Thread(target=build, args=(17.0, 600))
    for t in narrow + [wide]:
        t.start()
    wide.join(120)
    stop.set()
    for t in narrow:
        t.join(120)
    assert not errors, errors[0]
