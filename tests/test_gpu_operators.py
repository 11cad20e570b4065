"""The gradient operator with device pointers (SUNSET_PTR_DEVICE): the same values as with host
arrays and, on periodic sets, the restatement's, bit for bit; odd node counts, and an output that is
aligned to 8 bytes only."""
import ctypes as C

import numpy as np
import pytest
import torch

from sunset_viscoelastic_b200 import labfm
from sunset_viscoelastic_b200.nodesets import channel, jittered_lattice
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [jittered_lattice(9), jittered_lattice(41), channel(20)], ids=["81", "1681", "walls"])
def test_gradient_with_device_pointers(ns):
    kw = dict(form="di", order=6, h_over_s=0.0 if len(ns.x) != 81 else 1.5)
    O.set_pow_mode(True)
    try:
        ref = O.Oracle(**kw).build_domain(ns).setup()
    finally:
        O.set_pow_mode(False)
    g = labfm.Sunset(**kw).build_domain(ns).setup()
    n = g.sizes()[1]
    phi = np.random.default_rng(n).standard_normal(n)
    want = g.gradient(phi)
    if not (ns.node_type <= 2).any():  # walls: atan and cos of their frames may differ in the last bit
        assert np.array_equal(want, ref.gradient(phi))
    lib = C.CDLL(labfm.library_path())
    x = torch.from_numpy(phi).cuda()
    for out in (torch.full((n, 2), float("nan"), dtype=torch.float64, device="cuda"),
                torch.zeros(2 * n + 1, dtype=torch.float64, device="cuda")[1:]):  # 8-byte aligned only
        torch.cuda.synchronize()
        assert lib.sunset_calc_gradient(g.h, C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr()), 1) == 0
        assert np.array_equal(out.cpu().numpy().reshape(n, 2), want)


def test_gradient_after_queued_work():
    """Work queued on the default stream before the call and touching the output comes first: the
    array is filled behind a second or so of matrix products that are still running when the call
    is made, and read by a copy queued behind them, which must see the fill."""
    ns = jittered_lattice(41)
    g = labfm.Sunset(form="di", order=6, h_over_s=2.1).build_domain(ns).setup()
    n = g.sizes()[1]
    phi = np.random.default_rng(3).standard_normal(n)
    want = g.gradient(phi)
    lib = C.CDLL(labfm.library_path())
    x = torch.from_numpy(phi).cuda()
    a = torch.full((8192, 8192), 1.0 / 8192, device="cuda")
    out = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    a @ a
    torch.cuda.synchronize()
    for _ in range(40):
        a = a @ a
    out.fill_(7.0)
    before = out.clone()
    assert lib.sunset_calc_gradient(g.h, C.c_void_p(x.data_ptr()), C.c_void_p(out.data_ptr()), 1) == 0
    assert np.array_equal(out.cpu().numpy(), want)
    assert bool((before == 7.0).all())
    g.close()
