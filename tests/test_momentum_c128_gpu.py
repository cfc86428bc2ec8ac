"""The complex128 meson momentum projection: pairs of a site in integers or FP64
(MesonPairs), and the plane transform that takes sites x, Lx - x and rows y,
Ly - y together.  Where it can go wrong: sites and rows without a partner (the
first, the middle one of an even extent), lists without nx = 0, without the
partners +n / -n, with one component more than once modulo the extent, more Y
groups than one launch's chunk, every number of X groups; sites that the integer
form refuses.

Against the FP64 oracle, relative to max(|C|, sigma, L1), L1 the size of the
products: 1e-14.  The oracle's phases are exp() of an angle of up to 19, off by
2e-15; a wrong partner or sign is an error of order one, a lost low word 1e-9."""
import ctypes

import numpy as np
import pytest

from oracle import einsum_oracle as eo

pytestmark = pytest.mark.gpu
TOL = 1e-14
MOMENTA = {
    "zero": [(0, 0, 0)],
    "no zero": [(1, 0, 0), (-1, 1, 0), (1, 1, 1)],
    "unpaired": [(0, 0, 0), (1, 0, 0), (0, 2, 1), (0, -1, 0)],
    "modulo": [(0, 0, 0), (1, 1, 0), (7, 1, 2), (1, 6, 0), (-5, -4, 0), (6, 5, 5)],
    "27": list(map(tuple, eo.momentum_list(1))),
    "125": list(map(tuple, eo.momentum_list(2))),
    "one nx, 25 ny": [(0, n, 0) for n in range(-12, 13)],
    "eight nx": [(n, n * n - 3, 1) for n in range(8)],
    "28 groups": [(x, y, 0) for x in range(-3, 4) for y in range(-3, 4)],
}


@pytest.fixture(scope="module")
def lib():
    from contract_gb300 import _lib, build, pycontract
    build.build()
    pycontract.init(0)
    lib = _lib.lib()
    lib.contract_set_error_mode(1)
    return lib


def run(lib, pi, pj, latt, moms, prec=0):
    import torch
    dt = torch.complex64 if prec else torch.complex128
    a = torch.from_numpy(np.ascontiguousarray(pi)).cuda().to(dt)
    b = a if pj is pi else torch.from_numpy(np.ascontiguousarray(pj)).cuda().to(dt)
    out = torch.full((len(moms), latt[3], 256), float("nan"), dtype=torch.complex128, device="cuda")
    flat = (ctypes.c_int * (3 * len(moms)))(*[n for m in moms for n in m])
    lib.contract_meson_all_gamma_momentum(out.data_ptr(), a.data_ptr(), b.data_ptr(), int(np.prod(latt)),
                                          (ctypes.c_int * 4)(*latt), flat, len(moms), prec)
    torch.cuda.synchronize()
    assert lib.contract_last_error() == 0, lib.contract_last_error_message()
    return out.cpu().numpy()


def check(latt, pi, pj, moms, got, tol=TOL):
    site = eo.meson_all_gamma(pi, pj).reshape(256, -1)
    ref = eo.momentum_project(site, latt, moms).transpose(1, 2, 0)
    sig = np.sqrt(eo.timeslice_sum(np.abs(site) ** 2, latt).real).T[None]
    scale = np.maximum(np.maximum(np.abs(ref), sig), eo.meson_product_l1(pi, pj, latt))
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) / scale).max() < tol, (latt, (np.abs(got - ref) / scale).max())


@pytest.mark.parametrize("moms", list(MOMENTA))
@pytest.mark.parametrize("latt", [(2, 1, 1, 1), (2, 2, 3, 2), (6, 5, 2, 3), (8, 4, 3, 2), (10, 7, 1, 2)])
def test_lists(lib, latt, moms):
    pi, pj = eo.make_propagator(latt, 3, 0.2), eo.make_propagator(latt, 4, 0.25)
    if moms == "27":
        pj = pi
    check(latt, pi, pj, MOMENTA[moms], run(lib, pi, pj, latt, MOMENTA[moms]))


@pytest.mark.parametrize("kind", ["spin rows", "uneven", "zero blocks", "large", "small", "some sites"])
def test_values(lib, kind):
    latt = (6, 5, 2, 3)
    rng = np.random.default_rng(5)
    pi, pj = eo.make_propagator(latt, 3, 0.2), eo.make_propagator(latt, 4, 0.25)
    v = pi.shape[0]
    if kind == "spin rows":
        pi = pi * np.array([1, 1e-3, 1, 1e-6])[None, :, None, None, None]
    elif kind == "uneven":
        pi, pj = (p * 2.0 ** rng.integers(-4, 5, (v, 4, 4, 1, 1)) for p in (pi, pj))
    elif kind == "zero blocks":
        pi = pi * (rng.random((v, 4, 4, 1, 1)) < 0.6)
        pi[::7] = 0
    elif kind == "large":
        pi, pj = pi * 1e120, pj * 1e30
    elif kind == "small":
        pi, pj = pi * 1e-120, pj * 1e-80
    else:  # sites of a warp that differ: one refused, one denormal
        pi[::5, 0] *= 1e-9
        pi[1] *= 1e-310
    check(latt, pi, pj, MOMENTA["27"], run(lib, pi, pj, latt, MOMENTA["27"]))


def test_every_value_at_its_largest(lib):
    """All components of a block at the top of their power of two, in phase: the
    integer sums at their largest."""
    latt = (4, 3, 2, 2)
    one = np.full((int(np.prod(latt)), 4, 4, 3, 3), np.nextafter(2.0, 0) * (1 + 1j))
    check(latt, one, one, MOMENTA["27"], run(lib, one, one, latt, MOMENTA["27"]))


def test_planes_of_the_mixed_form(lib):
    """The same transform in FP32 (the mixed form's three kernels)."""
    import subprocess
    import sys
    code = ("import sys; sys.path[:0] = %r\nimport test_momentum_c128_gpu as m, ctypes\n"
            "from contract_gb300 import _lib, pycontract\npycontract.init(0); lib = _lib.lib()\n"
            "eo = m.eo\n"
            "for latt in ((6, 5, 2, 3), (8, 4, 3, 2)):\n"
            "  pi, pj = eo.make_propagator(latt, 3, 0.2), eo.make_propagator(latt, 4, 0.25)\n"
            "  for k in ('modulo', '125', '28 groups'):\n"
            "    m.check(latt, pi, pj, m.MOMENTA[k], m.run(lib, pi, pj, latt, m.MOMENTA[k], 1), 1e-6)\n")
    import os
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, CONTRACT_MOMENTUM_UNFUSED="1")
    r = subprocess.run([sys.executable, "-c", code % ([here, os.path.dirname(here)],)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
