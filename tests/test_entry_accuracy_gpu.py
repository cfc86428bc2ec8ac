"""Complex128 results entry by entry, on fields whose colour blocks are near diagonal,
near triangular or of one size, and whose spin blocks differ: an entry made of small
values must keep the bits that FP64 keeps, whichever pipe sums it.

Each entry's error is measured against the sum of the sizes of the products that make
it, in extended precision.  Bounds: a sum of n products in FP64 is off by at most
n 2^-53 of that, and usually by its square root.  One entry of a field: 64 real
products at most (four wedges' complex products, twice, or the closed loop's), so
32 x 2^-53 = 3.6e-15 leaves a factor of five over what FP64 shows (6e-16 over 200 000
entries).  A correlator sums a few thousand products of three: sqrt(4000) is 64 and the
same bound holds.  Values cut at a common scale are off by the inverse of the ratio of
two entries: 1e-13 for a thousandth."""
from unittest import mock

import numpy as np
import pytest

from oracle import einsum_oracle as eo

pytestmark = pytest.mark.gpu
V = 12
BOUND = 32 * 2.0 ** -53
KINDS = ["gauss", "diagonal 0.3", "diagonal 0.1", "diagonal 1e-2", "diagonal 1e-4", "diagonal 1e-8", "diagonal 1e-12",
         "triangular 1e-3", "one entry 1e-5", "spin rows", "spin columns", "crossed"]


def field(rng, kind, which):
    p = rng.standard_normal((V, 4, 4, 3, 3)) + 1j * rng.standard_normal((V, 4, 4, 3, 3))
    name, _, eps = kind.rpartition(" ")
    if name == "diagonal":
        p = p * np.where(np.eye(3) > 0, 1, float(eps))
    elif name == "triangular":
        p = p * np.where(np.tri(3) > 0, 1, float(eps))
    elif name == "one entry":
        p[..., 1, 2] *= float(eps)
    elif kind == "spin rows":
        p = p * np.array([1, 1e-5, 1, 1e-3])[None, :, None, None, None]
    elif kind == "spin columns":
        p = p * np.array([1e-4, 1, 1e-7, 1])[None, None, :, None, None]
    elif kind == "crossed":  # the three fields have their large entries in different places
        p = p * np.where(np.roll(np.eye(3), which, axis=1) > 0, 1, 1e-6)
    return np.ascontiguousarray(p)


@pytest.fixture(scope="module")
def api():
    from contract_gb300 import api, build, pycontract
    build.build()
    pycontract.init(0)
    return api


def fields(kind):
    import torch
    rng = np.random.default_rng(KINDS.index(kind) + 40)
    ps = [field(rng, kind, k) for k in range(3)]
    return ps, [torch.from_numpy(p).cuda() for p in ps]


def exact(f, ps, *args):
    """f in extended precision, and the sum of the sizes of its products."""
    ref = f(*[p.astype(np.clongdouble) for p in ps], *args)
    with mock.patch.multiple(eo, EPS=np.abs(eo.EPS), GAMMA=np.abs(eo.GAMMA), G5=np.abs(eo.G5)):
        size = np.abs(f(*[np.abs(p).astype(complex) for p in ps], *[np.abs(a) if isinstance(a, np.ndarray) else a for a in args]))
    return ref, size


def check(got, ref, size, what):
    err = np.abs(got.astype(np.clongdouble).reshape(ref.shape) - ref).astype(float)
    assert (err[size == 0] == 0).all(), what
    worst = (err[size > 0] / size[size > 0]).max()
    assert worst <= BOUND, (what, worst)


@pytest.mark.parametrize("kind", KINDS)
def test_fields(api, kind):
    from contract_gb300 import pycontract as pc
    ps, dev = fields(kind)
    check(pc.baryonDiquark(dev[0], dev[1], 6, 13).cpu().numpy(), *exact(eo.baryon_diquark, ps[:2], 6, 13), "diquark")
    for t in range(6):
        for slot in range(3):
            d = [x.clone() for x in dev]
            pc.baryonSequentialTwoPoint(*d, t, slot, 6, 13, 9)
            check(d[slot].cpu().numpy(), *exact(eo.baryon_sequential, ps, t, slot, 6, 13, 9), (t, slot))


@pytest.mark.parametrize("kind", KINDS)
def test_correlators(api, kind):
    ps, dev = fields(kind)
    pp = api.projector_plus_minus()
    rng = np.random.default_rng(11)
    wd = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    every = api.baryon_all_types(*dev, 6, 13, pp).cpu().numpy()
    one = api.baryon_all_types(*dev, 6, 13, pp[:1]).cpu().numpy()
    for t in range(6):
        for k, w in enumerate(pp):
            ref, size = exact(eo.baryon_general_two_point, ps, t, 6, 13, w.reshape(4, 4))
            check(every[t, k], ref, size, ("all types", t, k))
            if k == 0:
                check(one[t, 0], ref, size, ("all types, one projector", t))
                check(api.baryon(*dev, t, 6, 13, project_mn=w).cpu().numpy(), ref, size, ("rank 2", t))
        for name, w in (("dense", wd), ("rank 1", np.outer(wd[0], wd[1]))):
            check(api.baryon(*dev, t, 6, 13, project_mn=w).cpu().numpy(),
                  *exact(eo.baryon_general_two_point, ps, t, 6, 13, w), (name, t))
        check(api.baryon(*dev, t, 6, 13, gamma_mn=9).cpu().numpy(), *exact(eo.baryon_two_point, ps, t, 6, 13, 9), ("gamma", t))


@pytest.mark.parametrize("kind", KINDS)
def test_mesons(api, kind):
    from contract_gb300 import pycontract as pc
    ps, dev = fields(kind)
    for g in (6, 9):
        for source in (True, False):
            got = np.array([x.cpu().numpy() for x in pc._meson_all(dev[0], dev[1], g, source)])
            check(got.reshape(16, V), *exact(eo.meson_all_source if source else eo.meson_all_sink, ps[:2], g), (g, source))
