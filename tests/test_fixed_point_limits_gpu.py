"""The complex128 all-types pass where a block of the open diquark does not suit the
integer dots although P_n does: NaN and infinity in P_i or P_j, and products at both
ends of the exponent range.

Every output that the oracle makes non-finite must be non-finite, for every type and
projector; finite ones keep the 2e-15 of the norm that the two forms are off by 1.5 to
3e-16 of."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LATT = (4, 3, 3, 4)
V = int(np.prod(LATT))
BAD_SITE = 7
TOL = 2e-15


@pytest.fixture(scope="module")
def api():
    from contract_gb300 import api, build, pycontract
    build.build()
    pycontract.init(0)
    return api


def fields(sizes, same=False):
    rng = np.random.default_rng(3)
    ps = [s * (rng.standard_normal((V, 4, 4, 3, 3)) + 1j * rng.standard_normal((V, 4, 4, 3, 3))) for s in sizes]
    if same:
        ps[1] = ps[0]
    return ps


def run(api, ps, nproj=2, latt=None):
    import torch
    dev = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in ps]
    if ps[1] is ps[0]:
        dev[1] = dev[0]
    return api.baryon_all_types(*dev, 5, 5, api.projector_plus_minus()[:nproj], latt=latt).cpu().numpy()


def oracle(api, c_oracle, ps, nproj=2):
    pp = api.projector_plus_minus()[:nproj]
    return np.array([[c_oracle.baryon_general_two_point(*ps, t, 5, 5, w) for w in pp] for t in range(6)])


def off(got, ref):
    """Norm of the difference over the norm, in units near the largest value."""
    unit = 2.0 ** -np.floor(np.log2(np.abs(ref).max()))
    return np.linalg.norm((got - ref) * unit) / np.linalg.norm(ref * unit)


def timeslices(site):
    """Whether any site of each timeslice is marked: [Lt]."""
    return site.reshape(2, LATT[3], -1).any(axis=(0, 2))


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("size_n", [1e-2, 0.3, 1.0, 2.5, 10.0, 1e3])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, complex(0, np.nan)])
def test_not_finite(api, bad, size_n, same):
    ps = fields((1, 1, size_n), same)
    fine = [run(api, ps, n, latt) for n, latt in ((2, None), (2, LATT), (1, None))]
    for field in range(0, 3, 2 if same else 1):
        qs = list(ps)
        qs[field] = ps[field].copy()
        if field < 2:
            qs[field][BAD_SITE, 1, 2, 0, 1] = bad  # every type reads every entry of P_i and P_j
        else:
            qs[field][BAD_SITE] = bad  # a projector reads half of P_n
        if same and field == 0:
            qs[1] = qs[0]
        site = np.arange(V) == BAD_SITE
        for ref, n, latt, where in zip(fine, (2, 2, 1), (None, LATT, None), (site, timeslices(site), site)):
            got = run(api, qs, n, latt)
            assert not np.isfinite(got[:, :, where]).any(), (field, n, latt)
            # (the site that shares the warp takes the other form)
            assert off(got[:, :, ~where], ref[:, :, ~where]) <= TOL


# sizes of P_i, P_j and P_n: P_n suits the integer form, the diquark's blocks are at a limit
@pytest.mark.parametrize("sizes", [(1e-108, 1e-108, 1e-90), (1e-105, 1e-105, 1e-88), (1e-150, 1e-135, 1e-20),
                                   (1e107, 1e107, 1e88), (1e135, 1e85, 1e80), (1e-140, 1e120, 1.0)])
def test_limits(api, c_oracle, sizes):
    ps = fields(sizes)
    ref, got = oracle(api, c_oracle, ps), run(api, ps)
    assert np.isfinite(ref).all() and np.isfinite(got).all()
    assert off(got, ref) <= TOL, off(got, ref)


def test_overflow_and_underflow(api, c_oracle):
    ps = fields((1e112, 1e112, 1e90))  # results near 1e314
    assert not np.isfinite(oracle(api, c_oracle, ps)).any()
    assert not np.isfinite(run(api, ps)).any()
    ps = fields((1e-120, 1e-120, 1e-80))  # near 1e-320: a few units of the smallest number
    got, ref = run(api, ps), oracle(api, c_oracle, ps)
    assert np.isfinite(got).all() and np.abs(got - ref).max() < 1e-320
    ps = fields((1e-154, 1e-156, 1e80))  # a diquark of denormal numbers
    got, ref = run(api, ps), oracle(api, c_oracle, ps)
    assert off(got, ref) <= 1e-12


def test_wedge_of_small_colour_rows(api):
    """Two colour rows and columns far below the third, at the least field scale of the
    integer form, and a wedge's entry that cancels to a few of its units: its exponent
    must not run out of a double's range.  No entry exceeds the sizes of its products."""
    import torch
    from contract_gb300 import pycontract as pc
    s = 2.0 ** -100
    x = np.array([[1, s, s], [s, s * s, s * s * (1 + 2.0 ** -40)], [s, 0, 0]]) * 2.0 ** -299
    y = np.array([[1, s, s], [s, 0, 0], [s, s * s, s * s]]) * 2.0 ** -299
    rows = np.array([1, 1, 1, 0.5])[:, None, None, None]  # whatever the signs of Gamma_ij, they do not cancel
    pi = np.broadcast_to(rows * x, (V, 4, 4, 3, 3)).astype(complex, order="C")
    pj = np.broadcast_to(y, (V, 4, 4, 3, 3)).astype(complex, order="C")
    got = pc.baryonDiquark(torch.from_numpy(pi).cuda(), torch.from_numpy(pj).cuda(), 5, 5).cpu().numpy()
    size = np.zeros((3, 3))
    for a in range(3):
        for e in range(3):
            for b, c in ((1, 2), (2, 1)):
                for f, g in ((1, 2), (2, 1)):
                    size[a, e] += x[(a + b) % 3, (e + f) % 3] * y[(a + c) % 3, (e + g) % 3]
    assert (np.abs(got.reshape(V, 4, 4, 3, 3)) <= 4 * size).all()
