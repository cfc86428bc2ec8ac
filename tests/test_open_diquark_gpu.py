"""The all-types pass (open diquark, one warp per tile) where it can go wrong:
half-timeslices of one site and of sizes no tile divides, every way of
applying the open spin slot, one field or two for P_i and P_j, both precisions,
per site and per timeslice, and every pair of Gamma matrices, against the FP64
oracle.

Tolerances: complex128 outputs are sums of about 3000 products per site, so
their rounding is a few 1e-15 of the largest value; 1e-12 as in the other
complex128 tests.  complex64: 1e-6 of max(|C|, the largest per-timeslice
spread of the call's outputs), the bound of the mixed forms (types that vanish
identically for one field are rounding noise on that scale)."""
import numpy as np
import pytest

from oracle import einsum_oracle as eo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from contract_gb300 import api, build, pycontract
    build.build()
    pycontract.init(0)
    return api


def projectors():
    g, e = eo.GAMMA, np.eye(4)
    k = np.arange(16.0).reshape(4, 4)
    dense = np.cos(1 + 1.7 * k) + 1j * np.sin(0.3 + 0.61 * k * k)
    rank2 = np.outer(dense[0], dense[1]) + np.outer(dense[2], dense[3])
    return {"one term": [1j * g[7]], "one term, two projectors": [g[8], -2 * g[8]],
            "two terms": [(e + g[8]) / 2], "two terms, rank 4": [e + 0.5 * g[9]],
            "two projectors": [(e + g[8]) / 2, (e - g[8]) / 2], "imaginary terms": [e + 1j * g[3], g[3] - 2 * e],
            "rank 1": [(e + g[8]) @ (e - 1j * g[3]) / 4], "rank 2": [rank2], "dense": [dense],
            "dense, two projectors": [dense, dense.T + e], "zero": [np.zeros((4, 4))]}


def check(api, c_oracle, latt, ws, gij, gkl, same, c64, seed=1):
    import torch
    ps = [eo.make_propagator(latt, 40 * seed + s, 0.2) for s in range(3)]
    if same:
        ps[1] = ps[0]
    ws = np.ascontiguousarray(np.asarray(ws, np.complex128).reshape(-1, 16))
    site = np.array([[c_oracle.baryon_general_two_point(*ps, t, gij, gkl, w) for w in ws] for t in range(6)])
    ref = eo.timeslice_sum(site, latt)
    dev = [torch.from_numpy(p).cuda().to(torch.complex64 if c64 else torch.complex128) for p in ps]
    if same:
        dev[1] = dev[0]
    got = api.baryon_all_types(*dev, gij, gkl, ws, latt=latt).cpu().numpy()
    got_site = api.baryon_all_types(*dev, gij, gkl, ws).cpu().numpy()
    spread = np.sqrt(eo.timeslice_sum(np.abs(site) ** 2, latt).real).max()
    for a, b in ((got, ref), (got_site, site)):
        assert np.isfinite(a).all()
        if c64:
            assert np.abs(a - b).max() <= 1e-6 * max(spread, np.abs(b).max())
        else:
            assert np.abs(a - b).max() <= 1e-12 * max(spread, np.abs(b).max())


@pytest.mark.parametrize("c64", [False, True])
@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("kind", list(projectors()))
def test_open_slot(api, c_oracle, kind, same, c64):
    for k, latt in enumerate([(2, 1, 1, 3), (2, 3, 3, 5), (6, 5, 3, 4)]):
        check(api, c_oracle, latt, projectors()[kind], 5, 10, same, c64, k + 1)


@pytest.mark.parametrize("same", [False, True])
def test_every_gamma_pair(api, c_oracle, same):
    e, g4 = np.eye(4), eo.GAMMA[8]
    for gij in range(16):
        for gkl in range(16):
            check(api, c_oracle, (2, 1, 3, 2), [(e + g4) / 2, (e - g4) / 2], gij, gkl, same, False)


def test_large_volume_matches_two_halves(api):
    """More tiles than the grid has warps: the timeslices of a lattice equal those of its two halves in time."""
    import torch
    latt = (12, 11, 10, 12)
    half = 12 * 11 * 10 // 2
    ps = [torch.from_numpy(eo.make_propagator(latt, 90 + s, 0.1)).cuda().to(torch.complex64) for s in range(3)]
    pp = api.projector_plus_minus()
    whole = api.baryon_all_types(*ps, 5, 5, pp, latt=latt).cpu().numpy()
    for t0 in (0, 6):
        cut = [p.view(2, 12, half, 4, 4, 3, 3)[:, t0:t0 + 6].reshape(-1, 4, 4, 3, 3).contiguous() for p in ps]
        part = api.baryon_all_types(*cut, 5, 5, pp, latt=latt[:3] + (6,)).cpu().numpy()
        assert np.abs(part - whole[:, :, t0:t0 + 6]).max() <= 1e-12 * np.abs(whole).max()
