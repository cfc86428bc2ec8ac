"""Per-timeslice sums against the sums of the same call's per-site results, over the
lattices where the cut into chunks changes: one tile a chunk, levelled rounds of a few
tiles with a short last one, plain chunks of more; fewer chunks than CTAs, than warps, and
several rounds of them.

One value per site (loop, triangle and meson forms): both calls form the same site values to
the bit, and a chunk sums FP32 values as a high and a low word, so only the FP64 sums
differ: 1e-12 of the sum of the sizes.  The all-types pass combines its terms after the
sum, per site before it, in FP32: 12 terms of 2^-24, 1e-6 of the sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LATTS = [(2, 2, 2, 4), (4, 4, 4, 8), (6, 5, 6, 12), (8, 8, 8, 16), (10, 9, 11, 20), (12, 12, 12, 24), (16, 15, 16, 32),
         (18, 17, 20, 33)]


@pytest.fixture(scope="module")
def api():
    from contract_gb300 import api, build, pycontract
    build.build()
    pycontract.init(0)
    return api


def sums(site, latt):
    """[.., V] to [.., Lt] and the sums of the sizes."""
    s = site.reshape(site.shape[:-1] + (2, latt[3], -1))
    return s.sum((-1, -3)), s.abs().sum((-1, -3))


@pytest.mark.parametrize("latt", LATTS)
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_sums(api, latt, dtype):
    import torch
    from contract_gb300 import pycontract as pc
    v = int(np.prod(latt))
    if dtype == "complex128" and v > 50000:
        pytest.skip("the plain rule holds in complex128")
    g = torch.Generator(device="cuda")
    g.manual_seed(v)
    p = [torch.view_as_complex(torch.randn((v, 4, 4, 3, 3, 2), generator=g, device="cuda")).to(getattr(torch, dtype))
         for _ in range(3)]
    pp = api.projector_plus_minus()
    rng = np.random.default_rng(1)
    wd = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    r1 = np.outer([1, 0.5, -2, 0.25j], [3, 1, 0.75j, 5]).astype(complex)
    pairs = [("meson", api.meson_timeslice(p[0], p[1], latt, 15, 5), pc.mesonTwoPoint(p[0], p[1], 15, 5), 1e-12)]
    for source, f in ((True, pc.mesonAllSourceTwoPoint), (False, pc.mesonAllSinkTwoPoint)):
        site = torch.stack([x.reshape(v) for x in f(p[0], p[1], 5)])
        pairs.append(("all partners", api.meson_all_timeslice(p[0], p[1], latt, 5, source=source), site, 1e-12))
    for name, t, kw in (("loop", 0, dict(gamma_mn=8)), ("gamma", 3, dict(gamma_mn=8)), ("dense", 3, dict(project_mn=wd)),
                        ("rank 2", 3, dict(project_mn=pp[0])), ("rank 1", 5, dict(project_mn=r1))):
        pairs.append((name, api.baryon(*p, t, 5, 5, latt=latt, **kw), api.baryon(*p, t, 5, 5, **kw), 1e-12))
    for same in (False, True):
        q = [p[0], p[0] if same else p[1], p[2]]
        pairs.append(("all types", api.baryon_all_types(*q, 5, 5, pp, latt=latt), api.baryon_all_types(*q, 5, 5, pp), 1e-6))
    for name, got, site, tol in pairs:
        site = site.reshape(got.shape[:-1] + (v,))
        ref, size = sums(site, latt)
        err = ((got - ref).abs() / size.amax()).max().item() if name == "all types" else ((got - ref).abs() / size).max().item()
        assert err <= tol, (name, latt, err)
