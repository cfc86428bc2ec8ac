"""The contractions of a call (ring_kernel) and of the all-types pass (warp_kernel),
and the integer-pipe form that complex128 takes there (fixed.cuh), over inputs
that it takes and inputs that it must leave to the FP64 form: Gaussian fields, a
coherent part, colour rows and spin rows of different size, zero blocks and
sites, colour-diagonal blocks, very large, very small and denormal values,
NaN and infinity.

Tolerance: 2e-15 of the norm of a call's outputs.  The results are off by 1.5 to
3e-16 of that norm (measured against extended precision) in either form and the
oracle's own FP64 by as much; a dropped low word or a wrong scale is off by 1e-9
or more."""
import numpy as np
import pytest

from oracle import einsum_oracle as eo

pytestmark = pytest.mark.gpu
LATT = (4, 3, 3, 4)
V = int(np.prod(LATT))
TOL = 2e-15


def gauss(rng):
    return rng.standard_normal((V, 4, 4, 3, 3)) + 1j * rng.standard_normal((V, 4, 4, 3, 3))


def blocks(rng, kind):
    p = gauss(rng)
    if kind == "coherent":
        p = p + gauss(rng)[:1]
    elif kind == "colour rows":
        p = p * np.array([1, 1e-3, 1e-6])[:, None]
    elif kind == "colour columns":
        p = p * np.array([1e5, 1, 1e-9])[None, :]
    elif kind == "spin rows":
        p = p * np.array([1, 1e-2, 1, 1e-5])[None, :, None, None, None]
    elif kind == "uneven blocks":
        p = p * 2.0 ** rng.integers(-6, 7, (V, 4, 4, 1, 1))
    elif kind == "zeros":
        p[:, 1, 2] = 0
        p[:, 3] *= rng.random((V, 4, 1, 1)) < 0.5
        p[::5] = 0
    elif kind == "colour diagonal":
        p = p * np.eye(3)
    elif kind == "large":
        p = p * 1e95
    elif kind == "small":
        p = p * 1e-95
    elif kind == "mixed sites":
        p = p * 10.0 ** rng.integers(-60, 60, (V, 1, 1, 1, 1))
    elif kind == "denormal":
        p[:, 0, 0, 1, 1] = 3e-310
        p[3] = 4e-311 + 5e-312j
    elif kind == "powers of two":
        p = np.sign(p.real) * 2.0 ** rng.integers(-1, 2, p.shape) + 0j
    return p


KINDS = ["gauss", "coherent", "colour rows", "colour columns", "spin rows", "uneven blocks", "zeros", "colour diagonal",
         "large", "small", "mixed sites", "denormal", "powers of two"]


@pytest.fixture(scope="module")
def api():
    from contract_gb300 import api, build, pycontract
    build.build()
    pycontract.init(0)
    return api


def norm(a):
    m = np.abs(a).max()
    return m * np.sqrt((np.abs(a / m) ** 2).sum()) if m > 0 else 0.0


def close(got, ref, kind):
    """Per site where sites differ in scale, else over the call."""
    got, ref = np.asarray(got), np.asarray(ref)
    assert np.isfinite(got).all(), kind
    if kind == "mixed sites":
        scale = np.abs(ref).max(axis=tuple(range(ref.ndim - 1)), keepdims=True)
        got, ref = got / scale, ref / scale
    assert norm(got - ref) <= TOL * norm(ref), (kind, norm(got - ref) / norm(ref))


def fields(kind, same=False):
    import torch
    rng = np.random.default_rng(KINDS.index(kind) + 1)
    ps = [np.ascontiguousarray(blocks(rng, kind)) for _ in range(3)]
    if same:
        ps[1] = ps[0]
    dev = [torch.from_numpy(p).cuda() for p in ps]
    if same:
        dev[1] = dev[0]
    return ps, dev


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_all_types(api, c_oracle, kind, same):
    ps, dev = fields(kind, same)
    pp = api.projector_plus_minus()
    ref = np.array([[c_oracle.baryon_general_two_point(*ps, t, 5, 5, w) for w in pp] for t in range(6)])
    got = api.baryon_all_types(*dev, 5, 5, pp).cpu().numpy()
    if same:  # types that vanish identically are rounding noise on the scale of the others
        ref, got = ref.reshape(12, V), got.reshape(12, V)
    close(got, ref, kind)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite(api, c_oracle, bad):
    """A value that is not finite spoils its own site and no other."""
    ps, dev = fields("gauss")
    pp = api.projector_plus_minus()
    ref = np.array([[c_oracle.baryon_general_two_point(*ps, t, 5, 5, w) for w in pp] for t in range(6)])
    for field in range(3):
        ps2 = [p.copy() for p in ps]
        ps2[field][7, 1, 2, 0, 1] = bad
        dev[field].copy_(__import__("torch").from_numpy(ps2[field]))
        got = api.baryon_all_types(*dev, 5, 5, pp).cpu().numpy()
        dev[field].copy_(__import__("torch").from_numpy(ps[field]))
        assert not np.isfinite(got[:, :, 7]).all()
        keep = np.arange(V) != 7
        close(got[:, :, keep], ref[:, :, keep], "gauss")


def per_call(api, ps, dev, form):
    """(result, oracle) of one call of a per-site form."""
    from contract_gb300 import pycontract as pc
    rng = np.random.default_rng(11)
    wd = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    pp = api.projector_plus_minus()
    if form in ("source", "sink"):
        got = pc._meson_all(dev[0], dev[1], 6, form == "source")
        ref = (eo.meson_all_source if form == "source" else eo.meson_all_sink)(ps[0], ps[1], 6)
        return np.array([g.cpu().numpy() for g in got]).reshape(16, V), np.asarray(ref)
    if form == "meson":
        return pc.mesonTwoPoint(dev[0], dev[1], 6, 13).cpu().numpy().reshape(V), eo.meson_two_point(ps[0], ps[1], 6, 13)
    if form == "gamma":
        return (api.baryon(*dev, 3, 6, 13, gamma_mn=9).cpu().numpy().reshape(V),
                eo.baryon_two_point(*ps, 3, 6, 13, 9))
    t, w = {"loop": (0, pp[1]), "dense": (4, wd), "rank 2": (5, pp[0]), "rank 1": (1, np.outer(wd[0], wd[1])),
            "rank 2, general": (4, np.outer(wd[0], wd[1]) + np.outer(wd[2], wd[3])),
            "rank 1, phases": (3, np.outer([1, 0, 1j, 0], [0, 1, 0, -1]))}[form]
    return api.baryon(*dev, t, 6, 13, project_mn=w).cpu().numpy().reshape(V), eo.baryon_general_two_point(*ps, t, 6, 13, w)


FORMS = ["loop", "gamma", "dense", "rank 1", "rank 2", "rank 2, general", "rank 1, phases", "meson", "source", "sink"]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("kind", KINDS)
def test_per_call(api, form, kind):
    ps, dev = fields(kind)
    got, ref = per_call(api, ps, dev, form)
    if kind == "mixed sites":  # in units of each site's own values
        unit = np.prod([np.abs(p).max(axis=(1, 2, 3, 4)) for p in ps[:2 if form in ("meson", "source", "sink") else 3]], axis=0)
        got, ref, kind = got / unit, ref / unit, "gauss"
    close(got, ref, kind)


@pytest.mark.parametrize("form", FORMS)
def test_per_call_not_finite(api, form):
    ps, dev = fields("gauss")
    ref = per_call(api, ps, dev, form)[1]
    keep = np.arange(V) != 7
    for field in range(2 if form in ("meson", "source", "sink") else 3):
        for bad in (np.nan, np.inf):
            p = ps[field].copy()
            p[7] = bad
            d = list(dev)
            d[field] = __import__("torch").from_numpy(p).cuda()
            got = per_call(api, ps, d, form)[0]
            assert not np.isfinite(got[..., 7]).any()
            close(got[..., keep], ref[..., keep], "gauss")


def field_call(ps, dev, form):
    """(result, oracle) of a propagator-shaped call."""
    from contract_gb300 import pycontract as pc
    if form == "diquark":
        return pc.baryonDiquark(dev[0], dev[1], 6, 13).cpu().numpy().reshape(-1, 144), eo.baryon_diquark(ps[0], ps[1], 6, 13)
    t, slot = form
    d = [x.clone() for x in dev]
    pc.baryonSequentialTwoPoint(*d, t, slot, 6, 13, 9)
    for k in range(3):
        assert k == slot or (d[k] == dev[k]).all() or not np.isfinite(ps[k]).all()
    return d[slot].cpu().numpy().reshape(-1, 144), eo.baryon_sequential(*ps, t, slot, 6, 13, 9)


FIELD_FORMS = ["diquark"] + [(t, slot) for t in (0, 2, 1, 5) for slot in range(3)]


@pytest.mark.parametrize("form", FIELD_FORMS)
@pytest.mark.parametrize("kind", KINDS)
def test_fields(api, form, kind):
    ps, dev = fields(kind)
    got, ref = field_call(ps, dev, form)
    ref = np.asarray(ref).reshape(-1, 144)
    if kind == "mixed sites":  # in units of each site's own values
        used = [p for k, p in enumerate(ps) if (k < 2 if form == "diquark" else k != form[1])]
        unit = np.prod([np.abs(p).max(axis=(1, 2, 3, 4)) for p in used], axis=0)[:, None]
        got, ref, kind = got / unit, ref / unit, "gauss"
    close(got, ref, kind)


@pytest.mark.parametrize("form", FIELD_FORMS)
def test_fields_not_finite(api, form):
    ps, dev = fields("gauss")
    ref = np.asarray(field_call(ps, dev, form)[1]).reshape(-1, 144)
    keep = np.arange(V) != 7
    for field in range(2 if form == "diquark" else 3):
        if form != "diquark" and field == form[1]:
            continue
        p = ps[field].copy()
        p[7] = np.nan
        d = list(dev)
        d[field] = __import__("torch").from_numpy(p).cuda()
        got = field_call([p if k == field else q for k, q in enumerate(ps)], d, form)[0]
        bad = ~np.isfinite(got[7])
        assert bad.all() or (form in ((0, 2), (2, 2)) and bad.sum() == 36)  # four blocks, the others are zero
        close(got[keep], ref[keep], "gauss")


@pytest.mark.parametrize("volume", [1, 2, 3, 31, 1217])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_field_edges(api, volume, dtype):
    """One live site in a warp, fewer tiles than warps, stages used once and again."""
    import torch
    rng = np.random.default_rng(volume)
    tol = 2e-15 if dtype == "complex128" else 1e-6
    ps = [(rng.standard_normal((volume, 4, 4, 3, 3)) + 1j * rng.standard_normal((volume, 4, 4, 3, 3))).astype(dtype)
          for _ in range(3)]
    dev = [torch.from_numpy(p).cuda() for p in ps]
    ps = [p.astype(np.complex128) for p in ps]
    for form in FIELD_FORMS:
        got, ref = field_call(ps, dev, form)
        ref = np.asarray(ref).reshape(-1, 144)
        assert norm(got - ref) <= tol * norm(ref), form


@pytest.mark.parametrize("latt", [(2, 1, 1, 1), (2, 1, 1, 3), (6, 3, 1, 5), (10, 3, 3, 2)])
@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
def test_per_call_edges(api, latt, dtype):
    """Half-timeslices of 1, 9 and 45 sites: warps with one live site, a last tile
    part full, fewer tiles than warps."""
    import torch
    from contract_gb300 import pycontract as pc
    rng = np.random.default_rng(sum(latt))
    n, tol = int(np.prod(latt)), 2e-15 if dtype == "complex128" else 2e-6
    ps = [(rng.standard_normal((n, 4, 4, 3, 3)) + 1j * rng.standard_normal((n, 4, 4, 3, 3))).astype(dtype) for _ in range(3)]
    dev = [torch.from_numpy(p).cuda() for p in ps]
    # the reference in extended precision: a sum of two sites can cancel, and the
    # oracle's own FP64 rounding is then as large as the bound
    ps = [p.astype(np.clongdouble) for p in ps]
    pp = api.projector_plus_minus()
    wd = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    calls = [(t, w) for t, w in ((0, pp[0]), (1, pp[1]), (4, wd), (3, np.outer(wd[0], wd[1])))]
    pairs = [(api.baryon(*dev, t, 5, 7, project_mn=w, latt=l), eo.baryon_general_two_point(*ps, t, 5, 7, w), l)
             for t, w in calls for l in (None, latt)]
    pairs += [(api.baryon(*dev, 1, 5, 7, gamma_mn=8, latt=l), eo.baryon_two_point(*ps, 1, 5, 7, 8), l) for l in (None, latt)]
    pairs += [(api.meson_timeslice(dev[0], dev[1], latt, 15, 5), eo.meson_two_point(ps[0], ps[1], 15, 5), latt)]
    for src in (True, False):
        ref = (eo.meson_all_source if src else eo.meson_all_sink)(ps[0], ps[1], 5)
        pairs += [(api.meson_all_timeslice(dev[0], dev[1], latt, 5, source=src), ref, latt)]
    for got, ref, l in pairs:
        got, ref = got.cpu().numpy(), np.asarray(ref)
        if l is not None:
            ref = np.array([eo.timeslice_sum(r, latt) for r in ref.reshape(-1, n)])
        assert norm(got.ravel() - ref.ravel()) <= tol * norm(ref), (latt, l)
