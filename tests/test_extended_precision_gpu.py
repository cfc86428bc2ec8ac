"""Complex128 results against extended precision, in the norm: the momentum projection,
all partners of one meson Gamma, and every baryon type.

A reference in plain FP64 is itself off by 1.8e-16 (mesons) to 3.8e-16 (projections) of
the norm, as much as what is measured, so it cannot tell which of two forms is nearer.
Bounds: what the FP64 kernels left on these inputs (18 x 15 x 20 x 2, a part common to
all sites plus noise), 3.2e-16 for the projection, 1.75e-16 for mesons, 2.3e-16 for
baryons; the integer forms are not to be further off."""
import ctypes

import numpy as np
import pytest

from oracle import einsum_oracle as eo

pytestmark = pytest.mark.gpu
LATT = (18, 15, 20, 2)
L = np.clongdouble


@pytest.fixture(scope="module")
def api():
    from contract_gb300 import api, build, pycontract
    build.build()
    pycontract.init(0)
    return api


def propagators(latt, n, seed):
    """exp(-m |t|) (W + noise(x)) / sqrt 2, W the same at every site."""
    rng = np.random.default_rng(seed)
    v, t = int(np.prod(latt)), eo.eo_coords(latt)[3]
    out = []
    for k in range(n):
        p = rng.standard_normal((v, 288)) + rng.standard_normal(288)
        p *= 0.5 ** 0.5 * np.exp(-(0.2 + 0.05 * k) * np.minimum(t, latt[3] - t))[:, None]
        out.append(np.ascontiguousarray(p).view(complex).reshape(v, 4, 4, 3, 3))
    return out


def off(got, ref):
    return float(np.sqrt((np.abs(got.astype(L) - ref) ** 2).sum() / (np.abs(ref) ** 2).sum()))


def wave(n, length):
    pi = np.longdouble("3.14159265358979323846264338327950288")
    angle = 2 * pi * ((n[:, None] * np.arange(length)) % length).astype(np.longdouble) / length
    return np.cos(angle) + 1j * np.sin(angle)


@pytest.mark.parametrize("seed", [1, 2])
def test_projection(api, seed):
    import torch
    from contract_gb300 import _lib
    lx, ly, lz, lt = LATT
    moms = np.ascontiguousarray(eo.momentum_list(2), dtype=np.int32)
    a, b = propagators(LATT, 2, seed)
    dev = [torch.from_numpy(p).cuda() for p in (a, b)]
    out = torch.empty((len(moms), lt, 256), dtype=torch.complex128, device="cuda")
    _lib.lib().contract_meson_all_gamma_momentum(out.data_ptr(), dev[0].data_ptr(), dev[1].data_ptr(), len(a),
                                                 (ctypes.c_int * 4)(*LATT),
                                                 moms.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), len(moms), 0)
    got = out.cpu().numpy()
    a, b = (p.reshape(2, lt, lz, ly, lx // 2, 16, 9) for p in (a, b))
    n, ref = np.arange(-2, 3), np.empty((len(moms), lt, 256), L)
    g = np.array([eo.G5 @ m for m in eo.GAMMA]).astype(L)
    for t in range(lt):
        s = np.empty((5, lz, ly, 256), L)
        for z in range(lz):
            rows = np.empty((ly, lx, 256), L)
            for y in range(ly):
                for par in range(2):
                    prod = np.einsum("hkc,hlc->hkl", a[par, t, z, y].astype(L), b[par, t, z, y].conj().astype(L))
                    rows[y, 2 * np.arange(lx // 2) + ((par + t + z + y) & 1)] = prod.reshape(lx // 2, 256)
            s[:, z] = np.einsum("nx,yxg->nyg", wave(n, lx), rows)
        s = np.einsum("lz,mnzg->lmng", wave(n, lz), np.einsum("my,nzyg->mnzg", wave(n, ly), s))
        ref[:, t] = np.einsum("Aji,Bkl,pikjl->pAB", g, g, s.reshape(-1, 4, 4, 4, 4), optimize=True).reshape(-1, 256)
    assert off(got, ref) <= 3.2e-16, off(got, ref)


@pytest.mark.parametrize("source", [True, False])
def test_mesons(api, source):
    import torch
    from contract_gb300 import pycontract as pc
    a, b = (p[:2000] for p in propagators(LATT, 2, 3))
    got = pc._meson_all(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), 5, source)
    got = np.array([x.cpu().numpy().ravel() for x in got])
    ref = (eo.meson_all_source if source else eo.meson_all_sink)(a.astype(L), b.astype(L), 5)
    assert off(got, ref) <= 1.75e-16, off(got, ref)


def test_baryons(api):
    import torch
    ps = [p[:400] for p in propagators(LATT, 3, 4)]
    dev = [torch.from_numpy(p).cuda() for p in ps]
    pp = api.projector_plus_minus()
    got = api.baryon_all_types(*dev, 5, 5, pp).cpu().numpy()
    ps = [p.astype(L) for p in ps]
    ref = np.array([[eo.baryon_general_two_point(*ps, t, 5, 5, w) for w in pp] for t in range(6)])
    one = np.array([[api.baryon(*dev, t, 5, 5, project_mn=w).cpu().numpy().ravel() for w in pp] for t in range(6)])
    assert off(got, ref) <= 2.3e-16 and off(one, ref) <= 2.45e-16, (off(got, ref), off(one, ref))
