"""The row kernel of the mixed meson momentum projection where it can go wrong:
fewer rows than warps, planes that begin inside a batch of rows, one site pair a
row, every number of X groups with and without nx = 0, one (nx, ny) pair and
the most, a batch of uneven lattices, two fields and one.

Against the FP64 oracle, relative to max(|C|, sigma, L1), L1 the size of the
products that the FP32 sums are made of (oracle.einsum_oracle.meson_product_l1):
at most a few hundred FP32 roundings of 6e-8 that add up like their square root,
1e-6 as for the other mixed projections."""
import ctypes

import numpy as np
import pytest

from oracle import einsum_oracle as eo

pytestmark = pytest.mark.gpu
TOL = 1e-6
MOMENTA = {
    "zero": [(0, 0, 0)],
    "no zero": [(1, 0, 0), (-1, 1, 0), (1, 1, 1)],
    "two groups, no zero": [(1, 0, 0), (2, 1, 0), (-2, 0, 1)],
    "three groups, no zero": [(1, 0, 0), (2, 1, 0), (-3, 0, 1), (3, -1, 0)],
    "unpaired": [(0, 0, 0), (1, 0, 0), (0, 2, 1)],
    "27": list(map(tuple, eo.momentum_list(1))),
    "125": list(map(tuple, eo.momentum_list(2))),
    "one nx, 25 ny": [(0, n, 0) for n in range(-12, 13)],
}


@pytest.fixture(scope="module")
def lib():
    from contract_gb300 import _lib, build, pycontract
    build.build()
    pycontract.init(0)
    lib = _lib.lib()
    lib.contract_set_error_mode(1)
    return lib


def fields(latt, seed, same):
    pi = eo.make_propagator(latt, seed, 0.2)
    return pi, (pi if same else eo.make_propagator(latt, seed + 1, 0.25))


def check(latt, pi, pj, moms, got):
    site = eo.meson_all_gamma(pi, pj).reshape(256, -1)
    ref = eo.momentum_project(site, latt, moms).transpose(1, 2, 0)
    sig = np.sqrt(eo.timeslice_sum(np.abs(site) ** 2, latt).real).T[None]
    scale = np.maximum(np.maximum(np.abs(ref), sig), eo.meson_product_l1(pi, pj, latt))
    assert np.isfinite(got).all()
    assert (np.abs(got - ref) / scale).max() < TOL, latt


def device(pi, pj, same):
    import torch
    a = torch.from_numpy(pi).cuda().to(torch.complex64)
    return a, (a if same else torch.from_numpy(pj).cuda().to(torch.complex64))


@pytest.mark.parametrize("same", [False, True])
@pytest.mark.parametrize("name", list(MOMENTA))
def test_momentum_lists(lib, name, same):
    import torch
    moms = np.ascontiguousarray(np.array(MOMENTA[name], dtype=np.int32))
    for latt in ((2, 3, 5, 3), (10, 5, 7, 4), (6, 26, 2, 2)):
        pi, pj = fields(latt, 11, same)
        a, b = device(pi, pj, same)
        out = torch.full((len(moms), latt[3], 256), float("nan"), dtype=torch.complex128, device="cuda")
        lib.contract_meson_all_gamma_momentum(out.data_ptr(), a.data_ptr(), b.data_ptr(), pi.shape[0],
                                              (ctypes.c_int * 4)(*latt),
                                              moms.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), len(moms), 1)
        got = out.cpu().numpy()
        assert lib.contract_last_error() == 0, lib.contract_last_error_message()
        check(latt, pi, pj, moms, got)


@pytest.mark.parametrize("same", [False, True])
def test_batch_of_uneven_rows(lib, same):
    import torch

    from test_batch_mixed_gpu import MesonItem
    latts = [(6, 5, 3, 4), (4, 13, 4, 3), (16, 3, 5, 2), (6, 5, 3, 4)]
    moms = np.ascontiguousarray(eo.momentum_list(1).astype(np.int32))
    arr, keep = (MesonItem * len(latts))(), []
    for k, latt in enumerate(latts):
        pi, pj = fields(latt, 60 + 2 * k, same)
        a, b = device(pi, pj, same)
        out = torch.full((len(moms), latt[3], 256), float("nan"), dtype=torch.complex128, device="cuda")
        arr[k] = MesonItem(a.data_ptr(), b.data_ptr(), out.data_ptr(), (ctypes.c_int * 4)(*latt))
        keep.append((latt, pi, pj, a, b, out))
    lib.contract_meson_all_gamma_momentum_batch(arr, len(latts), moms.ctypes.data_as(ctypes.POINTER(ctypes.c_int)),
                                                len(moms), 1)
    torch.cuda.synchronize()
    assert lib.contract_last_error() == 0, lib.contract_last_error_message()
    for latt, pi, pj, _, _, out in keep:
        check(latt, pi, pj, moms, out.cpu().numpy())
