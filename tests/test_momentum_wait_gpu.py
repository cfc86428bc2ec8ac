"""The complex128 momentum projection's bounded waits, made to run out: the copies of
one row's first pair of sites are withheld (contract_test_withhold_chunk), so the pair
warp that needs them gives up, the warps that wait for it follow, the call ends within
a few of the short limits set here, contract_check_device() reports the timeout and the
next call gives the usual bits.  Nothing faults, traps or spins without a limit."""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CONTRACT_ERROR_DEVICE_TIMEOUT = 3
LATT = (8, 8, 8, 8)
LIMIT_NS = 50_000_000  # 50 ms per wait
MOMS = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 1), (2, -1, 1), (3, 0, 0)]


@pytest.mark.parametrize("nmom", [1, 5, 6])  # one, three and four X groups: 4 or 8 warps for the X sums
def test_wait_runs_out_and_context_recovers(nmom):
    import torch

    from contract_gb300 import _lib, build
    from contract_gb300.lattice import synthetic_propagator
    build.build()
    lib = _lib.lib()
    lib.contract_set_error_mode(1)
    lib.init(0)
    a, b = (synthetic_propagator(LATT, s, 0.3, device="cuda:0") for s in (71, 72))
    moms = (ctypes.c_int * (3 * nmom))(*[n for m in MOMS[:nmom] for n in m])

    def call():
        out = torch.zeros((nmom, LATT[3], 256), dtype=torch.complex128, device="cuda:0")
        lib.contract_meson_all_gamma_momentum(out.data_ptr(), a.data_ptr(), b.data_ptr(), int(np.prod(LATT)),
                                              (ctypes.c_int * 4)(*LATT), moms, nmom, 0)
        return out

    ref = call()
    assert lib.contract_check_device() == 0
    lib.contract_set_wait_limit(LIMIT_NS)
    lib.contract_test_withhold_chunk(3)
    try:
        t0 = time.monotonic()
        call()
        rc = lib.contract_check_device()
        elapsed = time.monotonic() - t0
    finally:
        lib.contract_test_withhold_chunk(-1)
        lib.contract_set_wait_limit(0)
        lib.contract_clear_error()
    assert rc == CONTRACT_ERROR_DEVICE_TIMEOUT
    assert elapsed < 20.0
    assert torch.equal(call(), ref) and lib.contract_check_device() == 0
