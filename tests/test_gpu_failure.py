"""Failure detection without a GPU fault: a bounded device wait that runs out
(a counter nothing increments) reports through the status word within its
limit, and the device keeps working afterwards."""
import ctypes
import time

import pytest

from conftest import golden_graph

pytestmark = pytest.mark.gpu


def test_bounded_wait_times_out_and_reports(cuda_device):
    from qtensor_b200 import _lib
    lib = _lib.lib()
    _lib.check(lib.qtb_init(0))
    status = ctypes.c_int32(-1)
    t0 = time.perf_counter()
    _lib.check(lib.qtb_selftest_wait_timeout(1 << 14, ctypes.byref(status)))
    assert time.perf_counter() - t0 < 30
    assert status.value == _lib.STATUS_WAIT_TIMEOUT
    # the context is intact: a normal contraction still matches the reference
    from qtensor_b200.engine import QAOAEnergyEngine
    G, w = golden_graph('cfg2')
    eng = QAOAEnergyEngine()
    E = eng.energy_expectation(G, w['gamma'], w['beta'])
    assert abs(E - w['energy']) <= 1e-5 * abs(w['energy'])
    assert eng.compile(G, 3, w['gamma'], w['beta']).plan.device_status() == 0


def test_selftest_rejects_bad_arguments(cuda_device):
    from qtensor_b200 import _lib
    status = ctypes.c_int32(0)
    assert _lib.lib().qtb_selftest_wait_timeout(0, ctypes.byref(status)) == _lib.QTB_ERR_ARG
    assert _lib.lib().qtb_selftest_wait_timeout(16, None) == _lib.QTB_ERR_ARG


@pytest.mark.parametrize('K,F,M,N,parts', [(544, 1, 100, 60, 8), (894, 4, 1309, 574, 2)])
def test_contract_timeout_leaves_the_tile_unwritten(cuda_device, K, F, M, N, parts):
    """K of one tile is split over `parts` CTAs; where one of them gives up,
    its part is missing from the tile's sums, so the others store nothing
    either (every row of the output keeps what it held)."""
    import numpy as np
    import torch
    from qtensor_b200 import _lib, tcontract
    lib = _lib.lib()
    gen = torch.Generator(device=cuda_device).manual_seed(K)
    a = torch.randn((K, F, M), dtype=torch.complex64, device=cuda_device, generator=gen)
    b = torch.randn((K, F, N), dtype=torch.complex64, device=cuda_device, generator=gen)
    c = torch.full((F, M, N), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)
    scratch = torch.empty(tcontract.contract_sum_scratch_bytes(K, F, M, N, 'tensor'), dtype=torch.uint8,
                          device=cuda_device)
    stream = torch.cuda.current_stream().cuda_stream

    def run(part):
        return lib.qtb_selftest_contract_timeout(a.data_ptr(), b.data_ptr(), c.data_ptr(), K, F, M, N,
                                                 scratch.data_ptr(), scratch.numel(), 1 << 14, part, stream)

    assert run(parts) == _lib.QTB_ERR_ARG
    for part in (0, parts - 1):
        _lib.check(run(part))
        torch.cuda.synchronize()
        assert int(scratch[:4].view(torch.int32).item()) == 2
        assert bool(torch.isnan(c.real).all())
    # the device and the scratch are as good as before
    tcontract.mkl_contract_sum(a, b, c, mode='tensor', scratch=scratch)
    ref = a.to(torch.complex128).permute(1, 2, 0) @ b.to(torch.complex128).permute(1, 0, 2)
    assert int(scratch[:4].view(torch.int32).item()) == 0
    assert (c - ref).abs().max().item() <= 1e-5 * ref.abs().max().item()
