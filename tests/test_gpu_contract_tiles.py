"""Edges of the tensor-core contract-sum's 128 x 64 tiles (the wider ones are in
test_gpu_contract_wide_tiles.py): one and more column tiles, rows past the
last tile, K split over 1 to 8 CTAs with even and uneven parts, odd N (8-byte
stores) and a C that is only 8-byte aligned.  The bar is
the repository's for this path: 1e-5 of the largest output magnitude."""
import numpy as np
import pytest
import torch

from qtensor_b200 import tcontract

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize('K,F,M,N', [
    (32, 1, 1, 1), (33, 1, 128, 64), (64, 1, 129, 65), (160, 2, 127, 128), (257, 1, 64, 129),
    (300, 40, 130, 130),        # more tiles than SMs
    (1000, 1, 100, 96),         # two tiles, K in eight parts
    (544, 2, 300, 250),
])
@pytest.mark.parametrize('shift', [0, 1])
def test_contract_tile_edges(cuda_device, K, F, M, N, shift):
    rng = np.random.default_rng(K + M + N)
    A = ((rng.standard_normal((K, F, M)) + 1j * rng.standard_normal((K, F, M))) / np.sqrt(2)).astype(np.complex64)
    B = ((rng.standard_normal((K, F, N)) + 1j * rng.standard_normal((K, F, N))) / np.sqrt(2)).astype(np.complex64)
    a, b = torch.from_numpy(A).to(cuda_device), torch.from_numpy(B).to(cuda_device)
    buf = torch.full((F * M * N + 2 * shift,), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)
    c = buf[shift:shift + F * M * N].view(F, M, N)
    scratch = torch.full((tcontract.contract_sum_scratch_bytes(K, F, M, N, 'tensor'),), 255, dtype=torch.uint8,
                         device=cuda_device)
    for _ in range(2):
        tcontract.mkl_contract_sum(a, b, c, mode='tensor', scratch=scratch)
    torch.cuda.synchronize()
    assert int(scratch[:4].view(torch.int32).item()) == 0
    ref = np.matmul(A.astype(np.complex128).transpose(1, 2, 0), B.astype(np.complex128).transpose(1, 0, 2))
    assert np.max(np.abs(c.cpu().numpy() - ref)) <= TOL * np.max(np.abs(ref))
    if shift:                                   # nothing outside the output is written
        assert bool(torch.isnan(buf[:shift].real).all()) and bool(torch.isnan(buf[shift + F * M * N:].real).all())
