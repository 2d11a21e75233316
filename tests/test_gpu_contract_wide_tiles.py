"""The contract-sum's 128 x 128 tiles, which it takes where tiles of half the
width need more than one round of CTAs: K in 1 to 8 parts (even and uneven),
rows and columns past the last tile, odd N (8-byte stores) and a C that is
only 8-byte aligned.  The kernel's name and grid, read from a captured call,
say which tile and how many parts a shape took.  The bar is the repository's
for this path: 1e-5 of the largest output magnitude."""
import numpy as np
import pytest
import torch

from graph_nodes import captured_kernels
from qtensor_b200 import tcontract

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize('K,F,M,N,parts', [
    (32, 4, 193, 1796, 1), (1024, 2, 1024, 1023, 1), (894, 4, 1309, 574, 2), (3075, 4, 741, 73, 4),
    (3606, 6, 853, 74, 8),
])
@pytest.mark.parametrize('shift', [0, 1])
def test_wide_tile_edges(cuda_device, K, F, M, N, parts, shift):
    gen = torch.Generator(device=cuda_device).manual_seed(K + M + N)
    a = torch.randn((K, F, M), dtype=torch.complex64, device=cuda_device, generator=gen)
    b = torch.randn((K, F, N), dtype=torch.complex64, device=cuda_device, generator=gen)
    buf = torch.full((F * M * N + 2 * shift,), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)
    c = buf[shift:shift + F * M * N].view(F, M, N)
    scratch = torch.full((tcontract.contract_sum_scratch_bytes(K, F, M, N, 'tensor'),), 255, dtype=torch.uint8,
                         device=cuda_device)
    kernels = captured_kernels(lambda stream: tcontract.mkl_contract_sum(a, b, c, mode='tensor', scratch=scratch))
    product = [k for k in kernels if 'qtb_tc_contract_kernel' in k.name]
    assert len(product) == 1 and 'ILj128E' in product[0].name
    assert product[0].grid == -(-N // 128) * parts
    assert int(scratch[:4].view(torch.int32).item()) == 0
    ref = a.to(torch.complex128).permute(1, 2, 0) @ b.to(torch.complex128).permute(1, 0, 2)
    assert (c - ref).abs().max().item() <= TOL * ref.abs().max().item()
    if shift:                                   # nothing outside the output is written
        assert bool(torch.isnan(buf[:shift].real).all()) and bool(torch.isnan(buf[shift + F * M * N:].real).all())
