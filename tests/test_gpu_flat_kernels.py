"""Edges of the CUDA-core products and of the large-bucket kernel: rows per
thread and pairs of columns with remainders, outputs too few for either,
pointers that are only 8-byte aligned, buckets around the size where chunks
take over and with operands that lack the low variables.

Tolerances: a complex64 product of k factors has a relative error of at most
about 3 k eps (eps = 2^-24), and a sum of K products at most (K + 4) eps of
the sum of their magnitudes; inputs have unit variance, so magnitudes stay
below 8 per factor over the sizes here."""
import ctypes

import numpy as np
import pytest
import torch

from qtensor_b200 import _lib, tcontract

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def _rand(rng, n, shift, device):
    """complex64 values on the device starting `shift` elements into a buffer."""
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    buf = torch.empty(n + shift, dtype=torch.complex64, device=device)
    buf[shift:] = torch.from_numpy(x).to(device)
    return x, buf[shift:]


@pytest.mark.parametrize('n,m,k', [(1, 1, 1), (3, 5, 1), (1, 1, 4097), (7, 1023, 130), (5, 1021, 129),
                                   (600, 1, 1100), (2, 3, 110001)])
@pytest.mark.parametrize('shift', [0, 1])
def test_outer_edges(cuda_device, n, m, k, shift):
    rng = np.random.default_rng(n + m + k)
    A, a = _rand(rng, n * m, shift, cuda_device)
    B, b = _rand(rng, n * k, shift, cuda_device)
    c = torch.full((n * m * k + shift,), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)[shift:]
    tcontract.mkl_contract_complex(a.view(n, m), b.view(n, k), c.view(n, m, k))
    ref = A.astype(np.complex128).reshape(n, m, 1) * B.astype(np.complex128).reshape(n, 1, k)
    got = c.cpu().numpy().reshape(n, m, k)
    assert np.max(np.abs(got - ref)) <= 4 * EPS * np.max(np.abs(ref))


@pytest.mark.parametrize('K,F,M,N', [(1, 1, 1, 1), (2, 3, 1023, 130), (3, 7, 301, 257), (17, 1, 9, 30001),
                                     (2, 640, 1, 1000), (33, 2, 63, 5)])
@pytest.mark.parametrize('shift', [0, 1])
def test_simt_sum_edges(cuda_device, K, F, M, N, shift):
    rng = np.random.default_rng(K + F + M + N)
    A, a = _rand(rng, K * F * M, shift, cuda_device)
    B, b = _rand(rng, K * F * N, shift, cuda_device)
    c = torch.full((F * M * N + shift,), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)[shift:]
    scratch = torch.full((64,), 255, dtype=torch.uint8, device=cuda_device)
    tcontract.mkl_contract_sum(a.view(K, F, M), b.view(K, F, N), c.view(F, M, N), mode='simt', scratch=scratch)
    A, B = A.astype(np.complex128).reshape(K, F, M), B.astype(np.complex128).reshape(K, F, N)
    ref = np.einsum('kfm,kfn->fmn', A, B)
    bound = np.einsum('kfm,kfn->fmn', np.abs(A), np.abs(B))
    got = c.cpu().numpy().reshape(F, M, N)
    assert int(scratch[:4].view(torch.int32).item()) == 0
    assert np.all(np.abs(got - ref) <= 2 * (K + 4) * EPS * bound + 1e-30)


@pytest.mark.parametrize('N', [4096, 4098])
@pytest.mark.parametrize('K', [1, 3])
def test_evict_first_line(cuda_device, K, N):
    # 3 x 1109 rows: just below and just above the size from which outputs
    # are stored evict-first, with a remainder of rows
    F, M = 3, 1109
    assert (F * M * 4096 * 8 < 104 << 20) and (F * M * 4098 * 8 >= 104 << 20)
    gen = torch.Generator(device=cuda_device).manual_seed(K * N)
    a = torch.randn((K, F, M), dtype=torch.complex64, device=cuda_device, generator=gen)
    b = torch.randn((K, F, N), dtype=torch.complex64, device=cuda_device, generator=gen)
    c = torch.full((F, M, N), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)
    if K == 1:
        tcontract.mkl_contract_complex(a[0], b[0], c)
    else:
        tcontract.mkl_contract_sum(a, b, c, mode='simt')
    for f in range(F):
        ref = a[:, f].to(torch.complex128).T @ b[:, f].to(torch.complex128)
        bound = a[:, f].abs().double().T @ b[:, f].abs().double()
        assert bool(((c[f] - ref).abs() <= 2 * (K + 4) * EPS * bound).all())


@pytest.mark.parametrize('u,sum_first', [(17, 1), (17, 0), (18, 1), (19, 0), (21, 1)])
@pytest.mark.parametrize('shift', [0, 1])
def test_large_bucket_edges(cuda_device, u, sum_first, shift):
    lib = _lib.lib()
    _lib.check(lib.qtb_init(cuda_device.index))
    rng = np.random.default_rng(u * 2 + sum_first)
    top = 1 << (u - 1)
    masks = [(1 << u) - 1, top | 0x3ff, top | (0x155 << 4), top | 0x200, 1, 0, top >> 1]
    host, ins = zip(*[_rand(rng, 1 << bin(x).count('1'), shift, cuda_device) for x in masks])
    w = u - sum_first
    out = torch.full(((1 << w) + shift,), complex(np.nan, 0), dtype=torch.complex64, device=cuda_device)[shift:]
    desc = _lib.BucketDesc()
    desc.n_inputs, desc.n_vars, desc.sum_first = len(masks), u, sum_first
    for t, x in enumerate(masks):
        desc.masks[t] = x
    ptrs = (ctypes.c_void_p * len(masks))(*[x.data_ptr() for x in ins])
    _lib.check(lib.qtb_bucket_c64(ctypes.byref(desc), ptrs, ctypes.c_void_p(out.data_ptr()),
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    j = np.arange(1 << u, dtype=np.int64)
    ref, mag = np.ones(1 << u, dtype=np.complex128), np.ones(1 << u)
    for x, data in zip(masks, host):
        off = np.zeros(1 << u, dtype=np.int64)
        bits = [b for b in range(u) if (x >> b) & 1]
        for i, b in enumerate(bits):
            off |= ((j >> b) & 1) << i
        ref = ref * data[off]
        mag = mag * np.abs(data[off])
    if sum_first:
        ref, mag = ref.reshape(2, -1).sum(0), mag.reshape(2, -1).sum(0)
    got = out.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 4 * len(masks) * EPS * mag + 1e-30)
