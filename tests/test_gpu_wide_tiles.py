"""The wide executor's tiles at their edges: ops of one chunk, of several
groups of chunks, runs of small ops and whole small phases, with 16-byte
loads and, where the caller's scratch is only 8-byte aligned, without; on
the whole GPU and on half of every SM.  Every term equals the plain
per-bucket path's, an independent execution of the same plan, within the
repository's bar of 1e-5 for terms of magnitude at most 1."""
import numpy as np
import pytest
import torch

import graphs
from qtensor_b200.plan import NetworkPlan, graph_csr

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.mark.parametrize('family,n,seed,order_trials,shift,half', [
    ('regular', 60, 3, 4, 0, 0),      # one network just too large for shared memory
    ('regular', 60, 3, 4, 8, 0),      # 8-byte aligned scratch
    ('er', 60, 2, 0, 0, 0),           # reference orders: widths up to 23
    ('er', 60, 2, 0, 8, 1),
])
def test_wide_tiles_match_plain_path(cuda_device, family, n, seed, order_trials, shift, half):
    p = 3
    G = graphs.regular(n, seed=seed) if family == 'regular' else graphs.erdos_renyi(n, seed)
    gamma, beta = graphs.angles(p, seed=3)
    params = np.concatenate([gamma, beta])
    plan = NetworkPlan(2 * p)
    plan.set_order_trials(order_trials)
    plan.set_max_width(24, 1024)
    plan.set_wave_ctas_per_sm(half)
    plan.add_lightcones(graph_csr(G), np.array(list(G.edges())), p, 0, params)
    plan.upload()
    count = len(plan)
    scratch_bytes = plan.scratch_bytes(0, count)
    assert scratch_bytes > 0                       # some network runs in a wave
    dev = cuda_device
    params_dev = torch.from_numpy(params).to(dev)
    scratch = torch.empty(scratch_bytes + 16, dtype=torch.uint8, device=dev)
    terms = torch.empty(count, dtype=torch.complex64, device=dev)
    energy = torch.empty(1, dtype=torch.float64, device=dev)
    stream = torch.cuda.current_stream().cuda_stream
    for _ in range(2):                             # the queue and its counters start over
        terms.fill_(complex(np.nan, np.nan))
        plan.run(0, count, params_dev, terms, energy, scratch.data_ptr() + shift, stream)
        torch.cuda.synchronize()
        assert plan.device_status() == 0
    assert any(c[3] & 4 for c in plan.last_launch_config())
    plain_scratch = torch.empty(max(8, plan.plain_scratch_bytes(0, count)), dtype=torch.uint8, device=dev)
    plain = torch.empty_like(terms)
    plain_energy = torch.empty_like(energy)
    plan.run_plain(0, count, params_dev, plain, plain_energy, plain_scratch, stream)
    torch.cuda.synchronize()
    assert (terms - plain).abs().max().item() < TOL
    assert abs(energy.item() - plain_energy.item()) <= TOL * abs(plain_energy.item())
