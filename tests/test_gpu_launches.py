"""Which kernels a call launches, where a test of results cannot tell."""
import numpy as np
import pytest
import torch

import graphs
from graph_nodes import captured_kernels
from qtensor_b200.plan import NetworkPlan, graph_csr

pytestmark = pytest.mark.gpu

TOL = 1e-5


def test_plain_path_shares_no_kernel_with_the_waves(cuda_device):
    """The plain path is what the wide waves are compared with, so its
    buckets go through the simple bucket kernel, not through the chunks that
    the waves contract their large ops by, at the sizes from which a bucket
    on its own does (2^17 outputs)."""
    p = 3
    G = graphs.erdos_renyi(60, 2)
    params = np.concatenate(graphs.angles(p, seed=3))
    plan = NetworkPlan(2 * p)
    plan.set_order_trials(0)
    plan.set_max_width(24, 1024)
    plan.add_lightcones(graph_csr(G), np.array(list(G.edges())), p, 0, params)
    plan.upload()
    infos = plan.infos()
    widest = max(range(len(plan)), key=lambda i: infos[i]['treewidth'])
    assert infos[widest]['treewidth'] > 18
    params_dev = torch.from_numpy(params).to(cuda_device)
    scratch = torch.empty(plan.plain_scratch_bytes(widest, 1), dtype=torch.uint8, device=cuda_device)
    term = torch.empty(1, dtype=torch.complex64, device=cuda_device)
    kernels = captured_kernels(lambda stream: plan.run_plain(widest, 1, params_dev, term, None, scratch, stream))
    names = set(k.name for k in kernels)
    assert sum('qtb_bucket_kernel' in k.name for k in kernels) == infos[widest]['n_ops']
    assert not any('wide' in name for name in names), names


@pytest.mark.parametrize('others,timed', [(0, False), (2000, True)])
def test_autotuner_beside_a_wide_network(cuda_device, monkeypatch, capfd, others, timed):
    """One network too large for shared memory beside the others of its graph,
    and beside those of a graph of `others` nodes more: the schedules are timed
    where most of the work is not in the wave, with the same terms."""
    import networkx as nx
    p = 3
    G = graphs.regular(60, seed=3)
    if others:
        G = nx.disjoint_union(G, graphs.regular(others, seed=1))
    params = np.concatenate(graphs.angles(p, seed=3))
    params_dev = torch.from_numpy(params).to(cuda_device)
    plan = NetworkPlan(2 * p)
    plan.set_order_trials(4)
    plan.add_lightcones(graph_csr(G), np.array(list(G.edges())), p, 0, params)
    plan.upload()
    scratch = torch.empty(plan.scratch_bytes(0, len(plan)), dtype=torch.uint8, device=cuda_device)
    energy = torch.empty(1, dtype=torch.float64, device=cuda_device)
    monkeypatch.setenv('QTB_AUTOTUNE_LOG', '1')
    stream = torch.cuda.current_stream().cuda_stream
    seen = []
    for tune in (False, True):
        terms = torch.zeros(len(plan), dtype=torch.complex64, device=cuda_device)
        plan.set_autotune(tune)
        plan.run(0, len(plan), params_dev, terms, energy, scratch, stream)
        torch.cuda.synchronize()
        assert plan.device_status() == 0
        assert sum(c[0] for c in plan.last_launch_config() if c[3] & 4) == 1
        seen.append((terms, energy.item(), capfd.readouterr().err))
    assert 'autotune' not in seen[0][2]
    assert ('persistent schedule' in seen[1][2]) == timed
    assert (seen[0][0] - seen[1][0]).abs().max().item() < TOL
    assert abs(seen[0][1] - seen[1][1]) <= TOL * abs(seen[0][1])
