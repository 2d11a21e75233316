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


@pytest.mark.parametrize('n,p,seed,schedule,capped,ctas_per_sm', [
    (1000, 2, 1, 'persistent:128', True, 8),     # compact records only, two networks per CTA without
    (300, 2, 1, 'persistent:512', True, 2),
    (1000, 3, 0, 'persistent:128', True, 7),     # shared memory holds seven
    (300, 2, 1, 'persistent:256', False, 2),     # 450 networks, 296 CTAs
    (300, 3, 1, 'persistent:512', True, 2),      # wide records
    (1000, 3, 1, 'persistent:256', True, 3),
    (100, 3, 1, 'persistent:512', False, 1),     # a CTA for nearly every network
    (1000, 3, 1, 'persistent:128', False, 3),    # as many CTAs as shared memory holds either way
    (1000, 3, 1, 'hybrid12:512', True, 12),      # the 96-thread queue
])
def test_persistent_launches_keep_their_ctas(cuda_device, monkeypatch, n, p, seed, schedule, capped, ctas_per_sm):
    """The persistent kernel's three forms: where a CTA would take two
    networks or more, registers leave as many CTAs per SM as shared memory and
    64 registers allow; the 96-thread queue does not spill (24 bytes of frame
    are the angles' range reduction); the terms are those of the class
    schedule."""
    G = graphs.regular(n, seed=seed)
    params = np.concatenate(graphs.angles(p, seed=3))
    params_dev = torch.from_numpy(params).to(cuda_device)
    plan = NetworkPlan(2 * p)
    plan.set_order_trials(16)
    plan.add_lightcones(graph_csr(G), np.array(list(G.edges())), p, 0, params)
    plan.upload()
    count = len(plan)
    assert plan.scratch_bytes(0, count) == 0
    classes = torch.zeros(count, dtype=torch.complex64, device=cuda_device)
    plan.run(0, count, params_dev, classes, None, None, torch.cuda.current_stream().cuda_stream)
    monkeypatch.setenv('QTB_SCHEDULE', schedule)
    terms = torch.zeros_like(classes)
    kernels = captured_kernels(lambda stream: plan.run(0, count, params_dev, terms, None, None, stream))
    assert plan.device_status() == 0
    threads = 96 if schedule.startswith('hybrid12') else int(schedule.split(':')[1])
    queue = [k for k in kernels if k.threads == threads and 'ELb1ELi' in k.name]   # kPersistent
    assert len(queue) == 1
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    assert queue[0].grid == min(count, ctas_per_sm * sms) or threads == 96
    if capped:
        assert queue[0].registers * threads * ctas_per_sm <= 65536
        assert queue[0].local_bytes <= 24
    assert (terms - classes).abs().max().item() < TOL
