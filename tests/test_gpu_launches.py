"""Which kernels a call launches, where a test of results cannot tell."""
import numpy as np
import pytest
import torch

import graphs
from graph_nodes import captured_kernels
from qtensor_b200.plan import NetworkPlan, graph_csr

pytestmark = pytest.mark.gpu


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
