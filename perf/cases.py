"""Performance cases of the framework: QAOA energies, bucket contractions,
merged-index products and amplitude batches, each through its public entry
point.

``listed()`` names the standing cases, ``draw(rng)`` gives one more of the
same ranges, ``prepare`` makes what a program holds before the call, ``run``
makes one call, ``work`` counts what the call cannot do without, and
``exact`` gives the call's result in 64 bits from plain torch and numpy.
Sizes are those of this repository's benchmark, tests and profiles
(3-regular N = 20 .. 1000 and Erdos-Renyi N = 400 graphs, the 24-variable
bucket, the K = 1024 contract-sum) or lie between them.
"""
import math
import random

import numpy as np
import torch


# ------------------------------------------------------------------ graphs
class Graph:
    """Nodes 0..n-1 and an undirected edge list, with the part of networkx's
    interface that the engine reads."""

    def __init__(self, n, edges):
        self._adj = {v: {} for v in range(n)}
        self._edges = [(int(a), int(b)) for a, b in edges]
        for a, b in self._edges:
            self._adj[a][b] = {}
            self._adj[b][a] = {}

    def nodes(self):
        return list(self._adj)

    def edges(self):
        return list(self._edges)

    def number_of_nodes(self):
        return len(self._adj)

    def number_of_edges(self):
        return len(self._edges)

    def neighbors(self, v):
        return iter(self._adj[v])

    def __len__(self):
        return len(self._adj)

    def __iter__(self):
        return iter(self._adj)

    def __getitem__(self, v):
        return self._adj[v]


def regular_graph(n, d, seed):
    """Random d-regular graph: a random pairing of the n d half-edges, loops
    and repeated edges removed by random edge swaps."""
    rng = random.Random(seed)
    stubs = [v for v in range(n) for _ in range(d)]
    rng.shuffle(stubs)
    pairs = [(stubs[i], stubs[i + 1]) for i in range(0, n * d, 2)]

    def key(e):
        return (min(e), max(e))

    count = {}
    for e in pairs:
        count[key(e)] = count.get(key(e), 0) + 1

    def bad(e):
        return e[0] == e[1] or count[key(e)] > 1

    todo = [i for i, e in enumerate(pairs) if bad(e)]
    while todo:
        i = todo.pop()
        while bad(pairs[i]):
            j = rng.randrange(len(pairs))
            (a, b), (c, e) = pairs[i], pairs[j]
            if i == j or a == e or c == b or count.get(key((a, e)), 0) or count.get(key((c, b)), 0):
                continue
            for k in (i, j):
                count[key(pairs[k])] -= 1
            pairs[i], pairs[j] = (a, e), (c, b)
            for k in (i, j):
                count[key(pairs[k])] = count.get(key(pairs[k]), 0) + 1
    return Graph(n, sorted(key(e) for e in pairs))


def erdos_renyi_graph(n, mean_degree, seed):
    rng = random.Random(seed)
    q = mean_degree / (n - 1)
    edges = [(a, b) for a in range(n) for b in range(a + 1, n) if rng.random() < q]
    return Graph(n, edges or [(0, 1)])


def make_graph(case):
    if case['family'] == 'regular':
        return regular_graph(case['n'], 3, case['graph_seed'])
    return erdos_renyi_graph(case['n'], 3.0, case['graph_seed'])


# ----------------------------------------------------------- qtree stand-ins
class Var:
    """A binary contraction index, as QTensor's simulators hand them to a backend."""

    def __init__(self, identity, size=2):
        self.identity = identity
        self.size = size
        self.name = 'v_{}'.format(identity)

    def copy(self, identity=None, size=None, name=None):
        return Var(self.identity if identity is None else identity, self.size if size is None else size)

    def __int__(self):
        return self.identity

    __index__ = __int__

    def __hash__(self):
        return hash((self.identity, self.size))

    def __eq__(self, other):
        return isinstance(other, Var) and (self.identity, self.size) == (other.identity, other.size)


class Tensor:
    """A named tensor over indices."""

    def __init__(self, name, indices, data_key=None, data=None):
        self.name = name
        self.indices = tuple(indices)
        self.data_key = data_key
        self.data = data

    def copy(self, name=None, indices=None, data_key=None, data=None):
        return Tensor(self.name if name is None else name, self.indices if indices is None else indices,
                      self.data_key if data_key is None else data_key, self.data if data is None else data)


class Gate:
    """A circuit gate: name, qubits, parameters."""

    def __init__(self, name, qubits, alpha=None):
        self.name = name
        self.qubits = tuple(qubits)
        self.parameters = {} if alpha is None else {'alpha': alpha}


# -------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest energy a user asks for: one angle pair on a graph that
        # a classroom example uses; launch and call latency
        {'name': 'energy_regular_n20_p1', 'kind': 'energy', 'family': 'regular', 'n': 20, 'p': 1, 'graph_seed': 0},
        # an ordinary angle-search call: a hundred nodes, three layers
        {'name': 'energy_regular_n100_p3', 'kind': 'energy', 'family': 'regular', 'n': 100, 'p': 3, 'graph_seed': 0},
        # the benchmark's headline call: 1500 edge networks, all in shared memory
        {'name': 'energy_regular_n1000_p3', 'kind': 'energy', 'family': 'regular', 'n': 1000, 'p': 3,
         'graph_seed': 0},
        # four layers: some edge networks outgrow shared memory
        {'name': 'energy_regular_n256_p4', 'kind': 'energy', 'family': 'regular', 'n': 256, 'p': 4, 'graph_seed': 0},
        # an irregular graph, networks of every width, the widest energy here
        {'name': 'energy_er_n400_p3', 'kind': 'energy', 'family': 'er', 'n': 400, 'p': 3, 'graph_seed': 6},
        # one bucket of a QTensor simulation through the drop-in backend, of the
        # size most buckets have; call latency
        {'name': 'bucket_v6', 'kind': 'bucket', 'vars': 6, 'tensors': 3, 'no_sum': False, 'shape_seed': 1},
        # the widest bucket of the profiles: one operand over nearly all of 24
        # variables, a smaller one and a gate
        {'name': 'bucket_v24', 'kind': 'bucket', 'vars': 24, 'tensors': 3, 'no_sum': False, 'shape_seed': 0},
        # a merged contraction with a long summed index: tensor cores
        {'name': 'contract_k1024', 'kind': 'contract', 'K': 1024, 'F': 2, 'M': 1024, 'N': 1024},
        # the same on odd sizes that no tile divides
        {'name': 'contract_k500_ragged', 'kind': 'contract', 'K': 500, 'F': 3, 'M': 333, 'N': 190},
        # the extended backend's own bucket: the sum over one binary variable
        {'name': 'contract_k2', 'kind': 'contract', 'K': 2, 'F': 64, 'M': 512, 'N': 512},
        # the extended backend's merge of two tensors over their common indices
        {'name': 'outer_n256', 'kind': 'outer', 'n': 256, 'm': 256, 'k': 256},
        # amplitudes of a circuit seen once: conversion, compile, upload,
        # contraction and read-back are all part of the call
        {'name': 'amplitudes_q12_b4', 'kind': 'amplitudes', 'qubits': 12, 'layers': 4, 'batch': 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['energy', 'energy', 'energy', 'bucket', 'contract', 'contract', 'outer', 'amplitudes'])
    if kind == 'energy':
        seed = rng.randrange(1000)
        if rng.random() < 0.25:
            # Erdos-Renyi graphs of one or two layers: three layers reach
            # widths whose cost has no bound on random graphs
            return {'kind': kind, 'family': 'er', 'n': _log_int(rng, 20, 400), 'p': rng.randint(1, 2),
                    'graph_seed': seed}
        p = rng.choice([1, 2, 3, 3, 4])
        # three layers from 60 nodes on and four from 256: below, the
        # lightcones cover the whole graph and their width is the graph's
        lo, hi = {1: (16, 1000), 2: (30, 1000), 3: (60, 1000), 4: (256, 320)}[p]
        return {'kind': kind, 'family': 'regular', 'n': 2 * (_log_int(rng, lo, hi) // 2), 'p': p, 'graph_seed': seed}
    if kind == 'bucket':
        return {'kind': kind, 'vars': rng.randint(3, 23), 'tensors': rng.randint(2, 6),
                'no_sum': rng.random() < 0.25, 'shape_seed': rng.randrange(1 << 30)}
    if kind == 'contract':
        if rng.random() < 0.5:
            K, F = _log_int(rng, 32, 1024), rng.randint(1, 2)
            return {'kind': kind, 'K': K, 'F': F, 'M': _log_int(rng, 64, 1024), 'N': _log_int(rng, 64, 1024)}
        K = rng.choice([1, 2, 2, 2, 4, 8])
        return {'kind': kind, 'K': K, 'F': _log_int(rng, 1, 64), 'M': _log_int(rng, 2, 500), 'N': _log_int(rng, 2, 500)}
    if kind == 'outer':
        return {'kind': kind, 'n': _log_int(rng, 1, 256), 'm': _log_int(rng, 1, 256), 'k': _log_int(rng, 1, 256)}
    return {'kind': kind, 'qubits': rng.randint(4, 12), 'layers': rng.randint(1, 4), 'batch': rng.randint(0, 4)}


# ------------------------------------------------------------------- inputs
def _angles(case, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0, np.pi, case['p']), rng.uniform(0, np.pi, case['p'])


def _device():
    return torch.device('cuda', torch.cuda.current_device()) if torch.cuda.is_available() else torch.device('cpu')


def _complex(shape, seed):
    """Unit-variance complex64 values on the device, from the seed."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex64, device=dev, generator=gen)


def bucket_indices(case):
    """Index ids of every tensor of the bucket, sorted; all hold the bucket
    variable 0.  The first is over nearly all variables, as the message from
    an earlier bucket is; the others are gates and smaller messages."""
    rng = random.Random(case['shape_seed'])
    u = case['vars']
    rest = list(range(1, u))
    if case['shape_seed'] == 0:
        return [list(range(u - 1)), [0] + list(range(u // 2, u)), [0, u - 1]][:case['tensors']]
    out = [[0] + [v for v in rest if rng.random() < 0.9]]
    for _ in range(case['tensors'] - 1):
        size = rng.choice([1, 1, 2, 3, max(1, u // 3), max(1, u // 2)])
        out.append([0] + sorted(rng.sample(rest, min(size, len(rest)))))
    held = set(v for ix in out for v in ix)
    out[0] = sorted(set(out[0]) | (set(range(u)) - held))
    return out


def _bucket_arrays(case, seed):
    return [_complex([2] * len(ix), seed * 64 + t) for t, ix in enumerate(bucket_indices(case))]


def _circuit(case, seed):
    """Layers of Hadamards and rotations on every qubit and entangling gates
    on random pairs, over every gate name the simulator takes."""
    shape = random.Random(case['qubits'] * 1009 + case['layers'])     # the circuit's layout
    rng = random.Random(seed)                                         # its angles
    n, qc = case['qubits'], []
    for q in range(n):
        qc.append(('H', (q,), None))
    for _ in range(case['layers']):
        order = list(range(n))
        shape.shuffle(order)
        for a, b in zip(order[::2], order[1::2]):
            name = shape.choice(['cZ', 'cX', 'ZZ'])
            qc.append((name, (a, b), rng.uniform(0, 2) if name == 'ZZ' else None))
        for q in range(n):
            name = shape.choice(['XPhase', 'YPhase', 'ZPhase', 'T', 'H'])
            qc.append((name, (q,), rng.uniform(0, 2) if name.endswith('Phase') else None))
    return qc


def prepare(case, seed):
    kind = case['kind']
    if kind == 'energy':
        from qtensor_b200.engine import QAOAEnergyEngine
        G = make_graph(case)
        gamma, beta = _angles(case, seed)
        engine = QAOAEnergyEngine()
        compiled = engine.compile(G, case['p'], gamma, beta)
        return {'kind': kind, 'engine': engine, 'G': G, 'gamma': gamma, 'beta': beta, 'compiled': compiled}
    if kind == 'bucket':
        from qtensor_b200.backend import B200Backend
        ids, arrays = bucket_indices(case), _bucket_arrays(case, seed)
        bucket = [Tensor('T{}'.format(t), [Var(v) for v in ix], data=a) for t, (ix, a) in enumerate(zip(ids, arrays))]
        return {'kind': kind, 'backend': B200Backend(), 'bucket': bucket, 'no_sum': case['no_sum']}
    if kind == 'contract':
        K, F, M, N = case['K'], case['F'], case['M'], case['N']
        return {'kind': kind, 'a': _complex([K, F, M], 2 * seed), 'b': _complex([K, F, N], 2 * seed + 1),
                'c': torch.empty([F, M, N], dtype=torch.complex64, device=_device())}
    if kind == 'outer':
        n, m, k = case['n'], case['m'], case['k']
        return {'kind': kind, 'a': _complex([n, m], 2 * seed), 'b': _complex([n, k], 2 * seed + 1),
                'c': torch.empty([n, m, k], dtype=torch.complex64, device=_device())}
    from qtensor_b200.simulator import QtreeSimulator
    return {'kind': kind, 'sim': QtreeSimulator(), 'circuit': [Gate(*g) for g in _circuit(case, seed)],
            'batch': case['batch']}


def run(state):
    kind = state['kind']
    if kind == 'energy':
        # the energy, and the edge terms the plan keeps on the device
        energy = state['engine'].energy_expectation(state['G'], state['gamma'], state['beta'])
        return {'energy': energy, 'terms': state['compiled'].terms}
    if kind == 'bucket':
        return state['backend'].process_bucket(state['bucket'], no_sum=state['no_sum']).data
    from qtensor_b200 import tcontract
    if kind == 'contract':
        return tcontract.mkl_contract_sum(state['a'], state['b'], state['c'])
    if kind == 'outer':
        return tcontract.mkl_contract_complex(state['a'], state['b'], state['c'])
    return state['sim'].simulate_batch(state['circuit'], state['batch'])


# --------------------------------------------------------------------- work
def work(case):
    """bytes: inputs read once, outputs written once.  flops: of an energy or
    an amplitude batch, the products and sums of its networks' buckets (6 per
    complex product, 2 per complex sum) in the elimination orders that the
    plan compiler finds; of a bucket or a contraction, its own."""
    kind = case['kind']
    if kind == 'energy':
        from qtensor_b200.plan import NetworkPlan, graph_csr
        G = make_graph(case)
        plan = NetworkPlan(2 * case['p'])
        plan.set_order_trials(16)
        plan.set_max_width(29, 1024)
        plan.add_lightcones(graph_csr(G), np.array(G.edges(), dtype=np.int32), case['p'], 0, np.concatenate(_angles(case, 0)))
        flops = sum(i['alg_flops'] for i in plan.infos())
        return {'bytes': 16 * case['p'] + 8 + 8 * len(plan), 'flops': flops}
    if kind == 'bucket':
        ids = bucket_indices(case)
        out = case['vars'] - (0 if case['no_sum'] else 1)
        return {'bytes': 8 * (sum(2 ** len(ix) for ix in ids) + 2 ** out),
                'flops': 6 * (len(ids) - 1) * 2 ** case['vars'] + (0 if case['no_sum'] else 2 * 2 ** out)}
    if kind == 'contract':
        K, F, M, N = case['K'], case['F'], case['M'], case['N']
        return {'bytes': 8 * F * (K * (M + N) + M * N), 'flops': 8 * F * M * N * K}
    if kind == 'outer':
        n, m, k = case['n'], case['m'], case['k']
        return {'bytes': 8 * n * (m + k + m * k), 'flops': 6 * n * m * k}
    n, out = case['qubits'], 2 ** case['batch']
    gates = len(_circuit(case, 0))
    return {'bytes': 24 * gates + 16 * out, 'flops': 8 * gates * out + 8 * 2 ** n}


# -------------------------------------------------------------------- exact
def _eliminate(factors, device):
    """Sum over all variables of the product of ``factors`` (index tuple,
    complex128 array over them): buckets in least-degree order."""
    factors = dict(enumerate(factors))
    holds, nbrs = {}, {}
    for k, (ix, _) in factors.items():
        for v in ix:
            holds.setdefault(v, set()).add(k)
            nbrs.setdefault(v, set()).update(ix)
    for v in nbrs:
        nbrs[v].discard(v)
    by_degree = {}
    for v, s in nbrs.items():
        by_degree.setdefault(len(s), set()).add(v)
    scalar, fresh = 1.0 + 0.0j, len(factors)
    pending = []
    for _ in range(len(nbrs)):
        v = None
        for deg in range(len(nbrs) + 1):
            if by_degree.get(deg):
                v = min(by_degree[deg])
                break
        near = nbrs.pop(v)
        by_degree[len(near)].discard(v)
        for w in near:
            by_degree[len(nbrs[w])].discard(w)
        for w in near:
            nbrs[w] |= near
            nbrs[w] -= {w, v}
        for w in near:
            by_degree.setdefault(len(nbrs[w]), set()).add(w)
        out = sorted(near)
        members = sorted(holds.pop(v), key=lambda k: len(factors[k][0]))
        place = {w: i for i, w in enumerate([v] + out)}
        args = []
        for k in members:
            ix, t = factors.pop(k)
            args += [t, [place[w] for w in ix]]
            for w in ix:
                if w != v:
                    holds[w].discard(k)
        if device.type == 'cpu':
            r = np.einsum(*args, list(range(1, len(out) + 1))) if len(args) <= 4 else None
            if r is None:
                acc, acc_ix = args[0], args[1]
                for t, ix in zip(args[2::2], args[3::2]):
                    both = sorted(set(acc_ix) | set(ix))
                    acc, acc_ix = np.einsum(acc, acc_ix, t, ix, both), both
                r = np.einsum(acc, acc_ix, list(range(1, len(out) + 1)))
        else:
            r = torch.einsum(*args, list(range(1, len(out) + 1)))
        if out:
            factors[fresh] = (tuple(out), r)
            for w in out:
                holds[w].add(fresh)
            fresh += 1
        else:
            pending.append(complex(r) if device.type == 'cpu' else r)
    for r in pending:
        scalar = scalar * r
    return complex(scalar)


def _edge_term(G, edge, gamma, beta, device):
    """<psi| Z_u Z_v |psi> of the MaxCut ansatz as a sum over basis paths: a
    node at distance d from the edge keeps its mixers of layers 1..p-d (the
    later ones cancel against their inverses), a graph edge its phases of
    the layers up to one of its ends' last mixer."""
    p = len(gamma)
    dist = {edge[0]: 0, edge[1]: 0}
    shell = [edge[0], edge[1]]
    for d in range(1, p + 1):
        shell = [w for v in shell for w in G[v] if w not in dist and not dist.update({w: d})]
    mixers = {v: p - d for v, d in dist.items()}
    names, top = {}, [0]

    def var(v, level, side):
        key = (v, level, 0 if level == mixers[v] else side)   # the last one is shared
        if key not in names:
            names[key] = top[0]
            top[0] += 1
        return names[key]

    spin = np.array([1.0, -1.0])
    factors = []

    def put(ix, t):
        order = np.argsort(ix)
        t = np.ascontiguousarray(np.transpose(t, order))
        factors.append((tuple(ix[i] for i in order), torch.from_numpy(t).to(device) if device.type != 'cpu' else t))

    for v, m in mixers.items():
        put([var(v, m, 0)], np.array([0.5, 0.5]) if v not in edge else 0.5 * spin + 0j * spin)
        for side in (0, 1):
            for layer in range(m):
                c, s = math.cos(math.pi * beta[layer]), math.sin(math.pi * beta[layer])
                mix = np.array([[c, -1j * s], [-1j * s, c]])
                put([var(v, layer, side), var(v, layer + 1, side)], mix if side == 0 else mix.conj())
    seen = set()
    for a in mixers:
        for b in G[a]:
            if b not in mixers or (min(a, b), max(a, b)) in seen:
                continue
            seen.add((min(a, b), max(a, b)))
            for layer in range(min(p, max(mixers[a], mixers[b]))):
                for side in (0, 1):
                    phase = np.exp(-1j * np.pi * gamma[layer] * np.outer(spin, spin))
                    ia, ib = var(a, min(layer, mixers[a]), side), var(b, min(layer, mixers[b]), side)
                    put([ia, ib], phase if side == 0 else phase.conj())
    factors = [(ix, (t.to(torch.complex128) if device.type != 'cpu' else t.astype(np.complex128))) for ix, t in factors]
    return _eliminate(factors, device)


def _cone_key(G, edge, p):
    """The cone's own numbering (breadth first from the edge) and edges, so
    that edges whose cones are numbered alike are contracted once."""
    number = {edge[0]: 0, edge[1]: 1}
    order = [edge[0], edge[1]]
    dist = {edge[0]: 0, edge[1]: 0}
    for v in order:
        if dist[v] == p:
            continue
        for w in G[v]:
            if w not in number:
                number[w] = len(order)
                dist[w] = dist[v] + 1
                order.append(w)
    return tuple(sorted((min(number[a], number[b]), max(number[a], number[b]))
                        for a in order for b in G[a] if b in number and a < b))


def _state_vector(qc, n):
    psi = np.zeros([2] * n, dtype=np.complex128)
    psi[(0,) * n] = 1.0
    r = math.sqrt(0.5)
    fixed = {'H': np.array([[r, r], [r, -r]]), 'T': np.diag([1, np.exp(0.25j * np.pi)]),
             'cZ': np.diag([1, 1, 1, -1.0]), 'cX': np.eye(4)[[0, 1, 3, 2]]}
    for name, qubits, alpha in qc:
        if name in fixed:
            u = fixed[name]
        elif name == 'ZZ':
            u = np.diag(np.exp(-0.5j * np.pi * alpha * np.array([1, -1, -1, 1])))
        else:
            c, s, g = math.cos(math.pi * alpha / 2), math.sin(math.pi * alpha / 2), np.exp(0.5j * math.pi * alpha)
            u = {'XPhase': g * np.array([[c, -1j * s], [-1j * s, c]]), 'YPhase': g * np.array([[c, -s], [s, c]]),
                 'ZPhase': np.diag([1, np.exp(1j * math.pi * alpha)])}[name]
        k = len(qubits)
        u = np.asarray(u, dtype=np.complex128).reshape([2] * (2 * k))
        psi = np.moveaxis(np.tensordot(u, psi, axes=(list(range(k, 2 * k)), list(qubits))), list(range(k)), list(qubits))
    return psi


def exact(case, seed):
    kind, device = case['kind'], _device()
    if kind == 'energy':
        G = make_graph(case)
        gamma, beta = _angles(case, seed)
        known, terms = {}, []
        for e in G.edges():
            key = _cone_key(G, e, case['p'])
            if key not in known:
                known[key] = _edge_term(G, e, gamma, beta, device)
            terms.append(known[key])
        terms = np.array(terms)
        return {'energy': float((len(terms) - math.fsum(terms.real)) / 2), 'terms': terms}
    if kind == 'bucket':
        arrays = [a.to(torch.complex128) for a in _bucket_arrays(case, seed)]
        acc = None
        for ix, a in zip(bucket_indices(case), arrays):
            # bring each operand to the union's axes, merged where it has or
            # lacks neighbouring ones together
            shape = [2 if v in ix else 1 for v in range(case['vars'])]
            a = a.reshape(shape).expand([2] * case['vars'])
            a = a.reshape(-1)
            acc = a if acc is None else acc * a
        if not case['no_sum']:
            acc = acc.reshape(2, -1).sum(0)
        return acc.reshape([2] * (case['vars'] - (0 if case['no_sum'] else 1)))
    if kind in ('contract', 'outer'):
        state = prepare(case, seed)
        a, b = state['a'].to(torch.complex128), state['b'].to(torch.complex128)
        if kind == 'outer':
            return a[:, :, None] * b[:, None, :]
        return torch.matmul(a.permute(1, 2, 0), b.permute(1, 0, 2))
    psi = _state_vector(_circuit(case, seed), case['qubits'])
    return psi.reshape(2 ** case['batch'], -1)[:, 0]
