"""The work that programs have this framework do, as cases that can be timed and checked.

Every case goes through a public entry point: the synchronous engine call on host arrays, the
reference-shaped `solve_accelerated_box`, the continuous-batching server, re-runs of resident
solves (single and batched), the plugin-level iteration, the device verification calls and the
constrained-QP inner solve.  Problems are the framework's planted families (random-graph
Laplacians, 2-D grids, the tridiagonal scale family) with sizes, tolerances and distributions of
its benchmark configurations, odd sizes among them; they are made here from the seed alone, so the
planted optimum is known without any of the framework's code.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / 'hypergrey-sih-26_gb300'))
import boxqp  # noqa: E402
from boxqp.serve import BoxQPServer  # noqa: E402

STEPS = 25          # plugin steps per pass: the reference's loop checks every 25 iterations
ADMM_ROW = 8        # entries per constraint row of the ADMM system
ADMM_SIGMA = 1e-8   # the reference's regularisation of the x-update


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one request of the serving stream (latency and launches)
        {'name': 'serve_one', 'kind': 'serve', 'count': 1, 'n_lo': 1000, 'n_hi': 1000},
        # the reference's API with its defaults (FP64, tolerance 1e-7) on the small configuration
        {'name': 'api_graph10k_fp64', 'kind': 'api', 'family': 'graph', 'n': 10000, 'epv': 5, 'tol': 1e-7,
         'precision': 'fp64'},
        # a burst of the serving stream: sizes 1k to 200k, both tolerances, overlapping on the device
        {'name': 'serve_burst', 'kind': 'serve', 'count': 16, 'n_lo': 1000, 'n_hi': 200000},
        # a re-run of a resident uneven batch (the batched configuration, at 256 instances)
        {'name': 'batch_uneven', 'kind': 'batch', 'count': 256, 'n_lo': 64, 'n_hi': 16384, 'tol': 1e-6},
        # the reference's plugin contract: 25 device iterations between two host checks
        {'name': 'plugin_graph', 'kind': 'plugin', 'family': 'graph', 'n': 300007, 'epv': 5},
        # verification of a candidate and the convexity gate on caller-owned device arrays
        {'name': 'verify_graph', 'kind': 'verify', 'family': 'graph', 'n': 1000000, 'epv': 7},
        # the ill-conditioned grid configuration at its tight tolerance, resident
        {'name': 'resident_grid_mixed', 'kind': 'resident', 'family': 'grid', 'n': 1024 * 1024, 'epv': 0, 'tol': 1e-8,
         'precision': 'mixed'},
        # the headline configuration, resident in device memory
        {'name': 'resident_graph1m_mixed', 'kind': 'resident', 'family': 'graph', 'n': 1000000, 'epv': 7, 'tol': 1e-6,
         'precision': 'mixed'},
        # the headline configuration end to end from host arrays
        {'name': 'solve_graph1m_mixed', 'kind': 'solve', 'family': 'graph', 'n': 1000000, 'epv': 7, 'tol': 1e-6,
         'precision': 'mixed'},
        # the constrained-QP inner solve on a 1M-variable system
        {'name': 'admm_graph1m', 'kind': 'admm', 'family': 'graph', 'n': 1000000, 'epv': 7, 'rows': 500000},
        # the reference's published scale family with its own numerics (FP64, 1e-7)
        {'name': 'resident_tridiagonal_fp64', 'kind': 'resident', 'family': 'tridiagonal', 'n': 1000000, 'epv': 0,
         'tol': 1e-7, 'precision': 'fp64'},
        # the largest: the plain FP64 engine on the headline problem
        {'name': 'resident_graph1m_fp64', 'kind': 'resident', 'family': 'graph', 'n': 1000000, 'epv': 7, 'tol': 1e-6,
         'precision': 'fp64'},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges; odd sizes come by themselves."""
    kind = rng.choice(['solve', 'solve', 'resident', 'resident', 'resident', 'api', 'serve', 'batch', 'plugin',
                       'verify', 'admm'])
    if kind == 'serve':
        lo = _log_int(rng, 1000, 20000)
        return {'kind': kind, 'count': rng.randint(1, 16), 'n_lo': lo, 'n_hi': _log_int(rng, lo, 200000)}
    if kind == 'batch':
        return {'kind': kind, 'count': _log_int(rng, 16, 256), 'n_lo': 64, 'n_hi': _log_int(rng, 1000, 16384),
                'tol': rng.choice([1e-4, 1e-6, 1e-8])}
    family = 'graph' if kind in ('api', 'verify', 'admm') else rng.choice(['graph', 'graph', 'grid', 'tridiagonal'])
    precision = rng.choice(['mixed', 'mixed', 'fp64', 'fp64', 'fp64_exact'])
    n = _log_int(rng, 1000, 50000 if kind == 'api' else 200000 if precision == 'fp64_exact' else 1000000)
    if family == 'grid':
        n = max(32, math.isqrt(n)) ** 2
    epv = rng.randint(2, 7) if family == 'graph' else 0
    case = {'kind': kind, 'family': family, 'n': n, 'epv': epv}
    if kind == 'admm':
        case['rows'] = n // 2
    if kind in ('solve', 'resident', 'api'):
        case['precision'] = 'fp64' if kind == 'api' else precision
        case['tol'] = rng.choice([1e-4, 1e-6, 1e-8]) if case['precision'] == 'mixed' else rng.choice([1e-6, 1e-7])
    return case


# ------------------------------------------------------------------------------------------
# planted problems
# ------------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    return g


def _host(t):
    return t.cpu().numpy()


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device='cuda', dtype=torch.float64)


def _row_sums(p, terms):
    return np.add.reduceat(terms, p['rowptr'][:-1])  # every row has its diagonal entry


def _times(p, x):
    return _row_sums(p, p['val'] * x[p['col']])


def _csr(n, rows, cols, vals):
    """Host CSR of entries already in row-major order."""
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device='cuda')
    rowptr[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return {'n': n, 'rowptr': _host(rowptr.to(torch.int32)), 'col': _host(cols.to(torch.int32)), 'val': _host(vals)}


def _banded(n, offsets, valid, values):
    """Rows of fixed offsets from the diagonal: column i + offset where valid(i) holds."""
    i = torch.arange(n, device='cuda')
    cols = torch.stack([i + o for o in offsets], 1)
    mask = torch.stack([valid[k](i) for k in range(len(offsets))], 1)
    vals = torch.tensor(values, dtype=torch.float64, device='cuda').expand(n, -1)
    rows = i[:, None].expand_as(cols)
    return _csr(n, rows[mask], cols[mask], vals[mask])


def _graph(g, n, epv):
    """Weighted Laplacian of a random graph plus a positive diagonal."""
    a = torch.randint(n, (epv * n,), generator=g, device='cuda')
    b = torch.randint(n, (epv * n,), generator=g, device='cuda')
    w = _uniform(g, epv * n, 0.1, 1.0)
    key = torch.minimum(a, b) * n + torch.maximum(a, b)
    key, order = torch.sort(torch.where(a == b, torch.full_like(key, -1), key), stable=True)
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]
    first &= key >= 0
    key, w = key[first], w[order][first]
    lo, hi = key // n, key % n
    i = torch.arange(n, device='cuda')
    rows, cols = torch.cat([lo, hi, i]), torch.cat([hi, lo, i])
    vals = torch.cat([-w, -w, torch.zeros(n, dtype=torch.float64, device='cuda')])
    order = torch.argsort(rows * n + cols)
    rows, cols = rows[order], cols[order]
    p = _csr(n, rows, cols, vals[order])
    at = _host(torch.nonzero(rows == cols)[:, 0])
    p['val'][at] = -_row_sums(p, p['val']) + _host(_uniform(g, n, 0.5, 2.0))
    return p


def _plant(g, p, lower, upper, share, inner):
    """Bounds, the planted optimum x* (`share` of the rows at each bound) and c = -Q x* + z."""
    n = p['n']
    u = torch.rand(n, generator=g, device='cuda', dtype=torch.float64)
    inside = lower + (upper - lower) * _uniform(g, n, *inner)
    dual = _uniform(g, n, 0.1, 1.0)
    at_lower, at_upper = u < share, (u >= share) & (u < 2 * share)
    x = torch.where(at_lower, lower, torch.where(at_upper, upper, inside))
    z = torch.where(at_lower, dual, torch.where(at_upper, -dual, torch.zeros_like(dual)))
    p['lower'], p['upper'], p['x'] = _host(lower), _host(upper), _host(x)
    p['c'] = -_times(p, p['x']) + _host(z)
    return p


def _full(n, v):
    return torch.full((n,), float(v), dtype=torch.float64, device='cuda')


def _problem(family, n, epv, seed):
    g = _generator(seed)
    if family == 'tridiagonal':
        p = _banded(n, [-1, 0, 1], [lambda i: i > 0, lambda i: i >= 0, lambda i: i < n - 1], [-1.0, 2.02, -1.0])
        x = 0.5 + torch.randint(10001, (n,), generator=g, device='cuda').to(torch.float64) / 10000
        p['lower'], p['upper'], p['x'] = np.zeros(n), np.full(n, 3.0), _host(x)
        p['c'] = -_times(p, p['x'])
        return p
    if family == 'grid':
        s = math.isqrt(n)
        p = _banded(n, [-s, -1, 0, 1, s], [lambda i: i >= s, lambda i: i % s > 0, lambda i: i >= 0,
                                           lambda i: i % s < s - 1, lambda i: i < n - s], [-1.0, -1.0, 4.001, -1.0, -1.0])
        return _plant(g, p, _uniform(g, n, -1.0, -0.5), _uniform(g, n, 0.5, 1.0), 0.2, (0.05, 0.95))
    p = _graph(g, n, epv)
    if epv >= 7:
        return _plant(g, p, _full(n, -1), _full(n, 1), 0.25, (0.05, 0.95))
    return _plant(g, p, _full(n, 0), _full(n, 1), 0.3, (0.1, 0.9))


def _mix(case, seed):
    """The problems of a serving burst or of an uneven batch: sizes log-uniform in the range, the
    same for every seed (the answers keep their shapes), the problems themselves from the seed."""
    rng = np.random.default_rng([case['count'], case['n_lo'], case['n_hi']])
    got = []
    for k in range(case['count']):
        n = int(np.exp(rng.uniform(np.log(case['n_lo']), np.log(case['n_hi']))) + 0.5)
        epv = 5 if case['kind'] == 'serve' else int(rng.integers(2, 7))
        got.append(_problem('graph', n, epv, seed * 4099 + k))
    return got


def _arrays(p):
    return p['rowptr'], p['col'], p['val'], p['c'], p['lower'], p['upper']


def _objective(p):
    x = p['x']
    return float(0.5 * np.dot(x, _times(p, x)) + np.dot(p['c'], x))


def _lipschitz(p):
    return float(np.max(_row_sums(p, np.abs(p['val']))))


def _lower_triplets(p):
    rows = np.repeat(np.arange(p['n'], dtype=np.int64), np.diff(p['rowptr']))
    keep = p['col'] <= rows
    return rows[keep], p['col'][keep].astype(np.int64), p['val'][keep]


def _momenta():
    t, got = 1.0, []
    for _ in range(STEPS):
        nt = (1.0 + math.sqrt(1.0 + 4.0 * t * t)) / 2.0
        got.append((t - 1.0) / nt)
        t = nt
    return got


def _candidate(p, seed):
    """A point near the optimum, inside the box, as a solver would hand it to the verification."""
    noise = np.random.default_rng(seed + 7).uniform(-1e-3, 1e-3, p['n'])
    return np.clip(p['x'] + noise, p['lower'], p['upper'])


def _constraints(case, seed):
    """A of the ADMM system (rows of ADMM_ROW entries), rho per row and a right-hand side."""
    rng = np.random.default_rng(seed + 11)
    n, m = case['n'], case['rows']
    cols = np.sort(rng.integers(0, n, size=(m, ADMM_ROW)), axis=1)
    return {'rowptr': (np.arange(m + 1) * ADMM_ROW).astype(np.int32), 'col': cols.reshape(-1).astype(np.int32),
            'val': rng.normal(size=m * ADMM_ROW), 'rho': np.where(rng.random(m) < 0.1, 10.0, 0.1),
            'rhs': rng.normal(size=n)}


def _accuracy(rhs):
    return 1e-7 * (1.0 + float(np.max(np.abs(rhs))))  # the reference's first-iteration accuracy


# ------------------------------------------------------------------------------------------
# what a program keeps, and one pass
# ------------------------------------------------------------------------------------------
class _Resident:
    """Solved problems kept resident in the process's engine, released with this object."""

    def __init__(self, problems, options):
        self.engine = boxqp.default_engine()
        self.ids = [self.engine.submit(*_arrays(p), options) for p in problems]
        for i in self.ids:
            self.engine.wait(i)
        ends = np.cumsum([p['n'] for p in problems])
        self.x = np.zeros(int(ends[-1]))
        self.views = np.split(self.x, ends[:-1])

    def run(self):
        self.engine.resolve(self.ids)
        stats = []
        for i, view in zip(self.ids, self.views):
            self.engine.wait(i)
            stats.append(self.engine.fetch(i, view.shape[0], out=view)[1])
        return self.x, stats

    def __del__(self):
        for i in self.ids:
            self.engine.release(i)


_servers = []


def _server():
    if not _servers:
        _servers.append(BoxQPServer())
    return _servers[0]


def prepare(case, seed):
    kind = case['kind']
    if kind == 'serve':
        return {'kind': kind, 'server': _server(), 'requests': [(_arrays(p), 1e-4 if k % 2 == 0 else 1e-8)
                                                                for k, p in enumerate(_mix(case, seed))]}
    if kind == 'batch':
        return {'kind': kind, 'solves': _Resident(_mix(case, seed), boxqp.options_struct(case['tol'], 60.0, 200000, 'mixed'))}
    p = _problem(case['family'], case['n'], case['epv'], seed)
    if kind in ('solve', 'resident'):
        options = boxqp.options_struct(case['tol'], 60.0, 200000, case['precision'])
        state = {'kind': kind, 'counted': case['precision'] != 'mixed'}
        if kind == 'resident':
            return dict(state, solves=_Resident([p], options))
        return dict(state, engine=boxqp.default_engine(), arrays=_arrays(p), options=options)
    if kind == 'api':
        rows, cols, vals = _lower_triplets(p)
        return {'kind': kind, 'options': boxqp.QpOptions(tolerance=case['tol'], precision=case['precision']),
                'problem': boxqp.QuadraticProblem(cost=p['c'], lower=p['lower'], upper=p['upper'], hessian_row=rows,
                                                  hessian_col=cols, hessian_val=vals)}
    if kind == 'plugin':
        return {'kind': kind, 'box': boxqp.make_cuda_box(*_arrays(p), _lipschitz(p)), 'momenta': _momenta()}
    if kind == 'verify':
        names = ('rowptr', 'col', 'val', 'c', 'lower', 'upper')
        state = {k: torch.from_numpy(p[k]).cuda() for k in names}
        state.update(kind=kind, n=case['n'], x=torch.from_numpy(_candidate(p, seed)).cuda())
        state['diag'] = torch.empty_like(state['c'])
        torch.cuda.synchronize()  # the calls run on streams of their own
        return state
    a = _constraints(case, seed)
    system = boxqp.AdmmSystem(p['rowptr'], p['col'], p['val'], a['rowptr'], a['col'], a['val'], case['n'])
    system.set_rho(a['rho'], ADMM_SIGMA)
    return {'kind': kind, 'system': system, 'rhs': a['rhs'], 'x0': np.zeros(case['n']), 'accuracy': _accuracy(a['rhs']),
            'most': min(4000, 2 * case['n'] + 20)}


def _answer(x, st, counted):
    got = {'x': x, 'objective': st.objective, 'status': int(st.status)}
    if counted:  # the FP64 engines keep the reference's iterations
        got['iterations'] = int(st.iterations)
    return got


def _verify(s):
    lib, n = boxqp.lib(), s['n']
    st, flags = boxqp.Stats(), (np.zeros(1), np.zeros(1, np.int32), np.zeros(1, np.int32))
    lipschitz, indefinite, nondominant = flags
    native = boxqp._native
    rc = lib.bqp_gate_device(n, s['rowptr'].data_ptr(), s['col'].data_ptr(), s['val'].data_ptr(), s['diag'].data_ptr(),
                             native.ptr(lipschitz, native.c_double), native.ptr(indefinite, native.c_int32),
                             native.ptr(nondominant, native.c_int32))
    rc |= lib.bqp_check_device(n, s['rowptr'].data_ptr(), s['col'].data_ptr(), s['val'].data_ptr(), s['x'].data_ptr(),
                               s['c'].data_ptr(), s['lower'].data_ptr(), s['upper'].data_ptr(), 1e-6, 0.0, 0, st)
    if rc:
        raise RuntimeError('device verification failed')
    return {'diag': s['diag'], 'lipschitz': lipschitz, 'indefinite': indefinite, 'nondominant': nondominant,
            'objective': st.objective, 'primal_residual': st.primal_residual,
            'stationarity': st.stationarity_residual, 'dual_bound': st.dual_bound, 'gap': st.relative_gap,
            'verified': int(st.verified)}


def run(state):
    kind = state['kind']
    if kind == 'serve':
        futures = [state['server'].submit(*arrays, tolerance=tol) for arrays, tol in state['requests']]
        return [{'x': r.x, 'objective': r.objective} for r in [f.result(timeout=60) for f in futures]]
    if kind == 'batch':
        x, stats = state['solves'].run()
        return {'x': x, 'objective': np.array([st.objective for st in stats]),
                'status': np.array([st.status for st in stats], np.int32)}
    if kind == 'resident':
        x, stats = state['solves'].run()
        return _answer(x, stats[0], state['counted'])
    if kind == 'solve':
        x, st = state['engine'].solve(*state['arrays'], state['options'])
        return _answer(x, st, state['counted'])
    if kind == 'api':
        r = boxqp.solve_accelerated_box(state['problem'], state['options'])
        return {'x': r.primal, 'objective': r.objective, 'iterations': r.iterations, 'verified': r.optimality_verified}
    if kind == 'plugin':
        for beta in state['momenta']:
            state['box'].step(beta)
        return state['box'].primal()
    if kind == 'verify':
        return _verify(state)
    x, inner, _ = state['system'].solve(state['rhs'], state['x0'], state['accuracy'], state['most'])
    return {'x': x, 'inner': inner}


# ------------------------------------------------------------------------------------------
# what one pass cannot do without
# ------------------------------------------------------------------------------------------
def _entries(case):
    n = case['n']
    return {'graph': (2 * case['epv'] + 1) * n, 'grid': 5 * n, 'tridiagonal': 3 * n}[case['family']]


def _products(case):
    """Matrix products of one pass: about the iterations that the method needs on the family."""
    if case['kind'] == 'plugin':
        return STEPS
    if case['kind'] == 'verify':
        return 1
    if case['kind'] == 'admm':
        return 95
    if case['precision'] == 'mixed':
        return {'graph': 22, 'grid': 50, 'tridiagonal': 35}[case['family']]
    return {'graph': 500, 'grid': 225, 'tridiagonal': 1700}[case['family']]


def work(case):
    """Each input read once and the answer written once; two operations per entry and product."""
    if case['kind'] in ('serve', 'batch'):
        lo, hi = case['n_lo'], case['n_hi']
        n = case['count'] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)  # mean of the log-uniform sizes
        nnz = n * (11 if case['kind'] == 'serve' else 9)
        return {'bytes': 12 * nnz + 36 * n, 'flops': 2 * nnz * 30}
    n, nnz = case['n'], _entries(case)
    if case['kind'] == 'admm':
        a = ADMM_ROW * case['rows']
        return {'bytes': 12 * nnz + 12 * a + 12 * case['rows'] + 24 * n, 'flops': (2 * nnz + 4 * a) * _products(case)}
    return {'bytes': 12 * nnz + 36 * n + 4, 'flops': 2 * nnz * _products(case)}


# ------------------------------------------------------------------------------------------
# the answers in 64 bits
# ------------------------------------------------------------------------------------------
def _matrix(p):
    return torch.sparse_csr_tensor(torch.from_numpy(p['rowptr']).long().cuda(), torch.from_numpy(p['col']).long().cuda(),
                                   torch.from_numpy(p['val']).cuda(), (p['rowptr'].shape[0] - 1, p.get('cols', p.get('n'))))


def _plugin_exact(p):
    q = _matrix(p)
    c, lo, up = (torch.from_numpy(p[k]).cuda() for k in ('c', 'lower', 'upper'))
    step = _lipschitz(p)
    x = torch.clamp(torch.zeros_like(c), lo, up)
    w = x
    for beta in _momenta():
        nx = torch.clamp(w - (q @ w + c) / step, lo, up)
        w = nx + beta * (nx - x)
        x = nx
    return _host(x)


def _verify_exact(p, seed):
    x = _candidate(p, seed)
    qx = _times(p, x)
    g = qx + p['c']
    objective = float(0.5 * np.dot(x, qx) + np.dot(p['c'], x))
    moved = np.clip(x - g, p['lower'], p['upper'])
    target = np.where(g > 0, p['lower'], p['upper'])
    bound = objective + float(np.sum(g * (target - x)))
    rows = np.repeat(np.arange(p['n']), np.diff(p['rowptr']))
    return {'diag': p['val'][p['col'] == rows], 'lipschitz': np.array([_lipschitz(p)]), 'indefinite': None,
            'nondominant': None, 'objective': objective, 'primal_residual': 0.0,
            'stationarity': float(np.max(np.abs(x - moved) / (1.0 + np.abs(x)))), 'dual_bound': bound,
            'gap': abs(objective - bound) / (1.0 + abs(objective)), 'verified': None}


def _admm_exact(case, p, seed):
    """K x = rhs by conjugate gradients in 64 bits, run well past the accuracy asked for."""
    a = _constraints(case, seed)
    h = _matrix(p)
    m = _matrix({'rowptr': a['rowptr'], 'col': a['col'], 'val': a['val'], 'cols': case['n']})
    rows = torch.arange(case['rows'], device='cuda').repeat_interleave(ADMM_ROW)
    mt = torch.sparse_coo_tensor(torch.stack([torch.from_numpy(a['col']).long().cuda(), rows]),
                                 torch.from_numpy(a['val']).cuda(), (case['n'], case['rows'])).coalesce().to_sparse_csr()
    rho, b = torch.from_numpy(a['rho']).cuda(), torch.from_numpy(a['rhs']).cuda()
    x, r = torch.zeros_like(b), b
    d, rr = r, torch.dot(r, r)
    for _ in range(4000):
        kd = h @ d + ADMM_SIGMA * d + mt @ (rho * (m @ d))
        alpha = rr / torch.dot(d, kd)
        x = x + alpha * d
        r = r - alpha * kd
        new = torch.dot(r, r)
        d = r + (new / rr) * d
        rr = new
        if float(rr) <= 1e-26 * float(torch.dot(b, b)):
            break
    return {'x': _host(x), 'inner': None}


def exact(case, seed):
    kind = case['kind']
    if kind == 'serve':
        return [{'x': p['x'], 'objective': _objective(p)} for p in _mix(case, seed)]
    if kind == 'batch':
        problems = _mix(case, seed)
        return {'x': np.concatenate([p['x'] for p in problems]),
                'objective': np.array([_objective(p) for p in problems]), 'status': None}
    p = _problem(case['family'], case['n'], case['epv'], seed)
    if kind == 'plugin':
        return _plugin_exact(p)
    if kind == 'verify':
        return _verify_exact(p, seed)
    if kind == 'admm':
        return _admm_exact(case, p, seed)
    return {'x': p['x'], 'objective': _objective(p)}
