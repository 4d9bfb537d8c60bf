"""Performance cases: the work that users of this package have it do.

Each case is one call of a public entry point on a seeded Rydberg lattice:
products H x for a caller's own eigensolver, ground states, pulse ramps and
quenches, Chebyshev moments (density of states, thermodynamics), batches of
small ground states, pulse gradients and fixed-excitation scans, on the full
2^N basis, chain, ring and lattice blockade sectors and fixed-excitation
sectors.  Energies are in cyclic MHz, times in ns, positions in um.

Values that are computed from 32-bit vectors (float32 / complex64 options)
come back in the digits that option has.
"""
import math

import numpy as np
import torch

C6 = 862690.0                  # MHz um^6
CONV = 2.0 * math.pi * 1e-3    # phase per MHz ns
DEV = 'cuda'


def listed():
    return [
        # a block of 8 vectors times H on the 31-site blockaded chain (dim 3.5 M)
        dict(name='apply_chain31_x8', kind='apply', lattice='chain', n=31, dtype='complex64', nvec=8),
        # one product on an unconstrained 21-site chain, for a user's own Krylov code
        dict(name='apply_full21', kind='apply', lattice='full', n=21, dtype='complex128', nvec=1),
        # one product on the blockade sector of a 5 x 6 square lattice (dim 470 k)
        dict(name='apply_grid30', kind='apply', lattice='grid', n=30, rows=5, dtype='float64', nvec=1),
        # ground state and gap of a 4 x 4 lattice on the full basis, with its vector
        dict(name='ground_full16', kind='ground', lattice='full', n=16, rows=4),
        # detuning ramp of the 31-site chain in piecewise-constant steps
        dict(name='ramp_chain31', kind='ramp', lattice='chain', n=31, steps=24, dtype='complex64'),
        # quench of a 4 x 4 lattice on the full basis, site observables at 21 times
        dict(name='quench_full16', kind='quench', lattice='full', n=16, rows=4, times=21, dtype='complex128'),
        # density-of-states moments of the 5 x 5 lattice on the full basis, 32 probes
        dict(name='moments_full25', kind='moments', lattice='full', n=25, rows=5, num=96, nvec=32,
             dtype='float32'),
        # the same for thermodynamics in the blockade sector of a 24-site chain, 64 probes
        dict(name='moments_chain24', kind='moments', lattice='chain', n=24, num=200, nvec=64, dtype='float32'),
        # 512 disordered blockaded chains of 16..22 sites in one go
        dict(name='batch_chain512', kind='batch', count=512, lo=16, hi=22),
        # the smallest solve: one 12-site chain on the full basis, 64 bits
        dict(name='single_full12', kind='single', lattice='full', n=12),
        # gradient of a 200-step pulse on a blockaded ring of 20 sites
        dict(name='gradient_ring20', kind='gradient', n=20, steps=200, dtype='complex64'),
        # every excitation sector of a 16-site dipolar XY chain
        dict(name='scan_xy16', kind='scan', n=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['apply', 'apply', 'ground', 'ramp', 'quench', 'moments', 'moments', 'batch', 'single',
                       'gradient', 'scan'])
    if kind == 'apply':
        lattice = rng.choice(['chain', 'ring', 'full', 'grid'])
        c = dict(kind=kind, lattice=lattice, dtype=rng.choice(['float32', 'float64', 'complex64', 'complex128']),
                 nvec=rng.choice([1, 1, 2, 4, 8, 16]))
        if lattice == 'grid':
            c['rows'] = rng.randint(2, 5)
            c['n'] = c['rows'] * rng.randint(3, 6)
        else:
            c['n'] = rng.randint(9, 22) if lattice == 'full' else rng.randint(12, 31)
        return c
    if kind == 'ground':
        lattice = rng.choice(['chain', 'ring', 'full', 'grid'])
        c = dict(kind=kind, lattice=lattice)
        if lattice == 'grid':
            c['rows'] = rng.randint(3, 5)
            c['n'] = c['rows'] * rng.randint(3, 5)
        else:
            c['n'] = rng.randint(10, 17) if lattice == 'full' else rng.randint(14, 25)
        return c
    if kind == 'ramp':
        return dict(kind=kind, lattice=rng.choice(['chain', 'chain', 'ring']), n=rng.randint(15, 30),
                    steps=rng.randint(5, 24), dtype=rng.choice(['complex64', 'complex128']))
    if kind == 'quench':
        n = rng.randint(8, 16)
        return dict(kind=kind, lattice='full', n=n, rows=rng.choice([r for r in (1, 2, 3, 4) if n % r == 0]),
                    times=rng.randint(5, 21), dtype=rng.choice(['complex64', 'complex128']))
    if kind == 'moments':
        lattice = rng.choice(['full', 'chain', 'ring'])
        n = rng.randint(9, 22) if lattice == 'full' else rng.randint(14, 25)
        return dict(kind=kind, lattice=lattice, n=n, num=_log_int(rng, 40, 300), nvec=rng.randint(8, 64),
                    dtype=rng.choice(['float32', 'float32', 'float64']))
    if kind == 'batch':
        lo = rng.randint(8, 18)
        return dict(kind=kind, count=_log_int(rng, 12, 512), lo=lo, hi=rng.randint(lo, 21))
    if kind == 'single':
        lattice = rng.choice(['full', 'chain', 'ring'])
        return dict(kind=kind, lattice=lattice, n=rng.randint(7, 12) if lattice == 'full' else rng.randint(9, 17))
    if kind == 'gradient':
        return dict(kind=kind, n=rng.randint(11, 21), steps=_log_int(rng, 20, 200),
                    dtype=rng.choice(['complex64', 'complex64', 'complex128']))
    return dict(kind=kind, n=rng.randint(9, 16))


# ------------------------------------------------------------------- inputs

def _positions(case, rng):
    """Sites of the case's lattice, each a little off its place."""
    n, lat = case['n'], case.get('lattice', 'chain')
    if lat == 'ring':
        t = 2.0 * np.pi * np.arange(n) / n
        p = 5.5 / (2.0 * np.sin(np.pi / n)) * np.stack([np.cos(t), np.sin(t)], 1)
    elif case.get('rows', 1) > 1:
        cols = n // case['rows']
        p = 6.0 * np.array([[i // cols, i % cols] for i in range(n)], float)
    else:
        p = np.stack([5.5 * np.arange(n), np.zeros(n)], 1)
    return p + rng.uniform(-0.1, 0.1, p.shape)


def _edges(case):
    """Nearest-neighbour blockade of the lattice; None on the full basis."""
    n, lat = case['n'], case.get('lattice', 'chain')
    if lat == 'full':
        return None
    if lat == 'grid':
        cols = n // case['rows']
        return ([[i, i + 1] for i in range(n) if (i + 1) % cols] + [[i, i + cols] for i in range(n - cols)])
    return [[i, i + 1] for i in range(n - 1)] + ([[n - 1, 0]] if lat == 'ring' else [])


def _lattice(case, seed):
    """Positions, drive and detunings of one lattice: plain arrays."""
    rng = np.random.default_rng([17, int(seed)])
    pos = _positions(case, rng)
    n = case['n']
    return dict(n=n, pos=pos, edges=_edges(case), Om=np.full(n, rng.uniform(1.5, 2.5)),
                delta=-rng.uniform(-3.0, 3.0, n))


def _pairs(pos):
    i, j = np.triu_indices(len(pos), 1)
    return i, j, C6 / np.linalg.norm(pos[i] - pos[j], axis=1) ** 6


def _calib(pos):
    return dict(atoms=[dict(id=q, pos=[float(p[0]), float(p[1]), 0.0]) for q, p in enumerate(pos)],
                pairs=[dict(i=int(i), j=int(j), V=float(v), J=0.0, A=0.0) for i, j, v in zip(*_pairs(pos))])


def _plan(edges):
    return None if edges is None else dict(projected=True, blockade_edges=edges, constraint=dict(kind='blockade'))


def _vectors(dim, case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    shape = (dim,) if case['nvec'] == 1 else (dim, case['nvec'])
    return torch.randn(shape, generator=g, device=DEV, dtype=getattr(torch, case['dtype']))


def _ramp(case, seed):
    """(lattice, segments): a detuning sweep -6 .. +6 MHz at Omega about 2 MHz, 10 ns a step."""
    L = _lattice(case, seed)
    n, steps = L['n'], case['steps']
    s = (np.arange(steps) + 0.5) / steps
    seg = [dict(t0=10.0 * k, Om=L['Om'], delta=np.full(n, 6.0 - 12.0 * s[k]) + 0.1 * L['delta']) for k in range(steps)]
    return L, seg


def _pulse(case, seed):
    """(lattice, tau, Omega_k, Delta_k): a smooth pulse in 10 ns steps, Delta from -6 to +6 MHz."""
    L = _lattice(dict(case, lattice='ring'), seed)
    rng = np.random.default_rng([29, int(seed)])
    K = case['steps']
    s = (np.arange(K) + 0.5) / K
    om, de = np.full(K, 2.0), -6.0 + 12.0 * s
    for q in range(1, 5):
        om += rng.uniform(-0.3, 0.3) * np.sin(np.pi * q * s + rng.uniform(0, 2 * np.pi))
        de += rng.uniform(-0.5, 0.5) * np.sin(np.pi * q * s + rng.uniform(0, 2 * np.pi))
    return L, np.full(K, 10.0), om, de


def _batch(case, seed):
    rng = np.random.default_rng([41, int(seed)])
    out = []
    for q in range(case['count']):
        n = int(rng.integers(case['lo'], case['hi'] + 1))
        pos = np.stack([5.5 * np.arange(n) + rng.uniform(-0.3, 0.3, n), np.zeros(n)], 1)
        out.append(dict(n=n, pos=pos, edges=[[i, i + 1] for i in range(n - 1)], Om=np.full(n, 2.0),
                        delta=np.full(n, -2.0 * rng.uniform(0.0, 3.0))))
    return out


def _xy(case, seed):
    """Dipolar XY chain: J_ij on every pair, a weak V, random detunings."""
    rng = np.random.default_rng([53, int(seed)])
    n = case['n']
    pos = np.stack([5.5 * np.arange(n) + rng.uniform(-0.1, 0.1, n), np.zeros(n)], 1)
    i, j, v = _pairs(pos)
    return dict(n=n, pos=pos, i=i, j=j, V=1e-3 * v, J=-0.7 * (5.5 / np.abs(pos[i, 0] - pos[j, 0])) ** 3,
                delta=rng.uniform(-1.0, 1.0, n))


def prepare(case, seed):
    from energy_level_b200 import adjoint, batched, model, sector_scan
    kind = case['kind']
    if kind == 'batch':
        return dict(case=case, batch=batched.BatchedGroundStates(
            [dict(calib=_calib(b['pos']), Om=b['Om'], delta=b['delta'], edges=b['edges'])
             for b in _batch(case, seed)], dtype='float32'))
    if kind == 'scan':
        X = _xy(case, seed)
        calib = _calib(X['pos'])
        for p, v, jj in zip(calib['pairs'], X['V'], X['J']):
            p.update(V=float(v), J=float(jj))
        return dict(case=case, scan=sector_scan.SectorScan(calib, X['delta'], terms=['I1', 'I2']))
    if kind == 'gradient':
        L, tau, om, de = _pulse(case, seed)
        n = L['n']
        prob = adjoint.PulseProblem(_calib(L['pos']), 'g' * n, target='rg' * (n // 2) + 'g' * (n % 2),
                                    plan=_plan(L['edges']), dtype=case['dtype'])
        return dict(case=case, problem=prob, pulse=(tau, om, de))
    if kind == 'ramp':
        L, seg = _ramp(case, seed)
        return dict(case=case, calib=_calib(L['pos']), plan=_plan(L['edges']), segments=seg,
                    t=np.array([0.0, 10.0 * case['steps']]))
    L = _lattice(case, seed)
    state = dict(case=case, calib=_calib(L['pos']), plan=_plan(L['edges']), Om=L['Om'], delta=L['delta'], seed=seed)
    if kind == 'apply':
        ctx, basis, ham, _ = model.build(state['calib'], L['Om'], L['delta'], plan=state['plan'])
        state.update(basis=basis, ham=ham, x=_vectors(basis.dim, case, seed))
    elif kind == 'single':
        state['instances'] = [dict(calib=state['calib'], Om=L['Om'], delta=L['delta'], edges=L['edges'])]
    return state


# --------------------------------------------------------------------- runs

def _digits(dtype, v):
    """Values in the digits of the vectors they were computed from."""
    v = np.asarray(v)
    if dtype in ('float32', 'complex64'):
        return v.astype(np.complex64 if v.dtype.kind == 'c' else np.float32)
    return v


def run(s):
    from energy_level_b200 import batched, engine, kpm, matrix_free
    c = s['case']
    kind = c['kind']
    if kind == 'apply':
        return s['ham'].hv(s['x'])
    if kind == 'ground':
        r = matrix_free.b200_lanczos_ground_state(s['calib'], s['Om'], s['delta'], plan=s['plan'], tol=1e-11,
                                                  return_state=True)
        return dict(E0=r['E0'], gap=r['gap'], vec=r['vec'].real)
    if kind in ('ramp', 'quench'):
        if kind == 'ramp':
            r = engine.evolve_manybody(s['calib'], 'g' * c['n'], s['t'], plan=s['plan'], segments=s['segments'],
                                       dtype=c['dtype'], want_entropy=False, record_psi=True)
        else:
            r = engine.evolve_manybody(s['calib'], 'g' * c['n'], np.linspace(0.0, 50.0 * (c['times'] - 1), c['times']),
                                       Om=s['Om'], delta=s['delta'], dtype=c['dtype'], want_entropy=False,
                                       record_psi=True)
        return dict({k: _digits(c['dtype'], r[k]) for k in ('pops_atom', 'norms', 'corr', 'psi_amp')},
                    sm=_digits(c['dtype'], r['observables']['sm']),
                    xy=_digits(c['dtype'], r['observables']['xy_corr']))
    if kind == 'moments':
        mu, cen, rad = kpm.kpm_moments_b200(dict(calib=s['calib'], Om=s['Om'], delta=s['delta'], plan=s['plan']),
                                            num=c['num'], nvec=c['nvec'], seed=s['seed'], dtype=c['dtype'])
        return dict(mu=_digits(c['dtype'], mu), c=cen, r=rad)
    if kind == 'batch':
        s['batch'].run()
        r = s['batch'].results()
        return dict(E0=_digits('float32', r['E0']), gap=_digits('float32', r['gap']))
    if kind == 'single':
        r = batched.batched_ground_states(s['instances'], dtype='float64', tol=1e-11)
        return {k: r[k] for k in ('E0', 'gap', 'n_atom')}
    if kind == 'gradient':
        F, go, gd = s['problem'].evaluate(*s['pulse'])
        return dict(F=_digits(c['dtype'], F), go=_digits(c['dtype'], go), gd=_digits(c['dtype'], gd))
    rows = s['scan'].run()
    return dict(E0=np.array([r['E0'] for r in rows]), gap=np.array([r['gap'] for r in rows]))


# --------------------------------------------------------------------- work

def _dim(case):
    n, lat = case['n'], case.get('lattice', 'chain')
    if case['kind'] == 'gradient':
        lat = 'ring'
    if lat == 'full' or case['kind'] == 'scan':
        return 1 << n
    if lat == 'grid':
        return len(_codes(n, _edges(case)))
    f = [0, 1]
    while len(f) < n + 3:
        f.append(f[-1] + f[-2])
    return f[n + 2] if lat == 'chain' else f[n + 1] + f[n - 1]


def _size(dtype):
    return {'float32': 4, 'float64': 8, 'complex64': 8, 'complex128': 16}[dtype]


def work(case):
    """What a pass cannot do without.  A product reads its block and writes
    the result; a Krylov or Chebyshev solve does that once for each of its
    steps, with the recurrence's third vector; about 0.7 n flips a row in a
    blockade sector, n on the full basis, one multiply-add each (two for
    complex vectors).  Step counts are those of typical inputs."""
    kind = case['kind']
    if kind == 'batch':
        nbar = 0.5 * (case['lo'] + case['hi'])
        rows = case['count'] * np.mean([1.17 * 1.618 ** q for q in range(case['lo'], case['hi'] + 1)])
        return dict(bytes=90 * rows * 4 * 3, flops=90 * rows * (1.4 * nbar + 8))
    dim, n = _dim(case), case['n']
    es = _size(case.get('dtype', 'float64'))
    flips = (n if case.get('lattice') == 'full' else 0.72 * n) * (4 if es == 16 or case.get('dtype') == 'complex64' else 2)
    if kind == 'apply':
        return dict(bytes=2.0 * dim * case['nvec'] * es, flops=dim * case['nvec'] * flips)
    steps = {'ground': 150, 'single': 150, 'scan': 90, 'ramp': 18 * case.get('steps', 0),
             'quench': 90 * (case.get('times', 1) - 1), 'gradient': 25 * case.get('steps', 0),
             'moments': 0.5 * case.get('num', 0) * case.get('nvec', 0)}[kind]
    if kind == 'scan':
        flips = 0.5 * n * n
    return dict(bytes=3.0 * steps * dim * es, flops=steps * dim * (flips + 6))


# ---------------------------------------------------- the same in 64 bits

def _codes(n, edges):
    """Ascending codes of the independent sets (site 0 = top bit); all codes without edges."""
    adj = [0] * n
    for a, b in edges or []:
        adj[n - 1 - a] |= 1 << (n - 1 - b)
        adj[n - 1 - b] |= 1 << (n - 1 - a)
    c = np.zeros(1, np.int64)
    for k in range(n):
        c = np.concatenate([c, c[(c & adj[k]) == 0] | (1 << k)])
    return c


class _H:
    """H in 64 bits: diagonal and, for each bit, the rows its flip leads to
    (on the full basis the flip is a reversal of one axis)."""

    def __init__(self, L, full):
        n = self.n = L['n']
        self.om = 0.5 * np.asarray(L['Om'])[::-1]
        self.full = full
        codes = None if full else torch.as_tensor(_codes(n, L['edges']), device=DEV)
        self.codes = torch.arange(1 << n, device=DEV) if full else codes
        self.dim = len(self.codes)
        self.occ = lambda q: ((self.codes >> (n - 1 - q)) & 1).double()
        self.V = torch.zeros(self.dim, dtype=torch.float64, device=DEV)
        for i, j, v in zip(*_pairs(L['pos'])):
            self.V += v * self.occ(int(i)) * self.occ(int(j))
        self.set(L['Om'], L['delta'])
        if not full:
            t = []
            for k in range(n):
                w = self.codes ^ (1 << k)
                p = torch.searchsorted(self.codes, w).clamp_(max=self.dim - 1)
                t.append(torch.where(self.codes[p] == w, p, self.dim).to(torch.int32))
            self.t = t

    def set(self, Om, delta):
        self.om = 0.5 * np.asarray(Om, float)[::-1]
        self.D = self.V.clone()
        for q in range(self.n):
            self.D += float(delta[q]) * self.occ(q)

    def flips(self, x, amp=None):
        amp = self.om if amp is None else amp
        y = torch.zeros_like(x)
        if self.full:
            for k in range(self.n):
                v = x.reshape((1 << (self.n - 1 - k), 2, -1))
                o = y.view(v.shape)
                o[:, 0].add_(v[:, 1], alpha=float(amp[k]))
                o[:, 1].add_(v[:, 0], alpha=float(amp[k]))
            return y
        z = torch.cat([x, torch.zeros_like(x[:1])])
        for k in range(self.n):
            y.add_(z[self.t[k]], alpha=float(amp[k]))
        return y

    def __call__(self, x):
        return self.flips(x).add_((self.D if x.dim() == 1 else self.D[:, None]) * x)

    def expm(self, x, tau):
        """exp(-i CONV H tau) x by a Taylor series about the middle of the diagonal."""
        mid = 0.5 * float(self.D.max() + self.D.min())
        b = CONV * abs(tau) * (0.5 * float(self.D.max() - self.D.min()) + float(np.abs(self.om).sum()))
        parts = max(1, math.ceil(b / 4.0))
        for _ in range(parts):
            u, acc = x, x.clone()
            for m in range(1, 200):
                u = (self(u) - mid * u) * (-1j * CONV * tau / parts / m)
                acc += u
                if m % 4 == 0 and float(u.abs().max()) < 1e-17:
                    break
            x = acc * np.exp(-1j * CONV * tau / parts * mid)
        return x


def _lanczos(h, dim, steps, count=1):
    """alpha, beta [count, k] and basis of a Lanczos with full reorthogonalisation."""
    g = torch.Generator(device=DEV)
    g.manual_seed(1)
    steps = min(steps, dim)
    Q = torch.empty((count, steps, dim), dtype=torch.float64, device=DEV)
    a = torch.zeros((count, steps), dtype=torch.float64, device=DEV)
    b = torch.zeros((count, steps), dtype=torch.float64, device=DEV)
    v = torch.randn((count, dim), generator=g, device=DEV, dtype=torch.float64)
    Q[:, 0] = v / v.norm(dim=1, keepdim=True)
    for j in range(steps):
        w = h(Q[:, j])
        a[:, j] = (w * Q[:, j]).sum(1)
        for _ in range(2):
            B = Q[:, :j + 1]
            w = w - torch.bmm(torch.bmm(B, w[:, :, None]).transpose(1, 2), B)[:, 0]
        b[:, j] = w.norm(dim=1)
        if j + 1 < steps:
            Q[:, j + 1] = w / b[:, j:j + 1].clamp_min(1e-300)
    return a, b, Q


def _ritz(a, b):
    T = torch.diag_embed(a) + torch.diag_embed(b[:, :-1], 1) + torch.diag_embed(b[:, :-1], -1)
    return torch.linalg.eigh(T)


def _two_lowest(h, dim, steps):
    a, b, Q = _lanczos(lambda x: h(x[0])[None], dim, steps)
    e, y = _ritz(a, b)
    x = (y[0, :, 0][None] @ Q[0])[0]
    return float(e[0, 0]), float(e[0, 1] - e[0, 0]) if e.shape[1] > 1 else 0.0, x / x.norm()


def _extremes(h, dim, steps=400):
    """Lowest and highest eigenvalue, by a plain three-term Lanczos on large bases."""
    if dim * steps * 8 < 8e9:
        a, b, _ = _lanczos(lambda x: h(x[0])[None], dim, steps)
        e, _ = _ritz(a, b)
        return float(e[0, 0]), float(e[0, -1])
    g = torch.Generator(device=DEV)
    g.manual_seed(1)
    v = torch.randn(dim, generator=g, device=DEV, dtype=torch.float64)
    v /= v.norm()
    p, be, al, bs = torch.zeros_like(v), 0.0, [], []
    for _ in range(steps):
        w = h(v) - be * p
        al.append(float(w @ v))
        w -= al[-1] * v
        be = float(w.norm())
        bs.append(be)
        p, v = v, w / be
    e = np.linalg.eigvalsh(np.diag(al) + np.diag(bs[:-1], 1) + np.diag(bs[:-1], -1))
    return float(e[0]), float(e[-1])


def _signs(seed, probe, dim):
    """The counter-based +-1 probes: top bit of splitmix64(key(probe) + row)."""
    def lsr(x, k):
        return (x >> k) & ((1 << (64 - k)) - 1)

    def signed(v):
        v &= (1 << 64) - 1
        return v - (1 << 64) if v >> 63 else v

    def mix(x):
        x = x + signed(0x9E3779B97F4A7C15)
        x = (x ^ lsr(x, 30)) * signed(0xBF58476D1CE4E5B9)
        x = (x ^ lsr(x, 27)) * signed(0x94D049BB133111EB)
        return x ^ lsr(x, 31)

    key = torch.tensor([signed(seed ^ ((probe + 1) * 0xD1B54A32D192ED03))], dtype=torch.int64, device=DEV)
    return torch.where(mix(mix(key) + torch.arange(dim, device=DEV)) < 0, -1.0, 1.0).double()


def _site_values(h, x):
    """n_i, sigma^-_i, <n_i n_j> - <n_i><n_j> and <sigma+_i sigma-_j> of a state."""
    n = h.n
    z = torch.cat([x, torch.zeros_like(x[:1])])
    p = x.abs().square()
    occ = torch.stack([h.occ(q) for q in range(n)])
    ni = occ @ p
    # s_q: sigma^-_q x, site q from r to g
    low = []
    for q in range(n):
        k = n - 1 - q
        src = (h.codes ^ (1 << k)) if h.full else h.t[k].long()
        low.append(torch.where(occ[q] == 0, z[src], torch.zeros_like(x)))
    sm = torch.stack([torch.vdot(x, s) for s in low])
    S = torch.stack(low)
    # <sigma+_i sigma-_j> = <sigma-_i x, sigma-_j x>
    xy = S.conj() @ S.T
    nn = (occ * p) @ occ.T
    corr = nn - torch.outer(ni, ni)
    xy = xy - torch.diag(torch.diag(xy)) + torch.diag(ni.to(xy.dtype))
    return ni, sm, corr, xy


def _exact_evolution(case, seed):
    if case['kind'] == 'ramp':
        L, seg = _ramp(case, seed)
        h = _H(L, False)
        x = torch.zeros(h.dim, dtype=torch.complex128, device=DEV)
        x[0] = 1.0
        states = [x]
        for s in seg:
            h.set(s['Om'], s['delta'])
            x = h.expm(x, 10.0)
        states.append(x)
    else:
        L = _lattice(case, seed)
        h = _H(L, True)
        x = torch.zeros(h.dim, dtype=torch.complex128, device=DEV)
        x[0] = 1.0
        states = [x]
        for _ in range(case['times'] - 1):
            x = h.expm(x, 50.0)
            states.append(x)
    vals = [_site_values(h, v) for v in states]
    return dict(pops_atom=torch.stack([v[0] for v in vals]), norms=torch.stack([v.abs().square().sum() for v in states]),
                corr=vals[-1][2], psi_amp=x, sm=torch.stack([v[1] for v in vals]), xy=vals[-1][3])


def _exact_moments(case, seed):
    L = _lattice(case, seed)
    h = _H(L, case['lattice'] == 'full')
    lo, hi = _extremes(h, h.dim)
    c, r = 0.5 * (lo + hi), 0.5 * (hi - lo) * (1.0 + 1e-3) + 1e-12
    mu = np.zeros(case['num'] + 1)
    for p in range(case['nvec']):
        z = _signs(seed, p, h.dim)
        a, b = z, (h(z) - c * z) / r
        mu[0] += float(a @ a)
        mu[1] += float(a @ b)
        m0, m1 = float(a @ a), float(a @ b)
        for m in range(1, case['num'] // 2 + 1):
            mu[2 * m] += 2.0 * float(b @ b) - m0
            a, b = b, (h(b) - c * b).mul_(2.0 / r).sub_(a)
            if 2 * m + 1 <= case['num']:
                mu[2 * m + 1] += 2.0 * float(a @ b) - m1
    return dict(mu=mu / (case['nvec'] * h.dim), c=c, r=r)


def _exact_batch(case, seed):
    items = _batch(case, seed)
    E0, gap = np.zeros(len(items)), np.zeros(len(items))
    for n in sorted({b['n'] for b in items}):
        ids = [q for q, b in enumerate(items) if b['n'] == n]
        h = _H(items[ids[0]], False)
        occ = torch.stack([h.occ(q) for q in range(n)])
        D = []
        for q in ids:
            W = torch.zeros((n, n), dtype=torch.float64, device=DEV)
            i, j, v = _pairs(items[q]['pos'])
            W[torch.as_tensor(i, device=DEV), torch.as_tensor(j, device=DEV)] = torch.as_tensor(v, device=DEV)
            D.append(((W @ occ) * occ).sum(0) + torch.as_tensor(items[q]['delta'], device=DEV) @ occ)
        D = torch.stack(D)
        for lo in range(0, len(ids), 96):
            d = D[lo:lo + 96]
            a, b, _ = _lanczos(lambda x: h.flips(x.T.contiguous()).T + d * x, h.dim, 160, count=len(d))
            e = _ritz(a, b)[0].cpu().numpy()
            E0[ids[lo:lo + 96]] = e[:, 0]
            gap[ids[lo:lo + 96]] = e[:, 1] - e[:, 0]
    return dict(E0=E0, gap=gap)


def _exact_gradient(case, seed):
    """F and its gradient: dU_k = -i CONV int U(tau - s) G U(s) ds by Gauss-Legendre nodes."""
    L, tau, om, de = _pulse(case, seed)
    n, K = L['n'], case['steps']
    h = _H(L, False)
    ones = np.ones(n)
    nocc = sum(h.occ(q) for q in range(n))
    x = torch.zeros(h.dim, dtype=torch.complex128, device=DEV)
    x[0] = 1.0
    want = sum(1 << (n - 1 - q) for q in range(0, 2 * (n // 2), 2))
    target = torch.zeros_like(x)
    target[int(torch.searchsorted(h.codes, torch.tensor(want, device=DEV)))] = 1.0
    psi = [x]
    for k in range(K):
        h.set(om[k] * ones, -de[k] * ones)
        psi.append(h.expm(psi[-1], tau[k]))
    ov = torch.vdot(target, psi[-1])
    nodes, wts = np.polynomial.legendre.leggauss(14)
    go, gd = np.zeros(K), np.zeros(K)
    chi = target * ov     # F = |<target|psi>|^2, dF = 2 Re <chi|dpsi>
    for k in range(K - 1, -1, -1):
        h.set(om[k] * ones, -de[k] * ones)
        s = 0.5 * tau[k] * (nodes + 1.0)
        back = h.expm(chi, -tau[k])
        pair, t = torch.stack([psi[k], back], 1), 0.0
        for w, sq in zip(0.5 * tau[k] * wts, s):
            pair, t = h.expm(pair, sq - t), sq
            p, q = pair[:, 0], pair[:, 1]
            go[k] += w * 2.0 * float((-1j * CONV * torch.vdot(q, h.flips(p.contiguous(), 0.5 * ones))).real)
            gd[k] += w * 2.0 * float((1j * CONV * torch.vdot(q, nocc * p)).real)
        chi = back
    return dict(F=float(ov.abs() ** 2), go=go, gd=gd)


def _exact_scan(case, seed):
    X = _xy(case, seed)
    n = X['n']
    every = torch.arange(1 << n, device=DEV)
    pop = sum((every >> k) & 1 for k in range(n))
    E0, gap = [], []
    for k in range(n + 1):
        codes = every[pop == k]
        dim = len(codes)
        bit = lambda q: (codes >> (n - 1 - int(q))) & 1
        D = sum(float(X['delta'][q]) * bit(q).double() for q in range(n))
        row = []
        for i, j, v, jj in zip(X['i'], X['j'], X['V'], X['J']):
            D = D + float(v) * (bit(i) * bit(j)).double()
            m = (1 << (n - 1 - int(i))) | (1 << (n - 1 - int(j)))
            src = torch.searchsorted(codes, codes ^ m).clamp_(max=dim - 1)
            row.append((src, (bit(i) != bit(j)).double() * float(jj)))
        S, A = torch.stack([r[0] for r in row]), torch.stack([r[1] for r in row])
        h = lambda x: D * x + (A * x[S]).sum(0)
        if dim <= 600:
            M = torch.diag(D)
            M.index_put_((torch.arange(dim, device=DEV).expand_as(S), S), A, accumulate=True)
            e = torch.linalg.eigvalsh(M)
            E0.append(float(e[0]))
            gap.append(float(e[1] - e[0]) if dim > 1 else 0.0)
        else:
            e, g, _ = _two_lowest(h, dim, 300)
            E0.append(e)
            gap.append(g)
    return dict(E0=np.array(E0), gap=np.array(gap))


def exact(case, seed):
    kind = case['kind']
    if kind in ('ramp', 'quench'):
        return _exact_evolution(case, seed)
    if kind == 'moments':
        return _exact_moments(case, seed)
    if kind == 'batch':
        return _exact_batch(case, seed)
    if kind == 'gradient':
        return _exact_gradient(case, seed)
    if kind == 'scan':
        return _exact_scan(case, seed)
    L = _lattice(case, seed)
    h = _H(L, case['lattice'] == 'full')
    if kind == 'apply':
        x = _vectors(h.dim, case, seed)
        return h(x.to(torch.complex128 if x.is_complex() else torch.float64))
    e, g, x = _two_lowest(h, h.dim, 320)
    if kind == 'ground':
        return dict(E0=e, gap=g, vec=None)
    return dict(E0=np.array([e]), gap=np.array([g]),
                n_atom=torch.stack([h.occ(q) @ x.square() for q in range(h.n)])[None])
