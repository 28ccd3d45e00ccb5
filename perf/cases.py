"""The work that a user of this library has it do, as timed cases.

Every case goes through a public entry point (``intception_b200.eri``, ``.jk``,
``.twoidx``) on synthetic inputs with the shapes and distributions of the
repository's own configurations: random contracted shells, jittered lattices
and primitive pairs.  ``exact`` evaluates the same integrals by the
McMurchie-Davidson scheme in torch float64, with none of the library's code.  The angular momenta,
contraction lengths and quartet lists of a case are the same for every seed;
the seed makes its exponents, coefficients, centres and densities.
"""
import functools
import math

import numpy as np
import torch

from intception_b200 import basis, eri, jk, twoidx

DEV = torch.device('cuda')
SCREEN = 1e-12     # quartets whose bound is smaller are written as zeros
PRIM_TOL = 1e-18   # primitive quartets whose bound is smaller are skipped
EXACT_WORK = 6e10  # Hermite contraction products that exact() takes on at most


# ------------------------------------------------------------------ cases
def _case(kind, **kw):
    """A random-shell case: l in 0..lmax and K in 1..kmax per shell unless fixed."""
    c = dict(kind=kind, nq=1, lmax=2, fixed_l=-1, kmin=1, kmax=6, alpha_lo=0.05, alpha_hi=1e4, box=30.0,
             spherical=True)
    c.update(kw)
    return c


def listed():
    return [
        # one call of the emitted function's drop-in from a host program that
        # loops over shell quartets: (pp|pp), K = 3, Cartesian
        dict(_case('dropin', kmin=3, kmax=3, alpha_lo=0.1, alpha_hi=100.0, box=10.0, spherical=False), la=1, lb=1,
             lc=1, ld=1, ncont=1, name='dropin_pppp'),
        # a few hundred quartets of a small molecule: launches and latency
        dict(_case('batch', nq=256, kmax=3, alpha_lo=0.1, alpha_hi=50.0, box=5.0), name='batch_256'),
        # one class, one contraction length: the plain (pp|pp) configuration
        dict(_case('batch', nq=4096, fixed_l=1, kmin=3, kmax=3, alpha_lo=0.1, alpha_hi=100.0, box=10.0,
                   spherical=False), name='pppp_4096'),
        # the uneven l <= 2 batch, every quartet in FP64 (the drop-ins' semantics)
        dict(_case('batch', nq=1000000), name='l2_fp64'),
        # the same batch as a program with screening runs it: bounds on the
        # device in the step, zero blocks, primitive screening
        dict(_case('screened', nq=1000000), name='l2_screened'),
        # the same screened work on batches that live in host memory
        dict(_case('host', nq=100000), batches=4, name='l2_host_pipeline'),
        # a basis whose shells many quartets share: the 200-atom l <= 3
        # lattice, Schwarz bounds, the mixed-precision tier
        dict(kind='lattice', natom=200, nq=1000000, mixed=True, name='lattice_l3'),
        # high angular momentum, long contractions, a wide exponent range
        dict(_case('batch', nq=6000, lmax=4, kmax=8, alpha_lo=0.02, alpha_hi=1e5, box=10.0), kept=True,
             name='l4_fp64'),
        # J and K energies of a density, and with their nuclear gradient (autograd)
        dict(kind='energy', natom=27, name='jk_energy'),
        dict(kind='forces', natom=20, name='jk_forces'),
        # one-electron matrices over primitive pairs
        dict(kind='overlap', n=4000000, lmax=2, name='overlap_2idx'),
        dict(kind='nuclear', n=4000000, lmax=2, name='nuclear_2idx'),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['dropin', 'batch', 'batch', 'screened', 'host', 'lattice', 'l4', 'energy', 'forces', 'overlap',
                       'nuclear'])
    if kind == 'dropin':
        ls = [rng.choice([0, 1, 1, 2, 2, 3]) for _ in range(4)]
        k = rng.randint(1, 6)
        return dict(_case('dropin', kmin=k, kmax=k, alpha_lo=0.1, alpha_hi=100.0, box=rng.choice([5.0, 10.0]),
                          spherical=rng.random() < 0.5),
                    la=ls[0], lb=ls[1], lc=ls[2], ld=ls[3], ncont=rng.choice([1, 1, 2]))
    if kind in ('batch', 'screened'):
        return _case(kind, nq=_size(rng, 100, 600000), lmax=rng.choice([1, 2, 2, 2]), kmax=rng.randint(1, 6),
                     alpha_lo=rng.choice([0.05, 0.1]), alpha_hi=rng.choice([100.0, 1e4]),
                     box=rng.choice([5.0, 10.0, 30.0]) if kind == 'batch' else 30.0, spherical=rng.random() < 0.7)
    if kind == 'host':
        return dict(_case('host', nq=_size(rng, 1000, 100000), kmax=rng.randint(2, 6)), batches=rng.randint(2, 4))
    if kind == 'lattice':
        return dict(kind='lattice', natom=rng.randint(30, 200), nq=_size(rng, 5000, 1000000),
                    mixed=rng.random() < 0.5)
    if kind == 'l4':
        return dict(_case('batch', nq=_size(rng, 50, 6000), lmax=rng.choice([3, 4, 4]), kmax=rng.randint(3, 8),
                          alpha_lo=0.02, alpha_hi=1e5, box=10.0, spherical=rng.random() < 0.7), kept=True)
    if kind == 'energy':
        return dict(kind='energy', natom=rng.randint(4, 27))
    if kind == 'forces':
        return dict(kind='forces', natom=rng.randint(3, 18))
    return dict(kind=kind, n=_size(rng, 1000, 4000000), lmax=rng.choice([1, 2, 2, 3]))


# ------------------------------------------------------------------ inputs
def _random_shells(g, ls, ks, lo, hi, box, dev):
    """Shell table over ls, ks: exponents log-uniform in [lo, hi], coefficients
    uniform [0.1, 1] then normalised, centres uniform in a cube."""
    n, K = ls.numel(), int(ks.max())
    u = lambda *s: torch.rand(*s, dtype=torch.float64, device=dev, generator=g)  # noqa: E731
    on = torch.arange(K, device=dev)[None, :] < ks[:, None]
    e = torch.exp(math.log(lo) + (math.log(hi) - math.log(lo)) * u(n, K))
    c = (0.1 + 0.9 * u(n, K)) * on
    xyz = box * u(n, 3)
    p = (ls + 1.5)[:, None]
    s = torch.zeros(n, dtype=torch.float64, device=dev)
    for i in range(K):
        s += (c[:, i:i + 1] * c * (2.0 * torch.sqrt(e[:, i:i + 1] * e) / (e[:, i:i + 1] + e)) ** p).sum(1)
    dfact = torch.tensor([float(np.prod(np.arange(2 * l - 1, 0, -2))) for l in range(8)], dtype=torch.float64,
                         device=dev)
    c = c / torch.sqrt(s)[:, None] * (2.0 * e / math.pi) ** 0.75 * (4.0 * e) ** (0.5 * ls[:, None])
    c = c / torch.sqrt(dfact[ls])[:, None]
    ptr = torch.cumsum(ks, 0) - ks
    h = lambda t, d: t.cpu().numpy().astype(d)  # noqa: E731
    return h(ls, np.int32), h(ks, np.int32), h(ptr, np.int32), h(xyz, np.float64), h(e[on], np.float64), \
        h(c[on], np.float64)


def _random_batch(case, seed, nq, dev=DEV, versions=1):
    """nq quartets over four fresh shells each (versions: so many times the same
    angular momenta and contraction lengths, one after the other)."""
    g = torch.Generator(device=dev)
    g.manual_seed(7)
    n = 4 * nq
    ls = torch.randint(0, case['lmax'] + 1, (n,), device=dev, generator=g)
    if case['fixed_l'] >= 0:
        ls.fill_(case['fixed_l'])
    ks = torch.randint(case['kmin'], case['kmax'] + 1, (n,), device=dev, generator=g)
    ls, ks = ls.repeat(versions), ks.repeat(versions)
    nq, n = nq * versions, n * versions
    g.manual_seed(seed)
    sh = _random_shells(g, ls, ks, case['alpha_lo'], case['alpha_hi'], case['box'], dev)
    quartets = np.arange(n, dtype=np.int32).reshape(nq, 4)
    off, total = basis.packed_offsets(sh[0], quartets, case['spherical'])
    return basis.ShellBatch(*sh, quartets, off, case['spherical'], total)


def _kept_batch(case, seed):
    """nq quartets, each the first of eight versions whose analytic bound passes the screen."""
    cand = _random_batch(case, seed, case['nq'], versions=8)
    keep = eri.EriEngine(cand).analytic_bounds().cpu().numpy().reshape(8, -1) >= SCREEN
    return cand.subset(keep.argmax(0) * case['nq'] + np.arange(case['nq']))


def _lattice_schwarz(shells):
    a, b = np.tril_indices(len(shells[0]))
    pairs = np.stack([a, b], axis=1).astype(np.int32)
    one = basis.ShellBatch(*shells, np.zeros((1, 4), np.int32), np.zeros(1, np.int64), True, 1)
    return pairs, eri.EriEngine(one).schwarz(torch.from_numpy(pairs).to(DEV)).cpu().numpy()


def _lattice(case, seed):
    """The jittered l <= 3 lattice of the seed and its Schwarz bounds, for a
    sample of the screened quartets of one such lattice."""
    rng, *sh = basis.lattice_shells(natom=case['natom'], seed=2)
    pairs, q = _lattice_schwarz(sh)
    quartets, _ = basis.sample_screened_quartets(q, pairs, case['nq'], rng, SCREEN)
    sh = basis.lattice_shells(natom=case['natom'], seed=seed)[1:]
    q = _lattice_schwarz(sh)[1]
    off, total = basis.packed_offsets(sh[0], quartets, True)
    at = lambda i, j: np.maximum(i, j).astype(np.int64) * (np.maximum(i, j) + 1) // 2 + np.minimum(i, j)  # noqa: E731
    bounds = q[at(quartets[:, 0], quartets[:, 1])] * q[at(quartets[:, 2], quartets[:, 3])]
    return basis.ShellBatch(*sh, quartets, off, True, total), bounds


def _dropin_args(case, seed):
    """Argument dicts of one drop-in call; functions of one index are adjacent
    in the output (component, then contracted function), a fastest."""
    ls = [case['la'], case['lb'], case['lc'], case['ld']]
    rng = np.random.default_rng(seed)
    k, nc = case['kmax'], case['ncont']
    shells, stride = [], 1
    for l in ls:
        e = np.exp(rng.uniform(math.log(case['alpha_lo']), math.log(case['alpha_hi']), k))
        coef = np.concatenate([basis.normalize_shell(l, e, rng.uniform(0.1, 1.0, k)) for _ in range(nc)])
        n = 2 * l + 1 if case['spherical'] else (l + 1) * (l + 2) // 2
        sh = dict(x=e, cen=rng.uniform(0.0, case['box'], 3), l=l, n=n, iskip=stride, nprim=k, ncont=nc,
                  iskip_cont=stride * n, coef=coef)
        if case['spherical']:
            sh['T'] = basis.sph_matrix(l)
        stride *= n * nc
        shells.append(sh)
    return shells, stride


def _pairs(case, seed):
    p = twoidx.make_pairs(case['n'], lmax=case['lmax'], seed=seed)
    rng = np.random.default_rng(7)
    p['la'], p['lb'] = rng.integers(0, case['lmax'] + 1, (2, case['n'])).astype(np.int32)
    return p


def prepare(case, seed):
    kind = case['kind']
    if kind == 'dropin':
        shells, size = _dropin_args(case, seed)
        fn = eri.cont_sph_main if case['spherical'] else eri.cont_cart_main
        return dict(kind=kind, shells=shells, fn=fn, out=np.zeros(size))
    if kind in ('batch', 'screened'):
        b = _kept_batch(case, seed) if case.get('kept') else _random_batch(case, seed, case['nq'])
        s = dict(kind=kind, eng=eri.EriEngine(b), out=torch.empty(b.out_size, dtype=torch.float64, device=DEV))
        if kind == 'screened':
            s['bounds'] = torch.empty(b.nq, dtype=torch.float64, device=DEV)
        return s
    if kind == 'lattice':
        b, bounds = _lattice(case, seed)
        return dict(kind=kind, eng=eri.EriEngine(b), out=torch.empty(b.out_size, dtype=torch.float64, device=DEV),
                    bounds=torch.from_numpy(bounds).to(DEV), prec=eri.PREC_MIXED if case['mixed'] else eri.PREC_FP64)
    if kind == 'host':
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).pin_memory()  # noqa: E731
        hb, outs = [], []
        for i in range(case['batches']):
            b = _random_batch(case, 64 * seed + i, case['nq'])
            hb.append({k: pin(getattr(b, k)) for k in ('shell_l', 'shell_k', 'shell_ptr', 'shell_xyz', 'prim_exp',
                                                       'prim_coef', 'quartets', 'out_off')})
            outs.append(torch.empty(b.out_size, dtype=torch.float64).pin_memory())
        return dict(kind=kind, pipe=eri.HostPipeline(case['spherical']), batches=hb, outs=outs, lmax=case['lmax'])
    if kind in ('energy', 'forces'):
        system, xyz = jk.lattice_system(natom=case['natom'], seed=seed, device=DEV)
        return dict(kind=kind, system=system, xyz=torch.from_numpy(xyz).to(DEV))
    tb = twoidx.TwoIndexBatch(_pairs(case, seed), device=DEV)
    return dict(kind=kind, tb=tb, out=torch.empty(tb.size, dtype=torch.float64, device=DEV),
                op=twoidx.NUCLEAR if kind == 'nuclear' else twoidx.OVERLAP)


def run(state):
    kind = state['kind']
    if kind == 'dropin':
        state['fn'](state['shells'], state['out'])
        return state['out']
    if kind == 'batch':
        return state['eng'].compute(out=state['out'])
    if kind == 'screened':
        eng = state['eng']
        eng.analytic_bounds(out=state['bounds'])
        eri.set_prim_tol(PRIM_TOL)
        out = eng.compute(out=state['out'], bounds=state['bounds'], skip_below=SCREEN)
        eri.set_prim_tol(0.0)
        return out
    if kind == 'lattice':
        return state['eng'].compute(out=state['out'], precision=state['prec'], bounds=state['bounds'],
                                    fp32_below=1e-4, mixed_tol=5e-11)
    if kind == 'host':
        for h, out in zip(state['batches'], state['outs']):
            state['pipe'].submit(h, out, skip_below=SCREEN, lmax=state['lmax'])
        state['pipe'].synchronize()
        return state['outs']
    if kind == 'energy':
        return state['system'].energy(state['xyz'])
    if kind == 'forces':
        x = state['xyz'].detach().requires_grad_(True)
        e = jk.jk_energy(x, state['system'])
        e.backward()
        return e.detach(), x.grad
    return state['tb'].compute(state['op'], out=state['out'])


# ------------------------------------------------------------------ work
def _nc(l):
    return (l + 1) * (l + 2) // 2


def _vrr_flops(la, lb, lc, ld):
    """Operations of one primitive quartet's vertical recurrences (about five
    per intermediate of the [e0|f0] tables) with its setup and Boys values."""
    E, F = la + lb, lc + ld
    n = sum(_nc(i) * (F + E - i + 1) for i in range(1, E + 1))
    n += sum(_nc(j) * (F - j + 1) * sum(_nc(i) for i in range(max(la - F + j, 0), E + 1)) for j in range(1, F + 1))
    return 5.0 * n + 74 + 2 * (E + F)


def _pair_r(xyz, s):
    return ((xyz[s[:, 0]] - xyz[s[:, 1]]) ** 2).sum(1)


def _live(l, k, ptr, xyz, e, c, s):
    """Primitive pairs of the shell pairs s whose Gaussian factor is not zero."""
    r2, n = _pair_r(xyz, s), np.zeros(len(s))
    for i in range(int(k.max())):
        for j in range(int(k.max())):
            on = (i < k[s[:, 0]]) & (j < k[s[:, 1]])
            x, y = e[np.where(on, ptr[s[:, 0]] + i, 0)], e[np.where(on, ptr[s[:, 1]] + j, 0)]
            n += on & (x * y / (x + y) * r2 < 745.0)
    return n


def _schwarz_estimate(l, k, ptr, xyz, e, c, s):
    """Size of a shell pair's charge distribution (its largest s-type primitive pair)."""
    r2, q = _pair_r(xyz, s), np.zeros(len(s))
    for i in range(int(k.max())):
        for j in range(int(k.max())):
            on = (i < k[s[:, 0]]) & (j < k[s[:, 1]])
            pi, pj = np.where(on, ptr[s[:, 0]] + i, 0), np.where(on, ptr[s[:, 1]] + j, 0)
            z = e[pi] + e[pj]
            v = np.abs(c[pi] * c[pj]) * np.exp(-e[pi] * e[pj] / z * r2) * z ** (-1.25 - 0.5 * (l[s[:, 0]] + l[s[:, 1]]))
            q = np.maximum(q, np.where(on, v, 0.0))
    return q


def _quartet_flops(l, nprim):
    """Summed VRR operations of quartets with angular momenta l [n, 4] and nprim live primitive quartets."""
    code = l @ np.array([512, 64, 8, 1])
    return sum(_vrr_flops(*l[code == u][0]) * nprim[code == u].sum() for u in np.unique(code))


@functools.lru_cache(maxsize=None)
def _work(items):
    case = dict(items)
    kind = case['kind']
    if kind in ('overlap', 'nuclear'):
        lm, by, fl = case['lmax'], 0.0, 0.0
        for a in range(lm + 1):
            for b in range(lm + 1):
                f, w = twoidx.algorithmic_cost(twoidx.NUCLEAR if kind == 'nuclear' else twoidx.OVERLAP, a, b)
                by, fl = by + w, fl + f
        return case['n'] * by / (lm + 1) ** 2, case['n'] * fl / (lm + 1) ** 2
    if kind == 'dropin':
        ls, nc = [case['la'], case['lb'], case['lc'], case['ld']], case['ncont']
        n = np.prod([2 * l + 1 if case['spherical'] else _nc(l) for l in ls]) * nc ** 4
        return 8.0 * n + 4 * 8 * case['kmax'] * (1 + nc), case['kmax'] ** 4 * nc ** 4 * _vrr_flops(*ls)
    if kind in ('energy', 'forces'):
        # unique quartets above the Schwarz screen (estimated), each with its
        # live primitive quartets; the gradient's blocks have an index raised
        # or lowered at three of the four centres
        rng = np.random.default_rng(0)
        sh = basis.lattice_shells(natom=case['natom'], seed=3, shells=((0, 6), (0, 3), (1, 3), (2, 1)))[1:]
        l = sh[0].astype(np.int64)
        a, b = np.tril_indices(len(l))
        pairs = np.stack([a, b], axis=1)
        q, live = _schwarz_estimate(*sh, pairs), _live(*sh, pairs)
        i, j = rng.integers(0, len(pairs), (2, 40000))
        keep = q[i] * q[j] >= 1e-15
        lq = np.concatenate([l[pairs[i]], l[pairs[j]]], axis=1)[keep]
        # (forces run the energy and then the gradient)
        up = [np.array(v) for v in ((0, 0, 0, 0), (1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 1, 0))]
        fl = sum(_quartet_flops(lq + v, (live[i] * live[j])[keep]) for v in (up if kind == 'forces' else up[:1]))
        return 8.0 * len(sh[4]) * 2 + 24 * len(l), fl / 40000 * len(pairs) * (len(pairs) + 1) / 2
    nq = case['nq']
    if kind == 'lattice':
        m = min(nq, 20000)
        rng = np.random.default_rng(0)
        sh = basis.lattice_shells(natom=case['natom'], seed=2)[1:]
        l = sh[0].astype(np.int64)
        a, b = np.tril_indices(len(l))
        pairs = np.stack([a, b], axis=1)
        quart, _ = basis.sample_screened_quartets(_schwarz_estimate(*sh, pairs), pairs, m, rng, SCREEN)
        lq, sph = l[quart], True
        inputs = 8.0 * (2 * len(sh[4]) + 3 * len(l)) + (16 + 8 + 8) * nq
        keep = np.ones(m, bool)
    else:
        m = min(nq, 4000) if not case.get('kept') else 4000
        b = _random_batch(case, 0, m, torch.device('cpu'))
        sh = (b.shell_l, b.shell_k, b.shell_ptr, b.shell_xyz, b.prim_exp, b.prim_coef)
        quart, sph = b.quartets, case['spherical']
        lq = b.shell_l.astype(np.int64)[quart]
        keep = np.ones(m, bool)
        if kind in ('screened', 'host') or case.get('kept'):
            keep = _schwarz_estimate(*sh, quart[:, :2]) * _schwarz_estimate(*sh, quart[:, 2:]) >= SCREEN
        if case.get('kept') and keep.any():
            quart, lq, keep = quart[keep], lq[keep], keep[keep]
            m = len(quart)
        inputs = (8.0 * 2 * len(sh[4]) / len(sh[0]) + 24) * 4 * nq + (16 + 8) * nq
    nprim = _live(*sh, quart[:, :2]) * _live(*sh, quart[:, 2:])
    n = (2 * lq + 1) if sph else (lq + 1) * (lq + 2) // 2
    by = inputs + 8.0 * n.prod(1).mean() * nq
    fl = _quartet_flops(lq[keep], nprim[keep]) / m * nq
    k = case.get('batches', 1)
    return by * k, fl * k


def work(case):
    by, fl = _work(tuple(sorted((k, v) for k, v in case.items() if k != 'name')))
    return {'bytes': float(by), 'flops': float(fl)}


# ------------------------------------------------------------------ exact values
def _cart(l):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


def _herm(L):
    return [(t, u, n - t - u) for n in range(L + 1) for t in range(n, -1, -1) for u in range(n - t, -1, -1)]


def _sph(l):
    """Real solid harmonics m = -l..l over the Cartesians of l, each scaled to
    the norm of x^l: z-recurrence on top of Re, Im (x + iy)^|m|."""
    def mul(p, q):
        r = {}
        for (a, b, c), v in p.items():
            for (d, e, f), w in q.items():
                k = (a + d, b + e, c + f)
                r[k] = r.get(k, 0.0) + v * w
        return r

    def lin(x, p, y, q):
        r = {k: x * v for k, v in p.items()}
        for k, v in q.items():
            r[k] = r.get(k, 0.0) + y * v
        return r
    X, Y, Z = {(1, 0, 0): 1.0}, {(0, 1, 0): 1.0}, {(0, 0, 1): 1.0}
    R2 = {(2, 0, 0): 1.0, (0, 2, 0): 1.0, (0, 0, 2): 1.0}
    df = lambda n: float(np.prod(np.arange(n, 0, -2))) if n > 0 else 1.0  # noqa: E731
    T = np.zeros((_nc(l), 2 * l + 1))
    for m in range(-l, l + 1):
        re, im = {(0, 0, 0): 1.0}, {}
        for _ in range(abs(m)):
            re, im = lin(1.0, mul(re, X), -1.0, mul(im, Y)), lin(1.0, mul(re, Y), 1.0, mul(im, X))
        p0, p1 = {}, (re if m >= 0 else im)
        for n in range(abs(m), l):  # (n+1-m) P_{n+1} = (2n+1) z P_n - (n+m) r^2 P_{n-1}
            p0, p1 = p1, lin((2 * n + 1) / (n + 1 - abs(m)), mul(Z, p1), -(n + abs(m)) / (n + 1 - abs(m)), mul(R2, p0))
        col = np.array([p1.get(k, 0.0) for k in _cart(l)])
        nrm = 0.0
        for x, k in zip(col, _cart(l)):
            for y, q in zip(col, _cart(l)):
                s = [a + b for a, b in zip(k, q)]
                if not any(v % 2 for v in s):
                    nrm += x * y * df(s[0] - 1) * df(s[1] - 1) * df(s[2] - 1)
        T[:, m + l] = col * math.sqrt(df(2 * l - 1) / nrm)
    return T


def _boys(T, L):
    """F_0..F_L(T), [L + 1, n]: ascending series and downward recursion below
    T = 40, the complete function and upward recursion above."""
    F = torch.empty((L + 1,) + T.shape, dtype=torch.float64, device=T.device)
    t = T.clamp(max=40.0)
    term = torch.full_like(t, 1.0 / (2 * L + 1))
    s = term.clone()
    for k in range(1, 180):
        term = term * (2.0 * t / (2 * L + 2 * k + 1))
        s += term
    e = torch.exp(-t)
    F[L] = e * s
    for m in range(L - 1, -1, -1):
        F[m] = (2.0 * t * F[m + 1] + e) / (2 * m + 1)
    big = T > 40.0
    if bool(big.any()):
        x = T[big]
        f = 0.5 * torch.sqrt(math.pi / x) * torch.erf(torch.sqrt(x))
        ex = torch.exp(-x)
        for m in range(L + 1):
            F[m][big] = f
            f = ((2 * m + 1) * f - ex) / (2.0 * x)
    return F


def _E(la, lb, p, PA, PB):
    """Hermite expansion coefficients of x_A^i x_B^j over exp(-p x_P^2), {(i, j): [n, i + j + 1]}."""
    E = {(0, 0): torch.ones(p.shape[0], 1, dtype=torch.float64, device=p.device)}

    def raise_(src, X):
        n = src.shape[1]
        out = torch.zeros(src.shape[0], n + 1, dtype=torch.float64, device=p.device)
        out[:, 1:] += src / (2.0 * p)[:, None]
        out[:, :n] += X[:, None] * src
        if n > 1:
            out[:, :n - 1] += torch.arange(1, n, dtype=torch.float64, device=p.device) * src[:, 1:]
        return out
    for i in range(la + 1):
        if i:
            E[i, 0] = raise_(E[i - 1, 0], PA)
        for j in range(1, lb + 1):
            E[i, j] = raise_(E[i, j - 1], PB)
    return E


def _pair_hermite(la, lb, p, PA, PB, sign=False):
    """[n, ncart(la) ncart(lb), nherm(la + lb)] expansion of the Cartesian pairs (a fastest)."""
    H, nt = _herm(la + lb), la + lb + 1
    pairs = [(a, b) for b in _cart(lb) for a in _cart(la)]
    out = torch.ones(1, dtype=torch.float64, device=p.device)
    for d in range(3):
        E = _E(la, lb, p, PA[:, d], PB[:, d])
        flat = torch.zeros(p.shape[0], (la + 1) * (lb + 1) * nt, dtype=torch.float64, device=p.device)
        for (i, j), v in E.items():
            flat[:, (i * (lb + 1) + j) * nt:][:, :v.shape[1]] = v
        at = torch.tensor([[(a[d] * (lb + 1) + b[d]) * nt + h[d] for h in H] for a, b in pairs], device=p.device)
        out = out * flat[:, at]
    if sign:
        out = out * torch.tensor([(-1.0) ** sum(h) for h in H], dtype=torch.float64, device=p.device)
    return out


def _R(L, rho, PQ):
    """Hermite Coulomb integrals R_tuv, t + u + v <= L, [nherm(L), n]."""
    F = _boys(rho * (PQ ** 2).sum(1), L)
    cur = {(0, 0, 0): [(-2.0 * rho) ** n * F[n] for n in range(L + 1)]}
    for tot in range(1, L + 1):
        for h in _herm(tot)[-_nc(tot):]:
            d = next(i for i in range(3) if h[i])
            lo = tuple(v - (i == d) for i, v in enumerate(h))
            lo2 = tuple(v - 2 * (i == d) for i, v in enumerate(h))
            cur[h] = [PQ[:, d] * cur[lo][n + 1] + ((h[d] - 1) * cur[lo2][n + 1] if h[d] > 1 else 0.0)
                      for n in range(L - tot + 1)]
    return torch.stack([cur[h][0] for h in _herm(L)])


def _exact_quartets(b):
    """Blocks of every quartet of the batch b (flat, at out_off), or None."""
    dev = DEV
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    l = b.shell_l[b.quartets].astype(np.int64)
    nprim = b.shell_k[b.quartets].astype(np.int64).prod(1)
    H = lambda n: (n + 1) * (n + 2) * (n + 3) // 6  # noqa: E731
    nab, ncd = _nc(l[:, 0]) * _nc(l[:, 1]), _nc(l[:, 2]) * _nc(l[:, 3])
    hb, hk = H(l[:, 0] + l[:, 1]), H(l[:, 2] + l[:, 3])
    cost = (nab * hb + ncd * hk + hb * hk) * 4 + nab * hb * hk + nab * hk * ncd + 20 * H(l.sum(1)) * (l.sum(1) + 1)
    if float((cost * nprim).sum()) > EXACT_WORK:
        return None
    out = torch.zeros(b.out_size, dtype=torch.float64, device=dev)
    code = l @ np.array([512, 64, 8, 1])
    xyz, e, c = t(b.shell_xyz), t(b.prim_exp), t(b.prim_coef)
    for u in np.unique(code):
        sel = np.nonzero(code == u)[0]
        la, lb, lc, ld = l[sel[0]]
        L = int(la + lb + lc + ld)
        gather = torch.tensor([[_herm(L).index(tuple(x + y for x, y in zip(h, g))) for g in _herm(lc + ld)]
                               for h in _herm(la + lb)], device=dev)
        per = int((4 * (nab * hb + ncd * hk) + 2 * hb * hk + nab * (hk + ncd))[sel[0]])
        step = max(1, int(2e8 / per))  # primitive quartets at a time
        blocks = torch.zeros(len(sel), _nc(la) * _nc(lb), _nc(lc) * _nc(ld), dtype=torch.float64, device=dev)
        quart, npr = t(b.quartets[sel].astype(np.int64)), nprim[sel]
        first = np.cumsum(npr) - npr
        k, ptr = t(b.shell_k.astype(np.int64)), t(b.shell_ptr.astype(np.int64))
        for p0 in range(0, int(npr.sum()), step):
            p1 = min(p0 + step, int(npr.sum()))
            q = t(np.searchsorted(first, np.arange(p0, p1), side='right') - 1)
            w = torch.arange(p0, p1, device=dev) - t(first)[q]
            s = quart[q]
            idx = [None] * 4
            for i in (3, 2, 1, 0):
                ki = k[s[:, i]]
                idx[i] = ptr[s[:, i]] + w % ki
                w = w // ki
            x = [e[i] for i in idx]
            X = [xyz[s[:, i]] for i in range(4)]
            z, n = x[0] + x[1], x[2] + x[3]
            P = (x[0][:, None] * X[0] + x[1][:, None] * X[1]) / z[:, None]
            Q = (x[2][:, None] * X[2] + x[3][:, None] * X[3]) / n[:, None]
            pre = 2.0 * math.pi ** 2.5 / (z * n * torch.sqrt(z + n))
            pre = pre * torch.exp(-x[0] * x[1] / z * ((X[0] - X[1]) ** 2).sum(1)) * c[idx[0]] * c[idx[1]]
            pre = pre * torch.exp(-x[2] * x[3] / n * ((X[2] - X[3]) ** 2).sum(1)) * c[idx[2]] * c[idx[3]]
            on = torch.nonzero(pre != 0.0).flatten()
            if not on.numel():
                continue
            g = lambda v: v[on]  # noqa: E731
            bra = _pair_hermite(la, lb, g(z), g(P - X[0]), g(P - X[1])) * g(pre)[:, None, None]
            ket = _pair_hermite(lc, ld, g(n), g(Q - X[2]), g(Q - X[3]), sign=True)
            R = _R(L, g(z * n / (z + n)), g(P - Q)).T[:, gather]
            blocks.index_add_(0, q[on], bra @ R @ ket.transpose(1, 2))
        v = blocks.view(len(sel), _nc(lb), _nc(la), _nc(ld), _nc(lc))
        if b.spherical:
            Ta, Tb, Tc, Td = (t(_sph(int(x))) for x in (la, lb, lc, ld))
            v = torch.einsum('nbadc,ai,bj,ck,dl->njilk', v, Ta, Tb, Tc, Td)
        v = v.permute(0, 3, 4, 1, 2).reshape(len(sel), -1)  # [d][c][b][a]
        at = t(b.out_off[sel])[:, None] + torch.arange(v.shape[1], device=dev)[None, :]
        out[at.reshape(-1)] = v.reshape(-1)
    return out


def _exact_pairs(case, p):
    """Overlap or nuclear-attraction blocks of primitive pairs (flat, packed)."""
    off, size = twoidx.block_offsets(p['la'], p['lb'])
    out = torch.zeros(size, dtype=torch.float64, device=DEV)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    for la in range(case['lmax'] + 1):
        for lb in range(case['lmax'] + 1):
            sel_all = np.nonzero((p['la'] == la) & (p['lb'] == lb))[0]
            for sel in np.array_split(sel_all, max(1, len(sel_all) // 100000)):
                if not len(sel):
                    continue
                xa, xb, A, B = t(p['xa'][sel]), t(p['xb'][sel]), t(p['ca'][sel]), t(p['cb'][sel])
                z = xa + xb
                P = (xa[:, None] * A + xb[:, None] * B) / z[:, None]
                K = torch.exp(-xa * xb / z * ((A - B) ** 2).sum(1))
                h = _pair_hermite(la, lb, z, P - A, P - B)
                if case['kind'] == 'overlap':
                    v = h[:, :, 0] * (K * (math.pi / z) ** 1.5)[:, None]
                else:
                    R = _R(la + lb, z, P - t(p['cc'][sel])).T
                    v = (h @ R[:, :, None])[:, :, 0] * (K * 2.0 * math.pi / z)[:, None]
                at = t(off[sel])[:, None] + torch.arange(v.shape[1], device=DEV)[None, :]
                out[at.reshape(-1)] = v.reshape(-1)
    return out


def _exact_dropin(case, seed):
    shells, size = _dropin_args(case, seed)
    nc, sph = case['ncont'], case['spherical']
    ls = np.repeat([s['l'] for s in shells], nc).astype(np.int32)
    ks = np.full(4 * nc, case['kmax'], np.int32)
    ptr = (np.arange(4 * nc) * case['kmax']).astype(np.int32)
    e = np.concatenate([np.tile(s['x'], nc) for s in shells])
    c = np.concatenate([s['coef'] for s in shells])
    xyz = np.repeat(np.stack([s['cen'] for s in shells]), nc, axis=0)
    combos = np.array(np.meshgrid(*[np.arange(nc)] * 4, indexing='ij')).reshape(4, -1).T
    quart = (combos + nc * np.arange(4)).astype(np.int32)
    off, total = basis.packed_offsets(ls, quart, sph)
    v = _exact_quartets(basis.ShellBatch(ls, ks, ptr, xyz, e, c, quart, off, sph, total)).cpu().numpy()
    n = [s['n'] for s in shells]
    out = np.zeros(size)
    comp = np.array(np.meshgrid(*[np.arange(m) for m in n[::-1]], indexing='ij')).reshape(4, -1)[::-1]
    step = np.array([s['iskip'] for s in shells])
    for w, o in zip(combos, off):
        at = (w * np.array([s['iskip_cont'] for s in shells])).sum() + (comp * step[:, None]).sum(0)
        out[at] = v[o:o + comp.shape[1]]
    return out


def exact(case, seed):
    kind = case['kind']
    if kind == 'dropin':
        return _exact_dropin(case, seed)
    if kind in ('overlap', 'nuclear'):
        return _exact_pairs(case, _pairs(case, seed))
    if kind in ('batch', 'screened'):
        return _exact_quartets(_kept_batch(case, seed) if case.get('kept') else _random_batch(case, seed, case['nq']))
    if kind == 'lattice':
        return _exact_quartets(_lattice(case, seed)[0])
    return None  # whole energies, gradients and streamed batches: over the time that a check can take
