"""Device table of Rys quadrature roots and weights, generated with mpmath at
build time.

For N roots and a Boys argument T the quadrature satisfies
``sum_r w_r u_r^k = F_k(T)``, k = 0..2N-1 (u = t^2 in (0, 1)): the Gauss rule of
the weight ``exp(-T u) / (2 sqrt(u))`` (Dupuis, Rys, King, J. Chem. Phys. 65,
111 (1976)).  Its nodes and weights follow from the moments F_k by the Chebyshev
algorithm (recurrence coefficients), Newton's iteration on the orthogonal
polynomial and the Christoffel numbers, all in 60-digit arithmetic.

Between 0 and RYS_TMAX[N] each root and weight is a polynomial of degree
RYS_DEG in x = 2 (4 T - row) - 1 on the interval [row/4, (row + 1)/4)
(interpolation at the Chebyshev nodes: at most 6e-17 relative error).  Above RYS_TMAX[N] the rule is the half-range Hermite one,
u_r = h_r / T, w_r = v_r / sqrt(T), within 1e-16 relative.

Layout per N, in doubles: rows x (RYS_DEG + 1) x N x (root, weight), then
N x (h_r, v_r).
"""
import json
import os
import subprocess
import sys

RYS_H_INV = 4            # intervals per unit T
RYS_DEG = 8
RYS_NMIN, RYS_NMAX = 2, 13   # 13: l = 6 on all four shells
RYS_TMAX = {2: 47, 3: 54, 4: 60, 5: 66, 6: 72, 7: 78, 8: 84, 9: 90, 10: 95, 11: 100, 12: 105, 13: 110}


def _moments(T, n):
    import mpmath as mp
    if T == 0:
        return [mp.mpf(1) / (2 * m + 1) for m in range(n)]
    c = [None] * n
    c[-1] = mp.hyp1f1(n - mp.mpf(1) / 2, n + mp.mpf(1) / 2, -T) / (2 * n - 1)
    e = mp.exp(-T)
    for m in range(n - 2, -1, -1):
        c[m] = (2 * T * c[m + 1] + e) / (2 * m + 1)
    return c


def _gauss(N, mu):
    """Nodes and weights of the N-point rule with moments mu[0..2N-1]."""
    import mpmath as mp
    import numpy as np
    a, b = [mu[1] / mu[0]], [mu[0]]
    prev, cur = [mp.mpf(0)] * (2 * N), list(mu[:2 * N])
    for k in range(1, N):
        nxt = [mp.mpf(0)] * (2 * N)
        for m in range(k, 2 * N - k):
            nxt[m] = cur[m + 1] - a[k - 1] * cur[m] - b[k - 1] * prev[m]
        a.append(nxt[k + 1] / nxt[k] - cur[k] / cur[k - 1])
        b.append(nxt[k] / cur[k - 1])
        prev, cur = cur, nxt
    J = np.diag([float(x) for x in a])
    for k in range(1, N):
        J[k, k - 1] = J[k - 1, k] = float(mp.sqrt(b[k]))
    us, ws = [], []
    for x0 in np.linalg.eigvalsh(J):
        x = mp.mpf(float(x0))
        for _ in range(3):
            p0, p1, d0, d1 = mp.mpf(0), mp.mpf(1), mp.mpf(0), mp.mpf(0)
            for k in range(N):
                bk = b[k] if k else mp.mpf(0)
                p0, p1, d0, d1 = p1, (x - a[k]) * p1 - bk * p0, d1, p1 + (x - a[k]) * d1 - bk * d0
            x -= p1 / d1
        s, h, p0, p1 = mp.mpf(0), b[0], mp.mpf(0), mp.mpf(1)
        for k in range(N):
            s += p1 * p1 / h
            p0, p1 = p1, (x - a[k]) * p1 - (b[k] * p0 if k else 0)
            if k + 1 < N:
                h *= b[k + 1]
        us.append(x)
        ws.append(1 / s)
    return us, ws


def _row(row):
    """Polynomial coefficients of row (interval index) for every N whose table reaches it."""
    import mpmath as mp
    mp.mp.dps = 60
    n = RYS_DEG + 1
    xs = [mp.cos((2 * i + 1) * mp.pi / (2 * n)) for i in range(n)]
    mus = [_moments((row + (x + 1) / 2) / RYS_H_INV, 2 * RYS_NMAX) for x in xs]
    out = {}
    for N in range(RYS_NMIN, RYS_NMAX + 1):
        if row >= RYS_TMAX[N] * RYS_H_INV:
            continue
        rules = [_gauss(N, mu) for mu in mus]
        coef = []
        for r in range(N):
            for which in (0, 1):
                # Chebyshev series through the nodes, then powers of x
                c = [2 * sum(rules[i][which][r] * mp.cos(k * (2 * i + 1) * mp.pi / (2 * n)) for i in range(n)) / n
                     for k in range(n)]
                c[0] /= 2
                mono = [mp.mpf(0)] * n
                t0, t1 = [mp.mpf(1)], [mp.mpf(0), mp.mpf(1)]
                for k in range(n):
                    for j, v in enumerate(t0):
                        mono[j] += c[k] * v
                    t2 = [mp.mpf(0)] + [2 * v for v in t1]
                    for j, v in enumerate(t0):
                        t2[j] -= v
                    t0, t1 = t1, t2
                coef.append([float(v) for v in mono])
        out[N] = coef
    return out


def _asymptotic(N):
    import mpmath as mp
    mp.mp.dps = 60
    u, w = _gauss(N, [mp.gamma(k + mp.mpf(1) / 2) / 2 for k in range(2 * N)])
    return [(float(a), float(b)) for a, b in zip(u, w)]


def write_headers(outdir):
    """rys_table.h (sizes) and rys_table_data.h (the values).  The values take
    about five minutes of one core; they are kept while this file is unchanged."""
    from .boys_table import _write
    import hashlib
    with open(os.path.abspath(__file__), 'rb') as fh:
        key = hashlib.sha1(fh.read()).hexdigest()
    data = os.path.join(outdir, 'rys_table_data.h')
    off, offs = 0, {}
    for N in range(RYS_NMIN, RYS_NMAX + 1):
        offs[N] = off
        off += RYS_TMAX[N] * RYS_H_INV * (RYS_DEG + 1) * N * 2 + 2 * N
    pick = lambda d: ' : '.join('N == %d ? %d' % kv for kv in sorted(d.items())) + ' : 0'  # noqa: E731
    _write(os.path.join(outdir, 'rys_table.h'), [
        '/* Generated by intception_b200/emit/rys_table.py. */',
        '#pragma once',
        '#define IB_RYS_H_INV %d' % RYS_H_INV,
        '#define IB_RYS_DEG %d' % RYS_DEG,
        '#define IB_RYS_NMAX %d' % RYS_NMAX,
        '#define IB_RYS_SIZE %d' % off,
        'extern const double ib_rys_host_table[IB_RYS_SIZE];',
        '__host__ __device__ inline constexpr int ib_rys_off(int N) { return %s; }' % pick(offs),
        '__host__ __device__ inline constexpr int ib_rys_tmax(int N) { return %s; }' % pick(RYS_TMAX)])
    if os.path.exists(data):
        with open(data) as fh:
            if key in fh.readline():
                return
    # the rows dealt to child interpreters (this file run as a script)
    jobs = min(16, os.cpu_count() or 1)
    procs = [subprocess.Popen([sys.executable, os.path.abspath(__file__), str(j), str(jobs)], stdout=subprocess.PIPE)
             for j in range(jobs)]
    got = {}
    for p in procs:
        text = p.communicate()[0]
        if p.returncode:
            raise RuntimeError('rys_table: a worker failed')
        got.update((int(row), {int(N): c for N, c in cs.items()}) for row, cs in json.loads(text).items())
    lines = ['/* %s: generated by intception_b200/emit/rys_table.py. */' % key, '#pragma once', '#include "rys_table.h"',
             'const double ib_rys_host_table[IB_RYS_SIZE] = {']
    for N in range(RYS_NMIN, RYS_NMAX + 1):
        for row in range(RYS_TMAX[N] * RYS_H_INV):
            c = got[row][N]
            for k in range(RYS_DEG + 1):
                lines.append('  ' + ', '.join('%.17g, %.17g' % (c[2 * r][k], c[2 * r + 1][k]) for r in range(N)) + ',')
        lines.append('  ' + ', '.join('%.17g, %.17g' % v for v in _asymptotic(N)) + ',')
    lines.append('};')
    _write(data, lines)


if __name__ == '__main__':
    first, step = int(sys.argv[1]), int(sys.argv[2])
    print(json.dumps({row: _row(row) for row in range(first, max(RYS_TMAX.values()) * RYS_H_INV, step)}))
