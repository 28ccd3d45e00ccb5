"""The warp-per-quartet kernels where their layout changes: batch sizes either
side of the small-batch and merged-kernel limits, pair counts either side of the
64-pair tile, and the Rys table's rows and range ends."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import tolerance
from intception_b200 import basis, eri
from intception_b200.emit import rys_table
from oracle import loader


@pytest.mark.parametrize('N', [2, 5, 9])
def test_rys_rule_reproduces_boys_moments(N):
    """sum_r w_r u_r^k = F_k(T), k < 2N, from the stored polynomials (first row,
    one inside, the last) and from the rule beyond the table.  Table values are
    rounded to double (2^-53 each) and u^k multiplies u's error by k."""
    import mpmath as mp
    mp.mp.dps = 60
    last = rys_table.RYS_TMAX[N] * rys_table.RYS_H_INV - 1
    checks = []
    for row in (0, 17, last):
        coef = rys_table._row(row)[N]
        for x in (-1.0, -0.3, 0.999):
            v = [sum(mp.mpf(c) * mp.mpf(x) ** k for k, c in enumerate(cs)) for cs in coef]
            checks.append(((row + (mp.mpf(x) + 1) / 2) / rys_table.RYS_H_INV, v[0::2], v[1::2]))
    for T in (mp.mpf(rys_table.RYS_TMAX[N]), mp.mpf(500)):
        hw = rys_table._asymptotic(N)
        checks.append((T, [h / T for h, _ in hw], [w / mp.sqrt(T) for _, w in hw]))
    for T, u, w in checks:
        F = rys_table._moments(T, 2 * N)
        for k in range(2 * N):
            s = sum(wr * ur ** k for ur, wr in zip(u, w))
            assert abs(s / F[k] - 1) <= (2 * k + 4) * 2.0 ** -52, (N, T, k)


@pytest.mark.gpu
@pytest.mark.parametrize('sph', [False, True])
@pytest.mark.parametrize('lmax', [1, 2])
def test_batch_sizes_around_the_path_limits(sph, lmax):
    """The first quartets of one list, evaluated in batches of 1, 296, 297, 3072
    and 3073 quartets (small-batch kernel, merged kernel, one kernel per
    class), unscreened and screened, against the oracle."""
    import torch
    b = basis.independent_quartet_batch(31, 3073, list(range(lmax + 1)), [1, 2, 3, 5], 0.1, 60.0, 6.0, sph)
    head = b.subset(np.arange(300))
    ref = loader.oracle_batch(head, basis.sph_matrices(6))
    for nq in (1, 296, 297, 3072, 3073):
        eng = eri.EriEngine(b.subset(np.arange(nq)))
        n = int(head.out_off[min(nq, 300) - 1]) if nq < 300 else head.out_size
        out = torch.full((eng.out_size,), 7.0, dtype=torch.float64, device='cuda')
        eng.compute(out=out)
        assert np.abs(out.cpu().numpy()[:n] - ref[:n]).max(initial=0.0) <= tolerance(ref), nq
        bounds = eng.analytic_bounds()
        out.fill_(7.0)
        eri.set_prim_tol(1e-18)
        eng.compute(out=out, bounds=bounds, skip_below=1e-9)
        eri.set_prim_tol(0.0)
        # a zeroed block is off by at most its bound, 5^4 dropped primitives by 1e-18 each
        got, kept = out.cpu().numpy(), bounds.cpu().numpy() >= 1e-9
        assert np.abs(got[:n] - ref[:n]).max(initial=0.0) <= 1e-9 + tolerance(ref)
        assert (got != 7.0).all()
        for q in np.nonzero(kept[:300])[0]:
            o, m = int(head.out_off[q]), int(np.prod(head.block_dims(q)))
            assert np.abs(got[o:o + m] - ref[o:o + m]).max() <= 625e-18 + tolerance(ref)
        assert eng.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize('ls', [(0, 0, 0, 0), (1, 0, 1, 0), (1, 1, 1, 1), (2, 1, 1, 1), (2, 2, 2, 1), (2, 2, 2, 2)])
@pytest.mark.parametrize('ks', [(1, 1, 1, 1), (8, 8, 4, 8), (9, 8, 8, 8), (13, 11, 5, 13)])
def test_pair_counts_around_the_tile(ls, ks):
    """Pair counts 1, 64, 72 and 143 a side (one tile of pairs holds 64), with
    and without primitive screening at 1e-18."""
    rng = np.random.default_rng(7)
    n = 3
    sh = basis.make_shells(rng, np.tile(ls, n), np.tile(ks, n), 0.2, 8.0, 1.5)
    q = np.arange(4 * n, dtype=np.int32).reshape(n, 4)
    off, total = basis.packed_offsets(sh[0], q, True)
    b = basis.ShellBatch(*sh, q, off, True, total)
    ref = loader.oracle_batch(b, basis.sph_matrices(6))
    eng = eri.EriEngine(b)
    assert np.abs(eng.compute().cpu().numpy() - ref).max() <= tolerance(ref)
    eri.set_prim_tol(1e-18)
    out = eng.compute().cpu().numpy()
    eri.set_prim_tol(0.0)
    assert np.abs(out - ref).max() <= tolerance(ref) + np.prod(np.array(ks, float)) * 1e-18


@pytest.mark.gpu
@pytest.mark.parametrize('nq', [8, 400])
@pytest.mark.parametrize('between', [8, 400])
def test_status_after_graph_replay(nq, between):
    """The status read after a replay is the replayed batch's, on the small-batch
    kernel and on the pipeline, whichever of them ran in between."""
    import torch
    bad = eri.EriEngine(basis.independent_quartet_batch(5, nq, [2], [1, 2], 0.1, 60.0, 6.0, True))
    bad._basis.lmax = 1  # declared lmax below the shells' l
    good = eri.EriEngine(basis.independent_quartet_batch(6, between, [0, 1, 2], [1, 2], 0.1, 60.0, 6.0, True))
    g = bad.graph(torch.empty(bad.out_size, dtype=torch.float64, device='cuda'))
    good.compute()
    assert good.device_status() == 0
    g.launch()
    assert bad.device_status() == eri.IB_ERR_ARG
    good.compute()
    assert good.device_status() == 0
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize('lmax', [2, 3])
def test_graph_replay_after_larger_batches(lmax):
    """A graph replays on the work buffers it was captured with: batches of more
    quartets and of a higher l in between move the library on to larger ones.
    Same kernels on the same inputs in a fixed order: the same bits; the counts
    are the replayed batch's, also once the graph is closed."""
    import torch
    eng = eri.EriEngine(basis.independent_quartet_batch(8, 400, list(range(lmax + 1)), [4, 6], 0.01, 1e5, 4.0, True))
    out = torch.empty(eng.out_size, dtype=torch.float64, device='cuda')
    g = eng.graph(out)
    ref, redo = eng.compute().cpu().numpy(), eri.last_hrr_redo()
    assert redo > 0
    for nq, l in ((5000, 2), (20000, 4)):
        big = eri.EriEngine(basis.independent_quartet_batch(9, nq, [0, 1, l], [1, 2], 0.1, 60.0, 6.0, True))
        big.compute()
        out.fill_(7.0)
        g.launch()
        assert np.array_equal(out.cpu().numpy(), ref)
        assert eri.last_hrr_redo() == redo and eng.device_status() == 0 and eng.fp32_rejected() == 0
    g.close()
    assert eri.last_hrr_redo() == redo
    assert np.array_equal(eng.compute().cpu().numpy(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize('sph', [False, True])
@pytest.mark.parametrize('lmax', [1, 2])
def test_every_quartet_of_batches_at_the_path_limits(sph, lmax):
    """Every block of the batches either side of the path limits, the last
    quartet's among them, against the oracle (out starts from 7, which no
    evaluated element keeps)."""
    import torch
    b = basis.independent_quartet_batch(32, 3073, list(range(lmax + 1)), [1, 2, 3, 5], 0.1, 60.0, 6.0, sph)
    ref = loader.oracle_batch(b, basis.sph_matrices(6))
    for nq in (1, 296, 297, 3072, 3073):
        eng = eri.EriEngine(b.subset(np.arange(nq)))
        out = torch.full((eng.out_size,), 7.0, dtype=torch.float64, device='cuda')
        got = eng.compute(out=out).cpu().numpy()
        assert eng.out_size == b.out_off[nq - 1] + np.prod(b.block_dims(nq - 1))
        assert np.abs(got - ref[:eng.out_size]).max() <= tolerance(ref), nq


@pytest.mark.gpu
@pytest.mark.parametrize('sph', [False, True])
@pytest.mark.parametrize('lmax', [1, 2, 3])
def test_short_quartets_of_large_batches(sph, lmax):
    """Batches of few primitives a shell, large enough that quartets of up to 31
    primitive quartets (fewer in the wider classes) go to the lane-group
    kernels: against the same quartets in two batches of half the size, which
    stay below that size, and against the oracle; screened too, with more and
    with fewer evaluated quartets than that."""
    import torch
    nq = 8192 if lmax == 1 else 32768  # mean K 1.5
    b = basis.independent_quartet_batch(41, nq, list(range(lmax + 1)), [1, 1, 1, 3], 0.1, 60.0, 5.0, sph)
    eng = eri.EriEngine(b)
    got = eng.compute().cpu().numpy()
    halves = [eri.EriEngine(b.subset(np.arange(i, i + nq // 2))) for i in (0, nq // 2)]
    want = np.concatenate([e.compute().cpu().numpy() for e in halves])
    assert np.abs(got - want).max() <= tolerance(want)
    head = b.subset(np.arange(1500))
    ref = loader.oracle_batch(head, basis.sph_matrices(6))
    assert np.abs(got[:head.out_size] - ref).max() <= tolerance(want)
    two = eri.EriEngine(b.subset(np.concatenate([np.arange(nq)] * 2)))
    bounds = two.analytic_bounds()
    for cut in np.quantile(bounds.cpu().numpy(), [0.3, 0.7]):
        out = torch.full((two.out_size,), 7.0, dtype=torch.float64, device='cuda')
        two.compute(out=out, bounds=bounds, skip_below=float(cut))
        d = np.abs(out.cpu().numpy() - np.concatenate([want, want]))
        off = two.out_off.cpu().numpy()
        worst = np.maximum.reduceat(d, off)  # packed: largest difference in each quartet's block
        kept = bounds.cpu().numpy() >= cut
        assert worst[kept].max() <= tolerance(want) and (worst[~kept] <= 1.000001 * bounds.cpu().numpy()[~kept]).all()


@pytest.mark.gpu
@pytest.mark.parametrize('sph', [False, True])
def test_merged_kernel_limit_with_few_primitives(sph):
    """Mean K 1.5: 24576 quartets take the merged kernel, one more a kernel per
    class; the same values, and the oracle's."""
    b = basis.independent_quartet_batch(43, 24577, [0, 1, 2], [1, 1, 2, 2], 0.1, 60.0, 5.0, sph)
    more = eri.EriEngine(b).compute().cpu().numpy()
    less = eri.EriEngine(b.subset(np.arange(24576))).compute().cpu().numpy()
    assert np.abs(more[:len(less)] - less).max() <= tolerance(more)
    head = b.subset(np.arange(1500))
    ref = loader.oracle_batch(head, basis.sph_matrices(6))
    assert np.abs(less[:head.out_size] - ref).max() <= tolerance(more)
    tail = b.subset(np.arange(24300, 24577))
    assert np.abs(more[-tail.out_size:] - loader.oracle_batch(tail, basis.sph_matrices(6))).max() <= tolerance(more)


CAPTURED = '''
import sys
import numpy as np
import torch
from intception_b200 import basis, eri
own = sys.argv[1] == 'own'  # captured on the caller's own stream, not by eri_graph_create
eng = eri.EriEngine(basis.independent_quartet_batch(8, 500, [0, 1, 2, 3], [4, 6], 0.01, 1e5, 4.0, True))
out = torch.empty(eng.out_size, dtype=torch.float64, device='cuda')
ref = eng.compute(out=out).cpu().numpy()
if own:
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        eng.compute(out=out)
    replay = g.replay
else:
    replay = eng.graph(out).launch
for nq, l in ((6000, 2), (30000, 5)):
    eri.EriEngine(basis.independent_quartet_batch(9, nq, [0, 1, l], [1], 0.1, 60.0, 6.0, True)).compute()
    out.fill_(7.0)
    replay()
    assert np.array_equal(out.cpu().numpy(), ref)
'''


@pytest.mark.gpu
@pytest.mark.parametrize('how', ['own', 'library'])
def test_captured_batch_after_larger_batches_in_a_new_process(how):
    """In a process of its own, where no earlier test has grown the work
    buffers: a captured batch, by the library or on the caller's stream, replays
    to the same bits after the library has moved on to larger buffers."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, '-c', CAPTURED, how], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
