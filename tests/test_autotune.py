"""The autotuner's host logic (no GPU): merging the tuning runs of the two
chain-order builds, and the tables the build bakes from the result."""
import json
import os

import pytest

from intception_b200 import autotune
from intception_b200.emit import eri_emitter


def _run(order, ms_by_tag):
    classes = {}
    for tag, (fp64, fp32) in ms_by_tag.items():
        classes[tag] = {'minb': [0, 1, 2, 3] if order == 'level' else [3, 2, 1, 0],
                        'ms': {'fp64_cart': [fp64, fp64 + 1], 'fp64_sph': [fp64 + 0.5, fp64],
                               'fp32_cart': [fp32, fp32 + 1], 'fp32_sph': [fp32 + 1, fp32]}}
    return {'meta': {'chain_order': order}, 'classes': classes}


def test_merge_picks_the_faster_order_and_fp32(tmp_path):
    a = tmp_path / 'dfs.json'
    b = tmp_path / 'level.json'
    a.write_text(json.dumps(_run('dfs', {'2221': (10.0, 7.0), '1000': (1.0, 1.5)})))
    b.write_text(json.dumps(_run('level', {'2221': (9.0, 6.5), '1000': (1.2, 1.6)})))
    out = tmp_path / 'tuning.json'
    merged = autotune.merge([str(a), str(b)], str(out))
    assert merged['2221']['order'] == 'level' and merged['2221']['minb'] == [0, 1, 2, 3]
    assert merged['1000']['order'] == 'dfs' and merged['1000']['minb'] == [3, 2, 1, 0]
    assert merged['2221']['fp32'] is True   # FP32 kernel at least 3 % faster in both outputs
    assert merged['1000']['fp32'] is False  # slower: the FP32 tier leaves this class in FP64
    assert json.loads(out.read_text())['classes'] == merged


def test_committed_tuning_covers_every_tuned_class():
    path = os.path.join(os.path.dirname(autotune.__file__), 'tuning.json')
    with open(path) as fh:
        tun = json.load(fh)['classes']
    tags = {'%d%d%d%d' % c for c in eri_emitter.canonical_classes(2)}
    # and the emitted f classes in canonical order (autotune --classes f)
    tags |= {'%d%d%d%d' % c for c, _ in eri_emitter.emitted_classes()
             if max(c) == 3 and c[0] >= c[1] and c[2] >= c[3]}
    assert tags == set(tun)
    for ent in tun.values():
        assert len(ent['minb']) == 4 and all(0 <= m < len(autotune.MINB_VALUES) for m in ent['minb'])
        assert ent['order'] in ('dfs', 'level') and isinstance(ent['fp32'], bool)


@pytest.mark.gpu
def test_tuner_times_the_fp32_kernels(monkeypatch):
    """The FP32 columns are of the FP32 kernel even where the built-in default
    has it off: its result differs from the FP64 kernel's (by 2^-24 of the
    intermediates, so by far more than FP64 rounding)."""
    from intception_b200 import eri
    out, rel = {}, []

    def fake(eng, o, precision, reps, warmup=2):
        kw = dict(bounds=eng._tune_bounds, skip_below=0.0, fp32_below=2.0, mixed_tol=1e300)
        eng.compute(out=o, precision=precision, **(kw if precision == eri.PREC_MIXED else {}))
        r = o.cpu()
        if precision == eri.PREC_FP64:
            out['ref'] = r
        else:
            rel.append(float((r - out['ref']).abs().max() / out['ref'].abs().max()))
        return 1.0
    monkeypatch.setattr(autotune, 'time_variant', fake)
    try:
        autotune.tune(nq=400, reps=1, classes=[(2, 1, 1, 1)], log=lambda *a: None)
    finally:
        for v4 in range(4):
            eri.set_class_minb((2, 1, 1, 1), v4, 0)
    assert len(rel) == 2 * len(autotune.MINB_VALUES) and all(1e-12 < x < 1e-4 for x in rel), rel


@pytest.mark.gpu
def test_bench_names_the_tier_that_runs():
    """The bench labels a mixed run by the tuned table: with no FP32 class on by
    default the mixed path gives the FP64 path's bits, with one it does not."""
    import numpy as np
    import torch
    import bench
    from intception_b200 import basis, eri
    eng = eri.EriEngine(basis.independent_quartet_batch(3, 4000, [0, 1, 2], [2, 3, 5], 0.1, 40.0, 4.0, True))
    bounds = torch.ones(eng.nq, dtype=torch.float64, device='cuda')
    mixed = eng.compute(precision=eri.PREC_MIXED, bounds=bounds, fp32_below=2.0, mixed_tol=1e300).cpu().numpy()
    assert np.array_equal(mixed, eng.compute().cpu().numpy()) == (not bench.fp32_tier_on())


def test_classes_without_an_unrolled_kernel():
    """Up to g shells only (gg|gg), whose tables exceed a block's shared memory,
    and (gg|ss), whose accumulators exceed a lane's registers, are left to the
    generic kernel."""
    emitted = {c for c, _ in eri_emitter.emitted_classes()}
    assert set(eri_emitter.canonical_classes(4)) - emitted == {(4, 4, 4, 4), (4, 4, 0, 0)}
