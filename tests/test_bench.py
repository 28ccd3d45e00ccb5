"""The bench's reference arm runs the reference's own code or says that it is not there."""
import json
import os
import subprocess
import sys

import pytest

from oracle import loader

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize('workload', ['eri', 'overlap_2idx'])
def test_reference_arm_without_the_reference(workload):
    if (loader.load_ref('sph') if workload == 'eri' else loader.load_ref_2idx()) is not None:
        pytest.skip('the reference is built here')
    r = subprocess.run([sys.executable, 'bench.py', '--impl', 'reference', '--workload', workload, '--steps', '1',
                        '--warmup', '0'], cwd=ROOT, capture_output=True, text=True, timeout=300)
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert r.returncode == 0 and line['impl'] == 'reference' and line['unavailable'] and 'value' not in line
