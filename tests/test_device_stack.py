"""No device function of the pair bounds recurses: a recursive call's stack is in
no kernel's stack size, so it runs past the end of a thread's local memory."""
import os
import subprocess
import sys

import pytest

from intception_b200 import build

KERNEL = '''
#include "ib_eri_device.cuh"
template <int LA, int LB, int LC, int LD>
__device__ __noinline__ int2 lists(const double* pe, const double* pc, int k, double r2, unsigned char* lst) {
  return ib_live_pairs_screened<LA, LB, LC, LD, true>(pe, pc, 0, k, k, 2 * k, 3 * k, k, r2, r2, 0, k * k, 0, k * k,
                                                      lst, threadIdx.x & 31, 32, 0xffffffffu, 0, 1e-18);
}
__global__ void screened(const double* pe, const double* pc, int k, double r2, int2* out) {
  __shared__ unsigned char lst[256];
  out[threadIdx.x] = lists<%s>(pe, pc, k, r2, lst);
}
'''


@pytest.mark.parametrize('cls', ['2, 2, 2, 2', '4, 4, 4, 4'])
def test_screened_lists_call_no_function(tmp_path, cls):
    src = tmp_path / 'screened.cu'
    src.write_text(KERNEL % cls)
    if not os.path.exists(os.path.join(build.GEN, 'rys_table.h')):
        build._generate()
    cmd = [build.NVCC] + build.ARCH + build.FLAGS + ['-Xptxas', '-v', '-c', str(src), '-o', str(tmp_path / 'o.o')]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    names = [ln.split()[-1] for ln in (r.stdout + r.stderr).splitlines() if 'Function properties for' in ln]
    assert sum('lists' in n for n in names) == 1 and len(names) == 2, names  # the kernel and the function above


ALONE = '''
import numpy as np
from intception_b200 import basis, eri
for nq in (256, 1000):
    eng = eri.EriEngine(basis.independent_quartet_batch(3, nq, [0, 1, 2], [1, 2, 4], 0.05, 100.0, 12.0, True))
    bounds = eng.analytic_bounds()
    eri.set_prim_tol(1e-18)
    out = eng.compute(bounds=bounds, skip_below=1e-12).cpu().numpy()
    eri.set_prim_tol(0.0)
    # screened blocks by 1e-12, up to 4^4 skipped primitives by 1e-18 each
    assert np.abs(out - eng.compute().cpu().numpy()).max() <= 1.001e-12
    assert eng.device_status() == 0
'''


@pytest.mark.gpu
def test_screened_small_batches_in_a_new_process():
    """Alone in a process: no earlier kernel has made the local memory larger."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, '-c', ALONE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
