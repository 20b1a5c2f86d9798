"""mlb_init loads the library's modules, not every kernel in them: a kernel is loaded
by its first launch.  Seen by the device memory that init takes in a fresh process:
46 MB when it set the limits of every kernel, 2 MB now."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _fresh(code):
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert out.returncode == 0, out.stderr
    return out.stdout.strip().splitlines()[-1]


def test_memory_of_init():
    mb = float(_fresh("import torch; torch.zeros(1, device='cuda'); torch.cuda.synchronize();"
                      "a = torch.cuda.mem_get_info()[0]; import maglua_b200 as M; M.init(0);"
                      "print((a - torch.cuda.mem_get_info()[0]) / 2**20)"))
    assert mb <= 16


@pytest.mark.parametrize("dims,precision", [((32, 8, 2), "f32"), ((34, 6, 2), "f64"), ((512, 4, 1), "f32")])
def test_first_call_is_a_captured_run(dims, precision):
    """A run, a scheme's graph step and a plan as the first calls of a process: their
    kernels are loaded while they are captured."""
    code = ("import numpy as np, maglua_b200 as M; M.init(0);"
            "dims, prec = %r, %r; n = int(np.prod(dims)); llg = M.LLG.new('Quaternion');"
            "ss = M.SpinSystem(*dims, precision=prec); ss.setSpinArrays(np.zeros(n), np.full(n, .6), np.full(n, .8));"
            "ss.setTimeStep(0.01); dip = M.Dipole(ss); dip.setTruncation(4);"
            "ani = M.Anisotropy(ss); ani.addMany(np.arange(n), np.tile([1.0, 0, 0], (n, 1)), np.full(n, .1));"
            "M.run(ss, [ani, dip], llg, 30);"
            "rk = M.RungeKutta(ss, 'RK4', [ani, dip], llg); rk.step(4);"
            "M.Plan(ss, [ani, dip], llg).launch(9);"
            "print(ss.status(), np.abs(np.stack(ss.spinArrays()[:3])).max())") % (dims, precision)
    status, top = _fresh(code).split()
    assert status == "0" and 0 < float(top) <= 1.000001
