"""A process with a second CUDA context on the device: a simulation made there runs
as in the first (the coarse cluster launch needs its kernel's attributes set in
each context).  In a child process, which makes the contexts itself."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C, numpy as np
from smokesim_b200 import Sim, abi, scene
cu = C.CDLL("libcuda.so.1")
def ok(rc): assert rc == 0, rc
ok(cu.cuInit(0))
out = []
for dim, n in ((3, (64, 64, 64)), (2, (256, 256, 1))):
    for prec in (abi.PREC_FP32, abi.PREC_MIXED):
        fields = []
        for k in range(2):
            ctx = C.c_void_p()
            ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, 0))
            g = Sim(abi.make_desc(dim, n, cell_size=1.0, density_channels=1, enclosed=1, min_coarse=8))
            r = np.random.default_rng(1)
            for f in (abi.FIELD_VX, abi.FIELD_VY):
                g.set_field(f, r.standard_normal(g.shape(f)).astype(np.float32))
            p = scene.workload_params(ref_quirks=0, precision=prec, n_vcycles=2)
            g.step(p, 2)
            fields.append(g.get_field(abi.FIELD_PRESSURE))
            g.close()
            ok(cu.cuCtxDestroy_v2(ctx))
        assert np.isfinite(fields[0]).all() and np.abs(fields[0]).max() > 0
        assert np.array_equal(*fields)
print("same")
"""


def test_second_context():
    repo = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=repo, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True,
                       timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout
