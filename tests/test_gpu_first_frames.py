"""The first frames of a simulation solved to a tolerance on the default stream:
its tolerance loop runs on the host, so that a new simulation does not pay for
recording the device loop's graphs there (SMOKESIM_DEVICE_LOOP=0 runs the host loop
by request: the same calls, so the same time; the graphs double it)."""
import time

import numpy as np
import pytest

from smokesim_b200 import abi, scene

pytestmark = pytest.mark.gpu


def test_first_frames_on_the_default_stream(monkeypatch):
    import torch
    from smokesim_b200 import Sim
    p = scene.workload_params(ref_quirks=0, precision=abi.PREC_MIXED, tol=1e-6, n_vcycles=40)
    r = np.random.default_rng(3)
    vel = [r.standard_normal(k).astype(np.float32) for k in (257 * 256, 256 * 257)]

    def two_frames(loop):
        monkeypatch.setenv("SMOKESIM_DEVICE_LOOP", loop)
        g = Sim(abi.make_desc(2, (256, 256, 1), cell_size=1.0, density_channels=1, enclosed=1, min_coarse=8))
        for f, a in zip((abi.FIELD_VX, abi.FIELD_VY), vel):
            g.set_field(f, a)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(2):
            g.step(p)
        torch.cuda.synchronize()
        t = time.perf_counter() - t0
        assert g.stats().vcycles > 0
        g.close()
        return t

    two_frames("1"), two_frames("0")
    # the quickest of nine, in turn: the machine's other work only ever adds time
    t = np.array([[two_frames("1"), two_frames("0")] for _ in range(9)]).min(0)
    assert t[0] <= 1.4 * t[1], t
