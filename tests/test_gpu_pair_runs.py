"""Which mixed kernel a launch runs, by the kernels' names in a device trace (a
process of its own): two fits per CTA for launches of more fits than fit slots
wherever two slots fit a CTA, whole, screened and packed, also where one fit's
parked relative rows fill the shared memory."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
import torch
from periodsearch_gb300 import Engine, Pack, PS_FORM_MIXED, learned, read_input, synth

n_sparse, n_dense, points, lmax, nrows = map(int, sys.argv[2:7])
cfg = synth.SynthConfig(name="pair", n_sparse=n_sparse, n_dense=n_dense, dense_points=points, lmax=lmax,
                        lmax_truth=lmax, nrows=nrows, n_periods=200, stop_condition=3)
synth.write_object(sys.argv[1], cfg, seed=4)
weights, _ = learned.load_default()
with Engine(read_input(sys.argv[1]), form=PS_FORM_MIXED) as eng, Pack([eng], PS_FORM_MIXED) as pack:
    n, conw = eng.info.slots + 9, eng.info.conw_r0
    per, pole = np.arange(n) % 150 + 1, np.arange(n) % 10 + 1
    calls = {"few": lambda: eng.fit_batch(conw, per[:9], pole[:9]), "fits": lambda: eng.fit_batch(conw, per, pole),
             "screen": lambda: eng.screen(conw, 1, n // 10 + 1, weights, 4),
             "pack": lambda: pack.fit([conw], np.zeros(n, int), per, pole)}
    for name, call in [("warm-up", calls["few"]), *calls.items()]:   # (a process's first trace is empty)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            call()
            torch.cuda.synchronize()
        kernels = [e.key for e in prof.key_averages() if "kernel" in e.key]
        print(name, "pair" if any("_kernel_pair" in k for k in kernels) else "single" if kernels else "none")
"""


@pytest.mark.parametrize("sizes,kind", [((200, 0, 60, 6, 6), "pair"), ((0, 3, 43, 6, 6), "pair"),
                                        ((20, 1, 315, 6, 6), "pair"), ((40, 1, 20, 2, 3), "pair"),
                                        ((100, 0, 60, 6, 7), "single")])
def test_kernel_of_a_launch(engine_lib, tmp_path, sizes, kind):
    r = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "period_search_in"), *map(str, sizes)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = dict(line.split() for line in r.stdout.splitlines() if len(line.split()) == 2)
    del got["warm-up"]
    assert got == {"few": "single", "fits": kind, "screen": kind, "pack": kind}
