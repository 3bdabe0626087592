"""The mixed form off the tensor cores (more than 64 coefficients, basis in
L2): its shape contraction, which takes most of such a fit, at no less than 5 %
of the device's FP32 rate over the whole launch (4 % inlined, sharing its
registers with the partial sums of the normal matrix, 7.5 % as a function)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_simt_contraction_rate(engine_lib, tmp_path):
    from periodsearch_gb300 import Engine, PS_FORM_MIXED, read_input, synth

    cfg = synth.SynthConfig(name="wide", n_sparse=500, n_dense=8, lmax=8, nrows=8, n_periods=200, stop_condition=20)
    path = tmp_path / "period_search_in"
    synth.write_object(path, cfg, seed=5)
    fp64, fp32 = C.c_double(), C.c_double()
    assert engine_lib.ps_device_fma_peaks(0, C.byref(fp64), C.byref(fp32)) == 0
    with Engine(read_input(path), form=PS_FORM_MIXED, tensor_cores=False) as eng:
        n = 2 * eng.info.slots
        per, pole = np.arange(n) % 150 + 1, np.arange(n) % 10 + 1
        ms, i = [], eng.info
        for _ in range(3):
            fits = eng.fit_batch(i.conw_r0, per, pole)
            ms.append(eng.timing()["kernel_ms"])
    flops = 2.0 * i.ndata * i.nfac * i.ncoef * (fits["niter"] + 1).sum()
    assert flops / (min(ms) * 1e-3) >= 0.05 * fp32.value * 1e12
