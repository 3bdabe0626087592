"""Steps decided on chi^2 alone (chi2_fp64, chi2_mixed: alpha and beta are
evaluated for accepted steps only), at the sizes where their chunks and tiles
end: below, at and above a chunk of points, relative lightcurves of odd
lengths, longer than a chunk and longer than the buffer (which falls back to
whole evaluations), more lightcurves than warps.

Fits of two LM steps against the oracle.  FP64: one evaluation agrees within
1e-10 and two steps amplify that little (12 steps stay within 1e-12 on the
traced fits): 1e-8.  Mixed form: one evaluation's chi^2 is within 1e-5, its
alpha within 1e-4; a left-out or misplaced tile moves chi^2 by percents:
5e-3."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(383, 0, 60, 6), (385, 0, 60, 6), (40, 3, 33, 3), (1000, 20, 31, 6), (70, 1, 385, 6), (1300, 1, 1000, 6),
         (0, 17, 64, 8)]


@pytest.mark.parametrize("n_sparse,n_dense,points,nrows", SIZES)
def test_steps_against_oracle(engine_lib, oracle, tmp_path, n_sparse, n_dense, points, nrows):
    from periodsearch_gb300 import Engine, PS_FORM_FP64, PS_FORM_MIXED, read_input, synth

    cfg = synth.SynthConfig(name="steps", n_sparse=n_sparse, n_dense=n_dense, dense_points=points, nrows=nrows,
                            n_periods=50, stop_condition=2, sparse_block=500)
    path = tmp_path / "period_search_in"
    synth.write_object(path, cfg, seed=n_sparse + points)
    ora = oracle.OracleProblem(path)
    conw_r = ora.info()["conw_r"]
    want = [ora.fit_n(7, pole) for pole in range(1, 11)]
    data = read_input(path)
    for form, tol in ((PS_FORM_FP64, 1e-8), (PS_FORM_MIXED, 5e-3)):
        with Engine(data, form=form) as eng:
            got = eng.fit_batch(conw_r, np.full(10, 7), np.arange(1, 11))
        for g, w in ((got["chisq"], "chisq"), (got["dev"], "dev"), (got["totarea"], "totarea")):
            np.testing.assert_allclose(g, [x[w] for x in want], rtol=tol)
