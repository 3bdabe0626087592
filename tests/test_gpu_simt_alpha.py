"""The SIMT accumulation of the mixed form's normal matrix (units of four rows
by 32 columns) at the edges of its units and above 4096 elements, and the
basis operand of both tensor-core paths: one evaluation against the oracle
within the mixed form's policy (chi^2 1e-5, alpha 1e-4, beta 1e-3 of their
largest entry)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Laplace degree, facet rows, tensor cores, free Lambert weight: 15 to 107 free
# parameters, around multiples of 4 and 32
@pytest.mark.parametrize("lmax,nrows,tensor,free_cl", [(2, 3, False, 1), (4, 4, False, 1), (5, 5, False, 0),
                                                       (7, 6, False, 0), (8, 7, False, 1), (9, 8, True, 0),
                                                       (9, 7, True, 1), (8, 6, True, 1), (7, 5, True, 0),
                                                       (3, 8, True, 0), (6, 3, True, 1)])
def test_evaluation_against_oracle(engine_lib, oracle, tmp_path, lmax, nrows, tensor, free_cl):
    from periodsearch_gb300 import Engine, PS_FORM_MIXED, read_input, synth

    cfg = synth.SynthConfig(name="alpha", n_sparse=330, n_dense=2, dense_points=45, lmax=lmax, lmax_truth=min(lmax, 6),
                            nrows=nrows, n_periods=50, ia_cl=free_cl)
    path = tmp_path / "period_search_in"
    synth.write_object(path, cfg, seed=lmax)
    ora = oracle.OracleProblem(path)
    conw_r = ora.info()["conw_r"]
    cg = ora.initial_cg(3, 6)
    want = ora.eval(cg)
    with Engine(read_input(path), form=PS_FORM_MIXED, tensor_cores=tensor) as eng:
        got = eng.eval(conw_r, cg)
    for g, w, tol in zip(got, want, (1e-4, 1e-3, 1e-5, 1e-12)):
        assert np.abs(np.asarray(g) - w).max() <= tol * np.abs(w).max()
