"""FP64 fits and evaluations on clusters of up to 16 CTAs: the cluster sizes
that small launches get (as many CTAs per fit as leave every fit a resident
cluster), bit for bit the one-CTA fits; objects with fewer tiles than CTAs,
with a relative lightcurve longer than the staging area, and with more
lightcurves than a set-up group has warps.  Evaluations against the oracle
(1e-10, the FP64 policy)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("dev", "chisq", "period_h", "lambda_deg", "beta_deg", "dark", "totarea", "niter", "err_code")
OBJECTS = {"two_tiles": (33, 0, 60), "long_relative": (0, 1, 450), "many": (5, 17, 33)}


@pytest.mark.parametrize("name", sorted(OBJECTS))
def test_cluster_fits_and_evaluation(engine_lib, oracle, tmp_path, name):
    from periodsearch_gb300 import Engine, PS_FORM_FP64, read_input, synth

    n_sparse, n_dense, points = OBJECTS[name]
    cfg = synth.SynthConfig(name=name, n_sparse=n_sparse, n_dense=n_dense, dense_points=points, n_periods=60,
                            stop_condition=7)
    path = tmp_path / "period_search_in"
    synth.write_object(path, cfg, seed=5)
    ora = oracle.OracleProblem(path)
    conw_r = ora.info()["conw_r"]
    with Engine(read_input(path), form=PS_FORM_FP64) as eng:
        n = eng.info.slots // 2 + 1
        per, pole = np.arange(n) % 50 + 1, np.arange(n) % 10 + 1
        whole = eng.fit_batch(conw_r, per, pole)
        assert eng.timing()["cluster_size"] == 1
        sizes = set()
        for k in (1, 7, 8, 13, 15, 23, 28, 36, 46):
            part = eng.fit_batch(conw_r, per[:k], pole[:k])
            sizes.add(eng.timing()["cluster_size"])
            for f in FIELDS:
                np.testing.assert_array_equal(part[f], whole[f][:k], err_msg=f"{name} {k} {f}")
        assert (max(sizes) > 4) == (name != "two_tiles")
        cg = ora.initial_cg(3, 6)
        got, want = eng.eval(conw_r, cg), ora.eval(cg)
        for g, w in zip(got, want):
            assert np.abs(np.asarray(g) - w).max() <= 1e-10 * np.abs(w).max()
