"""Steps decided on chi^2 by a cluster, where the solve between two passes is
shortest (few free parameters): objects of one and of three chunks of points,
clusters of many sizes, launch after launch bit for bit the one-CTA fits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("dev", "chisq", "period_h", "lambda_deg", "beta_deg", "dark", "totarea", "niter", "err_code")


@pytest.mark.parametrize("n_sparse,n_dense", [(40, 0), (130, 2), (700, 2)])
def test_repeated_cluster_fits(engine_lib, tmp_path, n_sparse, n_dense):
    from periodsearch_gb300 import Engine, PS_FORM_FP64, read_input, synth

    cfg = synth.SynthConfig(name="few", n_sparse=n_sparse, n_dense=n_dense, lmax=2, lmax_truth=2, nrows=3,
                            n_periods=60, stop_condition=25)
    path = tmp_path / "period_search_in"
    synth.write_object(path, cfg, seed=3)
    with Engine(read_input(path), form=PS_FORM_FP64) as eng:
        n = eng.info.slots // 2 + 1
        per, pole = np.arange(n) % 50 + 1, np.arange(n) % 10 + 1
        whole = eng.fit_batch(eng.info.conw_r0, per, pole)
        assert eng.timing()["cluster_size"] == 1
        for k in (3, 9, 19, 36) * 3:
            part = eng.fit_batch(eng.info.conw_r0, per[:k], pole[:k])
            assert eng.timing()["cluster_size"] > 1
            for f in FIELDS:
                np.testing.assert_array_equal(part[f], whole[f][:k], err_msg=f"{k} {f}")
