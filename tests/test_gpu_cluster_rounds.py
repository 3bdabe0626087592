"""Cluster sizes of FP64 launches around the numbers of clusters that a device
of 152 SMs holds at once: every fit has its cluster in one round (there are 36
clusters of 4 CTAs, not 152 / 4), bit for bit the one-CTA fits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("dev", "chisq", "period_h", "lambda_deg", "beta_deg", "dark", "totarea", "niter", "err_code")


@pytest.mark.parametrize("n_sparse", [15, 130])
def test_one_round_of_clusters(engine_lib, tmp_path, n_sparse):
    from periodsearch_gb300 import Engine, PS_FORM_FP64, read_input, synth

    cfg = synth.SynthConfig(name="rounds", n_sparse=n_sparse, lmax=3, lmax_truth=3, nrows=4, n_periods=60,
                            stop_condition=6)
    path = tmp_path / "period_search_in"
    synth.write_object(path, cfg, seed=2)
    with Engine(read_input(path), form=PS_FORM_FP64) as eng:
        if eng.info.slots != 152:
            pytest.skip("another device")
        n = 77
        per, pole = np.arange(n) % 50 + 1, np.arange(n) % 10 + 1
        whole = eng.fit_batch(eng.info.conw_r0, per, pole)
        assert eng.timing()["cluster_size"] == 1
        for k, size in ((36, 4), (37, 3), (38, 3), (76, 2)):
            part = eng.fit_batch(eng.info.conw_r0, per[:k], pole[:k])
            assert eng.timing()["cluster_size"] == size, k
            for f in FIELDS:
                np.testing.assert_array_equal(part[f], whole[f][:k], err_msg=f"{k} {f}")
