"""Objects whose slot comes within a few hundred bytes of the shared memory of a
CTA, by the length of a relative lightcurve whose rows are parked: each is
prepared, packed and fitted."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# form, Laplace degree, facet rows, lengths of the relative lightcurve
@pytest.mark.parametrize("form,lmax,nrows,lengths", [
    (1, 6, 6, range(302, 320)), (1, 8, 8, range(138, 152)), (1, 8, 9, range(100, 112)), (0, 6, 6, range(86, 106)),
    (0, 8, 8, (20, 21, 58, 59)), (0, 3, 4, (*range(686, 692), *range(750, 757))), (0, 2, 4, range(966, 973)),
    (0, 4, 8, range(29, 34))])
def test_slots_at_the_limit(engine_lib, tmp_path, form, lmax, nrows, lengths):
    from periodsearch_gb300 import Engine, Pack, read_input, synth

    for n in lengths:
        cfg = synth.SynthConfig(name="edge", n_sparse=20, n_dense=1, dense_points=n, lmax=lmax, lmax_truth=2,
                                nrows=nrows, n_periods=60, stop_condition=2)
        path = tmp_path / str(n)
        synth.write_object(path, cfg, seed=1)
        with Engine(read_input(path), form=form) as eng, Pack([eng], form) as pack:
            conw = eng.info.conw_r0
            want = eng.fit_batch(conw, [3], [2])
            got = pack.fit([conw], [0], [3], [2])
            assert np.isfinite(want["dev"]).all()
            for f in ("dev", "chisq", "period_h", "totarea"):
                np.testing.assert_array_equal(got[f], want[f], err_msg=f"{n} {f}")
