"""Two mixed fits per CTA (launches of more fits than fit slots): every fit bit
for bit the one that the kernel with one fit per CTA gives, whole, screened
and packed; facet grids at the edges of what fits the Tensor Memory of two
slots, relative rows in shared and in global memory, padded facet counts,
Gauss-Jordan fallbacks (relative lightcurves only)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("dev", "chisq", "period_h", "lambda_deg", "beta_deg", "dark", "totarea", "niter", "err_code", "pred_dev")
# sparse points, dense lightcurves, their points, Laplace degree, facet rows
OBJECTS = {"plain": (200, 0, 60, 6, 6), "relative": (0, 3, 43, 6, 6), "long_relative": (20, 1, 700, 6, 5),
           "padded": (61, 2, 33, 3, 7), "small": (40, 1, 20, 2, 3), "too_wide": (100, 0, 60, 6, 7)}


def _engine(tmp_path, name, seed=4, **opt):
    from periodsearch_gb300 import Engine, PS_FORM_MIXED, read_input, synth

    n_sparse, n_dense, points, lmax, nrows = OBJECTS[name]
    cfg = synth.SynthConfig(name=name, n_sparse=n_sparse, n_dense=n_dense, dense_points=points, lmax=lmax,
                            lmax_truth=lmax, nrows=nrows, n_periods=200, stop_condition=9)
    path = tmp_path / f"{name}_{seed}"
    synth.write_object(path, cfg, seed=seed)
    return Engine(read_input(path), form=PS_FORM_MIXED, **opt)


@pytest.mark.parametrize("name", sorted(OBJECTS))
def test_paired_fits_bit_identical(engine_lib, tmp_path, name):
    from periodsearch_gb300 import learned

    weights, _ = learned.load_default()
    with _engine(tmp_path, name) as eng, _engine(tmp_path, name, ctas_per_sm=1) as one:
        assert eng.info.tensor_cores == 1
        conw_r, slots = eng.info.conw_r0, eng.info.slots
        n = 2 * slots + 9
        per, pole = np.arange(n) % 150 + 1, np.arange(n) % 10 + 1
        got, want = eng.fit_batch(conw_r, per, pole), one.fit_batch(conw_r, per, pole)
        few = eng.fit_batch(conw_r, per[:slots], pole[:slots])
        for f in FIELDS:
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
            np.testing.assert_array_equal(few[f], want[f][:slots], err_msg=f)
        hi = (slots + 30) // 10 + 1
        a, b = eng.screen(conw_r, 1, hi, weights, 8), one.screen(conw_r, 1, hi, weights, 8)
        for f in FIELDS:
            np.testing.assert_array_equal(a[f], b[f], err_msg=f)


def test_paired_pack_bit_identical(engine_lib, tmp_path):
    from periodsearch_gb300 import Pack, PS_FORM_MIXED

    engines = [_engine(tmp_path, "plain", seed=s) for s in (4, 5)]
    try:
        slots, conw = engines[0].info.slots, [e.info.conw_r0 for e in engines]
        n = slots + 77
        ob, per, pole = np.arange(n) % 2, np.arange(n) % 90 + 1, np.arange(n) % 10 + 1
        with Pack(engines, PS_FORM_MIXED) as pack:
            got = pack.fit(conw, ob, per, pole)
        for k, e in enumerate(engines):
            want = e.fit_batch(conw[k], per[ob == k], pole[ob == k])
            for f in FIELDS:
                np.testing.assert_array_equal(got[f][ob == k], want[f], err_msg=f)
    finally:
        for e in engines:
            e.close()
