"""The plain FP64 evaluation from the columns (no mass or width free) against
the general FP64 kernel's sums through the same chain rule, at set sizes
around its tiles of 128 events and for every kind of model that takes it
(identical-particle swaps, per-event charges; toy_vvp's columns exceed a
block's shared memory and keep the general kernel).  Tolerance: FP64
rounding of the columns and of sums of up to 4e4 terms, 1e-12 of the largest
derivative of each set."""
import numpy as np
import pytest

from common import golden_data, load_golden, load_model

pytestmark = pytest.mark.gpu

SIZES = ((1, 1), (1, 300), (127, 129), (128, 128), (129, 1), (2000, 31), (31, 40_001),
         (40_001, 1000))


@pytest.mark.parametrize("case", ["d2kpipi", "lc2pkpi", "b2dstkpi", "dp2kpipi_ident",
                                  "b2dstkpi_cc", "ident_fermions", "epem_cp", "toy_vvp"])
def test_eval_cols(case):
    from tf_pwa_b200.engine import FORM_PLAIN_F64, PLAIN_F64, Engine

    g, meta = load_golden(case)
    dc, vm, plan = load_model(meta["config"])
    vm.set_all(meta["variables"])
    names = list(vm.variables)
    train = [n for n in vm.trainable_vars if not n.endswith(("_mass", "_width"))]
    values = [meta["variables"][n] for n in names]
    x, w = golden_data(g, meta)
    xm = g["fields_mc"]
    eng = Engine(dc.decay_group, plan, vm)
    eng.set_host_program(names, train)
    hp = eng.host_program(names, train)
    rng = np.random.default_rng(3)
    P = len(train)
    for nd, nm in SIZES:
        i, j = rng.integers(0, x.shape[1], nd), rng.integers(0, xm.shape[1], nm)
        wm = rng.uniform(0.5, 1.5, nm)
        eng.upload(x[:, i], w[i], xm[:, j], wm)
        got = eng.pieces_vars(values, FORM_PLAIN_F64)
        sd, sm = eng.eval_sums(eng.consts(meta["variables"]), PLAIN_F64)
        ref = hp.pieces(values, sd, sm, eng._sw)
        assert np.allclose(got[:3], ref[:3], rtol=1e-12, atol=0), (case, nd, nm)
        for a in (slice(3, 3 + P), slice(3 + P, 3 + 2 * P)):
            assert np.max(np.abs(got[a] - ref[a])) <= 1e-12 * np.abs(ref[a]).max(), (case, nd, nm)
    hp.close()
    eng.close()
