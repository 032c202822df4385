"""The one-kernel Gram matrix (columns and products together) against the
oracle's columns, at the edges of its event tiles and for models on both
sides of its dispatch (toy_vvp's tile exceeds a block's shared memory and
keeps the two-kernel form).  Tolerance: FP64 rounding of 40 000-term sums
and of the columns, 1e-12 of the largest entry."""
import numpy as np
import pytest

from common import load_golden, load_model

pytestmark = pytest.mark.gpu

SIZES = (1, 3, 31, 127, 128, 129, 148 * 128 * 2 + 5)


@pytest.mark.parametrize("case", ["d2kpipi", "lc2pkpi", "b2dstkpi", "dp2kpipi_ident",
                                  "b2dstkpi_cc", "toy_vvp"])
def test_gram_fused(case):
    from oracle.pwa_oracle import OracleModel
    from tf_pwa_b200.engine import Engine

    g, meta = load_golden(case)
    dc, vm, plan = load_model(meta["config"])
    vm.set_all(meta["variables"])
    om = OracleModel(dc.decay_group, plan)
    x0 = g["fields_mc"][:, :200]
    F, _ = om.columns(x0, meta["variables"], {})
    F = F.reshape(F.shape[0], F.shape[1], -1)
    eng = Engine(dc.decay_group, plan, vm)
    rng = np.random.default_rng(7)
    for n in SIZES:
        idx = rng.integers(0, x0.shape[1], n)
        w = rng.uniform(0.5, 1.5, n)
        w[1::7] *= -0.2  # negative weights among them; the sum stays positive
        eng.upload(g["fields_data"][:, :5], np.ones(5), x0[:, idx], w)
        M = eng.build_gram(eng.consts(meta["variables"]))
        wn = w / w.sum()
        we = np.bincount(idx, weights=wn, minlength=x0.shape[1])
        ref = np.einsum("n,nko,nlo->kl", we, np.conj(F), F)
        assert np.max(np.abs(M - ref)) <= 1e-12 * np.abs(ref).max(), (case, n)
    eng.close()
