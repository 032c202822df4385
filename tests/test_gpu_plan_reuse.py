"""The first evaluation of a new plan waits for its own result.

The cached kernel's result comes through pinned host memory with a call
number written last.  The allocator may hand a new plan the memory of a
closed one, whose number must not pass for the new plan's own.
"""
import numpy as np
import pytest

from common import golden_data, load_golden, load_model

pytestmark = pytest.mark.gpu


def _fcn(shift):
    from tf_pwa_b200.api import FCN, EventData

    class Cfg:
        pass

    g, meta = load_golden("lc2pkpi")
    dc, vm, plan = load_model(meta["config"])
    vm.set_all(meta["variables"])
    vm.set_all([v + shift for v in vm.get_all_val()])
    cfg = Cfg()
    cfg.vm, cfg.decay_group, cfg.plan = vm, dc.decay_group, plan
    x, w = golden_data(g, meta)
    return FCN(cfg, EventData(x, w), EventData(g["fields_mc"]), precision="mixed")


def test_first_evaluation_of_a_new_plan(monkeypatch):
    monkeypatch.setenv("PWA_AUTOTUNE", "0")
    seen = []
    for k in range(4):
        fcn = _fcn(0.05 * k)  # one evaluation each: every plan's call number is 1
        seen.append(fcn.nll_grad())
        fcn.eng.close()
    for k, (nll, grad) in enumerate(seen):
        fcn = _fcn(0.05 * k)
        fcn.nll_grad()
        n2, g2 = fcn.nll_grad()  # call number 2: not the closed plans'
        fcn.eng.close()
        assert nll == n2
        assert np.array_equal(grad, g2)
