"""Engine.fields_from_p4 hands the library a pointer and the tensor's own
strides: what is read through them equals the tensor's values, for every kind
of view (host tensors, the library call recorded)."""
import ctypes

import numpy as np
import pytest
import torch

from common import load_model


class _Recorder:
    """Reads the momenta as pwa_fields_from_strided would."""

    def __init__(self, n_final):
        self.n_final, self.seen = n_final, None

    def pwa_fields_from_strided(self, h, p4, n, se, sf, sc, out, ld_out, stream):
        a = np.empty((n, self.n_final, 4))
        for i, f, c in np.ndindex(*a.shape):
            a[i, f, c] = ctypes.c_double.from_address(p4 + 8 * (i * se + f * sf + c * sc)).value
        self.seen = a
        return 0


def _views(v):
    z = torch.complex(torch.zeros_like(v), -v)
    wide = torch.zeros((v.shape[0], v.shape[1], 6), dtype=v.dtype)
    wide[:, :, 1:5] = v
    return {
        "plain": v,
        "component-major": v.permute(1, 2, 0).contiguous().permute(2, 0, 1),
        "inside wider rows": wide[:, :, 1:5],
        "every other event": v.repeat_interleave(2, 0)[::2],
        "one event expanded": v[:1].expand(3, -1, -1),
        "float32": v.to(torch.float32),
        "lazily negated": z.conj().imag,
        "no events": v[:0],
    }


@pytest.mark.parametrize("kind", list(_views(torch.zeros(2, 3, 4, dtype=torch.float64))))
def test_values_read(kind, monkeypatch):
    from tf_pwa_b200 import engine

    dc, vm, plan = load_model("d2kpipi.yml")
    eng = engine.Engine(dc.decay_group, plan, vm, compile=False)
    nfin = eng.code.kin.nfin
    v = torch.as_tensor(np.random.default_rng(5).normal(size=(5, nfin, 4)))
    p4 = _views(v)[kind]
    lib = _Recorder(nfin)
    monkeypatch.setattr(engine, "load_library", lambda: lib)
    out = eng.fields_from_p4(p4)
    monkeypatch.undo()
    assert out.shape == (plan.n_fields, p4.shape[0])
    np.testing.assert_array_equal(lib.seen, p4.to(torch.float64).resolve_neg().numpy())
