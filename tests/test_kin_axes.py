"""The kinematics code on momenta where its axes degenerate, and on moving
parents, against the step-by-step host algorithm (``kinematics.event_fields``,
the reference's), one event at a time on the CPU; and the device kernel's
ways of reading momenta.  Angles within 1e-11 modulo 2 pi (the fold's edge
may fall either way), masses within 1e-12."""
import numpy as np
import pytest

from common import load_model
from hostexec import HostModel


def _host_model(config, tmp):
    from tf_pwa_b200.engine import Engine

    dc, vm, plan = load_model(config)
    eng = Engine(dc.decay_group, plan, vm, compile=False)
    return plan, HostModel(eng.code, str(tmp))


def _boosted(p, beta):
    """Momenta (n, 4) boosted by velocity beta (3,)."""
    b2 = beta @ beta
    g = 1.0 / np.sqrt(1.0 - b2)
    bp = p[:, 1:] @ beta
    k = (g - 1.0) / b2 * bp + g * p[:, 0]
    return np.concatenate([(g * (p[:, 0] + bp))[:, None], p[:, 1:] + k[:, None] * beta], 1)


def _events(plan, rng, n=64):
    """Momenta (n, n_final, 4): random, the total at rest."""
    m = [next(o.mass for o in plan.group.outs if str(o) == f) for f in plan.order]
    p = rng.normal(size=(n, len(m), 3))
    p -= p.mean(1, keepdims=True)
    e = np.sqrt((p ** 2).sum(2) + np.array(m) ** 2)
    return np.concatenate([e[:, :, None], p], 2)


def _compare(plan, hm, p4):
    from tf_pwa_b200.kinematics import event_fields, p4_dict

    ref = event_fields(plan, p4_dict(p4, plan.order)).numpy()
    got = hm.kin(p4)
    for f, a, b in zip(plan.fields, got, ref):
        assert np.array_equal(np.isnan(a), np.isnan(b)), f
        ok = ~np.isnan(b)
        d = np.abs(a - b)[ok]
        if not f.split("|")[-1].startswith("m/"):
            d = np.minimum(d, np.abs(d - 2 * np.pi))
        assert np.all(d < 1e-11), (f, d.max())


@pytest.mark.parametrize("config", ["d2kpipi.yml", "lc2pkpi.yml", "b2dstkpi.yml",
                                    "dp2kpipi_ident.yml", "toy_vvp.yml"])
def test_kinematics_axes(config, tmp_path):
    plan, hm = _host_model(config, tmp_path)
    rng = np.random.default_rng(5)
    p4 = _events(plan, rng)
    _compare(plan, hm, p4)
    # a moving parent
    flat = p4.reshape(-1, 4)
    _compare(plan, hm, _boosted(flat, np.array([0.3, -0.2, 0.4])).reshape(p4.shape))
    # first final along +z and -z: the axes of the decays that hold it alone
    for sign in (1.0, -1.0):
        q = p4[:8].copy()
        q[:, 0, 1:3] = 0.0
        q[:, 0, 3] = sign * np.linalg.norm(p4[:8, 0, 1:], axis=1)
        rest = q[:, 1:, 1:].mean(1, keepdims=True) + q[:, :1, 1:] / (q.shape[1] - 1)
        q[:, 1:, 1:] -= rest
        m = [next(o.mass for o in plan.group.outs if str(o) == f) for f in plan.order]
        q[:, :, 0] = np.sqrt((q[:, :, 1:] ** 2).sum(2) + np.array(m) ** 2)
        _compare(plan, hm, q)


@pytest.mark.gpu
@pytest.mark.parametrize("config", ["d2kpipi.yml", "b2dstkpi.yml"])
def test_momenta_of_any_layout(config):
    import torch

    from tf_pwa_b200.engine import Engine, load_library

    dc, vm, plan = load_model(config)
    eng = Engine(dc.decay_group, plan, vm)
    rng = np.random.default_rng(9)
    for n in (1, 127, 129, 5000):
        p4 = _events(plan, rng, n)
        nf = p4.shape[1]
        t = torch.as_tensor(p4, device="cuda")
        ref = eng.fields_from_p4(t)
        wide = torch.zeros((n, nf, 5), dtype=torch.float64, device="cuda")
        wide[:, :, :4] = t
        odd = torch.zeros(n * nf * 4 + 1, dtype=torch.float64, device="cuda")
        odd[1:] = t.reshape(-1)
        for v in (t.permute(1, 2, 0).contiguous().permute(2, 0, 1),   # component-major
                  t.permute(1, 0, 2).contiguous().permute(1, 0, 2),   # final-major
                  wide[:, :, :4],                                     # padded rows
                  odd[1:].reshape(n, nf, 4),                          # 8-byte aligned only
                  torch.cat([t, t[:, :1]], 1)):                       # a final more than read
            assert torch.equal(eng.fields_from_p4(v), ref)
        soa = t.permute(1, 2, 0).reshape(-1, n).contiguous()
        out = torch.empty_like(ref)
        assert load_library().pwa_fields_from_p4(eng.h, soa.data_ptr(), n, n, out.data_ptr(), n, 0) == 0
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    with pytest.raises(ValueError):
        eng.fields_from_p4(t[:, 1:])
    eng.close()
