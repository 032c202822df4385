"""Which models take the column kernel (pwa_eval_cols) in the plain form, and
what it does at the ends of its inputs.

The route is read from the names of the kernels that ran (and a model that
keeps the general FP64 kernel returns that kernel's sums bit for bit).
Values: as the general kernel within FP64 rounding of columns and sums, 1e-12 of the largest derivative of
each set; what is not a number there is not one here."""
import numpy as np
import pytest

from common import golden_data, load_golden, load_model

pytestmark = pytest.mark.gpu

# 110 KB of shared memory hold (pairs + outputs) x 128 events x 16 bytes:
# epem_cp needs 126 KB, toy_vvp 684 KB
TAKES = {"d2kpipi": True, "lc2pkpi": True, "b2dstkpi": True, "dp2kpipi_ident": True,
         "b2dstkpi_cc": True, "ident_fermions": True, "epem_cp": False, "toy_vvp": False}


class _Plan:
    def __init__(self, case):
        from tf_pwa_b200.engine import Engine

        g, meta = load_golden(case)
        dc, vm, plan = load_model(meta["config"])
        vm.set_all(meta["variables"])
        self.names = list(vm.variables)
        train = [n for n in vm.trainable_vars if not n.endswith(("_mass", "_width"))]
        self.vals = dict(meta["variables"])
        self.x, self.w = golden_data(g, meta)
        self.xm = g["fields_mc"]
        self.eng = Engine(dc.decay_group, plan, vm)
        self.eng.set_host_program(self.names, train)
        self.hp = self.eng.host_program(self.names, train)
        self.P = len(train)
        self.rng = np.random.default_rng(13)

    def upload(self, nd, nm, edit=None):
        i = self.rng.integers(0, self.x.shape[1], nd)
        j = self.rng.integers(0, self.xm.shape[1], nm)
        x, w = self.x[:, i].copy(), self.w[i].copy()
        xm, wm = self.xm[:, j].copy(), self.rng.uniform(0.5, 1.5, nm)
        if edit:
            edit(x, w, xm, wm)
        self.eng.upload(x, w, xm, wm)

    def both(self, vals=None):
        """(piece vector as evaluated, the same from the general kernel)."""
        from tf_pwa_b200.engine import FORM_PLAIN_F64, PLAIN_F64

        vals = vals or self.vals
        v = [vals[n] for n in self.names]
        got = self.eng.pieces_vars(v, FORM_PLAIN_F64)
        sd, sm = self.eng.eval_sums(self.eng.consts(vals), PLAIN_F64)
        return got, self.hp.pieces(v, sd, sm, self.eng._sw)

    def kernels(self):
        """Names of the kernels of one evaluation."""
        import torch
        from torch.profiler import ProfilerActivity, profile

        from tf_pwa_b200.engine import FORM_PLAIN_F64

        v = [self.vals[n] for n in self.names]
        with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as prof:
            self.eng.pieces_vars(v, FORM_PLAIN_F64)
            torch.cuda.synchronize()
        return {e.name for e in prof.events()}

    def close_to(self, got, ref):
        np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
        assert np.allclose(got[:3], ref[:3], rtol=1e-12, atol=0, equal_nan=True)
        for a in (slice(3, 3 + self.P), slice(3 + self.P, 3 + 2 * self.P)):
            d, top = np.abs(got[a] - ref[a]), np.abs(ref[a])
            if not np.isnan(top).all():
                assert np.nanmax(d) <= 1e-12 * np.nanmax(top)

    def close(self):
        self.hp.close()
        self.eng.close()


@pytest.mark.parametrize("case", sorted(TAKES))
def test_route(case):
    p = _Plan(case)
    src = p.eng.src
    fits = (p.eng.code.nf + p.eng.code.nout) * p.eng.tpb * 16 <= 110 * 1024
    assert ("#define PWA_COLS_EVAL 1" in src and fits) == TAKES[case]
    p.upload(40_001, 1000)
    got, ref = p.both()
    p.close_to(got, ref)
    if not TAKES[case]:
        np.testing.assert_array_equal(got, ref)
    ran = p.kernels()
    if not ran:
        pytest.skip("no kernel trace here (another profiler holds it)")
    assert any("pwa_eval_cols" in k for k in ran) == TAKES[case], ran
    assert any("pwa_eval_f64" in k for k in ran) != TAKES[case], ran
    p.close()


@pytest.mark.parametrize("case", ["d2kpipi", "lc2pkpi", "b2dstkpi"])
def test_one_set(case):
    p = _Plan(case)
    for nd, nm in ((1, 0), (129, 0), (40_001, 0), (0, 1), (0, 128), (0, 40_001)):
        p.upload(nd, nm)
        p.close_to(*p.both())
    p.close()


def _nan_data(x, w, xm, wm):
    x[0, 5] = np.nan


def _nan_mc(x, w, xm, wm):
    xm[0, 7] = np.nan


def _no_weight(x, w, xm, wm):
    w[::2] = 0.0
    wm[1::2] = 0.0


@pytest.mark.parametrize("case", ["d2kpipi", "lc2pkpi", "b2dstkpi"])
def test_values_at_the_ends(case):
    p = _Plan(case)
    for edit in (_nan_data, _nan_mc, _no_weight):
        p.upload(300, 1000, edit)
        p.close_to(*p.both())
    # no amplitude at all: the clipped logarithm's value and slope at zero
    p.upload(300, 1000)
    zero = {n: 0.0 if n.endswith("_0r") or n.endswith("r") else v for n, v in p.vals.items()}
    got, ref = p.both(zero)
    assert np.isfinite(got).all()
    p.close_to(got, ref)
    p.close()


@pytest.mark.parametrize("case", ["d2kpipi", "b2dstkpi"])
def test_streams_in_turn(case):
    """One plan, two streams in turn with nothing between the calls: each call
    returns its own point's sums."""
    import torch

    from tf_pwa_b200.engine import FORM_PLAIN_F64

    p = _Plan(case)
    p.upload(2000, 30_000)
    pts = []
    for k in range(3):
        v = {n: x * (1.0 + 0.01 * k) if n.endswith("r") else x for n, x in p.vals.items()}
        pts.append([v[n] for n in p.names])
    want = [p.eng.pieces_vars(v, FORM_PLAIN_F64) for v in pts]
    streams = [torch.cuda.Stream().cuda_stream, torch.cuda.Stream().cuda_stream, 0]
    for k in range(300):
        got = p.eng.pieces_vars(pts[k % 3], FORM_PLAIN_F64, stream=streams[(k // 2) % 3])
        np.testing.assert_array_equal(got, want[k % 3])
    p.close()
