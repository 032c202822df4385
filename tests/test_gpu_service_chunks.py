"""One launch over many fits: fit sizes around its tiles (128 events), chunks
(a fit of up to 128 tiles has one-tile chunks, 129 tiles two-tile ones) and
groups of chunks.  A fit's pieces are bitwise the same alone, in any order
and beside other fits, and equal the one-fit cached path's, which forms the
same FP32 sums per warp and tile (FP64 from there on: 1e-12 of the largest
derivative)."""
import numpy as np
import pytest

from common import CONFIGS, load_golden

pytestmark = pytest.mark.gpu

SIZES = (1, 31, 128, 129, 1024, 1025, 16_384, 16_385, 40_000)


@pytest.mark.parametrize("case", ["d2kpipi", "lc2pkpi", "b2dstkpi"])
def test_service_chunks(case):
    import torch

    from tf_pwa_b200.api import FCN, ConfigLoader, EventData
    from tf_pwa_b200.serving import FitJob, FitServer

    g, meta = load_golden(case)
    cl = ConfigLoader(f"{CONFIGS}/{meta['config']}", precision="mixed")
    cl.set_params(meta["variables"])
    rng = np.random.default_rng(11)
    x = torch.as_tensor(g["fields_data"], device="cuda")
    mc = EventData(torch.as_tensor(g["fields_mc"], device="cuda"))
    truth = np.array(cl.vm.get_all_val())
    fields = [x[:, torch.as_tensor(rng.integers(0, x.shape[1], n), device="cuda")].contiguous()
              for n in SIZES]
    srv = FitServer(cl, mc, 1e9, max_active=len(SIZES), run=False)
    jobs = [srv.submit(FitJob(i, f, truth + rng.normal(0, 0.1, truth.shape)))
            for i, f in enumerate(fields)]
    srv._admit(start=False)
    V = np.repeat(srv.base_vars[None, :], len(jobs), axis=0)
    for r, j in enumerate(jobs):
        V[r, srv.train_idx] = j.x0

    def run(order):
        out = srv.eng.pieces_multi([jobs[r].tiles[0] for r in order],
                                   [jobs[r].tiles[1] for r in order], V[order],
                                   [float(jobs[r].n) for r in order])
        return {r: row for r, row in zip(order, out)}

    order = list(range(len(jobs)))
    batch = run(order)
    for other in (order[::-1], list(rng.permutation(order)), order[::2]):
        got = run([int(r) for r in other])
        for r, row in got.items():
            assert np.array_equal(row, batch[r]), (case, SIZES[r])
    for r, f in enumerate(fields):
        assert np.array_equal(run([r])[r], batch[r]), (case, SIZES[r])
    # more requests than the plan's own pinned block holds arguments for
    many = order * 40
    out = srv.eng.pieces_multi([jobs[r].tiles[0] for r in many], [jobs[r].tiles[1] for r in many],
                               V[many], [float(jobs[r].n) for r in many])
    for r, row in zip(many, out):
        assert np.array_equal(row, batch[r])
    srv.close()
    P = len(truth)
    for r, f in enumerate(fields):
        cl.set_params(meta["variables"])
        fcn = FCN(cl, EventData(f), mc, precision="mixed")
        fcn.eng.set_cached_variant(2)
        ref = fcn.eng.pieces_cached(V[r])
        fcn.eng.close()
        assert np.allclose(batch[r][:3], ref[:3], rtol=1e-12, atol=0), (case, SIZES[r])
        for a in (slice(3, 3 + P), slice(3 + P, 3 + 2 * P)):
            assert np.max(np.abs(batch[r][a] - ref[a])) <= 1e-12 * np.abs(ref[a]).max()
