"""A captured pwa_eval_enqueue stays valid beside the plan's other calls on
the same events: building the Gram matrix and evaluating from the columns do
not move the block rows that the captured launch writes.  After replays among
them every call returns its own sums, bit for bit those from before."""
import numpy as np
import pytest

from common import golden_data, load_golden, load_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["d2kpipi", "lc2pkpi", "b2dstkpi"])
def test_replay_beside_other_calls(case):
    import torch

    from tf_pwa_b200.engine import FORM_PLAIN_F64, MIXED_F32, PLAIN_F64, Engine

    g, meta = load_golden(case)
    dc, vm, plan = load_model(meta["config"])
    vm.set_all(meta["variables"])
    names = list(vm.variables)
    train = [n for n in vm.trainable_vars if not n.endswith(("_mass", "_width"))]
    values = [meta["variables"][n] for n in names]
    x, w = golden_data(g, meta)
    xm = g["fields_mc"]
    rng = np.random.default_rng(7)
    i, j = rng.integers(0, x.shape[1], 3000), rng.integers(0, xm.shape[1], 200_000)
    eng = Engine(dc.decay_group, plan, vm)
    eng.set_host_program(names, train)
    eng.upload(x[:, i], w[i], xm[:, j], rng.uniform(0.5, 1.5, len(j)))
    C = eng.consts(meta["variables"])
    before = [eng.eval_sums(C, p) for p in (PLAIN_F64, MIXED_F32)]
    stream = torch.cuda.Stream()
    graphs = []
    for p in (PLAIN_F64, MIXED_F32):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1], stream=stream):
            eng.eval_enqueue(C, p, mc=True, stream=stream.cuda_stream)

    def replay():
        for gr in graphs:
            gr.replay()
        torch.cuda.synchronize()

    pieces, gram = [], []
    for _ in range(3):
        pieces.append(eng.pieces_vars(values, FORM_PLAIN_F64))
        replay()
        gram.append(eng.set_gram(meta["variables"]))
        replay()
    for p, b in zip((PLAIN_F64, MIXED_F32), before):
        for got, want in zip(eng.eval_sums(C, p), b):
            np.testing.assert_array_equal(got, want)
        replay()
    for k in (1, 2):
        np.testing.assert_array_equal(pieces[k], pieces[0])
        np.testing.assert_array_equal(np.asarray(gram[k]), np.asarray(gram[0]))
    del graphs
    eng.close()
