"""A call that cannot finish reports CUDA's own reason.  A stream under capture
refuses the synchronisation that ends a wait (nothing runs, nothing faults):
every call that returns sums raises with that reason, and the plan evaluates
afterwards exactly as before."""
import ctypes
import time

import numpy as np
import pytest

from common import CONFIGS, load_golden

pytestmark = pytest.mark.gpu

RELAXED = 2  # CU_STREAM_CAPTURE_MODE_RELAXED


class _Capture:
    """`stream` under capture; what was captured is dropped."""

    def __init__(self, stream):
        self.cu, self.s = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(stream.cuda_stream)

    def __enter__(self):
        assert self.cu.cuStreamBeginCapture_v2(self.s, RELAXED) == 0

    def __exit__(self, *exc):
        graph = ctypes.c_void_p()
        if self.cu.cuStreamEndCapture(self.s, ctypes.byref(graph)) == 0 and graph:
            self.cu.cuGraphDestroy(graph)


def _flat(v):
    return np.concatenate([np.ravel(x) for x in (v if isinstance(v, (tuple, list)) else [v])])


@pytest.fixture(scope="module")
def calls():
    import torch

    from tf_pwa_b200.api import FCN, ConfigLoader, EventData
    from tf_pwa_b200.engine import FORM_PLAIN_F64, PLAIN_F64
    from tf_pwa_b200.serving import FitJob, FitServer

    g, meta = load_golden("d2kpipi")
    vals = meta["variables"]
    cl = ConfigLoader(f"{CONFIGS}/{meta['config']}", precision="mixed")
    cl.set_params(vals)
    x = torch.as_tensor(g["fields_data"], device="cuda")
    mc = EventData(torch.as_tensor(g["fields_mc"], device="cuda"))
    truth = np.array(cl.vm.get_all_val())
    fcn = FCN(cl, EventData(x), mc, precision="mixed")
    plain = FCN(cl, EventData(x), mc, precision="plain")
    v = [cl.vm.variables[k] for k in fcn._var_names]
    C = plain.eng.consts(vals)
    srv = FitServer(cl, mc, 1e9, max_active=2, run=False)
    jobs = [srv.submit(FitJob(k, x, truth)) for k in range(2)]
    srv._admit(start=False)
    V = np.repeat(srv.base_vars[None, :], 2, axis=0)
    V[:, srv.train_idx] = truth
    tiles = [[j.tiles[q] for j in jobs] for q in (0, 1)]
    yield {
        "cached": lambda s: fcn.eng.nll_grad_cached(v, stream=s),
        "columns": lambda s: plain.eng.pieces_vars(v, FORM_PLAIN_F64, stream=s),
        "plain": lambda s: plain.eng.eval_sums(C, PLAIN_F64, stream=s),
        "hessian": lambda s: fcn.eng.hessian_cached_exact(v, stream=s),
        "gram": lambda s: plain.eng.build_gram(C, stream=s),
        "batch": lambda s: srv.eng.pieces_multi(*tiles, V, [float(j.n) for j in jobs], stream=s),
    }
    srv.close()
    fcn.eng.close()
    plain.eng.close()


KINDS = ("cached", "columns", "plain", "hessian", "gram", "batch")


@pytest.mark.parametrize("kind", KINDS)
def test_reason_reported(calls, kind):
    import torch

    from tf_pwa_b200.engine import PWAError

    call, stream = calls[kind], torch.cuda.Stream()
    before = _flat(call(stream.cuda_stream))
    with _Capture(stream):
        with pytest.raises(PWAError, match="captur"):
            call(stream.cuda_stream)
    np.testing.assert_array_equal(_flat(call(stream.cuda_stream)), before)


@pytest.mark.parametrize("kind", ("hessian", "gram", "batch"))
def test_capture_refused_at_once(calls, kind):
    """Set-up and service calls synchronise in any case: they refuse a stream
    under capture without polling for a result first (evaluations poll for up
    to a second)."""
    import torch

    from tf_pwa_b200.engine import PWAError

    call, stream = calls[kind], torch.cuda.Stream()
    call(stream.cuda_stream)
    with _Capture(stream):
        t0 = time.perf_counter()
        with pytest.raises(PWAError):
            call(stream.cuda_stream)
        dt = time.perf_counter() - t0
    assert dt < 0.5, dt
