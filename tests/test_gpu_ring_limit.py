"""The column cache of a model whose ring of three tiles leaves less shared
memory than the streaming kernel's own arrays take: the ring variant does not
exist for it, and the cache is built and evaluated by the others (36 columns
of one output in tiles of 256 events: 222 KB of a block's 227)."""
import numpy as np
import pytest
import yaml

from common import CONFIGS

pytestmark = pytest.mark.gpu


def _config(n):
    with open(f"{CONFIGS}/d2kpipi.yml") as f:
        c = yaml.safe_load(f)
    c["particle"] = {k: v for k, v in c["particle"].items() if k.startswith("$")}
    c["decay"] = {"A": [[f"R{i}", "D"] for i in range(n)]}
    for i in range(n):
        c["decay"][f"R{i}"] = ["B", "C"]
        c["particle"][f"R{i}"] = {"J": i % 2, "P": (-1) ** (i % 2), "mass": 0.7 + 0.01 * i,
                                  "model": "one"}
    return c


def test_cache_beside_the_limit():
    from tf_pwa_b200.api import ConfigLoader
    from tf_pwa_b200.engine import FORM_PLAIN_F64, Engine
    from tf_pwa_b200.workload import generate

    cl = ConfigLoader(_config(36))
    rng = np.random.default_rng(2)
    cl.vm.set_all({n: float(rng.uniform(0.5, 1.5)) for n in cl.vm.trainable_vars})
    eng = Engine(cl.decay_group, cl.plan, cl.vm, tpb=256)
    assert eng.code.nf == 36
    x = generate(eng, 6000, 3)[0].cpu().numpy()
    eng.upload(x[:, :1000], np.ones(1000), x[:, 1000:])
    vals = cl.vm.get_all_dic()
    names, train = list(cl.vm.variables), list(cl.vm.trainable_vars)
    v = [cl.vm.variables[n] for n in names]
    eng.set_host_program(names, train)
    ref = eng.pieces_vars(v, FORM_PLAIN_F64)
    eng.set_gram(vals)
    eng.cache_data(vals)
    eng.set_param_layout(names, train)
    # FP32 columns and warp sums: as the cached form's tests on the golden models
    for variant in (0, 1, 2, 3):
        eng.set_cached_variant(variant)
        got = eng.pieces_cached(v)
        assert np.allclose(got[:3], ref[:3], rtol=1e-6), variant
        P = len(train)
        for a in (slice(3, 3 + P), slice(3 + P, 3 + 2 * P)):
            assert np.max(np.abs(got[a] - ref[a])) <= 1e-6 * np.abs(ref[a]).max(), variant
    eng.close()
