"""Every function of a model's GPU source is called by a kernel (or by a
function that one calls): what only the host tests use stands between
#ifndef __CUDACC__ and #endif, which the GPU build skips."""
import os
import re

import pytest

from common import ROOT, load_model


def _strip(text):
    text = re.sub(r"#ifndef __CUDACC__\n.*?\n#endif\n", "", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


@pytest.mark.parametrize("cfg", ["d2kpipi.yml", "lc2pkpi.yml", "d2kpipi_float.yml",
                                 "lc2pkpi_pol.yml"])
def test_every_model_function_is_called(cfg):
    from tf_pwa_b200.engine import Engine

    dc, vm, plan = load_model(cfg)
    src = _strip(Engine(dc.decay_group, plan, vm, compile=False).code.source())
    with open(os.path.join(ROOT, "tf-pwa_b200", "csrc", "pwa_kernels.cuh")) as f:
        text = src + _strip(f.read())
    names = set(re.findall(r"__device__ __forceinline__ \w+(?:<\w+>)?\*? (model_\w+)\(", src))
    assert {"model_amp", "model_columns", "model_bw", "model_cols_ns"} <= names
    for n in sorted(names):
        uses = len(re.findall(rf"\b{n}\b", text)) - len(
            re.findall(rf"__device__ __forceinline__ [^\n(]*\b{n}\(", text))
        assert uses > 0, n
