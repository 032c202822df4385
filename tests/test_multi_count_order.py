"""The service kernel hands rows from block to block by counters: one lane
adds to a counter, then a whole warp reads rows that other blocks wrote.  A
vote or a shuffle orders no memory, so between that lane's count and the
warp's reads stand its fence and a warp barrier, and before a count stands a
fence behind the barrier that ends the block's writes.  (Read from the source:
the order of what the kernel does cannot be provoked by running it.)"""
import os
import re

from common import ROOT


def _steps():
    with open(os.path.join(ROOT, "tf-pwa_b200", "csrc", "pwa_kernels.cuh")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[text.index("    pwa_eval_multi(const long long*"):]
    body = body[:body.index("\n}\n")]
    kinds = ("__syncthreads()", "__threadfence()", "__threadfence_system()", "__syncwarp()",
             "atomicAdd(count + g,", "atomicAdd(count + n_groups + qq,",
             "atomicAdd(count + n_groups + n_req,", "__ballot_sync", "__shfl_sync",
             "multi_sum_rows(rows", "multi_sum_rows(grow", "(double)seq")
    found = sorted((m.start(), k) for k in kinds for m in re.finditer(re.escape(k), body))
    return [k for _, k in found]


def _between(steps, a, b):
    i = steps.index(a)
    return steps[i + 1:steps.index(b, i)]


def _ordered(part, *want):
    it = iter(part)
    return all(w in it for w in want)


def test_counts_order_the_rows():
    s = _steps()
    # the block's rows -> its count
    assert _ordered(_between(s, "__syncthreads()", "atomicAdd(count + g,"), "__threadfence()")
    # a full group's count -> the warp's reads of its rows
    assert _ordered(_between(s, "atomicAdd(count + g,", "multi_sum_rows(rows"),
                    "__threadfence()", "__syncwarp()")
    # the group's row -> the request's count -> the warp's reads of the group rows
    assert _ordered(_between(s, "multi_sum_rows(rows", "atomicAdd(count + n_groups + qq,"),
                    "__threadfence()")
    assert _ordered(_between(s, "atomicAdd(count + n_groups + qq,", "multi_sum_rows(grow"),
                    "__threadfence()", "__syncwarp()")
    # a request's sums in host memory -> its count -> the call number
    assert _ordered(_between(s, "multi_sum_rows(grow", "atomicAdd(count + n_groups + n_req,"),
                    "__threadfence_system()")
    assert _ordered(_between(s, "atomicAdd(count + n_groups + n_req,", "(double)seq"),
                    "__threadfence_system()")
