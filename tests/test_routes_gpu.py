"""Which kernels a call launches: the tests of the results cannot tell the routes apart."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import ae296_b200 as L
from lora_testlib import Case

pytestmark = pytest.mark.gpu


def launched(fn):
    """Names of the kernels that one call of ``fn`` launches, in order."""
    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    events = sorted((e for e in prof.events() if "_kernel" in e.name), key=lambda e: e.time_range.start)
    if not events:
        pytest.skip("kernel tracing is not available here")
    return [e.name for e in events]


def kinds(names):
    known = ("plan_build", "bgmv_cluster", "bgmv_shrink_tma", "bgmv_expand_tma", "bgmv_shrink", "bgmv_expand")
    return [next((k for k in known if k in n), n) for n in names]


@pytest.mark.parametrize("kind,T,want", [
    ("packed", 12, ["bgmv_cluster"]),                           # few tokens: one launch
    ("packed", 200, ["bgmv_shrink_tma", "bgmv_expand_tma"]),
    ("padded", 12, ["bgmv_shrink_tma", "bgmv_expand_tma"]),     # ranks below R
    ("general", 12, ["bgmv_shrink", "bgmv_expand"]),            # widths that are no multiple of 128
])
def test_kernels_of_an_apply(kind, T, want):
    h = 328 if kind == "general" else 1024
    ranks = [12, 40] if kind == "padded" else [16]
    c = Case(T, 12, h, h, np.resize(np.array(ranks, np.int32), 12), "fp16", dense=kind == "padded", seed=T)
    batch = L.LoraBatch(T, 12, h, 1).set_ids(c.ids_dev, c.pool)
    y = torch.zeros(T, h, dtype=torch.float16, device="cuda")
    names = launched(lambda: batch.apply([(c.x, y, c.pool)], 0))
    assert kinds(names) == want


@pytest.mark.parametrize("T,want", [(7, ["bgmv_cluster"]), (64, ["plan_build", "bgmv_shrink_tma", "bgmv_expand_tma"])])
def test_kernels_of_a_static_call(T, want):
    c = Case(T, 12, 4096, 4096, 16, "fp16", dense=True, seed=T)
    y = torch.zeros(T, 4096, dtype=torch.float16, device="cuda")
    names = launched(lambda: L.add_lora_bgmv_static(y, c.x, c.pool.wa, c.pool.wb, c.ids_dev, 0, 1.0))
    assert kinds(names) == want
