"""Tensors that the native host path cannot read: a Python exception, as the same access raises in Python, and a
process that goes on (one of its own here, because the failure guarded against ends it)."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import types, numpy as np, torch
import ae296_b200 as L
from ae296_b200 import _lib
from torch._subclasses.fake_tensor import FakeTensorMode
host = _lib.host()

def fake(*shape, dtype=torch.float16):           # a CUDA tensor without storage, on any machine
    with FakeTensorMode(allow_non_fake_inputs=True):
        return torch.empty(*shape, dtype=dtype, device="cuda")

def raises(fn):
    try:
        fn()
    except Exception as e:
        print("raised", type(e).__name__, flush=True)
        return
    raise SystemExit("nothing raised")

ids = fake(2, dtype=torch.int32)
x, y, wa, wb = fake(2, 128), fake(2, 128), fake(1, 1, 8, 128), fake(1, 1, 128, 8)
pool = types.SimpleNamespace(wa=wa, wb=wb, h_in=128, h_out=128, ranks=None, scalings=None, cum_ranks=None, n_adapters=1,
                             n_layers=1, r_pool=8, packed=False, ranks_host=np.full(1, 8, np.int32),
                             cum_host=np.array([0, 8]))
plan = types.SimpleNamespace(buf=fake(512, dtype=torch.int64), nbytes=4096, max_tokens=2, n_tokens=2)
ws = types.SimpleNamespace(buf=fake(4096, dtype=torch.uint8), nbytes=4096)
ad = L.ops._adapters_struct(1, 1, 8)
"""

CASES = {
    "static": "raises(lambda: L.add_lora_bgmv_static(y, x, wa, wb, ids, 0, 1.0))",
    "operator": "raises(lambda: host.bgmv(y, x, wa, wb, ids, 0, 1.0))",
    "apply": "raises(lambda: host.apply([(x, y, pool)], plan, 0, ws, 2, ad))",
    "apply_vmap": "raises(lambda: torch.vmap(lambda a: host.apply([(a, y, pool)], plan, 0, ws, 2, ad) and a)(fake(3, 2, 128)))",
    "plan_build": "raises(lambda: host.plan_build(plan, ids, ad))",
    "plan_segments": "raises(lambda: host.plan_segments(plan, fake(2, dtype=torch.int32), fake(1, dtype=torch.int32), 2, ad))",
}


def test_unreadable_tensors_raise_and_the_process_goes_on():
    code = PRELUDE + "".join(f"print({name!r}); {call}\n" for name, call in CASES.items()) + "print('still here')\n"
    res = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr[-2000:]
    assert res.stdout.count("raised") == len(CASES) and "still here" in res.stdout
