"""Which kernels a call launches, and how, seen in a captured graph. Environment settings are read once per
process, so each setting has a child of its own."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

OVERLAP = r"""
import json, torch
from aila_b200 import backend as be, linear as nf4
from tests.helpers import captured, make_weight
lin = nf4.Bnb4BitLinear()
assert lin.init(make_weight(1, 512, 512), 0), lin.last_error
sc = nf4.Bnb4BitLinearScratch(0)
sc.ensure(512, 512, 512, True)
bf = dict(dtype=torch.bfloat16, device="cuda")
x, y, cache = torch.ones(512, 512, **bf), torch.ones(512, 512, **bf), torch.ones(1, 64, 64, **bf)
freq, w = torch.ones(32, device="cuda"), torch.ones(64, **bf)
def call():
    for m in (1, 4, 16, 77, 512):
        lin.forward(sc, x, y, m)
    for _ in range(2):
        be.decode_prepare_qkv(y, y[1], y[2], freq, w, w, cache, cache, 3, 4, 1, 64, 1e-6)
        be.attention_decode(y, cache, cache, x, 4, 1, 64, 4)
call()
print(json.dumps(captured(call)))
"""


def child(code, **env):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT, **env),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-1000:] + r.stderr[-3000:]
    return json.loads(r.stdout.splitlines()[-1])


def test_launches_overlap_unless_switched_off():
    names, overlapped = child(OVERLAP)
    assert len(names) == 10 and overlapped >= 8, (names, overlapped)   # (all but the first and the dequantisation pass)
    off_names, off = child(OVERLAP, AILA_NF4_PDL="0")
    assert off_names == names and off == 0, (off_names, off)
