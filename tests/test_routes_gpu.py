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


ROUTES = r"""
import json, re, torch
from aila_b200 import linear as nf4
from tests.helpers import captured, make_weight
lin = nf4.Bnb4BitLinear()
assert lin.init(make_weight(1, 512, 2048), 0), lin.last_error
sc = nf4.Bnb4BitLinearScratch(0)
sc.ensure(512, 2048, 512, True)
x, y = (torch.ones(512, k, dtype=torch.bfloat16, device="cuda") for k in (2048, 512))
def route(m):
    lin.forward(sc, x, y, m)
    names = [n for n in captured(lambda: lin.forward(sc, x, y, m))[0] if "dequant" not in n]
    kinds = {re.search("gemv_stream|gemv_rows|gemm_midrows|gemm_bf16_tcgen05_kernelILb[01]", n)[0] for n in names}
    assert len(kinds) == 1, names
    return kinds.pop()
print(json.dumps({m: route(m) for m in (4, 9, 17, 32, 48, 49, 77, 300, 385)}))
"""
STREAM, SLICED, MID, GEMM, FUSED = ("gemv_stream", "gemv_rows", "gemm_midrows", "gemm_bf16_tcgen05_kernelILb0",
                                    "gemm_bf16_tcgen05_kernelILb1")


@pytest.mark.parametrize("env,want", [
    ({}, [STREAM] + [MID] * 7 + [GEMM]),
    (dict(AILA_NF4_DECODE_ROWS_MAX="17"), [STREAM, SLICED, SLICED, MID, MID, MID, MID, MID, GEMM]),
    (dict(AILA_NF4_DECODE_ROWS_MAX="48"), [STREAM] + [SLICED] * 4 + [MID] * 3 + [GEMM]),
    (dict(AILA_NF4_DECODE_ROWS_MAX="0"), [GEMM] + [MID] * 7 + [GEMM]),
    (dict(AILA_NF4_ROWS_KERNEL="0"), [STREAM] * 5 + [MID] * 3 + [GEMM]),
    (dict(AILA_NF4_ROWS_KERNEL="1"), [SLICED] * 5 + [MID] * 3 + [GEMM]),
    (dict(AILA_NF4_ROWS_KERNEL="2"), [STREAM] + [MID] * 7 + [GEMM]),
    (dict(AILA_NF4_FUSED_PREFILL="0"), [STREAM] + [MID] * 4 + [GEMM] * 4),
    (dict(AILA_NF4_FUSED_PREFILL="1"), [STREAM] + [MID] * 4 + [FUSED] * 4),
    (dict(AILA_NF4_MID_ROWS_MIN="49", AILA_NF4_MID_ROWS_MAX="77"), [STREAM] + [SLICED] * 4 + [MID] * 2 + [GEMM] * 2),
    (dict(AILA_NF4_MID_ROWS_MAX="0"), [STREAM] + [SLICED] * 4 + [GEMM] * 4)],
    ids=lambda v: "-".join(f"{k[9:]}={n}" for k, n in v.items()) or "default" if isinstance(v, dict) else "")
def test_settings_choose_the_kernel(env, want):
    assert list(child(ROUTES, **env).values()) == want


@pytest.mark.parametrize("n,k,rows,want", [
    (18944, 256, (9, 49, 256), [MID] * 3), (18945, 256, (9, 17, 48, 49), [SLICED, MID, MID, GEMM]),
    (18945, 192, (48,), [SLICED]), (18945, 448, (256,), [GEMM]), (18945, 512, (16, 17, 256, 257), [SLICED, MID, MID, GEMM]),
    (18945, 960, (16, 384), [SLICED, GEMM]), (18945, 1024, (9, 384), [MID, GEMM]),
    (512, 1472, (256, 257), [MID, GEMM]), (512, 1536, (256, 257), [MID, MID]), (65536, 1024, (384,), [MID])])
def test_shapes_choose_the_kernel(n, k, rows, want):
    """Both sides of every line of the rule, 148 tiles of 128 rows and one more among them."""
    import re

    import torch

    from aila_b200 import linear as nf4, synth
    from tests.helpers import captured
    packed = torch.randint(256, (n * k // 2,), dtype=torch.uint8).numpy()
    w = synth.Nf4Tensors(n, k, 64, packed, None, torch.ones(n * k // 64).numpy(), synth.nf4_codebook(), None, None)
    lin = nf4.Bnb4BitLinear()
    assert lin.init(w, 0), lin.last_error
    sc = nf4.Bnb4BitLinearScratch(0)
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes for 148 SMs")
    got = []
    for m in rows:
        x, y = (torch.zeros(m, c, dtype=torch.bfloat16, device="cuda") for c in (k, n))
        lin.forward(sc, x, y, m)
        names = captured(lambda: lin.forward(sc, x, y, m))[0]
        got.append(re.search("gemv_stream|gemv_rows|gemm_midrows|gemm_bf16_tcgen05_kernelILb[01]", names[-1])[0])
    assert got == want
    lin.close()
    sc.close()


def test_gemm_route_at_fewer_rows():
    """The prefill tests at 49 to 384 rows once more with the tensor-memory kernel switched off: the dequantisation
    pass and the GEMM's 128-row tiles, which serve linears that the kernel does not take."""
    r = subprocess.run([sys.executable, "-m", "pytest", "tests/test_parity_gpu.py", "-q", "-m", "gpu", "-p", "no:cacheprovider",
                        "-k", "prefill or small_batch_routes_agree"], cwd=ROOT,
                       env=dict(os.environ, AILA_NF4_MID_ROWS_MAX="0", PYTHONPATH=ROOT), capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and " passed" in r.stdout, r.stdout[-3000:] + r.stderr[-1000:]
