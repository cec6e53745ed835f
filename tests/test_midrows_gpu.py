"""The tensor-memory kernel behind aila_nf4_forward / aila_nf4_forward_gate_up_swiglu for a few to a few
hundred rows, against its weights in float64: above 48 rows the bit-exact dequantised weight, up to 48 rows
the code-book value rounded to bf16 times the fp32 absmax, which is what the small-batch decode kernels
multiply by and closer to the unrounded weight. With the weights equal, what is left is the order of an fp32
sum and the rounding of the result to bf16 (8 significant bits: at most 2^-8 of the value; twice more where
gate and up pass through bf16)."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from tests.helpers import make_weight

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nf4():
    from aila_b200 import linear
    return linear


@pytest.fixture(scope="module")
def scratch(nf4):
    return nf4.Bnb4BitLinearScratch(0)


def _linear(nf4, *args):
    l = nf4.Bnb4BitLinear()
    assert l.init(make_weight(*args), 0), l.last_error
    return l


def _weight(lin, tensors, m):
    """[in_features, out_features] in float64: what a call of m rows multiplies by."""
    if m > 48:
        return lin.dequantize_weight().double()
    code = torch.from_numpy(np.asarray(tensors[0].quant_map, np.float32)).cuda().to(torch.bfloat16).double()
    packed = torch.from_numpy(np.concatenate([t.packed for t in tensors])).cuda()
    nibbles = torch.stack((packed >> 4, packed & 15), dim=1).view(lin.out_features(), -1, tensors[0].blocksize)
    absmax = lin.expand_absmax(tensors[0].blocksize).double()
    return (code[nibbles.int()] * absmax.unsqueeze(2)).view(lin.out_features(), -1).T


def _x(seed, m, k):
    return torch.randn(m, k, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).cuda()


# rows: both sides of the 16-row operand steps, of an x stage per chunk and per block, one and two accumulator
# buffers, one launch and two;
# shapes: fewer rows than a tile, ragged tiles, a tile per CTA and less, a tile over many CTAs, K of one
# block, absmax blocks of 128 and 256 weights, fp32 absmax
@pytest.mark.parametrize("n,k,blocksize,nested", [
    (16, 64, 64, True), (100, 448, 64, False), (129, 1024, 256, True), (1000, 9728, 64, True),
    (6144, 2560, 64, True), (40000, 128, 128, False)])
@pytest.mark.parametrize("m", [9, 16, 17, 77, 96, 97, 128, 129, 256, 257, 384])
def test_linear(nf4, scratch, n, k, blocksize, nested, m):
    lin = _linear(nf4, 31 + n, n, k, blocksize, nested)
    w = _weight(lin, [make_weight(31 + n, n, k, blocksize, nested)], m)
    x, res = _x(m, m, k), _x(m + 1, m, n)
    y = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    first = None
    for r in (None, res, res):
        lin.forward(scratch, x, y[:m], m, r)
        want = x.double() @ w + (0 if r is None else r.double())
        bound = 2 ** -8 * want.abs() + 1e-5 * (x.double().abs() @ w.abs())
        assert ((y[:m].double() - want).abs() <= bound).all()
        assert (y[m] == 7.0).all()
        if r is not None:       # the same bits from one run to the next
            assert first is None or torch.equal(first, y)
            first = y.clone()
    scratch.check()


@pytest.mark.parametrize("n,k,blocksize,nested", [
    (16, 64, 64, True), (100, 448, 64, False), (129, 1024, 256, True), (1000, 9728, 64, True),
    (6144, 2560, 64, True), (40000, 128, 128, False)])
@pytest.mark.parametrize("m", [31, 32, 33, 47, 48, 49])
def test_linear_at_the_edges_of_the_block_scaled_form(nf4, scratch, n, k, blocksize, nested, m):
    """Its widths of 32 and 48 rows, and the first row count of the other form."""
    test_linear(nf4, scratch, n, k, blocksize, nested, m)


def test_absmax_is_not_rounded_up_to_48_rows(nf4, scratch):
    """A code of +-1 is the block's absmax itself: with only such codes and one block per row the result is
    absmax times a sum of x that fp32 holds exactly, rounded once."""
    from aila_b200 import synth
    n, k = 512, 64
    gen = torch.Generator().manual_seed(3)
    absmax = torch.rand(n, generator=gen) + 0.5
    signs = torch.randint(2, (n, k), generator=gen)
    quant_map = synth.nf4_codebook()
    assert quant_map[0] == -1 and quant_map[15] == 1
    codes = (signs * 15).to(torch.uint8)
    packed = ((codes[:, 0::2] << 4) | codes[:, 1::2]).reshape(-1).numpy()
    lin = nf4.Bnb4BitLinear()
    assert lin.init(synth.Nf4Tensors(n, k, 64, packed, None, absmax.numpy(), quant_map, None, None), 0), lin.last_error
    for m in (9, 32, 40):
        x = torch.randint(-128, 128, (m, k), generator=gen).to(torch.bfloat16)   # |sums| <= 2^13: exact
        y = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        lin.forward(scratch, x.cuda(), y, m)
        sums = x.double() @ (2 * signs - 1).double().T
        want = (absmax * sums.float()).to(torch.bfloat16)
        assert torch.equal(y.cpu(), want)


@pytest.mark.parametrize("ff,k", [(16, 64), (80, 448), (1040, 512), (9728, 2560)])
@pytest.mark.parametrize("m", [9, 31, 77, 200, 300])
def test_gate_up(nf4, scratch, ff, k, m):
    g, u = _linear(nf4, 5, ff, k), _linear(nf4, 6, ff, k)
    f = nf4.Bnb4BitLinear()
    assert f.init_fused_rows(g, u), f.last_error
    w = _weight(f, [make_weight(5, ff, k), make_weight(6, ff, k)], m)
    x = _x(m, m, k)
    out = torch.full((m + 1, ff), 7.0, dtype=torch.bfloat16, device="cuda")
    assert nf4.Bnb4BitLinear.try_forward_decode_gate_up_swiglu(f, scratch, x, out[:m], ff, m)
    gate, up = (x.double() @ w).chunk(2, dim=1)
    want = torch.nn.functional.silu(gate) * up
    # to first order: 2^-8 of gate moves the product by at most |silu'| <= 1.1 times 2^-8 |gate| |up|, 2^-8 of
    # up and of the result by 2^-8 of the product each; 1.02 for the products of two such errors
    size = (x.double().abs() @ w.abs()).chunk(2, dim=1)
    bound = (1.02 * 2 ** -8 * (2 * want.abs() + 1.1 * (gate * up).abs())
             + 1e-5 * (size[0] * up.abs() + size[1] * gate.abs()) + 1e-6)
    assert ((out[:m].double() - want).abs() <= bound).all()
    assert (out[m] == 7.0).all()
    scratch.check()


def test_captured_call_outlives_larger_calls(nf4):
    """A captured call whose tiles span CTAs (152 tiles over the whole chip) keeps the address of the partial
    tiles: calls with more rows on the same scratch must neither move nor free them. Every size of the row
    range between the capture and the replay, then the same bits again."""
    ff, k = 9728, 2560
    g, u = _linear(nf4, 5, ff, k), _linear(nf4, 6, ff, k)
    f = nf4.Bnb4BitLinear()
    assert f.init_fused_rows(g, u), f.last_error
    sc = nf4.Bnb4BitLinearScratch(0)
    sc.ensure(64, k, 2 * ff, False)
    x = _x(64, 64, k)
    out = torch.empty(64, ff, dtype=torch.bfloat16, device="cuda")
    call = nf4.Bnb4BitLinear.try_forward_decode_gate_up_swiglu
    assert call(f, sc, x, out, ff, 64)
    want = out.clone()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            assert call(f, sc, x, out, ff, 64)
    larger = [(m, _x(m, m, k), torch.empty(m, ff, dtype=torch.bfloat16, device="cuda")) for m in (77, 200, 256, 384)]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for m, xm, om in larger:
        assert call(f, sc, xm, om, ff, m)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free, "the calls allocated or freed device memory"
    # had the address been given back, an allocation of that size would now sit where the graph writes
    guard = [torch.zeros(n * 2 ** 20 // 4, dtype=torch.int32, device="cuda") for n in (10, 12, 20, 31, 39)]
    with torch.cuda.stream(st):
        out.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert all(int(t.count_nonzero()) == 0 for t in guard)
    sc.check()


@pytest.mark.parametrize("before", ["weight buffer", "prompt", "other split"])
def test_capture_after(nf4, before):
    """What makes a call of 77 rows capturable: a reservation of the weight buffer alone, a longer prompt
    through the dequantise + GEMM route, a call that took the other split and needed no partial tiles."""
    n, k = 19456, 2560
    lin = _linear(nf4, 9, n, k)
    sc = nf4.Bnb4BitLinearScratch(0)
    if before == "weight buffer":
        sc.ensure(1, k, n, True)
    elif before == "prompt":
        lin.forward(sc, _x(1, 400, k), torch.empty(400, n, dtype=torch.bfloat16, device="cuda"), 400)
    else:
        small = _linear(nf4, 10, 2560, 4096)
        small.forward(sc, _x(2, 77, 4096), torch.empty(77, 2560, dtype=torch.bfloat16, device="cuda"), 77)
    x, y = _x(77, 77, k), torch.empty(77, n, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            lin.forward(sc, x, y, 77)
        graph.replay()
    torch.cuda.synchronize()
    got = y.clone()
    lin.forward(sc, x, y, 77)
    assert torch.equal(got, y)
    sc.check()


@pytest.mark.parametrize("m", [32, 77])
def test_captured_first_call(nf4, m):
    """Nothing can be allocated in a captured first call: the tiles that would be cut over the whole chip go to
    clusters."""
    n, k = 19456, 2560
    lin = _linear(nf4, 9, n, k)
    w = _weight(lin, [make_weight(9, n, k)], m)
    sc = nf4.Bnb4BitLinearScratch(0)
    x, y = _x(m, m, k), torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            lin.forward(sc, x, y, m)
        graph.replay()
    torch.cuda.synchronize()
    want = x.double() @ w
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * (x.double().abs() @ w.abs())).all()
    sc.check()


@pytest.mark.parametrize("m", [16, 77])
def test_residual_of_the_launch_before(nf4, m):
    """The residual is what the launch before has just written, at the same address on every replay: it must
    not come from a cache that an earlier replay filled."""
    a, b = _linear(nf4, 41, 512, 512), _linear(nf4, 42, 512, 512)
    sc = nf4.Bnb4BitLinearScratch(0)
    sc.ensure(m, 512, 512, True)
    x, y1, y2 = (torch.zeros(m, 512, dtype=torch.bfloat16, device="cuda") for _ in range(3))
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            for _ in range(4):
                a.forward(sc, x, y1, m)
                b.forward(sc, y1, y2, m, y1)
                a.forward(sc, y2, y1, m, y2)
                b.forward(sc, y1, x, m, y1)
    for rep in range(20):
        start = _x(1000 + rep, m, 512)
        t1, t2, t = torch.empty_like(start), torch.empty_like(start), start.clone()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            x.copy_(start)
            graph.replay()
        torch.cuda.synchronize()
        for _ in range(4):
            for lin, src, dst, res in ((a, t, t1, None), (b, t1, t2, t1), (a, t2, t1, t2), (b, t1, t, t1)):
                dst.fill_(float("nan"))
                torch.cuda.synchronize()
                lin.forward(sc, src, dst, m, None if res is None else res.clone())
                torch.cuda.synchronize()
        assert torch.equal(t, x), rep
    sc.check()


@pytest.mark.parametrize("m", [9, 40, 77, 256, 384])
def test_linear_it_does_not_take(nf4, scratch, m):
    """More than 256 absmax codes per row: no table of row scales, so batched decode launches up to 48 rows and
    the dequantise + GEMM route above serve these row counts (sums of the former in no fixed order)."""
    n, k = 200, 25600
    lin = _linear(nf4, 61, n, k)
    w = _weight(lin, [make_weight(61, n, k)], m)
    x, res = _x(m, m, k), _x(m + 1, m, n)
    y = torch.full((m + 1, n), 7.0, dtype=torch.bfloat16, device="cuda")
    lin.forward(scratch, x, y[:m], m, res)
    want = x.double() @ w + res.double()
    assert ((y[:m].double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5 * (x.double().abs() @ w.abs())).all()
    assert (y[m] == 7.0).all()
    scratch.check()


SPLITS = r"""
import torch
from aila_b200 import linear as nf4
from tests import test_midrows_gpu as t
sc = nf4.Bnb4BitLinearScratch(0)
# K of 1, 5, 7, 16 and 65 blocks: shares of a cluster's CTAs that are equal, unequal and short of a chunk
for n, k, bs, nested in ((200, 64, 64, True), (129, 320, 64, False), (100, 448, 64, True), (300, 1024, 128, True),
                         (1000, 4160, 64, False)):
    for m in (9, 17, 48, 49, 129, 256):
        t.test_linear(nf4, sc, n, k, bs, nested, m)
for ff, k in ((80, 448), (1040, 512)):
    for m in (9, 40, 77, 200):
        t.test_gate_up(nf4, sc, ff, k, m)
print("splits ok")
"""


@pytest.mark.parametrize("split", range(9))
def test_every_split(split):
    """The stream split and clusters of one to eight CTAs, each forced on small ragged shapes (the choice is read
    once per process)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, AILA_NF4_MID_SPLIT=str(split), PYTHONPATH=root)
    r = subprocess.run([sys.executable, "-c", SPLITS], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "splits ok" in r.stdout, r.stdout[-1000:] + r.stderr[-3000:]
