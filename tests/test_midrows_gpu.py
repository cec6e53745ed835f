"""The tensor-memory kernel behind aila_nf4_forward / aila_nf4_forward_gate_up_swiglu for a few to a few
hundred rows, against the bit-exact dequantised weight in float64. With the weights equal, what is left is
the order of an fp32 sum and the rounding of the result to bf16 (8 significant bits: at most 2^-8 of the
value; twice more where gate and up pass through bf16)."""
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
    w = lin.dequantize_weight().double()
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


@pytest.mark.parametrize("ff,k", [(16, 64), (80, 448), (1040, 512), (9728, 2560)])
@pytest.mark.parametrize("m", [9, 31, 77, 200, 300])
def test_gate_up(nf4, scratch, ff, k, m):
    g, u = _linear(nf4, 5, ff, k), _linear(nf4, 6, ff, k)
    f = nf4.Bnb4BitLinear()
    assert f.init_fused_rows(g, u), f.last_error
    w = f.dequantize_weight().double()
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
