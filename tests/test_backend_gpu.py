"""The decode-step operators between the linears (embedding, per-head norm + RoPE + cache append,
single-token attention) and the Qwen3 NF4 backend skeleton built on the library, against the numpy /
C oracle. Through the C ABI.
"""
import numpy as np
import pytest
import torch

from oracle import backend_numpy as ref
from tests.helpers import bf16_bits, make_weight

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def be():
    from aila_b200 import backend
    assert torch.cuda.is_available()
    return backend



def _rand_bf16(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen) * scale).to(torch.bfloat16)


def _close(got_bits, want_bits, rel, what):
    got, want = ref.to_f32(got_bits).astype(np.float64), ref.to_f32(want_bits).astype(np.float64)
    err = np.abs(got - want).max()
    assert err <= rel * max(np.abs(want).max(), 1e-6), f"{what}: max err {err} vs {np.abs(want).max()}"


def test_embedding_lookup(be):
    gen = torch.Generator().manual_seed(1)
    table = _rand_bf16(gen, 1000, 256)
    ids = torch.tensor([0, 999, 17, 17, 512], dtype=torch.int32)
    out = torch.empty(5, 256, dtype=torch.bfloat16, device="cuda")
    be.embedding_lookup(table.cuda(), ids.cuda(), out)
    torch.cuda.synchronize()
    assert np.array_equal(bf16_bits(out), ref.embedding_lookup(bf16_bits(table), ids.numpy()))


@pytest.mark.parametrize("heads,kv,hd,pos", [(4, 2, 64, 0), (32, 8, 128, 37), (16, 16, 128, 1000), (8, 1, 256, 5)])
def test_decode_prepare_qkv(be, heads, kv, hd, pos):
    gen = torch.Generator().manual_seed(100 + heads + pos)
    max_len = 1024
    qkv = _rand_bf16(gen, 1, (heads + 2 * kv) * hd)
    qw, kw = (1 + 0.1 * torch.randn(hd, generator=gen)).to(torch.bfloat16), \
        (1 + 0.1 * torch.randn(hd, generator=gen)).to(torch.bfloat16)
    freq = ref.rope_freq(hd, 1e6)
    kc = torch.zeros(kv, max_len, hd, dtype=torch.bfloat16, device="cuda")
    vc = torch.zeros_like(kc)
    dq = qkv.cuda()
    q, k, v = dq[:, :heads * hd], dq[:, heads * hd:(heads + kv) * hd], dq[:, (heads + kv) * hd:]
    be.decode_prepare_qkv(q, k, v, torch.from_numpy(freq).cuda(), qw.cuda(), kw.cuda(), kc, vc, pos, heads, kv, hd,
                          1e-6)
    torch.cuda.synchronize()
    bits = bf16_bits(qkv).reshape(-1)
    kc_w = np.zeros((kv, max_len, hd), np.uint16)
    vc_w = np.zeros_like(kc_w)
    q_w = ref.decode_prepare_qkv(bits[:heads * hd], bits[heads * hd:(heads + kv) * hd], bits[(heads + kv) * hd:], freq,
                                 bf16_bits(qw), bf16_bits(kw), kc_w, vc_w, pos, heads, kv, hd, 1e-6)
    # cos/sin of angles up to 1000 rad differ in the last bits between libraries: one bf16 ulp
    _close(bf16_bits(dq).reshape(-1)[:heads * hd], q_w, 1e-2, "q")
    _close(bf16_bits(kc)[:, pos].reshape(-1), kc_w[:, pos].reshape(-1), 1e-2, "k cache")
    assert np.array_equal(bf16_bits(vc)[:, pos], vc_w[:, pos])
    assert not bf16_bits(kc)[:, pos + 1:].any() and not bf16_bits(kc)[:, :pos].any()


@pytest.mark.parametrize("hd", [20478, 20480, 20482, 40000, 120000])
def test_decode_prepare_qkv_long_heads(be, hd):
    """Both sides of the row that fits in the shared memory of every launch, and a row that fits nowhere."""
    test_decode_prepare_qkv(be, 2, 1, hd, 3)


@pytest.mark.parametrize("heads,kv,hd,length", [(4, 2, 64, 1), (32, 8, 128, 300), (16, 16, 128, 2047), (8, 1, 256, 33)])
def test_attention_decode(be, heads, kv, hd, length):
    gen = torch.Generator().manual_seed(200 + heads + length)
    max_len = 2048
    q = _rand_bf16(gen, 1, heads * hd)
    kc = _rand_bf16(gen, kv, max_len, hd)
    vc = _rand_bf16(gen, kv, max_len, hd)
    out = torch.empty(1, heads * hd, dtype=torch.bfloat16, device="cuda")
    be.attention_decode(q.cuda(), kc.cuda(), vc.cuda(), out, heads, kv, hd, length)
    torch.cuda.synchronize()
    want = ref.attention_decode(bf16_bits(q), bf16_bits(kc), bf16_bits(vc), heads, kv, hd, length)
    _close(bf16_bits(out).reshape(-1), want, 1e-2, "attention")


@pytest.mark.parametrize("heads,kv,hd,length", [
    (4, 4, 64, 2), (6, 2, 64, 65), (8, 4, 128, 64), (8, 4, 128, 65), (12, 3, 128, 129), (4, 1, 256, 257),
    (2, 2, 256, 1001), (32, 8, 128, 1023), (4, 1, 128, 2500), (3, 1, 128, 9), (4, 2, 64, 9000), (4, 2, 96, 40)])
def test_attention_decode_cluster(be, heads, kv, hd, length):
    """Both sides of the steps in CTAs per head, lengths that leave CTAs without a position or take several
    tiles, head groups of one, two and four, a head size the cluster form does not take; the cache is larger
    than the length and holds NaN behind it; with the position on the device the launch is sized for the
    whole cache. The same bits as the one-block form, which a cache off the 16-byte grid is sent to."""
    gen = torch.Generator().manual_seed(length)
    q = _rand_bf16(gen, heads, hd)
    kc, vc = _rand_bf16(gen, kv, length + 7, hd), _rand_bf16(gen, kv, length + 7, hd)
    s = torch.einsum("hd,htd->ht", q.double(), kc[:, :length].double().repeat_interleave(heads // kv, 0)) / hd ** 0.5
    want = torch.einsum("ht,htd->hd", torch.softmax(s, -1), vc[:, :length].double().repeat_interleave(heads // kv, 0))
    kc[:, length:] = float("nan")
    vc[:, length:] = float("nan")

    def off_grid(t):
        return torch.cat([torch.zeros(1, dtype=t.dtype), t.reshape(-1)]).cuda()[1:].view(t.shape)
    got = []
    for k, v in ((kc.cuda(), vc.cuda()), (off_grid(kc), vc.cuda())):
        for where in (None, torch.tensor([length - 1], dtype=torch.int32, device="cuda")):
            out = torch.zeros(heads * hd, dtype=torch.bfloat16, device="cuda")
            be.attention_decode(q.cuda(), k, v, out, heads, kv, hd, length if where is None else length + 7, where)
            got.append(bf16_bits(out))
    assert all((g == got[0]).all() for g in got)
    # one bf16 rounding of the result (2^-8), fp32 sums of at most 9000 terms before it
    assert torch.allclose(out.cpu().double().view(heads, hd), want, rtol=2 ** -8, atol=1e-4)


@pytest.mark.parametrize("heads,kv,hd,length", [
    (32, 8, 128, 1000), (32, 8, 128, 4000), (64, 8, 128, 1000), (64, 8, 128, 4000), (48, 8, 64, 2000), (40, 8, 128, 300)])
def test_attention_decode_head_groups(be, heads, kv, hd, length):
    """Groups of one, two and four heads by what runs at once, more clusters than run at once, heads per key/value
    head that only pairs or single heads divide."""
    test_attention_decode_cluster(be, heads, kv, hd, length)


def test_step_replayed_with_new_inputs(be):
    """q, k, v and the position are written by the launches right before and sit at the same addresses on
    every replay; the kernels that read them start before those launches end. 200 replayed steps against the
    same calls on fresh tensors with a wait after each."""
    from aila_b200 import linear as nf4
    heads, kv, hd, window, K = 8, 2, 64, 256, 512
    qkv = nf4.Bnb4BitLinear()
    assert qkv.init(make_weight(77, (heads + 2 * kv) * hd, K), 0), qkv.last_error
    o = nf4.Bnb4BitLinear()
    assert o.init(make_weight(78, K, heads * hd), 0), o.last_error
    sc = nf4.Bnb4BitLinearScratch(0)
    gen = torch.Generator().manual_seed(5)
    w = torch.ones(hd, dtype=torch.bfloat16, device="cuda")
    freq = (1e4 ** (-2 * torch.arange(hd // 2, dtype=torch.float64) / hd)).float().cuda()

    def step(x, buf, att, y, kc, vc, pos, wait):
        q, k, v = buf[0].split([heads * hd, kv * hd, kv * hd])
        qkv.forward(sc, x, buf, 1)
        wait()
        be.decode_prepare_qkv(q, k, v, freq, w, w, kc, vc, 0, heads, kv, hd, 1e-6, pos)
        wait()
        be.attention_decode(q, kc, vc, att, heads, kv, hd, window, pos)
        wait()
        o.forward(sc, att.view(1, -1), y, 1)
        wait()

    def tensors():
        z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda")
        return z(1, (heads + 2 * kv) * hd), z(heads * hd), z(1, K)
    caches = [[torch.zeros(kv, window, hd, dtype=torch.bfloat16, device="cuda") for _ in range(2)] for _ in range(2)]
    pos = torch.zeros(1, dtype=torch.int32, device="cuda")
    x = torch.zeros(1, K, dtype=torch.bfloat16, device="cuda")
    buf, att, y = tensors()
    st = torch.cuda.Stream()
    step(x, buf, att, y, *caches[0], pos, torch.cuda.synchronize)
    with torch.cuda.stream(st):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            step(x, buf, att, y, *caches[0], pos, lambda: None)
    inputs = _rand_bf16(gen, 200, 1, K).cuda()
    torch.cuda.synchronize()
    for t in range(200):
        with torch.cuda.stream(st):
            x.copy_(inputs[t])
            pos.fill_(t)
            graph.replay()
        torch.cuda.synchronize()
        fresh = tensors()
        step(inputs[t].clone(), *fresh, *caches[1], pos.clone(), torch.cuda.synchronize)
        assert all(torch.equal(a, b) for a, b in zip((buf, att, y, *caches[0]), (*fresh, *caches[1]))), t
    sc.check()


def test_backend_rejects_bad_arguments(be):
    from aila_b200 import _lib
    q = torch.zeros(1, 128, dtype=torch.bfloat16, device="cuda")
    kc = torch.zeros(1, 16, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(_lib.Nf4Error):
        be.attention_decode(q, kc, kc, q, 2, 1, 64, 17)      # beyond the cache
    with pytest.raises(_lib.Nf4Error):
        be.attention_decode(q, kc, kc, q, 3, 2, 64, 4)       # heads not a multiple of kv heads
    f = torch.zeros(32, dtype=torch.float32, device="cuda")
    w = torch.ones(64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(_lib.Nf4Error):
        be.decode_prepare_qkv(q, q, q, f, w, w, kc, kc, 16, 2, 1, 64, 1e-6)   # context window exceeded


def test_qwen3_backend_decodes_like_the_oracle(be, oracle):
    """A two-layer model with grouped-query attention: six tokens through forward(), the logits of
    every step against the oracle's decode step, the greedy token where the oracle's margin is clear,
    and the reference's error for a full context."""
    cfg = be.Qwen3Config(hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=4,
                         num_key_value_heads=2, head_dim=64, vocab_size=640, rms_norm_eps=1e-6, rope_theta=1e6)
    H, QD, KVD, FF = 256, 256, 128, 512
    gen = torch.Generator().manual_seed(4242)
    embed = _rand_bf16(gen, cfg.vocab_size, H)
    lm_head = _rand_bf16(gen, cfg.vocab_size, H, scale=0.05)
    final_norm = (1 + 0.1 * torch.randn(H, generator=gen)).to(torch.bfloat16)
    layers, ref_layers = [], []
    for i in range(cfg.num_hidden_layers):
        w = dict(q=make_weight(900 + 10 * i, QD, H), k=make_weight(901 + 10 * i, KVD, H),
                 v=make_weight(902 + 10 * i, KVD, H), o=make_weight(903 + 10 * i, H, QD),
                 gate=make_weight(904 + 10 * i, FF, H), up=make_weight(905 + 10 * i, FF, H),
                 down=make_weight(906 + 10 * i, H, FF))
        norms = {k: (1 + 0.1 * torch.randn(n, generator=gen)).to(torch.bfloat16)
                 for k, n in (("input_ln", H), ("post_attn_ln", H), ("q_norm", 64), ("k_norm", 64))}
        layers.append(be.Qwen3LayerWeights(**w, **norms))
        ref_layers.append({**w, **{k: bf16_bits(v) for k, v in norms.items()}})
    model = be.Qwen3Bnb4Backend(cfg, 0, max_seq_len=8)
    model.load(embed, layers, final_norm, lm_head)
    golden = ref.Qwen3Reference(oracle, cfg, bf16_bits(embed), ref_layers, bf16_bits(final_norm), bf16_bits(lm_head), 8)
    tokens = [3, 600, 17, 17, 255, 1]
    # a prompt of three tokens in one call, then one token per call
    logits = model.forward(torch.tensor(tokens[:3], dtype=torch.int32))
    torch.cuda.synchronize()
    model.scratch.check()
    want = [golden.step(t) for t in tokens[:3]][-1]
    _close(bf16_bits(logits).reshape(-1), want, 3e-2, "logits after the prompt")
    for t in tokens[3:]:
        logits = model.forward(torch.tensor([t], dtype=torch.int32))
        tok = int(model.greedy_token().cpu()[0])
        model.scratch.check()
        want = golden.step(t)
        _close(bf16_bits(logits).reshape(-1), want, 3e-2, f"logits of token {t}")
        w32 = ref.to_f32(want)
        top2 = np.sort(w32)[-2:]
        if top2[1] - top2[0] > 0.05 * np.abs(w32).max():
            assert tok == int(np.argmax(w32))
    assert model.current_length == 6
    with pytest.raises(RuntimeError, match="context window exceeded"):
        model.forward(torch.tensor([1, 2, 3], dtype=torch.int32))
    # greedy generation replayed from one captured step must choose what step-by-step calls choose
    prompt = torch.tensor(tokens[:3], dtype=torch.int32)
    model.reset()
    model.forward(prompt)
    by_hand = []
    for _ in range(4):
        tok = model.greedy_token().clone()
        by_hand.append(int(tok.cpu()[0]))
        model.forward(tok)
    last_by_hand = bf16_bits(model.logits).copy()
    model.reset()
    model.forward(prompt)
    replayed = model.generate(2).cpu().tolist() + model.generate(2).cpu().tolist()
    torch.cuda.synchronize()
    model.scratch.check()
    assert replayed == by_hand
    assert np.array_equal(bf16_bits(model.logits), last_by_hand)
    assert model.current_length == 7
    with pytest.raises(RuntimeError, match="context window exceeded"):
        model.generate(2)
    model.close()
