"""Kernels that start under the tail of the one before them (programmatic launches): captured graphs replayed on changed inputs,
buffers used again by the next launches of a chain, buffers handed from stream to stream. Same bits as plain calls everywhere."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    import rapid_h3_b200 as r
    assert torch.cuda.is_available()
    return r


def replayed(fn, inputs):
    """fn() captured once, then for every dict of values of `inputs`: the values copied into fn's tensors, a replay, a copy of its output."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        fn()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = fn()
    got = []
    for values in inputs:
        for tensor, value in values:
            tensor.copy_(value)
        graph.replay()
        got.append(out.clone())
    torch.cuda.synchronize()
    return got


@pytest.mark.parametrize("mode,rotate", [("int8_rowwise", False), ("int8_rot", True)])
@pytest.mark.parametrize("grid,audio", [((3, 4, 5), 7), ((5, 12, 17), 0)])
def test_captured_block(pkg, mode, rotate, grid, audio):
    r = pkg
    cfg = r.model.H3Config.tiny(text_dim=256, mlp_hidden=768)
    model = torch.nn.Module()
    model.blocks = torch.nn.ModuleList([r.model.init_weights(r.model.DiTBlock(cfg), seed=1).cuda()])
    fb = r.nodes.RapidH3LinearQuant().patch(model, mode)[0].block_forward[0]
    _, _, t_emb, rope, ctx = r.step.make_inputs(cfg, grid, audio, 1, 48, seed=3)
    n = grid[0] * grid[1] * grid[2]
    segs = [(0, n, 0)] + ([(n, n + audio, 1)] if audio else [])
    rope, t_emb = rope.cuda(), t_emb[0].cuda()
    xs = [torch.randn(n + audio, cfg.d_model, generator=torch.Generator().manual_seed(i)).to(torch.bfloat16).cuda() for i in range(3)]
    cs = [ctx[0].cuda() * (i + 1) for i in range(3)]
    r.nodes.ATTN_ROTATE = rotate
    try:
        want = [fb.forward(x.clone(), t_emb, segs, rope, c) for x, c in zip(xs, cs)]
        x_in, c_in = torch.empty_like(xs[0]), torch.empty_like(cs[0])
        got = replayed(lambda: fb.forward(x_in, t_emb, segs, rope, c_in), [((x_in, x), (c_in, c)) for x, c in zip(xs, cs)])
    finally:
        r.nodes.ATTN_ROTATE = False
    r._lib.check_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("lq,lk,heads", [(300, 300, 8), (257, 129, 2), (1500, 512, 4)])
def test_captured_attention(pkg, rotate, lq, lk, heads):
    A = pkg.attn_int8
    qkv = [[torch.randn(n, heads, 128, device="cuda", generator=torch.Generator("cuda").manual_seed(3 * i + j)).to(torch.bfloat16)
            for j, n in enumerate((lq, lk, lk))] for i in range(3)]
    want = [A.attention(*t, rotate=rotate) for t in qkv]
    held = [t.clone() for t in qkv[0]]
    got = replayed(lambda: A.attention(*held, rotate=rotate), [list(zip(held, t)) for t in qkv])
    pkg._lib.check_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_captured_decode(pkg):
    dec = pkg.vae.VAEDecoder(seed=0, widths=(128, 64, 64))
    zs = [torch.randn(1, 16, 2, 5, 7, device="cuda", generator=torch.Generator("cuda").manual_seed(i)).to(torch.bfloat16) for i in range(3)]
    want = [dec.decode(z) for z in zs]
    held = zs[0].clone()
    got = replayed(lambda: dec.decode(held), [[(held, z)] for z in zs])
    pkg._lib.check_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("m,n,k", [(37, 1024, 1024), (300, 256, 2048), (1, 4096, 256)])
def test_chain_that_uses_its_buffers_again(pkg, m, n, k):
    """Quantizer and GEMM over 24 inputs through one pair of code buffers, nothing else in between: every launch overwrites what
    the one before it reads."""
    r = pkg
    g = torch.Generator("cuda").manual_seed(m)
    x = torch.randn(24, m, k, device="cuda", generator=g).to(torch.bfloat16)
    qw = r.kernels.quantize_weight((0.02 * torch.randn(n, k, device="cuda", generator=g)).to(torch.bfloat16), "int8_rowwise")
    want = [r.kernels.linear(x[i], qw, "int8_rowwise") for i in range(24)]
    torch.cuda.synchronize()
    q = torch.zeros(m, k, device="cuda", dtype=torch.int8)
    s = torch.zeros(m, 1, device="cuda")
    out = torch.zeros(24, m, n, device="cuda", dtype=torch.bfloat16)
    for i in range(24):
        r._lib.call("rh3_quant_rows_i8", x[i].data_ptr(), k, m, k, q.data_ptr(), k, s.data_ptr(), r._lib.stream())
        r.gemm.int8_gemm(q, s, qw.q, qw.scale, out=out[i])
    r._lib.check_status()
    assert all(torch.equal(out[i], want[i]) for i in range(24))


def test_buffers_handed_from_stream_to_stream(pkg):
    """One stream's chain fills a buffer, another stream's chain reads it, and the first one fills it again once an event says so."""
    r = pkg
    m, k, n, rounds = 300, 1024, 512, 16
    g = torch.Generator("cuda").manual_seed(0)
    x = torch.randn(rounds, m, k, device="cuda", generator=g).to(torch.bfloat16)
    w1, w2 = (r.kernels.quantize_weight((0.02 * torch.randn(a, b, device="cuda", generator=g)).to(torch.bfloat16), "int8_rowwise")
              for a, b in ((n, k), (256, n)))

    def first(i, out):
        q, s = r.quantizers.quant_rows_i8(x[i])
        return r.gemm.int8_gemm(q, s, w1.q, w1.scale, out=out)

    def second(y, out):
        q, s = r.quantizers.quant_rows_i8(y)
        return r.gemm.int8_gemm(q, s, w2.q, w2.scale, out=out)

    want = torch.stack([second(first(i, None), None) for i in range(rounds)])
    torch.cuda.synchronize()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    y = torch.empty(2, m, n, device="cuda", dtype=torch.bfloat16)
    got = torch.empty_like(want)
    filled, read = [torch.cuda.Event() for _ in range(rounds)], [torch.cuda.Event() for _ in range(rounds)]
    for st in (a, b):
        st.wait_stream(torch.cuda.current_stream())
    for i in range(rounds):
        with torch.cuda.stream(a):
            if i >= 2:
                a.wait_event(read[i - 2])
            first(i, y[i % 2])
            filled[i].record(a)
        with torch.cuda.stream(b):
            b.wait_event(filled[i])
            second(y[i % 2], got[i])
            read[i].record(b)
    torch.cuda.synchronize()
    r._lib.check_status()
    assert torch.equal(got, want)
