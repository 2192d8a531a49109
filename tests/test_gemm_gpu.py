"""Parity of the tcgen05 W8A8 GEMM kernels (through the C ABI) with the CPU oracle.
int32 accumulators: bit-exact. bf16 outputs: rel-L2 <= 1e-3 against the emulation of the same op
(in practice they are equal up to rare 1-ulp differences)."""
import pytest
import torch

from oracle import inputs
from oracle import linear as ol

pytestmark = pytest.mark.gpu
TOL = 1e-3


def rel_l2(a, b):
    a, b = a.float(), b.float()
    return ((a - b).norm() / b.norm().clamp_min(1e-20)).item()


@pytest.fixture(scope="module")
def ops():
    from rapid_h3_b200 import _lib, gemm, kernels
    assert torch.cuda.is_available()
    return gemm, kernels, _lib


def _rand_codes(m, n, k, seed):
    g = inputs.gen(seed)
    xq = torch.randint(-127, 128, (m, k), generator=g, dtype=torch.int8)
    wq = torch.randint(-127, 128, (n, k), generator=g, dtype=torch.int8)
    xs = torch.rand(m, 1, generator=g) * 1e-3 + 1e-5
    ws = torch.rand(1, n, generator=g) * 1e-3 + 1e-5
    return xq, wq, xs, ws


@pytest.mark.parametrize("shape", [(128, 256, 128), (128, 256, 512), (256, 512, 4096), (300, 264, 1040),
                                   (1, 8, 16), (1000, 4096, 4096), (515, 12288, 4096)])
def test_int8_accumulators_bit_exact(ops, shape):
    # reference check: bench/gemm_tune.py:44-52 (random int8 codes, small random scales, torch.equal)
    gemm, kernels, lib = ops
    m, n, k = shape
    xq, wq, xs, ws = _rand_codes(m, n, k, seed=m + n + k)
    acc = torch.full((m, n), 123456789, dtype=torch.int32, device="cuda")
    y = gemm.int8_gemm(xq.cuda(), xs.cuda(), wq.cuda(), ws.cuda(), acc_dump=acc)
    lib.check_status()
    ref = ol.int_mm(xq, wq)
    assert torch.equal(acc.cpu(), ref)
    yr = ol.dequant(ref, xs, ws)
    assert torch.equal(y.cpu(), yr)


def test_config0_linear(ops):
    """X [4096,4096] with 1% outlier channels, W ~ N(0,0.02), bias ~ N(0,0.01), seed 0."""
    gemm, kernels, lib = ops
    x, w, b = inputs.linear_case(4096, 4096, 4096, seed=0)
    xd, wd, bd = x.cuda(), w.cuda(), b.cuda()
    qw = kernels.quantize_weight(wd, "int8_rowwise")
    xq, xs = kernels.quantize_rows(xd, "int8_rowwise")
    acc = torch.empty((4096, 4096), dtype=torch.int32, device="cuda")
    y = gemm.int8_gemm(xq, xs, qw.q, qw.scale, bias=bd, acc_dump=acc)
    lib.check_status()
    wq_r, ws_r = ol.quantize_weight(w, "int8_rowwise")
    xq_r, xs_r = ol.quantize_rows(x, "int8_rowwise")
    assert torch.equal(qw.q.cpu(), wq_r) and torch.equal(qw.scale.cpu(), ws_r)
    assert torch.equal(xq.cpu(), xq_r) and torch.equal(xs.cpu(), xs_r)
    acc_r = ol.int_mm(xq_r, wq_r)
    assert torch.equal(acc.cpu(), acc_r)
    y_r = ol.dequant(acc_r, xs_r, ws_r, b)
    assert rel_l2(y.cpu(), y_r) <= TOL
    assert (y.cpu() != y_r).float().mean() < 1e-4
    # the front end gives the same result as the explicit pipeline (bias is added by the caller there)
    y2 = kernels.linear(xd, qw, "int8_rowwise")
    assert torch.equal(y2.cpu(), ol.dequant(acc_r, xs_r, ws_r))
    # quantization error against the bf16 product stays in the reference's range (bench/int8_bench.py:41-48)
    full = x.float() @ w.float().t() + b.float()
    assert rel_l2(y.cpu(), full) < 0.12


@pytest.mark.parametrize("case", ["a", "b"])
def test_linear_matches_reference_golden(ops, golden_linear, case):
    gemm, kernels, lib = ops
    c = golden_linear[case]
    g = c["int8_rowwise"]
    qw = kernels.QWeight(g["wq"].cuda(), g["ws"].cuda())
    y = kernels.linear(c["x"].cuda(), qw, "int8_rowwise")
    assert torch.equal(y.cpu(), g["y"])
    g8 = c["fp8_rowwise"]
    qw8 = kernels.QWeight(g8["wq"].view(torch.float8_e4m3fn).cuda(), g8["ws"].cuda())
    y8 = kernels.linear(c["x"].cuda(), qw8, "fp8_rowwise")
    assert rel_l2(y8.cpu(), g8["y"]) < 4e-3  # the reference rounds the product to bf16 before scaling


def test_fp8_tensor_mode(ops, golden_tensor):
    """One scale per tensor (kernels.py:63-65, :125-128): codes and scales bit-exact against the oracle and the
    reference-made fixture, the product within the bf16 tolerance."""
    gemm, kernels, lib = ops
    c = golden_tensor
    qw = kernels.quantize_weight(c["w"].cuda(), "fp8_tensor")
    assert torch.equal(qw.q.cpu().view(torch.uint8), c["wq"])
    assert torch.equal(qw.scale.cpu(), c["ws"].reshape(1, 1).expand(1, c["w"].shape[0]))
    xq, xs = kernels.quantize_rows(c["x"].cuda(), "fp8_tensor")
    xq_r, xs_r = ol.quantize_rows(c["x"], "fp8_tensor")
    assert torch.equal(xq.cpu().view(torch.uint8), xq_r.view(torch.uint8)) and torch.equal(xs.cpu(), xs_r)
    y = kernels.linear(c["x"].cuda(), qw, "fp8_tensor")
    lib.check_status()
    y_r = ol.linear(c["x"], *ol.quantize_weight(c["w"], "fp8_tensor"), "fp8_tensor")
    assert rel_l2(y.cpu(), y_r) <= TOL
    assert rel_l2(y.cpu(), c["y"]) < 4e-3
    # a larger ragged case with an all-zero tensor row block and a strided view
    x, w, _ = inputs.linear_case(333, 1024, 264, seed=9, outlier_frac=0.01)
    x[7] = 0
    xq, xs = kernels.quantize_rows(x.cuda(), "fp8_tensor")
    xq_r, xs_r = ol.quantize_rows(x, "fp8_tensor")
    assert torch.equal(xq.cpu().view(torch.uint8), xq_r.view(torch.uint8)) and torch.equal(xs.cpu(), xs_r)
    z = torch.zeros(16, 64, dtype=torch.bfloat16)
    zq, zs = kernels.quantize_rows(z.cuda(), "fp8_tensor")
    assert torch.equal(zs.cpu(), torch.full((16, 1), 1e-12)) and not zq.view(torch.uint8).any()


@pytest.mark.parametrize("shape", [(256, 256, 256), (777, 1024, 2048)])
def test_fp8_gemm(ops, shape):
    gemm, kernels, lib = ops
    m, n, k = shape
    x, w, b = inputs.linear_case(m, k, n, seed=7)
    xq, xs = ol.quantize_rows(x, "fp8_rowwise")
    wq, ws = ol.quantize_weight(w, "fp8_rowwise")
    y = gemm.fp8_gemm(xq.cuda(), xs.cuda(), wq.cuda(), ws.cuda(), bias=b.cuda())
    lib.check_status()
    y_r = ol.dequant(ol.fp8_mm(xq, wq), xs, ws, b)
    assert rel_l2(y.cpu(), y_r) <= TOL


def test_gated_residual_segments(ops):
    # reference check: bench/fusion_test.py:38-50 (per-segment gated GEMM == int8_gemm + addcmul_)
    gemm, kernels, lib = ops
    m, n, k = 1000, 512, 1024
    xq, wq, xs, ws = _rand_codes(m, n, k, seed=21)
    g = inputs.gen(22)
    resid = torch.randn(m, n, generator=g).to(torch.bfloat16)
    gates = (0.5 * torch.randn(3, n, generator=g)).to(torch.bfloat16)
    segs = [(0, 600, 0), (600, 900, 1), (900, m, 2)]
    rd = resid.cuda()
    xqd, xsd, wqd, wsd = xq.cuda(), xs.cuda(), wq.cuda(), ws.cuda()
    for a, b_, row in segs:
        out = gemm.int8_gemm_gated_residual(xqd[a:b_], xsd[a:b_], wqd, wsd, gates[row].cuda(), rd[a:b_])
        assert out.data_ptr() == rd[a:b_].data_ptr()
    gemm.int8_gemm_gated_residual(xqd[:0], xsd[:0], wqd, wsd, gates[0].cuda(), rd[:0])  # M == 0 is a no-op
    lib.check_status()
    acc = ol.int_mm(xq, wq)
    ref = torch.empty_like(resid)
    for a, b_, row in segs:
        ref[a:b_] = ol.gated_residual(acc[a:b_], xs[a:b_], ws, gates[row], resid[a:b_])
    assert rel_l2(rd.cpu(), ref) <= TOL
    assert (rd.cpu() != ref).float().mean() < 1e-4


def test_swiglu_epilogue(ops):
    # reference check: bench/swiglu_epi_test.py:28-36 (epilogue h == bf16(silu(g) * u) of the plain GEMM)
    gemm, kernels, lib = ops
    m, k, f = 700, 1024, 1024
    xq, wq, xs, ws = _rand_codes(m, 2 * f, k, seed=31)
    xs, ws = xs * 30, ws * 30
    perm = gemm.swiglu_perm(2 * f, "cuda")
    assert torch.equal(perm.cpu(), ol.swiglu_perm(2 * f))
    wqd, wsd = wq.cuda()[perm].contiguous(), ws.cuda()[:, perm].contiguous()
    h = gemm.int8_gemm_swiglu(xq.cuda(), xs.cuda(), wqd, wsd)
    lib.check_status()
    assert h.shape == (m, f)
    acc = ol.int_mm(xq, wq)
    p = ol.swiglu_perm(2 * f)
    ref = ol.swiglu_epilogue(acc[:, p], xs, ws[:, p])
    assert rel_l2(h.cpu(), ref) <= TOL
    y = ol.dequant(acc, xs, ws).float()
    plain = (torch.nn.functional.silu(y[:, :f]) * y[:, f:])
    assert rel_l2(h.cpu(), plain) < 5e-3


def test_argument_errors(ops):
    gemm, kernels, lib = ops
    xq, wq, xs, ws = _rand_codes(16, 16, 32, seed=1)
    with pytest.raises(RuntimeError):
        gemm.int8_gemm(xq.cuda(), xs.cuda(), wq.cuda()[:, :16], ws.cuda())
    with pytest.raises(RuntimeError):
        gemm.int8_gemm(xq.cuda().float(), xs.cuda(), wq.cuda(), ws.cuda())
    with pytest.raises(RuntimeError):
        gemm.int8_gemm(xq, xs, wq, ws)


def test_epilogues_on_rows_that_are_only_16_byte_aligned(ops):
    """Outputs and residuals whose rows are 32-byte aligned go through 32-byte stores and loads, others through the
    16-byte path: both give the same bits (plain, gated residual, SwiGLU), here with a row stride of N + 8 elements
    and a base 16 bytes off a 32-byte boundary."""
    gemm, kernels, lib = ops
    m, n, k = 300, 512, 256
    x, w, _ = inputs.linear_case(m, k, n, seed=31)
    xq, xs = (t.cuda() for t in ol.quantize_rows(x, "int8_rowwise"))
    wq, ws = (t.cuda() for t in ol.quantize_weight(w, "int8_rowwise"))
    g = inputs.gen(5)
    gate = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
    resid0 = torch.randn(m, n, generator=g).to(torch.bfloat16).cuda()

    def odd_view(rows, cols):   # [rows, cols] view: row stride cols + 8, base 16 bytes into a 32-byte aligned buffer
        buf = torch.zeros(rows * (cols + 8) + 8, dtype=torch.bfloat16, device="cuda")
        v = buf[8:].view(rows, cols + 8)[:, :cols]
        assert v.data_ptr() % 32 == 16 and v.stride(0) % 16 == 8
        return v

    y = gemm.int8_gemm(xq, xs, wq, ws)
    y_odd = odd_view(m, n)
    gemm.int8_gemm(xq, xs, wq, ws, out=y_odd)
    assert torch.equal(y_odd, y)
    r = resid0.clone()
    gemm.int8_gemm_gated_residual(xq, xs, wq, ws, gate, r)
    r_odd = odd_view(m, n)
    r_odd.copy_(resid0)
    gemm.int8_gemm_gated_residual(xq, xs, wq, ws, gate, r_odd)
    assert torch.equal(r_odd, r)
    s = gemm.int8_gemm_swiglu(xq, xs, wq, ws)
    s_odd = odd_view(m, n // 2)
    gemm.int8_gemm_swiglu(xq, xs, wq, ws, out=s_odd)
    lib.check_status()
    assert torch.equal(s_odd, s)


@pytest.mark.parametrize("shape", [(1, 8, 16), (37, 264, 1040), (128, 256, 128), (300, 264, 1040), (515, 4096, 512)])
@pytest.mark.parametrize("kind", ["int8", "fp8"])
def test_bias_after_equals_a_separate_addition(ops, shape, kind):
    gemm, kernels, lib = ops
    m, n, k = shape
    xq, wq, xs, ws = (t.cuda() for t in _rand_codes(m, n, k, seed=m + k))
    if kind == "fp8":
        xq, wq = (xq.float() / 16).to(torch.float8_e4m3fn), (wq.float() / 16).to(torch.float8_e4m3fn)
    bias = torch.randn(n, generator=inputs.gen(7)).to(torch.bfloat16).cuda()
    y = gemm.gemm_bias_after(xq, xs, wq, ws, bias)
    plain = (gemm.fp8_gemm if kind == "fp8" else gemm.int8_gemm)(xq, xs, wq, ws)
    lib.check_status()
    assert torch.equal(y, plain + bias)


@pytest.mark.parametrize("m", [100, 128, 129, 300])
@pytest.mark.parametrize("n", [120, 128, 136, 392])
def test_epilogue_column_split(ops, m, n):
    """A tile's 256 columns are drained by two warps per row group: widths that end just before, at and just after the
    border between them, alone and after a full tile, through the one-CTA and the pair kernel, every bf16 epilogue."""
    gemm, kernels, lib = ops
    k = 256
    xq, wq, xs, ws = _rand_codes(m, n, k, seed=m * n)
    acc = ol.int_mm(xq, wq)
    dev = [t.cuda() for t in (xq, xs, wq, ws)]
    assert torch.equal(gemm.int8_gemm(*dev).cpu(), ol.dequant(acc, xs, ws))
    g = inputs.gen(m + n)
    gate, res = torch.randn(n, generator=g).to(torch.bfloat16), torch.randn(m, n, generator=g).to(torch.bfloat16)
    y = ol.dequant(acc, xs, ws).float()
    want = torch.addcmul(res.double(), y.double(), gate.double()).float().to(torch.bfloat16)
    got = gemm.int8_gemm_gated_residual(*dev, gate.cuda(), res.cuda())
    lib.check_status()
    assert (got.cpu() != want).float().mean() < 1e-4  # one fused rounding on the device, two here (fp64, then bf16)
    if n % 16 == 0:
        h = gemm.int8_gemm_swiglu(*dev)
        lib.check_status()
        assert h.shape == (m, n // 2)
        gu = y.to(torch.bfloat16).float().view(m, n // 8, 2, 4)
        ref = (gu[:, :, 0] / (1 + torch.exp(-gu[:, :, 0])) * gu[:, :, 1]).reshape(m, n // 2)
        assert rel_l2(h.cpu(), ref) <= 3e-3  # bf16 rounding, 2^-9 at worst


@pytest.mark.parametrize("m,split", [(5, 0), (5, 2), (5, 5), (128, 100), (300, 255), (300, 256), (515, 400)])
@pytest.mark.parametrize("n", [136, 512])
def test_gated_residual_with_two_gates(ops, m, split, n):
    """One launch over both modalities against one per modality with the bf16 gate rows: the same bits."""
    gemm, kernels, lib = ops
    k = 384
    xq, wq, xs, ws = _rand_codes(m, n, k, seed=m + split)
    dev = [t.cuda() for t in (xq, xs, wq, ws)]
    g = inputs.gen(m + n)
    gates = torch.randn(3, n, generator=g).cuda()
    res = torch.randn(m, n, generator=g).to(torch.bfloat16).cuda()
    want = res.clone()
    for a, b, row in ((0, split, 2), (split, m, 0)):
        if b > a:
            gemm.int8_gemm_gated_residual(dev[0][a:b], dev[1][a:b], dev[2], dev[3], gates[row].to(torch.bfloat16), want[a:b])
    got = gemm.int8_gemm_gated_residual2(*dev, gates[2], gates[0], split, res)
    lib.check_status()
    assert torch.equal(got, want)


def tile_of(lib, m, n, k):
    import ctypes
    rows, columns = ctypes.c_int64(), ctypes.c_int64()
    lib.call("rh3_gemm_tile", m, n, k, ctypes.addressof(rows), ctypes.addressof(columns))
    return rows.value, columns.value


# tests/test_epilogue_rules_cpu.py holds that these reach all six tiles
WIDTH_CASES = [(1, 8, 16), (9, 72, 144), (37, 4104, 1168), (100, 12288, 400), (128, 4096, 640), (129, 1032, 656), (200, 4096, 1168),
               (300, 4136, 1296), (513, 4096, 272), (1500, 4096, 144), (2049, 8192, 272), (100, 36864, 1168)]


@pytest.mark.parametrize("kind", ["i8", "f8"])
@pytest.mark.parametrize("m,n,k", WIDTH_CASES)
def test_gemm_tile_widths(m, n, k, kind):
    """The rule for the tile's width at rows, columns and K slabs that fill no tile: narrow and full tiles, single CTAs and pairs, one
    to four K slabs per stage with the last stage partly past K, and A boxes of fewer than 128 rows. The accumulators of int8
    are exact; e4m3 codes are small integers here, so theirs are as well."""
    from rapid_h3_b200 import _lib, gemm
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    top = 127 if kind == "i8" else 8
    a, b = (torch.randint(-top, top + 1, (r, k), device="cuda", generator=g) for r in (m, n))
    dtype = torch.int8 if kind == "i8" else torch.float8_e4m3fn
    xq, wq = (t.to(torch.float32).to(dtype) for t in (a, b))
    xs, ws = torch.rand(m, device="cuda", generator=g), torch.rand(n, device="cuda", generator=g)
    acc = torch.zeros(m, n, device="cuda", dtype=torch.int32)
    out = (gemm.int8_gemm if kind == "i8" else gemm.fp8_gemm)(xq, xs, wq, ws, acc_dump=acc)
    _lib.check_status()
    ref = a.double() @ b.double().t()   # sums below 2^53: exact in fp64
    assert torch.equal((acc if kind == "i8" else acc.view(torch.float32)).double(), ref)
    assert torch.equal(out, ((ref.float() * xs[:, None]) * ws[None]).bfloat16())


EPILOGUES = ["plain", "fp8", "bias", "bias_fp8", "gated", "gated2", "swiglu", "fp16", "fp16_resid", "fp16_swiglu", "fp32", "fp32_add"]


@pytest.mark.parametrize("epilogue", EPILOGUES)
def test_every_epilogue_has_the_same_bits_on_every_tile(ops, epilogue):
    """2,049 x 8,192 outputs on 256-column tiles of CTA pairs and of single CTAs (pairs off) against slices of their rows, which run on
    tiles of 64 and 128 columns: rows do not depend on one another, and every product here is exact (integers, or e4m3 codes that
    are small integers), so a row's bits are the same whatever tile it is computed on."""
    from rapid_h3_b200 import te_quant, vae_fast
    gemm, kernels, lib = ops
    m, n, k = 2049, 8192, 512
    g = torch.Generator(device="cuda").manual_seed(EPILOGUES.index(epilogue))
    f8 = epilogue.endswith("fp8")
    xq, wq = (torch.randint(-8 if f8 else -127, 9 if f8 else 128, (r, k), device="cuda", generator=g).to(torch.int8) for r in (m, n))
    if f8:
        xq, wq = xq.to(torch.float8_e4m3fn), wq.to(torch.float8_e4m3fn)
    xs, ws = (1e-3 * torch.rand(r, device="cuda", generator=g) + 1e-5 for r in (m, n))
    vec = torch.randn(3, n, device="cuda", generator=g)
    resid = torch.randn(m, n, device="cuda", generator=g)
    x32 = torch.randn(m, k, device="cuda", generator=g)
    x32[::7, 256:512] += 6.0 * (16.0 * ol.regular_hadamard(256)[5]).float().cuda()   # outlier rows: the second product adds to these
    te = te_quant._TELinear(kernels.QWeight(wq, ws[None]), vec[0].contiguous(), "int8_rot" if epilogue == "fp32_add" else "int8_rot_plain") if not f8 else None

    def run(a, b):
        xa, sa = xq[a:b], xs[a:b].contiguous()
        if epilogue in ("plain", "fp8"):
            return (gemm.fp8_gemm if f8 else gemm.int8_gemm)(xa, sa, wq, ws)
        if epilogue.startswith("bias"):
            return gemm.gemm_bias_after(xa, sa, wq, ws, vec[0].to(torch.bfloat16))
        if epilogue == "gated":
            return gemm.int8_gemm_gated_residual(xa, sa, wq, ws, vec[0].to(torch.bfloat16), resid[a:b].to(torch.bfloat16))
        if epilogue == "gated2":
            return gemm.int8_gemm_gated_residual2(xa, sa, wq, ws, vec[0], vec[1], min(max(1000 - a, 0), b - a), resid[a:b].to(torch.bfloat16))
        if epilogue == "swiglu":
            return gemm.int8_gemm_swiglu(xa, sa, wq, ws)
        if epilogue == "fp16":
            return vae_fast.vae_gemm(xa, wq, sa, ws, vec[0].half())
        if epilogue == "fp16_resid":
            return vae_fast.vae_gemm(xa, wq, sa, ws, vec[0].half(), vec[1].half(), resid[a:b].half())
        if epilogue == "fp16_swiglu":
            return vae_fast.vae_gemm_swiglu(xa, wq, sa, ws, vec[0].half())
        return te(x32[a:b])

    assert tile_of(lib, m, n, k) == (256, 256) and tile_of(lib, 200, n, k) == (256, 128) and tile_of(lib, 100, n, k) == (128, 64)
    full = run(0, m)
    for a, b in ((0, 100), (100, 300), (995, 1195), (1949, 2049), (2048, 2049)):
        assert torch.equal(run(a, b), full[a:b])
    prev = lib.lib().rh3_gemm_use_pairs(0)
    try:
        assert tile_of(lib, m, n, k) == (128, 256) and tile_of(lib, 200, n, k) == (128, 128)
        assert torch.equal(run(0, m), full) and torch.equal(run(100, 300), full[100:300])
    finally:
        lib.lib().rh3_gemm_use_pairs(prev)
    lib.check_status()
    if epilogue in ("plain", "fp8"):   # the anchor: these bits against the product in 64 bits
        want = (xq.double() @ wq.double().t()).float()
        assert torch.equal(full, ((want * xs[:, None]) * ws[None]).bfloat16())
