"""The text encoder's int8_rot linear with its outlier-row residual pass against the CPU oracle."""
import pytest
import torch

from oracle import inputs
from oracle import linear as ol
from oracle import quant as oq

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def te():
    from rapid_h3_b200 import _lib, kernels, te_quant
    assert torch.cuda.is_available()
    _lib.lib()
    return te_quant, kernels, _lib


def _case(m, k, n, seed):
    g = inputs.gen(seed)
    x = torch.randn(m, k, generator=g)
    # every 7th row carries a pattern that the rotation concentrates into ONE channel (a row of H256 itself):
    # these are the rows whose rotated abs-max towers over their rms, the ones the residual pass exists for
    x[::7, 256:512] += 6.0 * (ol.regular_hadamard(256)[5] * 16.0).float()
    w = (torch.randn(n, k, generator=g) / k ** 0.5).to(torch.bfloat16)
    return x, w


def test_residual_quantizer_bit_exact(te):
    te_quant, kernels, lib = te
    x, _ = _case(300, 1024, 8, 1)
    q1, s1 = oq.rot_quant_rows_i8(x.to(torch.bfloat16))
    rows = torch.tensor([0, 7, 14, 299, 5], dtype=torch.int64)
    q2, s2 = te_quant.rot_residual_quant_rows_i8(x.cuda(), q1.cuda(), s1.cuda(), rows.cuda())
    lib.check_status()
    q2r, s2r = oq.rot_residual_quant_rows_i8(x, q1, s1, rows)
    assert torch.equal(s2.cpu(), s2r) and torch.equal(q2.cpu(), q2r)


@pytest.mark.parametrize("mode", ["int8_rot", "int8_rot_plain"])
def test_te_linear_matches_oracle_and_helps_outlier_rows(te, mode):
    te_quant, kernels, lib = te
    m, k, n = 400, 2048, 512
    x, w = _case(m, k, n, 2)
    b = 0.1 * torch.randn(n, generator=inputs.gen(3))
    qw = kernels.quantize_weight(w.cuda(), "int8_rot")
    lin = te_quant._TELinear(qw, b.cuda(), mode, outlier_ratio=8.0)
    y = lin(x.cuda().reshape(4, 100, k))
    lib.check_status()
    assert y.shape == (4, 100, n) and y.dtype == torch.float32
    # oracle: the same two passes on CPU
    wq, ws = ol.quantize_weight(w, "int8_rot")
    q1, s1 = oq.rot_quant_rows_i8(x.to(torch.bfloat16))
    yr = ol.dequant(ol.int_mm(q1, wq), s1, ws).float()
    n_out = 0
    if mode == "int8_rot":
        ratio = 127.0 * s1[:, 0] / x.pow(2).mean(-1).sqrt().clamp_min(1e-12)
        rows = (ratio > 8.0).nonzero()[:, 0]
        n_out = rows.numel()
        assert 0 < n_out < m // 2
        q2, s2 = oq.rot_residual_quant_rows_i8(x, q1, s1, rows)
        yr[rows] += ol.dequant(ol.int_mm(q2, wq), s2, ws).float()
    yr = yr + b
    assert torch.allclose(y.cpu().reshape(m, n), yr, rtol=0, atol=1e-5 * yr.abs().max().item())
    ref = x.double() @ w.double().t() + b.double()
    err = ((y.cpu().reshape(m, n).double() - ref).norm(dim=1) / ref.norm(dim=1))
    print(mode, "rows with residual pass:", n_out, "median / max row error:", err.median().item(), err.max().item())
    if mode == "int8_rot":
        assert err.max().item() < 0.02


@pytest.mark.parametrize("shape", [(1, 256, 8), (130, 256, 264), (37, 2304, 512), (300, 8192, 128), (1500, 1024, 256)])
@pytest.mark.parametrize("rows", ["some", "none", "all"])
def test_fused_route_equals_the_separate_steps(te, shape, rows):
    """The three-kernel route against quantizer, product, row selection, residual quantizer and second product as separate
    calls: the same bits (row widths with idle threads, one row, more rows than blocks; no, some and only outlier rows).
    The rows here lie far from the ratio: one next to it may be an outlier on one route only (its squares are summed in
    another order)."""
    te_quant, kernels, lib = te
    m, k, n = shape
    x, w = _case(m, max(k, 512), n, m + k)
    x, w = x[:, :k].contiguous(), w[:, :k].contiguous()
    qw = kernels.quantize_weight(w.cuda(), "int8_rot")
    ratio = {"some": 8.0, "none": 1e9, "all": 0.0}[rows]
    for bias in (None, 0.1 * torch.randn(n, generator=inputs.gen(3)).cuda()):
        lin = te_quant._TELinear(qw, bias, "int8_rot", outlier_ratio=ratio)
        xd = torch.cat([x, torch.full((m, 4), 1e30)], 1).cuda()[:, :k]  # a strided view
        assert lin._can_fuse(xd)
        seen = te_quant._ROWS[1]
        taken = te_quant.residual_share() * seen
        y = lin(xd)
        if rows != "some":
            assert round(te_quant.residual_share() * te_quant._ROWS[1] - taken) == (m if rows == "all" else 0)
        assert te_quant._ROWS[1] == seen + m
        lib.check_status()
        xc = x.cuda()
        ref = lin._matmul(xc).float()
        ref = ref if bias is None else ref + bias
        assert torch.equal(y, ref)
        plain = te_quant._TELinear(qw, bias, "int8_rot_plain")(xd)
        p = kernels.linear(xc.to(torch.bfloat16), qw, "int8_rot").float()
        assert torch.equal(plain, p if bias is None else p + bias)


def _row_scales(x):
    from rapid_h3_b200 import quantizers
    return quantizers.rot_quant_rows_i8(x.to(torch.bfloat16))[1]


def test_residual_share_counts_what_ran(te, monkeypatch):
    """Rows seen and rows that took the residual pass stay in step: calls, replays of a captured call (which are not the
    captures), a call on another stream that nobody waited for, a graph whose capture is the linear's first call."""
    te_quant, kernels, lib = te
    monkeypatch.setattr(te_quant, "_ROWS", [0, 0])
    monkeypatch.setattr(te_quant, "_DEVICE_ROWS", {})
    m, k, n = 50, 512, 64
    x, w = _case(m, k, n, 8)
    x = x.cuda()
    qw = kernels.quantize_weight(w.cuda(), "int8_rot")
    lin = te_quant._TELinear(qw, None, "int8_rot", outlier_ratio=8.0)
    out = lin._outlier_rows(x, _row_scales(x)).numel()
    assert 0 < out < m
    assert te_quant.residual_share() == 0.0

    def totals():
        te_quant.residual_share()  # waits
        t, s = te_quant._DEVICE_ROWS[x.device].tolist()
        return te_quant._ROWS[0] + t, te_quant._ROWS[1] + s

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = lin(x)
    assert totals() == (0, 0)  # captured, not run
    for _ in range(5):
        graph.replay()
    assert totals() == (5 * out, 5 * m) and te_quant.residual_share() == out / m
    assert torch.equal(lin(x), y)
    assert totals() == (6 * out, 6 * m)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        lin(x)
    assert totals() == (7 * out, 7 * m)
    lib.check_status()


def test_no_rows_set_the_count_to_zero(te):
    te_quant, kernels, lib = te
    count = torch.full((1,), 77, dtype=torch.int32, device="cuda")
    lib.call("rh3_te_quant", None, 256, 0, 256, 8.0, None, None, None, count.data_ptr(), None, None, None, None, lib.stream())
    lib.check_status()
    assert count.item() == 0


def test_products_refuse_rows_their_stores_cannot_write(te):
    te_quant, kernels, lib = te
    q, f = torch.zeros(4, 256, dtype=torch.int8, device="cuda"), torch.ones(64, device="cuda")
    w, out = torch.zeros(64, 256, dtype=torch.int8, device="cuda"), torch.zeros(4 * 72 + 4, device="cuda")
    for offset, ldo in ((4, 64), (0, 68), (0, 56)):
        with pytest.raises(RuntimeError, match="32-byte"):
            lib.call("rh3_te_gemm", q.data_ptr(), f.data_ptr(), w.data_ptr(), f.data_ptr(), None, 4, 64, 256, None, None, None, None,
                     None, out.data_ptr() + 4 * offset, ldo, lib.stream())
