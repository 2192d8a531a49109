"""int8_rot linears of the text encoder: the W8A8 rotated linear plus a second int8 pass on the quantization
residual of outlier rows.

Mirrors `_TELinear` of the reference's custom_nodes/rapid_h3/te_quant.py:45-115 for its `int8_rot` and
`int8_rot_plain` modes (fp32 in, fp32 out, like the module it replaces). The weight is passed as a
`kernels.QWeight` holding int8 codes of W . blockdiag(H256)^T and per-row scales (what the reference adopts from an
int8_convrot checkpoint, `:33-42`). ComfyUI's CLIP cloning, weight casting contexts and the bf16 attention wrapper
are outside this path. CPU tensors raise: there is no fallback.
"""
import torch

from . import _lib, gemm, kernels, nodes, quantizers

# how often the second pass ran: [rows that took it, rows seen]; `residual_share()` reads it. The fused route counts its
# outlier rows on the device, where the host need not wait for them: an int64 pair per device, [rows that took the pass,
# rows seen by graph launches]. A call outside a capture runs once, so its rows are counted as seen here, on the host; a
# captured call runs whenever its graph is replayed, so there the kernel counts both.
_ROWS = [0, 0]
_DEVICE_ROWS = {}


def residual_share():
    """Fraction of the rows seen so far that were given the residual pass (0.0 before any call). Waits for the devices
    that ran the fused route, so that calls still queued on any stream are in it."""
    taken, seen = _ROWS
    for device, pair in list(_DEVICE_ROWS.items()):
        torch.cuda.synchronize(device)
        t, s = pair.tolist()
        taken, seen = taken + t, seen + s
    return taken / seen if seen else 0.0


def _device_rows(device, capturing):
    """This device's pair. None in a capture that comes before the first linear of the device was made or called: a
    tensor made there would belong to the graph's pool, and such a graph's rows are counted nowhere."""
    pair = _DEVICE_ROWS.get(device)
    if pair is None and not capturing:
        pair = torch.zeros(2, dtype=torch.int64, device=device)
        torch.cuda.current_stream(device).synchronize()  # the zeros are there before another thread or stream can add
        pair = _DEVICE_ROWS.setdefault(device, pair)
    return pair


def rot_residual_quant_rows_i8(x, q1, s1, rows):
    """int8 row quantizer of rotate(x[rows]) - q1[rows] * s1[rows] -> (q2 int8 [n, K], s2 fp32 [n, 1]); x fp32."""
    _lib.require_cuda(x, q1, s1, rows)
    if x.dtype != torch.float32 or x.ndim != 2 or x.stride(1) != 1:
        raise RuntimeError("x must be fp32 [M, K] with unit column stride")
    n, k = rows.numel(), x.shape[1]
    rows = rows.to(torch.int32).contiguous()
    q2 = torch.empty((n, k), device=x.device, dtype=torch.int8)
    s2 = torch.empty((n, 1), device=x.device, dtype=torch.float32)
    _lib.call("rh3_rot_residual_quant_rows_i8", x.data_ptr(), x.stride(0), q1.data_ptr(), q1.stride(0), s1.data_ptr(),
              rows.data_ptr(), n, k, q2.data_ptr(), s2.data_ptr(), _lib.stream())
    return q2, s2


class _TELinear:
    """Replacement forward for one linear of the language model (fp32 in, fp32 out)."""

    def __init__(self, qweight, bias=None, mode="int8_rot", outlier_ratio=8.0):
        if mode not in ("int8_rot", "int8_rot_plain"):
            raise NotImplementedError(f"text-encoder mode {mode!r} is not implemented")
        self.qweight, self.bias, self.mode, self.outlier_ratio = qweight, bias, mode, outlier_ratio
        if mode == "int8_rot" and qweight.q.is_cuda:  # here, so that a first call under capture finds it
            _device_rows(qweight.q.device, torch.cuda.is_current_stream_capturing())

    def _outlier_rows(self, x32, s1):
        """Indices of the rows whose rotated peak is more than `outlier_ratio` times their rms. H256 is orthonormal,
        so the rotated row has the rms of the input row, and its abs-max is 127 * s1 by construction of the scale:
        nothing has to be rotated again to find them (selection rule of the reference, te_quant.py:97-99)."""
        rms = x32.square().mean(dim=-1).sqrt().clamp_min(1e-12)
        peak_over_rms = (127.0 * s1.reshape(-1)) / rms
        return torch.nonzero(peak_over_rms > self.outlier_ratio).reshape(-1)

    def _matmul(self, x2):
        """x2 [M, K] in the caller's dtype -> W8A8 product in bf16 or, when rows took the second pass, fp32."""
        qw = self.qweight
        x16 = x2.to(torch.bfloat16).contiguous()
        if self.mode == "int8_rot_plain":
            return kernels.linear(x16, qw, "int8_rot")
        q1, s1 = quantizers.rot_quant_rows_i8(x16)
        y = gemm.int8_gemm(q1, s1, qw.q, qw.scale)
        x32 = x2.float().contiguous()
        rows = self._outlier_rows(x32, s1)
        _ROWS[1] += x2.shape[0]
        if rows.numel() == 0:
            return y
        # second int8 pass on what the first quantization lost on those rows: rotate(x) - q1 * s1, quantized with
        # its own row scale and multiplied with the same weight; the two products add up in fp32
        q2, s2 = rot_residual_quant_rows_i8(x32, q1, s1, rows)
        y = y.float()
        y[rows] += gemm.int8_gemm(q2, s2, qw.q, qw.scale).float()
        _ROWS[0] += rows.numel()
        return y

    def _fused(self, x2):
        """Both passes for fp32 x2 [M, K] in three kernels: the input side (te_quant_kernel) and the two products, whose
        epilogues write fp32 and add the bias. The number of outlier rows stays on the device. The bits of the separate
        steps (_matmul), except for a row whose peak-over-rms lies within rounding of `outlier_ratio`: the two sum its
        squares in different orders, and it may take the second pass on one route only."""
        qw, dev = self.qweight, x2.device
        m, k = x2.shape
        n = qw.q.shape[0]
        second = self.mode == "int8_rot"
        ws = qw.scale.reshape(-1)
        bias = self.bias
        if bias is not None:
            bias = bias.to(torch.float32).contiguous()
        out = torch.empty((m, n), device=dev, dtype=torch.float32)
        # one workspace: q1 | q2 | s1 | s2 | rows | count | flags (every piece starts on a 16-byte boundary: K % 256 == 0).
        # Without a second pass no row is an outlier, and q2 is never written: it gets no room of its own.
        m4 = (m + 3) // 4 * 4
        codes = m * k * (2 if second else 1)
        work = torch.empty(codes + 3 * 4 * m4 + 16 + m, device=dev, dtype=torch.uint8)
        q1 = work.data_ptr()
        q2, s1 = q1 + codes - m * k, q1 + codes
        s2, rows, count = s1 + 4 * m4, s1 + 8 * m4, s1 + 12 * m4
        flags = count + 16
        ratio, taken, seen = float("inf"), None, None
        if second:
            ratio = float(self.outlier_ratio)
            capturing = torch.cuda.is_current_stream_capturing()
            pair = _device_rows(dev, capturing)
            if pair is not None:
                taken = pair.data_ptr()
                seen = taken + 8 if capturing else None
            if not capturing:
                _ROWS[1] += m
        _lib.call("rh3_te_quant_counted", x2.data_ptr(), x2.stride(0), m, k, ratio, q1, s1, flags, count, rows, q2, s2,
                  taken, seen, _lib.stream())
        _lib.call("rh3_te_gemm", q1, s1, qw.q.data_ptr(), ws.data_ptr(), _lib.ptr(bias), m, n, k, flags, count,
                  rows if second else None, q2, s2, out.data_ptr(), n, _lib.stream())
        return out

    def _can_fuse(self, x2):
        """What the fused route takes: fp32 rows the kernel can read in place, a plain row-ordered int8 weight and a bias
        torch need not see being added. Everything else goes through the separate steps."""
        qw, k = self.qweight, x2.shape[1]
        return (type(x2) is torch.Tensor and x2.dtype == torch.float32 and x2.shape[0] > 0 and k % 256 == 0 and k <= 8192
                and x2.stride(1) == 1 and x2.stride(0) % 4 == 0 and x2.stride(0) >= k and x2.data_ptr() % 16 == 0
                and qw.q.device == x2.device and qw.q.dtype == torch.int8 and qw.q.is_contiguous() and qw.q.shape[1] == k
                and qw.q.shape[0] % 8 == 0 and qw.scale.device == x2.device and qw.scale.dtype == torch.float32
                and qw.scale.numel() == qw.q.shape[0] and qw.scale.is_contiguous()
                and (self.bias is None or nodes._plain_bias(self.bias, qw.q.shape[0], x2.device)))

    def __call__(self, x):
        if x.device.type != "cuda":
            raise NotImplementedError("_TELinear: CUDA tensors only (no fallback path)")
        lead, k = x.shape[:-1], x.shape[-1]
        x2 = x.reshape(-1, k)
        if self._can_fuse(x2):
            return self._fused(x2).reshape(*lead, self.qweight.q.shape[0])
        y = self._matmul(x2).to(x.dtype)
        if self.bias is not None:
            y = y + self.bias.to(y.dtype)
        return y.reshape(*lead, y.shape[-1])
