"""Which biases a quantized linear may leave to the GEMM's epilogue, and which must stay an operation of torch's own."""
import torch

from rapid_h3_b200 import nodes


def test_only_inert_plain_tensors_go_to_the_epilogue():
    cpu = torch.device("cpu")
    b = torch.zeros(8)
    assert nodes._plain_bias(b, 8, cpu)
    assert not nodes._plain_bias(b, 16, cpu) and not nodes._plain_bias(b.view(1, 8), 8, cpu)
    assert not nodes._plain_bias(b, 8, torch.device("cuda", 0))
    p = torch.nn.Parameter(torch.zeros(8))
    assert not nodes._plain_bias(p, 8, cpu)  # would want its gradient
    with torch.no_grad():
        assert nodes._plain_bias(p, 8, cpu)
    seen = []
    torch.func.vmap(lambda t: (seen.append(nodes._plain_bias(t, 8, cpu)), t * 2)[1])(torch.zeros(3, 8))
    torch.func.jvp(lambda t: (seen.append(nodes._plain_bias(t, 8, cpu)), t * 2)[1], (b,), (b,))
    with torch.autograd.forward_ad.dual_level():
        seen.append(nodes._plain_bias(torch.autograd.forward_ad.make_dual(b, b), 8, cpu))
    assert seen == [False] * 3

    class Sub(torch.Tensor):
        pass

    assert not nodes._plain_bias(b.as_subclass(Sub), 8, cpu)
