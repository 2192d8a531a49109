"""Which biases and gates a GEMM's epilogue takes over, and which stay with the general path."""
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


def test_two_gates_takes_one_or_two_plain_spans_only():
    two, tab = nodes.FusedBlock._two_gates, torch.zeros(2, 8)

    class OnGpu(torch.Tensor):  # the rule asks for a device tensor; nothing is computed here
        is_cuda = True

    gpu = tab.as_subclass(OnGpu)
    assert two([(0, 10, 0)], 10, gpu) == (0, 0, 10)
    assert two([(0, 7, 1), (7, 10, 0)], 10, gpu) == (1, 0, 7)
    assert two([(0, 7, 1), (7, 7, 0), (7, 10, 0)], 10, gpu) == (1, 0, 7)   # an empty span
    for segs in ([], [(0, 7, 0)], [(1, 10, 0)], [(0, 6, 0), (7, 10, 1)], [(7, 10, 1), (0, 7, 0)], [(0, 3, 0), (3, 6, 1), (6, 10, 0)],
                 [(0, 10, torch.zeros(10))], [(0, 10, 2)], [(0, 10, -1)]):
        assert two(segs, 10, gpu) is None
    assert two([(0, 10, 0)], 10, tab) is None and two([(0, 10, 0)], 10, gpu.to(torch.bfloat16)) is None
    assert two([(0, 10, 0)], 10, torch.zeros(8, 2).t().as_subclass(OnGpu)) is None


def test_the_shapes_of_the_tile_test_reach_every_tile():
    from test_gemm_gpu import WIDTH_CASES, tile_of
    from rapid_h3_b200 import _lib
    assert {tile_of(_lib, *c) for c in WIDTH_CASES} == {(r, c) for r in (128, 256) for c in (64, 128, 256)}
    # a call of the e4m3 recipe and one of a transformer block run at full width, a few rows on narrow tiles
    assert tile_of(_lib, 5003, 12288, 4096) == (256, 256) and tile_of(_lib, 36436, 4096, 4096) == (256, 256)
    assert tile_of(_lib, 37, 4096, 4096) == (128, 64)
    prev = _lib.lib().rh3_gemm_use_pairs(0)
    try:
        assert tile_of(_lib, 5003, 12288, 4096) == (128, 256)
    finally:
        _lib.lib().rh3_gemm_use_pairs(prev)
