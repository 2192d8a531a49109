"""What the compiler says about the kernels whose speed rests on it."""
import os

from rapid_h3_b200 import _build


def test_gemm_kernels_do_not_spill(tmp_path):
    """A spilled word of an epilogue thread is written and read once per 32 columns of every tile, in the time the next
    tile's products take: the gated epilogues lost a tenth of the output projection's time to 40-72 bytes of it."""
    log = _build._compile(_build._nvcc(), os.path.join(_build.CSRC, "gemm.cu"), str(tmp_path / "gemm.o"), verbose=False)
    assert "spilled" not in log, log
