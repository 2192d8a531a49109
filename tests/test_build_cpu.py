"""What the compiler says about the kernels whose speed rests on it."""
import os
import re

from rapid_h3_b200 import _build


def compiler_log(source, tmp_path, verbose=False):
    return _build._compile(_build._nvcc(), os.path.join(_build.CSRC, source), str(tmp_path / "out.o"), verbose=verbose)


def test_gemm_kernels_do_not_spill(tmp_path):
    """A spilled word of an epilogue thread is written and read once per 32 columns of every tile, in the time the next
    tile's products take: the gated epilogues lost a tenth of the output projection's time to 40-72 bytes of it."""
    log = compiler_log("gemm.cu", tmp_path)
    assert "spilled" not in log, log


def test_convolution_kernels_keep_their_arrays_in_registers(tmp_path):
    """An array indexed by a run-time value goes to local memory, which -warn-spills does not mention: the GroupNorm partials of
    an epilogue thread did."""
    log = compiler_log("conv.cu", tmp_path, verbose=True)
    frames = re.findall(r"Function properties for (\w+)\s+(\d+) bytes stack frame", log)
    assert sum("conv3d" in name for name, _ in frames) == 4
    assert [f for f in frames if f[1] != "0"] == []
