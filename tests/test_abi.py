"""The C-ABI shared library builds, loads and exports every symbol include/rapidh3_b200.h declares.
No compute call is made here (there is no GPU on the CPU test box)."""
import ctypes

from rapid_h3_b200 import _build, _lib


def test_library_builds_and_exports_declared_symbols():
    path = _build.build()
    handle = ctypes.CDLL(path)
    declared = _lib.declared_symbols()
    assert len(declared) >= 10
    for name in declared:
        assert hasattr(handle, name), f"{name} declared in the header but not exported"


def test_signature_table_covers_the_header():
    declared = set(_lib.declared_symbols()) - {"rh3_last_error_string"}
    assert declared == set(_lib.SIGNATURES), declared ^ set(_lib.SIGNATURES)


def test_argument_errors_are_reported_without_a_gpu():
    lib = _lib.lib()
    assert lib.rh3_version() >= 100
    # K not a multiple of 8 is rejected before anything touches the device
    rc = lib.rh3_quant_rows_i8(None, 8, 4, 7, None, 8, None, None)
    assert rc < 0 and b"multiple of 8" in lib.rh3_last_error_string()
    rc = lib.rh3_gemm_w8a8(None, 16, None, None, None, None, 4, 8, 16, 7, None, 8, None, None)
    assert rc < 0 and b"kind" in lib.rh3_last_error_string()


def test_argument_errors_of_the_later_entry_points():
    """Shape rules that the host side relies on are enforced by the library itself, before any CUDA call."""
    lib = _lib.lib()
    err = lib.rh3_last_error_string
    # rotated widths are whole groups of 256 channels
    assert lib.rh3_rot_quant_rows_i8(None, 384, 0, 384, None, 384, None, None) < 0 and b"256" in err()
    assert lib.rh3_swiglu_rot_quant_rows_i8(None, 1024, 0, 128, None, 128, None, None) < 0 and b"256" in err()
    # fp16 VAE quantizer: D must divide 256 and H*D be a multiple of 256
    assert lib.rh3_vae_out_quant(None, 1, 4, 8, 48, None, None, None) < 0
    assert lib.rh3_vae_quant_rows(None, 512, 4, 384, None, None, None) < 0 and b"256" in err()
    # fp16 SwiGLU GEMM: N in whole groups of 16 columns (M = 0: the null-pointer check is skipped)
    assert lib.rh3_vae_gemm_swiglu(None, 256, None, None, None, None, 0, 24, 256, None, 16, None) < 0 and b"16" in err()
    # scatter attention: 1..8 destinations
    assert lib.rh3_attn_int8_scatter(None, None, None, None, None, None, None, 256, 256, 128, 128, 1, 0.1, None, None,
                                     0, 128, 128, None) < 0 and b"n_dst" in err()
    assert lib.rh3_rope_scatter_heads(None, 1536, 4, 4, 3, 0, None, None, 1e-6, None, None, None) < 0  # 4 heads over 3 ranks
    assert lib.rh3_rot_residual_quant_rows_i8(None, 100, None, 100, None, None, 2, 100, None, None, None) < 0
    # the no-allocation statistics entry refuses what its built-in scratch cannot hold
    assert lib.rh3_attn_kv_stats_noalloc(None, 128, 128, None, 128, 128, 1 << 22, 64, None, None, None, None) < 0


def test_argument_errors_at_the_edges_of_the_fused_entries():
    lib = _lib.lib()
    err = lib.rh3_last_error_string
    p = ctypes.c_void_p(4096)  # an address that is never touched: the argument checks come first
    for count in (0.0, -1.0, float("nan")):
        assert lib.rh3_gn_silu_from_sums(p, p, count, 1e-5, p, p, 1, 8, 256, p, None) < 0 and b"count" in err()
    # no rows: nothing to do, and no count to set
    for fn, extra in ((lib.rh3_te_quant, ()), (lib.rh3_te_quant_counted, (None,))):
        assert fn(None, 256, 0, 256, 8.0, None, None, None, None, None, None, None, None, *extra, None) == 0


def test_argument_errors_of_the_block_entry():
    lib = _lib.lib()
    err = lib.rh3_last_error_string
    from rapid_h3_b200 import nodes
    ints = [115, 256, 2, 512, 33, 256, 0, 1, 108, 1536, 0, 0, 1]   # tokens, widths, gate rows, recipe flags
    pack = lambda v: nodes._BLOCK_ARGS.pack(*v, *[1e-6] * 5, 0, 256, *[0] * 18, 0, 256, *[0] * 14)  # noqa: E731
    p = 4096  # an address that is never touched
    need = lib.rh3_block_workspace_bytes(pack(ints))
    assert need >= 115 * (256 + 2 * 768) + 2 * 256 * 128
    assert lib.rh3_block_forward(None, p, need, None) < 0 and lib.rh3_block_forward(pack(ints), None, need, None) < 0
    assert lib.rh3_block_forward(pack(ints), p, need - 1, None) < 0 and b"needed" in err()
    assert lib.rh3_block_forward(pack(ints), p + 16, need, None) < 0 and b"aligned" in err()
    for i in (0, 1, 2, 3, 4, 5):
        bad = list(ints)
        bad[i] = 0
        assert lib.rh3_block_forward(pack(bad), p, need, None) < 0 and b"bad shape" in err()


def test_upsampling_refuses_what_its_32_bit_indices_do_not_hold():
    lib = _lib.lib()
    p = 4096  # an address that is never touched
    assert lib.rh3_upsample_causal2x(p, p, 1, 1, 1 << 20, 1 << 10, 64, None) < 0 and b"too large" in lib.rh3_last_error_string()
