"""The C-ABI library loads and exports every symbol include/smoe_b200.h declares (no compute calls: no GPU here)."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "smoe_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(smoe_[a-z0-9_]+)\s*\(", text)))


def test_header_declares_the_hot_path_entry_points():
    syms = declared_symbols()
    for must in ("smoe_topk_metadata", "smoe_count_cumsum", "smoe_quant_rows", "smoe_quant_cols_t", "smoe_quant_iso32",
                 "smoe_gemm_gated", "smoe_gemm_varlen_m", "smoe_gemm_dgated", "smoe_gemm_wgrad", "smoe_combine"):
        assert must in syms


def test_library_exports_every_declared_symbol(built_library):
    lib = ctypes.CDLL(built_library)
    missing = [s for s in declared_symbols() if not hasattr(lib, s)]
    assert not missing, missing


def test_binding_covers_every_declared_symbol(built_library):
    from sonicmoe import _lib
    assert sorted(_lib.SIGNATURES) == declared_symbols()


def test_host_side_argument_checks(built_library):
    """Shape / argument errors are reported by return code before anything touches a device."""
    from sonicmoe._lib import lib
    assert lib.smoe_quant_rows(None, 4, 48, None, None, None, None) == 1          # K % 32
    assert lib.smoe_gemm_varlen_m(None, None, None, None, None, None, 100, 128, 128, 1, None, None) == 1
    assert lib.smoe_gemm_gated(None, 1, None, None, None, None, None, None, None, None, None, 128, 128, 128, 1, None,
                               None) == 1                                           # N % 256
    assert lib.smoe_topk_metadata(None, None, 4, 17, 8, 128, 0, 0, 0, 0, None, None, None, None, None, None, None,
                                  None, None, None) == 1                            # top-k > 16
    assert lib.smoe_topk_metadata_workspace(64, 8) > 0
    assert lib.smoe_combine(None, None, None, None, None, 4, 12, None) == 1        # H % 8


def test_column_quantizers_refuse_misaligned_buffers(built_library):
    """Every column kernel moves 16 bytes at a time: a source or payload off that boundary is an error code, never a launch."""
    from sonicmoe._lib import lib
    for dim in (64, 128):
        for src, q, isa in ((8, 16, 16), (16, 24, 16), (16, 16, 18)):
            assert lib.smoe_quant_cols_t(src, None, None, 128, dim, q, isa, None) == 2
            assert lib.smoe_requant_cols_t(src, 16, None, None, 128, dim, q, isa, None) == 2
    assert lib.smoe_quant_iso32(8, 128, 128, 16, 16, None, 16, None) == 2
    assert lib.smoe_quant_iso32(16, 128, 128, 16, 16, 8, 16, None) == 2


@pytest.mark.parametrize("N,tile", [(768, 256), (3072, 256), (6144, 256), (512, 256), (1920, 384), (576, 192), (640, 128)])
def test_column_tile_of_the_plain_gemm_does_not_depend_on_the_allocation(built_library, N, tile):
    """A table with masked slots is sized for all of them: rows that are allocated say nothing about rows that are routed."""
    from sonicmoe._lib import lib
    for E in (1, 8, 64):
        for K in (128, 1536, 6144):
            assert {lib.smoe_internal_plain_tile(128 * E * t, N, K, E) for t in (1, 2, 12, 24, 64)} == {tile}


@pytest.mark.parametrize("k_tiles,busy,E,tiles,loads", [
    (740, 148, 148, 1776, 1), (741, 148, 148, 1776, 0), (740, 148, 148, 1775, 0), (700, 147, 148, 1776, 0),
    (8, 8, 8, 1152, 0), (16, 16, 16, 128, 0), (96, 32, 256, 12288, 0), (28, 8, 8, 4608, 1), (0, 0, 8, 4608, 0)])
def test_old_gradients_are_loaded_ahead_only_where_hbm_is_what_every_sum_waits_for(built_library, k_tiles, busy, E, tiles, loads):
    """Five K tiles an expert, every expert with rows and 24 tiles for each of 74 CTA pairs, and one less or more of each; launches
    of few tiles and of mostly idle experts, which the loads would hold up."""
    from sonicmoe._lib import lib
    assert lib.smoe_internal_reduce_loads(k_tiles, busy, E, tiles, 74) == loads


@pytest.mark.parametrize("H,I,E", [(256, 128, 8), (512, 768, 16), (3072, 1536, 8), (4096, 4096, 8), (1024, 1280, 37)])
def test_arena_sizes_follow_from_the_arguments_alone(built_library, H, I, E):
    """A caller may remember an arena's size by the problem: forcing another column tile between asking and running must not make
    the layer need more than was asked for."""
    from sonicmoe._lib import LayerArgs, lib
    a = LayerArgs(512, H, I, E, 4, 2048, 2048 + E * 128)
    a.keep_z, a.dw1_mode, a.dw2_mode, a.out = 1, 1, 1, 16
    want = [lib.smoe_layer_bytes(a, which) for which in (0, 1, 2)]
    assert min(want) > 0
    for knobs in (128, 192, 256, 384, 128 | (1 << 17), 1 << 17):
        lib.smoe_internal_gemm_knobs(knobs)
        try:
            got = [lib.smoe_layer_bytes(a, which) for which in (0, 1, 2)]
        finally:
            lib.smoe_internal_gemm_knobs(0)
        assert got == want, knobs
