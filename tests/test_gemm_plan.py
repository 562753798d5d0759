"""Host-side choices of the native library that need no GPU: the K split of accumulating GEMMs and the
number of copy drivers of the fused all-gather kernels."""
import ctypes

import pytest

from kareus_b200.kernels import build


def _lib():
    if not build.LIB.exists():
        pytest.skip("native library not built")
    L = ctypes.CDLL(str(build.LIB))
    L.kb_gemm_accum_plan.argtypes = [ctypes.c_int] * 4 + [ctypes.POINTER(ctypes.c_int)] * 3
    L.kb_gemm_accum_plan.restype = None
    L.kb_gemm_accum_scratch_floats.argtypes = [ctypes.c_int] * 4
    L.kb_gemm_accum_scratch_floats.restype = ctypes.c_long
    return L


def _plan(L, n_out, n_in, tokens, sms=148):
    """(tile width, K split), checked against the number of split tiles and the workspace of an ordered sum."""
    bn, ks, split = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    L.kb_gemm_accum_plan(n_out, n_in, tokens, sms, ctypes.byref(bn), ctypes.byref(ks), ctypes.byref(split))
    bn, ks, split = bn.value, ks.value, split.value
    assert bn in (64, 128, 192, 256)
    tiles = -(-n_out // 256) * -(-n_in // bn)
    assert split == (tiles % (sms // 2) if ks > 1 else 0)      # the tiles after the last full wave
    # outputs that 128-row tiles do not fill the chip with once may add their parts as they come: no workspace
    tiles128 = -(-n_out // 128) * -(-n_in // (128 if n_in <= 128 or 0 < n_in % 256 <= 128 else 256))
    scratch = L.kb_gemm_accum_scratch_floats(n_out, n_in, tokens, sms)
    assert scratch == split * (ks - 1) * 256 * bn or (scratch == 0 and tiles128 <= sms)
    return bn, ks


def test_weight_gradients_with_few_tiles_split_k():
    L = _lib()
    tokens = 16384
    # TP8 shards of a 3B Llama layer: 36-96 tiles for 148 SMs → more than one CTA per tile
    for n_out, n_in in [(640, 3072), (3072, 384), (2048, 3072), (3072, 1024)]:
        tile, ks = _plan(L, n_out, n_in, tokens)
        assert 2 <= ks <= 8, (n_out, n_in, tile, ks)
    # the LM head has thousands of tiles: no split
    assert _plan(L, 128256, 3072, tokens) == (256, 1)
    # a split never leaves fewer than eight 64-deep K steps per part
    for k in (512, 1024, 2048):
        _, ks = _plan(L, 640, 3072, k)
        assert ks == 1 or (k // 64) // ks >= 8
    # more tiles than SM pairs: what is left over after the full waves is split, in order
    for n_out, n_in in [(16384, 3072), (5120, 3072), (3072, 8192)]:
        bn, ks = _plan(L, n_out, n_in, tokens)
        assert ks > 1 and L.kb_gemm_accum_scratch_floats(n_out, n_in, tokens, 148) > 0, (n_out, n_in, bn, ks)
    # the choice follows the number of SMs given to the GEMM
    assert _plan(L, 2048, 3072, tokens, sms=32)[1] <= _plan(L, 2048, 3072, tokens, sms=148)[1]


def test_kernel_choice_for_plain_outputs():
    L = _lib()
    L.kb_gemm_plan.argtypes = [ctypes.c_int] * 5
    plan = lambda m, n, k, b_mn=0: L.kb_gemm_plan(m, n, k, b_mn, 148)
    # one wave of 128-row tiles instead of two of pairs; latency-bound calls; K of up to two steps
    assert plan(776, 5120, 3072) == -256
    for m, n, k in [(104, 13760, 512), (1024, 4096, 512), (4096, 1024, 256), (2048, 1024, 128), (64, 1024, 128), (15720, 4344, 128)]:
        assert plan(m, n, k) < 0, (m, n, k)
    # long or wide problems stay on pairs of SMs, as do rows whose length is no multiple of 16 bytes
    for m, n, k in [(16384, 16384, 3072), (16384, 3072, 8192), (16384, 640, 3072), (4096, 6144, 4096), (8192, 8192, 8192)]:
        assert plan(m, n, k) > 0, (m, n, k)
    assert plan(776, 5124, 3072) > 0
    # an MN-major B of 192 columns comes in as many bytes as one of 256
    assert plan(2048, 8192, 3072, 1) == 256


def test_long_calls_and_parts_of_k_for_plain_outputs():
    L = _lib()
    L.kb_gemm_plan.argtypes = [ctypes.c_int] * 5
    L.kb_gemm_scratch_floats.argtypes = [ctypes.c_int] * 5
    L.kb_gemm_scratch_floats.restype = ctypes.c_long
    # beyond 50 us wide tiles on pairs: one-SM tiles took 668 us here and 521 on pairs, 192 columns 137 and 256 columns 120
    assert L.kb_gemm_plan(3934, 14264, 5640, 0, 148) == 256 and L.kb_gemm_plan(11384, 2072, 2584, 1, 148) == 256
    # long sums over few tiles and long sums with a short last wave go in parts, in whole tiles of 256 rows
    for shape in [(203, 504, 15384, 0), (128, 1024, 8192, 0), (3800, 2048, 12288, 0), (4096, 3072, 128256, 1)]:
        n = L.kb_gemm_scratch_floats(*shape, 148)
        assert n > 0 and n % (256 * 64) == 0 and 4 * n <= 64e6, (shape, n)
    # not full waves, narrow outputs of many rows, or sums too short for a part of four steps and a caller's workspace
    for shape in [(16384, 16384, 3072, 0), (16384, 640, 3072, 0), (8192, 8192, 8192, 0), (128, 1024, 1016, 0), (128, 1024, 64, 1)]:
        assert L.kb_gemm_scratch_floats(*shape, 148) == 0, shape


def test_copy_driver_count_scales_with_output_width_and_budget():
    from kareus_b200.ops.fused import FusedAGGemm as F
    assert F.auto_drivers(12, 640) == 36 and F.auto_drivers(12, 1024) == 24 and F.auto_drivers(12, 2048) == 12
    # a kernel confined to 72 SMs keeps two thirds of them for the GEMM
    assert F.auto_drivers(12, 640, 72) == 24 and F.auto_drivers(12, 2048, 72) == 12
    # a plan's own number is never lowered by the cap
    assert F.auto_drivers(40, 4096, 72) == 40
