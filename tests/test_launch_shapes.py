"""The launch shape the engine picks for every mat-vec of the 8B, 70B and 7B models (warps per CTA, warps sharing a 32-row
unit, ring stages per warp) — pure host arithmetic (b200_op_launch_shape), pinned here so that a change of the selection
rule or of the shared-memory budget shows up as a deliberate diff. Q6_K tiles of 6.7 KB halve the warps that fit."""
import ctypes as C

import pytest

from booster_b200 import _lib

Q4_K, Q5_K, Q6_K, Q8_0 = 12, 13, 14, 8
SHAPES = [
    # name,                          types,        units, k,     norm, (W, G, S)
    ("8B qkv, all Q4_K",             [Q4_K],        192,  4096, 1, (16, 8, 2)),
    ("8B qkv, attn_v Q6_K",          [Q4_K, Q6_K],  192,  4096, 1, (8, 4, 4)),      # 6.7 KB tiles: half the warps fit
    ("8B wo",                        [Q4_K],        128,  4096, 0, (16, 16, 2)),
    ("8B gate|up",                   [Q4_K],        896,  4096, 1, (14, 2, 3)),
    ("8B ffn_down Q4_K",             [Q4_K],        128, 14336, 0, (14, 14, 2)),
    ("8B ffn_down Q6_K",             [Q6_K],        128, 14336, 0, (8, 8, 3)),
    ("8B output Q6_K",               [Q6_K],       4008,  4096, 1, (16, 1, 2)),
    ("70B qkv, attn_v Q5_K",         [Q4_K, Q5_K],  320,  8192, 1, (12, 4, 3)),
    ("70B gate|up",                  [Q4_K],       1792,  8192, 1, (14, 1, 3)),
    ("70B ffn_down Q6_K",            [Q6_K],        256, 28672, 0, (8, 4, 3)),
    ("Mistral-7B Q5_K_M gate|up",    [Q5_K],        896,  4096, 1, (16, 2, 2)),
    ("8B Q8_0 gate|up",              [Q8_0],        896,  4096, 1, (16, 2, 4)),
]


@pytest.mark.parametrize("name,types,units,k,norm,want", SHAPES, ids=[s[0] for s in SHAPES])
def test_launch_shape(name, types, units, k, norm, want):
    L = _lib.lib()
    t = (C.c_int32 * len(types))(*types)
    out = (C.c_int32 * 3)()
    assert L.b200_op_launch_shape(t, len(types), units, k, norm, 148, out) == 0
    W, G, S = tuple(out)
    assert (W, G, S) == want
    tiles_unit = k // (32 if types[0] == Q8_0 else 256)
    assert W % G == 0 and tiles_unit % G == 0 and S >= 2          # the kernel's structural requirements
    assert G == 1 or units * G <= 148 * W                          # K-split only inside one wave


def test_launch_shape_rejects_oversized_vectors():
    L = _lib.lib()
    t = (C.c_int32 * 1)(Q6_K)
    out = (C.c_int32 * 3)()
    assert L.b200_op_launch_shape(t, 1, 128, 256 * 1024, 0, 148, out) != 0
    assert b"shared-memory" in L.b200_last_error()


@pytest.mark.parametrize("kv,gqa,past,n,want", [
    (8, 4, 6000, 512, 16), (8, 4, 0, 512, 16), (8, 4, 1234, 77, 16), (16, 1, 0, 512, 16), (8, 8, 8000, 74, 16),   # many keys or heads: whole tiles
    (2, 8, 0, 16, 1), (2, 8, 300, 64, 2), (8, 4, 0, 16, 1), (2, 8, 0, 512, 8),             # few: 16 tokens x 8 heads in two blocks took 24 us a layer more
    (8, 8, 0, 256, 8), (1, 8, 8000, 128, 16), (8, 4, 1000, 64, 16)])
def test_score_tile(kv, gqa, past, n, want):
    """tokens per block of a prompt batch's score kernel: few enough that the grid fills 148 SMs"""
    assert _lib.lib().b200_op_score_tokens(kv, gqa, past, n, 148) == want


@pytest.mark.parametrize("types,rows,k,T,want", [
    ([Q4_K], 28672, 4096, 8, 2), ([Q5_K], 28672, 4096, 8, 2), ([Q4_K], 2048, 1024, 512, 2), ([Q5_K], 9536, 256, 32, 2),    # a second wave of 64 x 32 tiles
    ([Q4_K], 4096, 4096, 32, 2), ([Q6_K], 1024, 2816, 8, 2), ([Q4_K, Q6_K], 6144, 4096, 32, 2),                            # one wave, long rows
    ([Q5_K], 4096, 4096, 32, 1), ([Q5_K, Q6_K], 2560, 2048, 33, 1), ([Q4_K], 768, 512, 100, 1), ([Q4_K], 4096, 1792, 8, 1),
    ([Q8_0], 4096, 4096, 32, 3), ([Q4_K], 96, 4096, 512, 0), ([Q4_K, Q8_0], 128, 4096, 32, 0)])
def test_prompt_product_kernel(types, rows, k, T, want):
    """which kernel a prompt product takes (2 tcgen05, 1 mma.sync, 3 Q8_0's tcgen05, 0 dp4a); an odd number of 32-row units goes to dp4a"""
    assert _lib.lib().b200_op_prompt_kernel((C.c_int32 * len(types))(*types), len(types), rows // 32, k, T, 148) == want


BF16, F32 = 0, 1


@pytest.mark.parametrize("dtype,T,N,K,glu,want", [
    (BF16, 1, 16000, 2048, 0, 2), (BF16, 1, 2048, 8192, 0, 2), (BF16, 1, 16384, 2048, 1, 2), (F32, 1, 4096, 1024, 0, 2), (F32, 1, 16000, 4096, 1, 2),
    (BF16, 1, 2048, 1536, 0, 2), (BF16, 1, 2048, 1536, 1, 0), (BF16, 1, 2048, 3072, 1, 2), (BF16, 1, 2048, 3072, 0, 0),      # three quarters of a block's lanes
    (BF16, 1, 5120, 4096, 1, 2), (BF16, 1, 8192, 4096, 1, 0), (BF16, 1, 10240, 4096, 1, 2), (F32, 1, 8192, 4096, 1, 0),     # a gated unit's waves
    (BF16, 1, 2048, 1024, 0, 0), (BF16, 1, 8192, 3072, 1, 0), (F32, 1, 2048, 3072, 0, 0),          # lanes without entries: 1.2 times as long
    (BF16, 1, 16000, 16384, 0, 0), (F32, 1, 16000, 8192, 0, 0),                  # eight chunks a lane: 1.4 and 1.2 times
    (BF16, 1, 512, 2048, 0, 1), (BF16, 4, 16000, 2048, 0, 0), (BF16, 1, 2048, 2044, 0, 0),
    (F32, 300, 1024, 4096, 0, 4), (F32, 600, 1024, 512, 0, 4), (F32, 64, 4096, 2048, 0, 4),
    (F32, 64, 512, 512, 0, 4), (F32, 64, 512, 496, 0, 7), (F32, 64, 9472, 1024, 0, 4), (F32, 64, 9600, 1024, 0, 7), (F32, 64, 16000, 2048, 0, 7), (F32, 600, 4096, 4096, 0, 7),      # two blocks' worth of k, two SMs a tile
    (F32, 64, 512, 256, 0, 7), (F32, 300, 1024, 4096, 1, 7), (F32, 64, 64, 64, 0, 7), (F32, 64, 64, 4096, 0, 7), (F32, 64, 128, 4096, 0, 4),
    (F32, 63, 512, 512, 0, 6), (F32, 64, 63, 512, 0, 6), (F32, 64, 512, 60, 0, 6), (F32, 64, 512, 510, 0, 6),
    (BF16, 64, 128, 64, 0, 3), (BF16, 63, 128, 64, 0, 5), (BF16, 64, 128, 60, 0, 6)])
def test_stack_product_kernel(dtype, T, N, K, glu, want):
    """which kernel a layer stack's product takes: 0 a warp per row, 1 a block per row, 2 a block per eight rows with x in registers, 3 tcgen05 (bfloat16), 4 and 7
    tcgen05 (float32) in K parts and whole, 5 mma.sync, 6 tiles on the fp32 pipe; the sizes on both sides of each line are among those measured"""
    assert _lib.lib().b200_stack_product_kernel(dtype, T, N, K, glu, 148) == want
