"""The launch shapes that the engine picks: pure host arithmetic, pinned here so that a change of a rule or of a shared-memory budget shows up as a deliberate diff.

One token's products (b200_op_lanes_shape): every mat-vec of the 8B, 70B, 405B and 7B models goes to k_matvec_q80 or k_matvec_kq. k_matvec's own shapes (b200_op_launch_shape: warps
per CTA, warps sharing a 32-row unit, ring stages per warp; the persistent per-token kernel's phases follow the same rule) are pinned at the same sizes. Q6_K tiles of 6.7 KB
halve the warps that fit."""
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


LANES = [
    # name,                    types,        units, k,    norm, qkv, (kernel, rows per thread, tiles per stage, teams, stages, blocks)
    ("8B qkv, all Q4_K",       [Q4_K],        192,  4096, 1, 1, (2, 1, 2, 2, 8, 148)),
    ("8B qkv, attn_v Q6_K",    [Q4_K, Q6_K],  192,  4096, 1, 1, (2, 1, 2, 2, 7, 148)),
    ("8B wo",                  [Q4_K],        128,  4096, 0, 0, (2, 1, 2, 1, 8, 128)),        # as many stages as the walk has
    ("8B gate|up",             [Q4_K],        896,  4096, 1, 0, (2, 2, 1, 7, 6, 148)),
    ("8B ffn_down Q4_K",       [Q4_K],        128, 14336, 0, 0, (2, 1, 2, 1, 16, 128)),
    ("8B ffn_down Q6_K",       [Q6_K],        128, 14336, 0, 0, (2, 1, 2, 1, 14, 128)),
    ("8B output Q6_K",         [Q6_K],       4008,  4096, 1, 0, (2, 2, 1, 8, 4, 148)),
    ("70B qkv, attn_v Q5_K",   [Q4_K, Q5_K],  320,  8192, 1, 1, (2, 1, 2, 3, 6, 148)),
    ("70B ffn_down Q6_K",      [Q6_K],        256, 28672, 0, 0, (2, 1, 2, 2, 6, 148)),
    ("405B qkv, attn_v Q6_K",  [Q4_K, Q6_K],  576, 16384, 1, 1, (2, 1, 2, 4, 3, 148)),
    ("405B ffn_down Q6_K",     [Q6_K],        512, 53248, 0, 0, (2, 1, 2, 4, 2, 148)),
    ("Mistral gate|up Q5_K",   [Q5_K],        896,  4096, 1, 0, (2, 2, 1, 7, 5, 148)),
    ("8B Q8_0 gate|up",        [Q8_0],        896,  4096, 1, 0, (1, 1, 16, 2, 6, 148)),
    ("8B Q8_0 ffn_down",       [Q8_0],        128, 14336, 0, 0, (1, 1, 16, 1, 12, 128)),
    ("toy ffn_down",           [Q4_K],         16,   768, 0, 0, (2, 1, 1, 1, 3, 16)),         # an odd number of blocks: one to a stage
    ("toy Q8_0 ffn_down",      [Q8_0],         16,   768, 0, 0, (1, 1, 8, 1, 24, 16)),
    ("four teams' units",      [Q4_K],        592,  4096, 1, 0, (2, 1, 2, 4, 6, 148)),
    ("one more",               [Q4_K],        593,  4096, 1, 0, (2, 2, 1, 5, 9, 148)),
    ("longest Q6_K vector",    [Q6_K],        593, 58368, 0, 0, (2, 2, 1, 5, 3, 148)),
    ("one block more",         [Q6_K],        593, 58624, 0, 0, (0, 1, 1, 1, 0, 148)),
    ("longest normed vector",  [Q6_K],        192, 16384, 1, 1, (2, 1, 2, 2, 6, 148)),
    ("Q8_0 beside a K-quant",  [Q4_K, Q8_0],  192,  4096, 0, 0, (0, 1, 1, 1, 0, 148)),
]


@pytest.mark.parametrize("name,types,units,k,norm,qkv,want", LANES, ids=[s[0] for s in LANES])
def test_lanes_shape(name, types, units, k, norm, qkv, want):
    out = (C.c_int32 * 7)()
    assert _lib.lib().b200_op_lanes_shape((C.c_int32 * len(types))(*types), len(types), units, k, norm, qkv, 148, out) == 0
    assert tuple(out[:6]) == want


@pytest.mark.parametrize("sm_count", [1, 20, 132, 148])
@pytest.mark.parametrize("types", [[Q4_K], [Q5_K], [Q6_K], [Q4_K, Q6_K], [Q5_K, Q6_K], [Q8_0]], ids=str)
def test_every_lanes_shape_is_one_the_kernel_takes(types, sm_count):
    """what the kernels assume of a launch, over rows of 1 to 5000 units and vectors of one block to past the longest: stages that divide the vector, a stage and a unit for every team,
    rings and teams within the barriers' arrays, shared memory within a block's, and a normed vector in one pass"""
    L, out = _lib.lib(), (C.c_int32 * 7)()
    q80 = types[0] == Q8_0
    for k in list(range(256, 6400, 256)) + [8192, 14336, 16384, 16640, 28672, 53248, 57088, 58112, 58368, 143616, 171008, 171264]:
        for units in (1, 2, 15, 16, 17, 19, 20, 21, 64, 131, 132, 133, 148, 149, 296, 297, 591, 592, 593, 896, 1184, 1185, 4008, 5000):
            for norm in (0, 1):
                assert L.b200_op_lanes_shape((C.c_int32 * len(types))(*types), len(types), units, k, norm, 1, sm_count, out) == 0
                kernel, rows, nb, teams, stages, blocks, smem = out
                if kernel == 0:
                    assert (norm and k > 16384) or k > 50000
                    continue
                assert kernel == (1 if q80 else 2) and not (norm and k > 16384)
                assert blocks == min(units, sm_count) and 1 <= teams and (teams - 1) * blocks < units
                assert (k // (32 if q80 else 256)) % nb == 0
                assert teams <= (2 if q80 else 4 * rows) and 1 <= stages <= (24 if q80 else 16)
                assert smem + (1024 if q80 else 2560) <= 227 * 1024


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


@pytest.mark.parametrize("heads", [1, 3, 4, 16, 32, 128])
@pytest.mark.parametrize("rank,rot", [(32, 8), (256, 64), (512, 64), (1000, 3)])
@pytest.mark.parametrize("window", [0, 1, 512, 8192])
def test_latent_attention_plan(heads, rank, rot, window):
    """what the kernels of a pass of few tokens assume: 16 queries a block and 64 key slices at most (k_latent_combine's lanes), slices and score rows that hold every key a tile can see,
    and a block's shared memory. Contexts for which nothing fits are refused when they are made, each at every number of tokens alike: more tokens never need more than one"""
    L, out = _lib.lib(), (C.c_int32 * 6)()
    for n_ctx in (1, 31, 64, 512, 4096, 5000, 32768, 65536, 98304, 131072, 200000, 400000, 900000, 1000000):
        for sm_count in (20, 132, 148):
            one = None
            for T in range(1, 8):
                assert L.b200_stack_latent_plan(heads, rank, rot, window, n_ctx, T, sm_count, out) == 0
                tq, hq, nsplit, smax, smem, staged = out
                assert 1 <= tq <= min(T, 4) and 1 <= hq <= heads and tq * hq <= 16 and 1 <= nsplit <= 64, tuple(out)
                keys = min(window + tq - 1, n_ctx) if window else n_ctx
                assert smax * nsplit >= keys
                if T == 1:
                    one = smem <= 227 * 1024
                assert (smem <= 227 * 1024) == one, (n_ctx, T, tuple(out))


BF16, F32 = 0, 1


@pytest.mark.parametrize("dtype,T,N,K,glu,want", [
    (BF16, 1, 16000, 2048, 0, 2), (BF16, 1, 2048, 8192, 0, 2), (BF16, 1, 16384, 2048, 1, 2), (F32, 1, 4096, 1024, 0, 2), (F32, 1, 16000, 4096, 1, 2),
    (BF16, 1, 1, 8, 0, 2), (BF16, 1, 2048, 1536, 1, 2), (BF16, 1, 8192, 4096, 1, 2), (BF16, 1, 512, 2048, 0, 2), (F32, 1, 16000, 8192, 0, 2),      # any number of rows
    (BF16, 1, 16000, 8200, 0, 0), (BF16, 1, 16000, 16384, 0, 0), (F32, 1, 16000, 8196, 0, 0), (BF16, 1, 2048, 2044, 0, 0), (F32, 1, 2048, 2046, 0, 0),      # rows beyond a block's registers, and of odd bytes
    (BF16, 1, 512, 16384, 0, 1), (BF16, 1, 513, 16384, 0, 0), (BF16, 1, 512, 16384, 1, 0), (BF16, 1, 512, 1020, 0, 0), (BF16, 1, 512, 1028, 0, 1),      # few of those that are long
    (BF16, 3, 16000, 2048, 0, 2), (BF16, 4, 16000, 2048, 0, 2), (BF16, 2, 12287, 2048, 0, 2), (BF16, 2, 12288, 2048, 0, 0), (F32, 2, 12287, 1024, 0, 2), (F32, 2, 12288, 1024, 0, 0),      # 48 MB
    (BF16, 5, 16000, 2044, 0, 6), (F32, 4, 16000, 8196, 0, 0),
    (F32, 300, 1024, 4096, 0, 4), (F32, 600, 1024, 512, 0, 4), (F32, 64, 4096, 2048, 0, 4),
    (F32, 64, 512, 512, 0, 4), (F32, 64, 512, 496, 0, 7), (F32, 64, 9472, 1024, 0, 4), (F32, 64, 9600, 1024, 0, 7), (F32, 64, 16000, 2048, 0, 7), (F32, 600, 4096, 4096, 0, 7),      # two blocks' worth of k, two SMs a tile
    (F32, 64, 512, 256, 0, 7), (F32, 300, 1024, 4096, 1, 7), (F32, 64, 64, 128, 0, 7), (F32, 64, 64, 124, 0, 6), (F32, 127, 512, 64, 0, 6), (F32, 128, 128, 64, 0, 7), (F32, 128, 127, 64, 0, 6), (F32, 64, 64, 4096, 0, 7), (F32, 64, 128, 4096, 0, 4),
    (F32, 63, 512, 512, 0, 6), (F32, 64, 63, 512, 0, 6), (F32, 64, 512, 60, 0, 6), (F32, 64, 512, 510, 0, 6),
    (BF16, 64, 128, 64, 0, 3), (BF16, 63, 128, 64, 0, 5), (BF16, 64, 128, 60, 0, 6)])
def test_stack_product_kernel(dtype, T, N, K, glu, want):
    """which kernel a layer stack's product takes: 0 a warp per row, 1 a block per row, 2 the ring kernel, 3 tcgen05 (bfloat16), 4 and 7
    tcgen05 (float32) in K parts and whole, 5 mma.sync, 6 tiles on the fp32 pipe; the sizes on both sides of each line are among those measured"""
    assert _lib.lib().b200_stack_product_kernel(dtype, T, N, K, glu, 148) == want


def product_plan(dtype, T, N, K, batch=1, seg=0, glu=0, sm_count=148):
    out = (C.c_int32 * 8)()
    assert _lib.lib().b200_stack_product_plan(dtype, T, N, K, batch, seg, glu, sm_count, out) == 0
    return tuple(out)


@pytest.mark.parametrize("dtype,T,N,K,batch,seg,glu,want", [
    (F32, 24, 64, 1024, 16, 1, 0, 1), (F32, 24, 64, 1024, 2, 1, 1, 1),                                  # experts' rows, however few
    (F32, 7, 4736, 1024, 1, 0, 0, 1), (F32, 7, 4672, 1024, 1, 0, 0, 0), (F32, 7, 64, 1024, 74, 0, 0, 1), (F32, 7, 64, 1024, 73, 0, 0, 0), (BF16, 7, 8192, 1020, 1, 0, 1, 1),      # 74 tiles of 64 rows
    (F32, 32, 1024, 1024, 1, 0, 0, 0), (F32, 33, 1024, 1024, 1, 0, 0, 1), (F32, 63, 1024, 1024, 1, 0, 0, 1), (F32, 64, 63, 1024, 1, 0, 0, 0)])
def test_large_grids_of_fp32_tiles_start_on_empty_sms(dtype, T, N, K, batch, seg, glu, want):
    assert product_plan(dtype, T, N, K, batch, seg, glu)[:2] == (6, want)


@pytest.mark.parametrize("T,N,K,batch,seg,want", [
    (5, 256, 64, 1, 0, 8), (5, 256, 56, 1, 0, 5), (5, 255, 64, 1, 0, 5), (63, 256, 64, 1, 0, 8), (63, 4096, 64, 1, 0, 8), (63, 254, 4096, 1, 0, 5), (5, 256, 196, 1, 0, 6),
    (5, 256, 192, 4, 1, 8), (63, 256, 192, 512, 1, 8), (63, 256, 192, 513, 1, 5), (63, 256, 192, 4, 0, 5),                       # experts, more of them than a block notes, heads
    (64, 256, 64, 1, 0, 8), (64, 128, 64, 1, 0, 8), (64, 127, 64, 1, 0, 5), (64, 128, 64, 513, 1, 3), (64, 128, 64, 4, 0, 3), (64, 128, 56, 1, 0, 5)])
def test_bfloat16_products_of_portions(T, N, K, batch, seg, want):
    """8 pairs of SMs, 3 a block per tile, 5 mma.sync: few tokens go to the tensor memory from 256 rows on, 64 and more from 128"""
    assert product_plan(BF16, T, N, K, batch, seg)[0] == want


@pytest.mark.parametrize("sm_count", [2, 20, 132, 148])
@pytest.mark.parametrize("seg", [0, 1, 8, 512])
def test_every_plan_of_a_pair_is_one_the_kernel_takes(seg, sm_count):
    """what k_gemm_bf16_pair assumes, over portions of 5 to 40000 tokens: accumulators that fit tensor memory and cover the tokens, a ring of two stages and more, K parts with a slice each whose
    sums fit their room, and at least one piece of work"""
    for T in (5, 31, 32, 33, 63, 64, 65, 96, 255, 256, 257, 300, 511, 512, 513, 700, 1024, 2048, 5000, 32768, 40000):
        for N in (128, 254, 256, 258, 512, 2048, 16384, 32000):
            for K in (64, 72, 192, 520, 2048, 8192, 16384):
                for glu in (0, 1):
                    route, _, acc, n, parts, stages, sets, work = product_plan(BF16, T, N, K, max(seg, 1), 1 if seg else 0, glu, sm_count)
                    if route != 8:
                        assert T < 64 and N < 256
                        continue
                    assert acc in (1, 2) and n % 32 == 0 and 32 <= n <= 256 and sets in (1, 2) and sets * acc * n <= 512
                    stage = (128 + acc * n // 2) * 64 * 2
                    assert 2 <= stages <= 8 and stages * stage <= 200 * 1024 and (stages == 8 or (stages + 1) * stage > 200 * 1024)
                    assert 1 <= parts <= max(1, (K + 63) // 64 // 2) and (parts == 1 or not (glu or seg)) and (parts == 1 or parts * T * N <= sm_count * 128 * 256)
                    rows = (N + 255) // 256
                    assert work == (rows * seg * ((T + 255) // 256) if seg else rows * -(-T // (acc * n)) * parts)


@pytest.mark.parametrize("T,N,K,glu,want", [
    (512, 16384, 2048, 1, (2, 256, 1, 4, 1, 64)), (512, 2048, 8192, 0, (1, 256, 4, 6, 2, 64)), (512, 2048, 2048, 0, (1, 64, 1, 8, 2, 64)),
    (16, 2048, 8192, 0, (1, 32, 8, 8, 2, 64)), (64, 16384, 2048, 1, (1, 64, 1, 8, 2, 64))])
def test_plans_of_pairs(T, N, K, glu, want):
    """the measured shapes: accumulators, columns of each, K parts, stages, sets, pieces of work"""
    assert product_plan(BF16, T, N, K, 1, 0, glu)[2:] == want


@pytest.mark.parametrize("gqa,n_ctx,units,q8_0,want", [
    (8, 1536, 320, 0, 1), (8, 1537, 320, 0, 0), (8, 512, 74, 1, 1), (8, 512, 73, 1, 0),                                           # 64 heads on 8; half of the SMs
    (4, 1024, 192, 1, 1), (4, 1025, 192, 1, 0), (4, 512, 192, 0, 0), (4, 512, 111, 1, 1), (4, 512, 110, 1, 0),                     # 32 heads on 8 in Q8_0; three quarters
    (2, 256, 400, 1, 0), (1, 256, 400, 1, 0)])
def test_one_launch_attention(gqa, n_ctx, units, q8_0, want):
    """whether a token's attention takes one launch a layer; the context's allocated size decides, wherever the token is in it"""
    assert _lib.lib().b200_op_attention_one_launch(gqa, n_ctx, units, q8_0, 148) == want
