"""Operator-level parity of the CUDA kernels (through the C-ABI, same kernels the engine launches) against
the golden vectors the reference produced and against the port oracle on seeded inputs.
EVERYTHING is bit-exact: the kernels reproduce the reference's fp32 operation order (see kernels.cuh)."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import q8k_equal, rel_err
from booster_b200 import _lib, engine, gguf_io as G
from oracle import port

pytestmark = pytest.mark.gpu
TYPES = {"Q8_0": 8, "Q4_K": 12, "Q5_K": 13, "Q6_K": 14}


@pytest.fixture(scope="module")
def ops(golden_dir):
    return np.load(os.path.join(golden_dir, "ops.npz"))


def test_quantize_q8_K_bit_exact_golden(ops):
    assert q8k_equal(engine.op_quantize_q8_K(ops["act_x"]), ops["act_q8_K"])


def test_quantize_q8_0_bit_exact_golden(ops):
    assert np.array_equal(engine.op_quantize_q8_0(ops["act_x"]), ops["act_q8_0"])


@pytest.mark.parametrize("k", [256, 4096, 14336, 28672])
def test_quantize_bit_exact_vs_port(k):
    rng = np.random.default_rng(k)
    x = (rng.standard_normal(k) * rng.choice([1e-3, 1.0, 50.0])).astype(np.float32)
    x[::97] = 0.0
    assert q8k_equal(engine.op_quantize_q8_K(x), port.quantize_row_q8_K(x))
    assert np.array_equal(engine.op_quantize_q8_0(x), port.quantize_row_q8_0(x))


@pytest.mark.parametrize("name", list(TYPES))
def test_dequantize_bit_exact_golden(ops, name):
    t, k = TYPES[name], 1536
    rb = G.row_bytes(t, k)
    for r in (0, 7, 15):
        assert np.array_equal(engine.op_dequantize_row(t, ops[f"w_{name}"][r * rb:(r + 1) * rb], k), ops[f"deq_{name}"][r])


@pytest.mark.parametrize("name", list(TYPES))
def test_mul_mat_vec_golden(ops, name):
    # the reference's own ggml_vec_dot_* results, bit for bit
    y = engine.op_mul_mat_vec(TYPES[name], ops[f"w_{name}"], 16, 1536, ops["act_x"])
    assert np.array_equal(y, ops[f"dot_{name}"]), f"max abs diff {np.abs(y - ops[f'dot_{name}']).max()}"


@pytest.mark.parametrize("name", list(TYPES))
@pytest.mark.parametrize("shape", [(64, 256), (64, 768), (1024, 4096), (6144, 4096), (256, 14336), (128, 8192), (64, 28672)])
def test_mul_mat_vec_vs_port(name, shape):
    n, k = shape
    t = TYPES[name]
    rng = np.random.default_rng(n * 31 + k)
    w = G.random_blocks(rng, t, n, k)
    x = rng.standard_normal(k).astype(np.float32)
    y, yr = engine.op_mul_mat_vec(t, w, n, k, x), port.mul_mat_vec(t, w, n, k, x)
    assert np.array_equal(y, yr), f"max abs diff {np.abs(y - yr).max()} rel {rel_err(y, yr)}"


def test_mul_mat_vec_edge_activations():
    # all-zero activation blocks, ties at +-max: the integer path must still be exact
    rng = np.random.default_rng(5)
    k, n = 1024, 32
    x = rng.standard_normal(k).astype(np.float32)
    x[:256] = 0.0
    x[300] = 9.0; x[400] = -9.0
    for t in TYPES.values():
        w = G.random_blocks(rng, t, n, k)
        assert np.array_equal(engine.op_mul_mat_vec(t, w, n, k, x), port.mul_mat_vec(t, w, n, k, x))


@pytest.mark.parametrize("k", [256, 4096, 8192])
def test_rms_norm(k):
    rng = np.random.default_rng(k)
    x = rng.standard_normal(k).astype(np.float32) * 3
    w = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    y, yr = engine.op_rms_norm(x, w, 1e-5), port.rms_norm(x, w, 1e-5)
    # double accumulation on both sides: identical unless the mean lands on a float rounding boundary
    assert np.array_equal(y, yr) or rel_err(y, yr) < 1e-7
    assert rel_err(engine.op_rms_norm(x, None, 1e-6), port.rms_norm(x, None, 1e-6)) < 1e-7


@pytest.mark.parametrize("pos", [0, 1, 17, 2047, 8191])
@pytest.mark.parametrize("base", [10000.0, 500000.0])
def test_rope(pos, base):
    rng = np.random.default_rng(pos)
    x = rng.standard_normal(8 * 128).astype(np.float32)
    y, yr = engine.op_rope(x, 8, 128, pos, base), port.rope(x, 8, 128, pos, base)
    # the table is built with the host libm exactly like ggml_rope_cache_init; rotation is un-fused mul/sub
    assert np.array_equal(y, yr)
    ff = (1 + rng.random(64)).astype(np.float32)
    assert np.array_equal(engine.op_rope(x, 8, 128, pos, base, 0.5, ff), port.rope(x, 8, 128, pos, base, 0.5, ff))


# (n_head, n_head_kv, n_kv): GQA 1/2/4/8; the contexts of the measured models (2048, 4096, 8192 and one position short of
# them); (64, 8, 8192) exceeds one CTA's shared memory for the GQA score rows and takes the long-context route
@pytest.mark.parametrize("cfg", [(4, 1, 1), (4, 1, 33), (32, 8, 257), (32, 8, 2048), (64, 8, 700), (8, 8, 64), (2, 1, 5), (32, 8, 3000),
                                 (16, 8, 1000), (32, 8, 4096), (32, 8, 8191), (32, 8, 8192), (64, 8, 4095), (64, 8, 4096), (64, 8, 8192),
                                 (8, 1, 12000), (8, 1, 70000)])
@pytest.mark.parametrize("round_q", [False, True])
def test_attention_bit_exact(cfg, round_q):
    _attention_case(cfg, round_q)


# the long-context three-kernel route (taken automatically only when a CTA's share of the context exceeds its shared
# memory, e.g. (8, 1, 70000) above) forced at ordinary sizes too
@pytest.mark.parametrize("cfg", [(4, 1, 33), (32, 8, 2048), (64, 8, 4095), (64, 8, 8192), (2, 1, 5), (16, 8, 1000)])
@pytest.mark.parametrize("round_q", [False, True])
def test_attention_long_context_route_bit_exact(cfg, round_q):
    engine.set_attention_route(1)
    try:
        _attention_case(cfg, round_q)
    finally:
        engine.set_attention_route(0)


# one launch per layer, a cluster of 16 or 8 blocks per KV head, against the two launches: fewer vectors than blocks, stages that end inside, more stages than the ring has, contexts it leaves
@pytest.mark.parametrize("cfg", [(4, 1, 1), (4, 1, 17), (8, 1, 33), (32, 8, 130), (32, 8, 333), (64, 8, 1029), (64, 16, 700), (16, 4, 2050), (128, 16, 300), (64, 8, 4200), (8, 1, 9000), (8, 2, 20011)])
@pytest.mark.parametrize("round_q", [False, True])
@pytest.mark.parametrize("route", [2, 3])
def test_attention_routes_bit_exact(cfg, round_q, route):
    engine.set_attention_route(route)
    try:
        _attention_case(cfg, round_q)
    finally:
        engine.set_attention_route(0)


@pytest.mark.parametrize("cfg,want", [((4, 1, 17), {16}), ((8, 1, 33), {16}), ((16, 4, 2050), {16}), ((32, 8, 130), {8, 16}), ((32, 8, 333), {8, 16}), ((64, 8, 1029), {8, 16}),
                                      ((64, 16, 700), {0, 8}), ((8, 1, 9000), {0}), ((8, 2, 20011), {0}), ((64, 32, 100), {0}), ((2, 2, 100), {0})])
def test_the_one_launch_attention_runs_where_it_is_asked_for(cfg, want):
    """blocks of a cluster: as many as fit beside one another (eight clusters of 16 do not on every GPU, nor sixteen of 8), whatever was asked for before; 0 where the routes test
    compares two launches with themselves"""
    ask = _lib.lib().b200_op_attention_cluster
    try:
        engine.set_attention_route(3)
        first = ask(*cfg)
        assert first in want
        for n_kv in (8000, 32, 4200, 1536):
            ask(cfg[0], cfg[1], n_kv)
        assert ask(*cfg) == first
        for route in (2, 1, 0):                               # (0: products by themselves stand behind no qkv)
            engine.set_attention_route(route)
            assert ask(*cfg) == 0
    finally:
        engine.set_attention_route(0)


@pytest.mark.parametrize("cfg", [(2, 2, 50176), (2, 2, 12000), (4, 2, 25088), (8, 2, 12544), (8, 1, 6272), (8, 2, 7200), (2, 2, 14208), (2, 2, 11360), (2, 2, 11361)])
def test_attention_where_v_goes_round_its_slots(cfg):
    """soft-max . V of one token: the longest context of each number of heads per key head (slots of 96 to 352 positions), and V that just fits its four slots and just does not"""
    _attention_case(cfg, False)


def _attention_case(cfg, round_q):
    n_head, n_head_kv, n_kv = cfg
    hd = 128
    rng = np.random.default_rng(n_kv)
    q = (rng.standard_normal(n_head * hd) * 2).astype(np.float32)
    k = rng.standard_normal((n_kv, n_head_kv * hd)).astype(np.float16)
    v = rng.standard_normal((n_kv, n_head_kv * hd)).astype(np.float16)
    scale = 1.0 / np.sqrt(hd)
    y = engine.op_attention(q, k, v, n_kv, n_head, n_head_kv, hd, scale, round_q)
    yr = port.attention(q, k, v, n_kv, n_head, n_head_kv, hd, scale, round_q)
    assert np.array_equal(y, yr), f"max abs diff {np.abs(y - yr).max()} rel {rel_err(y, yr)}"


# ---- batch > 1 mat-mul (prompt batches): k_mma_batch on the tensor cores for K-quants, k_matmul_batch (dp4a) for Q8_0 ----
@pytest.mark.parametrize("name", list(TYPES))
@pytest.mark.parametrize("shape", [(64, 256, 8), (128, 768, 33), (1024, 4096, 70), (96, 14336, 31), (320, 4096, 512)])
def test_mul_mat_batch_vs_port(name, shape):
    """x[T][k] through the prompt-batch kernels equals the reference arithmetic token by token (ragged T, rows that are not
    a multiple of 64, one K step and 56 of them)"""
    n, k, T = shape
    t = TYPES[name]
    rng = np.random.default_rng(n * 7 + k + T)
    w = G.random_blocks(rng, t, n, k)
    x = (rng.standard_normal((T, k)) * rng.choice([0.01, 1.0, 30.0], size=(T, 1))).astype(np.float32)
    x[min(3, T - 1), :256] = 0.0
    y = engine.op_mul_mat(t, w, n, k, x)
    for i in sorted(set([0, 1, T // 2, T - 2, T - 1])):
        yr = port.mul_mat_vec(t, w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"token {i}: max abs diff {np.abs(y[i] - yr).max()} rel {rel_err(y[i], yr)}"


def _extreme_blocks(name, n, k, rng):
    """rows of worst-case magnitudes for the exact-fp16 argument of prefill_mma.cuh: largest quants x largest sub-block
    scales (Q4_K 15*63, Q5_K 31*63, Q6_K -32*-128 and 31*127), mixed with random rows"""
    t = TYPES[name]
    w = G.random_blocks(rng, t, n, k).reshape(n, -1).copy()
    nb = k // 256
    if name == "Q4_K":
        blk = np.full(144, 0xFF, np.uint8); blk[0:4] = np.array([1.0, 0.5], np.float16).view(np.uint8)
    elif name == "Q5_K":
        blk = np.full(176, 0xFF, np.uint8); blk[0:4] = np.array([1.0, 0.5], np.float16).view(np.uint8)
    elif name == "Q6_K":
        blk = np.zeros(210, np.uint8); blk[192:208] = 0x80; blk[208:210] = np.array([1.0], np.float16).view(np.uint8)
    else:
        blk = np.full(34, 0x81, np.uint8); blk[0:2] = np.array([1.0], np.float16).view(np.uint8)
    per = blk.size
    reps = w.shape[1] // per
    w[0::4] = np.tile(blk, reps)
    if name == "Q6_K":   # q = 63 (w = +31, odd), scale +127
        b2 = np.full(210, 0xFF, np.uint8); b2[192:208] = 0x7F; b2[208:210] = np.array([1.0], np.float16).view(np.uint8)
        w[1::4] = np.tile(b2, nb)
    return w.reshape(-1)


@pytest.fixture
def prefill_mma():
    """engine.set_prefill_mma, which holds for the whole process: back at the default when the test ends"""
    yield engine.set_prefill_mma
    engine.set_prefill_mma(2)


@pytest.mark.parametrize("k", [1024, 4096])
@pytest.mark.parametrize("name", list(TYPES))
def test_mul_mat_batch_extremes(name, k):
    """every quant at +-127 against the largest weights: the integer sums reach their bounds (Q6_K: 32 * 4096 * 127 < 2^24)
    and must still come out of the fp16 tensor-core contraction exactly, through mma.sync (short rows, Q5_K) and tcgen05 (long ones)"""
    rng = np.random.default_rng(11)
    n, T = 64, 40
    w = _extreme_blocks(name, n, k, rng)
    x = rng.standard_normal((T, k)).astype(np.float32)
    x[0] = 3.0; x[1] = -3.0                          # every quant -127 / +127
    x[2] = np.where(np.arange(k) % 2 == 0, 5.0, -5.0)
    x[3, :] = 0.0; x[3, ::256] = 1.0                 # a single non-zero per block
    y = engine.op_mul_mat(TYPES[name], w, n, k, x)
    for i in range(T if name != "Q8_0" else 8):
        yr = port.mul_mat_vec(TYPES[name], w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"token {i}: max abs diff {np.abs(y[i] - yr).max()}"


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("shape", [(32, 2048, 1), (160, 2304, 32), (416, 4096, 65), (20480, 2048, 40), (9536, 256, 1), (9536, 2304, 32), (4800, 4096, 65)])
def test_mul_mat_batch_tcgen05_edges(name, shape, prefill_mma):
    """k_umma_batch where its tiles end: half of a 128-row tile (the operator pads to two units of 32 rows), one super-block, one token past a tile, more tiles
    than SMs (a CTA's second tile starts behind its first one's epilogue), and where its rule begins: one tile of mma.sync past a wave, for every type — the
    reference's bits, on the largest weights and, for the first and last token, the largest quants"""
    n, k, T = shape
    rng = np.random.default_rng(n + k + T)
    w = _extreme_blocks(name, n, k, rng)
    x = (rng.standard_normal((T, k)) * rng.choice([0.01, 1.0, 30.0], size=(T, 1))).astype(np.float32)
    x[0], x[-1] = 3.0, -3.0
    prefill_mma(2)
    if n > 1000 or name != "Q5_K":
        rows = (n + 63) // 64 * 64
        assert _lib.lib().b200_op_prompt_kernel((C.c_int32 * 1)(TYPES[name]), 1, rows // 32, k, T, 148) == 2
    y = engine.op_mul_mat(TYPES[name], w, n, k, x)
    for i in sorted({0, T // 2, T - 1}):
        yr = port.mul_mat_vec(TYPES[name], w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"token {i}: max abs diff {np.abs(y[i] - yr).max()}"


@pytest.mark.parametrize("name", list(TYPES))
@pytest.mark.parametrize("T", [1, 16, 48])
def test_mul_mat_batch_halves_without_tokens(name, T, prefill_mma):
    """tile halves without tokens, whose warps only hand super-blocks on: over rings that go round many times and several tiles per CTA, the last tile's half alone and every
    tile's — the reference's bits"""
    n, k = 20480, 4096
    rng = np.random.default_rng(T)
    w = G.random_blocks(rng, TYPES[name], n, k).reshape(-1)
    x = rng.standard_normal((T, k)).astype(np.float32)
    prefill_mma(2)
    y = engine.op_mul_mat(TYPES[name], w, n, k, x)
    for i in sorted({0, T - 1}):
        yr = port.mul_mat_vec(TYPES[name], w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"token {i}: max abs diff {np.abs(y[i] - yr).max()}"


@pytest.mark.parametrize("shape", [(64, 256, 1), (64, 512, 33), (192, 256, 31), (320, 4352, 32), (19072, 256, 40), (128, 14336, 65)])
def test_mul_mat_batch_q8_0_edges(shape):
    """k_umma_batch_q80 where its tiles and rings end: half of a 128-row tile, two to 112 stages of four blocks (the first fewer than the ring has), one token past a
    tile and one short of it, more tiles than SMs — the reference's bits, on the largest weights, zero blocks and scales at the end of fp16's range"""
    n, k, T = shape
    rng = np.random.default_rng(n + k + T)
    w = _extreme_blocks("Q8_0", n, k, rng).reshape(n, -1)
    w[1::4, :34] = 0                                                       # a block of zeros with a scale of zero
    w[2::4, 0:2] = np.array([6e-8], np.float16).view(np.uint8)             # a sub-normal scale
    x = (rng.standard_normal((T, k)) * rng.choice([1e-6, 0.01, 1.0, 30.0], size=(T, 1))).astype(np.float32)
    x[0], x[-1] = 3.0, -3.0
    x[T // 2, :32] = 0.0
    w = w.reshape(-1)
    y = engine.op_mul_mat(TYPES["Q8_0"], w, n, k, x)
    for i in sorted({0, T // 2, T - 1}):
        yr = port.mul_mat_vec(TYPES["Q8_0"], w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"token {i}: max abs diff {np.abs(y[i] - yr).max()}"


@pytest.mark.parametrize("shape", [(9472, 512, 17), (9472, 512, 32), (9536, 512, 32), (9536, 512, 17), (6272, 256, 33), (6272, 256, 48), (6336, 256, 48), (128, 4096, 49), (640, 768, 250), (192, 256, 512)])
def test_mul_mat_batch_q8_0_halves(shape):
    """k_umma_batch_q80 with a block per half of a token tile: as many of them as SMs and one row tile more (whole tiles), two, three and four halves, a half with one token, an odd
    number of units — the reference's bits at both ends of every half"""
    n, k, T = shape
    rng = np.random.default_rng(n + k + T)
    w = G.random_blocks(rng, TYPES["Q8_0"], n, k).reshape(-1)
    x = rng.standard_normal((T, k)).astype(np.float32)
    y = engine.op_mul_mat(TYPES["Q8_0"], w, n, k, x)
    for i in sorted({t for h in range(0, T, 16) for t in (h, min(h + 15, T - 1))}):
        yr = port.mul_mat_vec(TYPES["Q8_0"], w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"token {i}: max abs diff {np.abs(y[i] - yr).max()}"


@pytest.mark.parametrize("shape", [(32, 256), (96, 768), (4736, 512), (4768, 256), (9504, 768), (14240, 1280), (64, 14336), (160, 17408)])
def test_mul_mat_vec_q8_0_edges(shape):
    """k_matvec_q80 where its teams and rings end: one stage, stages of eight and of 16 blocks, as many units of 32 rows as SMs and one more (a block's second team), more
    than both teams take at once, a ring that goes round, a vector of more than one pass of the quantizer — the reference's bits"""
    n, k = shape
    rng = np.random.default_rng(n + k)
    w = _extreme_blocks("Q8_0", n, k, rng).reshape(n, -1)
    w[1::4, :34] = 0
    w[2::4, 0:2] = np.array([6e-8], np.float16).view(np.uint8)
    x = (rng.standard_normal(k) * rng.choice([1e-6, 1.0, 30.0], size=k)).astype(np.float32)
    x[32:64] = 0.0
    y = engine.op_mul_mat_vec(TYPES["Q8_0"], w.reshape(-1), n, k, x)
    yr = port.mul_mat_vec(TYPES["Q8_0"], w.reshape(-1), n, k, x)
    assert np.array_equal(y, yr), f"max abs diff {np.abs(y - yr).max()}"


@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K"])
@pytest.mark.parametrize("shape", [(32, 256), (96, 768), (4736, 512), (4768, 256), (9504, 768), (14240, 1280), (64, 14336), (160, 17408), (4768, 9216),
                                   (18944, 512), (18976, 512), (18976, 4352), (37888, 256), (37920, 256), (37952, 2304)])
def test_mul_mat_vec_k_quant_edges(name, shape):
    """k_matvec_kq where its teams and rings end: one block of K, stages of one and of two blocks, as many units of 32 rows as SMs and one more (a block's second team), as many as
    the four teams of one row per thread and one more (two rows per thread from there), as many as their eight teams and one more (a team's second unit, taken by some), rings
    that go round, vectors of one and of several blocks per warp and of more than one pass, worst-case weights — the reference's bits"""
    n, k = shape
    rng = np.random.default_rng(n + k)
    w = _extreme_blocks(name, n, k, rng)
    x = (rng.standard_normal(k) * rng.choice([1e-6, 1.0, 30.0], size=k)).astype(np.float32)
    x[:256] = np.where(rng.random(256) < 0.5, 30.0, -30.0).astype(np.float32)
    if k > 256:
        x[256:512] = 0.0
    y = engine.op_mul_mat_vec(TYPES[name], w.reshape(-1), n, k, x)
    yr = port.mul_mat_vec(TYPES[name], w.reshape(-1), n, k, x)
    assert np.array_equal(y, yr), f"max abs diff {np.abs(y - yr).max()}"


@pytest.mark.parametrize("name,shape", [("Q6_K", (64, 58368)), ("Q6_K", (64, 58624)), ("Q6_K", (4800, 60160)), ("Q8_0", (64, 171008)), ("Q8_0", (64, 171264))])
def test_mul_mat_vec_long_vectors(name, shape):
    """the longest vectors that the kernels with a chain per thread hold, and longer ones, which k_matvec takes — the reference's bits"""
    n, k = shape
    out = (C.c_int32 * 7)()
    assert _lib.lib().b200_op_lanes_shape((C.c_int32 * 1)(TYPES[name]), 1, n // 32, k, 0, 0, 148, out) == 0
    assert (out[0] == 0) == (k > (58368 if name == "Q6_K" else 171008))
    rng = np.random.default_rng(k)
    w = G.random_blocks(rng, TYPES[name], n, k).reshape(-1)
    x = rng.standard_normal(k).astype(np.float32)
    assert np.array_equal(engine.op_mul_mat_vec(TYPES[name], w, n, k, x), port.mul_mat_vec(TYPES[name], w, n, k, x))


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("name", ["Q4_K", "Q5_K", "Q6_K", "Q8_0"])
def test_mul_mat_batch_kernel_variants(name, mode, prefill_mma):
    """the batch kernels — mma.sync (1; Q8_0: the block-diagonal HMMA kernel), tcgen05 (2, default; K-quants), dp4a (0): A/B
    switch b200_set_prefill_mma — give the reference's bits, on random blocks and on the worst-case magnitudes"""
    rng = np.random.default_rng(3)
    n, k, T = 256, 2048, 100
    x = rng.standard_normal((T, k)).astype(np.float32)
    x[0] = 3.0; x[1] = -3.0
    w = _extreme_blocks(name, n, k, rng)
    prefill_mma(mode)
    y = engine.op_mul_mat(TYPES[name], w, n, k, x)
    for i in (0, 1, 2, 50, 99):
        yr = port.mul_mat_vec(TYPES[name], w, n, k, x[i])
        assert np.array_equal(y[i], yr), f"mode {mode} token {i}: max abs diff {np.abs(y[i] - yr).max()}"
