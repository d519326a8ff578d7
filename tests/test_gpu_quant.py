"""GPU parity for block-quantized weights: dequantise/quantise bit-exact with the oracle, linear and
embedding against the reference's golden vectors and against the oracle on seeded inputs."""
import numpy as np
import pytest
import torch

import effect_torch_b200 as et
import oracle as orc
from tests import helpers
from tests.golden import reference_vectors as gv
from tests.gpu_util import dev, empty, host, runtime

pytestmark = pytest.mark.gpu

ALL_CODECS = [gv.Q4_0, gv.Q8_0, gv.Q2_K, gv.Q3_K, gv.Q4_K, gv.Q5_K, gv.Q6_K]
SCALE_FIELDS = {gv.Q4_0: [0], gv.Q8_0: [0], gv.Q2_K: [80, 82], gv.Q3_K: [108], gv.Q4_K: [0, 2], gv.Q5_K: [0, 2], gv.Q6_K: [208]}
REL_TOL = 2e-3  # tolerance on f16/f32 linear outputs, as max |err| / max |ref|


def random_packed(codec, rows, columns, seed, spread=0.01):
    """Random packed bytes with finite f16 scale fields (every bit pattern of the code bytes is legal)."""
    rng = np.random.default_rng(seed)
    bb, bv = orc.block_bytes(codec), orc.block_values(codec)
    blocks = rows * columns // bv
    raw = rng.integers(0, 256, size=(blocks, bb), dtype=np.uint8)
    for off in SCALE_FIELDS[codec]:
        scale = rng.normal(0, spread, size=blocks).astype(np.float16)
        raw[:, off:off + 2] = scale.view(np.uint8).reshape(blocks, 2)
    return raw.reshape(rows, columns // bv * bb)


# Block scales of K-quants as files have them (weights near 0.01), and as random_packed draws them: effective scales below and
# from 2^-5 on, the line between the two forms of the expansion to f16.
K_SPREADS = ["model", "wide"]


def k_packed(codec, rows, columns, seed, spread):
    return random_packed(codec, rows, columns, seed, helpers.K_SCALE_SIGMA[codec] / 2 if spread == "model" else 0.01)


def whole_warps_below_the_line(scales, blocks):
    """scales [rows, 32-value blocks (, scales per block)] -> for each dequant warp (32 rows) and run of `blocks` blocks that it
    expands together, whether all of its scales are below 2^-5."""
    rows, total = scales.shape[:2]
    runs = np.abs(scales.astype(np.float64)).reshape(rows // 32, 32, total // blocks, -1)
    return runs.max(axis=(1, 3)) < 2.0 ** -5


@pytest.mark.parametrize("codec", [gv.Q2_K, gv.Q3_K, gv.Q4_K, gv.Q5_K, gv.Q6_K])
def test_k_quant_fixtures_decode_exactly_on_gpu(codec):
    block, _, _ = gv.K_QUANT_FIXTURES[codec]
    out = empty((1, 256))
    runtime().dequantize_into(codec, dev(block.reshape(1, -1)), 1, 256, out)
    np.testing.assert_array_equal(host(out)[0], gv.fixture_expected(codec))


@pytest.mark.parametrize("codec", ALL_CODECS)
def test_dequantize_is_bit_exact_with_the_oracle(codec):
    rows, columns = 37, 1024
    packed = random_packed(codec, rows, columns, seed=codec)
    out = empty((rows, columns))
    runtime().dequantize_into(codec, dev(packed), rows, columns, out)
    expected = orc.dequantize(codec, packed, rows, columns)
    np.testing.assert_array_equal(host(out).view(np.uint32), expected.view(np.uint32))


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
def test_quantizer_is_bit_exact_with_the_oracle(codec):
    rng = np.random.default_rng(2)
    w = rng.normal(0, 0.02, size=(64, 512)).astype(np.float32)
    w[0, :32] = 0.0                       # all-zero block
    w[1, :32] = 0.01                      # every magnitude ties
    w[2, :32] = np.linspace(-1, 1, 32)    # extreme at the first element
    w[3, :32] = np.linspace(1, -1, 32)
    packed = empty((64, orc.encoded_row_bytes(codec, 512)), dtype=torch.uint8)
    runtime().quantize_into(codec, dev(w), 64, 512, packed)
    np.testing.assert_array_equal(host(packed), orc.quantize(codec, w))


@pytest.mark.parametrize("case", [gv.linear_prefill_case(), gv.linear_lowered_case()])
def test_quantized_linear_golden_vectors(case):
    x = case["x"]
    out = empty((x.shape[0], case["rows"]))
    bias = None if case["bias"] is None else dev(case["bias"])
    runtime().qlinear_into(case["codec"], dev(x), x.shape[0], case["columns"], dev(case["packed"]), case["rows"], bias, out)
    np.testing.assert_array_equal(host(out), case["expected"])


@pytest.mark.parametrize("codec", ALL_CODECS)
@pytest.mark.parametrize("vectors", [1, 3, 11])
def test_generic_linear_matches_the_oracle(codec, vectors):
    rng = np.random.default_rng(100 + codec)
    rows, columns = 96, 1024
    packed = random_packed(codec, rows, columns, seed=50 + codec)
    x = rng.normal(size=(vectors, columns)).astype(np.float32)
    bias = rng.normal(size=rows).astype(np.float32)
    out = empty((vectors, rows))
    runtime().qlinear_into(codec, dev(x), vectors, columns, dev(packed), rows, dev(bias), out)
    expected = orc.qlinear(codec, x, packed, rows, columns, bias, threads=4)
    assert helpers.rel_err(host(out), expected) <= REL_TOL


@pytest.mark.parametrize("codec", ALL_CODECS)
@pytest.mark.parametrize("rows,windows,vectors", [(1, 1, 1), (9, 17, 2), (33, 5, 6), (4099, 9, 4), (70, 70, 9)])
def test_raw_kernels_at_the_edges_of_their_tiles(codec, rows, windows, vectors):
    """Rows that do not fill a warp, columns that end inside a 256-value window, several staged chunks, a second pass over the
    vectors; and decoding of value counts that do not fill a warp's four windows, at a 2-byte-aligned address."""
    rng = np.random.default_rng(7 * codec + rows)
    columns = windows * 256 if orc.block_values(codec) == 256 else windows * 256 - 96
    packed = random_packed(codec, rows, columns, seed=rows + codec)
    x = rng.normal(size=(vectors, columns)).astype(np.float32)
    out = empty((vectors, rows))
    runtime().qlinear_into(codec, dev(x), vectors, columns, dev(packed), rows, None, out)
    expected = x.astype(np.float64) @ orc.dequantize(codec, packed, rows, columns).astype(np.float64).T
    assert np.abs(host(out) - expected).max() <= 2e-6 * np.sqrt(columns) * np.abs(expected).max()
    shifted = dev(np.concatenate([np.zeros(2, np.uint8), packed.reshape(-1)]))
    decoded = empty((rows, columns))
    runtime().dequantize_into(codec, shifted[2:], rows, columns, decoded)
    np.testing.assert_array_equal(host(decoded).view(np.uint32), orc.dequantize(codec, packed, rows, columns).view(np.uint32))


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
@pytest.mark.parametrize("rows,columns", [(1, 32), (5, 1600), (255, 32), (257, 96)])
def test_quantizer_tails(codec, rows, columns):
    w = np.random.default_rng(rows).normal(0, 0.02, size=(rows, columns)).astype(np.float32)
    w[0, 3] = -w[0, 17]  # equal magnitudes: the first decides the sign
    packed = empty((rows, orc.encoded_row_bytes(codec, columns)), dtype=torch.uint8)
    runtime().quantize_into(codec, dev(w), rows, columns, packed)
    np.testing.assert_array_equal(host(packed), orc.quantize(codec, w))


@pytest.mark.parametrize("codec", [orc.Q4_0, orc.Q8_0])
@pytest.mark.parametrize("shift", [0, 1, 2, 4, 8])
def test_quantizer_of_inputs_on_any_boundary(codec, shift):
    """Loads of 32 bytes, of 16 and of single values; the last CTA has three blocks."""
    w = np.random.default_rng(shift).normal(0, 0.02, size=(43, 288)).astype(np.float32)
    held = empty((w.size + shift,))
    held[shift:] = dev(w).reshape(-1)
    packed = empty((43, orc.encoded_row_bytes(codec, 288)), dtype=torch.uint8)
    runtime().quantize_into(codec, held[shift:], 43, 288, packed)
    np.testing.assert_array_equal(host(packed), orc.quantize(codec, w))


@pytest.mark.parametrize("codec", [orc.Q4_0, orc.Q8_0, orc.Q4_K, orc.Q6_K])
@pytest.mark.parametrize("shift", [0, 1, 4, 8])
@pytest.mark.parametrize("rows", [1, 13])
def test_dequantize_to_any_boundary(codec, shift, rows):
    """Stores of 32 bytes, of 16 and of single values; the last warp has one or two of its four windows; nothing beyond the end is written."""
    columns = 1280 if codec not in (orc.Q4_0, orc.Q8_0) else 1312
    packed = random_packed(codec, rows, columns, seed=shift)
    out = empty((rows * columns + shift + 8,))
    runtime().dequantize_into(codec, dev(packed), rows, columns, out[shift:])
    got, expected = host(out), orc.dequantize(codec, packed, rows, columns).reshape(-1)
    np.testing.assert_array_equal(got[shift:shift + expected.size].view(np.uint32), expected.view(np.uint32))
    assert not got[:shift].any() and not got[shift + expected.size:].any()


@pytest.mark.parametrize("codec", [orc.Q4_0, orc.Q8_0])
def test_quantizer_of_blocks_with_values_that_are_not_finite(codec):
    """A NaN takes no part in its block's scale, wherever it stands; an infinity makes the scale infinite."""
    rng = np.random.default_rng(29)
    x = rng.normal(size=(40, 32)).astype(np.float32)
    x[np.arange(32), np.arange(32)] = np.nan
    x[32, ::8] = np.nan
    x[33, :31] = np.nan
    x[34] = np.nan
    x[35, 5] = np.inf
    x[36, 30] = -np.inf
    x[37, 0], x[37, 17] = np.nan, np.inf
    x[38] = 0.0
    x[39] = -0.0
    packed = empty((40, et.encoded_row_bytes(codec, 32)), dtype=torch.uint8)
    runtime().quantize_into(codec, dev(x), 40, 32, packed)
    np.testing.assert_array_equal(host(packed), orc.quantize(codec, x).reshape(40, -1))


def test_linear_rejects_bad_geometry_and_observes_cancellation():
    rt = runtime()
    x, w, out = empty((1, 256)), empty((1, 144), dtype=torch.uint8), empty((1, 1))
    with pytest.raises(et.BackendError, match="logical row width 255 is invalid for Q4_K"):
        rt.qlinear_into(gv.Q4_K, x, 1, 255, w, 1, None, out)
    with pytest.raises(et.BackendError, match="^operation aborted$") as e:
        rt.qlinear_into(gv.Q4_K, x, 1, 256, w, 1, None, out, cancelled=True)
    assert e.value.reason == "cancelled"


@pytest.mark.parametrize("i64", [False, True])
def test_embedding_selected_rows_both_index_types(i64):
    block, _, _ = gv.K_QUANT_FIXTURES[gv.Q5_K]
    packed = np.zeros((3, block.size), dtype=np.uint8)
    packed[1] = block
    idx = dev(np.asarray([1, 1], dtype=np.int64 if i64 else np.uint32))
    out = empty((2, 256))
    runtime().qembedding_into(gv.Q5_K, idx, i64, 2, dev(packed), 3, 256, out)
    got = host(out)
    np.testing.assert_array_equal(got[0], gv.fixture_expected(gv.Q5_K))
    np.testing.assert_array_equal(got[1], gv.fixture_expected(gv.Q5_K))


@pytest.mark.parametrize("index", [-1, 1])
def test_embedding_reports_out_of_range_indexes(index):
    block, _, _ = gv.K_QUANT_FIXTURES[gv.Q2_K]
    out = empty((1, 256))
    runtime().qembedding_into(gv.Q2_K, dev(np.asarray([index], dtype=np.int64)), True, 1, dev(block.reshape(1, -1)), 1, 256, out)
    with pytest.raises(et.BackendError, match=r"outside 0\.\.1") as e:
        runtime().synchronize()
    assert e.value.reason == "execution-failed"
    runtime().synchronize()  # the status word was cleared: the runtime stays usable


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
def test_tiling_preserves_every_weight(codec):
    """x = identity picks out single weights: the tensor-core tiling must hold the same dequantised values
    (to f16 rounding of scale*code, the operand precision of the MMA path)."""
    rng = np.random.default_rng(7)
    rows, columns = 48, 128
    w = rng.normal(0, 0.02, size=(rows, columns)).astype(np.float32)
    packed = orc.quantize(codec, w)
    deq = orc.dequantize(codec, packed, rows, columns)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    eye = dev(np.eye(columns, dtype=np.float32))
    out = empty((columns, rows))
    qw.linear_into(eye, columns, out)
    got = host(out).T
    np.testing.assert_allclose(got, deq, rtol=2.0 ** -10, atol=1e-9)


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
@pytest.mark.parametrize("vectors", [32, 128, 200])
def test_expansion_is_exact_for_every_code_and_scale(codec, vectors):
    """Both forms of the expansion to f16 (block scales below and from 2^-5 on) give each weight scale * code rounded once to
    f16: all codes under scales at the line between the forms, subnormal, tiny, large and of either sign. x picks out single
    weights, whose f32 sums with zeros are exact."""
    columns, bb = 128, orc.block_bytes(codec)
    line = 2.0 ** -5
    scales = np.array([line, np.nextafter(np.float16(line), np.float16(0)), line * 1.5, 0.006, 6e-8, 6.1e-5, 0.0, 1.0, 200.0], np.float16)
    scales = np.concatenate([scales, -scales])
    rng = np.random.default_rng(5)
    # a warp (32 rows) of each scale, then three with scales below the line mixed and three with all of them mixed
    mixed = 3 * 32
    rows = 32 * len(scales) + 2 * mixed
    raw = rng.integers(0, 256, size=(rows, columns // 32, bb), dtype=np.uint8)
    held = np.empty((rows, columns // 32), np.float16)
    held[:-2 * mixed] = np.repeat(scales, 32)[:, None]
    held[-2 * mixed:-mixed] = rng.choice(scales[np.abs(scales) < line], size=(mixed, columns // 32))
    held[-mixed:] = rng.choice(scales, size=(mixed, columns // 32))
    raw[:, :, 0:2] = held[:, :, None].view(np.uint8).reshape(rows, columns // 32, 2)
    for blocks in (2, 4):  # that a warp of the two linears expands together
        small = whole_warps_below_the_line(held, blocks).all(axis=1)
        assert [int(small[:9].sum()), int(small[9:18].sum())] == [5, 5] and small[1] and small[18:21].all() and not small[21:].any()
    packed = raw.reshape(rows, -1)
    expected = orc.dequantize(codec, packed, rows, columns).astype(np.float16).astype(np.float32)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    x = np.zeros((vectors, columns), np.float32)
    x[np.arange(min(vectors, columns)), np.arange(min(vectors, columns))] = 1.0
    out = empty((vectors, rows))
    qw.linear_into(dev(x), vectors, out)
    n = min(vectors, columns)
    np.testing.assert_array_equal(host(out)[:n].T, expected[:, :n])


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
@pytest.mark.parametrize("rows,columns", [(256, 512), (200, 1024), (1024, 4096)])
@pytest.mark.parametrize("vectors", [1, 5, 8, 9, 16, 32, 40, 64, 100, 300])
def test_tiled_linear_matches_the_oracle(codec, rows, columns, vectors):
    rng = np.random.default_rng(rows + columns + vectors)
    w = rng.normal(0, 0.02, size=(rows, columns)).astype(np.float32)
    packed = orc.quantize(codec, w)
    x = rng.normal(size=(vectors, columns)).astype(np.float32)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    out = empty((vectors, rows))
    qw.linear_into(dev(x), vectors, out)
    expected = orc.qlinear(codec, x, packed, rows, columns, threads=8)
    assert helpers.rel_err(host(out), expected) <= REL_TOL


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
@pytest.mark.parametrize("vectors", [4, 32])
def test_tiled_linear_epilogues(codec, vectors):
    rng = np.random.default_rng(9)
    d, ffn = 512, 384
    gate = rng.normal(0, 0.05, size=(ffn, d)).astype(np.float32)
    up = rng.normal(0, 0.05, size=(ffn, d)).astype(np.float32)
    down = rng.normal(0, 0.05, size=(d, ffn)).astype(np.float32)
    pg, pu, pd = orc.quantize(codec, gate), orc.quantize(codec, up), orc.quantize(codec, down)
    x = rng.normal(size=(vectors, d)).astype(np.float32)
    residual = rng.normal(size=(vectors, d)).astype(np.float32)
    bias = rng.normal(size=d).astype(np.float32)
    rt = runtime()
    # fused gate/up with the SwiGLU epilogue
    qgu = et.QWeight(rt, codec, [dev(pg), dev(pu)], [ffn, ffn], d, interleave8=True)
    act = empty((vectors, ffn))
    qgu.linear_into(dev(x), vectors, act, epilogue=et.EPILOGUE_SWIGLU)
    expected_act = orc.silu_mul(orc.qlinear(codec, x, pg, ffn, d, threads=4), orc.qlinear(codec, x, pu, ffn, d, threads=4))
    assert helpers.rel_err(host(act), expected_act) <= REL_TOL
    # down projection with bias and the residual epilogue
    qd = et.QWeight(rt, codec, [dev(pd)], [d], ffn)
    out = empty((vectors, d))
    qd.linear_into(dev(expected_act), vectors, out, bias=dev(bias), residual=dev(residual), epilogue=et.EPILOGUE_RESIDUAL)
    expected = residual + orc.qlinear(codec, expected_act, pd, d, ffn, bias, threads=4)
    assert helpers.rel_err(host(out), expected) <= REL_TOL
    # concatenated q/k/v parts
    qkv = et.QWeight(rt, codec, [dev(pg), dev(pu)], [ffn, ffn], d)
    both = empty((vectors, 2 * ffn))
    qkv.linear_into(dev(x), vectors, both)
    expected_both = np.concatenate([orc.qlinear(codec, x, pg, ffn, d, threads=4), orc.qlinear(codec, x, pu, ffn, d, threads=4)], axis=1)
    assert helpers.rel_err(host(both), expected_both) <= REL_TOL


@pytest.mark.parametrize("codec,ffn,d,vectors", [(gv.Q4_0, 9728, 512, 20), (gv.Q4_0, 14336, 1024, 33), (gv.Q8_0, 9600, 256, 32)])
def test_single_split_launch_with_more_tiles_than_sms(codec, ffn, d, vectors):
    """More 128-row tiles than SMs and not a multiple of them (152, 224 and 150 tiles on 148 SMs), one split: the SwiGLU
    epilogue over interleaved gate/up rows and bias + residual over plain rows, each run twice and bit-identical."""
    rng = np.random.default_rng(ffn + d)
    gate = rng.normal(0, 0.05, size=(ffn, d)).astype(np.float32)
    up = rng.normal(0, 0.05, size=(ffn, d)).astype(np.float32)
    pg, pu = orc.quantize(codec, gate), orc.quantize(codec, up)
    x = rng.normal(size=(vectors, d)).astype(np.float32)
    rt = runtime()
    qgu = et.QWeight(rt, codec, [dev(pg), dev(pu)], [ffn, ffn], d, interleave8=True)
    expected_act = orc.silu_mul(orc.qlinear(codec, x, pg, ffn, d, threads=8), orc.qlinear(codec, x, pu, ffn, d, threads=8))
    runs = []
    for _ in range(2):
        act = empty((vectors, ffn))
        qgu.linear_into(dev(x), vectors, act, epilogue=et.EPILOGUE_SWIGLU)
        runs.append(host(act))
        assert helpers.rel_err(runs[-1], expected_act) <= REL_TOL
    np.testing.assert_array_equal(runs[0], runs[1])
    plain = et.QWeight(rt, codec, [dev(pg), dev(pu)], [ffn, ffn], d)
    bias = rng.normal(size=2 * ffn).astype(np.float32)
    residual = rng.normal(size=(vectors, 2 * ffn)).astype(np.float32)
    expected = residual + np.concatenate([orc.qlinear(codec, x, pg, ffn, d, bias[:ffn], threads=8),
                                          orc.qlinear(codec, x, pu, ffn, d, bias[ffn:], threads=8)], axis=1)
    runs = []
    for _ in range(2):
        out = empty((vectors, 2 * ffn))
        plain.linear_into(dev(x), vectors, out, bias=dev(bias), residual=dev(residual), epilogue=et.EPILOGUE_RESIDUAL)
        runs.append(host(out))
        assert helpers.rel_err(runs[-1], expected) <= REL_TOL
    np.testing.assert_array_equal(runs[0], runs[1])


def recut(codec, packed, rows, columns):
    """The re-cut form of K-quant rows, from what the oracle decodes of them with their fields replaced: f16 scales
    [rows, 32-value blocks, 1 or 2] (two where each half of a block has its own), f16 minima or None, and f64 codes [rows, columns]."""
    blocks = packed.reshape(-1, orc.block_bytes(codec))

    def decode(d, dmin, code_bytes=()):
        changed = blocks.copy()
        for off, value in zip(SCALE_FIELDS[codec], (d, dmin)):
            changed[:, off:off + 2] = np.array([value], np.float16).view(np.uint8)
        for first, last, value in code_bytes:
            changed[:, first:last] = value
        return orc.dequantize(codec, changed.reshape(rows, -1), rows, columns)

    def field(off):  # of each 256-value block, as f32, repeated over its 32-value blocks
        return np.repeat(np.ascontiguousarray(blocks[:, off:off + 2]).view(np.float16).astype(np.float32).reshape(rows, -1), 8, axis=1)

    ones = {gv.Q3_K: [(0, 32, 0xff), (32, 96, 0x55)], gv.Q4_K: [(16, 144, 0x11)], gv.Q5_K: [(16, 48, 0), (48, 176, 0x11)],
            gv.Q6_K: [(0, 128, 0x11), (128, 192, 0xaa)]}[codec]  # every code 1
    per_value = decode(1.0, 0.0, ones)  # the whole-number sub-scales
    minimum = codec in (gv.Q4_K, gv.Q5_K)
    sub = per_value.reshape(rows, columns // 32, 32)[:, :, ::32 if minimum else 16]
    scales = (field(SCALE_FIELDS[codec][0])[:, :, None] * sub).astype(np.float16)
    minima = None
    if minimum:
        zeros = [(16, 144, 0)] if codec == gv.Q4_K else [(16, 176, 0)]
        minima = (field(2) * -decode(0.0, 1.0, zeros).reshape(rows, columns // 32, 32)[:, :, 0]).astype(np.float16)
    codes = np.divide(decode(1.0, 0.0), per_value, out=np.zeros((rows, columns)), where=per_value != 0, dtype=np.float64)
    return scales, minima, codes


@pytest.mark.parametrize("codec", [gv.Q3_K, gv.Q4_K, gv.Q5_K, gv.Q6_K])
@pytest.mark.parametrize("spread", K_SPREADS)
@pytest.mark.parametrize("vectors", [32, 128, 512])
def test_k_quant_expansion_rounds_once(codec, spread, vectors):
    """Both forms of the expansion give a re-cut weight as scale * code (- minimum) of its f16 scales, rounded once to f16: at
    the scales of model files (whole warps below the line between the forms) and beyond it. x picks out single weights."""
    rows, columns = 128, 512
    packed = k_packed(codec, rows, columns, 17, spread)
    scales, minima, codes = recut(codec, packed, rows, columns)
    assert np.array_equal(codes, np.rint(codes)) and np.ptp(codes) == {gv.Q3_K: 7, gv.Q4_K: 15, gv.Q5_K: 31, gv.Q6_K: 63}[codec]
    for blocks in (2, 4):
        small = whole_warps_below_the_line(scales, blocks)
        assert small.all() if spread == "model" else not small.all()
    weights = np.repeat(scales.astype(np.float64), 32 // scales.shape[2], axis=2).reshape(rows, columns) * codes
    if minima is not None:
        weights -= np.repeat(minima.astype(np.float64), 32, axis=1)
    expected = weights.astype(np.float16).astype(np.float32)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    x = np.zeros((vectors, columns), np.float32)
    picked = np.sort(np.random.default_rng(1).permutation(columns)[:vectors])
    x[np.arange(vectors), picked] = 1.0
    out = empty((vectors, rows))
    qw.linear_into(dev(x), vectors, out)
    np.testing.assert_array_equal(host(out).T, expected[:, picked])


@pytest.mark.parametrize("codec", [gv.Q3_K, gv.Q4_K, gv.Q5_K, gv.Q6_K])
@pytest.mark.parametrize("spread", K_SPREADS)
def test_k_quant_tiling_preserves_every_weight(codec, spread):
    """The 256-value K-quant blocks are re-cut into 32-value blocks at load (effective scales rounded to f16): x = identity
    picks out single weights, which must equal the reference decode to the f16 precision of the MMA operands."""
    rows, columns = 40, 512
    packed = k_packed(codec, rows, columns, 11, spread)
    deq = orc.dequantize(codec, packed, rows, columns)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    out = empty((columns, rows))
    qw.linear_into(dev(np.eye(columns, dtype=np.float32)), columns, out)
    scale = np.abs(deq).max()
    np.testing.assert_allclose(host(out).T, deq, rtol=2.0 ** -9, atol=scale * 2.0 ** -10)


@pytest.mark.parametrize("codec", [gv.Q3_K, gv.Q4_K, gv.Q5_K, gv.Q6_K])
@pytest.mark.parametrize("rows,columns", [(256, 512), (200, 1024), (1024, 4096)])
@pytest.mark.parametrize("vectors", [1, 8, 17, 32, 64, 300])
@pytest.mark.parametrize("spread", K_SPREADS)
def test_k_quant_tiled_linear_matches_the_oracle(codec, rows, columns, vectors, spread):
    rng = np.random.default_rng(rows + columns + vectors)
    packed = k_packed(codec, rows, columns, rows + vectors, spread)
    x = rng.normal(size=(vectors, columns)).astype(np.float32)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    out = empty((vectors, rows))
    qw.linear_into(dev(x), vectors, out)
    expected = orc.qlinear(codec, x, packed, rows, columns, threads=8)
    assert helpers.rel_err(host(out), expected) <= REL_TOL


@pytest.mark.parametrize("codec", [gv.Q3_K, gv.Q4_K, gv.Q5_K, gv.Q6_K])
@pytest.mark.parametrize("spread", K_SPREADS)
def test_k_quant_fused_gate_up_and_residual_epilogues(codec, spread):
    rng = np.random.default_rng(21)
    d, ffn, vectors = 512, 256, 20
    pg, pu, pd = k_packed(codec, ffn, d, 1, spread), k_packed(codec, ffn, d, 2, spread), k_packed(codec, d, ffn, 3, spread)
    x = rng.normal(size=(vectors, d)).astype(np.float32)
    residual = rng.normal(size=(vectors, d)).astype(np.float32)
    rt = runtime()
    qgu = et.QWeight(rt, codec, [dev(pg), dev(pu)], [ffn, ffn], d, interleave8=True)
    act = empty((vectors, ffn))
    qgu.linear_into(dev(x), vectors, act, epilogue=et.EPILOGUE_SWIGLU)
    expected_act = orc.silu_mul(orc.qlinear(codec, x, pg, ffn, d, threads=4), orc.qlinear(codec, x, pu, ffn, d, threads=4))
    assert helpers.rel_err(host(act), expected_act) <= REL_TOL
    qd = et.QWeight(rt, codec, [dev(pd)], [d], ffn)
    out = empty((vectors, d))
    unit_act = (expected_act / np.abs(expected_act).max()).astype(np.float32)  # random code bytes make huge activations: keep f16 range
    qd.linear_into(dev(unit_act), vectors, out, residual=dev(residual), epilogue=et.EPILOGUE_RESIDUAL)
    expected = residual + orc.qlinear(codec, unit_act, pd, d, ffn, threads=4)
    assert helpers.rel_err(host(out), expected) <= REL_TOL


def test_tiled_weight_rejects_unsupported_geometry():
    rt = runtime()
    raw = empty((16, 18 * 3), dtype=torch.uint8)
    with pytest.raises(et.BackendError, match="multiple of 64"):
        et.QWeight(rt, gv.Q4_0, [raw], [16], 96)
    with pytest.raises(et.BackendError, match="Q4_0, Q8_0, Q3_K, Q4_K, Q5_K and Q6_K"):
        et.QWeight(rt, gv.Q2_K, [empty((16, 84), dtype=torch.uint8)], [16], 256)
    with pytest.raises(et.BackendError, match="multiple of 256"):
        et.QWeight(rt, gv.Q4_K, [raw], [16], 128)


@pytest.mark.parametrize("codec", [gv.Q4_0, gv.Q8_0])
@pytest.mark.parametrize("rows,columns,vectors", [(70, 64, 1), (130, 192, 16), (200, 704, 8), (4096, 1088, 9), (38100, 320, 3)])
def test_few_vectors_lose_no_weight_precision(codec, rows, columns, vectors):
    """Stages that K fills by half, one stage, odd stage counts, one CTA and a whole cluster per row tile: on inputs that f16
    holds exactly, the sums are those of exact weights."""
    rng = np.random.default_rng(rows + columns)
    packed = random_packed(codec, rows, columns, seed=rows)
    x = rng.normal(size=(vectors, columns)).astype(np.float16).astype(np.float32)
    qw = et.QWeight(runtime(), codec, [dev(packed)], [rows], columns)
    out = empty((vectors, rows))
    qw.linear_into(dev(x), vectors, out)
    expected = orc.qlinear(codec, x, packed, rows, columns, threads=8)
    assert helpers.rel_err(host(out), expected) <= 1e-5
