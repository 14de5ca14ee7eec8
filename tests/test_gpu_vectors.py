"""Vectorised forms of the memory-bound operators at the ends of their units: elementwise operators on int16 and on lengths that fill
no 16-byte unit, gates that repeat over the rows of an image, softmax rows of any length, the column walk of max pools on int16
and on ragged channels.  Bit-exact against the plain-C oracle."""
import ctypes as C

import numpy as np
import pytest

import cases
import checkers
import gpu_util
import test_gpu_ops
from espdl_b200 import abi

pytestmark = pytest.mark.gpu

BOTH = [abi.DTYPE_INT8, abi.DTYPE_INT16]
OPS = [abi.ELT_ADD, abi.ELT_SUB, abi.ELT_MUL, abi.ELT_MAX, abi.ELT_MIN, abi.ELT_DIV, abi.ELT_REQUANTIZE, abi.ELT_CLIP, abi.ELT_RELU, abi.ELT_LUT]


def check(case):
    got, want = test_gpu_ops.run_eltwise(case)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("shape", [(1,), (15,), (17,), (3, 5, 7, 11), (2, 9, 8, 24), (70001,)])
def test_lengths_that_fill_no_unit(shape, op, dtype):
    for round_mode in (abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN):
        check(cases.eltwise_case(op, seed=len(shape), dtype=dtype, out_shape=shape, round_mode=round_mode))


@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("op", [abi.ELT_ADD, abi.ELT_SUB, abi.ELT_MUL, abi.ELT_MAX, abi.ELT_MIN])
@pytest.mark.parametrize("shape,gate", [((3, 5, 7, 16), (3, 1, 1, 16)), ((2, 9, 4, 48), (1, 1, 1, 48)), ((1, 6, 6, 8), (1, 1, 1, 8)), ((4, 3, 3, 80), (4, 1, 1, 80)),
                                        ((3, 5, 7, 12), (3, 1, 1, 12)), ((2, 1, 9, 32), (1, 1, 1, 1)), ((3, 35, 24), (3, 1, 24)), ((2, 3, 5, 16), (2, 3, 1, 16)),
                                        ((5, 33, 20), (1, 1, 20)), ((2, 3, 5, 4), (1, 3, 1, 4))])
def test_gates(shape, gate, op, dtype):
    check(cases.eltwise_case(op, seed=shape[-1], dtype=dtype, out_shape=shape, in1_shape=gate))


# exponent -1 is the largest whose table stays finite (exp(63.5) < 3.4e38 < exp(127)): beyond it a row is inf / inf, and what the
# reference's float -> int conversion of that NaN gives is undefined
@pytest.mark.parametrize("round_mode", [abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN])
@pytest.mark.parametrize("e_in,rows,length", [(-4, 300, 17), (-3, 64, 1), (-6, 1000, 127), (-2, 257, 130), (-4, 77, 316), (-7, 4000, 64), (-1, 128, 33), (-3, 1, 5), (-4, 7, 100), (-4, 3, 1200)])
def test_softmax_codes(e_in, rows, length, round_mode):
    rng = np.random.default_rng(length)
    x = rng.integers(-128, 128, size=(rows, length), dtype=np.int8)
    x[: rows // 4] = np.clip(x[: rows // 4] // 8, -16, 15)  # flat rows: many codes near a rounding boundary
    table = np.exp(np.float32(2.0 ** e_in) * np.arange(-128, 128, dtype=np.float32)).astype(np.float32)
    want, got = np.zeros_like(x), np.zeros_like(x)
    d = abi.SoftmaxDesc()
    d.rows, d.len, d.out_dtype, d.out_exponent, d.in_exponent, d.round_mode = rows, length, abi.DTYPE_INT8, -7, e_in, round_mode
    d.input, d.output, d.exp_table = x.ctypes.data, want.ctypes.data, table.ctypes.data
    assert checkers.oracle().oracle_softmax(C.byref(d)) == 0
    with gpu_util.DeviceBuffers() as dev:
        out = dev.upload(got)
        d.input, d.output, d.exp_table = dev.upload(x), out, dev.upload(table)
        abi.check(dev.lib.espdl_b200_softmax(C.byref(d), None), "softmax")
        np.testing.assert_array_equal(dev.download(out, want), want)


@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("kw", [dict(n=2, h=21, w=9, c=24, kh=5, kw=5, pad=(2, 2, 2, 2)), dict(n=1, h=7, w=7, c=127, kh=5, kw=5, pad=(2, 2, 2, 2)),
                                dict(n=3, h=40, w=3, c=1, kh=3, kw=3, pad=(1, 1, 1, 1)), dict(n=1, h=64, w=64, c=17, kh=5, kw=5, pad=(2, 2, 2, 2)),
                                dict(n=2, h=5, w=6, c=8, kh=5, kw=5, pad=(0, 0, 1, 3)), dict(n=1, h=3, w=2, c=3, kh=3, kw=3, pad=(1, 1, 1, 1))])
def test_max_pool_walk(kw, dtype):
    pool_matches(cases.pool_case(abi.POOL_MAX, seed=kw["c"], dtype=dtype, stride=1, **kw))


# two and four elements a thread, segments of a column, pads wider than the window needs on one side
@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("kw", [dict(n=2, h=23, w=9, c=18, kh=5, kw=5, pad=(2, 2, 2, 2)), dict(n=1, h=64, w=7, c=20, kh=3, kw=3, pad=(1, 1, 1, 1)),
                                dict(n=3, h=6, w=5, c=2, kh=5, kw=5, pad=(4, 0, 1, 3)), dict(n=2, h=41, w=6, c=44, kh=5, kw=5, pad=(0, 0, 0, 0)),
                                dict(n=1, h=3, w=2, c=4, kh=3, kw=3, pad=(1, 1, 1, 1)), dict(n=60, h=40, w=40, c=6, kh=3, kw=3, pad=(2, 1, 0, 2)),
                                dict(n=31, h=41, w=40, c=28, kh=5, kw=5, pad=(2, 2, 2, 2)), dict(n=24, h=33, w=41, c=44, kh=3, kw=3, pad=(0, 2, 2, 0))])
def test_max_pool_walk_words(kw, dtype):
    pool_matches(cases.pool_case(abi.POOL_MAX, seed=kw["c"], dtype=dtype, stride=1, **kw))


def pool_matches(case):
    want = case["out"].copy()
    assert checkers.oracle().oracle_pool(cases.pool_desc(dict(case, out=want))) == 0
    with gpu_util.DeviceBuffers() as dev:
        ptrs = dict(input=dev.upload(case["x"]), output=dev.upload(case["out"]))
        abi.check(dev.lib.espdl_b200_pool(C.byref(cases.pool_desc(case, ptrs)), None), "pool")
        np.testing.assert_array_equal(dev.download(ptrs["output"], want), want)


# maps that go through shared memory: one band and several, windows past every edge, strides, pads of one side
@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("kw", [dict(n=1, h=10, w=10, c=32, kh=5, kw=5, pad=(2, 2, 2, 2), stride=1), dict(n=3, h=23, w=7, c=16, kh=3, kw=5, pad=(1, 1, 2, 2), stride=2),
                                dict(n=1, h=64, w=33, c=16, kh=2, kw=2, pad=(0, 0, 0, 0), stride=2), dict(n=2, h=5, w=6, c=48, kh=4, kw=3, pad=(3, 0, 0, 2), stride=1),
                                dict(n=1, h=1, w=300, c=16, kh=3, kw=9, pad=(1, 1, 4, 4), stride=3), dict(n=1, h=200, w=180, c=16, kh=9, kw=9, pad=(4, 4, 4, 4), stride=1)])
def test_max_pool_map(kw, dtype):
    pool_matches(cases.pool_case(abi.POOL_MAX, seed=kw["c"], dtype=dtype, **kw))


# one image over the blocks of a wide cluster
@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("shape", [(1, 131, 129, 32), (2, 97, 101, 64)])
def test_large_image_means(shape, dtype):
    n, h, w, c = shape
    case = cases.pool_case(abi.POOL_GLOBAL_AVG, seed=c, dtype=dtype, n=n, h=h, w=w, c=c)
    case["x"] = case["x"] // 4 + np.arange(c, dtype=case["x"].dtype) # channels with means apart
    pool_matches(case)


# windows of K x K taps, four channels a thread: maps smaller than the window, uneven strides and pads, channel slices
@pytest.mark.parametrize("act,lut,round_mode", [(abi.ACT_RELU, False, abi.ROUND_HALF_UP), (abi.ACT_LINEAR, True, abi.ROUND_HALF_EVEN)])
@pytest.mark.parametrize("kw", [dict(n=2, h=23, w=19, cin=64, kh=5, kw=5), dict(n=1, h=3, w=4, cin=20, kh=7, kw=7), dict(n=3, h=12, w=13, cin=36, kh=5, kw=5, stride=2),
                                dict(n=1, h=9, w=30, cin=8, kh=3, kw=3, stride=(2, 1)), dict(n=2, h=10, w=11, cin=16, kh=7, kw=7, stride=3, pad=(3, 0, 0, 2)),
                                dict(n=1, h=8, w=8, cin=12, kh=5, kw=5, in_stride=20, out_stride=24), dict(n=1, h=6, w=6, cin=1600, kh=5, kw=5)])
def test_depthwise_windows(kw, act, lut, round_mode):
    case = cases.conv_case(seed=kw["cin"], depthwise=True, cout=kw["cin"], per_channel=True, act=act, lut=lut, round_mode=round_mode, e_in=-7, e_out=-5, e_w=(-9, -7), **kw)
    want = gpu_util.run_conv_oracle(case)
    assert want.std() > 0
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)


# image means whose pixels take 1, 2, 3, 8, 32 and 40 lanes
@pytest.mark.parametrize("dtype", BOTH)
@pytest.mark.parametrize("shape", [(3, 19, 17, 16), (2, 24, 12, 32), (2, 15, 15, 48), (1, 23, 23, 128), (5, 9, 9, 512), (1, 20, 20, 640), (1, 60, 60, 4)])
def test_image_means(shape, dtype):
    n, h, w, c = shape
    case = cases.pool_case(abi.POOL_GLOBAL_AVG, seed=c, dtype=dtype, n=n, h=h, w=w, c=c)
    case["x"] = case["x"] // 4 + np.arange(c, dtype=case["x"].dtype) % 90
    pool_matches(case)
