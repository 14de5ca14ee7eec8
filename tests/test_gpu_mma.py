"""Small convs, Gemms and products on the warp-level matrix instructions: bit-exact against the plain-C oracle at the edges of
fragments, splits and chunks, for every alignment, epilogue and stride."""
import ctypes as C

import numpy as np
import pytest

import cases
import gpu_util
from espdl_b200 import abi

pytestmark = pytest.mark.gpu

P0 = dict(kh=1, kw=1, pad=(0, 0, 0, 0))
SHAPES = [
    dict(n=1, h=7, w=7, cin=160, cout=96, **P0),
    dict(n=1, h=1, w=1, cin=16, cout=8, **P0),
    dict(n=1, h=1, w=17, cin=1040, cout=9, **P0),
    dict(n=3, h=5, w=7, cin=28, cout=33, **P0),
    dict(n=1, h=10, w=10, cin=64, cout=64),
    dict(n=2, h=9, w=11, cin=16, cout=40, stride=2),
    dict(n=1, h=13, w=8, cin=12, cout=20, kh=5, kw=3, dil=2, pad=(4, 4, 2, 2)),
    dict(n=1, h=6, w=6, cin=128, cout=257, stride=2),
    dict(n=27, h=6, w=5, cin=32, cout=24, **P0),
    dict(n=1, h=40, w=40, cin=24, cout=24, **P0),
    dict(n=2, h=23, w=31, cin=3, cout=16, kh=7, kw=7, stride=2),       # ragged runs: 21 bytes a filter row
    dict(n=1, h=9, w=3, cin=1, cout=12, kh=3, kw=5, pad=(1, 1, 2, 2)),  # a window wider than the image
    dict(n=3, h=8, w=8, cin=5, cout=9, kh=5, kw=5, stride=(2, 1), dil=(2, 1), pad=(4, 4, 2, 2)),
    dict(n=1, h=1, w=50, cin=101, cout=40, **P0),
    dict(n=2, h=16, w=20, cin=3, cout=33, stride=2, pad=(0, 1, 0, 1)),
]


@pytest.fixture
def forced(monkeypatch):
    monkeypatch.setenv("ESPDL_B200_SMALL_MMA", "always")


@pytest.mark.parametrize("round_mode", [abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN])
@pytest.mark.parametrize("lut", [False, True, "channels"])
@pytest.mark.parametrize("i", range(len(SHAPES)))
def test_conv(i, lut, round_mode, forced):
    case = cases.conv_case(seed=i, per_channel=True, lut=lut, round_mode=round_mode, act=abi.ACT_LINEAR if lut else abi.ACT_RELU, **SHAPES[i])
    want = gpu_util.run_conv_oracle(case)
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)
    assert want.std() > 0


@pytest.mark.parametrize("in_stride,out_stride", [(0, 0), (64, 96), (52, 47)])
@pytest.mark.parametrize("e_w", [(-9, -6), (-1, 3), (-40, -25)])
def test_strides_residual_and_any_shift(in_stride, out_stride, e_w, forced):
    case = cases.conv_case(seed=3, n=2, h=6, w=9, cin=48, cout=45, per_channel=True, e_in=0, e_out=0, e_w=e_w, in_stride=in_stride, out_stride=out_stride, **P0)
    case["res"] = np.random.default_rng(3).integers(-128, 128, size=case["out"].shape, dtype=np.int8)
    case["residual_pixel_stride"] = case["out"].shape[-1]
    case["out"][...] = 0x55
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), gpu_util.run_conv_oracle(case))


@pytest.mark.parametrize("k,n", [(100, 100), (32, 17), (16, 3), (256, 64)])
def test_batch_of_products(k, n, forced):
    rng = np.random.default_rng(k)
    images, rows = 5, 21
    x = rng.integers(-100, 100, size=(images, 1, rows, k), dtype=np.int8)
    w = rng.integers(-100, 100, size=(images, n, 1, 1, k), dtype=np.int8)
    whole = cases.conv_case(seed=1, n=images, h=1, w=rows, cin=k, cout=n, bias=False, **P0)
    whole.update(x=x, w=w, filter_image_stride=n * k)
    got = gpu_util.run_conv_gpu(whole)
    for i in range(images):
        one = cases.conv_case(seed=1, n=1, h=1, w=rows, cin=k, cout=n, bias=False, **P0)
        one.update(x=x[i:i + 1], w=w[i], filter_exponent=whole["filter_exponent"])
        np.testing.assert_array_equal(got[i:i + 1], gpu_util.run_conv_oracle(one))


# short windows with few output channels on the CUDA cores: chunks of 16, 8 and 4 bytes, ragged channels, slices, every border
@pytest.mark.parametrize("act,lut,round_mode", [(abi.ACT_RELU, False, abi.ROUND_HALF_UP), (abi.ACT_LINEAR, True, abi.ROUND_HALF_EVEN)])
@pytest.mark.parametrize("kw", [dict(n=2, h=31, w=29, cin=16, cout=1, kh=2, kw=2, pad=(1, 1, 1, 1)), dict(n=1, h=40, w=17, cin=8, cout=16, kh=2, kw=2, pad=(0, 1, 0, 1)),
                                dict(n=1, h=9, w=9, cin=4, cout=30, kh=5, kw=5, stride=2), dict(n=3, h=7, w=20, cin=48, cout=6, kh=1, kw=3, in_stride=64, out_stride=12),
                                dict(n=1, h=12, w=12, cin=12, cout=32, kh=3, kw=4, dil=2, pad=(2, 2, 3, 3)), dict(n=70, h=60, w=50, cin=16, cout=3, kh=2, kw=2, pad=(1, 0, 1, 0))])
def test_narrow_windows(kw, act, lut, round_mode, monkeypatch):
    monkeypatch.setenv("ESPDL_B200_NARROW", "always")
    case = cases.conv_case(seed=kw["cin"] + kw["h"], per_channel=True, act=act, lut=lut, round_mode=round_mode, e_in=-7, e_out=-6, e_w=(-9, -7), **kw)
    want = gpu_util.run_conv_oracle(case)
    assert want.std() > 0
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)


@pytest.mark.parametrize("act", [abi.ACT_RELU, abi.ACT_LINEAR])
@pytest.mark.parametrize("sign", [1, -1])
def test_reductions_beyond_65536_terms(sign, act, forced):
    """73500 terms at the ends of int8 reach 1.2e9; with this bias the sum is 101 below (above) the end of int32, and only the rounding's
    half takes it across."""
    case = cases.conv_case(seed=1, n=1, h=8, w=8, cin=1500, cout=9, kh=7, kw=7, pad=(0, 0, 0, 0), per_channel=True, act=act, e_in=0, e_out=0, e_w=(-15, -15))
    case["x"][...], case["w"][...] = -128, -128 if sign > 0 else 127
    acc = 7 * 7 * 1500 * 128 * (128 if sign > 0 else -127)
    case["b"][...] = sign * (2 ** 31 - 101) - acc
    case["b"][1::3] = 5  # others take the one-add form
    want = gpu_util.run_conv_oracle(case)
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)
    assert want.max() == (127 if sign > 0 else 0 if act == abi.ACT_RELU else -128)


# int16 on byte planes: ragged reductions (runs of 64), pixels and channels around the tiles' edges, windows that leave the image on every side
SHAPES16 = [
    dict(n=4, h=40, w=40, cin=64, cout=64),
    dict(n=1, h=1, w=1, cin=8, cout=1, **P0),
    dict(n=1, h=1, w=65, cin=72, cout=33, **P0),
    dict(n=3, h=9, w=7, cin=24, cout=31, stride=2),
    dict(n=1, h=13, w=8, cin=16, cout=66, kh=5, kw=3, dil=2, pad=(4, 4, 2, 2)),
    dict(n=2, h=6, w=9, cin=40, cout=45, in_stride=56, out_stride=47),
    dict(n=1, h=1, w=33, cin=16384, cout=32, **P0),
    dict(n=40, h=20, w=20, cin=64, cout=64, **P0),
]


@pytest.mark.parametrize("act,round_mode", [(abi.ACT_RELU, abi.ROUND_HALF_UP), (abi.ACT_LINEAR, abi.ROUND_HALF_EVEN)])
@pytest.mark.parametrize("i", range(len(SHAPES16)))
def test_conv_int16(i, act, round_mode, monkeypatch):
    monkeypatch.setenv("ESPDL_B200_MMA16", "always")
    case = cases.conv_case(seed=20 + i, dtype=abi.DTYPE_INT16, per_channel=True, act=act, round_mode=round_mode, e_in=-13, e_out=-5, e_w=(-14, -11), **SHAPES16[i])
    want = gpu_util.run_conv_oracle(case)
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)
    assert want.size < 8 or want.std() > 0


# Runs of 64 elements of the reduction: all asked for at the start (up to five), whole and partial groups of three, the tiles of 64 x 64, 64 x 32 and 32 x 32
@pytest.mark.parametrize("k", [8, 64, 72, 320, 328, 384, 392, 512, 576, 640, 832])
@pytest.mark.parametrize("m,n", [(65, 40), (6400, 64), (40000, 72)])
def test_int16_runs_of_the_reduction(m, n, k, monkeypatch):
    monkeypatch.setenv("ESPDL_B200_MMA16", "always")
    case = cases.gemm_case(seed=m + k, dtype=abi.DTYPE_INT16, m=m, k=k, n_out=n, per_channel=True, e_in=-13, e_out=-6, e_w=(-14, -11))
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), gpu_util.run_conv_oracle(case))


@pytest.mark.parametrize("e_w", [(-60, -30), (-1, 3), (20, 40)])
def test_conv_int16_ends_of_the_range_and_any_shift(e_w, monkeypatch):
    """Every element at an end of the type, so that each plane's sum is as large as it gets; shifts from far left to beyond the sum."""
    monkeypatch.setenv("ESPDL_B200_MMA16", "always")
    case = cases.conv_case(seed=5, dtype=abi.DTYPE_INT16, n=1, h=4, w=9, cin=16384, cout=34, per_channel=True, e_in=0, e_out=0, e_w=e_w, act=abi.ACT_LINEAR, **P0)
    rng = np.random.default_rng(5)
    case["x"][...] = np.where(rng.random((1, 4, 9, 1)) < 0.5, -32768, 32767)
    case["w"][...] = np.where(rng.random((34, 1, 1, 1)) < 0.5, -32768, 32767)
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), gpu_util.run_conv_oracle(case))


def test_int16_product_in_place(monkeypatch):
    """Results that overwrite the inputs: the kernel that has copied its operands first, also where the other one is asked for.  Channels beside the inputs in the
    same rows are no such case."""
    monkeypatch.setenv("ESPDL_B200_MMA16", "always")
    for cin, cout, stride, ahead in ((64, 64, 0, 0), (256, 256, 0, 0), (64, 32, 96, 64)):
        case = cases.conv_case(seed=cin, dtype=abi.DTYPE_INT16, n=1, h=1, w=200, cin=cin, cout=cout, per_channel=True, e_in=-13, e_out=-5, e_w=(-14, -11),
                               in_stride=stride, out_stride=stride, **P0)
        want = gpu_util.run_conv_oracle(case)
        with gpu_util.DeviceBuffers() as dev:
            x = dev.upload(case["x"])
            ptrs = dict(input=x, output=x + 2 * ahead, filter=dev.upload(case["w"]), bias=dev.upload(case["b"]), filter_exponents=dev.upload(case["ew"]))
            abi.check(dev.lib.espdl_b200_conv2d(C.byref(cases.conv_desc(case, ptrs)), None), "conv2d")
            rows = dev.download(x, case["x"])
        np.testing.assert_array_equal(rows[..., ahead:ahead + cout], want[..., :cout])


@pytest.mark.parametrize("knob", ["always", "0"])
def test_int16_product_refuses_scratch_it_cannot_use(knob, monkeypatch):
    """Whichever kernel runs a product: scratch that is missing, short or not aligned to 16 bytes is an error."""
    monkeypatch.setenv("ESPDL_B200_MMA16", knob)
    case = cases.conv_case(seed=1, dtype=abi.DTYPE_INT16, n=1, h=1, w=100, cin=64, cout=48, per_channel=True, e_in=-13, e_out=-5, e_w=(-14, -11), **P0)
    with gpu_util.DeviceBuffers() as dev:
        out = dev.upload(case["out"])
        ptrs = dict(input=dev.upload(case["x"]), output=out, filter=dev.upload(case["w"]), bias=dev.upload(case["b"]), filter_exponents=dev.upload(case["ew"]))
        d, need = cases.conv_desc(case, ptrs), C.c_size_t(0)
        abi.check(dev.lib.espdl_b200_conv2d_workspace_bytes(C.byref(d), C.byref(need)), "workspace")
        scratch = dev.alloc(need.value + 16)
        assert need.value > 0
        for at, size in ((None, need.value), (scratch, need.value - 1), (scratch + 8, need.value)):
            assert dev.lib.espdl_b200_conv2d_ws(C.byref(d), at, size, None) == abi.ERR_INVALID_ARG
        abi.check(dev.lib.espdl_b200_conv2d_ws(C.byref(d), scratch, need.value, None), "conv2d_ws")
        want = gpu_util.run_conv_oracle(case)
        np.testing.assert_array_equal(dev.download(out, want), want)
