"""Half-to-even rounding in the fast epilogue form of every int8 conv kernel, and the reduction over pixels: bit-exact
against the plain-C oracle at the sizes where tiles end and where ties are common."""
import ctypes as C

import numpy as np
import pytest

import cases
import checkers
import gpu_util
from espdl_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_small_layers(monkeypatch, request):
    monkeypatch.setenv("ESPDL_B200_SMALL_MMA", "0")  # the kernels meant here, whatever the size
    if "dw-tma" in request.node.name:
        monkeypatch.setenv("ESPDL_B200_DW_TMA_NARROW", "1")
    if "dw-mma" in request.node.name:
        monkeypatch.setenv("ESPDL_B200_DW_MMA", "always")

# one shape per kernel: the tile kernel (staged, unaligned rows, residual), filter windows (one box per tap, one patch per
# tile stacked / unstaged), banded 8 / 16 channels, first layer, depthwise through the TMA unit, on the matrix instruction and from global memory
SHAPES = {
    "tile": dict(n=2, h=9, w=13, cin=64, cout=96, kh=1, kw=1, pad=(0, 0, 0, 0)),
    "tile-wide": dict(n=1, h=1, w=130, cin=512, cout=256, kh=1, kw=1, pad=(0, 0, 0, 0)),
    "tile-ragged": dict(n=1, h=1, w=77, cin=48, cout=17, kh=1, kw=1, pad=(0, 0, 0, 0)),
    "tile-residual": dict(n=1, h=1, w=200, cin=96, cout=32, kh=1, kw=1, pad=(0, 0, 0, 0)),
    "taps": dict(n=2, h=15, w=15, cin=48, cout=48, stride=2),
    "patch": dict(n=2, h=11, w=33, cin=64, cout=64),
    "patch-unstaged": dict(n=1, h=9, w=31, cin=128, cout=128),
    "band8": dict(n=2, h=12, w=24, cin=8, cout=16),
    "band16": dict(n=3, h=16, w=32, cin=16, cout=32, stride=2),
    "first": dict(n=2, h=32, w=48, cin=3, cout=16, stride=2),
    "dw-tma": dict(n=2, h=14, w=15, cin=96, depthwise=True),
    "dw-tma-s2": dict(n=2, h=15, w=14, cin=64, stride=2, depthwise=True),
    "dw-mma": dict(n=2, h=14, w=15, cin=96, depthwise=True),
    "dw-mma-slices": dict(n=3, h=9, w=7, cin=32, depthwise=True, in_stride=48, out_stride=64),
    "dw-narrow": dict(n=2, h=9, w=17, cin=24, depthwise=True),
    "dw-narrow-s2": dict(n=2, h=10, w=17, cin=32, stride=2, depthwise=True),
}


@pytest.mark.parametrize("act", [abi.ACT_LINEAR, abi.ACT_RELU])
@pytest.mark.parametrize("shift", [(1, 3), (7, 9), (20, 24)])
@pytest.mark.parametrize("name", list(SHAPES))
def test_half_even_fast_form(name, shift, act):
    e_w = (-shift[1], -shift[0])  # with e_in = e_out = 0 the shift of a channel is minus its filter exponent
    for lut in (False, True) if "dw" not in name and "residual" not in name else (False,):
        case = cases.conv_case(seed=len(name) + shift[0], per_channel=True, round_mode=abi.ROUND_HALF_EVEN, act=act, e_in=0, e_out=0, e_w=e_w, lut=lut,
                               bias_mag=1 << (shift[1] + 4), **SHAPES[name])
        if shift[1] <= 3:  # small sums: neither all saturated nor all zero, every second one a tie at shift 1
            case["x"] = np.clip(case["x"], -2, 2)
            case["w"] = np.clip(case["w"], -1, 1)
        if "residual" in name:
            case["res"] = np.random.default_rng(3).integers(-128, 128, size=case["out"].shape, dtype=np.int8)
        want = gpu_util.run_conv_oracle(case)
        np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)
        assert want.std() > 0


@pytest.mark.parametrize("round_mode", [abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN])
@pytest.mark.parametrize("name", list(SHAPES))
def test_shifts_and_biases_of_dead_channels(name, round_mode):
    """Channels whose weights were all but zero when the model was quantised carry shifts up to 39 and biases at the ends of int32."""
    case = cases.conv_case(seed=len(name), per_channel=True, round_mode=round_mode, act=abi.ACT_LINEAR, e_in=0, e_out=0, e_w=(-12, -7), **SHAPES[name])
    rng = np.random.default_rng(5)
    edge = [2 ** 31 - 1, -2 ** 31, 2 ** 30, -2 ** 30, 2 ** 29 + 7, -2 ** 29 - 7, 2 ** 31 - 2 ** 28, -2 ** 31 + 2 ** 28]
    for c in range(0, case["out_c"], 3):
        case["ew"][c] = -int(rng.integers(25, 41))
        # above 31 any bias gives 0; up to 31 the largest that leave the 32-bit sum in range
        case["b"][c] = edge[int(rng.integers(0, 8))] if case["ew"][c] < -31 else edge[int(rng.integers(4, 8))] // (1 if case["ew"][c] > -29 else 4)
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), gpu_util.run_conv_oracle(case))


# kernel -> (layer, switches, kernel asked for): the kernels that requantise channel by channel, and those that do so for channels outside
# the one-add form
GENERAL = {
    "mma": (dict(n=2, h=6, w=9, cin=48, cout=45, kh=1, kw=1, pad=(0, 0, 0, 0)), {"ESPDL_B200_SMALL_MMA": "always"}, abi.KERNEL_AUTO),
    "narrow": (dict(n=2, h=15, w=14, cin=16, cout=13, kh=2, kw=2, pad=(0, 1, 0, 1)), {"ESPDL_B200_NARROW": "always"}, abi.KERNEL_AUTO),
    "dw3": (dict(n=1, h=9, w=11, cin=20, depthwise=True), {}, abi.KERNEL_AUTO),
    "dw3-tma": (dict(n=2, h=14, w=15, cin=96, depthwise=True), {"ESPDL_B200_DW_TMA_NARROW": "1"}, abi.KERNEL_AUTO),
    "dw3-mma": (dict(n=2, h=14, w=15, cin=96, depthwise=True), {"ESPDL_B200_DW_MMA": "always"}, abi.KERNEL_AUTO),
    "dw3-mma-slices": (dict(n=3, h=9, w=7, cin=32, depthwise=True, in_stride=48, out_stride=64), {"ESPDL_B200_DW_MMA": "always"}, abi.KERNEL_AUTO),
    "dw5": (dict(n=1, h=9, w=11, cin=20, kh=5, kw=5, pad=(2, 2, 2, 2), depthwise=True), {}, abi.KERNEL_AUTO),
    "dw7": (dict(n=1, h=9, w=11, cin=24, kh=7, kw=7, pad=(3, 3, 3, 3), depthwise=True), {}, abi.KERNEL_AUTO),
    "dw-vec": (dict(n=1, h=9, w=11, cin=32, kh=3, kw=5, pad=(1, 1, 2, 2), depthwise=True), {}, abi.KERNEL_AUTO),
    "dw-any": (dict(n=1, h=9, w=11, cin=21, kh=3, kw=5, pad=(1, 1, 2, 2), depthwise=True), {}, abi.KERNEL_AUTO),
    "cores": (dict(n=1, h=7, w=9, cin=20, cout=18), {}, abi.KERNEL_SIMT),
    "cores-first": (dict(n=1, h=7, w=9, cin=3, cout=18), {}, abi.KERNEL_SIMT),
    "tile": (dict(n=1, h=1, w=130, cin=64, cout=48, kh=1, kw=1, pad=(0, 0, 0, 0)), {}, abi.KERNEL_TCGEN05),
    "patch": (dict(n=2, h=11, w=33, cin=64, cout=64), {}, abi.KERNEL_TCGEN05),
    "band": (dict(n=2, h=12, w=24, cin=8, cout=16), {}, abi.KERNEL_AUTO),
    "first": (dict(n=2, h=32, w=48, cin=3, cout=16, stride=2), {}, abi.KERNEL_AUTO),
}


@pytest.mark.parametrize("round_mode", [abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN])
@pytest.mark.parametrize("name", list(GENERAL))
def test_dead_channels_beside_channels_outside_the_fast_form(name, round_mode, monkeypatch):
    """A shift beyond 31 gives 0 for every 32-bit sum, also in the form that a neighbour with a left shift or a huge bias brings about."""
    kw, switches, kernel = GENERAL[name]
    for k, v in switches.items():
        monkeypatch.setenv(k, v)
    case = cases.conv_case(seed=len(name), per_channel=True, round_mode=round_mode, act=abi.ACT_LINEAR, e_in=0, e_out=0, e_w=(-12, -7), **kw)
    rng = np.random.default_rng(7)
    for c in range(0, case["out_c"], 4):
        case["ew"][c], case["b"][c] = -int(rng.integers(31, 41)), [2 ** 31 - 1, -2 ** 31, 2 ** 30 + 3, -2 ** 30 - 3][c // 4 % 4]
        if c + 2 < case["out_c"]:
            case["ew"][c + 2] = int(rng.integers(0, 3))  # a left shift: outside the one-add form
    for c in range(0, case["out_c"], 4):
        if case["ew"][c] == -31:  # within the reach of the sum
            case["b"][c] //= 2
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case, kernel=kernel), gpu_util.run_conv_oracle(case))


# pixels and channels around what a thread block covers at once, images shared by one, two and eight blocks
@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
@pytest.mark.parametrize("n,h,w,c", [(1, 184, 184, 32), (3, 23, 23, 48), (2, 33, 31, 6), (1, 3, 700, 1), (300, 7, 7, 1280), (2, 16, 16, 520), (1, 2048, 1, 3)])
def test_pool_and_reduce_over_all_pixels(n, h, w, c, dtype):
    t = np.int8 if dtype == abi.DTYPE_INT8 else np.int16
    case = cases.pool_case(abi.POOL_GLOBAL_AVG, seed=n + h, dtype=dtype, n=n, h=h, w=w, c=c, e_in=-4, e_out=-6)
    case["x"] = case["x"] // 2 + t(9)  # a mean away from zero
    want = case["out"].copy()
    assert checkers.oracle().oracle_pool(cases.pool_desc(dict(case, out=want))) == 0
    with gpu_util.DeviceBuffers() as dev:
        x, out = dev.upload(case["x"]), dev.upload(case["out"])
        d = cases.pool_desc(case, dict(input=x, output=out))
        abi.check(dev.lib.espdl_b200_pool(C.byref(d), None), "pool")
        np.testing.assert_array_equal(dev.download(out, want), want)
        for op in (abi.REDUCE_MEAN, abi.REDUCE_SUM, abi.REDUCE_MAX, abi.REDUCE_MIN, abi.REDUCE_L1, abi.REDUCE_SUM_SQUARE, abi.REDUCE_L2):
            r = abi.ReduceDesc()
            r.op, r.dtype, r.ndim, r.in_exponent, r.out_exponent, r.round_mode = op, dtype, 4, -4, (-5 if op == abi.REDUCE_MEAN else 4), abi.ROUND_HALF_EVEN
            for i, v in enumerate((n, h, w, c)):
                r.shape[i], r.reduce[i] = v, int(i in (1, 2))
            want_r = np.zeros((n, 1, 1, c), dtype=t)
            r.input, r.output = case["x"].ctypes.data, want_r.ctypes.data
            assert checkers.oracle().oracle_reduce(C.byref(r)) == 0
            r.input, r.output = x, out
            abi.check(dev.lib.espdl_b200_reduce(C.byref(r), None), "reduce")
            np.testing.assert_array_equal(dev.download(out, want_r), want_r)
