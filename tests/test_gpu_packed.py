"""Convs whose operands are packed for the tile kernel (int16 windows, reductions and channel counts that are no multiple of 16),
the int16 product's combined planes, and batches of products on the CUDA cores: bit-exact against the plain-C oracle at the
extremes of the types, around tile and chunk ends."""
import os
import subprocess
import sys

import numpy as np
import pytest

import cases
import gpu_util
from espdl_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def no_small_layers(monkeypatch):
    monkeypatch.setenv("ESPDL_B200_SMALL_MMA", "0")  # the kernels meant here, whatever the size
    monkeypatch.setenv("ESPDL_B200_MMA16", "0")

S16 = dict(dtype=abi.DTYPE_INT16, e_in=-14, e_w=(-15, -14), e_out=-11)
SHAPES = [
    dict(n=2, h=20, w=21, cin=32, cout=48),                        # 3x3
    dict(n=1, h=30, w=30, cin=24, cout=64, stride=2),              # channels no multiple of 16, stride
    dict(n=3, h=17, w=19, cin=20, cout=33, kh=5, kw=5, dil=2, pad=(4, 4, 4, 4)),
    dict(n=1, h=40, w=40, cin=40, cout=56, kh=1, kw=1, pad=(0, 0, 0, 0), in_stride=48, out_stride=72),
    dict(n=2, h=30, w=28, cin=3, cout=40, kh=7, kw=7, stride=2),
    dict(n=1, h=1, w=9, cin=1100, cout=300, kh=1, kw=1, pad=(0, 0, 0, 0)),   # few rows, a long reduction
    dict(n=1, h=1, w=700, cin=127, cout=257, kh=1, kw=1, pad=(0, 0, 0, 0)),
]


@pytest.mark.parametrize("round_mode", [abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN])
@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
@pytest.mark.parametrize("i", range(len(SHAPES)))
def test_packed_conv(i, dtype, round_mode):
    kw = dict(SHAPES[i], seed=i, per_channel=True, round_mode=round_mode)
    if dtype == abi.DTYPE_INT16:
        kw.update(S16, wide=True)
    case = cases.conv_case(**kw)
    want = gpu_util.run_conv_oracle(case)
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)
    assert want.std() > 0


def test_packed_convs_of_a_plan_that_share_scratch():
    """A tile kernel with a resident filter (two row tiles an SM and more) starts beside the packing that writes this filter: inside a model's scope, where other
    filters are read ahead, and with another layer's filter still in the scratch."""
    import ctypes as C
    layers = [cases.conv_case(seed=i, n=1, h=200, w=200, per_channel=True, **kw) for i, kw in enumerate((dict(cin=24, cout=64), dict(cin=40, cout=48), dict(cin=3, cout=64, kh=7, kw=7)))]
    want = [gpu_util.run_conv_oracle(case) for case in layers]
    with gpu_util.DeviceBuffers() as dev:
        descs, scratch_bytes = [], 0
        for case in layers:
            names = dict(input="x", filter="w", bias="b", filter_exponents="ew", output="out")
            descs.append(cases.conv_desc(case, {k: dev.upload(case[v]) for k, v in names.items()}))
            need = C.c_size_t(0)
            abi.check(dev.lib.espdl_b200_conv2d_workspace_bytes(C.byref(descs[-1]), C.byref(need)), "workspace_bytes")
            assert need.value >= 40000 * case["kh"] * case["kw"] * case["in_c"]  # the packed path
            scratch_bytes = max(scratch_bytes, need.value)
        scratch = dev.alloc(scratch_bytes)
        for _ in range(10):
            dev.lib.espdl_b200_model_scope(1)
            try:
                for d in descs:
                    abi.check(dev.lib.espdl_b200_conv2d_ws(C.byref(d), scratch, scratch_bytes, None), "conv2d_ws")
            finally:
                dev.lib.espdl_b200_model_scope(0)
            for d, w in zip(descs, want):
                np.testing.assert_array_equal(dev.download(d.output, w), w)


@pytest.mark.parametrize("m,k,n", [(129, 16, 16), (300, 16384, 8), (128, 4096, 129), (1000, 272, 260)])
@pytest.mark.parametrize("sign", [-1, 1, 0])
def test_int16_products_at_the_ends_of_the_type(m, k, n, sign):
    """All operands at an end of int16 (the largest partial sums there are), and mixed."""
    case = cases.gemm_case(seed=m, m=m, k=k, n_out=n, wide=True, **dict(S16, e_out=-4))
    if sign:
        case["x"][...] = 32767 if sign > 0 else -32768
        case["w"][...] = -32768 if sign > 0 else 32767
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), gpu_util.run_conv_oracle(case))


@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
@pytest.mark.parametrize("k,n", [(100, 100), (99, 17), (16, 3)])
def test_batch_of_products_on_the_cuda_cores(k, n, dtype):
    t = np.int8 if dtype == abi.DTYPE_INT8 else np.int16
    rng = np.random.default_rng(k)
    images, rows = 5, 13
    x = rng.integers(-100, 100, size=(images, 1, rows, k), dtype=t)
    w = rng.integers(-100, 100, size=(images, n, 1, 1, k), dtype=t)
    extra = dict(S16, e_out=-20) if dtype == abi.DTYPE_INT16 else {}
    whole = cases.conv_case(seed=1, n=images, h=1, w=rows, cin=k, cout=n, kh=1, kw=1, pad=(0, 0, 0, 0), bias=False, **extra)
    whole.update(x=x, w=w, filter_image_stride=n * k)
    got = gpu_util.run_conv_gpu(whole, kernel=abi.KERNEL_SIMT)
    for i in range(images):
        one = cases.conv_case(seed=1, n=1, h=1, w=rows, cin=k, cout=n, kh=1, kw=1, pad=(0, 0, 0, 0), bias=False, **extra)
        one.update(x=x[i:i + 1], w=w[i], filter_exponent=whole["filter_exponent"])
        np.testing.assert_array_equal(got[i:i + 1], gpu_util.run_conv_oracle(one))


# staged rows of every alignment: widths around the word, the 16-byte chunk and the tile, rows that start anywhere
@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
@pytest.mark.parametrize("m,k,n,stride,lut", [(130, 64, 15, 0, False), (257, 96, 17, 0, True), (100, 32, 127, 0, False), (300, 160, 129, 131, False), (128, 48, 301, 0, True),
                                              (64, 512, 333, 350, False), (1, 64, 1001, 0, False), (4096, 16, 9, 0, False), (20000, 64, 37, 0, False)])
def test_rows_of_any_alignment(m, k, n, stride, lut, dtype):
    kw = dict(S16, wide=True) if dtype == abi.DTYPE_INT16 else dict(lut=lut)
    for round_mode in (abi.ROUND_HALF_UP, abi.ROUND_HALF_EVEN):
        case = cases.gemm_case(seed=n, m=m, k=k, n_out=n, per_channel=True, round_mode=round_mode, out_stride=stride, **kw)
        case["out"][...] = 0x55
        want = gpu_util.run_conv_oracle(case)
        np.testing.assert_array_equal(gpu_util.run_conv_gpu(case), want)


@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
@pytest.mark.parametrize("kw", [dict(n=1, h=1, w=1, cin=40, cout=7, kh=1, kw=1, pad=(0, 0, 0, 0)), dict(n=3, h=5, w=4, cin=7, cout=5), dict(n=1, h=9, w=9, cin=8, cout=8, kh=5, kw=5),
                                dict(n=1, h=1, w=1, cin=1000, cout=3, kh=1, kw=1, pad=(0, 0, 0, 0)), dict(n=2, h=13, w=11, cin=12, cout=9, stride=2, dil=2)])
def test_reductions_shared_by_lanes(kw, dtype):
    extra = dict(S16, wide=True) if dtype == abi.DTYPE_INT16 else {}
    case = cases.conv_case(seed=4, per_channel=True, act=abi.ACT_LINEAR, **dict(extra, **kw))
    np.testing.assert_array_equal(gpu_util.run_conv_gpu(case, kernel=abi.KERNEL_SIMT), gpu_util.run_conv_oracle(case))


@pytest.mark.parametrize("sa,sb", [((3, 2, 5, 16), (1, 2, 16, 7)), ((4, 3, 9, 12), (4, 1, 12, 20)), ((2, 3, 6, 32), (1, 3, 32, 32))])
def test_matmul_whose_second_operand_repeats_over_some_slices(sa, sb, tmp_path):
    import checkers
    import graph_oracle
    from espdl_b200 import espdl_file, model
    rng = np.random.default_rng(5)
    w = rng.integers(-60, 60, size=sb, dtype=np.int8)
    g = espdl_file.GraphBuilder("matmul_spread", metadata={"target": "c"})
    g.add_input("a", np.int8, list(sa), -5)
    g.add_initializer("w", w, [-6])
    g.add_node("MatMul", "mm", ["a", "w"], ["y"], quant_type="S8", activation="Linear")
    so = [max(x, y) for x, y in zip(sa[:2], sb[:2])] + [sa[2], sb[3]]
    g.add_output("y", np.int8, so, -3)
    path = str(tmp_path / "m.espdl")
    g.save(path)
    m = model.Model(path)
    a = rng.integers(-60, 60, size=sa, dtype=np.int8)
    m.inputs[0].array[...] = a
    m.run()
    want = graph_oracle.matmul(checkers.oracle(), a, w, -5, -6, -3, abi.DTYPE_INT8, abi.ACT_LINEAR, abi.ROUND_HALF_UP)
    np.testing.assert_array_equal(np.asarray(m.outputs[0].array).reshape(so), want.reshape(so))
    m.close()


@pytest.mark.parametrize("dt", [abi.DTYPE_INT8, abi.DTYPE_INT16])
@pytest.mark.parametrize("rows,n", [(300, 768), (259, 33), (1000, 1), (257, 1022), (600, 100), (5000, 17), (256, 2050)])
def test_layer_norm_rows_side_by_side(rows, n, dt):
    import ctypes as C
    import checkers
    import test_norm
    for stats, round_mode in ((True, abi.ROUND_HALF_UP), (False, abi.ROUND_HALF_EVEN)):
        a = test_norm.make(abi.NORM_LAYER, dt, rows, n, seed=n, stats=stats, round_mode=round_mode)
        want = test_norm.fresh(a)
        assert checkers.oracle().oracle_norm(C.byref(test_norm.desc(want))) == 0
        with gpu_util.DeviceBuffers() as dev:
            ptrs = {k: dev.upload(a[k]) for k in ("x", "y", "scale", "bias", "mean", "inv") if a[k] is not None}
            abi.check(dev.lib.espdl_b200_norm(C.byref(test_norm.desc(a, ptrs)), None), "norm")
            for k in ("y", "mean", "inv"):
                if a[k] is not None:
                    np.testing.assert_array_equal(dev.download(ptrs[k], want[k]), want[k], err_msg=k)


def products_model(tmp_path, pairs, rng):
    """A model of parallel MatMuls by constants (test_recorded_plans.matmul_graph) run twice on fresh inputs, against the oracle."""
    import checkers
    import graph_oracle
    import test_recorded_plans
    from espdl_b200 import model
    g = test_recorded_plans.matmul_graph(pairs)
    path = str(tmp_path / "m.espdl")
    g.save(path)
    m = model.Model(path)
    weights = {name: arr for name, arr, _ in g.initializers}
    ins, outs = {t.name: t for t in m.inputs}, {t.name: t for t in m.outputs}
    for _ in range(2):
        for t in ins.values():
            t.array[...] = rng.integers(-60, 60, size=t.shape, dtype=t.array.dtype)
        m.run()
        for i, (sa, sb, qt) in enumerate(pairs):
            want = graph_oracle.matmul(checkers.oracle(), ins[f"a{i}"].array, weights[f"b{i}"], -5, -6, -3, abi.DTYPE_INT8 if qt == "S8" else abi.DTYPE_INT16,
                                       abi.ACT_LINEAR, abi.ROUND_HALF_UP)
            np.testing.assert_array_equal(np.asarray(outs[f"y{i}"].array).reshape(want.shape), want, err_msg=f"product {i}")
    m.close()


def test_parallel_products_that_share_the_scratch(tmp_path):
    """int8 products that pack their operands, in branches beside one another and an int16 one that splits its own."""
    products_model(tmp_path, [((4096, 100), (100, 512), "S8"), ((512, 128), (128, 64), "S16"), ((3000, 60), (60, 512), "S8"), ((4096, 100), (100, 512), "S8")],
                   np.random.default_rng(8))


def test_constants_that_repeat_over_slices_one_behind_the_other(tmp_path):
    """Each repeats its constant into the same scratch and multiplies by it from there."""
    products_model(tmp_path, [((3, 2, 64, 32), (1, 2, 32, 48), "S8"), ((5, 2, 33, 32), (1, 2, 32, 48), "S8"), ((4, 3, 9, 12), (1, 3, 12, 20), "S8")],
                   np.random.default_rng(9))


@pytest.mark.parametrize("n,m,k,cout", [(2, 256, 64, 256), (8, 300, 512, 129), (3, 200, 100, 300), (64, 16, 48, 24)])
def test_batch_of_int16_products_with_the_scratch_it_asks_for(n, m, k, cout):
    """Large slices run one by one on the tile kernel out of the scratch that the query names, small ones together; without the scratch
    every batch runs on the CUDA cores."""
    import ctypes as C
    rng = np.random.default_rng(k)
    whole = cases.conv_case(seed=1, n=n, h=1, w=m, cin=k, cout=cout, kh=1, kw=1, pad=(0, 0, 0, 0), bias=False, **dict(S16, e_out=-14))
    whole.update(x=rng.integers(-32768, 32768, size=(n, 1, m, k), dtype=np.int16), w=rng.integers(-32768, 32768, size=(n, cout, 1, 1, k), dtype=np.int16),
                 filter_image_stride=cout * k)
    want = np.zeros_like(whole["out"])
    for i in range(n):
        one = cases.conv_case(seed=1, n=1, h=1, w=m, cin=k, cout=cout, kh=1, kw=1, pad=(0, 0, 0, 0), bias=False, **dict(S16, e_out=-14))
        one.update(x=whole["x"][i:i + 1], w=whole["w"][i], filter_exponent=whole["filter_exponent"])
        want[i:i + 1] = gpu_util.run_conv_oracle(one)
    with gpu_util.DeviceBuffers() as dev:
        out = dev.upload(whole["out"])
        d = cases.conv_desc(whole, dict(input=dev.upload(whole["x"]), filter=dev.upload(whole["w"]), output=out))
        need = C.c_size_t(0)
        abi.check(dev.lib.espdl_b200_conv2d_workspace_bytes(C.byref(d), C.byref(need)), "workspace")
        assert (need.value > 0) == (n < 64)
        for size in {need.value, 0}:
            scratch = dev.upload(np.zeros(max(size, 1), dtype=np.uint8))
            abi.check(dev.lib.espdl_b200_conv2d_ws(C.byref(d), scratch if size else None, size, None), "conv2d_ws")
            np.testing.assert_array_equal(dev.download(out, want), want)


@pytest.mark.parametrize("pairs", [[((4, 3, 260, 64), (4, 3, 64, 256), "S16")], [((4, 3, 260, 64), (1, 3, 64, 256), "S16"), ((3, 2, 9, 12), (1, 2, 12, 5), "S16")]])
def test_matmul_of_int16_slices(pairs, tmp_path):
    """Slices of one matrix each, and second operands that repeat over some of them, on the tile kernel and on the CUDA cores."""
    products_model(tmp_path, pairs, np.random.default_rng(10))


def conv_on(lib, case, stream, dev, ptrs):
    """One espdl_b200_conv2d on `stream`; returns the output's address."""
    import ctypes as C
    out = dev.upload(np.full_like(case["out"], 0x55))
    abi.check(lib.espdl_b200_conv2d(C.byref(cases.conv_desc(case, dict(ptrs, output=out))), stream), "conv2d")
    return out


@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
def test_packed_convs_under_capture(dtype):
    """Packing is an option of espdl_b200_conv2d: a capture, also the first time this size is met, runs without the scratch."""
    import ctypes as C
    lib = gpu_util.lib()
    extra = dict(S16, wide=True) if dtype == abi.DTYPE_INT16 else {}
    case = cases.conv_case(seed=3, n=3, h=61, w=59, cin=20, cout=40, kh=5, kw=5, pad=(2, 2, 2, 2), per_channel=True, **extra)
    want = gpu_util.run_conv_oracle(case)
    stream, graph = C.c_void_p(), C.c_void_p()
    abi.check(lib.espdl_b200_stream_create(C.byref(stream)), "stream")
    with gpu_util.DeviceBuffers() as dev:
        ptrs = dict(input=dev.upload(case["x"]), filter=dev.upload(case["w"]), bias=dev.upload(case["b"]), filter_exponents=dev.upload(case["ew"]))
        out = dev.upload(np.full_like(case["out"], 0x55))
        d = cases.conv_desc(case, dict(ptrs, output=out))
        need = C.c_size_t(0)
        abi.check(lib.espdl_b200_conv2d_workspace_bytes(C.byref(d), C.byref(need)), "workspace")
        assert need.value > 0
        abi.check(lib.espdl_b200_graph_begin(stream), "begin")
        st = lib.espdl_b200_conv2d(C.byref(d), stream)
        end = lib.espdl_b200_graph_end(stream, C.byref(graph))
        assert (st, end) == (abi.OK, abi.OK)
        abi.check(lib.espdl_b200_graph_launch(graph, stream), "launch")
        abi.check(lib.espdl_b200_stream_sync(stream), "sync")
        np.testing.assert_array_equal(dev.download(out, want), want)
        lib.espdl_b200_graph_destroy(graph)
    lib.espdl_b200_stream_destroy(stream)


@pytest.mark.parametrize("dtype", [abi.DTYPE_INT8, abi.DTYPE_INT16])
def test_packed_convs_on_streams_of_their_own(dtype):
    """Streams that nothing orders, more of them than keep a scratch, sizes that grow: each its own inputs and results."""
    import ctypes as C
    lib = gpu_util.lib()
    extra = dict(S16, wide=True) if dtype == abi.DTYPE_INT16 else {}
    layers = [cases.conv_case(seed=i, n=1 + i % 3, h=40, w=37, cin=20, cout=40, per_channel=True, **extra) for i in range(6)]
    want = [gpu_util.run_conv_oracle(c) for c in layers]
    streams = [C.c_void_p() for _ in range(6)]
    for s in streams:
        abi.check(lib.espdl_b200_stream_create(C.byref(s)), "stream")
    with gpu_util.DeviceBuffers() as dev:
        ptrs = [dict(input=dev.upload(c["x"]), filter=dev.upload(c["w"]), bias=dev.upload(c["b"]), filter_exponents=dev.upload(c["ew"])) for c in layers]
        outs = []
        for i in [0, 1] * 8 + list(range(6)) * 3:
            outs.append((i, conv_on(lib, layers[i], streams[i], dev, ptrs[i])))
        for s in streams:
            abi.check(lib.espdl_b200_stream_sync(s), "sync")
        for i, out in outs:
            np.testing.assert_array_equal(dev.download(out, want[i]), want[i])
    for s in streams:
        lib.espdl_b200_stream_destroy(s)


@pytest.mark.parametrize("layer", [dict(n=19, h=17, w=20, cin=96, cout=12, kh=5, kw=5, pad=(2, 2, 2, 2)), dict(n=2, h=45, w=47, cin=256, cout=48, kh=5, kw=5, pad=(2, 2, 2, 2))])
def test_int16_windows_without_scratch(layer, monkeypatch):
    """Layers that pack their operands where they get scratch; without it the warp-level instructions run them (the CUDA cores take a hundred times as long)."""
    import ctypes as C
    monkeypatch.delenv("ESPDL_B200_MMA16")
    case = cases.conv_case(seed=7, per_channel=True, **dict(S16, wide=True), **layer)
    want = gpu_util.run_conv_oracle(case)
    with gpu_util.DeviceBuffers() as dev:
        out = dev.upload(np.full_like(case["out"], 0x55))
        d = cases.conv_desc(case, dict(input=dev.upload(case["x"]), filter=dev.upload(case["w"]), bias=dev.upload(case["b"]), filter_exponents=dev.upload(case["ew"]), output=out))
        need = C.c_size_t(0)
        abi.check(dev.lib.espdl_b200_conv2d_workspace_bytes(C.byref(d), C.byref(need)), "workspace")
        assert need.value > 0
        for size in (0, need.value - 1, need.value):
            scratch = dev.upload(np.zeros(max(size, 1), dtype=np.uint8))
            abi.check(dev.lib.espdl_b200_conv2d_ws(C.byref(d), scratch if size else None, size, None), "conv2d_ws")
            np.testing.assert_array_equal(dev.download(out, want), want)


CAPTURED_PRODUCT = r"""
import ctypes as C, sys
sys.path.insert(0, sys.argv[1])
import conftest
import numpy as np
import cases, gpu_util
from espdl_b200 import abi
lib = gpu_util.lib()
case = cases.gemm_case(seed=9, m=871, k=1920, n_out=139, per_channel=True, dtype=abi.DTYPE_INT16, **eval(sys.argv[2]))
want = gpu_util.run_conv_oracle(case)
stream, graph = C.c_void_p(), C.c_void_p()
abi.check(lib.espdl_b200_stream_create(C.byref(stream)), "stream")
with gpu_util.DeviceBuffers() as dev:
    out = dev.upload(np.full_like(case["out"], 0x55))
    d = cases.conv_desc(case, dict(input=dev.upload(case["x"]), filter=dev.upload(case["w"]), bias=dev.upload(case["b"]), filter_exponents=dev.upload(case["ew"]), output=out))
    abi.check(lib.espdl_b200_graph_begin(stream), "begin")
    st = lib.espdl_b200_conv2d(C.byref(d), stream)
    end = lib.espdl_b200_graph_end(stream, C.byref(graph))
    assert (st, end) == (abi.OK, abi.OK), (st, end)
    abi.check(lib.espdl_b200_graph_launch(graph, stream), "launch")
    abi.check(lib.espdl_b200_stream_sync(stream), "sync")
    np.testing.assert_array_equal(dev.download(out, want), want)
    lib.espdl_b200_graph_destroy(graph)
lib.espdl_b200_stream_destroy(stream)
"""


def test_an_int16_product_is_captured_before_any_scratch_is_there():
    """In a process of its own: a product beside the line between the kernels, whose scratch nothing could allocate any more."""
    here = os.path.dirname(os.path.abspath(__file__))
    opts = {k: v for k, v in S16.items() if k != "dtype"}
    env = {k: v for k, v in os.environ.items() if k != "ESPDL_B200_MMA16"}
    r = subprocess.run([sys.executable, "-c", CAPTURED_PRODUCT, here, repr(opts)], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
