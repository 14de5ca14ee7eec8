"""CPU-side checks of the C ABI: the built library loads and exports every symbol include/espdl_b200.h
declares, the ctypes mirrors have the C structs' sizes, and calls fail cleanly (no compute) without a GPU."""
import ctypes as C
import os
import re
import subprocess

import pytest

from espdl_b200 import abi

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "espdl_b200.h")


@pytest.fixture(scope="module")
def library():
    if not os.path.exists(abi.LIB_PATH):
        from espdl_b200 import build
        build.build()
    return abi.bind(C.CDLL(abi.LIB_PATH))


def test_every_declared_symbol_is_exported(library):
    text = open(HEADER).read()
    declared = set(re.findall(r"\b(espdl_b200_\w+)\s*\(", text))
    assert declared == set(abi.SYMBOLS), declared ^ set(abi.SYMBOLS)
    for name in declared:
        assert hasattr(library, name)


def test_struct_sizes_match_the_header(tmp_path):
    src = tmp_path / "sizes.c"
    src.write_text('#include <stdio.h>\n#include "espdl_b200.h"\nint main(void){printf("%zu %zu %zu %zu %zu %zu %zu %zu\\n",'
                   "sizeof(espdl_conv_desc),sizeof(espdl_eltwise_desc),sizeof(espdl_pool_desc),sizeof(espdl_resize_desc),"
                   "sizeof(espdl_copy_desc),sizeof(espdl_softmax_desc),sizeof(espdl_gather_desc),sizeof(espdl_norm_desc));return 0;}\n")
    exe = tmp_path / "sizes"
    subprocess.check_call(["/usr/bin/gcc", "-std=c99", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)])
    sizes = [int(x) for x in subprocess.check_output([str(exe)]).split()]
    mirrors = [abi.ConvDesc, abi.EltwiseDesc, abi.PoolDesc, abi.ResizeDesc, abi.CopyDesc, abi.SoftmaxDesc, abi.GatherDesc, abi.NormDesc]
    assert sizes == [C.sizeof(m) for m in mirrors]


def test_argument_validation_needs_no_gpu(library):
    assert library.espdl_b200_conv2d(None, None) == abi.ERR_INVALID_ARG
    assert library.espdl_b200_eltwise(None, None) == abi.ERR_INVALID_ARG
    assert library.espdl_b200_pool(None, None) == abi.ERR_INVALID_ARG
    assert library.espdl_b200_strerror(abi.ERR_TIMEOUT) == b"device-side wait timed out"
    assert library.espdl_b200_launch_count() == 0


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(abi, "LIB_PATH", str(tmp_path / "nope.so"))
    monkeypatch.setattr(abi, "_lib", None)
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        abi.load()


# windows of int16: pixels, filter, channels in and out; us on the warp-level instructions and on packed operands.  Only the latter asks for scratch.
INT16_TIMES = [((4, 40, 40), 3, 64, 64, 9.7, 12.3), ((47, 13, 12), 3, 96, 24, 12.9, 17.3), ((44, 14, 13), 3, 24, 128, 11.6, 13.7),
               ((3, 97, 98), 1, 24, 64, 14.3, 12.4), ((45, 11, 11), 3, 256, 80, 37.3, 22.1), ((1, 72, 70), 5, 32, 96, 17.8, 15.6), ((27, 13, 14), 5, 32, 80, 17.5, 15.2)]


@pytest.mark.parametrize("image,k,cin,cout,here,packed", INT16_TIMES)
def test_int16_windows_take_the_faster_kernel(library, image, k, cin, cout, here, packed):
    """Layers on both sides of the line, as measured; long reductions of few blocks were sent to the slower one."""
    d = abi.ConvDesc()
    d.input, d.filter, d.output = 1 << 20, 2 << 20, 3 << 20  # nothing is read
    d.dtype, d.n, d.in_h, d.in_w, d.in_c, d.out_c = abi.DTYPE_INT16, *image, cin, cout
    d.out_h, d.out_w, d.kh, d.kw, d.group = d.in_h, d.in_w, k, k, 1
    d.stride_h = d.stride_w = d.dilation_h = d.dilation_w = 1
    d.pad_top = d.pad_bottom = d.pad_left = d.pad_right = k // 2
    need = C.c_size_t(0)
    assert library.espdl_b200_conv2d_workspace_bytes(C.byref(d), C.byref(need)) == abi.OK
    assert (need.value == 0) == (here < packed)


# the same since rows of the reduction meet in threes here and results leave the tile kernel faster; a CUDA-core kernel asks for no scratch either
@pytest.mark.parametrize("image,k,cin,cout,here,packed", [((49, 101, 104), 3, 24, 24, 111.7, 304.8), ((4, 41, 43), 3, 8, 80, 6.1, 10.7), ((27, 98, 95), 1, 24, 12, 30.4, 49.2),
                                                          ((3, 46, 47), 7, 24, 48, 15.7, 25.2), ((63, 67, 66), 1, 24, 12, 33.5, 53.6), ((20, 91, 92), 3, 16, 32, 36.0, 57.6),
                                                          ((105, 8, 8), 5, 192, 12, 54.7, 33.6), ((19, 17, 20), 5, 96, 12, 29.4, 20.7)])
def test_int16_windows_since_both_kernels_changed(library, image, k, cin, cout, here, packed):
    test_int16_windows_take_the_faster_kernel(library, image, k, cin, cout, here, packed)
