"""What a model's plan hands to the device: the launches, their scratch and the order the captured streams keep them in, recorded by a
stand-in for the CUDA library (fake_device.c) in a process of its own.  No GPU."""
import os
import subprocess
import sys

import numpy as np
import pytest

from espdl_b200 import abi, espdl_file, model

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

CHILD = r"""
import ctypes as C, sys
host = C.CDLL(sys.argv[1])
host.espdl_model_create.restype = C.c_void_p
host.espdl_model_create.argtypes = [C.c_char_p, C.c_int, C.c_int]
for f in ("run", "destroy"):
    getattr(host, "espdl_model_" + f).argtypes = [C.c_void_p]
host.espdl_model_run_device.argtypes = [C.c_void_p, C.c_int]
host.espdl_model_arena_bytes.argtypes = [C.c_void_p]
host.espdl_model_arena_bytes.restype = C.c_size_t
h = host.espdl_model_create(sys.argv[2].encode(), int(sys.argv[3]), int(sys.argv[5]))
if not h:
    print("status none")
    sys.exit()
print("arena", host.espdl_model_arena_bytes(h))
for what in sys.argv[4].split(","):
    print(what, host.espdl_model_run(h) if what == "run" else host.espdl_model_run_device(h, 1))
host.espdl_model_destroy(h)
"""


@pytest.fixture(scope="session")
def fake(tmp_path_factory):
    """The host library beside a fake device library (it finds its device library through $ORIGIN)."""
    d = tmp_path_factory.mktemp("fake")
    host = d / os.path.basename(model.HOST_LIB_PATH)
    host.write_bytes(open(model.HOST_LIB_PATH, "rb").read())
    src = open(os.path.join(HERE, "fake_device.c")).read()
    names = subprocess.run(["nm", "-D", "--undefined-only", str(host)], capture_output=True, text=True, check=True).stdout.split()
    stubs = [n for n in names if n.startswith("espdl_b200_") and n + "(" not in src]
    (d / "fake.c").write_text(src + "".join(f'int {n}_stub(const void *d, void *s) __asm__("{n}");\n'
                                            f'int {n}_stub(const void *d, void *s) {{ line("{n[11:]} stream=%p scope=%d", s, scope); return 0; }}\n' for n in stubs))
    subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-Wno-unused-parameter", "-I" + os.path.join(ROOT, "include"), str(d / "fake.c"), "-o", str(d / "libespdl_b200.so"), "-ldl"])
    return str(host)


def record(fake, tmp_path, graph, calls="run", batch=0, child=CHILD, flags=0, **env):
    """[(call, {argument: value})] and the child's printed lines."""
    path, log = str(tmp_path / "g.espdl"), str(tmp_path / "log.txt")
    if isinstance(graph, str):
        path = graph
    else:
        graph.save(path)
    r = subprocess.run([sys.executable, "-c", child, fake, path, str(batch), calls, str(flags)], capture_output=True, text=True,
                       env=dict(os.environ, FAKE_DEVICE_LOG=log, REAL_DEVICE_LIB=abi.LIB_PATH, **env))
    assert r.returncode == 0, r.stderr
    lines = []
    for text in open(log).read().splitlines():
        name, *args = text.split()
        lines.append((name, dict(a.split("=") for a in args)))
    return lines, dict(t.split() for t in r.stdout.splitlines())


def captured(lines):
    """The calls between the first graph_begin and its graph_end."""
    names = [n for n, _ in lines]
    return lines[names.index("graph_begin") + 1:names.index("graph_end")]


def before(lines):
    """happens[j] = the captured calls that are done when call j starts: earlier ones of its stream and what its stream waited for."""
    done_of_stream, done_of_event, out = {}, {}, []
    for j, (name, a) in enumerate(lines):
        done = done_of_stream.setdefault(a.get("stream"), set())
        if name == "record":
            done_of_event[a["event"]] = set(done)
        elif name == "wait":
            done |= done_of_event[a["event"]]
        out.append(set(done))
        done.add(j)
    return out


def matmul_graph(pairs, second="constant"):
    """Parallel MatMuls: pairs = [(shape a, shape b, type)]; `second` operands are parameters or graph inputs."""
    rng = np.random.default_rng(5)
    g = espdl_file.GraphBuilder("products", metadata={"target": "c"})
    for i, (sa, sb, qt) in enumerate(pairs):
        t = np.int8 if qt == "S8" else np.int16
        g.add_input(f"a{i}", t, list(sa), -5)
        if second == "constant":
            g.add_initializer(f"b{i}", rng.integers(-60, 60, size=sb, dtype=t), [-6])
        else:
            g.add_input(f"b{i}", t, list(sb), -6)
        g.add_node("MatMul", f"mm{i}", [f"a{i}", f"b{i}"], [f"y{i}"], quant_type=qt, activation="Linear")
        lead = [max(x, y) for x, y in zip(sa[:-2], ([1] * (len(sa) - len(sb)) + list(sb))[:-2])]
        g.add_output(f"y{i}", t, lead + [sa[-2], sb[-1]], -3)
    return g


PACKED, PLAIN, WIDE = ((4096, 100), (100, 512), "S8"), ((256, 64), (64, 64), "S8"), ((512, 128), (128, 64), "S16")


def test_int8_products_that_pack_operands_are_ordered_by_their_scratch(fake, tmp_path):
    """Products whose reduction is no multiple of 16 pack their operands into the scratch: a step that uses it declares it, so that
    two of them in different branches never pack at the same time."""
    lines, _ = record(fake, tmp_path, matmul_graph([PACKED, WIDE, PACKED, PLAIN, PACKED]))
    caught = captured(lines)
    ordered = before(caught)
    users = [j for j, (n, a) in enumerate(caught) if n == "conv" and int(a["need"])]
    assert len(users) == 4
    for j in users:
        assert int(caught[j][1]["ws_bytes"]) >= int(caught[j][1]["need"]), "the plan has scratch for it"
    for i, a in enumerate(users):
        for b in users[i + 1:]:
            assert a in ordered[b], "two steps that write the scratch run side by side"


def test_products_without_scratch_of_their_own_get_none(fake, tmp_path):
    """Whether a product packs its operands does not depend on what other steps made the plan allocate."""
    lines, _ = record(fake, tmp_path, matmul_graph([WIDE, PLAIN, ((64, 30), (30, 17), "S8")]))
    small = [a for n, a in captured(lines) if n == "conv" and not int(a["need"])]
    assert len(small) == 2 and all(int(a["ws_bytes"]) == 0 for a in small)


def test_only_constants_are_read_ahead_of_the_previous_kernel(fake, tmp_path):
    """Inside a plan's scope kernels read their filter before the launches in front of them are done.  A filter that one of these
    writes - a constant repeated into the scratch, or another step's output - is launched outside of it; a constant inside."""
    repeated = ((3, 2, 64, 32), (1, 2, 32, 48), "S8")
    lines, _ = record(fake, tmp_path, matmul_graph([repeated, PLAIN]))
    caught = captured(lines)
    copies = {a["dst"] for n, a in caught if n == "copy"}
    scope = {(a["filter"] in copies): int(a["scope"]) for n, a in caught if n == "conv"}
    assert scope == {True: 0, False: 1}
    lines, _ = record(fake, tmp_path, matmul_graph([PLAIN], second="input"))
    assert [int(a["scope"]) for n, a in captured(lines) if n == "conv"] == [0]


def test_a_conv_whose_filter_another_step_writes(fake, tmp_path):
    g = espdl_file.GraphBuilder("dynamic", metadata={"target": "c"})
    g.add_input("x", np.int8, [1, 12, 12, 16], -5)
    g.add_input("f", np.int8, [1, 1, 16, 24], -6)
    g.add_initializer("w", np.ones((1, 1, 24, 16), dtype=np.int8), [-6])
    g.add_node("Conv", "c0", ["x", "f"], ["y"], quant_type="S8", activation="Linear", pads=[0, 0, 0, 0], strides=[1, 1], dilations=[1, 1], group=1)
    g.add_value_info("y", np.int8, [1, 12, 12, 24], -5)
    g.add_node("Conv", "c1", ["y", "w"], ["z"], quant_type="S8", activation="Linear", pads=[0, 0, 0, 0], strides=[1, 1], dilations=[1, 1], group=1)
    g.add_output("z", np.int8, [1, 12, 12, 16], -5)
    lines, _ = record(fake, tmp_path, g)
    assert [int(a["scope"]) for n, a in captured(lines) if n == "conv"] == [0, 1]


def test_int16_slices_have_the_scratch_of_the_tile_kernel(fake, tmp_path):
    """Batches of large int16 products run slice by slice on the tile kernel, which needs scratch for one: their own operand each, or one
    that repeats over some slices (then behind the repeated operand)."""
    lines, _ = record(fake, tmp_path, matmul_graph([((4, 3, 260, 64), (4, 3, 64, 256), "S16"), ((4, 3, 260, 64), (1, 3, 64, 256), "S16")]))
    convs = [a for n, a in captured(lines) if n == "conv"]
    spread = {int(a["dst"], 16) for n, a in captured(lines) if n == "copy"}
    assert len(convs) == 2 and len(spread) == 1
    for a in convs:
        assert int(a["need"]) and int(a["ws_bytes"]) >= int(a["need"])
        if int(a["filter"], 16) in spread:
            assert int(a["ws"], 16) >= int(a["filter"], 16) + 12 * 64 * 256 * 2


SCORING_CHILD = r"""
import ctypes as C, sys, threading
import numpy as np
host = C.CDLL(sys.argv[1])
host.espdl_model_create.restype = C.c_void_p
host.espdl_model_create.argtypes = [C.c_char_p, C.c_int, C.c_int]
host.espdl_model_run.argtypes = [C.c_void_p]
host.espdl_model_io_info.argtypes = [C.c_void_p, C.c_int, C.c_int] + [C.c_void_p] * 7
host.espdl_model_classify.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_float, C.c_int, C.POINTER(C.c_int), C.POINTER(C.c_float)]
host.espdl_model_detect.argtypes = [C.c_void_p, C.c_int, C.c_int, C.POINTER(C.c_char_p), C.POINTER(C.c_int), C.c_float, C.c_float, C.c_int, C.c_int, C.c_int, C.c_int,
                                    C.POINTER(C.c_int), C.POINTER(C.c_float)]
host.espdl_model_preprocess.argtypes = [C.c_void_p, C.c_void_p] + [C.c_int] * 4 + [C.POINTER(C.c_float)] * 2 + [C.c_int] * 2 + [C.c_void_p]
h = host.espdl_model_create(sys.argv[2].encode(), 0, 0)
assert host.espdl_model_run(h) == 0
name, ndim, shape, dtype, e, hp, dp = C.c_char_p(), C.c_int(), (C.c_int * 8)(), C.c_int(), C.c_int(), C.c_void_p(), C.c_void_p()
host.espdl_model_io_info(h, 1, 0, C.byref(name), C.byref(ndim), shape, C.byref(dtype), C.byref(e), C.byref(hp), C.byref(dp))
dims = list(shape[:ndim.value])
n = int(np.prod(dims))
logits = np.frombuffer((C.c_char * n).from_address(dp.value), dtype=np.int8).reshape(dims)  # the stand-in's device memory
logits[...] = np.random.default_rng(1).integers(-128, 128, size=dims, dtype=np.int8)

def classify(image, k=20):
    cat, score = (C.c_int * k)(), (C.c_float * k)()
    found = host.espdl_model_classify(h, image, k, 0.0, image % 2, cat, score)
    return found, list(cat[:max(found, 0)]), list(score[:max(found, 0)])

def detect(image, k=20):
    names = (C.c_char_p * 2)(b"y0", b"y0")
    box, score = (C.c_int * (5 * k))(), (C.c_float * k)()
    return host.espdl_model_detect(h, image, 1, names, (C.c_int * 1)(8), 0.5, 0.5, k, 64, 64, k, box, score)
"""


def test_images_outside_the_batch_have_no_results(fake, tmp_path):
    child = SCORING_CHILD + r"""
print("detect", ",".join(str(detect(i)) for i in (0, 1, 2, 7, -1)))
print("classify", ",".join(str(classify(i)[0]) for i in (2, 7, -1)))
"""
    _, said = record(fake, tmp_path, matmul_graph([((2, 4, 4, 16), (16, 64), "S8")]), child=child)
    assert said == {"detect": "0,0,0,0,0", "classify": "0,0,0"}


def test_several_threads_score_one_finished_batch(fake, tmp_path):
    """The objects that a handle keeps between calls serve one call at a time: threads that score different images, with and without
    softmax, detect and preprocess beside one another get what a single one gets."""
    child = SCORING_CHILD + r"""
want = [classify(i) for i in range(32)]
wrong = []
mean, std = (C.c_float * 3)(0, 0, 0), (C.c_float * 3)(1, 1, 1)
def score(part):
    for _ in range(40):
        for i in range(part, 32, 8):
            if classify(i) != want[i]:
                wrong.append(i)
def others(which):
    frames = np.zeros((1, 9 + which, 11, 1), dtype=np.uint8)
    for k in range(300):
        if detect(k % 32) != 0:
            wrong.append(-1)
        one = (C.c_float * 3)(k % 7, 0, 0)
        host.espdl_model_preprocess(h, frames.ctypes.data, 1, 9 + which, 11, 1, one, std, 0, -1, None)
threads = [threading.Thread(target=score, args=(p,)) for p in range(8)] + [threading.Thread(target=others, args=(w,)) for w in range(2)]
for t in threads: t.start()
for t in threads: t.join()
print("wrong", len(wrong))
"""
    _, said = record(fake, tmp_path, matmul_graph([((32, 1, 1, 16), (16, 64), "S8")]), child=child)
    assert said == {"wrong": "0"}


def test_no_memory_for_buffers_of_their_own_is_a_chain(fake, tmp_path):
    """Where the arena of a branched plan cannot be allocated the model takes the chain's, which loaded before there were branches."""
    from espdl_b200 import zoo
    g = zoo.yolo11n_style(seed=6, input_hw=96)
    lines, said = record(fake, tmp_path, g)
    branches = int(said["arena"])
    assert any(n == "wait" for n, _ in captured(lines))
    _, said = record(fake, tmp_path, g, ESPDL_B200_BRANCHES="0")
    chain = int(said["arena"])
    assert chain < branches
    lines, said = record(fake, tmp_path, g, FAKE_ARENA_LIMIT=str(branches))
    assert said == {"arena": str(chain), "run": "0"}
    assert not any(n == "wait" for n, _ in captured(lines))


def large_layer():
    """One 1x1 conv between tensors of 100 MB."""
    g = espdl_file.GraphBuilder("large", metadata={"target": "c"})
    g.add_input("x", np.int8, [1, 1024, 1024, 96], -5)
    g.add_initializer("w", np.ones((1, 1, 96, 96), dtype=np.int8), [-6])
    g.add_node("Conv", "c0", ["x", "w"], ["y"], quant_type="S8", activation="Linear", pads=[0, 0, 0, 0], strides=[1, 1], dilations=[1, 1], group=1)
    g.add_output("y", np.int8, [1, 1024, 1024, 96], -5)
    return g


def test_large_steps_are_plain_launches_however_buffers_are_planned(fake, tmp_path):
    for flags, env in ((0, {}), (0, {"ESPDL_B200_BRANCHES": "0"}), (2, {})):
        lines, _ = record(fake, tmp_path, large_layer(), calls="run_device", flags=flags, **env)
        assert [a["overlap"] for n, a in captured(lines) if n == "conv"] == ["0"], (flags, env)
    lines, _ = record(fake, tmp_path, matmul_graph([PLAIN]), calls="run_device")
    assert [a["overlap"] for n, a in captured(lines) if n == "conv"] == ["1"]


def test_run_and_run_device_share_the_graph_of_large_steps(fake, tmp_path):
    """The copies are part of the captured graph where a pass is short enough for launches to count."""
    lines, said = record(fake, tmp_path, large_layer(), calls="run,run_device,run")
    names = [n for n, _ in lines]
    assert names.count("graph_begin") == 1 and names.count("graph_launch") == 3 and said["run"] == "0"
    assert "upload" not in [n for n, _ in captured(lines)]
    lines, _ = record(fake, tmp_path, matmul_graph([PLAIN]), calls="run,run_device,run")
    names = [n for n, _ in lines]
    assert names.count("graph_begin") == 2 and "upload" in [n for n, _ in captured(lines)]


def test_a_capture_that_gets_no_stream_is_an_error(fake, tmp_path):
    """run() has no result of its own: what went wrong is the model's status, not the last pass's outputs in silence."""
    _, said = record(fake, tmp_path, matmul_graph([PLAIN, PLAIN, PLAIN]), calls="run,run_device", FAKE_STREAM_LIMIT="1")
    assert int(said["run"]) == abi.ERR_CUDA and int(said["run_device"]) != 0


def test_a_released_model_gives_its_tile_counters_back(fake, tmp_path):
    """Its graphs are idle by then: synchronised, then destroyed as such."""
    lines, _ = record(fake, tmp_path, matmul_graph([PLAIN]), calls="run,run_device")
    names = [n for n, _ in lines]
    assert names.count("graph_destroy_idle") == names.count("graph_begin") == 2 and "graph_destroy" not in names
    assert "stream_sync" in names[len(names) - 1 - names[::-1].index("graph_launch"):names.index("graph_destroy_idle")]
