"""Properties of the kernels' sources that no run can show: an ordering that one
machine happens to give, a limit that no test may wait for, an attribute of a
device that is not there."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rusty_h264_b200", "csrc")


def source(name):
    """A source file without its comments, white space folded."""
    with open(os.path.join(CSRC, name)) as f:
        t = f.read()
    t = re.sub(r"/\*.*?\*/", " ", t, flags=re.S)
    return re.sub(r"\s+", " ", re.sub(r"//[^\n]*", " ", t))


def body(name, head):
    """The text from `head` to the end of the braces that follow it."""
    t = source(name)
    i = t.index(head)
    j = t.index("{", i)
    depth = 0
    for k in range(j, len(t)):
        depth += (t[k] == "{") - (t[k] == "}")
        if depth == 0:
            return t[i:k + 1]
    raise AssertionError(head)


def test_column_sums_are_read_before_the_next_round_stores():
    """The lanes of a search exchange column sums through the warp's shared
    scratch: a __syncwarp between every read of a round and the next store."""
    for head in ("SearchOut search16(", "SearchOut search_parts("):
        b = body("mb_search.cuh", head)
        loop = b[b.index("bs.red"):]  # store, sync, read, ... and round again
        last = [m.end() for m in re.finditer(r"d \+= bs\.red\[[^;]*;", loop)][-1]
        # nothing but unconditional statements up to the __syncwarp
        m = re.match(r"((?:(?!\bif\b|\bcontinue\b|\bbreak\b|\bfor\b|\bwhile\b).)*?)__syncwarp\(\);", loop[last:])
        assert m, head


def test_deblocking_rows_wait_with_the_whole_warp():
    """Lane 0 alone acquires the row above's progress: a __syncwarp before the
    other lanes read that row's samples."""
    b = body("deblock.cu", "deblock_rows_kernel(")
    i = b.index("ld_acquire(gprog - 1)")
    reads = min(b.index("top_word(x)", i), b.index("db_strips + ((long long)(w - 1)", i))
    branch = b[i:reads]
    assert "__syncwarp();" in branch[branch.index("avail = W"):branch.index("if (top_shared) { if (lane < 20)")]


def test_motion_compensation_waits_with_the_whole_warp():
    """A lane may find in shared memory that another lane has seen a reference
    segment ready: a __syncwarp between those waits and the reads."""
    b = body("me.cu", "void frame_mb(")
    last = [m.end() for m in re.finditer(r"band_wait_px\(", b)][-1]
    for read in ("chroma_rows(", "plane_rows("):
        assert last < b.index(read), read
        assert "__syncwarp();" in b[last:b.index(read)], read


def test_an_mb_leaves_its_warp_scratch_to_the_next():
    """Lane 0 writes the warp's scratch for the next MB: a __syncwarp before
    every way out of an MB."""
    b = body("me.cu", "void frame_mb(")
    outs = [m.start() for m in re.finditer(r"\breturn;", b)] + [len(b) - 1]
    for o in outs:
        assert b[:o].rstrip().endswith("__syncwarp();"), b[max(0, o - 80):o + 8]


def test_wait_limits_are_times():
    """A wait's limit stands for polls SPIN_NS apart, about half a second: a
    loop that sleeps for another time scales it."""
    dev = source("h264a_device.cuh")
    ns = int(re.search(r"constexpr unsigned SPIN_NS = (\d+);", dev).group(1))
    limit = eval(re.search(r"constexpr int SPIN_LIMIT = ([\d *]+);", dev).group(1))
    scaled = re.search(r"int poll_limit\(int limit, unsigned ns\) \{ return int\((.*?)\); \}", dev).group(1)
    scaled = scaled.replace("(long long)", "").replace("/", "//")
    for every in (20, 40, 100, 200, 1000):
        polls = eval(scaled, {"limit": limit, "SPIN_NS": ns, "ns": every})
        assert polls * every == limit * ns >= 200_000_000
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        t = source(name)
        for m in re.finditer(r"__nanosleep\(([^;]*)\);", t):
            sleep = m.group(1)
            if sleep == "SPIN_NS":
                continue
            before = t[max(0, m.start() - 6000):m.start()]
            assert re.search(r"poll_limit\((spin_)?limit, %s\)" % re.escape(sleep), before), (name, sleep)


def test_network_kernels_opt_in_on_their_nets_device():
    """Dynamic shared memory above 48 KB is an attribute of a kernel on a
    device: mvnet_create sets it for every instantiation that is launched."""
    t = source("mvnet.cu")
    assert not re.search(r"static (const )?(bool|std::once_flag)", t)
    launched = {(k, re.sub(r"\s", "", a), op) for k, a, op in
                re.findall(r"\b(gemm|conv_gemm|wgrad)<([\d, ]+)>\((\w+(?:<[\d, ]+>)?)\{", t)}
    setup = body("mvnet.cu", "static int opt_in_kernels(")
    listed = {(k, re.sub(r"\s", "", a), op) for k, a, op in
              re.findall(r"H264A_CUDA\(\((\w+)_opt_in<((?:\d+, )*\d+), (\w+(?:<[\d, ]+>)?)>\(\)\)\)", setup)}
    assert len(launched) >= 12 and launched == listed
    assert "opt_in_kernels()" in body("mvnet.cu", "int h264a_mvnet_create(")


def test_multi_reference_kernels_opt_in_on_every_device():
    """As above for the frame kernels: no once-per-process opt-in."""
    t = source("me.cu")
    assert "once_flag" not in t and "call_once" not in t
    b = body("me.cu", "int h264a::mr_launch(")
    assert "me_mr_setup(" in b
    assert "cudaGetDevice(&dev)" in body("me.cu", "static int me_mr_setup(")


def test_network_waits_that_run_out_are_reported():
    """Every kernel that waits for the tensor cores has the net's status word,
    and every call on the net looks at it first."""
    t = source("mvnet.cu")
    for m in re.finditer(r"\b(\w+_tc_kernel|conv1_kernel)(<[^;{}]*?>)? ?<<<[^;]*;", t):
        assert m.group(0).endswith("z.status);"), m.group(0)[-60:]
    for call in ("forward", "grads", "propose", "get_params"):  # train_step calls grads
        assert "check_waits(" in body("mvnet.cu", "int h264a_mvnet_%s(" % call), call


def test_grid_opt_ins_do_not_depend_on_the_call():
    """Two threads' calls of different radius: the opt-in of one must not fall
    below what the other is about to launch with."""
    for m in re.finditer(r"cudaFuncSetAttribute\(fullpel_\w+, cudaFuncAttributeMaxDynamicSharedMemorySize, ([^)]*\)?)\)", source("grid.cu")):
        assert re.fullmatch(r"int\([A-Z_]+\)|[A-Z_]+", m.group(1)), m.group(1)
