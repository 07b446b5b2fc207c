"""The library's host code on a CUDA runtime without a GPU (fake_cudart.cpp):
what it copies and where to, what it launches, and what it does when a call
fails.  Kernels do not run, so no values are checked here."""
import ctypes as C
import importlib.util
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INC = "/usr/local/cuda/include"


class Fake:
    """The library linked with the fake runtime, and the runtime's log."""

    def __init__(self, path):
        from soapbubble_gb300 import _lib
        spec = importlib.util.spec_from_file_location("fake_sb_lib", _lib.__file__)
        self.m = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(self.m)
        self.m.LIB_PATH = path
        L = self.L = self.m.lib()
        L.fake_log.restype = L.fake_graph_node.restype = C.c_char_p
        L.fake_fail.argtypes = [C.c_char_p, C.c_int]

    def log(self, kind=""):
        lines = [self.L.fake_log(i).decode() for i in range(self.L.fake_log_size())]
        return [l for l in lines if l.startswith(kind)]

    def copies(self):
        return [tuple(int(v) for v in l.split()[1:]) for l in self.log("copy")]  # (to, from, bytes)

    def clear(self):
        self.L.fake_clear()

    def fail(self, name, nth=1):
        self.L.fake_fail(name.encode(), nth)

    def params(self, nT, **kw):
        p = self.m.SbParams()
        self.L.sb_default_params(C.byref(p))
        p.nTheta = nT
        for k, v in kw.items():
            setattr(p, k, v)
        return p

    def bubble(self, nT, **kw):
        h = C.c_void_p()
        p = self.params(nT, **kw)
        assert self.L.sb_create(C.byref(p), C.byref(h)) == 0, self.L.sb_last_error()
        return h

    def batch(self, members):
        arr = (C.c_void_p * len(members))(*[m.value for m in members])
        h = C.c_void_p()
        assert self.L.sb_batch_create(arr, len(members), C.byref(h)) == 0, self.L.sb_last_error()
        return h

    def field(self, name):
        return self.m.FIELD_ID[name]


def dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.fixture(scope="module")
def fake(gpulib, tmp_path_factory):
    from soapbubble_gb300 import build
    objs = [os.path.join(build.BUILD, os.path.splitext(s)[0] + ".o") for s in build.LIB_SOURCES]
    out = str(tmp_path_factory.mktemp("fake") / "libsb_fake.so")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-Wl,-Bsymbolic", "-I", CUDA_INC,
                    os.path.join(HERE, "fake_cudart.cpp"), *objs, "-o", out], check=True)
    return Fake(out)


@pytest.mark.parametrize("nT", [8, 64, 512])
@pytest.mark.parametrize("name", ["uair", "vair", "u_phi", "eta"])
def test_uploads_stay_inside_their_landing_place(fake, nT, name):
    """An FP64 array lands in scratch between steps: no copy may reach the
    landing place of another one (the four arrays of sb_upload_fields mark
    where each begins)."""
    h = fake.bubble(nT)
    N = 2 * nT * nT
    a = np.zeros(N + 1)
    fake.clear()
    assert fake.L.sb_upload_fields(h, dp(a), dp(a), dp(a), dp(a), None, None) == 0
    places = sorted(to for to, _, _ in fake.copies())
    assert len(places) == 4
    n = fake.L.sb_field_size(h, fake.field(name))
    fake.clear()
    assert fake.L.sb_upload_field(h, fake.field(name), dp(a), n) == 0
    copies = fake.copies()
    assert copies
    for to, _, size in copies:
        assert not any(to < p < to + size for p in places)
    fake.L.sb_destroy(h)


@pytest.mark.parametrize("call,nth", [("cudaMemcpyAsync", 2), ("cudaMemcpyAsync", 4), ("launch", 1)])
def test_a_failed_upload_leaves_no_copy_in_flight(fake, call, nth):
    """The caller may free its arrays as soon as an upload has returned, also
    with an error: every copy from them has been waited for."""
    h = fake.bubble(256)
    N = 2 * 256 * 256
    a = np.zeros(N + 1)

    def waited_for():
        log = fake.log()
        last = max((k for k, l in enumerate(log) if l.startswith("copy")), default=-1)
        return "synchronised" in log[last + 1:]

    fake.clear()
    fake.fail(call, nth)
    assert fake.L.sb_upload_fields(h, dp(a), dp(a), dp(a), dp(a), None, None) == fake.m.SB_ERR_CUDA
    assert fake.log("failed") and waited_for()
    for name in ("u_phi", "eta"):
        fake.clear()
        fake.fail(call, 1)
        rc = fake.L.sb_upload_field(h, fake.field(name), dp(a), N)
        assert rc == fake.m.SB_ERR_CUDA and waited_for()
    fake.clear()
    fake.L.sb_destroy(h)


@pytest.mark.parametrize("nT", [64, 1024])
def test_a_captured_step_makes_no_streams_or_events(fake, nT):
    """The first step of a handle or a batch captures its launches; the branch
    of the velocities beside maps and thickness is made of the capture's own
    dependencies, not of a stream and events made for it."""
    h = fake.bubble(nT)
    B = fake.batch([h])
    for step in (lambda: fake.L.sb_batch_step(B, 1, 0.0, 0.005), lambda: fake.L.sb_step(h, 1, 0.0, 0.005)):
        fake.clear()
        assert step() == 0, fake.L.sb_last_error()
        assert not fake.log("stream created") and not fake.log("event created")
        nodes = [fake.L.fake_graph_node(i).decode() for i in range(fake.L.fake_graph_size())]
        deps = [[int(d) for d in n.split(":")[1].split()] for n in nodes]
        at = {k: i for k in ("advect_maps", "velocity", "bimocq", "assemble") for i, n in enumerate(nodes) if k in n}
        assert len(nodes) == 9
        assert deps[at["advect_maps"]] == deps[at["velocity"]] == []
        assert deps[at["bimocq"]] == [at["advect_maps"]]
        assert sorted(deps[at["assemble"]]) == sorted([at["velocity"], at["bimocq"]])
        assert all(deps[i] == [i - 1] for i in range(at["assemble"] + 1, 9))
    # a capture that fails leaves the handle usable
    fake.clear()
    g = fake.bubble(nT)
    fake.fail("cudaStreamUpdateCaptureDependencies", 2)
    assert fake.L.sb_step(g, 1, 0.0, 0.005) == fake.m.SB_ERR_CUDA
    fake.clear()
    assert fake.L.sb_step(g, 1, 0.0, 0.005) == 0
    assert len(fake.log("launch")) == 9
    fake.L.sb_batch_destroy(B)
    fake.L.sb_destroy(h)
    fake.L.sb_destroy(g)


def test_a_batch_is_made_and_fed_without_pinning_or_blocking(fake):
    """A serving loop rebuilds its batch whenever requests join: the tables go
    up in one copy on the batch's own stream, and so do the step scalars."""
    members = [fake.bubble(n) for n in (64, 128, 64)]
    fake.clear()
    B = fake.batch(members)
    assert not fake.log("page-locked") and not fake.log("blocking")
    assert len(fake.log("copy")) == 1
    assert fake.log()[-1] == "synchronised"  # the tables' host copy is free again, errors are reported here
    for t in ([0.1, 0.2, 0.3], [0.2, 0.2, 0.4]):
        fake.clear()
        ts = np.array(t)
        assert fake.L.sb_batch_step_each(B, 1, dp(ts), 0.005) == 0
        log = fake.log()
        # the scalars are rewritten only after the stream has drained
        assert len(fake.log("copy")) == 1 and log[0] == "synchronised" and log[1].startswith("copy")
    fake.clear()
    assert fake.L.sb_batch_step_each(B, 1, dp(ts), 0.005) == 0
    assert not fake.log("copy")  # unchanged
    fake.L.sb_batch_destroy(B)
    for m in members:
        fake.L.sb_destroy(m)


@pytest.mark.parametrize("call", ["cudaMemcpyAsync", "launch"])
def test_step_scalars_that_did_not_arrive_are_sent_again(fake, call):
    """A batch step whose scalars could not be sent leaves the members' frame
    time unknown: the next call with the same time sends them."""
    h = fake.bubble(64)
    B = fake.batch([h])
    assert fake.L.sb_batch_step(B, 1, 0.0, 0.005) == 0
    fake.clear()
    fake.fail(call, 1)
    assert fake.L.sb_batch_step(B, 1, 0.5, 0.005) == fake.m.SB_ERR_CUDA
    fake.clear()
    assert fake.L.sb_batch_step(B, 1, 0.5, 0.005) == 0
    assert len(fake.log("copy")) == 1 and any("k_set_params" in l for l in fake.log("launch"))
    fake.L.sb_batch_destroy(B)
    fake.L.sb_destroy(h)


def test_launch_counts_include_the_step_scalars(fake):
    """sb_stats.launches counts the kernels that served a handle: a batch of
    one counts what the runtime saw."""
    h = fake.bubble(64)
    B = fake.batch([h])
    st = fake.m.SbStats()

    def count():
        assert fake.L.sb_get_stats(h, C.byref(st)) == 0
        return st.launches

    before = count()
    fake.clear()
    for t in (0.1, 0.1, 0.2):
        assert fake.L.sb_batch_step(B, 2, t, 0.005) == 0
    assert len(fake.log("launch")) == 3 * 2 * 9 + 2
    assert count() - before == len(fake.log("launch"))
    fake.L.sb_batch_destroy(B)
    fake.L.sb_destroy(h)


def test_a_smaller_smallest_tile_does_not_compile(tmp_path):
    """The parallel chain kernels deal kSampleCells cells to a block and are
    launched over the smallest tiles: another smallest tile is refused when
    they are compiled, and does not index out of their shared arrays."""
    import shutil
    from soapbubble_gb300 import build
    src = tmp_path / "csrc"
    shutil.copytree(build.CSRC, src)
    for f in src.iterdir():
        t = f.read_text()
        f.write_text(t.replace("kTileSizes[3] = {64, 128, 256}", "kTileSizes[3] = {32, 128, 256}"))
    cmd = [build.nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "--expt-relaxed-constexpr",
           "-I", os.path.join(build.ROOT, "include"), "-I", str(src), "--cuda", str(src / "sb_chain.cu"),
           "-o", str(tmp_path / "out.ii")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode != 0
    assert "static assertion" in r.stdout + r.stderr


@pytest.mark.parametrize("sizes,kw,fixed", [([64], {}, True), ([64, 64], {}, True), ([512], {}, False),
                                            ([64], {"storage": 1}, False), ([64, 1024], {}, False)])
def test_autotune_reports_the_tiles_in_use(fake, sizes, kw, fixed):
    """Small FP32 sets sample thickness and accumulation over 64-cell tiles
    whatever was timed; the sizes reported are the sizes used (the fake
    runtime times every size alike, which selects 128)."""
    members = [fake.bubble(n, **kw) for n in sizes]
    out = (C.c_int * 8)()
    if len(members) == 1:
        assert fake.L.sb_autotune(members[0], 0.0, 0.005, out) == 0
    else:
        B = fake.batch(members)
        assert fake.L.sb_batch_autotune(B, 0.0, 0.005, out) == 0
        fake.L.sb_batch_destroy(B)
    names = [fake.L.sb_stage_name(k).decode() for k in range(8)]
    got = dict(zip(names, out))
    want = 64 if fixed else 128
    assert got["k_bimocq"] == got["k_accum"] == want
    assert got["k_advect_maps"] == got["k_assemble"] == 128
    for m in members:
        fake.L.sb_destroy(m)


def test_the_chains_are_dealt_by_the_device_at_hand(fake):
    """Chains run in parallel below one thread per cell of the device, of
    however many multiprocessors it has."""
    def form(nT):
        h = fake.bubble(nT)
        fake.clear()
        assert fake.L.sb_step(h, 1, 0.0, 0.005) == 0
        names = [l for l in fake.log("launch") if "k_bimocq_chains" in l]
        fake.L.sb_destroy(h)
        assert len(names) == 1
        return int(names[0].split("Li")[1].split("E")[0])  # the kernel's PAR argument

    try:
        assert [form(n) for n in (64, 256, 512)] == [5, 5, 1]
        fake.L.fake_set_sms(8)
        assert [form(n) for n in (64, 128, 256)] == [5, 1, 1]
    finally:
        fake.L.fake_set_sms(152)


@pytest.mark.parametrize("nT,launches", [(16, 0), (128, 0), (256, 1)])
def test_small_fields_take_one_copy_and_no_kernel(fake, nT, launches):
    """FP32 arrays of up to 128 x 256 cells are rounded on the host: a kernel
    behind the copy would take longer than the host's loop."""
    h = fake.bubble(nT)
    a = np.zeros(2 * nT * nT)
    fake.clear()
    assert fake.L.sb_upload_field(h, fake.field("u_phi"), dp(a), a.size) == 0
    assert len(fake.log("copy")) == 1 and len(fake.log("launch")) == launches
    fake.L.sb_destroy(h)
