"""The host code of the context, the proposer and the statistics (auto_gb300/csrc/ctx.cu, mlp.cu, seed.cu) over stand-ins for
the CUDA runtime and the passes (tests/cpp/fake_cudart.cpp, fake_passes.cpp): what happens when a call of the runtime fails, and in which order copies and kernels touch the
caller's memory.  No GPU; the kernels are simple functions of the same arguments, so every value is exact."""
import ctypes
import mmap
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

from auto_gb300 import _lib
from auto_gb300.program import Kernel, World


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc) or not shutil.which("g++"):
        pytest.skip("needs nvcc and g++")
    d = str(tmp_path_factory.mktemp("runtime"))
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    objs = []
    for name in ("ctx", "mlp", "seed"):
        objs.append(os.path.join(d, name + ".o"))
        # PTX only: the kernels do not run here
        subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=compute_103a", "-O1", "-std=c++17", "-Xcompiler", "-fPIC",
                               "-I" + os.path.join(ROOT, "include"), "-c", os.path.join(ROOT, "auto_gb300", "csrc", name + ".cu"),
                               "-o", objs[-1]])
    so = os.path.join(d, "runtime_host.so")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + include,
                           "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(ROOT, "auto_gb300", "csrc")] +
                          [os.path.join(ROOT, "tests", "cpp", f) for f in ("fake_cudart.cpp", "fake_passes.cpp")] + objs + ["-o", so])
    return ctypes.CDLL(so)


def test_statistics_of_a_smaller_context_between_set_and_launch(lib):
    """The shared-memory limit belongs to the kernel, which all contexts share: a call for small worlds that comes between
    another thread's setting of the limit and its launch leaves that launch valid."""
    small = []
    hook = ctypes.CFUNCTYPE(None)(lambda: small.append(lib.fake_world_stats(4096 + 4096)))
    lib.fake_on_attribute(hook)
    assert lib.fake_world_stats(8192 + 8192)
    assert small == [1]
    assert lib.fake_world_stats(32 + 32)


IN, OUT, NPARAM, EINVAL, ECUDA = 16, 3, 70915, -1, -4
F = ctypes.POINTER(ctypes.c_float)


def ptr(a):
    return ctypes.cast(a.ctypes.data, F)


def floats(n, aligned=True):
    """n floats, 16-byte aligned or 4 bytes past such an address (which only a copy takes)."""
    a = np.zeros(n + 8, np.float32)
    k = -(a.ctypes.data // 4) % 4 + (0 if aligned else 1)
    return a[k:k + n]


def rows(n, aligned=True):
    """Rows whose sums are their numbers."""
    a = floats(n * IN, aligned)
    a[::IN] = np.arange(n)
    return a


def probabilities(n):
    return np.arange(n, dtype=np.float32)[:, None] + np.arange(OUT, dtype=np.float32)


@pytest.fixture
def mlp(lib):
    h = ctypes.c_void_p()
    lib.lenia_mlp_destroy.argtypes = [ctypes.c_void_p]
    lib.fake_reads_host(1)
    assert lib.lenia_mlp_create(1, 4096, ctypes.byref(h)) == 0
    yield h
    lib.fake_fail(b"", 0)
    lib.lenia_mlp_destroy(h)


def test_gradients_report_a_failed_download(lib, mlp):
    """Gradients that leave by copy: a copy that the runtime refuses is an error of this call, and of no later one."""
    x, y, loss = rows(100), floats(100 * OUT), ctypes.c_float()
    for aligned, want in ((False, ECUDA), (True, 0), (False, 0)):
        g = floats(NPARAM, aligned)
        if want:
            lib.fake_fail(b"cudaMemcpyAsync:down", 0)
        assert lib.lenia_mlp_gradients(mlp, ptr(x), ptr(y), 100, ptr(g), ctypes.byref(loss)) == want
        assert lib.fake_failed()
        if not want:
            assert (g == x.sum()).all() and loss.value == x[::IN].mean()


# the last two: rows of more than one half (38,912 rows), page-locked, so that copies are in flight as well
@pytest.mark.parametrize("call, count, aligned, locked, what, skip", [
    ("predict", 1000, (True, False), False, b"cudaMemcpyAsync:down", 0),
    ("predict", 100000, (True, True), False, b"cudaMemcpyAsync:down", 0),
    ("predict", 1000, (False, True), True, b"cudaMemcpyAsync:down", 0),
    ("predict", 100000, (False, True), True, b"cudaMemcpyAsync:up", 2),
    ("predict", 100000, (False, True), True, b"cudaMemcpyAsync:down", 1),
    ("gradients", 1000, (True, False), False, b"cudaMemcpyAsync:down", 0),
    ("gradients", 1000, (True, True), False, b"copy_out", 0),
    ("gradients", 1000, (False, True), True, b"cudaMemcpyAsync:up", 1),
    ("train_step", 1000, (True, True), False, b"adam", 0),
])
def test_a_failed_call_leaves_nothing_running(lib, mlp, call, count, aligned, locked, what, skip):
    """A call that fails half way waits for what it has queued: the caller may free its arrays.  The next call is
    as good as ever."""
    x, y = rows(count, aligned[0]), floats(count * OUT)
    out = floats(count * OUT if call == "predict" else NPARAM, aligned[1])
    loss = ctypes.c_float()
    if locked:
        lib.fake_lock(ptr(x), ctypes.c_size_t(x.nbytes))

    def run():
        if call == "predict":
            return lib.lenia_mlp_predict(mlp, ptr(x), count, ptr(out))
        if call == "gradients":
            return lib.lenia_mlp_gradients(mlp, ptr(x), ptr(y), count, ptr(out), ctypes.byref(loss))
        return lib.lenia_mlp_train_step(mlp, ptr(x), ptr(y), count, ctypes.c_float(0.1), ctypes.byref(loss))

    lib.fake_fail(what, skip)
    assert run() == ECUDA
    assert lib.fake_failed() and lib.fake_pending() == 0
    assert run() == 0 and lib.fake_pending() == 0
    if call == "predict":
        np.testing.assert_array_equal(out.reshape(-1, OUT), probabilities(count))
    elif call == "gradients":
        assert (out == x.sum(dtype=np.float64).astype(np.float32)).all()
    if locked:
        lib.fake_unlock(ptr(x))


def fresh(n):
    """n floats (zeros) in pages that nobody has touched."""
    return np.frombuffer(mmap.mmap(-1, 4 * n), np.float32)


@pytest.mark.parametrize("count", [1, 63, 64, 4000, 250001])
def test_every_page_is_touched_from_the_host_before_a_kernel_gets_it(lib, mlp, count):
    """A kernel that walked into a page that is not the caller's would take the GPU's context with it; the host's touch
    faults here.  So every page of a range that goes to a kernel in place has been touched."""
    loss = ctypes.c_float()
    x, probs = fresh(count * IN), fresh(count * OUT)
    assert lib.lenia_mlp_predict(mlp, ptr(x), count, ptr(probs)) == 0
    assert lib.fake_absent() == 0
    if count <= 4096:
        x, y, g = fresh(count * IN), fresh(count * OUT), fresh(NPARAM)
        assert lib.lenia_mlp_gradients(mlp, ptr(x), ptr(y), count, ptr(g), ctypes.byref(loss)) == 0
        assert lib.fake_absent() == 0
        x, y = fresh(count * IN), fresh(count * OUT)
        assert lib.lenia_mlp_train_step(mlp, ptr(x), ptr(y), count, ctypes.c_float(0.1), ctypes.byref(loss)) == 0
        assert lib.fake_absent() == 0


# in place in one launch and in two, copied in one half, two, three and four
@pytest.mark.parametrize("count, aligned", [(1000, True), (100000, True), (1048577, True), (38912, False), (38913, False), (77825, False),
                                            (150000, False)])
@pytest.mark.parametrize("at", [0, 4, 0.5, 1])
def test_probabilities_anywhere_over_their_own_rows(lib, mlp, count, aligned, at):
    """The probabilities of the first rows may lie over rows that are yet to be read."""
    k = int(at * (count * IN - count * OUT)) // 4 * 4 if at <= 1 else at  # floats from the rows' start; 1: at their end
    x = rows(count, aligned)
    assert lib.lenia_mlp_predict(mlp, ptr(x), count, ptr(x[k:])) == 0
    np.testing.assert_array_equal(x[k:k + count * OUT].reshape(-1, OUT), probabilities(count))
    assert lib.fake_pending() == 0


@pytest.mark.parametrize("count, aligned", [(1000, True), (100000, True), (100000, False)])
def test_a_launch_is_judged_by_its_own_status(lib, mlp, count, aligned):
    """An older error of the runtime's is no failure of this call; a refused launch is, on every route."""
    x, probs, y, g, loss = rows(count, aligned), floats(count * OUT), floats(4096 * OUT), floats(NPARAM), ctypes.c_float()

    def calls():
        yield b"mlp_rank", lambda: lib.lenia_mlp_predict(mlp, ptr(x), count, ptr(probs))
        yield b"mlp_tile", lambda: lib.lenia_mlp_gradients(mlp, ptr(x), ptr(y), 1000, ptr(g), ctypes.byref(loss))
        yield b"adam", lambda: lib.lenia_mlp_train_step(mlp, ptr(x), ptr(y), 1000, ctypes.c_float(0.1), ctypes.byref(loss))

    for kernel, call in calls():
        lib.fake_leave_error()
        assert call() == 0
        lib.fake_fail(kernel, 0)
        assert call() == ECUDA and lib.fake_failed() and lib.fake_pending() == 0
        assert call() == 0
    np.testing.assert_array_equal(probs.reshape(-1, OUT), probabilities(count))


# ---------------------------------------------------------------------- states

@pytest.fixture
def context(lib):
    """make(worlds): a context of one-kernel worlds of these (width, height)."""
    made = []
    lib.lenia_destroy.argtypes = [ctypes.c_void_p]
    lib.fake_reads_host(1)

    def make(worlds):
        descs = (_lib.LeniaWorldDesc * len(worlds))(*[World(w, h, [Kernel(radius=5.0)]).to_desc() for w, h in worlds])
        made.append(ctypes.c_void_p())
        assert lib.lenia_create(descs, len(worlds), 0, ctypes.byref(made[-1])) == 0
        return made[-1]

    yield make
    lib.fake_fail(b"", 0)
    for c in made:
        lib.lenia_destroy(c)


def size(n):
    return ctypes.c_size_t(n)


@pytest.mark.parametrize("refused", ["lenia_read_states", "lenia_mlp_get_params"])
def test_a_reported_error_does_not_come_back(lib, mlp, context, refused):
    """An error that a call has reported is not found again by a later, valid one."""
    n = 256 * 256
    ctx, state, out = context([(256, 256)]), floats(n), floats(n)
    state[:] = np.arange(n)
    lib.fake_fail(b"cudaMemcpyAsync:down", 0)
    if refused == "lenia_read_states":
        assert lib.lenia_read_states(ctx, ptr(out), size(n)) == ECUDA
    else:
        assert lib.lenia_mlp_get_params(mlp, ptr(floats(NPARAM)), size(NPARAM)) == ECUDA
    assert lib.fake_failed()
    assert lib.lenia_write_state(ctx, 0, ptr(state), size(n)) == 0
    assert lib.lenia_read_state(ctx, 0, ptr(out), size(n)) == 0
    np.testing.assert_array_equal(out, state)
    x, probs = rows(100), floats(100 * OUT)
    assert lib.lenia_mlp_predict(mlp, ptr(x), 100, ptr(probs)) == 0


@pytest.mark.parametrize("w, h", [(96, 32), (128, 128), (192, 128), (256, 256), (512, 512)])
def test_states_copied_in_place_are_touched_first(lib, context, w, h):
    n = w * h
    ctx, state, out = context([(w, h)]), fresh(n), fresh(n)
    assert lib.lenia_write_state(ctx, 0, ptr(state), size(n)) == 0
    assert lib.lenia_read_state(ctx, 0, ptr(out), size(n)) == 0
    assert lib.fake_absent() == 0 and lib.fake_pending() == 0


@pytest.mark.parametrize("worlds, want", [
    ([(256, 256)] * 4, (0, False)),                                  # one class
    ([(256, 256)] * 4 + [(512, 512)] * 2, (512 * 512 - 1, True)),     # within 128 MiB
    ([(512, 512)] * 2 + [(256, 512)], (512 * 512 - 1, True)),
    ([(1024, 1024)] * 16 + [(256, 256)], (384 * 384, False)),         # within 256 MiB
    ([(384, 256)] * 110 + [(256, 256)], (384 * 256 - 1, True)),
    ([(384, 256)] * 200 + [(256, 256)], (384 * 256 - 1, False)),
    ([(1024, 1024)] * 30 + [(256, 256)], (0, False)),                 # beyond
])
def test_the_default_branch_split(lib, context, worlds, want):
    """lenia_branch_split of a new context, by the bytes that its worlds touch in a step (9 a cell and a bit); lenia_set_branch_split
    replaces it, and cells = 0 turns it off."""
    ctx, cells, each = context(worlds), ctypes.c_int64(), ctypes.c_int32()

    def split():
        assert lib.lenia_branch_split(ctx, ctypes.byref(cells), ctypes.byref(each)) == 0
        return cells.value, bool(each.value)

    assert split() == want
    assert lib.lenia_set_branch_split(ctx, ctypes.c_int64(128 * 128), 1) == 0
    assert split() == (128 * 128, True)
    assert lib.lenia_set_branch_split(ctx, ctypes.c_int64(0), 0) == 0
    assert split() == (0, False)


@pytest.mark.parametrize("batch", [0, 4097, 0x7fffffff, 0x80000000, 0xffffffff])
def test_batches_beyond_the_handle_are_refused(lib, mlp, batch):
    x, y, g, loss = rows(1), floats(OUT), floats(NPARAM), ctypes.c_float()
    b = ctypes.c_uint32(batch)
    assert lib.lenia_mlp_gradients(mlp, ptr(x), ptr(y), b, ptr(g), ctypes.byref(loss)) == EINVAL
    assert lib.lenia_mlp_train_step(mlp, ptr(x), ptr(y), b, ctypes.c_float(0.1), ctypes.byref(loss)) == EINVAL
