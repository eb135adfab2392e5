"""The library's host code without a GPU: its objects linked with a fake CUDA runtime
(fake/fake_cuda.cpp) that logs the calls, keeps device memory on the host and fails
a named call.  Kernels do nothing there: only what the host does is tested."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from gaussmle_gb300 import _lib, build, serve
from gaussmle_gb300.constraints import default_constraints
from gaussmle_gb300.fitter import make_desc
from gaussmle_gb300.models import (AstigmaticXYZNB, GaussianXYNB, GaussianXYNBS,
                                   GaussianXYNBSXSY)

SMS = 152


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    build.build(force=not build.BUILD_DIR.exists())
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    objs = [str(build.BUILD_DIR / (u[1] + ".o")) for u in build.UNITS]
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{cuda}", "-o", str(out),
                    str(ROOT / "tests" / "fake" / "fake_cuda.cpp"), *objs, "-Wl,-Bsymbolic",
                    "-lpthread"], check=True)
    lib = C.CDLL(str(out))
    lib.fake_log.restype = C.c_char_p
    lib.gmle_last_error.restype = C.c_char_p
    yield lib
    out.unlink()


@pytest.fixture
def ctx(lib):
    lib.fake_host_pages(0)
    lib.fake_fail(b"", 0)
    c = C.c_void_p()
    assert lib.gmle_create(C.byref(c), 0) == 0
    yield c
    lib.fake_fail(b"", 0)
    lib.gmle_destroy(c)


def calls(lib, name):
    """(stream, *numbers) of every logged call of `name`."""
    rows = (r.split() for r in lib.fake_log().decode().splitlines())
    return [tuple(int(v) for v in r[1:]) for r in rows if r[0] == name]


def p(a):
    return a.ctypes.data_as(C.c_void_p) if a is not None else None


BOX = 3
CHUNK = (64 << 20) // (4 * BOX * BOX)  # gmle_fit's chunk, 64 MiB of pixels


def desc(box=BOX):
    psf = GaussianXYNB(1.3)
    return make_desc(psf, box, 20, default_constraints(psf, box), 0)


def host_fit(lib, ctx, data, n, fill=7.0):
    out = [np.full((n, 4), fill, np.float32), np.full((n, 4), fill, np.float32),
           np.full(n, fill, np.float32), np.full(n, int(fill), np.uint8)]
    return lib.gmle_fit(ctx, C.byref(desc()), p(data), None, None, C.c_int64(n),
                        *map(p, out)), out


@pytest.mark.parametrize("host_pages", [0, 1])
@pytest.mark.parametrize("name,nth", [("cudaMemcpyAsync", 6), ("launch", 3), ("cudaEventRecord", 9)])
def test_a_failed_fit_leaves_nothing_behind(lib, ctx, host_pages, name, nth):
    """Three chunks, an error in the second or third: every stream has run dry before
    the call returns, and the next call writes to its own buffers only."""
    lib.gmle_destroy(ctx)
    lib.fake_host_pages(host_pages)
    assert lib.gmle_create(C.byref(ctx), 0) == 0
    data = np.zeros((2 * CHUNK + 10, BOX * BOX), np.float32)
    lib.fake_clear()
    lib.fake_fail(name.encode(), nth)
    st, out = host_fit(lib, ctx, data, len(data))
    assert st != 0 and b"fake error" in lib.gmle_last_error(ctx)
    log = lib.fake_log().decode().splitlines()
    used = {r.split()[1] for r in log if r.startswith(("cudaMemcpyAsync", "launch"))}
    last = max(k for k, r in enumerate(log) if r.startswith(("cudaMemcpyAsync", "launch",
                                                             "cudaEventRecord")))
    waited = {r.split()[1] for r in log[last:] if r.startswith("cudaStreamSynchronize")}
    assert len(used) >= 2 and used <= waited
    before = [o.copy() for o in out]
    st, _ = host_fit(lib, ctx, data[:100], 100)
    assert st == 0
    for a, b in zip(before, out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("name", ["cudaMalloc", "cudaEventCreateWithFlags", "cudaMemcpyAsync"])
def test_a_fit_that_fails_before_its_results_leaves_the_outputs_alone(lib, ctx, name):
    """Where the GPU takes pageable memory as it is, its pages are mapped by the host
    first: without a change to the outputs, which hold the caller's values until results
    come."""
    lib.gmle_destroy(ctx)
    lib.fake_host_pages(1)
    assert lib.gmle_create(C.byref(ctx), 0) == 0
    data = np.zeros((40_000, BOX * BOX), np.float32)
    lib.fake_fail(name.encode(), 1)
    st, out = host_fit(lib, ctx, data, len(data))
    assert st != 0
    for o in out:
        assert (o == 7).all()
    st, out = host_fit(lib, ctx, data, len(data))
    assert st == 0 and (out[0] == 0).all()  # (the fake's results: zeros)


def test_inputs_that_are_not_resident(lib, ctx, tmp_path):
    """A read-only file mapping as input, as raw movies often are."""
    lib.gmle_destroy(ctx)
    lib.fake_host_pages(1)
    assert lib.gmle_create(C.byref(ctx), 0) == 0
    np.zeros((3000, BOX * BOX), np.float32).tofile(tmp_path / "rois.bin")
    m = np.memmap(tmp_path / "rois.bin", np.float32, "r", shape=(3000, BOX * BOX))
    st, out = host_fit(lib, ctx, m, len(m))
    assert st == 0 and (out[0] == 0).all()


PSF = {0: GaussianXYNB(1.3), 1: GaussianXYNBS(), 2: GaussianXYNBSXSY(),
       3: AstigmaticXYZNB(1.3, 1.3, 0.05, 0.05, 0.3, 0.3, 50.0, 100.0)}


def groups(kinds):
    """gmle_group array of (model, box, n); the fake's kernels read and write nothing."""
    some = np.zeros(1, np.float32)
    gs = []
    for model, box, n in kinds:
        g = serve.make_group(PSF[model], box, 0, default_constraints(PSF[model], box), some, some,
                             some, np.empty((n, 6), np.float32), some, some)
        gs.append(g)
    return (_lib.Group * len(gs))(*gs)


@pytest.mark.parametrize("kinds", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("large", [0, 1])
def test_the_launches_of_a_submission_take_every_stream(lib, ctx, kinds, large):
    """One launch per kind (a group of 65536 ROIs or more: its own), each on a stream of
    its own up to four; a single launch on the caller's."""
    gs = groups([(k % 4, 7 + k, 70_000 if k < large else 500) for k in range(kinds)])
    lib.fake_clear()
    assert lib.gmle_fit_mixed_device(ctx, gs, len(gs), C.c_void_p(999)) == 0
    streams = [c[0] for c in calls(lib, "launch")]
    assert len(streams) == kinds
    assert len(set(streams)) == min(kinds, 4)
    assert (streams == [999]) if kinds == 1 else (999 not in streams)


@pytest.mark.parametrize("n,threads,grid", [
    (300, 128, 10),          # four lanes, 32 ROIs per block
    (5_000, 128, 157),
    (100_000, 64, 4 * SMS),  # one thread, as many blocks as are resident (the fake's four per SM)
])
def test_the_launches_without_allocation_go_by_their_own_kinds_rois(lib, n, threads, grid):
    """gmle_fit_mixed_device_noalloc's launches run one after another, so that a kind's
    shape does not depend on how much else the call holds."""
    err = C.create_string_buffer(256)
    for others in ([(1, 9, 200_000)], [(1, 9, 3_000)]):
        shape = noalloc_shapes(lib, err, [(0, 11, n)] + others)[0]
        assert shape == (grid, threads)


def noalloc_shapes(lib, err, kinds):
    gs = groups(kinds)
    lib.fake_clear()
    assert lib.gmle_fit_mixed_device_noalloc(gs, len(gs), None, None, None, 0, 0,
                                             C.c_void_p(999), err, 256) == 0, err.value
    fits = [c for c in calls(lib, "launch") if c[1:3] != (1, 256)]  # (without the table writes)
    assert len(fits) == len(gs) and all(c[0] == 999 for c in fits)
    return [c[1:3] for c in fits]


@pytest.mark.parametrize("other,lanes", [(2_739, 32), (2_740, 4), (29_000, 4)])
def test_small_kinds_take_the_lanes_of_the_entry_point_with_a_context(lib, ctx, other, lanes):
    """A warp per ROI for all of a call below 20 ROIs per SM, else four lanes: as in
    gmle_fit_mixed_device, so that the two give the same bits."""
    kinds = [(0, 11, 300), (3, 15, other)]
    mine = noalloc_shapes(lib, C.create_string_buffer(256), kinds)[0]
    lib.fake_clear()
    gs = groups(kinds)
    assert lib.gmle_fit_mixed_device(ctx, gs, len(gs), C.c_void_p(999)) == 0
    theirs = [c[1:3] for c in calls(lib, "launch")]
    if lanes == 4:
        assert mine == (10, 128) and mine in theirs
    else:
        assert mine == (300, 32) and all(t <= 128 for _, t in theirs)


def get_tuning(lib, ctx, model, box, camera):
    t, r = C.c_int32(), C.c_int32()
    assert lib.gmle_get_tuning(ctx, model, box, camera, C.byref(t), C.byref(r)) == 0
    return t.value, r.value


def test_every_launch_shape_that_is_answered_can_be_set(lib, ctx):
    """A program that saves the shapes and sets them again: for every specialised box,
    and back to the default."""
    for model in range(4):
        for camera in range(3):
            for box in range(3, 17):
                shape = get_tuning(lib, ctx, model, box, camera)
                assert lib.gmle_set_tuning(ctx, model, box, camera, *shape) == 0, (
                    model, box, camera, shape, lib.gmle_last_error(ctx))
                assert get_tuning(lib, ctx, model, box, camera) == shape
                assert lib.gmle_set_tuning(ctx, model, box, camera, 0, 0) == 0


@pytest.mark.parametrize("box,camera,most", [(16, 1, 224), (16, 2, 224), (16, 0, 128), (15, 1, 128),
                                             (11, 2, 128)])
def test_one_thread_blocks_end_where_the_kernel_does(lib, ctx, box, camera, most):
    assert lib.gmle_set_tuning(ctx, 0, box, camera, 1, most) == 0
    assert lib.gmle_set_tuning(ctx, 0, box, camera, 1, most + 32) == 1
    assert str(most).encode() in lib.gmle_last_error(ctx)


@pytest.mark.parametrize("box", [17, 21, 33, 64])
def test_large_boxes_answer_the_shape_they_run_in(lib, ctx, box):
    n, some = 3000, np.zeros(1, np.float32)
    lib.fake_clear()
    assert lib.gmle_fit_device(ctx, C.byref(desc(box)), p(some), None, None, C.c_int64(n), p(some),
                               p(some), p(some), None, C.c_void_p(7)) == 0
    _, grid, threads, _ = calls(lib, "launch")[0]
    tpr, rpb = get_tuning(lib, ctx, 0, box, 0)
    assert tpr == 32 and threads == 32 * rpb and grid == -(-n // rpb)


def autotune(lib, ctx, box, camera, n, grid, threads):
    """Autotune where the launch of that grid and block is the fastest; (shape, kept)."""
    some, d = np.ones(4, np.float32), desc(box)
    d.camera = camera
    lib.fake_fastest(grid, threads)
    t, r, ms = C.c_int32(), C.c_int32(), C.c_float()
    if camera:
        assert lib.gmle_set_calibration(ctx, p(np.ones((64, 64), np.float32)), None, None, 64, 64) == 0
    st = lib.gmle_autotune(ctx, C.byref(d), p(some), p(some), p(some), C.c_int64(n), p(some), p(some),
                           p(some), None, C.byref(t), C.byref(r), C.byref(ms))
    assert st == 0, lib.gmle_last_error(ctx)
    lib.fake_clear()
    assert lib.gmle_fit_device(ctx, C.byref(d), p(some), p(some), p(some), C.c_int64(n), p(some),
                               p(some), p(some), None, C.c_void_p(7)) == 0
    _, g, b, _ = calls(lib, "launch")[0]
    return (t.value, r.value, ms.value), (g, b)


@pytest.mark.parametrize("box,camera,n,grid,threads,tpr", [
    (11, 0, 200, 200, 32, 32),        # a warp per ROI, the default of 200 ROIs
    (11, 0, 200, 25, 32, 4),          # another shape, where it is faster
    (16, 1, 100_000, 447, 224, 1),    # the blocks of large 16x16 sCMOS batches
    (16, 1, 100_000, 1042, 96, 1),
    (16, 0, 100_000, 1563, 64, 1)])
def test_autotune_times_the_default_shape_too(lib, ctx, box, camera, n, grid, threads, tpr):
    """The shape that a batch runs in afterwards is the fastest, also where that is the
    shape it would have had anyway."""
    (t, r, ms), ran = autotune(lib, ctx, box, camera, n, grid, threads)
    assert (t, t * r, ms) == (tpr, threads, 1.0) and ran == (grid, threads)
    if t == 32:  # not kept for the larger batches of the kind
        assert get_tuning(lib, ctx, 0, box, camera)[0] == 1
    else:
        assert get_tuning(lib, ctx, 0, box, camera) == (t, r)


def test_autotune_saves_no_shape_of_the_smallest_batches(tmp_path, monkeypatch):
    import json
    from gaussmle_gb300 import tuning
    monkeypatch.setattr(tuning, "CACHE", tmp_path / "tuning.json")
    monkeypatch.setattr(tuning, "_gpu_name", lambda device: "GB300")

    class Tensor:
        shape = (200, 4)

        def data_ptr(self):
            return 0

    class Ctx:
        handle, device, lib, shape = None, 0, None, None

        def gmle_autotune(self, *a):
            for q, v in zip(a[-3:], self.shape + (0.1,)):
                q._obj.value = v
            return 0

        def check(self, st):
            assert st == 0

    ctx, x = Ctx(), Tensor()
    ctx.lib = ctx
    for ctx.shape, want in [((1, 64), {"0/11/0": [1, 64]}), ((32, 1), {}), ((32, 4), {})]:
        assert tuning.autotune(ctx, desc(11), x, None, None, x, x, x)[:2] == ctx.shape
        assert json.loads(tuning.CACHE.read_text())["GB300"] == want
