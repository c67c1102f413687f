"""What a program sees around the solves that run whole levels in one launch: streams, captures, masks,
first solves, errors, and the buffers that the default path leaves."""
import ctypes
import subprocess
import threading

import numpy as np
import pytest

from tests.helpers import params, random_case

pytestmark = pytest.mark.gpu


def _solver(case, p, stream=None, fused=False, half=False):
    from vfs_b200.stereotgv import StereoTgv
    i0, i1, mask, tv, cv = case
    s = StereoTgv()
    s.set_solve_path(fused, half)
    h, w = i0.shape
    s.limitRange = p["limit_range"]
    s.initialize(w, h, p["beta"], p["gamma"], p["alpha0"], p["alpha1"], p["tsl"], p["lam"], p["n_levels"],
                 p["f_scale"], p["n_warp"], p["n_iter"])
    s.copyMaskToDevice(mask)
    s.loadVectorFields(tv, cv)
    if stream is not None:
        s.set_stream(stream)
    return s


def _disparity(s, case, masked=True):
    s.copyImagesToDevice(*case[:2])
    (s.solveStereoForwardMasked if masked else s.solveStereoForward)()
    return s.copy1DDisparityToHost()


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
def test_first_unmasked_solve_in_a_capture(gpu, half):
    """A handle that has only solved with its mask: its first unmasked solve goes into a caller's graph,
    and what it solves afterwards without one is right."""
    import torch
    case = random_case(150, 110, seed=7)
    p = params(n_levels=2, n_warp=2, n_iter=6)
    want = _disparity(_solver(case, p, fused=True, half=half), case, masked=False)
    assert want.any()
    st = torch.cuda.Stream()
    s = _solver(case, p, st, fused=True, half=half)
    s.set_graph(False)
    for _ in range(2):
        _disparity(s, case)
    i0, i1 = (torch.from_numpy(x).cuda() for x in case[:2])
    out = torch.zeros((110, 150), device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
            s.copy_images_from_device(i0, i1)
            s.solveStereoForward()
            s.copy_1d_disparity_to_device(out)
        captured = True
    except Exception:
        captured = False
        torch.cuda.synchronize()
    if captured:
        g.replay()
        torch.cuda.synchronize()
    assert np.array_equal(_disparity(s, case, masked=False), want)
    assert captured and np.array_equal(out.cpu().numpy(), want)


def test_circle_on_the_host(gpu, tmp_path):
    """The unmasked form's circle as the host finds it, row by row, and as the kernels evaluate it."""
    from vfs_b200.build import CSRC, NVCC_FLAGS, nvcc
    src = tmp_path / "t.cu"
    src.write_text(r"""
#include <cstdio>
#include "resident.cuh"
#include "tgv_pixel.cuh"
namespace vfs { int res_capacity(bool, bool, int, int) { return 0; } }
using namespace vfs;
__global__ void k_codes(uint8_t* c, int w, int h) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x < w) c[x + (size_t)y * w] = outside_circle(x, y, w, h) ? 0 : kOn;
}
int main() {
  uint8_t* d;
  if (cudaMalloc(&d, 1500 * 1500) != cudaSuccess) return 2;
  int bad = 0, n = 0;
  auto check = [&](int w, int h) {
    std::vector<uint8_t> dev((size_t)w * h);
    k_codes<<<dim3((w + 127) / 128, h), 128>>>(d, w, h);
    if (cudaMemcpy(dev.data(), d, dev.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    n++;
    if (dev != res_circle_codes(w, h)) std::printf("%d x %d\n", w, h), bad++;
    return true;
  };
  for (int w = 1; w < 70; w++)
    for (int h = 1; h < 70; h += 1 + w % 3)
      if (!check(w, h)) return 2;
  unsigned s = 1;
  for (int k = 0; k < 120; k++) {
    s = s * 1664525u + 1013904223u;
    if (!check(70 + (s >> 8) % 1400, 70 + (s >> 20) % 1400)) return 2;
  }
  std::printf("%d sizes\n", n);
  return bad != 0;
}
""")
    exe = tmp_path / "t"
    r = subprocess.run([nvcc(), *NVCC_FLAGS, f"-I{CSRC}", str(src), f"{CSRC}/resident_plan.cu", "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("fused,half", [(False, False), (True, False), (True, True)], ids=["dropin", "fp32", "fp16"])
@pytest.mark.parametrize("size", [(150, 110), (640, 480)])
def test_solves_return_after_enqueueing(gpu, size, fused, half):
    """Behind work that keeps the stream busy for some 0.3 s: the first solve with a mask, the first
    unmasked one and the first with another mask.  (A first handle loads the kernels.)"""
    import torch
    w, h = size
    case = random_case(w, h, seed=9)
    p = params(n_levels=3, n_warp=2, n_iter=8)
    i0, i1 = (torch.from_numpy(x).cuda() for x in case[:2])
    for warm in (True, False):
        st = torch.cuda.Stream()
        s = _solver(case, p, st, fused=fused, half=half)
        for masked, mask in ((True, None), (False, None), (True, np.ascontiguousarray(case[2][:, ::-1]) * (case[0] > 60))):
            if mask is not None:
                s.copyMaskToDevice(mask)
            s.copy_images_from_device(i0, i1)
            torch.cuda.synchronize()
            before = torch.cuda.Event()
            with torch.cuda.stream(st):
                if not warm:
                    torch.cuda._sleep(600_000_000)
                before.record()
            (s.solveStereoForwardMasked if masked else s.solveStereoForward)()
            waited = before.query()
            torch.cuda.synchronize()
            assert warm or not waited, (masked, mask is not None)


@pytest.mark.parametrize("fused", [False, True], ids=["dropin", "fp32"])
def test_plans_that_cannot_be_made(gpu, fused):
    """Device memory runs out at each step of a form's tile plans (one a level; the second form's own
    memory): the solve runs one iteration a launch, and the next mask has its plans."""
    from vfs_b200._native import lib
    from vfs_b200.stereotgv import StereoTgv
    case = random_case(150, 110, seed=31)
    p = params(n_levels=3, n_warp=1, n_iter=100)
    want = {m: _disparity(_solver(case, p), case, masked=m) for m in (True, False)}

    def launches(s, masked):
        n = StereoTgv.launch_count()
        assert np.array_equal(_disparity(s, case, masked), want[masked])
        return StereoTgv.launch_count() - n

    for failing in (1, 2, 3):
        s = _solver(case, p, fused=fused)
        s.set_autotune(False)
        assert lib().vfs_debug_fail_allocation(failing + (1 if fused else 0)) == 0  # the fused buffers come first
        assert launches(s, True) > 300
        assert launches(s, True) > 300
        s.copyMaskToDevice(case[2])
        assert launches(s, True) < 100
    assert lib().vfs_debug_fail_allocation(4) == 0  # the unmasked form's plans beside the masked form's
    assert launches(s, False) > 300 and launches(s, False) > 300
    assert launches(s, True) < 100
    assert lib().vfs_debug_fail_allocation(0) == 0
    assert s.check_guards() == 0


@pytest.mark.parametrize("stream", [1, 2], ids=["legacy", "per-thread"])
def test_default_path_on_the_default_streams(gpu, stream):
    """cudaStreamLegacy and cudaStreamPerThread as the handle's stream: the first cannot be captured."""
    case = random_case(150, 110, seed=17)
    p = params(n_levels=2, n_warp=2, n_iter=20)
    for masked in (True, False):
        want = _disparity(_solver(case, p), case, masked)
        s = _solver(case, p, stream)
        for _ in range(8):
            assert np.array_equal(_disparity(s, case, masked), want)


def test_default_path_beside_work_on_the_legacy_stream(gpu):
    """The handle on a stream that synchronises with the legacy default stream, on which another
    thread keeps working: both go on undisturbed."""
    import torch
    rt = ctypes.CDLL("libcudart.so.12")
    st = ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(st)) == 0
    case = random_case(150, 110, seed=19)
    p = params(n_levels=3, n_warp=2, n_iter=20)
    want = _disparity(_solver(case, p), case)
    s = _solver(case, p, st.value)
    x = torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    stop, errors, calls = threading.Event(), [], [0]

    def work():
        while not stop.is_set():
            e = rt.cudaMemsetAsync(ctypes.c_void_p(x.data_ptr()), 0, ctypes.c_size_t(4096), ctypes.c_void_p(1))
            if e:
                errors.append(e)
            calls[0] += 1
            if calls[0] % 64 == 0:
                rt.cudaStreamSynchronize(ctypes.c_void_p(1))

    t = threading.Thread(target=work)
    t.start()
    try:
        for k in range(12):
            s.copyMaskToDevice(case[2])  # the graphs of the last mask go
            for _ in range(5):
                assert np.array_equal(_disparity(s, case), want)
    finally:
        stop.set()
        t.join()
        s.close()
        rt.cudaStreamDestroy(st)
    assert not errors, errors[:3]
    assert calls[0] > 100


def test_states_that_come_once(gpu):
    """A new mask or limit for every frame: nothing is recorded that is not replayed, and a short solve
    makes its plans only when its mask comes a second time."""
    from vfs_b200._native import lib
    from vfs_b200.stereotgv import StereoTgv
    case = random_case(150, 110, seed=41)
    other = np.ascontiguousarray(case[2][:, ::-1])

    def pair(p):  # and the same frames through the one-iteration kernels
        s, t = _solver(case, p), _solver(case, p, fused=True)
        t.set_iteration_variant(1)
        return s, t

    def frame(st, mask=None, limit=None):
        u = []
        for s in st:
            if mask is not None:
                s.copyMaskToDevice(mask)
            if limit is not None:
                s.limitRange = limit
            n = StereoTgv.launch_count()
            u.append(_disparity(s, case))
            if s is st[0]:
                launches = StereoTgv.launch_count() - n
        assert np.array_equal(*u)
        return launches

    short, usual = params(n_levels=2, n_warp=1, n_iter=5), params(n_levels=2, n_warp=1, n_iter=6)
    st = pair(short)
    per_operation = frame(st)
    assert frame(st) < per_operation  # the mask's second solve
    for mask in (other, case[2]):
        assert frame(st, mask) == per_operation
    st = pair(usual)
    for k in range(6):
        assert frame(st, case[2], 0.1 + 0.01 * k) < per_operation
    assert lib().vfs_cached_graphs(st[0].handle) == 0
    for k in range(2):  # the two states that the solves alternate between
        frame(st)
    graphs = lib().vfs_cached_graphs(st[0].handle)
    assert graphs == 2
    for k in range(4):
        frame(st)
    assert lib().vfs_cached_graphs(st[0].handle) == graphs


@pytest.fixture
def muted(gpu):
    """Whole-level launches leave out a tile's first values: its neighbours' waits run out."""
    from vfs_b200._native import lib
    st = ctypes.c_int()
    lib().vfs_device_status(ctypes.byref(st))
    assert lib().vfs_debug_mute_tile(1) == 0
    yield lib()
    assert lib().vfs_debug_mute_tile(0) == 0
    lib().vfs_device_status(ctypes.byref(st))


# in one cluster and on the whole GPU
@pytest.mark.parametrize("size", [(60, 50), (300, 280)])
@pytest.mark.parametrize("fused,half", [(False, False), (True, True)], ids=["dropin", "fp16"])
def test_a_wait_that_runs_out_is_an_error(muted, size, fused, half):
    from vfs_b200._native import VfsError
    w, h = size
    case = random_case(w, h, seed=w)
    p = params(n_levels=1, n_warp=1, n_iter=40)
    s = _solver(case, p, fused=fused, half=half)
    s.check_solve()
    for call in (lambda: _disparity(s, case), s.copyDisparityToHost, s.synchronize, s.check_solve):
        with pytest.raises(VfsError) as e:  # the solve's copy, and every later question
            call()
        assert e.value.status == -6
    st = ctypes.c_int()
    assert muted.vfs_device_status(ctypes.byref(st)) == 0 and st.value == 1
    muted.vfs_debug_mute_tile(0)
    want = _disparity(_solver(case, p, fused=fused, half=half), case)
    s.copyMaskToDevice(case[2])  # (recorded launches stay muted)
    got = _disparity(s, case)
    from scipy.ndimage import binary_erosion
    on = binary_erosion(case[2] > 0, iterations=4)  # beyond the median's reach of masked-out pixels, which keep theirs
    assert on.any() and np.array_equal(got[on], want[on])
    s.check_solve()
    assert s.check_guards() == 0


def test_a_wait_that_runs_out_in_a_batch_and_a_server(muted):
    from vfs_b200._native import VfsError
    from vfs_b200.serving import StereoServer
    from vfs_b200.stereotgv import StereoBatch
    cases = [random_case(160, 120, seed=k) for k in range(2)]
    p = params(n_levels=1, n_warp=1, n_iter=40)
    b = StereoBatch(half_storage=True)
    for c in cases:
        b.add(_solver(c, p, fused=True, half=True))
    with pytest.raises(VfsError) as e:
        b.solve_host([c[:2] for c in cases])
    assert e.value.status == -6 and "pair 0" in str(e.value)
    for m in b.members:
        with pytest.raises(VfsError):
            m.check_solve()
    srv = StereoServer(lanes=1)
    srv.open_stream(0, 160, 120, cases[0][2], cases[0][3], cases[0][4], 1, dict(nWarpIters=1))
    bad = srv.submit(0, *cases[0][:2])
    srv.run_until_idle()
    assert bad.u is None and "-6" in bad.error and srv.stats()["failed"] == 1


def test_default_path_after_a_device_reset(gpu):
    """A program that resets the device between two handles (in a process of its own)."""
    import os
    import sys
    code = """
import ctypes, gc
import numpy as np
from tests.helpers import params, random_case, run_gpu
case, p = random_case(150, 110, seed=3), params(n_levels=2, n_warp=2, n_iter=20)
want = run_gpu(*case, p).copy1DDisparityToHost()
gc.collect()
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
for _ in range(2):
    assert np.array_equal(run_gpu(*case, p).copy1DDisparityToHost(), want)
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


# The form a level takes: 30-column tiles of the least rows that leave them at most 2,368 (two rows: three
# quarters of that), one cluster up to 208 tiles of two rows with half storage and 128 with float
@pytest.mark.parametrize("half,w,h,rows,cluster", [
    (True, 118, 104, 2, True), (True, 119, 106, 2, False), (False, 115, 64, 2, True), (False, 118, 66, 2, False),
    (True, 640, 100, 2, False), (False, 424, 400, 4, False), (True, 600, 520, 6, False), (False, 760, 480, 6, False),
    (True, 830, 560, 8, False), (False, 850, 560, 8, False), (True, 810, 760, 12, False), (True, 1078, 1009, 16, False),
    (False, 850, 760, 0, False), (True, 1200, 1100, 0, False)])
def test_the_form_of_a_level_and_pinning_it(gpu, half, w, h, rows, cluster):
    case = list(random_case(w, h, seed=w + h, circle=False))
    case[2][0] = case[2][:, 0] = 0
    p = params(n_levels=1, n_warp=1, n_iter=6)
    tiles = -(-w // 30) * -(-h // rows) if rows else 0
    want = [(rows, tiles, cluster)]
    s = _solver(case, p, fused=True, half=half)
    s.set_autotune(False)
    u = _disparity(s, case)
    assert s.level_launches() == want
    assert s.iteration_variants() == [14 if rows else 1]
    t = _solver(case, p, fused=True, half=half)
    t.set_iteration_variants(s.iteration_variants())  # pinned from the report
    assert np.array_equal(_disparity(t, case), u)
    assert t.level_launches() == want and t.iteration_variants() == s.iteration_variants()
    t.set_iteration_variants([])
    t.set_iteration_variant(14 if rows == 2 else 1)  # another kernel, the same bits
    t.copyMaskToDevice(case[2])
    f = _solver(case, p, fused=True, half=half)
    f.set_iteration_variant(1)
    assert np.array_equal(_disparity(f, case), u)
    _disparity(t, case)
    assert t.level_launches() == [(0, 0, False)] == f.level_launches()
    if not half:
        d = _solver(case, p)
        assert np.array_equal(_disparity(d, case), u)
        assert d.level_launches() == want


def test_exported_state_holds_the_edge_codes(gpu):
    """Where the fused buffers held them: a library that reads them from a state finds those of the
    mask and of the circle, level after level, with their guard zones."""
    w, h = 150, 110
    case = random_case(w, h, seed=61)
    s = _solver(case, params(n_levels=2, n_warp=1, n_iter=6), fused=True)
    _disparity(s, case)
    state = s.export_state()
    sizes = s.level_sizes()
    n = sizes[0][1] * sizes[0][2]

    def place(at, b):
        at = -(-at // 512) * 512
        return at, at + b + 256

    at = 0
    for b in (16 * n, 32 * n, 4 * n, 4 * n, 16 * n, 8 * n):  # the planes before them
        _, at = place(at, b)
    pool = int.from_bytes(state[48:56].tobytes(), "little")
    f = state[160 + pool:]
    for l, (lw, lh, ls) in enumerate(sizes):
        for masked in (True, False):
            lo, at = place(at, ls * lh)
            on = f[lo:lo + ls * lh].reshape(lh, ls)[:, :lw] & 1
            assert (f[lo + ls * lh:at] == 0xA5).all()
            yy, xx = np.mgrid[0:lh, 0:lw].astype(np.float32)
            r = np.sqrt((yy - np.float32(lh) / 2) ** 2 + (xx - np.float32(lw) / 2) ** 2)
            if not masked:
                assert np.array_equal(on, r < np.float32(lw) / np.float32(2.2))
            elif l == 0:
                assert np.array_equal(on, case[2] > 0)
    t = _solver(case, params(n_levels=2, n_warp=1, n_iter=6), fused=True)
    t.import_state(state)
    assert np.array_equal(_disparity(t, case, False), _disparity(s, case, False))


BUFFERS = (("u", 1), ("u_", 1), ("warpUV", 2), ("a", 1), ("b", 1), ("c", 1), ("etau", 1), ("etav1", 1), ("etav2", 1),
           ("Iu", 1), ("Iz", 1), ("i1warp", 1), ("tv2", 2), ("i0smooth", 1), ("p", 2), ("q", 4), ("v_", 2), ("Tp", 2),
           ("us", 1), ("u_s", 1), ("v_s", 2), ("du", 1), ("u_last", 1), ("warpUVs", 2), ("i1calibrated", 1))


@pytest.mark.parametrize("masked", [True, False], ids=["masked", "plain"])
@pytest.mark.parametrize("w,h,levels,warps,iters,kw", [
    (64, 48, 2, 1, 2, {}), (64, 48, 2, 2, 5, {}), (64, 48, 2, 0, 3, {}), (97, 53, 2, 2, 3, {}), (53, 97, 2, 2, 4, {}),
    (130, 60, 1, 1, 6, dict(alpha0=0.0)), (300, 280, 3, 2, 7, {}), (640, 480, 4, 1, 9, {})])
def test_default_path_leaves_every_buffer_as_a_kernel_per_operation_does(gpu, w, h, levels, warps, iters, kw, masked):
    """The same frames on two handles, the last ones of the second in a caller's capture, where the
    default path takes a kernel per operation: every buffer's bits, over a new mask in between."""
    import torch
    case = random_case(w, h, seed=w + h, circle=w != 64)
    case[2][0] = case[2][:, 0] = 0
    new = case[2].copy()
    new[h // 3:h // 2, w // 4:w // 2] = 0
    p = params(n_levels=levels, n_warp=warps, n_iter=iters, **kw)
    i0, i1 = (torch.from_numpy(x).cuda() for x in case[:2])
    out = []
    for captured in (False, True):
        st = torch.cuda.Stream()
        s = _solver(case, p, st)
        solve = s.solveStereoForwardMasked if masked else s.solveStereoForward
        frames = []
        for k in range(10):  # the first eight make the texture objects of every pointer state
            if k == 9:
                s.copyMaskToDevice(new)
            s.copy_images_from_device(i0, i1)
            torch.cuda.synchronize()
            if captured and k >= 8:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=st):
                    solve()
                assert not any(r for r, _, _ in s.level_launches())
                g.replay()
            else:
                solve()
                assert k < 6 or warps == 0 or k == 9 or all(r for r, _, _ in s.level_launches())
            torch.cuda.synchronize()
            if k >= 8:
                frames.append({n: s.debug_buffer(n, c) for n, c in BUFFERS})
        out.append(frames)
    for a, b in zip(*out):
        for n, _ in BUFFERS:
            assert np.array_equal(a[n], b[n], equal_nan=True), n
            assert np.array_equal(np.signbit(a[n]), np.signbit(b[n])), n


def test_fused_solve_in_a_captured_stream(gpu):
    """With the handle's own graphs off its launches go into the caller's graph, one iteration a launch;
    with them on the capture is refused, and the handle solves as before."""
    import torch
    from vfs_b200._native import VfsError
    case = random_case(150, 110, seed=23)
    p = params(n_levels=2, n_warp=2, n_iter=8)
    want = _disparity(_solver(case, p, fused=True, half=True), case)
    i0, i1 = (torch.from_numpy(x).cuda() for x in case[:2])
    st = torch.cuda.Stream()
    s = _solver(case, p, st, fused=True, half=True)
    out = torch.zeros((110, 150), device="cuda")

    def frame():
        s.copy_images_from_device(i0, i1)
        s.solveStereoForwardMasked()
        s.copy_1d_disparity_to_device(out)

    for _ in range(2):
        frame()
    torch.cuda.synchronize()
    with pytest.raises((VfsError, RuntimeError)):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=st, capture_error_mode="relaxed"):
            frame()
    torch.cuda.synchronize()
    assert np.array_equal(_disparity(s, case), want)
    assert all(r for r, _, _ in s.level_launches())
    s.set_graph(False)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
        frame()
    assert not any(r for r, _, _ in s.level_launches())
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(_disparity(s, case), want)


def _spreading_case(w, h, rows, seed):
    """Two equal images but for a strip near an end of the longer side: the disparity spreads from there by
    a pixel an iteration, each time smaller, down to zero.  rows: the images differ in the upper half too,
    alike in every column, so that a large vertical step stands beside the horizontal one that spreads."""
    rng = np.random.default_rng(seed)
    i0 = rng.uniform(0.2, 0.8, (h, w)).astype(np.float32)
    tv = np.zeros((h, w, 2), np.float32)
    tv[..., 0] = -1.0
    if rows:
        i0[:] = np.linspace(0.1, 0.9, h, dtype=np.float32)[:, None] ** 2
        tv[:] = (0.0, 1.0)
    i1 = i0.copy()
    if rows:
        i1[:h // 2] += np.float32(0.3)
    if w >= h:
        i1[2:h - 2, w // 8:w // 8 + 4] += np.float32(0.2)
    else:
        i1[h // 8:h // 8 + 4, 2:w - 2] += np.float32(0.2)
    mask = np.ones((h, w), np.float32)
    mask[0] = mask[:, 0] = 0
    return i0, i1, mask, tv, np.zeros((h, w, 2), np.float32)


# (30 x 240: in one cluster; the unmasked form's circle is too small for the values to shrink there)
@pytest.mark.parametrize("w,h,rows,masked", [(30, 240, False, True)] + [
    (w, h, rows, masked) for w, h in ((160, 160), (500, 400), (848, 640)) for rows in (False, True)
    for masked in (True, False)])
def test_values_down_to_the_smallest(gpu, w, h, rows, masked):
    """Disparities and dual variables that shrink to subnormal numbers, some beside a norm above 1: their
    quotients are the plain division's too."""
    case = _spreading_case(w, h, rows, w)
    p = params(n_levels=1, n_warp=2, n_iter=60, alpha0=1.0, lam=50.0)
    out = []
    for variant in (1, None):
        s = _solver(case, p, fused=True)
        if variant is not None:
            s.set_iteration_variant(variant)
        _disparity(s, case, masked)
        out.append({n: s.debug_buffer(n, c) for n, c in (("u", 1), ("u_", 1), ("us", 1), ("u_s", 1), ("v_", 2),
                                                         ("v_s", 2), ("Tp", 2))})
    assert s.level_launches()[0][0] > 0
    a = np.abs(out[0]["us"])
    assert ((a > 0) & (a < 2.0 ** -102)).any() and ((a > 0) & (a < 2.0 ** -126)).any()
    for n in out[0]:
        same = out[0][n].view(np.int32) == out[1][n].view(np.int32)
        assert same.all(), (n, int((~same).sum()), same.size)


def test_exact_quotients_of_any_dividend(gpu, tmp_path):
    """10^9 quotients by divisors from 2^-64 to 2^64, dividends from the smallest subnormal on (half of
    them below 2^-100), against the device's division.  Left out, as the header says: quotients exactly
    halfway between two subnormals, which take an integer divisor (a few in 10^9 here), and the sign of
    a zero divided by a negative number."""
    from vfs_b200.build import ARCH, CSRC, nvcc
    src = tmp_path / "t.cu"
    src.write_text(r"""
#include <cstdio>
#include "tgv_exact_pairs.cuh"
using namespace vfs;
namespace x2 = fast::x2;
__device__ unsigned long long bad, tiny, halfway;
__global__ void k_quot(int n) {
  unsigned long long s = 0x9E3779B97F4A7C15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
  for (int i = 0; i < n; i++) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    // exponents of b - 127: 0 .. 15 (as a norm's), or -64 .. 63; of a: 0 .. 31, or 0 .. 191
    const unsigned eb = (s >> 40) & 1 ? 127 + ((s >> 41) & 15) : 63 + ((s >> 41) & 127);
    const unsigned ea = (s >> 48) & 1 ? (s >> 49) & 31 : ((s >> 49) % 192);
    const float a = __uint_as_float((unsigned)(s >> 63) << 31 | ea << 23 | ((unsigned)s & 0x7fffff));
    const float b = __uint_as_float(eb << 23 | (unsigned)((s * 0xD1342543DE82EF95ull) >> 41));
    const float q = a / b;
    if (!(fabsf(q) <= 0x1p120f)) continue;
    const x2::f2 B = x2::pk(b, -b), Q = exact::quot(x2::pk(a, a), exact::Divisor(B, exact::recip(B)));
    if (fabsf(q) <= 0x1p-126f && fmod(fabs((double)a / (double)b) * 0x1p150, 2.0) == 1.0) {
      atomicAdd(&halfway, 1ull);
      if (b != rint(b)) atomicAdd(&bad, 1ull);
      continue;
    }
    if (__float_as_uint(x2::upk(Q).x) != __float_as_uint(q) ||
        (a != 0.0f && __float_as_uint(x2::upk(Q).y) != __float_as_uint(-q)))
      atomicAdd(&bad, 1ull);
    if (fabsf(q) < 0x1p-126f && q != 0.0f) atomicAdd(&tiny, 1ull);
  }
}
int main() {
  k_quot<<<1024, 256>>>(4000);
  unsigned long long h[3];
  if (cudaMemcpyFromSymbol(h, bad, 8) != cudaSuccess || cudaMemcpyFromSymbol(h + 1, tiny, 8) != cudaSuccess ||
      cudaMemcpyFromSymbol(h + 2, halfway, 8) != cudaSuccess) return 2;
  std::printf("%llu wrong, %llu subnormal, %llu halfway\n", h[0], h[1], h[2]);
  return h[0] != 0 || h[1] < 1000000 || h[2] > 1000;
}
""")
    exe = tmp_path / "t"
    r = subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-fmad=false", f"-I{CSRC}", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
