"""The register-resident iteration (all iterations of a level in one cooperative launch): the bits of
one launch per iteration, for every tile height, kind of tile and form, and the exact quotients and
roots its float form is built from."""
import ctypes
import subprocess

import numpy as np
import pytest

from tests.helpers import params, random_case

pytestmark = pytest.mark.gpu

OUT = (("u", 1), ("u_", 1), ("us", 1), ("u_s", 1), ("warpUV", 2), ("Tp", 2))


def _solve(case, p, half, masked, variant=None, frames=2):
    from vfs_b200.stereotgv import StereoTgv
    i0, i1, mask, tv, cv = case
    s = StereoTgv()
    s.set_solve_path(True, half)
    h, w = i0.shape
    s.limitRange = p["limit_range"]
    s.initialize(w, h, p["beta"], p["gamma"], p["alpha0"], p["alpha1"], p["tsl"], p["lam"], p["n_levels"],
                 p["f_scale"], p["n_warp"], p["n_iter"])
    if variant is not None:
        s.set_iteration_variant(variant)
    s.copyMaskToDevice(mask)
    s.loadVectorFields(tv, cv)
    for _ in range(frames):
        s.copyImagesToDevice(i0, i1)
        (s.solveStereoForwardMasked if masked else s.solveStereoForward)()
    out = {n: s.debug_buffer(n, c) for n, c in OUT}
    assert s.check_guards() == 0
    return out, s.iteration_variants()


def _same(case, p, half, masked, resident=True):
    """Both ping-pong buffers, so odd and even iteration counts and the kept values are covered."""
    from vfs_b200._native import lib
    want, _ = _solve(case, p, half, masked, variant=1)
    got, ran = _solve(case, p, half, masked)
    if resident is not None:
        assert (ran == [14] * p["n_levels"]) == resident, ran
    for n in want:
        assert np.array_equal(got[n], want[n], equal_nan=True), n
    st = ctypes.c_int(-1)
    assert lib().vfs_device_status(ctypes.byref(st)) == 0 and st.value == 0


# widths about one and two tiles of 30 columns, heights about the tile rows, one row or column over
@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
@pytest.mark.parametrize("masked", [True, False], ids=["masked", "plain"])
@pytest.mark.parametrize("size", [(29, 40), (30, 31), (31, 33), (61, 62), (90, 44), (91, 45), (121, 64)])
def test_tile_edges(gpu, size, masked, half):
    w, h = size
    for n_iter in (1, 2, 5):
        _same(random_case(w, h, seed=w * h), params(n_levels=1, n_warp=2, n_iter=n_iter), half, masked)


# enough pixels for tiles of 4, 6, 8 (and, half storage, 12) rows; an all-on mask fills them evenly
@pytest.mark.parametrize("size,half", [((640, 100), True), ((424, 400), False), ((600, 520), True), ((760, 480), False),
                                       ((830, 560), True), ((850, 560), False), ((810, 760), True)])
def test_tile_heights(gpu, size, half):
    w, h = size
    case = random_case(w, h, seed=w + h)
    yy, xx = np.mgrid[0:h, 0:w]
    inside = (xx > 0) & (yy > 0) & (xx < w - 1) & (yy < h - 1)
    _same((case[0], case[1], inside.astype(np.float32), case[3], case[4]), params(n_levels=1, n_warp=1, n_iter=3), half,
          True)


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
def test_masks_with_isolated_pixels(gpu, half):
    """Lone pixels, one-pixel gaps and thin lines: on pixels whose edge rules read masked-out ones,
    whose two ping-pong values alternate."""
    w, h = 100, 70
    i0, i1, mask, tv, cv = random_case(w, h, seed=3)
    rng = np.random.default_rng(5)
    for k in range(3):
        m = mask.copy()
        if k == 0:
            m[rng.random((h, w)) < 0.08] = 0
        elif k == 1:
            m[:] = 0
            m[20:50, 10:90:2] = 1
            m[10, 5:95] = 1
        else:
            m[:, 29:32] = 0
            m[33, :] = 0
            m[40, 60] = 1
        m[0] = m[:, 0] = 0
        for n_iter in (3, 4):
            _same((i0, i1, m, tv, cv), params(n_levels=1, n_warp=2, n_iter=n_iter), half, True)


@pytest.mark.parametrize("masked", [True, False], ids=["masked", "plain"])
@pytest.mark.parametrize("size", [(850, 702), (991, 999), (1078, 1009)])
def test_tall_tiles(gpu, size, masked):
    """Tiles of 12 and 16 rows (half storage): ragged right and lower edges, a disc that leaves masked-out
    pixels and isolated ones in them, and alpha0 = 0, where eta_v2 may vanish."""
    w, h = size
    i0, i1, mask, tv, cv = random_case(w, h, seed=w)
    yy, xx = np.mgrid[0:h, 0:w]
    m = ((xx > 0) & (yy > 0) & ((xx - w / 2) ** 2 + (yy - h / 2) ** 2 < (0.62 * w) ** 2)).astype(np.float32)
    m[np.random.default_rng(w).random((h, w)) < 0.001] = 0
    for kw in (dict(n_iter=1), dict(n_iter=4), dict(n_iter=3, alpha0=0.0)):
        _same((i0, i1, m, tv, cv), params(n_levels=1, n_warp=1, **kw), True, masked)


def test_levels_it_does_not_take(gpu):
    """A masked-in pixel of column 0 without its right neighbour, more iterations than one launch
    holds, a negative lambda: the one-iteration kernels, with the same results."""
    i0, i1, mask, tv, cv = random_case(70, 50, seed=8)
    m = mask.copy()
    m[20, 0], m[20, 1] = 1, 0
    _same((i0, i1, m, tv, cv), params(n_levels=1, n_warp=1, n_iter=4), False, True, resident=None)
    _same((i0, i1, mask, tv, cv), params(n_levels=1, n_warp=1, n_iter=128), True, True)
    for p in (params(n_levels=1, n_warp=1, n_iter=129), params(n_levels=1, n_warp=1, n_iter=3, lam=-1.0)):
        _, ran = _solve((i0, i1, mask, tv, cv), p, False, True, frames=1)
        assert ran != [14]


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
def test_zero_and_extreme_preconditioners(gpu, half):
    """alpha0 = 0 makes eta_v2 zero where the tensor is (columns beyond the reference's launch
    grid when w > h), which writes v.x twice; a huge alpha1 leaves the exact quotients' range."""
    case = random_case(130, 60, seed=12, circle=False)
    m = case[2]
    m[0] = m[:, 0] = 0
    for kw in (dict(alpha0=0.0), dict(alpha0=0.0, alpha1=1e-20), dict(alpha1=3e18)):
        _same(case, params(n_levels=1, n_warp=1, n_iter=4, **kw), half, True)


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
@pytest.mark.parametrize("masked", [True, False], ids=["masked", "plain"])
def test_values_whose_squares_overflow(gpu, masked, half):
    """Images with a patch of 1e24, infinities and NaN: dual variables whose norm overflows."""
    i0, i1, mask, tv, cv = random_case(130, 66, seed=13)
    for v in (1e24, np.inf, np.nan):
        a, b = i0.astype(np.float32) / 255, i1.astype(np.float32) / 255
        a[20:24, 40:52] = v
        b[40:41, 80:83] = v
        _same((a, b, mask, tv, cv), params(n_levels=1, n_warp=2, n_iter=6), half, masked)


def test_exact_quotients_and_roots(gpu, tmp_path):
    """Every significand of a divisor and every m in [1, 4) (and scaled by 2^26), and 10^9 random
    quotients, against the device's IEEE division and square root."""
    from vfs_b200.build import ARCH, CSRC, nvcc
    src = tmp_path / "t.cu"
    src.write_text(r"""
#include <cstdio>
#include "tgv_exact_pairs.cuh"
using namespace vfs;
namespace x2 = fast::x2;
__device__ unsigned long long bad[4];
__device__ bool ne(float a, float b) { return __float_as_uint(a) != __float_as_uint(b); }
__global__ void k_recip() {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  for (unsigned e = 40; e < 220; e += 29) {
    const float b = __uint_as_float((i & 1) << 31 | e << 23 | i);
    const float2 y = x2::upk(exact::recip(x2::pk(b, -b)));
    if (ne(y.x, 1.0f / b) || ne(y.y, -1.0f / b)) atomicAdd(&bad[0], 1ull);
  }
}
__global__ void k_root() {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  for (unsigned sh = 0; sh <= 26; sh += 26) {
    const float m = __uint_as_float(((127u + sh) << 23) + i);
    x2::f2 s, y;
    exact::root(x2::pk(m, m), s, y);
    const float r = sqrtf(m);
    if (ne(x2::upk(s).x, r) || ne(x2::upk(y).y, 1.0f / r)) atomicAdd(&bad[1], 1ull);
  }
}
__global__ void k_quot(int n) {
  unsigned long long s = 0x9E3779B97F4A7C15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
  for (int i = 0; i < n; i++) {
    s ^= s << 13; s ^= s >> 7; s ^= s << 17;
    const unsigned ma = s & 0x7fffff, mb = (s >> 60) ? (s >> 23) & 0x7fffff : 0x7fffff - ((s >> 46) & 7);
    const float a = __uint_as_float((unsigned)(s >> 63) << 31 | (unsigned)(87 + ((s >> 46) & 63)) << 23 | ma);
    const float b = __uint_as_float((unsigned)(97 + ((s >> 52) & 63)) << 23 | mb);
    const x2::f2 B = x2::pk(b, b), Q = exact::quot(x2::pk(a, -a), B, exact::recip(B));
    if (ne(x2::upk(Q).x, a / b) || ne(x2::upk(Q).y, -a / b)) atomicAdd(&bad[2], 1ull);
  }
}
int main() {
  k_recip<<<(1 << 23) / 256, 256>>>();
  k_root<<<(1 << 24) / 256, 256>>>();
  k_quot<<<1024, 256>>>(4000);
  unsigned long long h[4];
  if (cudaMemcpyFromSymbol(h, bad, sizeof(h)) != cudaSuccess) return 2;
  std::printf("%llu %llu %llu\n", h[0], h[1], h[2]);
  return h[0] || h[1] || h[2];
}
""")
    exe = tmp_path / "t"
    r = subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "-fmad=false", f"-I{CSRC}", str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def _dropin(case, p, stream=None):
    from vfs_b200.stereotgv import StereoTgv
    i0, i1, mask, tv, cv = case
    s = StereoTgv()
    h, w = i0.shape
    s.limitRange = p["limit_range"]
    s.initialize(w, h, p["beta"], p["gamma"], p["alpha0"], p["alpha1"], p["tsl"], p["lam"], p["n_levels"],
                 p["f_scale"], p["n_warp"], p["n_iter"])
    s.copyMaskToDevice(mask)
    s.loadVectorFields(tv, cv)
    if stream is not None:
        s.set_stream(stream)
    return s


@pytest.mark.parametrize("masked", [True, False], ids=["masked", "plain"])
def test_dropin_path_buffers(gpu, masked):
    """The drop-in path on the register-resident iteration (128 iterations) and on a kernel per
    operation (129, more than one launch holds): the fused path's one-iteration kernels' buffers, and
    p and q that are zero where nothing is solved."""
    case = random_case(64, 48, seed=21)
    i0, i1 = case[:2]
    for n_iter in (128, 129):
        p = params(n_levels=2, n_warp=1, n_iter=n_iter)
        s = _dropin(case, p)
        f, _ = _solve(case, p, False, masked, variant=1)
        for _ in range(2):
            s.copyImagesToDevice(i0, i1)
            (s.solveStereoForwardMasked if masked else s.solveStereoForward)()
        for n, c in OUT:
            assert np.array_equal(s.debug_buffer(n, c), f[n], equal_nan=True), (n_iter, n)
        on = case[2] > 0 if masked else None
        for n, c in (("p", 2), ("q", 4)):  # zero where nothing is solved
            v = s.debug_buffer(n, c)
            assert np.isfinite(v).all()
            if masked:
                assert not v[~on].any(), n
        assert s.check_guards() == 0


def test_dropin_solve_in_a_captured_stream(gpu):
    """The drop-in solve inside a caller's stream capture, after solves that made its texture objects:
    its launches go into the caller's graph."""
    import torch
    case = random_case(150, 110, seed=3)
    p = params(n_levels=2, n_warp=2, n_iter=6)
    i0, i1 = (torch.from_numpy(x).cuda() for x in case[:2])
    want = _dropin(case, p)
    want.copyImagesToDevice(*case[:2])
    want.solveStereoForwardMasked()
    u = want.copy1DDisparityToHost()
    st = torch.cuda.Stream()
    s = _dropin(case, p, st)
    out = torch.zeros((110, 150), device="cuda")
    torch.cuda.synchronize()

    def frame():
        s.copy_images_from_device(i0, i1)
        s.solveStereoForwardMasked()
        s.copy_1d_disparity_to_device(out)

    for _ in range(2):
        frame()
    torch.cuda.synchronize()
    out.zero_()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        frame()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), u)


def test_captured_dropin_solve_after_a_new_mask(gpu):
    """A caller's graph of the drop-in solve takes the mask that is there when it is replayed."""
    import torch
    case = random_case(150, 110, seed=5)
    p = params(n_levels=2, n_warp=2, n_iter=6)
    i0, i1 = (torch.from_numpy(x).cuda() for x in case[:2])
    yy, xx = np.mgrid[0:110, 0:150]
    new = ((xx > 20) & (xx < 140) & (yy > 30) & (yy < 100)).astype(np.float32)
    outs = []
    for capture in (False, True):
        st = torch.cuda.Stream()
        s = _dropin(case, p, st)
        out = torch.zeros((110, 150), device="cuda")
        torch.cuda.synchronize()

        def frame():
            s.copy_images_from_device(i0, i1)
            s.solveStereoForwardMasked()
            s.copy_1d_disparity_to_device(out)

        for _ in range(2):
            frame()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        if capture:
            with torch.cuda.graph(g, stream=st):
                frame()
        s.copyMaskToDevice(new)
        torch.cuda.synchronize()
        g.replay() if capture else frame()
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
    assert np.array_equal(*outs)


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
@pytest.mark.parametrize("masked", [True, False], ids=["masked", "plain"])
def test_cluster_sizes(gpu, masked, half):
    """Levels about the size where the tiles of one cluster give way to the whole GPU (208 tiles of two
    rows with half storage, 128 with float), one tile, and fewer tiles than blocks."""
    for w, h in ((28, 2), (30, 18), (61, 130), (115, 64), (118, 66), (118, 104), (119, 106)):
        case = random_case(w, h, seed=w * h)
        m = np.ones((h, w), np.float32)
        if h > 2:
            m[0] = m[:, 0] = 0
        case = case[:2] + (m,) + case[3:]
        for n_iter in (1, 2, 7):
            _same(case, params(n_levels=1, n_warp=2, n_iter=n_iter), half, masked, resident=None)
