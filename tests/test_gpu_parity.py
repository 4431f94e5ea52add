"""GPU parity: the sm_103a integrators against the CPU oracle, bit for bit.

Every case renders the same seeded plane through the library's C-ABI (host lambda plane -> GPU
integrator) and through the oracle (a C restatement of src/pixelwise.rs / src/grainwise.rs), and
requires the f32 output planes to be bit-identical (coverage counts equal, the same count * (1/N)).
"""
import os
import subprocess
import sys
import time

import numpy as np
import pytest

from film_grain_gb300 import workloads

pytestmark = pytest.mark.gpu


def _setup(fgl, orc, plane, radius=0.1, dist="const", sd=0.0, zoom=1.0, n=32, seed=5489, sigma=0.8,
           cell=None, maxr=None, size=None):
    h, w = plane.shape
    kw = dict(radius_mean=radius, radius_dist=fgl.RadiusDist.Lognorm if dist == "lognorm" else fgl.RadiusDist.Const,
              radius_stddev=sd, zoom=zoom, n_samples=n, seed=seed, sigma_px=sigma, cell_delta=cell, size=size)
    if maxr is not None:
        kw["max_radius"] = fgl.MaxRadius.Absolute(maxr)
    p = fgl.ParamsBuilder(**kw).build()
    d = fgl.derive_common(p, (w, h))
    norm, _ = fgl.normalize_plane(plane)
    lam = fgl.lambda_plane(norm, d.inv_e_pi_r2)
    op = orc.params_struct(dist, radius, sd, zoom, sigma, n, seed)
    od, offs, offs_in = orc.derive(op, w, h, ("absolute", maxr) if maxr is not None else ("quantile", 0.999), cell,
                                   size)
    onorm, _ = orc.normalize_plane(plane)
    olam = orc.lambda_plane(onorm, od.inv_e_pi_r2)
    assert np.array_equal(lam.view(np.uint32), olam.view(np.uint32)), "lambda planes differ"
    assert np.array_equal(d.offsets, offs) and np.array_equal(d.offsets_input, offs_in)
    assert (d.output_width, d.output_height, d.rm, d.delta) == (od.out_w, od.out_h, od.rm, od.delta)
    return p, d, lam, op, od, offs, offs_in


def _check(algo, fgl, orc, plane, **kw):
    p, d, lam, op, od, offs, offs_in = _setup(fgl, orc, plane, **kw)
    if algo == "pixel":
        got = fgl.render_pixelwise(lam, p, d)
        want, _ = orc.render("pixel", lam, op, od, offs_in)
    else:
        got = fgl.render_grainwise(lam, p, d)
        want, _ = orc.render("grain", lam, op, od, offs)
    assert got.shape == want.shape
    diff = np.count_nonzero(got.view(np.uint32) != want.view(np.uint32))
    assert diff == 0, f"{diff} of {got.size} pixels differ (max abs {np.abs(got - want).max()})"
    return got


def _blobs(w, h, seed=11):
    """A blob plane with blobs scaled to its size: dark background, mid tones and saturated spots."""
    return workloads.blobs_plane(w, h, seed, scale=workloads.small_scale(w, h))


# ------------------------------------------------------------------ pixel-wise
def test_pixelwise_ramp_256_n64(cuda, fgl, orc):
    """The 256x256 luma ramp workload: const radius 0.12, N=64, zoom 1, seed 42."""
    out = _check("pixel", fgl, orc, workloads.ramp_noise(256, 256, 42), radius=0.12, n=64, seed=42)
    slow, unstaged, subdiv, blocks = fgl.pixelwise_diagnostics()
    # interior blocks stage their windows; only border blocks, which own few samples, regenerate
    assert blocks > 0 and unstaged < blocks // 4 and slow < 0.05 * 256 * 256 * 64
    assert abs(float(out.mean()) - 0.5) < 0.01


@pytest.mark.parametrize("n", [1, 7, 37, 100])
def test_pixelwise_sample_counts(cuda, fgl, orc, n):
    _check("pixel", fgl, orc, _blobs(48, 40), radius=0.1, n=n, seed=3)


def test_pixelwise_lognormal(cuda, fgl, orc):
    _check("pixel", fgl, orc, _blobs(64, 48), radius=0.05, dist="lognorm", sd=0.025, n=40, seed=7)


@pytest.mark.parametrize("zoom", [0.5, 1.5, 2.0, 3.0])
def test_pixelwise_zoom(cuda, fgl, orc, zoom):
    _check("pixel", fgl, orc, _blobs(40, 36), radius=0.1, n=16, zoom=zoom, seed=9)


def test_pixelwise_cell_and_absolute_max_radius(cuda, fgl, orc):
    _check("pixel", fgl, orc, _blobs(40, 40), radius=0.15, n=20, cell=0.37, maxr=0.3, seed=13)


def test_pixelwise_rejection_regime(cuda, fgl, orc):
    """cell 1.0, radius 0.2: lambda*delta^2 >= 12 in bright areas (Poisson rejection branch)."""
    plane = np.clip(workloads.ramp_noise(32, 32, 5) * 1.2, 0, 1).astype(np.float32)
    _check("pixel", fgl, orc, plane, radius=0.2, n=16, cell=1.0, seed=17)


def test_pixelwise_dense_subdivides(cuda, fgl, orc):
    """A saturated plane with many samples per cell: every window overflows shared memory and, as the
    samples reach more than four windows' worth of cells, splits into quadrants."""
    plane = np.ones((24, 24), np.float32)
    _check("pixel", fgl, orc, plane, radius=0.05, n=256, seed=19)
    _, _, subdiv, _ = fgl.pixelwise_diagnostics()
    assert subdiv > 0


def test_pixelwise_dense_regenerates(cuda, fgl, orc):
    """A saturated plane whose blocks' samples reach about as many cells as a window holds: the whole
    plane runs the per-sample kernel (dense form)."""
    plane = np.ones((24, 24), np.float32)
    _check("pixel", fgl, orc, plane, radius=0.05, n=64, seed=19)
    slow, unstaged, subdiv, _ = fgl.pixelwise_diagnostics()
    assert subdiv == 0 and unstaged > 0 and slow == 24 * 24 * 64


def test_pixelwise_dense_block_regenerates(cuda, fgl, orc):
    """A saturated plane on the block kernel (samples reach 2.7 windows of cells): its overflowing
    dense windows regenerate per sample instead of subdividing."""
    plane = np.ones((24, 24), np.float32)
    _check("pixel", fgl, orc, plane, radius=0.05, n=128, seed=19)
    slow, unstaged, subdiv, _ = fgl.pixelwise_diagnostics()
    assert subdiv == 0 and unstaged > 0 and slow > 0


def test_pixelwise_mixed_density_blocks(cuda, fgl, orc):
    """A dark left half (0.1) and a bright right half (0.95) on the block kernel: sparse windows
    stage, dense ones regenerate."""
    plane = np.where(np.arange(64)[None, :] < 32, 0.1, 0.95).astype(np.float32).repeat(64, 0)
    _check("pixel", fgl, orc, plane, radius=0.05, n=128, seed=37)
    slow, unstaged, _, blocks = fgl.pixelwise_diagnostics()
    assert 0 < unstaged < blocks


@pytest.mark.parametrize("n", [16, 64])
def test_pixelwise_sparse_regenerates(cuda, fgl, orc, n):
    """Radius 0.025 (cells of 1/40 pixel) with few samples per pixel: the samples reach fewer cells
    than a staged window holds, so the plane runs the per-sample kernel (both forms: dark background
    and bright blobs)."""
    _check("pixel", fgl, orc, _blobs(48, 40), radius=0.025, n=n, seed=29)
    slow, unstaged, _, _ = fgl.pixelwise_diagnostics()
    assert unstaged > 0 and slow == 48 * 40 * n


def test_pixelwise_regen_zoom_and_lognormal(cuda, fgl, orc):
    """The per-sample kernel with zoom 2 and log-normal radii (ranges of 7 or 8 cells per axis: up to
    the full 64-cell mask)."""
    _check("pixel", fgl, orc, _blobs(40, 36), radius=0.05, dist="lognorm", sd=0.02, n=2, zoom=2.0, seed=41)
    slow, _, _, _ = fgl.pixelwise_diagnostics()
    assert slow == 80 * 72 * 2


def test_pixelwise_lognormal_small_radius(cuda, fgl, orc):
    """Log-normal radius 0.025/0.01 at N=256 (the large-frame workload's parameters): staged windows."""
    _check("pixel", fgl, orc, _blobs(40, 32), radius=0.025, dist="lognorm", sd=0.01, n=256, seed=31)


@pytest.mark.parametrize("n,zoom,dist,radius", [(256, 1.0, "lognorm", 0.04), (64, 1.0, "const", 0.08),
                                                (16, 1.0, "lognorm", 0.15), (256, 2.0, "lognorm", 0.04),
                                                (100, 0.5, "const", 0.1)])
def test_pixelwise_sparse_pass_forms(cuda, fgl, orc, n, zoom, dist, radius):
    """The sparse block pass (6 launches) in its forms: one offset per thread (N = 256) or several
    threads per offset sharing its rows (N 64, 16); rectangles within the 4 x 4 range table (zoom 1) or
    beyond it (zoom 2: cell ranges computed per sample); zoom 0.5; on a plane large enough for the
    4 x 4-pixel blocks, mixing dense and sparse regions.  The sample step runs grain-major (each staged
    grain tests the samples within its radius) at N = 256, sample-major where a grain can reach half a
    pixel (log-normal r 0.15: max radius 0.46)."""
    plane = _blobs(160, 128, seed=5)
    kw = dict(radius=radius, dist=dist, sd=0.4 * radius if dist == "lognorm" else 0.0, zoom=zoom, n=n, seed=41)
    p, d, *_ = _setup(fgl, orc, plane, **kw)
    assert fgl.pixelwise_kernel_count(p, d) == 6
    _check("pixel", fgl, orc, plane, **kw)
    sample_major, grain_major = fgl.pixelwise_sparse_forms()
    if n == 256:
        assert grain_major > 0
    if radius == 0.15:
        assert sample_major > 0 and grain_major == 0


@pytest.mark.parametrize("radius,n,zoom", [(0.025, 256, 1.0), (0.05, 128, 0.75), (0.1, 64, 1.0), (0.04, 32, 3.0),
                                           (0.08, 256, 1.0)])
def test_pixelwise_grain_major_form(cuda, fgl, orc, radius, n, zoom):
    """The sparse pass's grain-major form against the oracle: log-normal radii, zoom in and out (the
    phase bands wrap and span several bins), N from 32 to 256, a plane with dense blobs and empty
    regions.  At r 0.08, N 256 a grain has about 13 candidates, more than a warp's queue holds for 32
    grains, so the warps test their candidates lane by lane."""
    plane = _blobs(144, 112, seed=9)
    kw = dict(radius=radius, dist="lognorm", sd=0.4 * radius, zoom=zoom, n=n, seed=77)
    _check("pixel", fgl, orc, plane, **kw)
    sample_major, grain_major = fgl.pixelwise_sparse_forms()
    assert grain_major > 0


def test_pixelwise_empty_and_tiny(cuda, fgl, orc):
    _check("pixel", fgl, orc, np.zeros((16, 16), np.float32), radius=0.1, n=8)
    _check("pixel", fgl, orc, np.full((1, 1), 0.5, np.float32), radius=0.1, n=8)
    _check("pixel", fgl, orc, np.full((2, 3), 0.7, np.float32), radius=0.3, n=5, zoom=2.0)


def test_pixelwise_wide_filter(cuda, fgl, orc):
    _check("pixel", fgl, orc, _blobs(32, 32), radius=0.1, n=32, sigma=4.0, seed=21)


def test_pixelwise_forced_size(cuda, fgl, orc):
    """--size changes the output grid while the integrator keeps mapping with params.zoom."""
    _check("pixel", fgl, orc, _blobs(40, 30), radius=0.1, n=12, size=(50, None), seed=23)


# ------------------------------------------------------------------ grain-wise
def test_grainwise_blob_crop_lognormal_zoom2_n128(cuda, fgl, orc):
    """A 96x80 crop of the 1024^2 blob workload: lognormal 0.05/0.025, zoom 2, N=128."""
    plane = workloads.blobs_plane(1024, 1024, 0)[300:380, 400:496]
    _check("grain", fgl, orc, np.ascontiguousarray(plane), radius=0.05, dist="lognorm", sd=0.025, zoom=2.0, n=128,
           seed=42)


@pytest.mark.parametrize("n", [1, 31, 33, 200])
def test_grainwise_sample_counts(cuda, fgl, orc, n):
    _check("grain", fgl, orc, _blobs(40, 36), radius=0.1, n=n, seed=5)


@pytest.mark.parametrize("zoom", [0.5, 1.0, 1.5, 4.0])
def test_grainwise_zoom(cuda, fgl, orc, zoom):
    _check("grain", fgl, orc, _blobs(36, 30), radius=0.08, n=24, zoom=zoom, seed=29)


def test_grainwise_large_radius(cuda, fgl, orc):
    """radius_out > 0.5 px: the disks cover several pixel centres per offset."""
    _check("grain", fgl, orc, _blobs(24, 24), radius=0.8, n=16, zoom=2.0, maxr=1.0, seed=31)


def test_grainwise_empty_and_tiny(cuda, fgl, orc):
    _check("grain", fgl, orc, np.zeros((16, 16), np.float32), radius=0.1, n=8)
    _check("grain", fgl, orc, np.full((1, 1), 0.5, np.float32), radius=0.1, n=8)


def test_grainwise_forced_size(cuda, fgl, orc):
    _check("grain", fgl, orc, _blobs(40, 30), radius=0.1, n=12, size=(33, 70), seed=37)


# ------------------------------------------------------------------ whole-image path with the fused colour epilogue
@pytest.mark.parametrize("mode", ["luma", "rgb"])
@pytest.mark.parametrize("algo", ["pixel", "grain"])
def test_render_image_matches_oracle(cuda, fgl, orc, mode, algo):
    rgb = workloads.blobs_rgb(48, 40, 3, scale=workloads.small_scale(48, 40))
    p = fgl.ParamsBuilder(radius_mean=0.1, n_samples=24, zoom=1.5, seed=77,
                          color_mode=fgl.ColorMode.Luma if mode == "luma" else fgl.ColorMode.Rgb,
                          algo=fgl.Algo.Pixel if algo == "pixel" else fgl.Algo.Grain).build()
    got, stats = fgl.render_with_input_image(rgb, p)
    op = orc.params_struct("const", 0.1, 0.0, 1.5, 0.8, 24, 77)
    want, chosen = orc.render_image(rgb, mode, 2 if algo == "pixel" else 1, op)
    assert stats.algorithm == (fgl.Algo.Pixel if algo == "pixel" else fgl.Algo.Grain)
    assert got.shape == want.shape
    assert np.array_equal(got, want), f"{np.count_nonzero(got != want)} bytes differ"


def test_render_image_roi(cuda, fgl, orc):
    rgb = workloads.blobs_rgb(64, 64, 4, scale=workloads.small_scale(64, 64))
    p = fgl.ParamsBuilder(radius_mean=0.1, n_samples=16, seed=5, roi=fgl.Roi(8, 4, 40, 36)).build()
    got, stats = fgl.render_with_input_image(rgb, p)
    op = orc.params_struct("const", 0.1, 0.0, 1.0, 0.8, 16, 5)
    want, _ = orc.render_image(np.ascontiguousarray(rgb[4:36, 8:40]), "luma", 0, op)
    assert stats.input_size == (32, 32)
    assert np.array_equal(got, want)


def test_cancel_before_launch(cuda, fgl):
    plane = _blobs(16, 16)
    p = fgl.ParamsBuilder(n_samples=4).build()
    d = fgl.derive_common(p, (16, 16))
    lam = fgl.lambda_plane(fgl.normalize_plane(plane)[0], d.inv_e_pi_r2)
    with pytest.raises(fgl.CancelledError):
        fgl.render_pixelwise(lam, p, d, cancel=lambda: True)


def test_device_tensors_in_and_out(cuda, fgl, orc):
    """torch CUDA tensors go through the same entry point without host staging."""
    torch = cuda
    plane = _blobs(40, 32)
    p, d, lam, op, od, offs, offs_in = _setup(fgl, orc, plane, radius=0.1, n=16, seed=41)
    out = fgl.render_grainwise(torch.from_numpy(lam).cuda(), p, d)
    torch.cuda.synchronize()
    want, _ = orc.render("grain", lam, op, od, offs)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("n", [256, 257, 289, 512, 577])
def test_grainwise_sample_chunks(cuda, fgl, orc, n):
    """More samples than one chunk's masks hold: one chunk full, a last chunk of one sample's word, chunks of
    unequal width, two full ones, three."""
    _check("grain", fgl, orc, _blobs(37, 29), radius=0.07, n=n, zoom=1.5, seed=n)


@pytest.mark.parametrize("w,h,zoom,radius,n,dist", [
    (3, 1, 1.0, 0.05, 64, "const"),       # fewer pixels than warps: 32 lanes to a pixel
    (61, 9, 1.0, 0.02, 33, "lognorm"),    # saturated ramp end: parts of a few pixels, groups of 2 to 16 lanes
    (300, 40, 0.5, 0.04, 16, "lognorm"),  # one tile, lanes with a pixel each and refills
    (33, 35, 2.0, 0.4, 200, "const"),     # a grain reaches most samples: the pair queue overflows
])
def test_grainwise_lane_groups_and_queue(cuda, fgl, orc, w, h, zoom, radius, n, dist):
    plane = workloads.ramp_noise(w, h, 5)
    _check("grain", fgl, orc, plane, radius=radius, n=n, zoom=zoom, dist=dist, sd=0.4 * radius if dist == "lognorm" else 0.0,
           seed=41)


@pytest.mark.parametrize("w,h,radius,cell,zoom,n", [
    (41, 37, 0.02, None, 1.0, 33),    # per-sample kernel: rows of one lambda pixel and of two, two batches of 32
    (37, 29, 0.05, 0.31, 1.3, 5),     # three or four cells to a pixel, runs of a word's rows of three
    (70, 45, 0.45, 0.29, 0.5, 8),     # ranges over two pixels and more
    (64, 33, 0.4, 1.0, 1.0, 64),      # a lambda pixel row for every row of a bitmask word
    (300, 9, 0.3, 1.7, 1.0, 48),      # pixel rows left out between cell rows, more columns than a CTA
    (33, 70, 0.11, 0.07, 2.0, 100),   # runs that end inside a word
])
def test_pixelwise_screened_cells(cuda, fgl, orc, w, h, radius, cell, zoom, n):
    """The lambda pixels of a cell column's rows: in the plane's bitmask and in the per-sample kernel."""
    _check("pixel", fgl, orc, _blobs(w, h), radius=radius, cell=cell, zoom=zoom, n=n, seed=13)


@pytest.mark.parametrize("n", [1, 4, 5, 31, 33, 100])
def test_pixelwise_small_plane_parts(cuda, fgl, orc, n):
    """A small plane on the per-sample kernel, its samples in parts over several warps."""
    plane = _blobs(35, 9)
    p, d, *_ = _setup(fgl, orc, plane, radius=0.2, n=n, seed=3)
    if n <= 5:
        assert fgl.pixelwise_kernel_count(p, d) == 3
    _check("pixel", fgl, orc, plane, radius=0.2, n=n, seed=3)


@pytest.mark.parametrize("w,h,radius,dist,zoom,n,cell", [
    (128, 70, 0.15, "const", 1.0, 32, None),     # a word of bits a pixel
    (131, 67, 0.15, "const", 1.0, 33, None),     # two
    (97, 101, 0.1, "const", 1.0, 65, None),      # four
    (97, 101, 0.08, "lognorm", 1.0, 129, None),  # eight; ranges of several cells
    (103, 91, 0.05, "lognorm", 1.0, 256, None),
    (200, 180, 0.7, "const", 0.5, 50, None),     # grains wider than an input pixel
    (41, 33, 0.12, "const", 3.0, 40, None),      # reach 0.36 of a pixel
    (67, 49, 0.21, "const", 2.0, 22, None),      # reach 0.42
    (120, 90, 0.3, "const", 1.0, 64, 1.0),       # cells of a pixel, the rejection regime
    (110, 90, 0.3, "const", 1.0, 20, 0.04),      # ranges of 16 cells: no per-sample kernel
    (131, 67, 0.3, "const", 1.0, 128, None),     # 36 hits a grain: tiles and their footprints
    (320, 250, 0.12, "const", 1.0, 40, 0.02),    # tiles of many chunks
])
def test_pixelwise_stream_pass(cuda, fgl, orc, w, h, radius, dist, zoom, n, cell):
    """The stream pass: widths off the segments and tiles, every variant of words, dark, middle and saturated
    areas (the last on the per-sample kernel, where its ranges allow)."""
    plane = _blobs(w, h)
    plane[: h // 3, : w // 2] = 1.0
    plane[h // 2:, : w // 5] = 0.0
    kw = dict(radius=radius, dist=dist, sd=0.4 * radius if dist == "lognorm" else 0.0, zoom=zoom, n=n, cell=cell, seed=9)
    p, d, *_ = _setup(fgl, orc, plane, **kw)
    assert fgl.pixelwise_kernel_count(p, d) == 6
    _check("pixel", fgl, orc, plane, **kw)
    assert fgl.pixelwise_sparse_forms()[1] > 0


def test_pixelwise_stream_all_dense_and_empty(cuda, fgl, orc):
    _check("pixel", fgl, orc, np.ones((96, 100), np.float32), radius=0.1, n=64, seed=3)
    assert fgl.pixelwise_diagnostics()[0] == 96 * 100 * 64  # every segment on the per-sample kernel
    _check("pixel", fgl, orc, np.zeros((96, 100), np.float32), radius=0.1, n=64, seed=3)


@pytest.mark.parametrize("n", [2, 9, 33, 40])
def test_pixelwise_two_step_ranges(cuda, fgl, orc, n):
    """The per-sample kernel with ranges of five cells and more: samples that the middle cells leave uncovered,
    from none to all of a warp's (dark, middle and saturated areas), in one and two batches of 32."""
    plane = _blobs(70, 45)
    plane[:15, :40] = 0.02
    plane[30:, 20:] = 1.0
    _check("pixel", fgl, orc, plane, radius=0.03, dist="lognorm", sd=0.012, n=n, seed=21)


@pytest.mark.parametrize("radius,zoom,n", [(0.22, 2.0, 40), (0.2249, 2.0, 70), (0.2251, 2.0, 70), (0.004, 1.0, 64),
                                           (0.00002, 1.0, 33), (0.4, 1.0, 130)])
def test_grainwise_one_pixel_form(cuda, fgl, orc, radius, zoom, n):
    """Zoomed radii up to and beyond 0.45, where a pair's bounds can hold more than the nearest pixel, and radii
    around the coordinates' rounding, where every hit computes its bounds; the plane's edges."""
    plane = _blobs(37, 29)
    plane[:, -3:] = 0.9
    dim = 1e-7 if radius < 0.001 else 1e-3 if radius < 0.01 else 1.0  # grains a pixel: not too many
    _check("grain", fgl, orc, (plane * dim).astype(np.float32), radius=radius, zoom=zoom, n=n, seed=5)


@pytest.mark.parametrize("w,h,radius,zoom,n,kernels", [
    (96, 64, 0.1, 1.0, 32, 3),    # per-sample kernel
    (160, 128, 0.1, 1.0, 64, 6),  # stream pass
    (160, 128, 0.45, 1.0, 64, 6),  # sparse and fat passes
    (160, 128, 0.45, 0.5, 64, 6),  # an output smaller than lambda
    (160, 128, 0.2, 1.0, 300, 4),  # lean and fat passes
])
def test_pixelwise_in_place(cuda, fgl, w, h, radius, zoom, n, kernels):
    """An output that is lambda's own memory, or shares its end, gets what a separate one gets, through every
    pixel-wise entry point."""
    torch = cuda
    L = fgl.lib()
    p = fgl.ParamsBuilder(radius_mean=radius, zoom=zoom, n_samples=n, seed=3).build()
    d = fgl.derive_common(p, (w, h))
    lam = torch.from_numpy(fgl.lambda_plane(fgl.normalize_plane(_blobs(w, h))[0], d.inv_e_pi_r2)).cuda()
    assert fgl.pixelwise_kernel_count(p, d) == kernels
    want = fgl.render_pixelwise(lam, p, d).flatten()
    offs = np.ascontiguousarray(d.offsets_input, np.float32)
    st = torch.cuda.current_stream().cuda_stream
    for name in ("fg_render_pixelwise", "fg_render_pixelwise_async", "fg_render_pixelwise_noalloc"):
        for at in (0, w * h - 7):  # the output's first float in lambda
            buf = torch.cat([lam.flatten(), torch.full((want.numel(),), 0.5, device="cuda")])
            args = [buf.data_ptr(), p.c, d._c, offs.ctypes.data, buf[at:].data_ptr()]
            args += [None, st] if name == "fg_render_pixelwise" else [st]
            assert getattr(L, name)(*args) == 0, L.fg_last_error_message().decode()
            assert torch.equal(buf[at:at + want.numel()], want), (name, at)


def _fastest(torch, call, n=5):
    times = []
    for _ in range(n + 1):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        call()
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t0)
    return min(times[1:])


def _grain_plane(fgl, plane, **kw):
    p = fgl.ParamsBuilder(**kw).build()
    d = fgl.derive_common(p, (plane.shape[1], plane.shape[0]))
    return p, d, fgl.lambda_plane(fgl.normalize_plane(plane)[0], d.inv_e_pi_r2)


@pytest.mark.parametrize("n", [64, 128])
def test_grainwise_saturated_strip_keeps_pace(cuda, fgl, n):
    """A narrow plane that is half saturated (7000 grains a pixel, a few tens of thousands of such pixels) takes at
    most 1.85 times as long a grain as an even plane, whose pixels fill every lane: 1.97 (N 128: 45 ps against 23) with
    parts that were unequal and whose lanes repeated each other's draws."""
    torch = cuda
    rate = []
    for plane in (np.full((600, 600), 0.7, np.float32), workloads.blobs_plane(123, 1024, 3, scale=1024 / 1536)):
        p, d, lam = _grain_plane(fgl, plane, radius_mean=0.025, n_samples=n, seed=5)
        dl = torch.from_numpy(lam).cuda()
        rate.append(_fastest(torch, lambda: fgl.render_grainwise(dl, p, d)) / float(lam.astype(np.float64).sum()))
    assert rate[1] < 1.85 * rate[0], [r * 1e12 for r in rate]


def test_batch_not_slower_than_its_images(cuda, fgl):
    """One launch over images whose grains cost very different amounts (radius 0.025 with one candidate pair a grain,
    radius 0.2 with 44) takes no longer than the images one after the other (a tenth for noise)."""
    torch = cuda
    items, alone = [], 0.0
    for w, h, radius in ((123, 1024, 0.025), (500, 400, 0.2), (250, 1024, 0.1)):
        plane = workloads.blobs_plane(w, h, 3, scale=max(w, h) / 1536)
        p, d, lam = _grain_plane(fgl, plane, radius_mean=radius, n_samples=256, seed=5)
        dl = torch.from_numpy(lam).cuda()
        items.append((dl, p, d, fgl.Algo.Grain, lam))
        alone += _fastest(torch, lambda: fgl.render_grainwise(dl, p, d))
    batch = fgl.Batch(items)
    together = _fastest(torch, batch.run)
    assert together < 1.1 * alone, f"{together * 1e3:.1f} ms together, {alone * 1e3:.1f} ms one by one"


# A render whose device memory comes from a pool of a given size (the driver API's struct CUmemPoolProps).
_LIMITED_POOL = """
import ctypes, sys
import numpy as np, torch
import film_grain_gb300 as fg
from film_grain_gb300 import workloads

class Props(ctypes.Structure):
    _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("loc_type", ctypes.c_int),
                ("loc_id", ctypes.c_int), ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]

p = fg.ParamsBuilder(radius_mean=0.2, n_samples=256, seed=3).build()
d = fg.derive_common(p, (4096, 4096))
plane = workloads.ramp_noise(4096, 4096, 5)
lam = torch.from_numpy(fg.lambda_plane(plane, d.inv_e_pi_r2)).cuda()
want = fg.render_pixelwise(lam, p, d)
assert fg.pixelwise_sparse_forms()[0] == 0 and fg.pixelwise_sparse_forms()[1] > 0
cu = ctypes.CDLL("libcuda.so.1")
props = Props(alloc_type=1, loc_type=1, loc_id=0, max_size=int(sys.argv[1]) << 20)
pool = ctypes.c_void_p()
assert cu.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) == 0
assert cu.cuDeviceSetMemPool(0, pool) == 0
got = fg.render_pixelwise(lam, p, d)
assert torch.equal(got, want)
print("forms", *fg.pixelwise_sparse_forms(), "blocks", fg.pixelwise_diagnostics()[3])
"""


@pytest.mark.parametrize("mib,sparse", [(512, True), (288, False)])
def test_pixelwise_with_little_memory(cuda, fgl, mib, sparse):
    """4096^2, N 256: 256 MiB of cells, 50 of bitmask, 512 of the samples' bits.  Without room for the bits the plane
    takes the sparse pass, without room for the bitmask the lean pass."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _LIMITED_POOL, str(mib)], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    forms = r.stdout.split()
    assert int(forms[2]) == 0 and (int(forms[1]) > 0) == sparse and int(forms[4]) > 0, r.stdout


def test_refused_request_does_not_wait(cuda, fgl):
    """A request that is refused (too many samples for the grain-wise tile) returns while the caller's stream is still
    busy: an image and a plane behind a kernel of about 0.4 s."""
    torch = cuda
    p = fgl.ParamsBuilder(radius_mean=0.1, n_samples=20000, seed=3, algo=fgl.Algo.Grain).build()
    d = fgl.derive_common(p, (64, 48))
    lam = torch.from_numpy(fgl.lambda_plane(fgl.normalize_plane(_blobs(64, 48))[0], d.inv_e_pi_r2)).cuda()
    rgb = np.ascontiguousarray(workloads.blobs_rgb(64, 48, 3, scale=workloads.small_scale(64, 48)), np.float32)
    out = np.empty((48, 64, 3), np.uint8)
    stream = torch.cuda.Stream()
    for plane in (True, False):
        with torch.cuda.stream(stream):
            torch.cuda._sleep(800_000_000)
            done = torch.cuda.Event()
            done.record()
            if plane:
                with pytest.raises(fgl.RenderError, match="too large"):
                    fgl.render_grainwise(lam, p, d)
            else:
                assert fgl.lib().fg_render_image(rgb.ctypes.data, 64, 48, p.c, out.ctypes.data, None, None,
                                                 stream.cuda_stream) != 0
            assert not done.query()
        torch.cuda.synchronize()


@pytest.mark.parametrize("w,h,zoom,radius,n", [
    (61, 9, 1.0, 0.02, 33),    # a saturated ramp end: parts of a few pixels, 2 to 32 lanes to a pixel
    (97, 3, 2.0, 0.015, 20),   # parts that do not divide the tile
    (40, 1, 1.0, 0.01, 5),     # 32 lanes to a pixel of many thousand grains
    (130, 95, 0.5, 0.03, 64),  # one tile, groups of 1 and 2
])
def test_grainwise_parts_and_skipped_draws(cuda, fgl, orc, w, h, zoom, radius, n):
    """Constant radius: the lanes of a pixel stand at their own grains of its stream, in parts that take the tile's
    pixels in turn."""
    _check("grain", fgl, orc, workloads.ramp_noise(w, h, 5), radius=radius, n=n, zoom=zoom, seed=17)


@pytest.mark.parametrize("w,h,n,dist", [(37, 29, 33, "const"), (37, 29, 40, "lognorm"), (90, 31, 20, "const"),
                                        (23, 40, 200, "const")])
def test_grainwise_even_tiles(cuda, fgl, orc, w, h, n, dist):
    """Saturated planes, whose tiles are cut into parts that fill the lanes at once."""
    _check("grain", fgl, orc, np.ones((h, w), np.float32), radius=0.04, dist=dist, sd=0.012 if dist == "lognorm" else 0.0,
           n=n, seed=23)


def test_grainwise_fewer_samples_cost_less(cuda, fgl):
    """A saturated plane at N 128 takes less time than at N 256: the same grains with half of the samples.  Cut by cost
    alone, its parts of 675 pixels left a third of the lanes waiting, and it took 86 ms against 81."""
    torch = cuda
    times = []
    for n in (128, 256):
        p, d, lam = _grain_plane(fgl, np.ones((512, 1024), np.float32), radius_mean=0.025, n_samples=n, seed=5)
        dl = torch.from_numpy(lam).cuda()
        times.append(_fastest(torch, lambda: fgl.render_grainwise(dl, p, d), 3))
    assert times[0] < 0.95 * times[1], times
