"""Cancellation inside a running launch.

The crate's CPU integrators poll their cancel closure per row, pixel, grain and offset
(src/pixelwise.rs:28, src/grainwise.rs:30-93) and return RenderError::Cancelled; the viewer relies on
it to drop a superseded render (latest job wins).  Here the closure is polled by a host thread, the
library mirrors it into mapped memory and the persistent / block kernels stop at their next work
item.  Each case renders a plane that takes a few hundred milliseconds, cancels it a quarter of the
way in, and checks that the call returns early with the kernel-side stop reported, and that the next
render of the same plane is bit-identical to an uncancelled one.  No GPU fault is involved: the
kernels read a flag and return.
"""
import ctypes
import threading
import time

import numpy as np
import pytest

from film_grain_gb300 import workloads

pytestmark = pytest.mark.gpu

CASES = {
    # the block kernels (lean pass, deferred fat pass)
    "pixel_blocks": dict(size=4096, algo="pixel", kw=dict(radius_mean=0.025, radius_stddev=0.01, n_samples=256, seed=42,
                                                          lognorm=True)),
    # the per-sample kernel
    "pixel_per_sample": dict(size=4096, algo="pixel", kw=dict(radius_mean=0.025, n_samples=256, seed=7)),
    # the grain-wise persistent kernel on a saturated plane (u = 1: thousands of grains per pixel)
    "grain": dict(size=1024, algo="grain", level=1.0, kw=dict(radius_mean=0.025, n_samples=256, seed=42)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_cancel_stops_a_running_launch(cuda, fgl, name):
    torch = cuda
    case = CASES[name]
    kw = dict(case["kw"])
    if kw.pop("lognorm", False):
        kw["radius_dist"] = fgl.RadiusDist.Lognorm
    kw["algo"] = fgl.Algo.Pixel if case["algo"] == "pixel" else fgl.Algo.Grain
    p = fgl.ParamsBuilder(**kw).build()
    if "level" in case:
        plane = np.full((case["size"], case["size"]), case["level"], np.float32)
    else:
        plane = workloads.blobs_plane(case["size"], case["size"], 3)
    d = fgl.derive_common(p, (case["size"], case["size"]))
    lam = torch.from_numpy(fgl.lambda_plane(fgl.normalize_plane(plane)[0], d.inv_e_pi_r2)).cuda()
    render = fgl.render_pixelwise if case["algo"] == "pixel" else fgl.render_grainwise
    if case["algo"] == "pixel":
        want_kernels = (3,) if name == "pixel_per_sample" else (4, 6)
        assert fgl.pixelwise_kernel_count(p, d) in want_kernels  # the case exercises the kernel it names

    render(lam, p, d)  # warm-up
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    want = render(lam, p, d)
    torch.cuda.synchronize()
    full = time.perf_counter() - t0
    assert full > 0.1, f"plane too fast ({full * 1e3:.1f} ms) to cancel in flight"

    start = time.perf_counter()
    with pytest.raises(fgl.CancelledError) as err:
        render(lam, p, d, cancel=lambda: time.perf_counter() - start > 0.25 * full)
    elapsed = time.perf_counter() - start
    assert "inside a kernel" in str(err.value)
    assert elapsed < 0.75 * full, f"cancelled call took {elapsed * 1e3:.0f} ms of {full * 1e3:.0f} ms"

    again = render(lam, p, d)
    torch.cuda.synchronize()
    assert torch.equal(again.view(torch.int32), want.view(torch.int32))


def test_cancel_whole_image_inside_a_launch(cuda, fgl):
    """fg_render_image (render_with_input_image_cancelable, src/lib.rs:86-93) on a 2048^2 RGB frame."""
    rgb = workloads.blobs_rgb(2048, 2048, 1)
    p = fgl.ParamsBuilder(radius_mean=0.025, radius_dist=fgl.RadiusDist.Lognorm, radius_stddev=0.01, n_samples=256,
                          seed=42, algo=fgl.Algo.Pixel, color_mode=fgl.ColorMode.Rgb).build()
    want, _ = fgl.render_with_input_image(rgb, p)
    t0 = time.perf_counter()
    fgl.render_with_input_image(rgb, p)
    full = time.perf_counter() - t0
    start = time.perf_counter()
    with pytest.raises(fgl.CancelledError):
        fgl.render_with_input_image(rgb, p, cancel=lambda: time.perf_counter() - start > 0.25 * full)
    assert time.perf_counter() - start < 0.75 * full
    again, _ = fgl.render_with_input_image(rgb, p)
    assert np.array_equal(again, want)


@pytest.mark.parametrize("size,radius", [((96, 64), 0.1), ((512, 512), 0.1), ((512, 512), 0.05)])
def test_looking_at_the_flag_costs_little(cuda, fgl, size, radius):
    """A render with a cancel flag that stays clear takes less than 1.5 times one without a flag, plus 100 us (host
    work): the kernels do not read host memory for every short item of theirs."""
    torch = cuda
    L = fgl.lib()
    p = fgl.ParamsBuilder(radius_mean=radius, n_samples=32, seed=3).build()
    d = fgl.derive_common(p, size)
    plane = workloads.blobs_plane(size[0], size[1], 5, scale=workloads.small_scale(*size))
    lam = torch.from_numpy(fgl.lambda_plane(fgl.normalize_plane(plane)[0], d.inv_e_pi_r2)).cuda()
    out = torch.empty((d.output_height, d.output_width), device="cuda")
    offs = np.ascontiguousarray(d.offsets_input, np.float32)
    flag = ctypes.c_int32(0)

    def best(cancel):
        times = []
        for _ in range(30):
            t0 = time.perf_counter()
            assert L.fg_render_pixelwise(lam.data_ptr(), p.c, d._c, offs.ctypes.data, out.data_ptr(), cancel,
                                         torch.cuda.current_stream().cuda_stream) == 0
            times.append(time.perf_counter() - t0)
        return sorted(times)[10]

    without, clear = best(None), best(ctypes.addressof(flag))
    assert clear < 1.5 * without + 100e-6, f"{without * 1e6:.0f} us without a flag, {clear * 1e6:.0f} us with one"


@pytest.mark.parametrize("kernels,kw", [
    (6, dict(radius_mean=0.5, n_samples=256)),  # the sparse pass and the fat pass over what it leaves
    (4, dict(radius_mean=0.2, n_samples=300)),  # the lean pass
])
def test_cancel_stops_the_block_passes(cuda, fgl, kernels, kw):
    """As above, on the block passes, at the first plane size that takes 0.12 s."""
    torch = cuda
    p = fgl.ParamsBuilder(seed=9, algo=fgl.Algo.Pixel, **kw).build()
    for size in (2048, 4096, 8192, 12288):
        d = fgl.derive_common(p, (size, size))
        lam = torch.from_numpy(fgl.lambda_plane(workloads.ramp_noise(size, size, 3), d.inv_e_pi_r2)).cuda()
        fgl.render_pixelwise(lam, p, d)
        t0 = time.perf_counter()
        want = fgl.render_pixelwise(lam, p, d)
        full = time.perf_counter() - t0
        if full > 0.12:
            break
    assert fgl.pixelwise_kernel_count(p, d) == kernels
    assert fgl.pixelwise_sparse_forms()[1] == 0 and (fgl.pixelwise_sparse_forms()[0] > 0) == (kernels == 6)
    start = time.perf_counter()
    with pytest.raises(fgl.CancelledError) as err:
        fgl.render_pixelwise(lam, p, d, cancel=lambda: time.perf_counter() - start > 0.25 * full)
    assert "inside a kernel" in str(err.value)
    assert time.perf_counter() - start < 0.75 * full
    assert torch.equal(fgl.render_pixelwise(lam, p, d), want)


def test_cancel_stops_short_items(cuda, fgl):
    """The stream pass without tiles and the pass over its dense segments, whose warps look at the flag by the clock:
    a flag set a third of the way into a render of some milliseconds."""
    torch = cuda
    L = fgl.lib()
    p = fgl.ParamsBuilder(radius_mean=0.1, n_samples=256, seed=9).build()
    d = fgl.derive_common(p, (850, 850))
    lam = torch.from_numpy(fgl.lambda_plane(workloads.ramp_noise(850, 850, 3), d.inv_e_pi_r2)).cuda()
    out = torch.empty((d.output_height, d.output_width), device="cuda")
    offs = np.ascontiguousarray(d.offsets_input, np.float32)
    flag = ctypes.c_int32(0)
    stream = torch.cuda.current_stream().cuda_stream

    def call():
        return L.fg_render_pixelwise(lam.data_ptr(), p.c, d._c, offs.ctypes.data, out.data_ptr(),
                                     ctypes.addressof(flag), stream)

    assert call() == 0
    t0 = time.perf_counter()
    assert call() == 0
    full = time.perf_counter() - t0
    assert full > 1.5e-3 and fgl.pixelwise_sparse_forms()[1] > 0
    want = out.clone()
    setter = threading.Timer(full / 3, lambda: setattr(flag, "value", 1))
    setter.start()
    assert call() == 2  # FG_ERR_CANCELLED
    setter.join()
    assert b"inside a kernel" in L.fg_last_error_message()
    flag.value = 0
    assert call() == 0 and torch.equal(out, want)
