"""The surrogate's kernels against the CPU oracle (oracle/surrogate_ref.py), and what training gains.

Tolerances: the device and the oracle store the same tensors in bf16 at the same points and both
accumulate in f32, but in different orders, so a value within rounding distance of a bf16 boundary can
round to the neighbouring bf16 (one part in 256) and carry that into later layers.  Outputs are
therefore compared by max abs error (forward) and by relative L2 norm per gradient tensor (backward),
with the bounds stated in each test.
"""
import numpy as np
import pytest

from oracle import surrogate_ref as sr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg(cuda, fgl):
    from film_grain_gb300 import surrogate
    return surrogate


def _random_net(sg, torch, n_res=3, seed=1):
    net = sg.SurrogateNet(n_res=n_res, seed=seed)
    rng = np.random.default_rng(seed + 100)
    w = net.w32.cpu().numpy()
    net._np_view(w, "w_in")[:, :, :3] = rng.normal(0, 0.4, (32, 9, 3))
    net._np_view(w, "w_res")[:] = rng.normal(0, 0.06, (n_res, 32, 9, 32))
    net._np_view(w, "w_out")[0] = rng.normal(0, 0.05, (9, 32))
    net._np_view(w, "b_in")[:] = rng.normal(0, 0.1, 32)
    net._np_view(w, "b_res")[:] = rng.normal(0, 0.05, (n_res, 32))
    net._np_view(w, "b_out")[0] = 0.01
    net.w32.copy_(torch.from_numpy(w))
    net.wbf.copy_(net.w32.to(torch.bfloat16))
    net.ema.copy_(net.w32)
    return net


def _inputs(torch, nb, h, w, seed=5):
    rng = np.random.default_rng(seed)
    u = rng.uniform(0, 1, (nb, h, w)).astype(np.float32)
    t = np.clip(u + rng.normal(0, 0.1, u.shape), 0, 1).astype(np.float32)
    r = rng.uniform(0.03, 0.2, nb).astype(np.float32)
    return torch.from_numpy(u).cuda(), torch.from_numpy(r).cuda(), torch.from_numpy(t).cuda()


def test_make_input_channels_and_noise(sg, cuda):
    torch = cuda
    net = sg.SurrogateNet(n_res=1)
    u, r, _ = _inputs(torch, 2, 256, 256)
    net.forward(u, r, seed=77, keep=True)
    x = net._workspace(2, 256, 256)["x"].float().cpu().numpy()
    assert np.array_equal(x[..., 0], sr.bf16_round(u.cpu().numpy()))
    want_r = sr.bf16_round(r.cpu().numpy() * np.float32(net.radius_scale))
    assert np.array_equal(x[..., 2], np.broadcast_to(want_r[:, None, None], x[..., 2].shape))
    assert not x[..., 3:].any()
    z = x[..., 1].ravel()
    assert abs(z.mean()) < 0.01 and abs(z.std() - 1.0) < 0.01
    assert abs(np.mean(z ** 4) - 3.0) < 0.1  # Gaussian kurtosis
    net.forward(u, r, seed=77, keep=True)
    assert np.array_equal(net._workspace(2, 256, 256)["x"].float().cpu().numpy(), x)
    net.forward(u, r, seed=78, keep=True)
    assert not np.array_equal(net._workspace(2, 256, 256)["x"].float().cpu().numpy()[..., 1], x[..., 1])


@pytest.mark.parametrize("shape", [(2, 8, 32), (3, 37, 45), (1, 64, 64), (2, 40, 300)])
def test_forward_matches_oracle(sg, cuda, shape):
    """Max abs error of y within 2e-2 (y is O(1); one bf16 step of a hidden activation moves it ~1e-3).
    (2, 40, 300): the residual layers' tensor-core kernel with several 128-pixel column tiles (the last one
    partial) and 16-row strips (the last one partial)."""
    torch = cuda
    nb, h, w = shape
    net = _random_net(sg, torch)
    u, r, _ = _inputs(torch, nb, h, w)
    y = net.forward(u, r, seed=9, keep=True).cpu().numpy()
    x = net._workspace(nb, h, w)["x"].float().cpu().numpy()
    y_ref, _ = sr.forward(x, u.cpu().numpy(), net.numpy_net())
    err = np.abs(y - y_ref).max()
    assert err < 2e-2, err
    assert np.abs(y - u.cpu().numpy()).max() > 0.05  # the network is not the identity here
    y_inf = net.infer(u, r, seed=9).cpu().numpy()
    assert np.array_equal(y_inf.view(np.uint32), y.view(np.uint32)), "fg_sg_infer differs from the layer calls"


def _conv_inputs(torch, nb, h, w, seed):
    rng = np.random.default_rng(seed)
    bf = lambda a: sr.bf16_round(a.astype(np.float32))
    x = bf(np.maximum(rng.normal(0, 1, (nb, h, w, 32)), 0))
    return (x, bf(rng.normal(0, 0.06, (32, 9, 32))), rng.normal(0, 0.1, 32).astype(np.float32),
            bf(rng.normal(0, 1, (nb, h, w, 32))))


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 9, 128), (3, 17, 129), (700, 3, 5), (1, 400, 130)])
def test_tensor_core_convs_match_oracle(sg, cuda, fgl, shape):
    """The residual conv with its ReLU output and the data gradient on the tensor cores: one pixel, one full
    column tile, a column tile of one pixel, row ranges that span many images, ranges longer than the
    accumulator ring.  Outputs are f32 sums rounded to bf16: within one bf16 step (2^-7) of the oracle's,
    plus 2e-5 for 288 products of f32 rounding."""
    torch = cuda
    nb, h, w = shape
    x, wt, b, res = _conv_inputs(torch, nb, h, w, 3)
    dev = lambda a: torch.from_numpy(a).cuda().to(torch.bfloat16)
    X, Wt, R, B = dev(x), dev(wt), dev(res), torch.from_numpy(b).cuda()
    out, aux = torch.empty_like(X), torch.empty_like(X)
    st = torch.cuda.current_stream().cuda_stream
    call = lambda kind, r, o, a: fgl.lib().fg_sg_conv_forward(kind, X.data_ptr(), 32, Wt.data_ptr(), B.data_ptr(),
                                                              r.data_ptr(), None, o.data_ptr(), a, None, nb, h, w, st)
    close = lambda got, want: np.all(np.abs(got.float().cpu().numpy() - want) <= 2.0**-7 * np.abs(want) + 2e-5)
    z = sr.conv(x, wt)
    relu = np.maximum(z + b, 0)
    assert call(sg.CONV_RESIDUAL, X, out, aux.data_ptr()) == 0
    assert close(out, x + relu) and close(aux, relu)
    assert call(sg.CONV_DGRAD_RESIDUAL, R, out, None) == 0
    assert close(out, res + z)
    assert call(sg.CONV_DGRAD_RESIDUAL, R, R, None) == 0  # in place, as the backward pass runs it
    assert torch.equal(R, out)


def test_tensor_core_conv_repeats_bit_for_bit(sg, cuda, fgl):
    """Back-to-back launches over many small images (whose halo rows outside the image are filled with zeros at
    once, the tightest reuse of a row slot) all equal the first."""
    torch = cuda
    nb, h, w = 256, 64, 64
    gen = torch.Generator(device="cuda").manual_seed(2)
    X = torch.randn((nb, h, w, 32), generator=gen, device="cuda").relu_().to(torch.bfloat16)
    Wt = (torch.randn((32, 9, 32), generator=gen, device="cuda") * 0.05).to(torch.bfloat16)
    B = torch.zeros(32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    outs = [(torch.empty_like(X), torch.empty_like(X)) for _ in range(8)]
    for _ in range(6):
        for out, aux in outs:
            assert fgl.lib().fg_sg_conv_forward(sg.CONV_RESIDUAL, X.data_ptr(), 32, Wt.data_ptr(), B.data_ptr(), X.data_ptr(),
                                                None, out.data_ptr(), aux.data_ptr(), None, nb, h, w, st) == 0
        torch.cuda.synchronize()
        for out, aux in outs:
            assert torch.equal(aux, outs[0][1]) and torch.equal(out, outs[0][0])
            # the sum's two roundings (r and out, one bf16 step each)
            assert bool(((out.float() - X.float() - aux.float()).abs() <= 2.0**-7 * out.float().abs()).all())


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 9, 128), (3, 17, 129), (300, 3, 5)])
def test_tensor_core_dgrad_and_wgrad_match_oracle(sg, cuda, fgl, shape):
    """The masked data gradients and the weight gradients of the three conv kinds on the tensor cores.  Data
    gradients: one bf16 step (2^-7) plus 2e-5; the mask exactly.  Weight gradients: f32 sums of up to
    n = nb h w products (here n <= 4500) in another order, each within n 2^-23 of the sum of magnitudes."""
    torch = cuda
    nb, h, w = shape
    x, wt, _, res = _conv_inputs(torch, nb, h, w, 7)
    rng = np.random.default_rng(8)
    g = sr.bf16_round(rng.normal(0, 1, (nb, h, w, 32)).astype(np.float32))
    relu = np.maximum(rng.normal(0, 1, (nb, h, w, 32)), 0).astype(np.float32)
    dy = np.zeros((nb, h, w, 16), np.float32)
    dy[..., 0] = g[..., 0]
    w_out = np.zeros((8, 9, 32), np.float32)
    w_out[0] = wt[0]
    dev = lambda a: torch.from_numpy(a).cuda().to(torch.bfloat16)
    G, X, R, Wt, M, DY, WO = dev(g), dev(x), dev(res), dev(wt), dev(relu), dev(dy), dev(w_out)
    out, masked = torch.empty_like(G), torch.empty_like(G)
    L, st = fgl.lib(), torch.cuda.current_stream().cuda_stream
    close = lambda got, want: np.all(np.abs(got.float().cpu().numpy() - want) <= 2.0**-7 * np.abs(want) + 2e-5)
    for kind, gout, wts, want in ((sg.CONV_DGRAD_RESIDUAL, G, Wt, res + sr.conv_dgrad(g, wt)),
                                  (sg.CONV_DGRAD_OUTPUT, DY, WO, sr.conv_dgrad(dy[..., :8], w_out))):
        for dst in (out, None):
            assert L.fg_sg_conv_dgrad(kind, gout.data_ptr(), gout.shape[-1], wts.data_ptr(), R.data_ptr(), M.data_ptr(),
                                      None if dst is None else out.data_ptr(), masked.data_ptr(), nb, h, w, st) == 0
            if dst is not None:
                assert close(out, want)
            assert torch.equal(masked, torch.where(M > 0, out, torch.zeros_like(out)))
    x16 = torch.zeros((nb, h, w, 16), dtype=torch.bfloat16, device="cuda")
    x16[..., :3] = X[..., :3]
    for kind, gout, xin, co, ci in ((sg.CONV_RESIDUAL, G, X, 32, 32), (sg.CONV_INPUT, G, x16, 32, 16),
                                    (sg.CONV_OUTPUT, DY, X, 8, 32)):
        dw = torch.zeros((co, 9, ci), device="cuda")
        db = torch.zeros(co, device="cuda")
        assert L.fg_sg_conv_wgrad(kind, gout.data_ptr(), gout.shape[-1], xin.data_ptr(), xin.shape[-1], dw.data_ptr(),
                                  db.data_ptr(), nb, h, w, st) == 0
        gn, xn = gout.float().cpu().numpy()[..., :co].astype(np.float64), xin.float().cpu().numpy().astype(np.float64)
        bound = nb * h * w * 2.0**-23
        assert np.all(np.abs(dw.cpu().numpy() - sr.conv_wgrad(gn, xn)) <= bound * sr.conv_wgrad(np.abs(gn), np.abs(xn)))
        flat = gn.reshape(-1, co)
        assert np.all(np.abs(db.cpu().numpy() - flat.sum(0)) <= bound * np.abs(flat).sum(0))


@pytest.mark.parametrize("shape", [(2, 16, 32), (2, 19, 41)])
def test_gradients_match_oracle(sg, cuda, shape):
    """Every parameter gradient within 3e-2 relative L2 of the oracle's (bf16 activations, f32 sums)."""
    torch = cuda
    nb, h, w = shape
    net = _random_net(sg, torch)
    u, r, t = _inputs(torch, nb, h, w)
    net.forward(u, r, seed=11, keep=True)
    loss_sum = float(net.backward(u, t).item())
    ws = net._workspace(nb, h, w)
    x = ws["x"].float().cpu().numpy()
    y_ref, cache = sr.forward(x, u.cpu().numpy(), net.numpy_net())
    loss_ref, g_ref = sr.backward(y_ref, t.cpu().numpy(), cache, net.numpy_net())
    assert abs(loss_sum / (nb * h * w) - loss_ref) <= 1e-2 * loss_ref
    g = net.grad.cpu().numpy()
    for name in ("w_in", "b_in", "w_res", "b_res", "w_out", "b_out"):
        got, want = net._np_view(g, name), g_ref[name].astype(np.float32)
        if name == "w_in":  # channels 3..15 of the input are zero: their gradient must be exactly 0
            assert not got[:, :, 3:].any()
            got, want = got[:, :, :3], want[:, :, :3]
        if name in ("w_out", "b_out"):
            assert not got[1:].any(), "unused output channels must get no gradient"
            got, want = got[:1], want[:1]
        rel = np.linalg.norm(got - want) / np.linalg.norm(want)
        assert rel < 3e-2, (name, rel)


def test_adam_matches_oracle(sg, cuda):
    torch = cuda
    net = _random_net(sg, torch, n_res=2)
    u, r, t = _inputs(torch, 2, 16, 32)
    w0 = net.w32.cpu().numpy().astype(np.float64)
    m = np.zeros_like(w0)
    v = np.zeros_like(w0)
    ema = w0.copy()
    for step in (1, 2):
        net.forward(u, r, seed=step, keep=True)
        net.backward(u, t)
        g = net.grad.cpu().numpy().astype(np.float64)
        net.adam_step(lr=1e-3, ema_decay=0.999)
        w0, m, v = sr.adam(w0, m, v, g, step, lr=1e-3, decay=net.decay.cpu().numpy().astype(np.float64))
        d = (1.0 + step) / (10.0 + step)  # the decay's warm-up
        ema = d * ema + (1 - d) * w0
        got = net.w32.cpu().numpy()
        assert np.abs(got - w0).max() < 1e-6
        assert np.abs(net.ema.cpu().numpy() - ema).max() < 1e-6
        assert np.array_equal(net.wbf.float().cpu().numpy(), sr.bf16_round(got))


def test_checkpoint_resume(sg, cuda, tmp_path):
    torch = cuda
    net = _random_net(sg, torch, n_res=2)
    u, r, t = _inputs(torch, 4, 32, 32)
    for s in range(3):
        net.train_step(u, r, t, seed=s)
    path = str(tmp_path / "ck.npz")
    net.save(path)
    net2 = sg.SurrogateNet.load(path)
    assert net2.step == 3
    for a, b in ((net.w32, net2.w32), (net.wbf, net2.wbf), (net.m, net2.m), (net.v, net2.v), (net.ema, net2.ema)):
        assert torch.equal(a, b)
    # the gradient sums are float atomics, so the next step agrees to rounding, not bit for bit
    net.train_step(u, r, t, seed=3)
    net2.train_step(u, r, t, seed=3)
    torch.cuda.synchronize()
    assert torch.allclose(net.w32, net2.w32, rtol=0, atol=1e-6)
    assert torch.allclose(net.m, net2.m, rtol=1e-3, atol=1e-7)


def test_training_gains_over_no_network(sg, cuda):
    """A short grain-training run on plain N=256 renders of tiles (constant and lognormal radii), scored
    on held-out tiles.
    (a) With its noise weights zeroed the network predicts the expected render (the mean of 16
        independently seeded N=1024 renders: a single render carries a grain realisation and MC noise no
        predictor can know) with less than half the MAE of the method without a network (the intensity u
        itself) and of the untrained network, and beats the plain render at N=16.
    (b) With its noise input it renders grain: the spectrum of its residual against the expectation over
        1/64 .. 1/4 cycles/px is within half the error of u's (u has no grain) from the grain of a plain
        N=1024 render."""
    torch = cuda
    u_tr, r_tr, sd_tr, rn_tr = sg.training_set(4096, seed=1)
    t_tr = sg.render_tiles(u_tr, r_tr, n_samples=256, seed=1, radius_sd=sd_tr)
    u_te, r_te, sd_te, rn_te = sg.training_set(128, seed=99)
    refs = [sg.render_tiles(u_te, r_te, n_samples=1024, seed=99 + k, radius_sd=sd_te) for k in range(16)]
    ref = sum(refs) / 16
    low = sg.render_tiles(u_te, r_te, n_samples=16, seed=123, radius_sd=sd_te)
    ut, rt = torch.from_numpy(u_tr).cuda(), torch.from_numpy(rn_tr).cuda()
    ue, re = torch.from_numpy(u_te).cuda(), torch.from_numpy(rn_te).cuda()
    net = sg.SurrogateNet(n_res=8, seed=0)
    mae_untrained = float((net.infer(ue, re, seed=5, grain=False) - ref).abs().mean())
    hist = sg.train(net, ut, rt, t_tr, steps=2000, batch=64, lr=1e-3, seed=0, log_every=500, log=lambda s: None,
                    grain_n=256)
    net.use_ema()
    mae_net = float((net.infer(ue, re, seed=5, grain=False) - ref).abs().mean())
    mae_id = float((ue - ref).abs().mean())
    mae_low = float((low - ref).abs().mean())
    floor = float((refs[0] - refs[1]).abs().mean()) / np.sqrt(2)  # one N=1024 render's own deviation
    gb_net = sg.grain_band_error(net.infer(ue, re, seed=5), refs[0], ue, None, 1024)
    gb_id = sg.grain_band_error(ue, refs[0], ue, None, 1024)
    print(f"MAE vs mean of 16 N=1024 renders: trained {mae_net:.4f}, identity {mae_id:.4f}, "
          f"untrained {mae_untrained:.4f}, plain N=16 {mae_low:.4f}, single N=1024 render {floor:.4f}; "
          f"grain-band error vs an N=1024 render: trained {gb_net:.3f}, identity {gb_id:.3f}; train {hist}")
    assert mae_net < 0.5 * mae_id
    assert mae_net < 0.5 * mae_untrained
    assert mae_net < mae_low
    assert gb_net < 0.5 * gb_id


def test_evaluator_matches_oracle(sg, cuda):
    """The device spectrum metric (torch FFT) against the numpy oracle, and MAE / spectrum error on
    known pairs."""
    torch = cuda
    rng = np.random.default_rng(4)
    img = rng.normal(0, 1, (96, 128)).astype(np.float32) + np.linspace(0, 3, 128, dtype=np.float32)[None, :]
    got = sg.raps(torch.from_numpy(img).cuda()).cpu().numpy()
    want = sr.raps(img)
    assert np.allclose(got, want, rtol=1e-9, atol=1e-9 * want.max())
    a = torch.from_numpy(img).cuda()
    e = sg.evaluate(a, a)
    assert e["mae"] == 0.0 and e["raps_max"] < 1e-12  # the device bin sums are atomics: order-dependent
    e = sg.evaluate(a + 0.5, a)  # a constant offset changes the MAE but not the spectrum of (img - mean)
    assert abs(e["mae"] - 0.5) < 1e-6 and e["raps_max"] < 1e-6  # f32 rounding of img + 0.5
    e = sg.evaluate(2 * a, a)  # doubling the image quadruples its power
    assert abs(e["raps_max"] - 3.0) < 1e-9


@pytest.mark.parametrize("nb,h,w", [(200, 3, 1), (9, 11, 24), (7, 5, 30), (2, 9, 62), (5, 8, 64), (6, 7, 65), (3, 40, 67),
                                    (2, 5, 68)])
def test_narrow_images_sharing_row_tiles(sg, cuda, fgl, nb, h, w):
    """Images up to 67 pixels wide share row tiles, wherever the tiles cut them: every conv gives the bits that it
    gives for each image on its own (one image takes a row tile alone, and a pixel's sum runs in the same
    order)."""
    torch = cuda
    x, wt, b, res = _conv_inputs(torch, nb, h, w, 11)
    dev = lambda a: torch.from_numpy(a).cuda().to(torch.bfloat16)
    X, Wt, R, B = dev(x), dev(wt), dev(res), torch.from_numpy(b).cuda()
    W16 = Wt[:, :, :16].contiguous()
    X16 = X[..., :16].contiguous()
    U = torch.rand((nb, h, w), device="cuda")
    L, st = fgl.lib(), torch.cuda.current_stream().cuda_stream

    def run(n, s):
        sub = lambda t: t[s:s + n].contiguous()
        xs, x16, rs, us = sub(X), sub(X16), sub(R), sub(U)
        new = lambda: torch.empty_like(xs)
        out = [new() for _ in range(8)] + [torch.empty_like(us)]
        fwd = lambda kind, i, c, wgt, r, u, o, a, f: L.fg_sg_conv_forward(
            kind, i.data_ptr(), c, wgt.data_ptr(), B.data_ptr(), None if r is None else r.data_ptr(),
            None if u is None else u.data_ptr(), None if o is None else o.data_ptr(),
            None if a is None else a.data_ptr(), None if f is None else f.data_ptr(), n, h, w, st)
        assert fwd(sg.CONV_INPUT, x16, 16, W16, None, None, out[0], None, None) == 0
        assert fwd(sg.CONV_RESIDUAL, xs, 32, Wt, xs, None, out[1], None, None) == 0
        assert fwd(sg.CONV_RESIDUAL, xs, 32, Wt, xs, None, out[2], out[3], None) == 0
        assert fwd(sg.CONV_OUTPUT, xs, 32, Wt[:8].contiguous(), None, us, None, None, out[8]) == 0
        assert fwd(sg.CONV_DGRAD_RESIDUAL, xs, 32, Wt, rs, None, out[4], None, None) == 0
        assert L.fg_sg_conv_dgrad(sg.CONV_DGRAD_RESIDUAL, xs.data_ptr(), 32, Wt.data_ptr(), rs.data_ptr(), xs.data_ptr(),
                                  out[5].data_ptr(), out[6].data_ptr(), n, h, w, st) == 0
        assert L.fg_sg_conv_dgrad(sg.CONV_DGRAD_OUTPUT, x16.data_ptr(), 16, Wt[:8].contiguous().data_ptr(), None,
                                  rs.data_ptr(), None, out[7].data_ptr(), n, h, w, st) == 0
        torch.cuda.synchronize()
        return out

    together = run(nb, 0)
    for s in range(0, nb, max(1, nb // 5)):
        for a, t in zip(run(1, s), together):
            assert torch.equal(a[0], t[s])


@pytest.mark.parametrize("nb,h,w", [(256, 64, 64), (1, 720, 1280), (900, 24, 31), (3, 7, 9)])
def test_weight_gradient_of_long_sums(sg, cuda, fgl, nb, h, w):
    """Sums of one sign over up to a million pixels stay within 8e-7 plus 8e-7 a million pixels of 64 bits (relative
    L2), what the mma.sync kernels reach: a tensor-core accumulator cuts bits off at each addition, half of the last
    one on average, so a CTA may not keep adding to one for its whole share."""
    torch = cuda
    L, st = fgl.lib(), torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(4)
    for kind, co, ci, cg in ((sg.CONV_RESIDUAL, 32, 32, 32), (sg.CONV_INPUT, 32, 16, 32), (sg.CONV_OUTPUT, 8, 32, 16)):
        g = torch.rand((nb, h, w, cg), generator=gen, device="cuda").to(torch.bfloat16)
        x = torch.rand((nb, h, w, ci), generator=gen, device="cuda").to(torch.bfloat16)
        dw, db = torch.zeros((co, 9, ci), device="cuda"), torch.zeros(co, device="cuda")
        assert L.fg_sg_conv_wgrad(kind, g.data_ptr(), cg, x.data_ptr(), ci, dw.data_ptr(), db.data_ptr(), nb, h, w, st) == 0
        gd = g[..., :co].double().reshape(-1, co)
        xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
        want = torch.stack([gd.T @ xp[:, t // 3:t // 3 + h, t % 3:t % 3 + w].reshape(-1, ci) for t in range(9)], dim=1)
        bound = 8e-7 * (1 + nb * h * w / 1e6)
        for got, ref in ((dw, want), (db, gd.sum(0))):
            assert float((got.double() - ref).norm() / ref.norm()) < bound, kind


def test_a_wait_given_up_ends_training(sg, cuda, fgl, monkeypatch, tmp_path):
    """The flag that a kernel sets when a wait runs out is clear after a pass, and training raises where it reads a
    result (and writes no checkpoint) when the library reports it."""
    torch = cuda
    net = _random_net(sg, torch, n_res=1)
    u, r, t = _inputs(torch, 2, 16, 32)
    sg.train(net, u, r, t, steps=1, batch=2, log_every=1, log=lambda s: None)
    assert fgl.lib().fg_sg_check() == 0

    class Reporting:
        def __getattr__(self, name):
            return (lambda: 7) if name == "fg_sg_check" else getattr(fgl.lib(), name)  # FG_ERR_INTERNAL

    monkeypatch.setattr(sg, "lib", Reporting)
    path = tmp_path / "ck.npz"
    for kw in (dict(log_every=1), dict(checkpoint=str(path), checkpoint_every=1)):
        with pytest.raises(fgl.RenderError):
            sg.train(net, u, r, t, steps=net.step + 1, batch=2, log=lambda s: None, **kw)
    assert not path.exists()


def _misaligned(torch, shape, skip, fill=None):
    """A bf16 tensor of `shape` that starts `skip` elements behind a 16-byte boundary."""
    n = int(np.prod(shape))
    buf = torch.zeros(n + skip, dtype=torch.bfloat16, device="cuda")
    view = buf[skip:].view(shape)
    assert view.data_ptr() % 16
    if fill is not None:
        view.copy_(fill)
    return view


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 9, 33), (3, 17, 70)])
def test_mma_sync_kernels_match_oracle(sg, cuda, fgl, shape):
    """The kernels that take what the tensor-core ones refuse: outputs off a 16-byte boundary, a residual of another
    tensor, gradients off a boundary or of an odd channel stride; and the two passes that the backward pass ran beside
    them.  Bounds as for the tensor-core kernels."""
    torch = cuda
    nb, h, w = shape
    x, wt, b, res = _conv_inputs(torch, nb, h, w, 21)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(torch.bfloat16)
    X, X16, Wt, R, B = dev(x), dev(x[..., :16]), dev(wt), dev(res), torch.from_numpy(b).cuda()
    L, st = fgl.lib(), torch.cuda.current_stream().cuda_stream
    close = lambda got, want: np.all(np.abs(got.float().cpu().numpy() - want) <= 2.0**-7 * np.abs(want) + 2e-5)
    ptr = lambda t: None if t is None else t.data_ptr()
    call = lambda kind, i, c, wgt, r, o, a: L.fg_sg_conv_forward(kind, ptr(i), c, ptr(wgt), ptr(B), ptr(r), None, ptr(o),
                                                                  ptr(a), None, nb, h, w, st)
    z, relu = sr.conv(x, wt), np.maximum(sr.conv(x, wt) + b, 0)
    z16 = sr.conv(x[..., :16], wt[:, :, :16])
    out, aux = _misaligned(torch, X.shape, 2), _misaligned(torch, X.shape, 2)
    assert call(sg.CONV_RESIDUAL, X, 32, Wt, X, out, aux) == 0 and close(out, x + relu) and close(aux, relu)
    assert call(sg.CONV_DGRAD_RESIDUAL, X, 32, Wt, R, out, None) == 0 and close(out, res + z)
    W16 = Wt[:, :, :16].contiguous()
    assert call(sg.CONV_INPUT, X16, 16, W16, None, out, None) == 0 and close(out, np.maximum(z16 + b, 0))
    assert call(sg.CONV_DGRAD_OUTPUT, X16, 16, W16, None, out, None) == 0 and close(out, z16)
    whole, aux = torch.empty_like(X), torch.empty_like(X)
    assert call(sg.CONV_RESIDUAL, X, 32, Wt, R, whole, aux) == 0 and close(whole, res + relu) and close(aux, relu)

    g = sr.bf16_round(np.random.default_rng(22).normal(0, 1, (nb, h, w, 32)).astype(np.float32))
    bound = nb * h * w * 2.0**-23
    for skip, cs in ((4, 32), (0, 36)):
        G = torch.zeros(nb * h * w * cs + skip, dtype=torch.bfloat16, device="cuda")
        gv = G[skip:].view(nb, h, w, cs)
        gv[..., :32].copy_(dev(g))
        for kind, xin, co, ci in ((sg.CONV_RESIDUAL, X, 32, 32), (sg.CONV_INPUT, X16, 32, 16), (sg.CONV_OUTPUT, X, 8, 32)):
            dw, db = torch.zeros((co, 9, ci), device="cuda"), torch.zeros(co, device="cuda")
            assert L.fg_sg_conv_wgrad(kind, gv.data_ptr(), cs, xin.data_ptr(), ci, dw.data_ptr(), db.data_ptr(), nb, h, w,
                                      st) == 0
            gn, xn = g[..., :co].astype(np.float64), xin.float().cpu().numpy().astype(np.float64)
            assert np.all(np.abs(dw.cpu().numpy() - sr.conv_wgrad(gn, xn)) <= bound * sr.conv_wgrad(np.abs(gn), np.abs(xn)))
            flat = gn.reshape(-1, co)
            assert np.all(np.abs(db.cpu().numpy() - flat.sum(0)) <= bound * np.abs(flat).sum(0))

    masked = torch.empty_like(X)
    assert L.fg_sg_mask_grad(R.data_ptr(), X.data_ptr(), masked.data_ptr(), X.numel(), st) == 0
    assert torch.equal(masked, torch.where(X > 0, R, torch.zeros_like(R)))
    flipped = torch.empty((32, 9, 16), dtype=torch.bfloat16, device="cuda")
    W8 = Wt[:8].contiguous()
    assert L.fg_sg_flip_weights(W8.data_ptr(), flipped.data_ptr(), 8, 32, 16, 32, st) == 0
    want = torch.zeros_like(flipped)
    want[:, :, :8] = W8.flip(1).permute(2, 1, 0)
    assert torch.equal(flipped, want)
