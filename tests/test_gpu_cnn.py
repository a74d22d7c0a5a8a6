"""Learned-closure kernels on the GPU against the float64 CPU oracle
(oracle/cnn_oracle.py).

Tolerances (f32 kernels against f64 maths): layer outputs and gradients
within 1e-5 relative to the largest magnitude of the compared array; the
closure records within binary16 rounding (2e-3 relative); the per-cell
relaxation path bit-exact against a plain run at the same omega."""
import ctypes

import numpy as np
import pytest

from oracle import cnn_oracle as C

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda(cuda_ok):
    import torch
    return torch


def close(got, want, tol=1e-5, atol=0.0):
    got = np.asarray(got, np.float64)
    scale = max(np.abs(want).max(), 1e-30)
    err = np.abs(got - want).max()
    assert err <= tol * scale + atol, "max error %.3e of scale %.3e" % (err, scale)


def params_for(seed):
    from lbm_gb300 import closure
    return closure.unpack(closure.init_params(seed).astype(np.float64))


def test_gpu_conv_layers_forward_and_backward(lbm, torch_cuda, oracle_mod):
    torch = torch_cuda
    from lbm_gb300 import closure
    net = closure.ClosureNet(seed=5)
    ps = closure.unpack(net.numpy().astype(np.float64))
    rng = np.random.default_rng(1)
    N, H, W = 2, 13, 150
    feat = rng.normal(size=(N, 4, H, W)) * np.array([0.3, 0.6, 0.2, 1.0])[None, :, None, None]
    ft = torch.from_numpy(feat.astype(np.float32)).cuda()
    z = net.forward(ft)
    acts = C.forward(ps, feat.astype(np.float32).astype(np.float64))
    for l in range(1, 5):
        close(net._acts[l].cpu().numpy(), acts[l])
    gz = rng.normal(size=(N, 1, H, W))
    net.backward(torch.from_numpy(gz.astype(np.float32)).cuda())
    grads = C.backward(ps, acts, gz.astype(np.float32).astype(np.float64))
    got = closure.unpack(net.grads.cpu().numpy().astype(np.float64))
    for l in range(4):
        close(got[l][0], grads[l][0], 2e-5)
        close(got[l][1], grads[l][1], 2e-5)
    torch.cuda.synchronize()


def test_gpu_closure_loss_and_full_gradient(lbm, torch_cuda):
    torch = torch_cuda
    from lbm_gb300 import closure
    net = closure.ClosureNet(seed=7)
    ps = closure.unpack(net.numpy().astype(np.float64))
    rng = np.random.default_rng(2)
    N, H, W = 3, 17, 40
    feat = (rng.normal(size=(N, 4, H, W)) * 0.5).astype(np.float32)
    sxx, sxy = rng.normal(size=(2, N, H, W)) * 1e-2
    dxx = -0.02 * sxx + 1e-4 * rng.normal(size=sxx.shape)
    txy = -0.02 * sxy + 1e-4 * rng.normal(size=sxy.shape)
    coef = np.stack([(8 / 9) * (sxx ** 2 + sxy ** 2), -(4 / 3) * (dxx * sxx + txy * sxy),
                     2 * (dxx ** 2 + txy ** 2)], axis=1).astype(np.float32)
    norm = float(coef[:, 2].sum())
    z = net.forward(torch.from_numpy(feat).cuda())
    L, gz = net.loss(z, torch.from_numpy(coef).cuda(), norm)
    acts = C.forward(ps, feat.astype(np.float64))
    L64, gz64 = C.loss(acts[-1], coef.astype(np.float64), norm)
    assert float(L.item()) == pytest.approx(L64, rel=1e-5)
    close(gz.cpu().numpy(), gz64, 1e-4)
    net.backward(gz)
    g64 = C.backward(ps, acts, gz64)
    got = closure.unpack(net.grads.cpu().numpy().astype(np.float64))
    for l in range(4):
        close(got[l][0], g64[l][0], 2e-4)
        close(got[l][1], g64[l][1], 2e-4)


def test_gpu_adam_matches_oracle(lbm, torch_cuda):
    torch = torch_cuda
    from lbm_gb300 import closure
    net = closure.ClosureNet(seed=3)
    p = net.numpy().astype(np.float64)
    m = np.zeros_like(p)
    v = np.zeros_like(p)
    rng = np.random.default_rng(3)
    for t in range(1, 4):
        g = rng.normal(size=p.size).astype(np.float32)
        net.grads.copy_(torch.from_numpy(g))
        net.adam(1e-3)
        C.adam(p, g.astype(np.float64), m, v, t, 1e-3)
    close(net.numpy(), p, 1e-6)


def test_gpu_closure_samples_match_oracle(lbm, torch_cuda):
    """Samples of a real fine run (96 x 64 channel, circle) at three snapshots."""
    from lbm_gb300 import closure, geometry
    mask = geometry.single_circle(96, 64, 30, 31.5, 7)
    feat, coef, solid_c = closure.fine_samples(mask, 0.55, 0.06, 60, 20, 4, seed=1)
    with lbm.Lattice(96, 64, 1.0 / 0.55, lbm.EDGE_CHANNEL, lbm.F32) as lat:
        lat.set_inlet_velocity(0.06)
        lat.init_equilibrium(1.0, 0.06, 0.0, 1e-3, 1)
        lat.draw_mask(mask)
        for k in range(3):
            lat.iterate(20)
            pops = lat.populations().astype(np.float64)
            f64, c64 = C.sample(pops, mask, 4)
            close(feat[k].cpu().numpy(), f64, 1e-5)
            # the stresses are differences of O(u^2) f32 products (subgrid
            # variances ~1e-6 of u^2 ~ 4e-3): f32 leaves ~1e-3 relative on them
            for j in range(3):
                close(coef[k, j].cpu().numpy(), c64[j], 5e-3, atol=1e-16)
    np.testing.assert_array_equal(solid_c.cpu().numpy(), C.coarsen(pops, mask, 4)[-1])


@pytest.mark.parametrize("kernel", [0, 1])
def test_gpu_fused_inference_matches_oracle(lbm, torch_cuda, kernel):
    """The tile-fused network on a lattice's moments (kernel 0: tcgen05 tensor
    cores with BF16 activations; 1: CUDA cores with f32 activations) against
    the whole-image oracle network with the same BF16-rounded weights.  The
    tensor-core kernel rounds each layer's activations to BF16 (8-bit
    mantissa): its delta_tau is held to 2 % of the largest value."""
    from lbm_gb300 import closure, geometry
    nx, ny = 150, 70  # ragged tiles on both axes
    mask = geometry.single_circle(nx, ny, 40, 35, 8)
    flat = closure.init_params(11)
    flat[-1] = 0.3  # output bias
    L = lbm.load_library()
    with lbm.Lattice(nx, ny, 1.0 / 0.51, lbm.EDGE_CHANNEL, lbm.F32) as lat:
        lat.set_inlet_velocity(0.08)
        lat.init_equilibrium(1.0, 0.08, 0.0, 1e-2, 4)
        lat.draw_mask(mask)
        lat.iterate(30)
        p = flat.copy()
        lbm._check(L.lbm_closure_set_weights(lat.handle, p.ctypes.data_as(ctypes.c_void_p), p.size))
        lbm._check(L.lbm_closure_enable(lat.handle, 0.5))
        lbm._check(L.lbm_closure_set_inference(lat.handle, kernel))
        lbm._check(L.lbm_closure_infer(lat.handle))
        lat.synchronize()
        dt = np.zeros(nx * ny, np.float32)
        sp = np.zeros(nx * ny, np.float32)
        lbm._check(L.lbm_closure_read(lat.handle, dt.ctypes.data_as(ctypes.c_void_p),
                                      sp.ctypes.data_as(ctypes.c_void_p)))
        rho, jx, jy = lat.field("rho"), lat.field("jx"), lat.field("jy")
    fl = mask == 0
    r = np.where(fl, rho, 1.0).astype(np.float64)
    feat = np.stack([np.where(fl, (r - 1) * C.S_RHO, 0), np.where(fl, jx / r * C.S_U, 0),
                     np.where(fl, jy / r * C.S_U, 0), (~fl).astype(np.float64)])[None]
    ps = closure.unpack(closure.round_bf16(flat).astype(np.float64))
    z = C.forward(ps, feat)[-1][0, 0]
    want = C.delta_tau(z)
    got = dt.reshape(ny, nx)
    tol = 2e-3 if kernel == 1 else 2e-2
    err = np.abs(got - want)[fl].max() / want.max()
    print("kernel %d: max delta_tau error %.3e of %.3e" % (kernel, err, want.max()))
    assert err <= tol
    speed = np.hypot(jx, jy) / r
    assert np.abs(sp.reshape(ny, nx) - speed)[fl].max() <= 2e-3 * speed[fl].max()


@pytest.mark.parametrize("storage,sr", [(0, False), (1, False), (2, False), (1, True), (2, True)])
@pytest.mark.parametrize("kernel", [0, 1, 3, 8, 9, 11])
def test_gpu_closure_step_equals_plain_step_at_the_same_omega(lbm, torch_cuda, storage, sr, kernel):
    """All-zero weights give z = bias = 0, delta_tau = DT_MAX / 2 = 0.125
    exactly, so every fluid cell relaxes with 1 / (1 / omega + 0.125): that
    must reproduce a plain run at that omega bit for bit.  A NaN bias gives
    no valid prediction: every cell takes the plain omega and is counted.
    With stochastic rounding the closure kernels store cell by cell and the
    plain 16-bit kernels two cells per word, from the same random bits: the
    runs still agree bit for bit."""
    if storage == 0 and kernel == 8:
        kernel = 6
    from lbm_gb300 import closure, geometry
    nx, ny, steps = 300, 90, 25
    mask = geometry.random_layout(nx, ny, 0.08, 3, rmin=2.0, inlet_clearance=8)
    L = lbm.load_library()
    om0 = np.float32(1.0 / 0.52)
    om_eff = np.float32(1.0) / (np.float32(1.0) / om0 + np.float32(0.125))

    def run(omega, weights=None):
        with lbm.Lattice(nx, ny, float(omega), lbm.EDGE_CHANNEL, storage) as lat:
            lat.set_tuning(8, kernel)
            lat.set_inlet_velocity(0.07)
            lat.init_equilibrium(1.0, 0.07, 0.0, 1e-2, 2)
            lat.draw_mask(mask)
            if sr:
                lat.set_rounding(lbm.ROUND_STOCHASTIC, 31)
            fb = ctypes.c_uint64(0)
            if weights is not None:
                lbm._check(L.lbm_closure_set_weights(lat.handle, weights.ctypes.data_as(ctypes.c_void_p),
                                                     weights.size))
                lbm._check(L.lbm_closure_enable(lat.handle, 1e9))
                lbm._check(L.lbm_closure_infer(lat.handle))
            lat.iterate(steps)
            if weights is not None:
                lbm._check(L.lbm_closure_fallback_count(lat.handle, ctypes.byref(fb), 1))
            return lat.populations(), fb.value

    zero = np.zeros(closure.N_PARAMS, np.float32)
    nan = zero.copy()
    nan[-1] = np.nan
    ref_eff, _ = run(om_eff)
    ref_0, _ = run(om0)
    got, fb = run(om0, zero)
    np.testing.assert_array_equal(got, ref_eff)
    assert fb == 0
    got, fb = run(om0, nan)
    np.testing.assert_array_equal(got, ref_0)
    assert fb == int(((mask == 0)[:, 1:]).sum()) * steps


@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (1, 2, 63), (2, 9, 64), (1, 17, 65), (3, 8, 132), (4, 80, 256)])
@pytest.mark.parametrize("cin,cout", [(32, 32), (4, 32), (32, 1), (5, 32), (9, 1)])
def test_gpu_conv_tiles_and_channel_remainders(lbm, torch_cuda, n, h, w, cin, cout):
    """Each layer kernel at the edges of its 64 x 8 pixel tiles and 8- and
    4-channel steps, with 16-byte aligned rows and without, against float64.
    Sums of at most 9 * 32 (forward, data) or n h w (weights) products: errors
    stay below 1e-5 of the largest magnitude.  The bias gradient, which can
    cancel to far less than its partial sums, equals the f32 sums in the order
    the kernel documents."""
    torch = torch_cuda
    F = torch.nn.functional
    lib = lbm.load_library()
    gen = torch.Generator().manual_seed(1000 * h + w + cin)
    x = torch.randn(n, cin, h, w, generator=gen)
    wt = torch.randn(cout, cin, 3, 3, generator=gen)
    b = torch.randn(cout, generator=gen)
    g = torch.randn(n, cout, h, w, generator=gen)
    x64, w64, b64 = (t.double().requires_grad_(True) for t in (x, wt, b))
    y64 = torch.relu(F.conv2d(x64, w64, b64, padding=1))
    y64.backward(g.double())
    pad = 1 if h == 17 else 0  # rows that start off a 16-byte boundary

    def dev(t):
        flat = torch.zeros(t.numel() + pad, device="cuda")
        flat[pad:].copy_(t.reshape(-1))
        return flat[pad:]

    def ptr(t):
        return ctypes.c_void_p(t.data_ptr())

    dx, dw, db, dg = dev(x), dev(wt), dev(b), dev(g)
    y = dev(torch.zeros(n, cout, h, w))
    assert lib.lbm_cnn_conv_forward(ptr(dx), n, cin, h, w, ptr(dw), ptr(db), cout, 1, ptr(y), None) == 0
    close(y.cpu().view(n, cout, h, w).numpy(), y64.detach().numpy())
    size = lib.lbm_cnn_weight_scratch_bytes(cin, cout)
    scratch = torch.empty(size // 4, device="cuda")
    gw, gb = torch.empty(wt.numel(), device="cuda"), torch.empty(cout, device="cuda")
    assert lib.lbm_cnn_conv_backward_weight(ptr(dx), ptr(dg), ptr(y), n, cin, h, w, cout, ptr(gw), ptr(gb),
                                            ptr(scratch), size, None) == 0
    close(gw.cpu().view(wt.shape).numpy(), w64.grad.numpy(), atol=1e-6)
    gm = np.where(y.cpu().view(n, cout, h, w).numpy() > 0, g.numpy(), np.float32(0))
    tiles = np.zeros((n * h * ((w + 63) // 64), 64, cout), np.float32)
    rows = np.zeros((n * h, (w + 63) // 64 * 64, cout), np.float32)
    rows[:, :w] = gm.transpose(0, 2, 3, 1).reshape(n * h, w, cout)
    tiles[:] = rows.reshape(tiles.shape)
    blocks = min(len(tiles), 304)
    part = np.zeros((blocks, cout), np.float32)
    for t0 in range(0, len(tiles), blocks):  # one chain per block over its tiles' pixels
        some = tiles[t0:t0 + blocks]
        for px in range(64):
            part[:len(some)] += some[:, px]
    want = np.zeros(cout, np.float32)
    for v in part:
        want += v
    np.testing.assert_array_equal(gb.cpu().numpy(), want)
    if cin == 32:
        gx = dev(torch.zeros(n, cin, h, w))
        assert lib.lbm_cnn_conv_backward_data(ptr(dg), ptr(y), n, cin, h, w, ptr(dw), cout, ptr(gx), None) == 0
        close(gx.cpu().view(n, cin, h, w).numpy(), x64.grad.numpy(), atol=1e-6)


@pytest.mark.parametrize("factor", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("h,w", [(3, 3), (4, 63), (5, 64), (6, 300)])
def test_gpu_coarsened_blocks_by_whole_words_and_by_floats(lbm, torch_cuda, factor, h, w):
    """Blocks read as 8- or 16-byte words against the same populations at an
    address that only floats may be read from: the same bits; and against the
    float64 oracle where every fluid cell is near rest (f32 sums of 9 F^2 terms
    of order one: 1e-5 of the largest average)."""
    torch = torch_cuda
    from lbm_gb300 import closure
    rng = np.random.default_rng(factor * 1000 + h * 10 + w)
    hf, wf = h * factor, w * factor
    W = np.array([1, 4, 1, 4, 16, 4, 1, 4, 1], np.float64)[:, None, None] / 36
    pops = (W * (1 + 0.05 * rng.standard_normal((9, hf, wf)))).astype(np.float32)
    solid = (rng.random((hf, wf)) < 0.3).astype(np.uint8)
    s = torch.from_numpy(solid).cuda()
    lib, stream = lbm.load_library(), None
    out = []
    for shift in (0, 1):
        buf = torch.empty(9 * hf * wf + 4, dtype=torch.float32, device="cuda")
        p = buf[shift:shift + 9 * hf * wf].view(9, hf, wf)
        p.copy_(torch.from_numpy(pops))
        feat = torch.empty((4, h, w), dtype=torch.float32, device="cuda")
        coef = torch.empty((3, h, w), dtype=torch.float32, device="cuda")
        scratch = torch.empty(6 * h * w, dtype=torch.float32, device="cuda")
        solid_c = torch.empty((h, w), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        closure.sample(lib, stream, p, s, factor, feat, coef, scratch, solid_c)
        torch.cuda.synchronize()
        out.append([t.cpu().numpy() for t in (feat, coef, scratch, solid_c)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    want = C.coarsen(pops.astype(np.float64), solid, factor)
    np.testing.assert_array_equal(out[0][3], want[-1])
    avg = out[0][2].reshape(6, h, w)
    rho = np.asarray(want[0])
    np.testing.assert_allclose(avg[0], rho, rtol=0, atol=1e-5 * np.abs(rho).max())
