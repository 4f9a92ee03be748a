"""Learned-guess network: the CPU restatement (its gradients against finite
differences) and the device BF16 kernels against it.

Tolerances: the device GEMM against an FP64 product of the same BF16
operands 1e-5 relative (FP32 accumulation); network outputs and gradients
against the restatement with the same BF16 rounding points 2e-2 relative
in the L2 norm (a BF16 rounding that flips on FP32-vs-FP64 accumulation
propagates one BF16 ulp, 2^-8, through the layers that follow).
"""
import numpy as np
import pytest

from oracle import unet_oracle as uo

from helpers import rel_l2


def _tiny(rng, channels=(4, 4, 6, 6), n_in=5, n_out=3):
    convs = []
    cin = n_in
    for ch in channels:
        convs.append((rng.standard_normal((ch, 9 * cin)) * 0.3, rng.standard_normal(ch) * 0.1, True, True))
        convs.append((rng.standard_normal((ch, 9 * ch)) * 0.3, rng.standard_normal(ch) * 0.1, True, True))
        cin = ch
    for lv in range(len(channels) - 2, -1, -1):
        cin = channels[lv + 1] + channels[lv]
        convs.append((rng.standard_normal((channels[lv], 9 * cin)) * 0.3, rng.standard_normal(channels[lv]) * 0.1,
                      True, True))
        convs.append((rng.standard_normal((channels[lv], 9 * channels[lv])) * 0.3,
                      rng.standard_normal(channels[lv]) * 0.1, True, True))
    convs.append((rng.standard_normal((n_out, channels[0])) * 0.3, rng.standard_normal(n_out) * 0.1, False, False))
    return convs


@pytest.mark.parametrize("periodic", [0, 1])
def test_oracle_gradients_match_finite_differences(periodic):
    rng = np.random.default_rng(5)
    channels = (4, 4, 6, 6)
    convs = _tiny(rng, channels)
    x = rng.standard_normal((1, 8, 8, 5))
    net = uo.OracleUNet(convs, channels, bf16_points=False)
    dout = rng.standard_normal(net.forward(x, periodic).shape)
    grads = net.backward(dout, periodic)

    def loss():
        return float(np.sum(uo.OracleUNet(convs, channels, bf16_points=False).forward(x, periodic) * dout))

    h = 1e-6
    for i in (0, 3, 7, len(convs) - 2, len(convs) - 1):
        w, b, k3, act = convs[i]
        for (r, c) in ((0, 0), (w.shape[0] - 1, w.shape[1] - 1), (w.shape[0] // 2, w.shape[1] // 3)):
            old = w[r, c]
            w[r, c] = old + h
            lp = loss()
            w[r, c] = old - h
            lm = loss()
            w[r, c] = old
            fd = (lp - lm) / (2 * h)
            assert abs(fd - grads[i][0][r, c]) <= 1e-6 * max(1.0, abs(fd)), (i, r, c)
        old = b[0]
        b[0] = old + h
        lp = loss()
        b[0] = old - h
        lm = loss()
        b[0] = old
        assert abs((lp - lm) / (2 * h) - grads[i][1][0]) <= 1e-6 * max(1.0, abs(grads[i][1][0]))


def test_bf16_rounding_is_nearest_even():
    torch = pytest.importorskip("torch")
    x = np.random.default_rng(1).standard_normal(10000) * np.logspace(-8, 8, 10000)
    ref = torch.tensor(x, dtype=torch.float32).to(torch.bfloat16).to(torch.float64).numpy()
    assert np.array_equal(uo.bf16(x), ref)


# ---------------------------------------------------------------------
# device kernels
# ---------------------------------------------------------------------
def _net_from_oracle(convs, channels, n_out):
    import torch
    from cism_b200 import net as netmod

    w0, _, k30, _ = convs[0]
    n_in = w0.shape[1] // 9 if k30 else w0.shape[1]  # the restatement's input channels
    dev = netmod.UNet(n_out=n_out, channels=channels, n_in=n_in)
    for cv, (w, b, k3, act) in zip(dev.convs(), convs):
        cv.w.copy_(torch.tensor(w, dtype=torch.float32))
        cv.b.copy_(torch.tensor(b, dtype=torch.float32))
        cv.refresh()
    return dev


def _device_setup(periodic, B=2, H=16, W=24, channels=(8, 8, 16, 16), n_out=8, seed=7):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(seed)
    convs = _tiny(rng, channels, n_out=n_out)
    # the device keeps FP32 master weights; both sides see them rounded to BF16
    convs = [(uo.bf16(w).astype(np.float32).astype(np.float64), b.astype(np.float32).astype(np.float64), k3, a)
             for (w, b, k3, a) in convs]
    x = uo.bf16(rng.standard_normal((B, H, W, 5)))
    dev = _net_from_oracle(convs, channels, n_out)
    xt = torch.tensor(x, dtype=torch.float32, device="cuda").to(torch.bfloat16).contiguous()
    return torch, rng, convs, x, dev, xt


@pytest.mark.gpu
@pytest.mark.parametrize("kernel", ["tma", "tc", "mma"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (100, 40, 72), (7, 130, 8), (256, 96, 1160), (300, 24, 48),
                                   (96, 1440, 64), (130, 64, 1000), (200, 128, 640), (32, 288, 8192),
                                   (64, 200, 4104)])
def test_gemm_matches_bf16_product(shape, kernel):
    # the tcgen05 kernels -- operands by TMA boxes into a four-stage ring
    # ("tma", the default) or by register-staged loads in two stages ("tc");
    # 128 x 64, 128 x 32 (at most 32 columns) and 128 x 128 tiles (N = 96,
    # 128, 200); the last two shapes split K, the weight-gradient form -- and
    # the mma.sync one against the
    # FP64 product of the same BF16 operands
    torch = pytest.importorskip("torch")
    from cism_b200 import net as netmod

    M, N, K = shape
    rng = np.random.default_rng(3)
    a = uo.bf16(rng.standard_normal((M, K)))
    b = uo.bf16(rng.standard_normal((N, K)))
    bias = rng.standard_normal(N).astype(np.float32)
    at = torch.tensor(a, dtype=torch.float32, device="cuda").to(torch.bfloat16).contiguous()
    bt = torch.tensor(b, dtype=torch.float32, device="cuda").to(torch.bfloat16).contiguous()
    out = torch.empty((M, N), dtype=torch.float32, device="cuda")
    biast = torch.tensor(bias, device="cuda")
    netmod.gemm_tn(at, bt, out, biast, M, N, K, K, K, N, kernel=kernel)
    ref = a @ b.T + bias
    assert rel_l2(out.cpu().numpy(), ref) < 1e-5
    netmod.gemm_tn(at, bt, out, None, M, N, K, K, K, N, accum=True, kernel=kernel)
    assert rel_l2(out.cpu().numpy(), 2 * (a @ b.T) + bias) < 1e-5
    assert netmod.gemm_status() == 0  # no bounded wait of the tcgen05 kernel ran out


@pytest.mark.gpu
@pytest.mark.parametrize("periodic", [0, 1])
def test_unet_forward_and_gradients_match_oracle(periodic):
    torch, rng, convs, x, dev, xt = _device_setup(periodic)
    channels = (8, 8, 16, 16)
    ref = uo.OracleUNet(convs, channels, bf16_points=True)
    yo = ref.forward(x, periodic)
    yd = dev.forward(xt, periodic, train=True)
    torch.cuda.synchronize()
    assert rel_l2(yd.cpu().numpy(), yo) < 2e-2
    dout = rng.standard_normal(yo.shape)
    go = ref.backward(dout, periodic)
    dev.backward(torch.tensor(dout, dtype=torch.float32, device="cuda"))
    torch.cuda.synchronize()
    for cv, (gw, gb) in zip(dev.convs(), go):
        assert rel_l2(cv.gw.cpu().numpy(), gw) < 2e-2
        assert rel_l2(cv.gb.cpu().numpy(), gb) < 2e-2


@pytest.mark.gpu
def test_training_steps_reduce_the_loss():
    torch, rng, convs, x, dev, xt = _device_setup(1)
    from cism_b200 import net as netmod

    target = torch.tensor(np.tanh(x[..., :1].repeat(8, axis=-1)), dtype=torch.float32, device="cuda")
    mask = torch.ones(x.shape[:3], dtype=torch.float32, device="cuda")
    losses = []
    for t in range(1, 41):
        y = dev.forward(xt, 1, train=True)
        loss, dy = netmod.mse(y, target, mask)
        dev.backward(dy)
        dev.adam(3e-3, t)
        losses.append(loss)
    assert losses[-1] < 0.5 * losses[0]


def test_bindings_match_the_c_declarations():
    """Every ctypes signature of net.py has the parameter count of its
    extern "C" definition in net_kernels.cu (the library loads without a GPU)."""
    import os
    import re

    from cism_b200 import net as netmod

    src = open(os.path.join(os.path.dirname(netmod.__file__), "csrc", "net_kernels.cu")).read()
    body = src[src.index('extern "C" {'):]
    decl = {m.group(1): len([a for a in m.group(2).split(",") if a.strip()])
            for m in re.finditer(r"\bint\s+(bpnet_\w+)\s*\(([^)]*)\)", body)}
    L = netmod.lib()
    assert decl
    for name, n in decl.items():
        assert len(getattr(L, name).argtypes) == n, name


@pytest.mark.gpu
def test_shipped_network_reduces_iterations_on_held_out_slab(ctx):
    """The trained weights shipped in cism_b200/weights: on a slab drawn from
    the family with a seed outside the training seeds, the learned start
    needs fewer Picard and PCG iterations than the zero start, and both meet
    the same convergence criteria (Picard max speed change 1e-4, PCG 1e-8),
    so the answers agree to the Picard tolerance's scale."""
    import os

    from cism_b200 import configs, guess, net as netmod, solver

    path = os.path.join(os.path.dirname(netmod.__file__), "weights", "unet_slab.npz")
    model = netmod.UNet.load(path)
    m = configs.random_slab(np.random.default_rng(424242), n=96).copy(pcg_maxiters=3000)
    u0, v0, _, st0 = ctx.velo_higher_solve(m)
    gu, gv = guess.learned_guesses(model, [m])[0]
    prep, _, _ = solver.prepare(m)
    u1, v1, _, st1 = ctx.solve_prepared(prep, gu, gv)
    assert st0["status"] == 0 and st1["status"] == 0
    js, is_ = m.owned_vertex_slices()
    guess_err = rel_l2([gu[js, is_], gv[js, is_]], [u0[js, is_], v0[js, is_]])
    assert guess_err < 0.2
    assert st1["picard_iters"] < st0["picard_iters"]
    assert st1["pcg_iters_total"] < 0.8 * st0["pcg_iters_total"]
    assert rel_l2([u1, v1], [u0, v0]) < 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape", [(1, 2, 2, 8), (2, 6, 10, 6), (1, 4, 34, 24), (3, 8, 2, 33), (1, 2, 6, 1032)])
def test_pointwise_kernels_match_torch(shape, offset):
    """The 16-byte forms and the element forms (channel counts that are not
    multiples of 4 or 8; addresses one element past a 16-byte boundary) of the
    data-movement and pointwise kernels.  Copies and sums of at most nine terms
    in the kernels' order: equal bit for bit; GELU and its gradient to 4 ulp of
    FP32 before the BF16 rounding (one BF16 ulp, 2^-8); column sums of N terms
    in FP32 to N 2^-24 of the sum of magnitudes."""
    torch = pytest.importorskip("torch")
    from cism_b200 import net as netmod

    L = netmod.lib()
    B, H, W, C = shape
    P = B * H * W
    g = torch.Generator(device="cuda").manual_seed(P + C)

    def rand(*n, dtype=torch.float32):
        buf = torch.randn(int(np.prod(n)) + 8, generator=g, device="cuda").to(dtype)
        return buf[offset:offset + int(np.prod(n))].view(*n)

    def new(*n, dtype=torch.float32):
        buf = torch.full((int(np.prod(n)) + 8,), float("nan"), device="cuda").to(dtype)
        return buf[offset:offset + int(np.prod(n))].view(*n)

    bf = torch.bfloat16
    s = netmod._s()
    p = netmod._p
    x = rand(B, H, W, C, dtype=bf)
    for periodic in (0, 1):
        Kp = netmod.ceil8(9 * C)
        col = new(P, Kp, dtype=bf)
        assert L.bpnet_im2col(p(x), p(col), B, H, W, C, Kp, periodic, s) == 0
        pad = torch.nn.functional.pad(x.float().permute(0, 3, 1, 2), (1, 1, 1, 1),
                                      mode="circular" if periodic else "constant")
        ref = torch.stack([pad[:, :, dy:dy + H, dx:dx + W] for dy in range(3) for dx in range(3)], 1)
        ref = ref.permute(0, 3, 4, 1, 2).reshape(P, 9 * C).to(bf)
        assert torch.equal(col[:, :9 * C], ref) and not bool((col[:, 9 * C:] != 0).any())
        d = rand(P, 9 * C)
        dx_ = new(B, H, W, C)
        assert L.bpnet_col2im(p(d), p(dx_), B, H, W, C, 9 * C, periodic, s) == 0
        dd = d.view(B, H, W, 9, C)
        acc = torch.zeros(B, H, W, C, device="cuda")
        for tap in range(9):
            ty, tx = tap // 3 - 1, tap % 3 - 1
            r = torch.roll(dd[..., tap, :], (ty, tx), (1, 2))
            if not periodic:
                r = r.clone()
                if ty: r[:, 0 if ty > 0 else H - 1] = 0
                if tx: r[:, :, 0 if tx > 0 else W - 1] = 0
            acc = acc + r
        assert torch.equal(dx_, acc)
    z, dy = rand(P, C), rand(P, C)
    y = new(P, C + 8, dtype=bf)
    assert L.bpnet_act(p(z), p(y), P, C, C + 8, 8, 1, s) == 0
    ref = torch.nn.functional.gelu(z.double())
    assert bool(((y[:, 8:].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-7).all())
    dz, dzb, db, part = new(P, C), new(P, C, dtype=bf), new(C), new((P + 256) * C)
    assert L.bpnet_act_grad(p(z), p(dy), p(dz), P, C, C, 0, 1, s) == 0
    assert L.bpnet_act_grad_sum(p(z), p(dy), p(dzb), p(db), p(part), P, C, 1, s) == 0
    assert torch.equal(dzb, dz.to(bf)) and torch.equal(part[:P * C].view(P, C), dz)
    db1 = new(C)
    assert L.bpnet_colsum(p(dz), p(db1), P, C, s) == 0
    assert torch.equal(db, db1)
    mag = dz.double().abs().sum(0)
    assert bool(((db.double() - dz.double().sum(0)).abs() <= (P + 8) * 2.0 ** -24 * mag).all())
    c2 = new(B, H // 2, W // 2, C, dtype=bf)
    assert L.bpnet_pool(p(x), p(c2), B, H, W, C, s) == 0
    f = x.float()
    ref = f[:, ::2, ::2] + f[:, ::2, 1::2]
    ref = 0.25 * ((ref + f[:, 1::2, ::2]) + f[:, 1::2, 1::2])
    assert torch.equal(c2, ref.to(bf))
    cat = new(P, C + 8, dtype=bf)
    assert L.bpnet_up(p(c2), p(cat), B, H // 2, W // 2, C, C + 8, 0, s) == 0
    up = c2.repeat_interleave(2, 1).repeat_interleave(2, 2).reshape(P, C)
    assert torch.equal(cat[:, :C], up)
    assert L.bpnet_copy_slice(p(x), p(cat), P, C, C + 8, 8, s) == 0
    assert torch.equal(cat[:, 8:], x.reshape(P, C))
    dcat, a = rand(P, C + 8), rand(P, C)
    b = a.clone() if offset == 0 else new(P, C)
    b.copy_(a)
    assert L.bpnet_add_slice(p(dcat), p(b), P, C, C + 8, 8, s) == 0
    assert torch.equal(b, a + dcat[:, 8:])
    ug = new(B, H // 2, W // 2, C)
    assert L.bpnet_up_grad(p(dcat), p(ug), B, H // 2, W // 2, C, C + 8, 0, s) == 0
    q = dcat[:, :C].reshape(B, H, W, C)
    assert torch.equal(ug, ((q[:, ::2, ::2] + q[:, ::2, 1::2]) + q[:, 1::2, ::2]) + q[:, 1::2, 1::2])
    pg = new(B, H, W, C)
    pg.copy_(a.view(B, H, W, C))
    assert L.bpnet_pool_grad(p(ug), p(pg), B, H, W, C, C, 0, s) == 0
    assert torch.equal(pg, a.view(B, H, W, C) + 0.25 * ug.repeat_interleave(2, 1).repeat_interleave(2, 2))
    torch.cuda.synchronize()


@pytest.mark.gpu
@pytest.mark.parametrize("a_mn", [0, 1])
@pytest.mark.parametrize("b_mn", [0, 1])
@pytest.mark.parametrize("shape", [(64, 64, 64), (24, 40, 72), (136, 136, 8), (96, 864, 1000), (128, 1152, 2056),
                                   (32, 288, 8192), (264, 56, 4168), (40, 200, 16)])
def test_gemm_of_either_operand_order(shape, a_mn, b_mn):
    """K-major and MN-major operands of the TMA-fed kernel: rows that end
    within a box of 64 and within a tile of 128, K that is not a multiple of a
    slice or of 16, each tile width, split K; against the FP64 product of the
    same BF16 operands (1e-5, FP32 accumulation), and bitwise the register-staged
    kernel's product of the same operands in K-major order."""
    torch = pytest.importorskip("torch")
    from cism_b200 import net as netmod

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    A = a.t().contiguous() if a_mn else a
    B = b.t().contiguous() if b_mn else b
    out = torch.full((M, N + 8), float("nan"), device="cuda")
    assert netmod.gemm_major(a_mn, b_mn, A, B, out, M, N, K, M if a_mn else K, N if b_mn else K, N + 8)
    ref = a.double() @ b.double().t()
    assert float((out[:, :N].double() - ref).norm() / ref.norm()) < 1e-5
    assert bool(out[:, N:].isnan().all())
    tc = torch.empty((M, N), device="cuda")
    netmod.gemm_tn(a, b, tc, None, M, N, K, K, K, N, kernel="tc")
    assert torch.equal(out[:, :N], tc)
    assert netmod.gemm_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(130, 24, 56), (256, 96, 864), (64, 128, 1152)])
@pytest.mark.parametrize("act", [0, 1])
def test_gemm_with_its_activation(shape, act):
    """The fused epilogue against the separate kernels: bitwise."""
    torch = pytest.importorskip("torch")
    from cism_b200 import net as netmod

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda")
    z, z2 = torch.empty(M, N, device="cuda"), torch.empty(M, N, device="cuda")
    y, y2, y3 = (torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    L, p, s = netmod.lib(), netmod._p, netmod._s()
    assert L.bpnet_gemm_act(p(a), p(b), p(z), p(bias), p(y), M, N, K, K, K, act, s) == 0
    assert L.bpnet_gemm_act(p(a), p(b), None, p(bias), p(y3), M, N, K, K, K, act, s) == 0
    netmod.gemm_tn(a, b, z2, bias, M, N, K, K, K, N)
    assert L.bpnet_act(p(z2), p(y2), M, N, N, 0, act, s) == 0
    assert torch.equal(z, z2) and torch.equal(y, y2) and torch.equal(y, y3)


@pytest.mark.gpu
@pytest.mark.parametrize("periodic", [0, 1])
@pytest.mark.parametrize("shape", [(1, 8, 8, 32, 32), (2, 13, 26, 64, 96), (1, 130, 6, 32, 64), (1, 2, 200, 96, 32),
                                   (3, 64, 48, 192, 256), (1, 104, 184, 96, 32), (1, 104, 184, 64, 64),
                                   (1, 1, 1, 32, 32)])
def test_direct_input_gradient(shape, periodic):
    """The input gradient formed tap by tap in one kernel against the product
    over all taps and the gather: bitwise (the same products, the same order);
    rectangles that end outside the grid, single-row and single-slice cases,
    wrapped and zero borders."""
    torch = pytest.importorskip("torch")
    from cism_b200 import net as netmod

    B, H, W, cin, cout = shape
    P, Kp = B * H * W, 9 * cin
    g = torch.Generator(device="cuda").manual_seed(P)
    L, p, s = netmod.lib(), netmod._p, netmod._s()
    dzb = torch.randn(P, cout, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(cout, Kp, generator=g, device="cuda").to(torch.bfloat16)
    dx = torch.full((P, cin), float("nan"), device="cuda")
    assert L.bpnet_dgrad3(p(dzb), p(w), p(dx), B, H, W, cin, cout, Kp, periodic, s) == 0
    dcol = torch.empty(P, Kp, device="cuda")
    assert netmod.gemm_major(False, True, dzb, w, dcol, P, Kp, cout, cout, Kp, Kp)
    ref = torch.empty(P, cin, device="cuda")
    assert L.bpnet_col2im(p(dcol), p(ref), B, H, W, cin, Kp, periodic, s) == 0
    assert torch.equal(dx, ref)
    assert netmod.gemm_status() == 0


@pytest.mark.parametrize("M,N,K,registers", [(296 * 128, 32, 64, 1), (295 * 128, 32, 64, 0), (295 * 128 + 1, 32, 8, 1),
                                             (296 * 128, 32, 72, 0), (148 * 128, 128, 56, 1), (147 * 128, 128, 56, 0),
                                             (296 * 128, 96, 56, 1), (961, 32, 56, 0), (2 ** 20, 1152, 64, 1)])
def test_route_of_products_of_one_slice(M, N, K, registers):
    """Products of one K slice (64) with 296 tiles or more are the
    register-staged kernel's, and their activation, for whole groups of four
    channels, a pass of its own."""
    pytest.importorskip("torch")
    from cism_b200 import net as netmod

    L = netmod.lib()
    assert L.bpnet_gemm_by_registers(M, N, K) == registers
    assert L.bpnet_act_apart(M, N, K) == registers
    assert L.bpnet_act_apart(M, N + 2, K) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(296 * 128, 32, 56), (296 * 128 - 127, 32, 8), (295 * 128, 32, 56),
                                   (148 * 128, 128, 64), (300 * 128, 22, 32), (300 * 128, 24, 72)])
def test_products_of_one_slice_are_the_same_on_every_route(shape):
    """Either kernel, the fused activation and the separate one: the same sums
    in the same order, so bitwise."""
    torch = pytest.importorskip("torch")
    from cism_b200 import net as netmod

    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda")
    z = [torch.empty(M, N, device="cuda") for _ in range(4)]
    y = [torch.empty(M, N, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    L, p, s = netmod.lib(), netmod._p, netmod._s()
    for out, kernel in zip(z, ("tma", "tc", None)):
        netmod.gemm_tn(a, b, out, bias, M, N, K, K, K, N, kernel=kernel)
    assert L.bpnet_gemm_act(p(a), p(b), p(z[3]), p(bias), p(y[0]), M, N, K, K, K, 1, s) == 0
    assert L.bpnet_gemm_act(p(a), p(b), None, p(bias), p(y[1]), M, N, K, K, K, 1, s) == 0
    assert L.bpnet_act(p(z[0]), p(y[2]), M, N, N, 0, 1, s) == 0
    assert all(torch.equal(z[0], other) for other in z[1:])
    assert all(torch.equal(y[2], other) for other in y[:2])
