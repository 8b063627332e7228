"""Learned warm start on the GPU, through the C ABI (i3g_unet_*), against the CPU oracle
oracle/unet_ref.py: the tcgen05 convolution, the network's output and its parameter
gradients; then a small training run that must lower the loss and must never make a
held-out Stokes solve start from a worse residual than the default start."""
import numpy as np
import pytest

import unet_ref as U

pytestmark = pytest.mark.gpu

PAIRS = [(16, 16), (16, 32), (32, 16), (32, 32), (32, 64), (64, 32), (64, 64), (64, 128), (128, 64), (128, 128)]


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    torch.cuda.set_device(0)


def _rows(x):
    """[nz, nx, ny, C] interior -> padded rows [(nz+2)(nx+2)(ny+2), C]."""
    return np.pad(x, ((1, 1), (1, 1), (1, 1), (0, 0))).reshape(-1, x.shape[3])


@pytest.mark.parametrize("cin,cout", PAIRS)
def test_conv_matches_oracle(cin, cout):
    from i3elvis_b200 import warmstart as W
    rng = np.random.default_rng(cin * 1000 + cout)
    dims = (9, 7, 11)     # 11*9*13 = 1287 padded rows: ten 128-row tiles and a partial one
    x = U.bf16(rng.normal(size=dims + (cin,)))
    w = U.bf16(rng.normal(0, 1 / np.sqrt(27 * cin), size=(27, cout, cin)))
    b = rng.normal(0, 0.1, size=cout).astype(np.float32)
    add = U.bf16(rng.normal(0, 0.5, size=dims + (cout,)))
    out = W.conv_host(cin, cout, dims, U.bf16_bits(_rows(x)), U.bf16_bits(w), b, U.bf16_bits(_rows(add)), relu=True)
    ref = np.maximum(U.conv3(x, w, b.astype(np.float64)) + add, 0.0)
    got = out.reshape(dims[0] + 2, dims[1] + 2, dims[2] + 2, cout)
    inner = got[1:-1, 1:-1, 1:-1]
    # FP32 accumulation of <= 27*128 products against float64
    assert np.max(np.abs(inner - ref)) <= 2e-5 * np.max(np.abs(ref)) + 1e-6
    # rows of the zero halo are not written
    halo = got.copy()
    halo[1:-1, 1:-1, 1:-1] = 0
    assert not np.any(halo)


@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 16), (32, 32)])
def test_conv_many_tiles_per_cta(cin, cout):
    """64 x 49 x 33 nodes = 1280 output tiles of 1 x 16 x 8 (4 x 5 x 64, partial in x and y): every
    persistent CTA of the TMA-fed kernel walks four or more tiles, so its box slots and both TMEM
    accumulators are reused many times."""
    from i3elvis_b200 import warmstart as W
    rng = np.random.default_rng(7 + cin * 100 + cout)
    dims = (64, 49, 33)
    x = U.bf16(rng.normal(size=dims + (cin,)))
    w = U.bf16(rng.normal(0, 1 / np.sqrt(27 * cin), size=(27, cout, cin)))
    b = rng.normal(0, 0.1, size=cout).astype(np.float32)
    add = U.bf16(rng.normal(0, 0.5, size=dims + (cout,)))
    out = W.conv_host(cin, cout, dims, U.bf16_bits(_rows(x)), U.bf16_bits(w), b, U.bf16_bits(_rows(add)), relu=True)
    ref = np.maximum(U.conv3(x, w, b.astype(np.float64)) + add, 0.0)
    got = out.reshape(dims[0] + 2, dims[1] + 2, dims[2] + 2, cout)
    assert np.max(np.abs(got[1:-1, 1:-1, 1:-1] - ref)) <= 2e-5 * np.max(np.abs(ref)) + 1e-6
    halo = got.copy()
    halo[1:-1, 1:-1, 1:-1] = 0
    assert not np.any(halo)


def test_conv_brick_fallback_matches_oracle():
    """The same parity cases on the brick kernel, the path taken when the driver offers no
    tensor-map encoder (I3G_CONV_TMA=0), in a child process: the switch is read once per process."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, I3G_CONV_TMA="0")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", os.path.abspath(__file__),
                        "-k", "test_conv_matches_oracle or test_conv_many_tiles_per_cta"],
                       cwd=root, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
    assert " passed" in r.stdout and "skipped" not in r.stdout.splitlines()[-1], r.stdout[-500:]


@pytest.mark.parametrize("cin,cout", PAIRS)
def test_wgrad_matches_oracle(cin, cout):
    """Weight and bias gradients of one layer (tcgen05 for 16/32 channels, CUDA cores for the
    wider layers) against float64 sums of the same BF16 operands, on a grid whose tiles of
    2 x 8 x 8 nodes are partly outside it (ragged in every direction)."""
    from i3elvis_b200 import warmstart as W
    rng = np.random.default_rng(7 * cin + cout)
    dims = (9, 11, 13)
    x = U.bf16(rng.normal(size=dims + (cin,)))
    gy = U.bf16(rng.normal(size=dims + (cout,)))
    dw, db = W.wgrad_host(cin, cout, dims, U.bf16_bits(_rows(x)), U.bf16_bits(_rows(gy)))
    ref = U.conv3_wgrad(x, gy)
    # FP32 sums of 1287 products per weight (in several partial sums) against float64
    assert np.max(np.abs(dw - ref)) <= 1e-5 * np.max(np.abs(ref)), (cin, cout)
    assert np.allclose(db, gy.reshape(-1, cout).sum(axis=0), rtol=1e-5, atol=1e-4)


def _sample(dims, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(dims))
    nz, nx, ny = dims
    # smooth-ish fields so that every level sees structure
    zz, xx, yy = np.meshgrid(np.linspace(0, 1, nz), np.linspace(0, 1, nx), np.linspace(0, 1, ny), indexing="ij")
    le = 21 + 2 * np.sin(3 * xx + 2 * yy) * np.cos(2 * zz) + 0.3 * rng.normal(size=dims)
    ro = 3300 + 80 * np.cos(4 * yy + xx) + 10 * rng.normal(size=dims)
    v = [1e-10 * np.sin(k + 3 * xx * yy + zz) for k in range(3)]
    in5 = np.stack([le.ravel(), ro.ravel()] + [a.ravel() for a in v]).astype(np.float32)
    tg4 = np.stack([1e6 * np.cos(2 * xx + zz).ravel()] + [2e-10 * np.cos(k + xx + 2 * zz).ravel() for k in range(3)])
    return in5, tg4.astype(np.float32), n


def test_network_output_and_gradients_match_oracle():
    from i3elvis_b200.warmstart import UNet
    dims = (9, 17, 9)      # nz, nx, ny
    scales = (21.0, 0.5, 3300.0, 0.0125, 1e-10, 1e6)
    par = U.init_params(seed=11)
    net = UNet(dims[1], dims[2], dims[0], capacity=1, seed=3)
    assert net.nparams == par.size
    net.set_params(par)
    net.set_scales(*scales)
    assert np.array_equal(net.get_params(), par)
    in5, tg4, n = _sample(dims, 12)
    out4, loss, g = net.eval_host(in5, tg4, grads=True)
    ref = U.Net(par, dims, scales, round_bf16=True)
    out_ref = ref.output(in5)
    loss_ref, g_ref = ref.loss_grads(in5, tg4)
    err = np.linalg.norm(out4 - out_ref) / np.linalg.norm(out_ref)
    assert err < 3e-2, err
    assert abs(loss - loss_ref) <= 2e-2 * loss_ref, (loss, loss_ref)
    offs, _ = U.param_offsets()
    worst = 0.0
    for li, ((w, b), (cin, cout)) in enumerate(zip(offs, U.layer_shapes())):
        gw, gr = g[w:w + 27 * cin * cout], g_ref[w:w + 27 * cin * cout]
        e = np.linalg.norm(gw - gr) / max(np.linalg.norm(gr), 1e-30)
        worst = max(worst, e)
        assert e < 1e-1, (li, e)
        eb = np.linalg.norm(g[b:b + cout] - g_ref[b:b + cout]) / max(np.linalg.norm(g_ref[b:b + cout]), 1e-30)
        assert eb < 1e-1, (li, eb)
    assert np.linalg.norm(g - g_ref) / np.linalg.norm(g_ref) < 5e-2
    # padded input channels never receive a gradient
    g0 = g[:27 * 16 * 16].reshape(27, 16, 16)
    assert not np.any(g0[:, :, U.IN_CH:])
    # the same sample through the device data set gives the same loss
    net.set_sample(0, in5, tg4)
    assert abs(net.loss([0]) - loss) <= 1e-6 * loss


def test_gradients_do_not_depend_on_the_pass_before():
    """Weight gradients of the wide layers run on a second stream: a sample's gradients are the same after
    another sample's pass as in a new network, up to the order in which atomic adds meet (partial sums of at
    most a few hundred blocks in FP32: 1e-4 of a layer's norm is far above it), and the narrow layers', whose
    sums have a fixed order, bit for bit."""
    from i3elvis_b200.warmstart import UNet
    dims = (17, 25, 33)
    par = U.init_params(seed=4)
    a, b = _sample(dims, 1), _sample(dims, 2)

    def network():
        net = UNet(dims[1], dims[2], dims[0], capacity=1, seed=3)
        net.set_params(par)
        net.set_scales(21.0, 0.5, 3300.0, 0.0125, 1e-10, 1e6)
        return net
    fresh = network().eval_host(a[0], a[1], grads=True)
    net = network()
    net.eval_host(b[0], b[1], grads=True)
    net.eval_host(b[0])
    again = net.eval_host(a[0], a[1], grads=True)
    assert np.array_equal(fresh[0], again[0])
    offs, _ = U.param_offsets()
    for (w, _), (cin, cout) in zip(offs, U.layer_shapes()):
        x, y = fresh[2][w:w + 27 * cin * cout], again[2][w:w + 27 * cin * cout]
        assert np.linalg.norm(x) > 0
        if max(cin, cout) <= 32:
            assert np.array_equal(x, y), (cin, cout)
        assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(x), (cin, cout)


def test_training_lowers_loss_and_never_worsens_the_start():
    """A short training run on library solves of seeded 17^3 inclusion models lowers the loss;
    on held-out models the learned start (its correction scaled by the residual-minimising
    factor, kept only when its residual is lower) never starts the solve from a higher
    residual than the default start, and the solve still meets the tolerance in about as
    many V-cycles.  The gain itself is printed (and measured at larger sizes by
    ``python -m i3elvis_b200.learned``)."""
    from i3elvis_b200 import learned
    from i3elvis_b200.warmstart import UNet
    case = learned.Case(n=17, mnum=2, count=8, r_km=(15.0, 35.0))
    steps = 1   # cold starts: on some 17^3 seeds the second step's solve stalls near 2e-5
    net = UNet(case.n, case.n, case.n, capacity=32 * steps, seed=2)
    slots = learned.record(net, case, range(100, 132), steps)
    learned.fit_scales(net, slots)
    hist = learned.train(net, slots, iters=400, batch=4, lr=2e-3)
    first, last = float(np.mean(hist[:10])), float(np.mean(hist[-20:]))
    assert last < 0.7 * first, (first, last)
    rows = learned.compare(net, case, range(900, 906), steps)
    print("learned warm start, 17^3 held-out models:", learned.summarize(rows))
    for r in rows:
        assert r["guess_used"] in (0, 1), r
        # the solve starts from the better of the two starts of its own state
        assert r["learned_rel0"] <= r["rel_default"] * (1 + 1e-9), r
        # ... and never from a worse one than the separate default-start context on the same
        # state (one step per seed: both contexts hold identical models)
        assert r["learned_rel0"] <= r["default_rel0"] * (1 + 1e-9), r
        assert r["alpha"] >= 0.0, r
    print("guess accepted on", sum(r["guess_used"] == 1 for r in rows), "of", len(rows), "held-out solves")
    d = float(np.mean([r["default_cycles"] for r in rows]))
    g = float(np.mean([r["learned_cycles"] for r in rows]))
    assert g <= d + 3.0, (g, d)
