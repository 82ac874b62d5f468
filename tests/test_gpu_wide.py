"""Widened configuration (benchmark configuration 5: 56x56 input, 64 maps) on the GPU against the generalised
oracle; the same kernels at 28x28 / 6 maps against the fused path of the reference net."""
import numpy as np
import pytest

from conftest import rel_err, scaled_err

pytestmark = pytest.mark.gpu


def wide_inputs(n, H, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((n, H, H), dtype=np.float32)
    x[rng.random((n, H, H)) < 0.8] = 0.0          # MNIST-like sparsity
    labels = rng.integers(0, 10, n).astype(np.uint32)
    return x, labels


def wide_params(ob, H, F, seed):
    rng = np.random.default_rng(seed)
    n = ob.param_count(H, F)
    p = rng.uniform(-0.5, 0.5, n).astype(np.float32)
    S = F * ((H - 4) // 4) ** 2
    p[F * 25 + F + 17: F * 25 + F + 17 + 10 * S] *= np.float32(6.0 / np.sqrt(S))   # keep the FC out of saturation
    return p


def blocks(H, F):
    S = F * ((H - 4) // 4) ** 2
    o = [0, F * 25, F * 25 + F, F * 25 + F + 16, F * 25 + F + 17, F * 25 + F + 17 + 10 * S, F * 25 + F + 27 + 10 * S]
    return dict(zip(["Wc", "bc", "Ws", "bs", "Wf", "bf"], zip(o[:-1], o[1:])))


@pytest.mark.parametrize("H,F,n", [(56, 64, 6), (56, 64, 1), (28, 6, 40), (32, 5, 9)])
def test_wide_forward_and_gradient_match_oracle(cuda, pkg, ob, H, F, n):
    x, labels = wide_inputs(n, H, 1)
    params = wide_params(ob, H, F, 2)
    net = pkg.WideNet(H, F)
    assert net.n_params == ob.param_count(H, F)
    net.set_params(params)
    d_x = cuda.from_numpy(x).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
    net.forward(d_x, n, d_out, d_arg)
    cuda.cuda.synchronize()
    ref_out, ref_arg = ob.forward_batch(params, x, H=H, F=F)
    assert rel_err(d_out.cpu().numpy(), ref_out) < 1e-5
    top2 = np.sort(ref_out, axis=1)
    ok = (top2[:, -1] - top2[:, -2]) > 1e-5 * top2[:, -1]
    assert np.array_equal(d_arg.cpu().numpy()[ok], ref_arg[ok])
    d_g = cuda.full((net.n_padded,), 9.0, dtype=cuda.float32, device="cuda")
    net.grad_batch(d_x, d_lab, n, d_g)
    cuda.cuda.synchronize()
    g = d_g.cpu().numpy()
    G, err = ob.grad_batch(params, x, labels, H=H, F=F)
    for name, (lo, hi) in blocks(H, F).items():
        assert scaled_err(g[lo:hi], G[lo:hi]) < 1e-5, name
    assert abs(g[net.n_params + 1] - err) < 1e-5 * max(err, 1.0)
    assert g[net.n_params] == 0 and not g[net.n_params + 2:].any()
    # one minibatch step
    net.apply_update(d_g, 0.1 / n)
    cuda.cuda.synchronize()
    want = ob.apply_update(params, G, 0.1, n)
    assert scaled_err(net.get_params(), want) < 1e-5


def test_wide_kernels_agree_with_the_fused_reference_net(cuda, pkg, params0):
    """At 28x28 / 6 maps the widened path and the fused path are two implementations of one net."""
    n = 300
    images, labels = pkg.synth.synth_images(61, n)
    d_x = cuda.from_numpy(images).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    wide = pkg.WideNet(28, 6)
    wide.set_params(params0)
    net = pkg.Net(0)
    net.set_params(params0)
    o1 = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    o2 = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    wide.forward(d_x, n, o1, None)
    net.forward(d_x, n, o2, None)
    g1 = cuda.zeros(wide.n_padded, dtype=cuda.float32, device="cuda")
    g2 = cuda.zeros(2368, dtype=cuda.float32, device="cuda")
    wide.grad_batch(d_x, d_lab, n, g1)
    net.grad_batch(d_x, d_lab, n, g2)
    cuda.cuda.synchronize()
    assert rel_err(o1.cpu().numpy(), o2.cpu().numpy()) < 1e-5
    assert scaled_err(g1.cpu().numpy()[:2343], g2.cpu().numpy()[:2343]) < 1e-5


def test_wide_full_batch_runs_and_is_deterministic(cuda, pkg, ob):
    """benchmark configuration 5 size: batch 1,024 of 56x56 images, forward + backward twice, bit-identical."""
    H, F, n = 56, 64, 1024
    x, labels = wide_inputs(n, H, 3)
    net = pkg.WideNet(H, F)
    net.set_params(wide_params(ob, H, F, 4))
    d_x = cuda.from_numpy(x).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    ga = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
    gb = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
    net.grad_batch(d_x, d_lab, n, ga)
    net.grad_batch(d_x, d_lab, n, gb)
    cuda.cuda.synchronize()
    assert cuda.equal(ga, gb) and bool(cuda.isfinite(ga).all())
    # additivity over shards (what data-parallel training relies on)
    g1 = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
    g2 = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
    net.grad_batch(d_x[:512], d_lab[:512], 512, g1)
    net.grad_batch(d_x[512:], d_lab[512:], 512, g2)
    cuda.cuda.synchronize()
    s = (g1.double() + g2.double()).cpu().numpy()
    assert scaled_err(ga.cpu().numpy()[:net.n_params], s[:net.n_params]) < 1e-5


@pytest.mark.parametrize("mode,tol", [(2, 1e-5), (1, 3e-3)])
@pytest.mark.parametrize("H,F,n", [(56, 64, 1), (56, 64, 5), (28, 64, 33)])
def test_tensor_core_conv_matches_oracle(cuda, pkg, ob, H, F, n, mode, tol):
    """conv = 2: three passes of fp16 parts on tcgen05 keep the 1e-5 bar; conv = 1: one pass, 11 significant bits."""
    x, labels = wide_inputs(n, H, 5)
    params = wide_params(ob, H, F, 6)
    net = pkg.WideNet(H, F)
    net.set_params(params)
    net.set_option("conv", mode)
    d_x = cuda.from_numpy(x).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    net.forward(d_x, n, d_out, None)
    cuda.cuda.synchronize()
    assert net.status() == 0
    ref_out, _ = ob.forward_batch(params, x, H=H, F=F)
    assert rel_err(d_out.cpu().numpy(), ref_out) < tol
    d_g = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
    net.grad_batch(d_x, d_lab, n, d_g)
    cuda.cuda.synchronize()
    assert net.status() == 0
    G, _ = ob.grad_batch(params, x, labels, H=H, F=F)
    g = d_g.cpu().numpy()
    for name, (lo, hi) in blocks(H, F).items():
        assert scaled_err(g[lo:hi], G[lo:hi]) < tol * (1 if mode == 2 else 10), name


@pytest.mark.parametrize("H,F,n,mode,sigmoid,offset", [
    (8, 64, 1, 2, 1, 0),        # one window per image: half a row group is empty
    (8, 64, 300, 2, 0, 0),      # two image groups per FC cluster
    (12, 64, 601, 1, 1, 0),     # four, the last one ragged
    (28, 64, 33, 2, 2, 0),      # row groups of an image end in the middle of a group set
    (56, 128, 3, 2, 1, 0),      # two groups of maps
    (56, 64, 70, 2, 1, 0),      # units of a CTA: several hand-overs of the gradient accumulators and a rest
    (28, 64, 9, 2, 1, 1),       # images not 16-byte aligned: the fp32 path
    (30, 64, 9, 2, 1, 0),       # a height that is not a multiple of 4: the fp32 path
    (28, 16, 33, 2, 1, 0),      # maps that are not a multiple of 64: the fp32 path, in either mode
    (28, 16, 33, 1, 1, 0),
])
def test_tensor_core_edges_match_oracle(cuda, pkg, ob, H, F, n, mode, sigmoid, offset):
    x, labels = wide_inputs(n, H, 9)
    params = wide_params(ob, H, F, 10)
    net = pkg.WideNet(H, F)
    net.set_params(params)
    net.set_option("conv", mode)
    net.set_option("fast_sigmoid", sigmoid)
    d_x = cuda.zeros((n * H * H + offset,), dtype=cuda.float32, device="cuda")[offset:]
    d_x.copy_(cuda.from_numpy(x.reshape(-1)))
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_g = cuda.full((net.n_padded,), 9.0, dtype=cuda.float32, device="cuda")
    net.forward(d_x, n, d_out, None)
    net.grad_batch(d_x, d_lab, n, d_g)
    cuda.cuda.synchronize()
    assert net.status() == 0
    tol = 1e-5 if mode == 2 else 3e-3
    ref_out, _ = ob.forward_batch(params, x, H=H, F=F)
    assert rel_err(d_out.cpu().numpy(), ref_out) < tol
    G, err = ob.grad_batch(params, x, labels, H=H, F=F)
    g = d_g.cpu().numpy()
    for name, (lo, hi) in blocks(H, F).items():
        assert scaled_err(g[lo:hi], G[lo:hi]) < tol * (1 if mode == 2 else 10), name
    assert abs(g[net.n_params + 1] - err) < tol * max(err, 1.0)
    assert g[net.n_params] == 0 and not g[net.n_params + 2:].any()


@pytest.mark.parametrize("mode", [0, 2])
def test_wide_full_batch_matches_oracle(cuda, pkg, ob, mode):
    """Benchmark configuration 5 at its full size (batch 1,024 of 56x56 images, 64 maps) against the
    generalised oracle: forward outputs within 1e-5 relative, every gradient block within 1e-5 of its
    largest magnitude, for the fp32 SIMT convolution (conv = 0) and the three-pass tensor-core
    convolution (conv = 2)."""
    H, F, n = 56, 64, 1024
    x, labels = wide_inputs(n, H, 7)
    params = wide_params(ob, H, F, 8)
    net = pkg.WideNet(H, F)
    net.set_params(params)
    net.set_option("conv", mode)
    d_x = cuda.from_numpy(x).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
    net.forward(d_x, n, d_out, d_arg)
    d_g = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
    net.grad_batch(d_x, d_lab, n, d_g)
    cuda.cuda.synchronize()
    assert net.status() == 0
    ref_out, ref_arg = ob.forward_batch(params, x, H=H, F=F, threads=0)
    # The FC of this net adds 10,816 products: two fp32 evaluations in different orders already differ
    # by more than 1e-5 on some of the 10,240 outputs, so the yardstick here is the fp64 oracle -- 1e-5, or
    # twice the fp32 oracle's own distance from it where that is larger.
    ref64, _ = ob.forward_batch(params, x, H=H, F=F, threads=0, dtype=np.float64)
    e_lib, e_or = rel_err(d_out.cpu().numpy(), ref64), rel_err(ref_out, ref64)
    print("conv mode %d: outputs against the fp64 oracle: library %.3e, fp32 oracle %.3e" % (mode, e_lib, e_or))
    assert e_lib < max(1e-5, 2 * e_or)
    top2 = np.sort(ref_out, axis=1)
    ok = (top2[:, -1] - top2[:, -2]) > 1e-5 * top2[:, -1]
    print("conv mode %d: %d of %d rows below the 1e-5 argmax margin" % (mode, int((~ok).sum()), n))
    assert np.array_equal(d_arg.cpu().numpy()[ok], ref_arg[ok]) and (~ok).sum() <= 2
    # gradients: sums over 1,024 images (and 2,704 positions for the conv filter) -- the fp64 oracle
    # is the yardstick, with the fp32 oracle's own distance from it as the floor of what fp32 can deliver
    G, err = ob.grad_batch(params, x, labels, H=H, F=F, threads=0)
    G64, err64 = ob.grad_batch(params, x, labels, H=H, F=F, threads=0, dtype=np.float64)
    g = d_g.cpu().numpy()
    for name, (lo, hi) in blocks(H, F).items():
        e_lib, e_or = scaled_err(g[lo:hi], G64[lo:hi]), scaled_err(G[lo:hi], G64[lo:hi])
        print("  %s: library %.3e, fp32 oracle %.3e (against the fp64 oracle)" % (name, e_lib, e_or))
        assert e_lib < max(1e-5, 2 * e_or), name
    assert abs(g[net.n_params + 1] - err64) < 1e-5 * max(err64, 1.0)


@pytest.mark.parametrize("what", ["bright images", "all but one bright", "not finite", "huge filter", "huge FC weights", "dim"])
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("H,F,n", [(56, 64, 40), (8, 128, 301), (8, 64, 3500)])
def test_tensor_core_images_do_not_depend_on_their_neighbours(cuda, pkg, ob, H, F, n, mode, what):
    """One power of two scales the pixels of a call, so an image much brighter than others (or not finite) has to leave them
    untouched and come out right itself: both for the outputs, image by image, and for the gradient.  Weights of any magnitude
    too.  Yardstick: the fp64 oracle, which computes each image by itself, within the tolerance of the mode or four times the fp32
    kernels' own distance from it (pixels of 30,000 leave few bits to sums that a sigmoid does not saturate); where its values
    are not finite, the fp32 kernels."""
    x, labels = wide_inputs(n, H, 11)
    params = wide_params(ob, H, F, 12)
    S = F * ((H - 4) // 4) ** 2
    fc = slice(F * 26 + 17, F * 26 + 17 + 10 * S)
    spots = [0, n // 2, n - 1]
    if what == "bright images":
        x[spots[0], 3, 3], x[spots[1], H - 1, H - 1], x[spots[2], 4, 5] = 1e6, 1e30, -4e5
    elif what == "all but one bright":
        x[1:] *= np.float32(3e4)
    elif what == "not finite":
        x[spots[0], 3, 3], x[spots[1], 2, 2], x[spots[2], 4, 5] = np.nan, np.inf, -np.inf
    elif what == "huge filter":
        params[:F * 25] *= np.float32(1e25)
        x *= np.float32(1e-25)
    elif what == "huge FC weights":
        params[fc] *= np.float32(1e22)
    elif what == "dim":
        x[1:] *= np.float32(1e-3)
        x[spots[1]] = 0
    net = pkg.WideNet(H, F)
    net.set_params(params)
    d_x = cuda.from_numpy(x).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    outs, grads = {}, {}
    for conv in (0, mode):
        net.set_option("conv", conv)
        d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
        d_g = cuda.zeros(net.n_padded, dtype=cuda.float32, device="cuda")
        net.forward(d_x, n, d_out, None)
        net.grad_batch(d_x, d_lab, n, d_g)
        cuda.cuda.synchronize()
        assert net.status() == 0
        outs[conv], grads[conv] = d_out.cpu().numpy(), d_g.cpu().numpy()
    tol = 1e-5 if mode == 2 else 3e-3
    if what in ("not finite", "huge FC weights"):
        ref, G = outs[0], grads[0]
    else:
        ref, _ = ob.forward_batch(params, x, H=H, F=F, dtype=np.float64)
        G, _ = ob.grad_batch(params, x, labels, H=H, F=F, dtype=np.float64)
    assert np.array_equal(np.isnan(outs[mode]), np.isnan(ref))
    ok = ~np.isnan(ref).any(axis=1)
    assert ok.sum() >= n - 3
    e_tc, e_fp32 = (float(np.max(np.abs(outs[c][ok].astype(np.float64) - ref[ok]))) for c in (mode, 0))
    assert e_tc < max(tol, 4 * e_fp32)
    if what == "not finite":
        return
    for name, (lo, hi) in blocks(H, F).items():
        e_tc, e_fp32 = scaled_err(grads[mode][lo:hi], G[lo:hi]), scaled_err(grads[0][lo:hi], G[lo:hi])
        print("%s: tensor cores %.3e, fp32 kernels %.3e" % (name, e_tc, e_fp32))
        assert e_tc < max(tol * (1 if mode == 2 else 10), 4 * e_fp32), name
