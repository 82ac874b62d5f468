"""Fused training kernels (GPU): minibatch gradient, minibatch SGD and the per-sample SGD kernel
against the oracle and the reference's own kernels."""
import numpy as np
import pytest

from conftest import rel_err, scaled_err

pytestmark = pytest.mark.gpu

BLOCKS = {"Wc": (0, 150), "bc": (150, 156), "Ws": (156, 172), "bs": (172, 173), "Wf": (173, 2333),
          "bf": (2333, 2343)}


# In-place adds per step into one parameter: the reference (and the oracle, which follows it) adds
# every bias term straight into the bias, 576 times for a conv bias and 216 times for the subsample bias.
SEQUENTIAL_ADDS = {"Wc": 1, "bc": 576, "Ws": 1, "bs": 216, "Wf": 1, "bf": 1}


def increments_agree(p, p_other, p0, lo, hi, name, rtol=1e-4):
    """Compare parameter increments of one block.  An increment is only known to the rounding of the
    parameter it was added to (half an ulp of |p| per add, a random walk over the adds), so the bar
    is rtol of the block's largest increment plus 2*sqrt(adds) ulps of the block's largest parameter."""
    inc_a = p[lo:hi].astype(np.float64) - p0[lo:hi]
    inc_b = p_other[lo:hi].astype(np.float64) - p0[lo:hi]
    ulp = float(np.spacing(np.float32(np.max(np.abs(p0[lo:hi])))))
    slack = 2 * ulp * np.sqrt(SEQUENTIAL_ADDS[name])
    return np.max(np.abs(inc_a - inc_b)) <= rtol * np.max(np.abs(inc_b)) + slack


def to_dev(torch, images, labels):
    d_img = torch.from_numpy(np.ascontiguousarray(images)).cuda()
    d_lab = torch.from_numpy(np.ascontiguousarray(labels).astype(np.int32)).cuda()
    return d_img, d_lab


def gpu_grad(torch, net, images, labels):
    d_img, d_lab = to_dev(torch, images, labels)
    d_g = torch.full((2368,), 7.0, dtype=torch.float32, device="cuda")
    net.grad_batch(d_img, d_lab, images.shape[0], d_g)
    torch.cuda.synchronize()
    assert net.status() == 0
    return d_g.cpu().numpy()


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 147, 148, 149, 256, 1000])
def test_grad_batch_matches_oracle(cuda, pkg, ob, params0, n, fast):
    images, labels = pkg.synth.synth_images(31, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(fast)
    g = gpu_grad(cuda, net, images, labels)
    G, err = ob.grad_batch(params0, images, labels)
    for name, (lo, hi) in BLOCKS.items():
        assert scaled_err(g[lo:hi], G[lo:hi]) < 1e-5, name
    assert abs(g[2344] - err) < 1e-5 * max(err, 1.0)
    assert g[2343] == 0 and not g[2345:].any()
    # parameters are untouched by a gradient evaluation
    assert np.array_equal(net.get_params(), params0)


def test_grad_batch_empty_and_deterministic(cuda, pkg, params0):
    net = pkg.Net(0)
    net.set_params(params0)
    d_g = cuda.full((2368,), 3.0, dtype=cuda.float32, device="cuda")
    net.grad_batch(None, None, 0, d_g)
    cuda.cuda.synchronize()
    assert not d_g.cpu().numpy().any()
    images, labels = pkg.synth.synth_images(32, 500)
    a = gpu_grad(cuda, net, images, labels)
    b = gpu_grad(cuda, net, images, labels)
    assert np.array_equal(a, b)


def test_grad_is_additive_over_shards(cuda, pkg, params0):
    """What the data-parallel all-reduce relies on: grad(A+B) = grad(A) + grad(B) to rounding."""
    images, labels = pkg.synth.synth_images(33, 512)
    net = pkg.Net(0)
    net.set_params(params0)
    whole = gpu_grad(cuda, net, images, labels)[:2343]
    parts = sum(gpu_grad(cuda, net, images[i:i + 128], labels[i:i + 128])[:2343].astype(np.float64)
                for i in range(0, 512, 128))
    assert scaled_err(whole, parts) < 1e-5


def test_single_sgd_step_matches_oracle_and_reference(cuda, pkg, ob, params0, data64):
    images, labels = data64
    ref = ob.Reference(0) if ob.reference_available() else None
    for i in (0, 3, 40):
        net = pkg.Net(0)
        net.set_params(params0)
        d_img, d_lab = to_dev(cuda, images[i:i + 1], labels[i:i + 1])
        ran, mean_err = net.train_sgd_persample(d_img, d_lab, 1, 1)
        p = net.get_params()
        p_or, err_or, _ = ob.sgd_step(params0, images[i], int(labels[i]))
        assert ran == 1
        assert scaled_err(p, p_or) < 1e-5
        for name, (lo, hi) in BLOCKS.items():
            assert increments_agree(p, p_or, params0, lo, hi, name), name
        assert abs(float(mean_err[0]) - err_or) < 1e-5
        if ref is not None:
            ref.set_params(params0)
            err_ref = ref.train_step(images[i], int(labels[i]))
            p_ref = ref.get_params()
            assert scaled_err(p, p_ref) < 1e-5
            for name, (lo, hi) in BLOCKS.items():
                assert increments_agree(p, p_ref, params0, lo, hi, name), name
            assert abs(float(mean_err[0]) - err_ref) < 1e-5
    if ref is not None:
        ref.close()


@pytest.mark.parametrize("fast", [0, 1])
def test_persample_trajectory_matches_oracle(cuda, pkg, ob, params0, fast):
    """2,000 sequential SGD steps (two epochs of 1,000).  Rounding differences compound along the
    chain, so the bar on parameters is 1e-3 of the largest parameter here, with 1e-5 kept for the
    single step from identical state (previous test); the per-epoch mean error must agree to 1e-4
    relative."""
    n = 1000
    images, labels = pkg.synth.synth_images(34, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(fast)
    d_img, d_lab = to_dev(cuda, images, labels)
    ran, mean_err = net.train_sgd_persample(d_img, d_lab, n, 2)
    p_or, m_or, ran_or = ob.train_persample(params0, images, labels, 2)
    assert ran == ran_or == 2
    assert scaled_err(net.get_params(), p_or) < 1e-3
    assert np.allclose(mean_err, m_or, rtol=1e-4)
    # and the trained net classifies like the oracle's
    test_img, _ = pkg.synth.synth_images(35, 500)
    d_t = cuda.from_numpy(test_img).cuda()
    d_arg = cuda.empty((500,), dtype=cuda.int32, device="cuda")
    net.forward(d_t, 500, None, d_arg)
    cuda.cuda.synchronize()
    _, arg_or = ob.forward_batch(p_or, test_img)
    assert (d_arg.cpu().numpy() == arg_or).mean() > 0.99


def test_full_size_persample_epoch_matches_oracle(cuda, pkg, ob, params0):
    """Benchmark configuration 1 at its full size: one epoch of per-sample SGD over 10,000 images of
    seed 0 in file order, then the argmax of 2,000 held-out images, against the oracle run on the
    same data.  10,000 sequential steps compound rounding differences, so the parameters are held to
    2e-3 of the largest parameter (printed), the epoch's mean error to 1e-4 relative and the test-set
    predictions to 99 % agreement (labels are random, so accuracy itself is chance for both)."""
    n_train, n_test = 10000, 2000
    images, labels = pkg.synth.synth_images(0, n_train + n_test)
    d_img, d_lab = to_dev(cuda, images, labels)
    net = pkg.Net(0)
    net.set_params(params0)
    ran, mean_err = net.train_sgd_persample(d_img, d_lab, n_train, 1)
    p_or, m_or, ran_or = ob.train_persample(params0, images[:n_train], labels[:n_train], 1)
    err = scaled_err(net.get_params(), p_or)
    print("10,000 steps: parameter distance %.3e, mean error %.6f vs oracle %.6f" % (err, float(mean_err[0]), float(m_or[0])))
    assert ran == ran_or == 1
    assert err < 2e-3
    assert np.allclose(mean_err, m_or, rtol=1e-4)
    d_arg = cuda.empty((n_test,), dtype=cuda.int32, device="cuda")
    net.forward(d_img[n_train:], n_test, None, d_arg)
    cuda.cuda.synchronize()
    _, arg_or = ob.forward_batch(p_or, images[n_train:])
    agree = float((d_arg.cpu().numpy() == arg_or).mean())
    acc = float((d_arg.cpu().numpy().astype(np.uint32) == labels[n_train:]).mean())
    acc_or = float((arg_or.astype(np.uint32) == labels[n_train:]).mean())
    print("test set: %.4f of the predictions agree; accuracy %.4f vs oracle %.4f" % (agree, acc, acc_or))
    assert agree > 0.99 and abs(acc - acc_or) < 0.01


def test_full_size_minibatch_epoch_matches_oracle(cuda, pkg, ob, params0):
    """Benchmark configuration 4 at its full single-GPU size: one epoch of minibatch SGD, batch 256,
    over 60,000 images of seed 3, against the oracle's minibatch rule: parameters within 2e-5 of the
    largest parameter, the epoch's mean error within 1e-5 relative."""
    n, batch = 60000, 256
    images, labels = pkg.synth.synth_images(3, n)
    d_img, d_lab = to_dev(cuda, images, labels)
    net = pkg.Net(0)
    net.set_params(params0)
    d_me = cuda.zeros(1, dtype=cuda.float32, device="cuda")
    net.train_minibatch(d_img, d_lab, n, batch, 1, 0.1, d_me)
    cuda.cuda.synchronize()
    assert net.status() == 0
    p_or, me_or = ob.train_minibatch(params0, images, labels, batch, 1)
    err = scaled_err(net.get_params(), p_or)
    print("235 steps of 256: parameter distance %.3e, mean error %.7f vs oracle %.7f" % (err, float(d_me.item()), float(me_or[0])))
    assert err < 2e-5
    assert np.allclose(d_me.cpu().numpy(), me_or, rtol=1e-5)


def test_persample_early_stop_and_determinism(cuda, pkg, params0):
    images, labels = pkg.synth.synth_images(36, 200)
    d_img, d_lab = to_dev(cuda, images, labels)
    net = pkg.Net(0)
    net.set_params(params0)
    ran, mean_err = net.train_sgd_persample(d_img, d_lab, 200, 5, threshold=100.0)
    assert ran == 1 and mean_err.shape == (1,)
    p1 = net.get_params()
    net.set_params(params0)
    ran, _ = net.train_sgd_persample(d_img, d_lab, 200, 1)
    assert ran == 1 and np.array_equal(net.get_params(), p1)
    ran, _ = net.train_sgd_persample(d_img, d_lab, 0, 3)
    assert ran == 0


@pytest.mark.parametrize("kernel", [0, 1])
def test_persample_kernels_single_step_matches_oracle(cuda, pkg, ob, params0, kernel):
    """Three SGD steps from identical state with the reference sigmoid, for both per-sample kernels
    (0: single persistent block; 1: the default cluster of six CTAs): 1e-5 of the largest parameter,
    and the epoch's mean error norm."""
    images, labels = pkg.synth.synth_images(42, 3)
    d_img, d_lab = to_dev(cuda, images, labels)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(0)
    net.set_option("persample_kernel", kernel)
    ran, mean_err = net.train_sgd_persample(d_img, d_lab, 3, 1)
    p_or, m_or, _ = ob.train_persample(params0, images, labels, 1)
    assert ran == 1 and net.status() == 0
    assert scaled_err(net.get_params(), p_or) < 1e-5
    assert np.allclose(mean_err, m_or, rtol=1e-5)


@pytest.mark.parametrize("fast", [0, 1])
def test_persample_cluster_kernel_against_single_block(cuda, pkg, ob, params0, fast):
    """The cluster kernel adds the same terms in another order than the single-block kernel: over 3
    epochs of 700 samples both stay within the trajectory bar of the oracle and of each other, stop
    early alike, and the cluster kernel repeats itself bit for bit."""
    n = 700
    images, labels = pkg.synth.synth_images(43, n)
    d_img, d_lab = to_dev(cuda, images, labels)
    got = {}
    for kernel in (0, 1, 1):
        net = pkg.Net(0)
        net.set_params(params0)
        net.set_fast_sigmoid(fast)
        net.set_option("persample_kernel", kernel)
        ran, mean_err = net.train_sgd_persample(d_img, d_lab, n, 3)
        assert ran == 3 and net.status() == 0
        p = net.get_params()
        ran1, _ = net.train_sgd_persample(d_img, d_lab, 1, 4, threshold=100.0)   # stops after one epoch
        assert ran1 == 1 and net.status() == 0
        if kernel in got:
            assert np.array_equal(got[kernel][0], p) and np.array_equal(got[kernel][1], mean_err)
        got[kernel] = (p, np.asarray(mean_err))
    assert scaled_err(got[1][0], got[0][0]) < 1e-3
    assert np.allclose(got[1][1], got[0][1], rtol=1e-4)
    p_or, m_or, ran_or = ob.train_persample(params0, images, labels, 3)
    assert ran_or == 3
    for kernel in (0, 1):
        assert scaled_err(got[kernel][0], p_or) < 1e-3
        assert np.allclose(got[kernel][1], m_or, rtol=1e-4)


@pytest.mark.parametrize("n,batch", [(600, 256), (256, 256), (100, 7), (5, 1)])
def test_minibatch_training_matches_oracle(cuda, pkg, ob, params0, n, batch):
    images, labels = pkg.synth.synth_images(37, n)
    d_img, d_lab = to_dev(cuda, images, labels)
    net = pkg.Net(0)
    net.set_params(params0)
    d_me = cuda.zeros(2, dtype=cuda.float32, device="cuda")
    net.train_minibatch(d_img, d_lab, n, batch, 2, 0.1, d_me)
    cuda.cuda.synchronize()
    assert net.status() == 0
    p_or, me_or = ob.train_minibatch(params0, images, labels, batch, 2)
    assert scaled_err(net.get_params(), p_or) < 2e-5
    assert np.allclose(d_me.cpu().numpy(), me_or, rtol=1e-5)


def test_minibatch_epoch_in_a_cuda_graph_equals_eager(cuda, pkg, params0):
    """The step's two kernels are launched as programmatic dependents (each may set itself up while its
    predecessor still runs).  An epoch captured into a CUDA graph and replayed must leave exactly the
    parameters of the same epoch launched eagerly, and a second replay must continue from there."""
    n, batch = 2048 + 100, 256
    images, labels = pkg.synth.synth_images(39, n)
    d_img, d_lab = to_dev(cuda, images, labels)
    eager = pkg.Net(0)
    eager.set_params(params0)
    eager.train_minibatch(d_img, d_lab, n, batch, 2, 0.1, None)
    cuda.cuda.synchronize()
    p_eager = eager.get_params()
    net = pkg.Net(0)
    net.set_params(params0)
    net.train_minibatch(d_img, d_lab, batch, batch, 1, 0.1, None)       # scratch exists before the capture
    net.set_params(params0)
    side = cuda.cuda.Stream()
    with cuda.cuda.stream(side):
        graph = cuda.cuda.CUDAGraph()
        with cuda.cuda.graph(graph, stream=side):
            net.train_minibatch(d_img, d_lab, n, batch, 1, 0.1, None, cuda.cuda.current_stream())
    cuda.cuda.synchronize()
    graph.replay()
    graph.replay()
    cuda.cuda.synchronize()
    assert net.status() == 0
    assert np.array_equal(net.get_params(), p_eager)


def test_minibatch_of_one_equals_persample_kernel(cuda, pkg, params0):
    images, labels = pkg.synth.synth_images(38, 50)
    d_img, d_lab = to_dev(cuda, images, labels)
    a = pkg.Net(0); a.set_params(params0)
    b = pkg.Net(0); b.set_params(params0)
    a.train_minibatch(d_img, d_lab, 50, 1, 1, 0.1, None)
    b.train_sgd_persample(d_img, d_lab, 50, 1)
    cuda.cuda.synchronize()
    assert scaled_err(a.get_params(), b.get_params()) < 1e-5


def test_apply_update(cuda, pkg, params0):
    net = pkg.Net(0)
    net.set_params(params0)
    g = np.random.default_rng(0).standard_normal(2368).astype(np.float32)
    net.apply_update(cuda.from_numpy(g).cuda(), 0.01)
    cuda.cuda.synchronize()
    want = params0 + np.float32(0.01) * g[:2343]
    assert np.allclose(net.get_params(), want, rtol=1e-6, atol=1e-7)


def test_reference_trajectory_spread(cuda, pkg, ob, params0):
    """The reference itself is not bit-reproducible (float atomics).  Measure reference-vs-reference
    and library-vs-reference drift over the same 300 steps; the library must stay within a small
    multiple of the reference's own spread (floored at 1e-5 of the largest parameter)."""
    if not ob.reference_available():
        pytest.skip("reference kernels not built")
    n = 300
    images, labels = pkg.synth.synth_images(39, n)
    runs = []
    for _ in range(2):
        ref = ob.Reference(0)
        ref.set_params(params0)
        for i in range(n):
            ref.train_step(images[i], int(labels[i]))
        runs.append(ref.get_params())
        ref.close()
    spread = scaled_err(runs[0], runs[1])
    net = pkg.Net(0)
    net.set_params(params0)
    d_img, d_lab = to_dev(cuda, images, labels)
    net.train_sgd_persample(d_img, d_lab, n, 1)
    drift = scaled_err(net.get_params(), runs[0])
    print("reference-vs-reference spread %.3e, library-vs-reference drift %.3e" % (spread, drift))
    assert drift < max(20 * spread, 1e-4)


@pytest.mark.parametrize("n", [295, 296, 297, 1185])
def test_grad_batch_around_full_rounds(cuda, pkg, ob, params0, n):
    """Two images per block and turn, three image buffers per team: one image short of a full round, a full one, one image
    into the next, and a batch whose last turn reuses the buffers with a single live team."""
    images, labels = pkg.synth.synth_images(37, n)
    net = pkg.Net(0)
    net.set_params(params0)
    g = gpu_grad(cuda, net, images, labels)
    G, err = ob.grad_batch(params0, images, labels)
    for name, (lo, hi) in BLOCKS.items():
        assert scaled_err(g[lo:hi], G[lo:hi]) < 1e-5, name
    assert abs(g[2344] - err) < 1e-5 * err and g[2343] == 0 and not g[2345:].any()


# ---- the gradient of a large batch on the tensor cores (option "grad_path") ------------------------
def both_paths(cuda, pkg, params, images, labels):
    out = {}
    for path in (0, 1):
        net = pkg.Net(0)
        net.set_params(params)
        net.set_option("grad_path", path)
        out[path] = gpu_grad(cuda, net, images, labels)
        assert np.array_equal(out[path], gpu_grad(cuda, net, images, labels), equal_nan=True)      # fixed order
    return out


@pytest.mark.parametrize("n", [1, 4, 5, 6, 739, 740, 741, 148 * 5 * 4 + 3, 148 * 26])
def test_tensor_core_gradient_matches_oracle(cuda, pkg, ob, params0, n):
    """Tiles of five images: one image, a full tile, one image more, one tile per SM, and so many that every ring (two raw buffers,
    three accumulators, four delta operands, five slabs) goes round.  The bar is the other path's: 1e-5 of the block's largest
    entry."""
    images, labels = pkg.synth.synth_images(61, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("grad_path", 1)
    g = gpu_grad(cuda, net, images, labels)
    G, err = ob.grad_batch(params0, images, labels)
    for name, (lo, hi) in BLOCKS.items():
        assert scaled_err(g[lo:hi], G[lo:hi]) < 1e-5, name
    assert abs(g[2344] - err) < 1e-5 * max(err, 1.0) and g[2343] == 0 and not g[2345:].any()
    assert np.array_equal(g, gpu_grad(cuda, net, images, labels))


@pytest.mark.parametrize("where", ["first", "second tile", "middle", "last", "first of a share", "all"])
@pytest.mark.parametrize("what", ["fraction", "bright", "negative", "not a number"])
def test_tensor_core_gradient_leaves_other_pixels(cuda, pkg, params0, what, where):
    """A block stops at its first tile with a pixel that is not a whole number / 255 and leaves what follows to the CUDA-core kernel, wherever
    that is.  Yardstick: the CUDA-core path alone; two fp32 sums of the same terms, so 1e-5 of the block's largest entry."""
    n = 148 * 17 + 9
    share = -(-n // 148)
    images, labels = pkg.synth.synth_images(62, n)
    spot = {"first": [0], "second tile": [5], "middle": [share * 70 + 8], "last": [n - 1], "first of a share": [share * 3],
            "all": np.arange(n)}[where]
    images[spot, 3, 9] = {"fraction": 0.3337, "bright": 3.1e5, "negative": -0.25, "not a number": np.nan}[what]
    out = both_paths(cuda, pkg, params0, images, labels)
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    if what != "not a number":
        for name, (lo, hi) in BLOCKS.items():
            assert scaled_err(out[1][lo:hi], out[0][lo:hi].astype(np.float64)) < 1e-5, name
        assert abs(out[1][2344] - out[0][2344]) < 1e-5 * out[0][2344]


def some_other_pixels(images, which, seed=3):
    """`images` with other pixels than whole numbers / 255 in some of them."""
    n, rng = images.shape[0], np.random.default_rng(seed)
    images = images.copy()
    if which == "second half":
        images[n // 2:] *= np.float32(0.77)
    elif which == "all":
        images *= np.float32(0.77)
    elif which == "byte times reciprocal":
        images = np.rint(images * 255).astype(np.float32) * np.float32(1 / 255)
    else:
        images[rng.permutation(n)[:int(n * which)], 12, 12] = 0.3337
    return images


@pytest.mark.parametrize("n", [11, 740, 148 * 17 + 9, 148 * 180])
@pytest.mark.parametrize("which", [0.01, 0.1, 0.4, "second half", "all", "byte times reciprocal"])
def test_tensor_core_gradient_of_a_mixture(cuda, pkg, params0, which, n):
    """Tiles with other pixels are left out one by one, a share from the tile on where there are too many, or as a whole, and done on the CUDA cores
    in whatever order blocks finish; a net is left as it was for the next call.  Yardstick and bar as above."""
    images, labels = pkg.synth.synth_images(66, n)
    mixed = some_other_pixels(images, which)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("grad_path", 1)
    before = gpu_grad(cuda, net, images, labels)
    got = gpu_grad(cuda, net, mixed, labels)
    assert np.array_equal(got, gpu_grad(cuda, net, mixed, labels)) and np.array_equal(before, gpu_grad(cuda, net, images, labels))
    net.set_option("grad_path", 0)
    want = gpu_grad(cuda, net, mixed, labels).astype(np.float64)
    for name, (lo, hi) in BLOCKS.items():
        assert scaled_err(got[lo:hi], want[lo:hi]) < 1e-5, name
    assert abs(got[2344] - want[2344]) < 1e-5 * want[2344] and got[2343] == 0 and not got[2345:].any()


@pytest.mark.parametrize("which,n,bar", [(0.01, 60000, 1.0), ("second half", 4000, 1.25)])
def test_tensor_core_gradient_of_a_mixture_takes_no_longer(cuda, pkg, which, n, bar):
    """Images that the tensor-core kernel cannot take must not cost much more than on the CUDA cores alone.  Measured: 1 % of 60,000 images 392 us against
    643 (once 816), the second half of 4,000 56 us against 50 (once 70)."""
    images, labels = pkg.synth.synth_images(66, 1000)
    mixed = some_other_pixels(np.tile(images, (n // 1000, 1, 1)), which)
    d_img, d_lab = to_dev(cuda, mixed, np.tile(labels, n // 1000))
    d_g = cuda.empty(2368, dtype=cuda.float32, device="cuda")
    net = pkg.Net(0)
    times = {0: [], -1: []}
    for _ in range(9):
        for path, of_path in times.items():
            net.set_option("grad_path", path)
            start, stop = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
            net.grad_batch(d_img, d_lab, n, d_g)
            start.record()
            for _ in range(20):
                net.grad_batch(d_img, d_lab, n, d_g)
            stop.record()
            cuda.cuda.synchronize()
            of_path.append(start.elapsed_time(stop))
    assert net.status() == 0
    assert np.median(times[-1]) < bar * np.median(times[0])


def test_first_gradient_of_a_net_allocates_one_granule(cuda, pkg):
    """The training scratch comes with a net's first gradient call, so that call pays for it: a row per SM, 1.4 MB, which fits one 2 MiB granule of
    device memory.  Median over nets, because small allocations share granules."""
    images, labels = pkg.synth.synth_images(67, 2048)
    d_img, d_lab = to_dev(cuda, images, labels)
    d_g = cuda.empty(2368, dtype=cuda.float32, device="cuda")
    nets, taken = [], []
    for seed in range(9):
        nets.append(pkg.Net(seed))
        before = cuda.cuda.mem_get_info()[0]
        nets[-1].grad_batch(d_img, d_lab, 2048, d_g)
        cuda.cuda.synchronize()
        taken.append(before - cuda.cuda.mem_get_info()[0])
    assert sorted(taken)[len(taken) // 2] <= 2 << 20


@pytest.mark.parametrize("n", [5, 743])
@pytest.mark.parametrize("what", ["bright", "white", "inverted", "both"])
def test_tensor_core_gradient_of_dense_bright_images(cuda, pkg, what, n):
    """Bytes of 200 to 255, of 254 and 255, inverted strokes, and strokes of which every second image is inverted, with deltas of one sign: sums
    of 720 products that all add up, which the tensor core must not truncate (2^-23 for each of 48 additions, half of it on average, half of the
    sum on average: 1.4e-6).  Yardstick: the CUDA-core path, which shares the activations' approximations; what is left are fp32 roundings of
    a delta, its parts, the bias and the sums, five of 2^-24 on either side."""
    rng = np.random.default_rng(7)
    images, labels = pkg.synth.synth_images(65, n)
    pixels = np.rint(images * 255)
    if what == "bright":
        pixels = rng.integers(200, 256, pixels.shape)
    elif what == "white":
        pixels = rng.integers(254, 256, pixels.shape)
    elif what == "inverted":
        pixels = 255 - pixels
    else:
        pixels[::2] = 255 - pixels[::2]
    images = (pixels / 255).astype(np.float32)
    for seed in range(3):
        params = pkg.Net(seed).get_params()
        params[173:2333] = 0.02 * (1 + 0.3 * rng.random(2160))
        params[156:172] = 0.3 + 0.2 * rng.random(16)
        out = both_paths(cuda, pkg, params, images, labels)
        for name, (lo, hi) in BLOCKS.items():
            assert scaled_err(out[1][lo:hi], out[0][lo:hi].astype(np.float64)) < 10 * 2.0**-24, name


def fp64_gradient(torch, params, images, labels):
    """The gradient of a batch in fp64, from the formulas."""
    p = torch.from_numpy(params.astype(np.float64)).cuda()
    x, n = torch.from_numpy(images.astype(np.float64)).cuda(), images.shape[0]
    w_conv, w_sub, w_fc = p[:150].view(6, 25), p[156:172].view(4, 4), p[173:2333].view(10, 216)
    patches = torch.nn.functional.unfold(x.view(n, 1, 28, 28), 5)
    a = torch.sigmoid(torch.einsum("ft,ntp->nfp", w_conv, patches) + p[150:156, None]).view(n, 6, 6, 4, 6, 4)
    s = torch.sigmoid(torch.einsum("nfpiqj,ij->nfpq", a, w_sub) + p[172]).reshape(n, 216)
    d = torch.nn.functional.one_hot(torch.from_numpy(labels.astype(np.int64)).cuda(), 10) - torch.sigmoid(s @ w_fc.t() + p[2333:])
    ds = ((d @ w_fc) * s * (1 - s)).view(n, 6, 6, 6)
    dc = (ds.view(n, 6, 6, 1, 6, 1) * w_sub.view(1, 1, 1, 4, 1, 4) * a * (1 - a)).reshape(n, 6, 576) / 576
    parts = [torch.einsum("nfp,ntp->ft", dc, patches), dc.sum((0, 2)), torch.einsum("nfpq,nfpiqj->ij", ds, a), ds.sum()[None] / 216, d.t() @ s, d.sum(0)]
    return torch.cat([q.reshape(-1) for q in parts]).cpu().numpy()


@pytest.mark.parametrize("scale", [1, 30])
@pytest.mark.parametrize("what", ["strokes", "bright", "inverted"])
def test_tensor_core_gradient_is_as_close_to_fp64(cuda, pkg, what, scale):
    """Distance from fp64 of the whole gradient and of the conv weights' part, by the two paths, geometric mean over nets (where that part is not lost
    in saturation).  With conv weights 30 times as large pre-activations are the limit, and of dense bright images their common part.  Two fp32
    results of the same precision: half as far again, for chance."""
    images, labels = pkg.synth.synth_images(68, 743)
    pixels = np.rint(images * 255)
    if what == "bright":
        pixels = np.random.default_rng(5).integers(200, 256, pixels.shape)
    elif what == "inverted":
        pixels = 255 - pixels
    images = (pixels / 255).astype(np.float32)
    ratios = []
    for seed in range(1, 9):
        params = pkg.Net(seed).get_params()
        params[:150] *= np.float32(scale)
        want = fp64_gradient(cuda, params, images, labels)
        out = both_paths(cuda, pkg, params, images, labels)
        ratios.append([])
        for hi in (2343, 150):
            away = [np.linalg.norm(out[path][:hi] - want[:hi]) for path in (0, 1)]
            ratios[-1].append(away[1] / away[0] if np.linalg.norm(want[:hi]) > 1e-6 * np.linalg.norm(want) else np.nan)
    assert (np.exp(np.nanmean(np.log(ratios), axis=0)) < 1.5).all(), ratios


@pytest.mark.parametrize("what", ["conv weights x 1e-7", "conv weights x 5e-6", "conv weights x 1e-3", "conv weights x 30", "conv weights x 100",
                                  "conv weights x 500", "conv weights x 1e5", "infinite bias", "not a number", "large rest", "no subsample filter",
                                  "subsample filter of 6e7", "subsample filter of 5e8", "subsample filter of 5e9"])
def test_tensor_core_gradient_parameter_range(cuda, pkg, params0, what):
    """Conv weights below 2^-21 (x 1e-7) or from 2^11 on (x 1e5), and parameters that are not finite, go to the CUDA-core kernel; everything between
    through the scales that follow the largest weight and the tile's deltas.  Yardstick: the CUDA-core path.  With large weights a pre-activation
    of 25 terms up to 0.5 * factor is only known to 25 * 0.5 * factor * 2^-24 in fp32.  A subsample filter that saturates its sigmoids leaves deltas of
    zero, whose scale is the largest there is and must not take the filter's taps out of range (they go to the CUDA cores above 2^26)."""
    images, labels = pkg.synth.synth_images(63, 2100)
    params, factor = params0.copy(), 1.0
    if "conv weights" in what:
        factor = float(what.split()[-1])
        params[:150] *= np.float32(factor)
    elif what == "infinite bias":
        params[151] = np.inf
    elif what == "not a number":
        params[2000] = np.nan
    elif what == "large rest":
        params[156:] *= np.float32(30)
    else:
        params[156:172] = float(what.split()[-1]) if " of " in what else 0
    out = both_paths(cuda, pkg, params, images, labels)
    assert np.isfinite(out[0]).all() or what in ("infinite bias", "not a number")
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
    if not np.isnan(out[0]).any():
        bar = max(1e-5, 25 * 0.5 * factor * 2.0**-24) if factor < 1e5 else 1e-5
        for name, (lo, hi) in BLOCKS.items():
            if np.abs(out[0][lo:hi]).max() > 0:
                assert scaled_err(out[1][lo:hi], out[0][lo:hi].astype(np.float64)) < bar, name
            else:
                assert not out[1][lo:hi].any(), name


def test_gradient_kernel_choice_follows_batch_size(cuda, pkg, params0):
    """grad_path = -1, the default: tensor cores from 2,048 images on, bit for bit, in the gradient call and in the training loop (whose
    ragged last step is small), eager and replayed from a graph; the reference's sigmoid expression stays on the CUDA cores."""
    images, labels = pkg.synth.synth_images(64, 2048 * 2 + 300)
    d_img, d_lab = to_dev(cuda, images, labels)
    got = {}
    for path in (-1, 0, 1):
        net = pkg.Net(0)
        net.set_params(params0)
        net.set_option("grad_path", path)
        a, b = gpu_grad(cuda, net, images[:2047], labels[:2047]), gpu_grad(cuda, net, images[:2048], labels[:2048])
        err = cuda.zeros(2, dtype=cuda.float32, device="cuda")
        net.train_minibatch(d_img, d_lab, images.shape[0], 2048, 2, 0.1, err)
        cuda.cuda.synchronize()
        assert net.status() == 0
        got[path] = (a, b, net.get_params(), err.cpu().numpy())
    assert np.array_equal(got[-1][0], got[0][0]) and np.array_equal(got[-1][1], got[1][1])
    assert not np.array_equal(got[0][1], got[1][1])
    assert np.max(np.abs(got[-1][2] - got[0][2])) < 1e-5 * np.max(np.abs(got[0][2])) and np.allclose(got[-1][3], got[0][3], rtol=1e-5)
    net = pkg.Net(0)
    net.set_params(params0)
    err = cuda.zeros(2, dtype=cuda.float32, device="cuda")
    net.train_minibatch(d_img, d_lab, 2048, 2048, 1, 0.0, err)        # (scratch exists before the capture)
    stream = cuda.cuda.Stream()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph, stream=stream):
        net.train_minibatch(d_img, d_lab, images.shape[0], 2048, 2, 0.1, err, stream.cuda_stream)
    graph.replay()
    cuda.cuda.synchronize()
    assert np.array_equal(net.get_params(), got[-1][2])
    ref = {}
    for path in (0, 1):
        net = pkg.Net(0)
        net.set_params(params0)
        net.set_fast_sigmoid(0)
        net.set_option("grad_path", path)
        ref[path] = gpu_grad(cuda, net, images[:2100], labels[:2100])
    assert np.array_equal(ref[0], ref[1])
    with pytest.raises(Exception):
        net.set_option("grad_path", 2)
