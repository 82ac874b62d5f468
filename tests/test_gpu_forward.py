"""Fused batched forward (GPU) against the oracle, the reference kernels and itself."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def run_forward(torch, net, images, want_out=True, want_arg=True, offset_elems=0):
    n = images.shape[0]
    flat = torch.zeros(n * 784 + offset_elems + 4, dtype=torch.float32, device="cuda")
    d_img = flat[offset_elems:offset_elems + n * 784]
    if n:
        d_img.copy_(torch.from_numpy(np.ascontiguousarray(images).reshape(-1)))
    d_out = torch.full((n, 10), -1.0, dtype=torch.float32, device="cuda") if want_out else None
    d_arg = torch.full((n,), -1, dtype=torch.int32, device="cuda") if want_arg else None
    net.forward(d_img, n, d_out, d_arg)
    torch.cuda.synchronize()
    assert net.status() == 0
    return (d_out.cpu().numpy() if want_out else None), (d_arg.cpu().numpy() if want_arg else None)


def clear_margin(out, tol=1e-5):
    top2 = np.sort(out, axis=1)
    return (top2[:, -1] - top2[:, -2]) > tol * top2[:, -1]


def check_argmax(arg, ref_arg, ref_out, what, tol=1e-5, max_masked_frac=1e-3):
    """argmax must equal the oracle's on every row whose top-two margin exceeds ``tol`` relative
    (below that the reference's own run-to-run atomics order decides the winner); the number of rows
    excused that way is printed and must be tiny."""
    ok = clear_margin(ref_out, tol)
    masked = int((~ok).sum())
    mism = int((arg != ref_arg).sum())
    print("%s: %d rows, %d below the %.0e margin, %d argmax differences in all (%d on clear rows)"
          % (what, len(arg), masked, tol, mism, int((arg[ok] != ref_arg[ok]).sum())))
    assert np.array_equal(arg[ok], ref_arg[ok])
    assert masked <= max(1, int(max_masked_frac * len(arg)))


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 100, 2368 + 5, 4099])
def test_forward_matches_oracle(cuda, pkg, ob, params0, n, fast):
    images, _ = pkg.synth.synth_images(21, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(fast)
    out, arg = run_forward(cuda, net, images)
    ref_out, ref_arg = ob.forward_batch(params0, images)
    assert rel_err(out, ref_out) < 1e-5       # the 1e-5 relative bar on activations
    check_argmax(arg, ref_arg, ref_out, "n=%d flavour %d" % (n, fast))
    # the argmax written by the kernel is the lowest-index maximum of the row it wrote
    assert np.array_equal(arg, np.argmax(out, axis=1).astype(np.int32))


@pytest.mark.parametrize("path", [-1, 0])
@pytest.mark.parametrize("fast", [0, 1])
def test_full_size_forward_matches_oracle(cuda, pkg, ob, params0, fast, path):
    """Benchmark configuration 2 at its full size: 65,536 images of seed 1 against the oracle --
    every sigmoid within 1e-5 relative, argmax equal on every clear-margin row; the number of rows
    below the margin and the number of differing rows are printed (both are expected to be zero or a
    handful out of 65,536).  Run with the default kernel choice (at this size and with the short sigmoid
    form: the three-pass tensor-core kernel) and with the CUDA-core kernel forced."""
    n = 65536
    images, _ = pkg.synth.synth_images(1, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(fast)
    net.set_option("forward_path", path)
    out, arg = run_forward(cuda, net, images)
    ref_out, ref_arg = ob.forward_batch(params0, images, threads=0)
    err = rel_err(out, ref_out)
    print("full size, flavour %d, forward_path %d: max relative error of the sigmoids %.3e" % (fast, path, err))
    assert err < 1e-5
    check_argmax(arg, ref_arg, ref_out, "65,536 images flavour %d path %d" % (fast, path))
    assert np.array_equal(arg, np.argmax(out, axis=1).astype(np.int32))


def test_forward_empty_and_optional_outputs(cuda, pkg, ob, params0):
    net = pkg.Net(0)
    net.set_params(params0)
    net.forward(None, 0, None, None)
    images, _ = pkg.synth.synth_images(22, 50)
    out, _ = run_forward(cuda, net, images, want_arg=False)
    _, arg = run_forward(cuda, net, images, want_out=False)
    assert np.array_equal(arg, np.argmax(out, axis=1))


def test_forward_rejects_bad_arguments(cuda, pkg, params0):
    net = pkg.Net(0)
    d = cuda.zeros(784 * 4 + 8, dtype=cuda.float32, device="cuda")
    with pytest.raises(pkg.CnnError) as e:
        net.forward(d[1:], 2, None, None)   # 4-byte offset: not 16-byte aligned
    assert e.value.code == -1 and "16-byte" in str(e.value)
    with pytest.raises(pkg.CnnError):
        net.forward(d, -1, None, None)
    with pytest.raises(pkg.CnnError):
        net.forward(None, 3, None, None)
    # a 16-byte (4-float) offset is fine
    net.forward(d[4:], 2, None, None)
    cuda.cuda.synchronize()


def test_forward_is_deterministic_and_tie_breaks_low(cuda, pkg, params0):
    images, _ = pkg.synth.synth_images(23, 1000)
    net = pkg.Net(0)
    net.set_params(params0)
    a = run_forward(cuda, net, images)
    b = run_forward(cuda, net, images)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    # all-zero FC weights and equal biases: every output equal, index 0 must win
    p = params0.copy()
    p[173:2333] = 0
    p[2333:] = 0.25
    net.set_params(p)
    out, arg = run_forward(cuda, net, images[:20])
    assert np.all(out == out[0, 0]) and np.all(arg == 0)


def test_forward_host_pipeline(cuda, pkg, ob, params0):
    n = 8192 * 2 + 123          # spans three staging chunks
    images, _ = pkg.synth.synth_images(24, n)
    net = pkg.Net(0)
    net.set_params(params0)
    h_img = cuda.from_numpy(images).pin_memory()
    h_out = cuda.empty((n, 10), dtype=cuda.float32).pin_memory()
    h_arg = cuda.empty((n,), dtype=cuda.int32).pin_memory()
    net.forward_host(h_img, n, h_out, h_arg)
    d_out, d_arg = run_forward(cuda, net, images)
    bad = np.nonzero((h_out.numpy() != d_out).any(axis=1))[0]
    assert bad.size == 0, "rows differing between host pipeline and device call: %s ... (%d)" % (bad[:8], bad.size)
    assert np.array_equal(h_arg.numpy(), d_arg)
    # pageable host memory works too
    out2 = np.empty((n, 10), dtype=np.float32)
    net.forward_host(images, n, out2, None)
    assert np.array_equal(out2, d_out)


def test_forward_against_reference_kernels(cuda, pkg, ob, params0):
    if not ob.reference_available():
        pytest.skip("reference kernels not built")
    images, _ = pkg.synth.synth_images(25, 96)
    net = pkg.Net(0)
    net.set_params(params0)
    out, arg = run_forward(cuda, net, images)
    ref = ob.Reference(0)
    ref.set_params(params0)
    ref_out = np.zeros((96, 10), dtype=np.float32)
    ref_arg = np.zeros(96, dtype=np.int32)
    for i in range(96):
        ref_arg[i] = ref.classify(images[i])
        ref_out[i] = ref.read("f", "output")
    ref.close()
    assert rel_err(out, ref_out) < 1e-5
    check_argmax(arg, ref_arg, ref_out, "96 images against the reference kernels", max_masked_frac=0.05)


@pytest.mark.parametrize("path", [-1, 0])
def test_full_size_property_linearity_in_batch(cuda, pkg, params0, path):
    """benchmark configuration 2 size (65,536 images): results of a batch do not depend on where an image
    sits in it -- the full batch equals the concatenation of two half batches, bit for bit, and the
    device generator fills the same images as the host generator.  Holds for the default kernel choice
    (tensor cores at these sizes) and for the CUDA-core kernel."""
    n = 65536
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("forward_path", path)
    d_img = cuda.empty((n, 28, 28), dtype=cuda.float32, device="cuda")
    pkg.synth_images_device(1, 0, n, d_img)
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
    net.forward(d_img, n, d_out, d_arg)
    o2 = cuda.empty_like(d_out)
    a2 = cuda.empty_like(d_arg)
    half = n // 2 + 3 * 8       # keeps the second half on a tile boundary multiple
    net.forward(d_img, half, o2, a2)
    net.forward(d_img[half:], n - half, o2[half:], a2[half:])
    cuda.cuda.synchronize()
    assert cuda.equal(d_out, o2) and cuda.equal(d_arg, a2)
    host, _ = pkg.synth.synth_images(1, 2048, first_index=30000)
    assert np.array_equal(d_img[30000:32048].cpu().numpy(), host)


def test_device_generator_matches_host(cuda, pkg):
    n = 3000
    d_img = cuda.empty((n, 28, 28), dtype=cuda.float32, device="cuda")
    d_lab = cuda.empty((n,), dtype=cuda.int32, device="cuda")
    pkg.synth_images_device(9, 12345, n, d_img, d_lab)
    cuda.cuda.synchronize()
    h_img, h_lab = pkg.synth.synth_images(9, n, first_index=12345)
    assert np.array_equal(d_img.cpu().numpy(), h_img)
    assert np.array_equal(d_lab.cpu().numpy().astype(np.uint32), h_lab)


@pytest.mark.parametrize("n", [1, 9, 1000, 8192 + 77])
def test_uint8_input_is_bit_identical_to_fp32(cuda, pkg, params0, n):
    """uint8 pixels through the in-kernel pixel/255.0 table == fp32 images, through the CUDA-core kernels (the
    tensor-core kernel's ingest: test_tensor_core_forward_operand_range)."""
    pix = pkg.synth.synth_pixels_u8(26, n)
    images = pkg.synth.u8_to_float(pix)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("forward_path", 0)
    out_f, arg_f = run_forward(cuda, net, images)
    d_pix = cuda.from_numpy(pix).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
    net.forward_u8(d_pix, n, d_out, d_arg)
    cuda.cuda.synchronize()
    assert net.status() == 0
    assert np.array_equal(d_out.cpu().numpy(), out_f) and np.array_equal(d_arg.cpu().numpy(), arg_f)
    h_out = np.empty((n, 10), dtype=np.float32)
    h_arg = np.empty((n,), dtype=np.int32)
    net.forward_u8_host(pix, n, h_out, h_arg)
    assert np.array_equal(h_out, out_f) and np.array_equal(h_arg, arg_f)


def test_sigmoid_flavours_agree(cuda, pkg, ob, params0):
    """The default (short) sigmoid form against the reference expression on the full benchmark batch:
    maximum relative difference of the ten outputs between the two, and the distance of each from the
    fp64 oracle, beside the fp32 oracle's own distance from it."""
    n = 65536
    images, _ = pkg.synth.synth_images(1, n)
    d_img = cuda.from_numpy(images).cuda()
    ref64, _ = ob.forward_batch(params0, images, threads=0, dtype=np.float64)
    ref32, _ = ob.forward_batch(params0, images, threads=0)
    outs = {}
    for fl in (0, 1):
        net = pkg.Net(0)
        net.set_params(params0)
        net.set_fast_sigmoid(fl)
        net.set_option("forward_path", 0)      # the same kernel for both forms
        o = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
        net.forward(d_img, n, o, None)
        cuda.cuda.synchronize()
        outs[fl] = o.cpu().numpy().astype(np.float64)
    d = float(np.max(np.abs(outs[1] - outs[0]) / outs[0]))
    e0, e1, eo = rel_err(outs[0], ref64), rel_err(outs[1], ref64), rel_err(ref32, ref64)
    print("short form vs reference expression: %.3e; against the fp64 oracle: reference expression %.3e, "
          "short form %.3e, fp32 oracle %.3e" % (d, e0, e1, eo))
    assert d < 5e-6 and e1 < max(5e-6, 1.5 * e0)


def test_forward_host_is_ordered_behind_legacy_stream_work(cuda, pkg, params0):
    """A host-buffer forward issued right after an asynchronous parameter update on the legacy
    stream (no synchronisation in between) must see the updated parameters."""
    n = 4096
    images, labels = pkg.synth.synth_images(27, n)
    d_img = cuda.from_numpy(images).cuda()
    d_lab = cuda.from_numpy(labels.astype(np.int32)).cuda()
    h_img = cuda.from_numpy(images).pin_memory()
    outs = []
    for sync_between in (True, False):
        net = pkg.Net(0)
        net.set_params(params0)
        net.forward_host(h_img, 8, None, None)          # staging buffers and streams exist
        cuda.cuda.synchronize()
        h_out = cuda.empty((n, 10), dtype=cuda.float32).pin_memory()
        net.train_minibatch(d_img, d_lab, n, 64, 3, 0.1, None, None)   # asynchronous, stream NULL
        if sync_between:
            cuda.cuda.synchronize()
        net.forward_host(h_img, n, h_out, None)
        outs.append(h_out.numpy().copy())
    assert np.array_equal(outs[0], outs[1])
    assert not np.array_equal(outs[0][:8], 0 * outs[0][:8])


# ---- the convolution on the tensor cores (option "forward_path") ------------------------------------
@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("n", [1, 5, 16, 17, 100, 2368 + 5, 4099])
def test_tensor_core_forward_three_passes_matches_oracle(cuda, pkg, ob, params0, n, fast):
    """forward_path = 1: tcgen05 convolution in three passes of fp16 parts keeps the 1e-5 bar of the fp32 path."""
    images, _ = pkg.synth.synth_images(21, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(fast)
    net.set_option("forward_path", 1)
    out, arg = run_forward(cuda, net, images)
    ref_out, ref_arg = ob.forward_batch(params0, images)
    assert rel_err(out, ref_out) < 1e-5
    check_argmax(arg, ref_arg, ref_out, "tensor cores, three passes, n=%d flavour %d" % (n, fast))
    assert np.array_equal(arg, np.argmax(out, axis=1).astype(np.int32))


def test_tensor_core_forward_full_size(cuda, pkg, ob, params0):
    """Benchmark configuration 2 at full size on both tensor-core paths.  Path 1 (three passes): 1e-5
    on every sigmoid, argmax on every clear-margin row.  Path 2 (one pass of the high parts, tanh.approx sigmoid) is
    a reduced-precision mode: its bar is 5e-3 absolute on the sigmoids and argmax equality on every
    row whose top-two margin is clear of that error (1e-2 relative); both counts are printed."""
    n = 65536
    images, _ = pkg.synth.synth_images(1, n)
    ref_out, ref_arg = ob.forward_batch(params0, images, threads=0)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("forward_path", 1)
    out, arg = run_forward(cuda, net, images)
    err = rel_err(out, ref_out)
    print("three passes: max relative error of the sigmoids %.3e" % err)
    assert err < 1e-5
    check_argmax(arg, ref_arg, ref_out, "65,536 images, tensor cores, three passes")
    # bit-repeatable, and independent of where an image sits in the batch
    out2, arg2 = run_forward(cuda, net, images[1000:3000])
    assert np.array_equal(out2, out[1000:3000]) and np.array_equal(arg2, arg[1000:3000])
    net.set_option("forward_path", 2)
    out, arg = run_forward(cuda, net, images)
    abs_err = float(np.max(np.abs(out.astype(np.float64) - ref_out)))
    print("one pass + tanh: max absolute error of the sigmoids %.3e, mean %.3e"
          % (abs_err, float(np.mean(np.abs(out.astype(np.float64) - ref_out)))))
    assert abs_err < 5e-3
    check_argmax(arg, ref_arg, ref_out, "65,536 images, tensor cores, one pass + tanh", tol=1e-2,
                 max_masked_frac=0.05)
    assert np.array_equal(arg, np.argmax(out, axis=1).astype(np.int32))


def test_tensor_core_forward_optional_outputs_and_host_pipeline(cuda, pkg, params0):
    n = 8192 + 300
    images, _ = pkg.synth.synth_images(28, n)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("forward_path", 1)
    out, arg = run_forward(cuda, net, images)
    o2, _ = run_forward(cuda, net, images, want_arg=False)
    _, a2 = run_forward(cuda, net, images, want_out=False)
    assert np.array_equal(o2, out) and np.array_equal(a2, arg)
    h_out = np.empty((n, 10), dtype=np.float32)
    h_arg = np.empty((n,), dtype=np.int32)
    net.forward_host(images, n, h_out, h_arg)
    assert np.array_equal(h_out, out) and np.array_equal(h_arg, arg)


def test_default_kernel_choice_follows_batch_size(cuda, pkg, params0):
    """forward_path = -1 (the default): below 6,144 images per call the CUDA-core kernel answers, from
    6,144 on the three-pass tensor-core kernel -- bit for bit in both cases; with the reference's
    sigmoid expression selected the default stays on the CUDA-core kernel at every size."""
    images, _ = pkg.synth.synth_images(29, 6144)
    outs = {}
    for path in (-1, 0, 1):
        net = pkg.Net(0)
        net.set_params(params0)
        net.set_option("forward_path", path)
        outs[path] = (run_forward(cuda, net, images[:6143]), run_forward(cuda, net, images))
    assert np.array_equal(outs[-1][0][0], outs[0][0][0]) and np.array_equal(outs[-1][0][1], outs[0][0][1])
    assert np.array_equal(outs[-1][1][0], outs[1][1][0]) and np.array_equal(outs[-1][1][1], outs[1][1][1])
    assert not np.array_equal(outs[0][1][0], outs[1][1][0])     # the two kernels do differ in the last bits
    ref = {}
    for path in (-1, 0):
        net = pkg.Net(0)
        net.set_params(params0)
        net.set_fast_sigmoid(0)
        net.set_option("forward_path", path)
        ref[path] = run_forward(cuda, net, images)
    assert np.array_equal(ref[-1][0], ref[0][0])


@pytest.mark.parametrize("what", ["largest", "out of range", "not a number", "uint8", "tiny weights", "huge weights"])
@pytest.mark.parametrize("n", [3, 148 * 16 + 21])
def test_tensor_core_forward_operand_range(cuda, pkg, params0, what, n):
    """The tensor-core kernel's operands are fp16 parts of scaled values: pixels up to 65,519 / scale go through them, an
    image with a larger pixel or a NaN is computed in fp32 (its neighbours are not touched), weights of any magnitude
    are scaled with the pixels, and uint8 pixels give the bits of the fp32 images they stand for.  Reference: the fp32
    CUDA-core kernel."""
    pix = pkg.synth.synth_pixels_u8(41, n)
    images = pkg.synth.u8_to_float(pix)
    params = params0.copy()
    spots = [0, n // 2, n - 1]
    limit = 65520.0 / (255 * 2.0 ** (np.floor(np.log2(np.abs(params[:150]).max() * 1.442695)) - 3))
    if what == "largest":
        images[spots, 5, 7] = limit * (1 - 1e-4)
    elif what == "out of range":
        images[spots, 27, 27] = limit * (1 + 1e-6)
        images[spots[0], 0, 0] = -3e6
    elif what == "not a number":
        images[spots, 11, 12] = np.nan
    elif what.endswith("weights"):
        params[:150] *= np.float32(1e-6 if what == "tiny weights" else 1e6)
        images *= np.float32(1e4 if what == "tiny weights" else 1e-6)
    net = pkg.Net(0)
    net.set_params(params)
    outs = {}
    for path in (0, 1):
        net.set_option("forward_path", path)
        outs[path] = run_forward(cuda, net, images)
        assert net.status() == 0
    if what == "uint8":
        d_pix = cuda.from_numpy(pix).cuda()
        d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
        d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
        net.forward_u8(d_pix, n, d_out, d_arg)
        cuda.cuda.synchronize()
        assert np.array_equal(d_out.cpu().numpy(), outs[1][0]) and np.array_equal(d_arg.cpu().numpy(), outs[1][1])
    assert np.array_equal(np.isnan(outs[0][0]), np.isnan(outs[1][0]))
    keep = ~np.isnan(outs[0][0]).any(axis=1)
    assert keep.sum() == n - (len(set(spots)) if what == "not a number" else 0)
    assert rel_err(outs[1][0][keep], outs[0][0][keep]) < 1e-5


@pytest.mark.parametrize("what,tol", [("weights x 4000", 2e-3), ("weights x 1e5", 5e-2), ("infinite bias", 1e-5), ("not a number", 0),
                                      ("blank image, weights x 1e32", 1e-5)])
@pytest.mark.parametrize("n", [3, 148 * 16 + 21])
def test_tensor_core_forward_uint8_parameter_range(cuda, pkg, params0, what, tol, n):
    """uint8 pixels meet the same limits as the fp32 images they stand for: with weights whose pixel scale takes them out of fp16's
    range, or with parameters that are not finite, the tensor-core kernel computes them in fp32, to the fp32 images' bits.  Yardstick:
    the CUDA-core kernel; a pre-activation of 25 terms up to 0.5 * factor is only known to 25 * 0.5 * factor * 2^-24 in fp32,
    3e-3 and 7e-2 here, and a sigmoid's slope is at most 1/4 at the windows that it does not saturate."""
    pix = pkg.synth.synth_pixels_u8(47, n)
    params = params0.copy()
    if "weights" in what:
        params[:150] *= np.float32(what.split()[-1])
    if what.startswith("blank"):
        pix[:] = 0
    elif what == "infinite bias":
        params[150] = np.inf
    elif what == "not a number":
        params[77] = np.nan
    images = pkg.synth.u8_to_float(pix)
    d_pix = cuda.from_numpy(pix).cuda()
    outs = {}
    for path in (0, 1):
        net = pkg.Net(0)
        net.set_params(params)
        net.set_option("forward_path", path)
        d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
        d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
        net.forward_u8(d_pix, n, d_out, d_arg)
        cuda.cuda.synchronize()
        outs[path] = d_out.cpu().numpy()
        out, arg = run_forward(cuda, net, images)
        assert net.status() == 0
        assert np.array_equal(outs[path], out, equal_nan=True) and np.array_equal(d_arg.cpu().numpy(), arg)
    if what == "not a number":
        assert np.isnan(outs[0]).all() and np.isnan(outs[1]).all()
    else:
        assert float(np.max(np.abs(outs[1].astype(np.float64) - outs[0]))) < tol


@pytest.mark.parametrize("factor", [1e-9, 1e-6, 1e-3, 1.0, 30.0, 900.0])
@pytest.mark.parametrize("n", [5, 148 * 16 + 21])
def test_tensor_core_forward_bytes_beside_other_pixels(cuda, pkg, params0, factor, n):
    """Pixels that are bytes / 255 leave no fp16 remainder, and a tile of them skips the pass that multiplies remainders: they give the
    same bits as uint8 pixels and beside images with remainders, at every weight scale (the pixels' scale follows it, and the byte conversion
    has two ranges).  Yardstick for the others: the fp32 CUDA-core kernel; a pre-activation of 25 terms up to 0.5 * factor is
    known to 25 * 0.5 * factor * 2^-23 in fp32, a sigmoid's slope is at most 1/4, and 216 of them meet weights up to 0.5."""
    pix = pkg.synth.synth_pixels_u8(53, n)
    images = pkg.synth.u8_to_float(pix)
    params = params0.copy()
    params[:150] *= np.float32(factor)
    rng = np.random.default_rng(3)
    mixed = images.copy()
    mixed[2::7] *= rng.uniform(0.5, 1.0, mixed[2::7].shape).astype(np.float32)
    net = pkg.Net(0)
    net.set_params(params)
    net.set_option("forward_path", 1)
    out, arg = run_forward(cuda, net, images)
    out_m, _ = run_forward(cuda, net, mixed)
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    net.forward_u8(cuda.from_numpy(pix).cuda(), n, d_out, None)
    cuda.cuda.synchronize()
    assert np.array_equal(d_out.cpu().numpy(), out)
    same = np.arange(n) % 7 != 2
    assert np.array_equal(out_m[same], out[same])
    net.set_option("forward_path", 0)
    ref, _ = run_forward(cuda, net, mixed)
    assert net.status() == 0
    tol = max(1e-5, 216 * 0.5 / 4 / 4 * 25 * 0.5 * factor * 2.0 ** -23)
    assert rel_err(out_m, ref) < tol


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("n", [2, 297, 888, 889, 895, 2073])
def test_cuda_core_forward_around_its_dispatch(cuda, pkg, params0, n, fast):
    """The one-image kernel (up to six images per SM) and the tile kernel above it, at one image more than the resident
    blocks, at the dispatch line, at a ragged last tile and at one tile more than a round, fp32 and uint8.  Reference: the
    tensor-core kernel, which is checked against the oracle."""
    pix = pkg.synth.synth_pixels_u8(43, n)
    images = pkg.synth.u8_to_float(pix)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_fast_sigmoid(fast)
    net.set_option("forward_path", 1)
    ref, _ = run_forward(cuda, net, images)
    net.set_option("forward_path", 0)
    out, arg = run_forward(cuda, net, images)
    assert rel_err(out, ref) < 1e-5 and np.array_equal(arg, np.argmax(out, axis=1).astype(np.int32))
    d_pix = cuda.from_numpy(pix).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    net.forward_u8(d_pix, n, d_out, None)
    cuda.cuda.synchronize()
    assert net.status() == 0 and np.array_equal(d_out.cpu().numpy(), out)


@pytest.mark.parametrize("n", [370, 371, 444, 445, 666, 667, 1035, 1036, 1037, 2071, 2072, 2081, 4147])
def test_cuda_core_forward_tiles_of_equal_length(cuda, pkg, params0, n):
    """Both sides of the lines at 2.5, 3 and 4.5 images per SM (148 of them) between the one-image and the tile kernel, of a tile on each
    SM and of a round of tiles, and last tiles of two and three images with warps that have none.  Reference as above."""
    pix = pkg.synth.synth_pixels_u8(47, n)
    images = pkg.synth.u8_to_float(pix)
    net = pkg.Net(0)
    net.set_params(params0)
    net.set_option("forward_path", 1)
    ref, _ = run_forward(cuda, net, images)
    net.set_option("forward_path", 0)
    out, arg = run_forward(cuda, net, images)
    assert rel_err(out, ref) < 1e-5 and np.array_equal(arg, np.argmax(out, axis=1).astype(np.int32))
    d_pix, d_out = cuda.from_numpy(pix).cuda(), cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    net.forward_u8(d_pix, n, d_out, None)
    cuda.cuda.synchronize()
    assert net.status() == 0 and np.array_equal(d_out.cpu().numpy(), out)


@pytest.mark.parametrize("u8", [False, True])
@pytest.mark.parametrize("n", [41, 200, 1024, 1025, 9001, 17000])
def test_forward_host_buffers_pageable_and_pinned(cuda, pkg, params0, n, u8):
    """The host pipeline around its sizes: below and above staging, one and two chunks, pieces that wrap around the ring, a
    ragged end; pageable and pinned images, pageable and pinned results, either result left out -- always the bits of the
    device call.  A second net runs the same request from another thread (one of the two finds the copy threads busy)."""
    import threading
    pix = pkg.synth.synth_pixels_u8(44, n)
    images = pix if u8 else pkg.synth.u8_to_float(pix)
    nets = [pkg.Net(0), pkg.Net(0)]
    for net in nets:
        net.set_params(params0)
    d_img = cuda.from_numpy(images).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_arg = cuda.empty((n,), dtype=cuda.int32, device="cuda")
    (nets[0].forward_u8 if u8 else nets[0].forward)(d_img, n, d_out, d_arg)
    cuda.cuda.synchronize()
    want, want_arg = d_out.cpu().numpy(), d_arg.cpu().numpy()

    def check(net, img, out, arg):
        (net.forward_u8_host if u8 else net.forward_host)(img, n, out, arg)
        assert out is None or np.array_equal(np.asarray(out), want)
        assert arg is None or np.array_equal(np.asarray(arg), want_arg)

    def pageable():
        return np.full((n, 10), -1, np.float32), np.full(n, -1, np.int32)

    pinned_img = cuda.from_numpy(images).pin_memory()
    check(nets[0], images, *pageable())
    check(nets[0], images, pageable()[0], None)
    check(nets[0], images, None, pageable()[1])
    check(nets[0], pinned_img, *pageable())
    check(nets[0], pinned_img, cuda.empty((n, 10)).pin_memory(), cuda.empty(n, dtype=cuda.int32).pin_memory())
    failed = []

    def other():
        try:
            for _ in range(3):
                check(nets[1], images, *pageable())
        except Exception as e:      # reported by the main thread
            failed.append(e)
    t = threading.Thread(target=other)
    t.start()
    for _ in range(3):
        check(nets[0], images, *pageable())
    t.join()
    assert not failed


def test_forward_host_with_nets_that_come_and_go(cuda, pkg, params0):
    """Each net sets the pipeline up and, as the last of them, takes the shared threads and ring down again: pageable requests, a
    small one that is not staged first, results pinned or left out, always the bits of the device call."""
    n = 3000
    pix = pkg.synth.synth_pixels_u8(45, n)
    d_pix = cuda.from_numpy(pix).cuda()
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    for turn in range(4):
        net = pkg.Net(0)
        net.set_params(params0)
        net.forward_u8(d_pix, n, d_out, None)
        cuda.cuda.synchronize()
        want = d_out.cpu().numpy()
        if turn % 2:
            out = np.empty((20, 10), np.float32)
            net.forward_u8_host(pix[:20], 20, out, None)
            assert rel_err(out, want[:20]) < 1e-5      # (so few images go through another kernel)
        if turn == 2:
            net.forward_u8_host(pix, n, None, None)
        out = cuda.empty((n, 10)).pin_memory() if turn == 3 else np.empty((n, 10), np.float32)
        net.forward_u8_host(pix, n, out, None)
        assert np.array_equal(np.asarray(out), want)
        net.close()


@pytest.mark.parametrize("n", [1026, 2047, 41000])
def test_forward_host_last_chunk_is_shorter(cuda, pkg, params0, n):
    """Equal chunks and a last one, for pageable images of a quarter of the request, 512 at least and 2,048 at most (514 and 512, 1,535 and 512), for
    pinned ones of so few bytes of half of it (513 twice, 1,024 and 1,023); and six chunks in four slots, whose pageable results are handed over
    before a slot is used again; always the bits of the device call."""
    pix = pkg.synth.synth_pixels_u8(48, n)
    net = pkg.Net(0)
    net.set_params(params0)
    d_out = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    d_arg = cuda.empty(n, dtype=cuda.int32, device="cuda")
    net.forward_u8(cuda.from_numpy(pix).cuda(), n, d_out, d_arg)
    cuda.cuda.synchronize()
    for pinned in (False, True):
        img = cuda.from_numpy(pix).pin_memory() if pinned else pix
        out, arg = np.full((n, 10), -1, np.float32), np.full(n, -1, np.int32)
        net.forward_u8_host(img, n, out, arg)
        assert np.array_equal(out, d_out.cpu().numpy()) and np.array_equal(arg, d_arg.cpu().numpy())


def test_forward_host_memory_stays_whatever_the_order_of_sizes(cuda, pkg, params0):
    """The chunks of a larger request can be the shorter ones (10,000 images 7,952 and the rest, 11,000 two of 4,476): a net that has seen all sizes
    allocates nothing any more, whichever comes next, and the results are the bits of the device call at every one."""
    sizes = [10000, 11000, 20000, 1500]
    pix = pkg.synth.synth_pixels_u8(46, max(sizes))
    d_pix = cuda.from_numpy(pix).cuda()
    d_out = cuda.empty((max(sizes), 10), dtype=cuda.float32, device="cuda")
    net = pkg.Net(0)
    net.set_params(params0)
    free = []
    for turn in range(3):
        for n in sizes if turn < 2 else sizes[::-1]:
            out = np.empty((n, 10), np.float32)
            net.forward_u8_host(pix[:n], n, out, None)
            free.append((turn, cuda.cuda.mem_get_info()[0]))
            net.forward_u8(d_pix, n, d_out, None)
            cuda.cuda.synchronize()
            assert np.array_equal(out, d_out[:n].cpu().numpy())
    assert len({left for turn, left in free if turn > 0}) == 1


def test_forward_host_small_pinned_requests_run_in_halves(cuda, pkg, params0):
    """1,100 pinned images are two chunks of 550, for which a new net takes 3.5 MB of device memory (1,024 and 76: 6.5 MB).
    Behind a request of 20, which creates the streams; median over nets, because small allocations share granules."""
    n = 1100
    images = cuda.from_numpy(pkg.synth.u8_to_float(pkg.synth.synth_pixels_u8(49, n))).pin_memory()
    want = cuda.empty((n, 10), dtype=cuda.float32, device="cuda")
    nets, taken = [], []
    for _ in range(9):
        nets.append(pkg.Net(0))
        nets[-1].set_params(params0)
        out = cuda.empty((n, 10)).pin_memory()
        nets[-1].forward_host(images[:20], 20, out[:20], None)
        cuda.cuda.synchronize()
        before = cuda.cuda.mem_get_info()[0]
        nets[-1].forward_host(images, n, out, None)
        taken.append(before - cuda.cuda.mem_get_info()[0])
        nets[-1].forward(images.cuda(), n, want, None)
        cuda.cuda.synchronize()
        assert cuda.equal(out, want.cpu())
    assert sorted(taken)[len(taken) // 2] <= 4 << 20
