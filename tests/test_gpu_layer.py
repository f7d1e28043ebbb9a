"""Layer- and network-level parity on the GPU through the reference-facing API
(streambrain_b200.{StructuralPlasticityLayer, DenseLayer, Network}), against the
golden trajectories of the reference cpu backend and against the CPU oracle at
the MNIST-shaped configuration; full-size STL-10-shaped checks use properties that
do not need a full CPU run."""
import ctypes
import random

import numpy as np
import pytest

from conftest import TOL, load_golden, mask_mismatch_is_a_tie, rel_inf, weight_err

import oracle

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("contraction_path")]

DTYPES = [("f32", np.float32), ("f64", np.float64)]
PLASTIC_STATE = ("weights", "bias", "Ci", "Cj", "Cij", "kbi", "wmask")


@pytest.fixture(scope="module")
def B200():
    import streambrain_b200
    return streambrain_b200


def _layers_from_golden(B200, g, dtype):
    H, Mc, n_pix = int(g["H"]), int(g["Mc"]), int(g["n_pix"])
    np.random.seed(0)
    layer = B200.StructuralPlasticityLayer(2 * n_pix, H, Mc, float(g["hp_taupdt"]), float(g["hp_khalf"]),
                                           float(g["hp_pmin"]), float(g["hp_taubdt"]), float(g["hp_density"]), 16,
                                           (1, 1 / Mc, 1 / Mc), dtype=dtype)
    dense = B200.DenseLayer(H * Mc, 1, 10, float(g["dense_taupdt"]), (1 / Mc, 1 / 10, 1 / Mc / 10), dtype=dtype)
    for name in PLASTIC_STATE:
        setattr(layer, name, g["init_" + name])
    for name in ("weights", "bias", "Ci", "Cj", "Cij"):
        setattr(dense, name, g["dinit_" + name])
    return layer, dense


@pytest.mark.parametrize("tag,dtype", DTYPES)
def test_layer_steps_teacher_forced_vs_golden(B200, tag, dtype):
    g = load_golden("layer_%s.npz" % tag)
    tol = TOL[np.dtype(dtype)]
    layer, dense = _layers_from_golden(B200, g, dtype)
    B, steps, Mc = int(g["B"]), int(g["steps"]), int(g["Mc"])
    for s in range(steps):
        x = g["x"][s * B:(s + 1) * B]
        lab = g["labels"][s * B:(s + 1) * B]
        act = layer.compute_activation(x)
        assert rel_inf(act, g["act_%d" % s]) < tol, s
        assert rel_inf(dense.compute_activation(g["act_%d" % s]), g["dact_%d" % s]) < tol, s
        h = int(g["hs"][s])
        before = layer.wmask
        dense.train_step(g["act_%d" % s], lab)
        layer.train_step(x, g["act_%d" % s], None if h < 0 else h)
        for name in ("Ci", "Cj", "Cij", "kbi", "bias"):
            assert rel_inf(getattr(layer, name), g["s%d_%s" % (s, name)]) < tol, (s, name)
        got_mask = layer.wmask
        want = {n: g["s%d_%s" % (s, n)] for n in PLASTIC_STATE}
        if dtype == np.float64:
            assert np.array_equal(got_mask, want["wmask"]), s
        else:
            assert mask_mismatch_is_a_tie(got_mask, want["wmask"], max(h, 0), before, want,
                                          float(g["hp_taupdt"]) / 2, Mc, 1e-5), s
        if np.array_equal(got_mask, want["wmask"]):
            W = layer.weights
            assert weight_err(W, want["weights"]) < 10 * tol, s
            assert np.array_equal(W == 0, want["weights"] == 0), s
        for name in ("Ci", "Cj", "Cij"):
            assert rel_inf(getattr(dense, name), g["d%d_%s" % (s, name)]) < tol, (s, name)
        assert weight_err(dense.weights, g["d%d_weights" % s]) < 10 * tol, s
        for name in PLASTIC_STATE:
            setattr(layer, name, want[name])
        for name in ("weights", "Ci", "Cj", "Cij"):
            setattr(dense, name, g["d%d_%s" % (s, name)])
    dense.train_finalize()
    assert rel_inf(dense.bias, g["dfinal_bias"]) < tol


def test_layer_free_run_f64_vs_golden(B200):
    g = load_golden("layer_f64.npz")
    layer, _ = _layers_from_golden(B200, g, np.float64)
    B, steps = int(g["B"]), int(g["steps"])
    for s in range(steps):
        x = g["x"][s * B:(s + 1) * B]
        act = layer.compute_activation(x)
        h = int(g["hs"][s])
        layer.train_step(x, act, None if h < 0 else h)
        assert np.array_equal(layer.wmask, g["s%d_wmask" % s]), s
    assert rel_inf(layer.Cij, g["s%d_Cij" % (steps - 1)]) < 1e-10
    assert rel_inf(layer.weights, g["s%d_weights" % (steps - 1)]) < 1e-9


def test_device_tensor_path_equals_host_path(B200):
    """CUDA tensors in -> CUDA tensors out must give the same numbers as numpy in/out,
    and the fused host step (one upload) the same as forward + train_step."""
    import torch
    g = load_golden("layer_f32.npz")
    B = int(g["B"])
    x = g["x"][:B]
    la, _ = _layers_from_golden(B200, g, np.float32)
    lb, _ = _layers_from_golden(B200, g, np.float32)
    lc, _ = _layers_from_golden(B200, g, np.float32)
    ya = la.compute_activation(x)
    la.train_step(x, ya, 1)
    xt = torch.from_numpy(x).cuda()
    yb = lb.compute_activation(xt)
    lb.train_step(xt, yb, 1)
    torch.cuda.synchronize()
    yc = lc.step_host(x, None, 1)
    assert np.array_equal(ya, yb.cpu().numpy()) and np.array_equal(ya, yc)
    for name in PLASTIC_STATE:
        assert np.array_equal(getattr(la, name), getattr(lb, name)), name
        assert np.array_equal(getattr(la, name), getattr(lc, name)), name
    t = lb.state_tensor("Cij")
    assert t.is_cuda and np.array_equal(t.cpu().numpy(), lb.Cij)


def test_row_block_products_with_reserved_sms(B200):
    """The persistent row-block product may leave multiprocessors to a collective running beside
    it (sbb_set_reserved_sms): a smaller grid walks the same tiles and must give the same sums."""
    import torch
    from streambrain_b200._lib import check, lib

    class Done:
        def wait(self):
            pass

    g = load_golden("layer_f32.npz")
    B = int(g["B"])
    x = torch.from_numpy(np.ascontiguousarray(g["x"][:B])).cuda()
    full, _ = _layers_from_golden(B200, g, np.float32)
    fewer, _ = _layers_from_golden(B200, g, np.float32)
    y = full.compute_activation(x)
    full.dp_train_step(x, y, 1, 1, lambda t: Done(), row_blocks=2)
    try:
        check(lib.sbb_set_reserved_sms(140))
        fewer.dp_train_step(x, y, 1, 1, lambda t: Done(), row_blocks=2)
    finally:
        check(lib.sbb_set_reserved_sms(0))
    torch.cuda.synchronize()
    for name in PLASTIC_STATE:
        assert np.array_equal(getattr(fewer, name), getattr(full, name)), name


def test_async_host_steps_equal_blocking_host_steps(B200):
    """Five pipelined host-buffer steps (copies double-buffered against the steps, page-locked
    buffers) leave the same state and return the same activations as five blocking calls."""
    import torch
    g = load_golden("layer_f32.npz")
    B, steps = int(g["B"]), 5
    blocking, _ = _layers_from_golden(B200, g, np.float32)
    piped, _ = _layers_from_golden(B200, g, np.float32)
    xs = [torch.from_numpy(np.ascontiguousarray(g["x"][s * B:(s + 1) * B])).pin_memory() for s in range(steps)]
    outs = [torch.empty((B, piped.out_features), dtype=torch.float32).pin_memory() for _ in range(steps)]
    want = [blocking.step_host(xs[s].numpy(), None, s % 3) for s in range(steps)]
    for s in range(steps):
        piped.step_host_async(xs[s].numpy(), None, s % 3, out=outs[s].numpy())
    piped.wait()
    for s in range(steps):
        assert np.array_equal(outs[s].numpy(), want[s]), s
    for name in PLASTIC_STATE:
        assert np.array_equal(getattr(piped, name), getattr(blocking, name)), name
    # the blocking entry points work again after wait()
    assert np.array_equal(piped.step_host(xs[0].numpy(), None, 1), blocking.step_host(xs[0].numpy(), None, 1))


@pytest.mark.parametrize("tag,dtype", DTYPES)
def test_network_fit_and_evaluate_vs_golden(B200, tag, dtype):
    g = load_golden("network_%s.npz" % tag)
    n_pix, H, Mc, B = int(g["n_pix"]), int(g["H"]), int(g["Mc"]), int(g["B"])
    n_train, seed = int(g["n_train"]), int(g["seed"])
    np.random.seed(seed)
    random.seed(seed)
    net = B200.Network(dtype)
    net.verbose = False
    net.add_layer(B200.StructuralPlasticityLayer(2 * n_pix, H, Mc, 0.03, -40.0, 0.1, 0.05, 0.5, 16,
                                                 (1, 1 / Mc, 1 / Mc)))
    net.add_layer(B200.DenseLayer(H * Mc, 1, 10, 0.02, (1 / Mc, 1 / 10, 1 / Mc / 10)))
    x, lab = g["x"], g["labels"]
    net.fit(x[:n_train], lab[:n_train], B, [(0, 3)])
    net.fit(x[:n_train], lab[:n_train], B, [(1, 2)])
    correct, total = net.evaluate(x[n_train:], lab[n_train:], B)
    assert int(total[0]) == int(g["total"][0])
    if dtype == np.float64:
        assert np.array_equal(net._layers[0].wmask, g["l0_wmask"])
        for li, layer in enumerate(net._layers):
            for name in ("Ci", "Cj", "Cij", "bias", "weights"):
                assert rel_inf(getattr(layer, name), g["l%d_%s" % (li, name)]) < 1e-9, (li, name)
        assert int(correct[0]) == int(g["correct"][0])
        act = x[n_train:]
        for layer in net._layers:
            act = layer.compute_activation(act)
        assert np.array_equal(np.argmax(act, axis=1), g["test_pred"])
    else:
        for name in ("Ci", "Cj"):
            assert rel_inf(getattr(net._layers[0], name), g["l0_" + name]) < 1e-3, name


def _small_network(B200, g, dtype):
    n_pix, H, Mc = int(g["n_pix"]), int(g["H"]), int(g["Mc"])
    net = B200.Network(dtype)
    net.verbose = False
    net.add_layer(B200.StructuralPlasticityLayer(2 * n_pix, H, Mc, 0.03, -40.0, 0.1, 0.05, 0.5, 16,
                                                 (1, 1 / Mc, 1 / Mc)))
    net.add_layer(B200.DenseLayer(H * Mc, 1, 10, 0.02, (1 / Mc, 1 / 10, 1 / Mc / 10)))
    return net


def test_network_with_reduction_callbacks_reproduces_golden_run(B200):
    """The native loop with the data-parallel callbacks installed (one rank: the sum over ranks is the
    identity) runs the split step -- row-block products, reduction, row-block apply -- for every batch
    and must land on the reference's golden run like the fused step does."""
    g = load_golden("network_f64.npz")
    B, n_train, seed = int(g["B"]), int(g["n_train"]), int(g["seed"])
    np.random.seed(seed)
    random.seed(seed)
    net = _small_network(B200, g, np.float64)

    class Done:
        def wait(self):
            pass

    started = []
    net.set_data_parallel(0, 1, all_reduce=lambda t: started.append(t.numel()) or Done())
    x, lab = g["x"], g["labels"]
    net.fit(x[:n_train], lab[:n_train], B, [(0, 3)])
    net.fit(x[:n_train], lab[:n_train], B, [(1, 2)])
    correct, total = net.evaluate(x[n_train:], lab[n_train:], B)
    assert len(started) > 0
    assert np.array_equal(net._layers[0].wmask, g["l0_wmask"])
    for li, layer in enumerate(net._layers):
        for name in ("Ci", "Cj", "Cij", "bias", "weights"):
            assert rel_inf(getattr(layer, name), g["l%d_%s" % (li, name)]) < 1e-9, (li, name)
    assert int(correct[0]) == int(g["correct"][0]) and int(total[0]) == int(g["total"][0])


@pytest.mark.parametrize("tag,dtype", DTYPES)
def test_checkpoint_resume_equals_uninterrupted_run(B200, tmp_path, tag, dtype):
    """save() after two epochs, load() into a fresh network, continue: bit-identical to the run that was
    never interrupted (the random stream is carried over as well, as a resumed job would)."""
    g = load_golden("network_%s.npz" % tag)
    B, n_train = int(g["B"]), int(g["n_train"])
    x, lab = g["x"][:n_train], g["labels"][:n_train]

    np.random.seed(5)
    whole = _small_network(B200, g, dtype)
    whole.fit(x, lab, B, [(0, 2)])
    whole.fit(x, lab, B, [(0, 2), (1, 1)])

    np.random.seed(5)
    first = _small_network(B200, g, dtype)
    first.fit(x, lab, B, [(0, 2)])
    first.save(tmp_path / "ckpt.npz")
    rng = np.random.get_state()
    del first

    np.random.seed(99)                      # a fresh process: other initial weights, another stream
    resumed = _small_network(B200, g, dtype)
    resumed.load(tmp_path / "ckpt.npz")
    np.random.set_state(rng)
    resumed.fit(x, lab, B, [(0, 2), (1, 1)])
    for a, b in zip(whole._layers, resumed._layers):
        for name in a._state_names:
            assert np.array_equal(getattr(a, name), getattr(b, name)), name
    assert np.array_equal(whole.evaluate(g["x"][n_train:], g["labels"][n_train:], B)[0],
                          resumed.evaluate(g["x"][n_train:], g["labels"][n_train:], B)[0])
    with pytest.raises(ValueError):
        B200.Network(dtype).load(tmp_path / "ckpt.npz")     # layer count mismatch


def test_network_too_few_batches_for_the_mask_schedule(B200):
    np.random.seed(0)
    net = B200.Network(np.float32)
    net.verbose = False
    net.add_layer(B200.StructuralPlasticityLayer(8, 4, 2, 0.05, -10.0, 0.1, 0.1, 0.5, 16, (1, 0.5, 0.5)))
    net.add_layer(B200.DenseLayer(8, 1, 10, 0.05, (0.5, 0.1, 0.05)))
    from streambrain_b200 import synthetic
    x, lab = synthetic.make_inputs(16, 4, 0.5, np.float32)
    with pytest.raises(ZeroDivisionError):
        net.fit(x, lab, 8, [(0, 2)])
    net.fit(x, lab, 8, [(0, 1)])
    correct, total = net.evaluate(x, lab, 8)
    assert int(total[0]) == 16 and 0 <= int(correct[0]) <= 16


def _mnist_pair(B200, port_kernels, dtype, seed=0):
    from streambrain_b200 import synthetic
    p = synthetic.layer_params("mnist_f32" if dtype == np.float32 else "mnist_f64")
    hp = p["hidden"]
    np.random.seed(seed)
    dev = B200.StructuralPlasticityLayer(hp["in_features"], hp["hypercolumns"], hp["minicolumns"], hp["taupdt"],
                                         hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"], 16,
                                         hp["initial_counters"], dtype=dtype)
    np.random.seed(seed)
    ref = oracle.OracleLayer(port_kernels, "plastic", hp["in_features"], hp["hypercolumns"], hp["minicolumns"],
                             hp["taupdt"], hp["initial_counters"], dtype, khalf=hp["khalf"], pmin=hp["pmin"],
                             taubdt=hp["taubdt"], density=hp["density"])
    x, lab = synthetic.make_inputs(p["batch"] * 6, p["n_pixels"], p["sparsity"], dtype)
    return dev, ref, x, lab, p


@pytest.mark.parametrize("tag,dtype", DTYPES)
def test_mnist_shaped_layer_teacher_forced_vs_oracle(B200, port_kernels, tag, dtype):
    """1568 -> 30x100, batch 128: identical seeded initial state (the constructor draws
    from the global NumPy stream in the reference's order), six steps, mask update from
    the third step on, every step restarted from the oracle's state."""
    dev, ref, x, _, p = _mnist_pair(B200, port_kernels, dtype)
    tol = TOL[np.dtype(dtype)]
    for name in PLASTIC_STATE:
        assert np.array_equal(getattr(dev, name), getattr(ref, name)), name
    B = p["batch"]
    Mc = p["hidden"]["minicolumns"]
    for s in range(6):
        xb = x[s * B:(s + 1) * B]
        a_ref = ref.compute_activation(xb)
        a_dev = dev.compute_activation(xb)
        assert rel_inf(a_dev, a_ref) < tol, s
        h = (7 * s) % 30 if s >= 2 else None
        before = ref.wmask.copy()
        ref.train_step(xb, a_ref, h)
        dev.train_step(xb, a_ref, h)
        for name in ("Ci", "Cj", "Cij", "kbi", "bias"):
            assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, (s, name)
        got = dev.wmask
        if dtype == np.float64:
            assert np.array_equal(got, ref.wmask), s
        else:
            assert mask_mismatch_is_a_tie(got, ref.wmask, h or 0, before, ref.state(), p["hidden"]["taupdt"] / 2, Mc,
                                          1e-5), s
        if np.array_equal(got, ref.wmask):
            assert weight_err(dev.weights, ref.weights) < 10 * tol, s
        for name in PLASTIC_STATE:
            setattr(dev, name, getattr(ref, name))


def test_mnist_shaped_argmax_predictions_identical(B200, port_kernels):
    """Classifier argmax on held-out samples after identical (teacher-forced) training state."""
    from streambrain_b200 import synthetic
    dev, ref, x, lab, p = _mnist_pair(B200, port_kernels, np.float64)
    op = p["out"]
    np.random.seed(1)
    dev_out = B200.DenseLayer(op["in_features"], 1, 10, op["taupdt"], op["initial_counters"], dtype=np.float64)
    np.random.seed(1)
    ref_out = oracle.OracleLayer(port_kernels, "dense", op["in_features"], 1, 10, op["taupdt"],
                                 op["initial_counters"], np.float64)
    B = p["batch"]
    for s in range(4):
        xb, lb = x[s * B:(s + 1) * B], lab[s * B:(s + 1) * B]
        a = ref.compute_activation(xb)
        ref_out.train_step(a, lb)
        dev_out.train_step(a, lb)
    ref_out.train_finalize()
    dev_out.train_finalize()
    xt = x[4 * B:]
    hidden = ref.compute_activation(xt)
    assert np.array_equal(np.argmax(dev_out.compute_activation(hidden), axis=1),
                          np.argmax(ref_out.compute_activation(hidden), axis=1))
    assert np.array_equal(np.argmax(dev_out.compute_activation(dev.compute_activation(xt)), axis=1),
                          np.argmax(ref_out.compute_activation(hidden), axis=1))


def test_data_parallel_split_step_equals_single_step(B200):
    """Two ranks emulated on one GPU through the C ABI: each half batch fills its own
    delta buffer, the buffers are summed (standing in for the allreduce), and the
    apply calls must reproduce the single-device step on the whole batch."""
    import torch
    from streambrain_b200._lib import check, lib
    g = load_golden("layer_f64.npz")
    B = int(g["B"])
    x = torch.from_numpy(g["x"][:B]).cuda()
    single, _ = _layers_from_golden(B200, g, np.float64)
    split, _ = _layers_from_golden(B200, g, np.float64)
    y = single.compute_activation(x)
    single.train_step(x, y, 2)
    n = int(lib.sbb_layer_delta_elems(split._handle))
    N = split.in_features
    deltas = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    half = B // 2
    for r in range(2):
        xs, ys = x[r * half:(r + 1) * half].contiguous(), y[r * half:(r + 1) * half].contiguous()
        check(lib.sbb_layer_dp_local(split._handle, xs.data_ptr(), ys.data_ptr(), half, deltas[r].data_ptr(), 0, N, st))
    total = deltas[0] + deltas[1]
    check(lib.sbb_layer_dp_apply_vectors(split._handle, total.data_ptr(), B, st))
    check(lib.sbb_layer_dp_apply_rows(split._handle, total.data_ptr(), B, 0, N, st))
    check(lib.sbb_layer_dp_finish(split._handle, 2, st))
    torch.cuda.synchronize()
    assert np.array_equal(split.wmask, single.wmask)
    for name in ("Ci", "Cj", "Cij", "weights", "bias", "kbi"):
        assert rel_inf(getattr(split, name), getattr(single, name)) < 1e-12, name
    # the pipelined orchestration with a local stand-in for the reduction (world_size 1)
    piped, _ = _layers_from_golden(B200, g, np.float64)

    class Done:
        def wait(self):
            pass

    piped.dp_train_step(x, y, 2, 1, lambda t: Done(), row_blocks=3)
    torch.cuda.synchronize()
    for name in ("Ci", "Cj", "Cij", "weights", "bias", "kbi", "wmask"):
        assert rel_inf(getattr(piped, name), getattr(single, name)) < 1e-12, name


@pytest.mark.parametrize("tag,dtype", DTYPES)
def test_row_sharded_step_on_one_rank_equals_single_step(B200, tag, dtype):
    """The row-sharded step with a world of one rank (it owns every row; the scatter, the partial forward
    product, the activation and the row-block update all run locally) must reproduce forward + fused step."""
    import torch
    g = load_golden("layer_%s.npz" % tag)
    B = int(g["B"])
    x = torch.from_numpy(np.ascontiguousarray(g["x"][:B])).cuda()
    single, _ = _layers_from_golden(B200, g, dtype)
    sharded, _ = _layers_from_golden(B200, g, dtype)
    sharded.shard_rows(0, 1, lambda blob: [blob], B)
    assert sharded.owned_rows() == (0, sharded.in_features)
    tol = TOL[np.dtype(dtype)]
    done = type("Done", (), {"wait": lambda self: None})
    for h in (2, None, 0):
        y = single.compute_activation(x)
        single.train_step(x, y, h)
        ys = sharded.sharded_step(x, h, lambda t: done())
        torch.cuda.synchronize()
        assert rel_inf(ys.cpu().numpy(), y.cpu().numpy() if hasattr(y, "cpu") else y) < tol, h
        assert np.array_equal(sharded.wmask, single.wmask), h
        for name in ("Ci", "Cj", "Cij", "bias", "kbi"):
            assert rel_inf(getattr(sharded, name), getattr(single, name)) < tol, (h, name)
        assert weight_err(sharded.weights, single.weights) < 10 * tol, h
        for name in PLASTIC_STATE:          # both continue from the same state
            setattr(sharded, name, getattr(single, name))
    # the same with every next batch staged ahead on the side stream (three input buffers used in turn)
    xs = [torch.from_numpy(np.ascontiguousarray(g["x"][:B] * s)).cuda() for s in (1.0, 0.5, 0.25, 0.75, 1.0)]
    for k, h in enumerate((1, None, 3, 0)):
        y = single.compute_activation(xs[k])
        single.train_step(xs[k], y, h)
        ys = sharded.sharded_step(xs[k], h, lambda t: done(), next_inputs=xs[k + 1])
        torch.cuda.synchronize()
        assert rel_inf(ys.cpu().numpy(), y.cpu().numpy() if hasattr(y, "cpu") else y) < tol * 10 ** k, k
        assert np.array_equal(sharded.wmask, single.wmask), k
        for name in ("Ci", "Cj", "Cij", "bias", "kbi"):
            assert rel_inf(getattr(sharded, name), getattr(single, name)) < tol * 10 ** k, (k, name)
    with pytest.raises(ValueError):         # the batch staged ahead must be the next one passed
        sharded.sharded_step(xs[0], None, lambda t: done())
    sharded.drop_staged()
    sharded.sharded_step(xs[0], None, lambda t: done())
    with pytest.raises(Exception):          # the plain data-parallel step refuses a sharded layer
        sharded.dp_train_step(x, y, None, 1, lambda t: done())
    big = torch.zeros((B + 1, sharded.in_features), dtype=x.dtype, device="cuda")
    with pytest.raises(Exception):          # more samples than the gathered-input buffers were sized for
        sharded.sharded_step(big, None, lambda t: done())


def test_stl10_shaped_layer_full_size_properties(B200, port_kernels):
    """55296 -> 30x100, batch 256, float32 (663 MB trace matrix).  Checked without a full
    CPU run: (a) the forward pass of a sample of batch rows against the oracle;
    (b) the trace update of a sample of input rows against the oracle (row i of Cij
    depends only on column i of x); (c) identities that hold for every row --
    sum_j Cij[i, HC] moves with Ci[i] because each hypercolumn's activations sum to
    one, and complementary input pairs satisfy Cij[2k] + Cij[2k+1] = Cj's update."""
    from streambrain_b200 import synthetic
    p = synthetic.layer_params("stl10_f32")
    hp = p["hidden"]
    N, H, Mc, B = hp["in_features"], hp["hypercolumns"], hp["minicolumns"], p["batch"]
    M = H * Mc
    np.random.seed(0)
    dev = B200.StructuralPlasticityLayer(N, H, Mc, hp["taupdt"], hp["khalf"], hp["pmin"], hp["taubdt"],
                                         hp["density"], 16, hp["initial_counters"], dtype=np.float32)
    x, _ = synthetic.make_inputs(B, p["n_pixels"], 0.0, np.float32)
    W0, b0, mask0 = dev.weights, dev.bias, dev.wmask
    y = dev.compute_activation(x)
    rows = [0, 1, 100, 255]
    s = port_kernels.update_state(np.zeros((len(rows), M), dtype=np.float32), W0, b0, np.ascontiguousarray(x[rows]))
    want = port_kernels.softmax_minicolumns(s, H, Mc)
    # K = 55296 float32 accumulations: the oracle's own rounding (sequential sums) is of the
    # order of 1e-4 here, so both are measured against a float64 evaluation of the same rows.
    s64 = x[rows].astype(np.float64) @ W0.astype(np.float64) + b0.astype(np.float64)
    y64 = oracle.numpy_softmax_minicolumns(s64, H, Mc)
    err_dev, err_ref = rel_inf(y[rows], y64), rel_inf(want, y64)
    assert err_dev < max(2 * err_ref, 1e-5), (err_dev, err_ref)
    assert rel_inf(y[rows], want) < 1e-3
    assert np.allclose(y.reshape(B, H, Mc).sum(axis=2), 1.0, atol=1e-5)

    Ci0, Cj0, Cij0 = dev.Ci, dev.Cj, dev.Cij
    dev.train_step(x, y, 3)
    Ci1, Cj1, Cij1, W1, mask1 = dev.Ci, dev.Cj, dev.Cij, dev.weights, dev.wmask
    pick = np.r_[0:8, 27640:27656, N - 8:N]
    sub = [Ci0[pick].copy(), Cj0.copy(), np.ascontiguousarray(Cij0[pick]), np.ascontiguousarray(x[:, pick]), y]
    taupdt = hp["taupdt"]
    cw = np.zeros((len(pick), M), dtype=np.float32)
    port_kernels.update_weights(sub[0], sub[1], sub[2], sub[3], sub[4], taupdt, cw, taupdt / 2)
    assert rel_inf(Ci1[pick], sub[0]) < 1e-5 and rel_inf(Cj1, sub[1]) < 1e-5
    assert rel_inf(Cij1[pick], sub[2]) < 1e-5
    masked = np.repeat(mask1[pick], Mc, axis=1).astype(bool)
    assert rel_inf(W1[pick], np.where(masked, cw, 0)) < 1e-4
    assert (W1[np.repeat(mask1, Mc, axis=1) == 0] == 0).all()   # silent connections carry no weight
    # (c) identities over ALL rows
    t = np.float64(np.float32(taupdt))
    row_sum = Cij1.astype(np.float64).reshape(N, H, Mc).sum(axis=2)
    expect = (1 - t) * Cij0.astype(np.float64).reshape(N, H, Mc).sum(axis=2) + \
        t * x.astype(np.float64).mean(axis=0)[:, None]
    assert np.abs(row_sum - expect).max() < 1e-5
    pair = Cij1[0::2].astype(np.float64) + Cij1[1::2].astype(np.float64)
    expect = (1 - t) * (Cij0[0::2].astype(np.float64) + Cij0[1::2]) + t * y.astype(np.float64).mean(axis=0)[None, :]
    assert np.abs(pair - expect).max() < 1e-6
    # mask update moved at most 16 connections in hypercolumn 3 and nothing else
    assert np.array_equal(np.delete(mask1, 3, axis=1), np.delete(mask0, 3, axis=1))
    assert mask1[:, 3].sum() == mask0[:, 3].sum() and (mask1[:, 3] != mask0[:, 3]).sum() <= 32


def test_errors_are_reported_not_fatal(B200):
    from streambrain_b200 import _lib
    np.random.seed(0)
    layer = B200.StructuralPlasticityLayer(8, 2, 2, 0.01, -10.0, 0.1, 0.1, 0.5, 16, (1, 0.5, 0.5), dtype=np.float32)
    with pytest.raises(ValueError):
        layer.compute_activation(np.zeros((4, 9), dtype=np.float32))
    with pytest.raises(ValueError):
        layer.weights = np.zeros((3, 3))
    with pytest.raises(_lib.SbbError) as e:
        layer.train_step(np.zeros((4, 8), dtype=np.float32), np.zeros((4, 4), dtype=np.float32), 5)
    assert e.value.code == 1
    rc = _lib.lib.sbb_layer_forward(layer._handle, None, 4, None, None)
    assert rc == 1
    buf = np.zeros(3, dtype=np.float32)
    assert _lib.lib.sbb_layer_get_state(layer._handle, 0, _lib.host_ptr(buf), buf.nbytes) == 1
    dense = B200.DenseLayer(8, 1, 4, 0.01, (0.5, 0.25, 0.125), dtype=np.float32)
    with pytest.raises(AttributeError):
        dense.kbi
    # the layer still works after the rejected calls
    out = layer.compute_activation(np.random.rand(4, 8).astype(np.float32))
    assert np.allclose(out.reshape(4, 2, 2).sum(axis=2), 1.0, atol=1e-6)
    assert _lib.lib.sbb_kernel_launches() > 0


def test_outputs_too_short_for_the_samples_are_refused(B200):
    """The native calls read batch rows of every operand: arrays that hold fewer are refused before anything runs."""
    import torch
    layer = B200.DenseLayer(12, 2, 4, 0.01, (0.1, 0.1, 0.01), np.float32)
    before = layer.Cij
    x, y = torch.rand((6, 12), device="cuda"), torch.rand((6, 8), device="cuda")
    with pytest.raises(ValueError):
        layer.train_step(x, y[:5])
    with pytest.raises(ValueError):
        layer.dp_train_step(x, y[:5], None, 1, lambda t: None)
    xh, yh = x.cpu().numpy(), y.cpu().numpy()
    for bad_x, bad_y in ((xh[:, :11], yh), (xh.ravel(), yh), (xh, yh[:5]), (xh, yh[:, :7])):
        with pytest.raises(ValueError):
            layer.step_host(bad_x, bad_y)
    assert np.array_equal(layer.Cij, before)
    layer.train_step(x, y)
    layer.step_host(xh.reshape(6, 3, 4), yh)   # (any shape that holds the samples)
    assert not np.array_equal(layer.Cij, before)


@pytest.mark.parametrize("tag,dtype", [("f32", np.float32), ("f64", np.float64)])
@pytest.mark.parametrize("kind", ["dense", "plastic"])
@pytest.mark.parametrize("B,N,H,Mc", [(1, 1, 1, 2), (3, 31, 1, 8), (64, 33, 3, 3), (65, 512, 2, 8), (129, 513, 1, 10),
                                      (300, 700, 5, 5), (700, 1040, 4, 8), (2500, 96, 1, 6), (130, 2050, 16, 2)])
def test_layers_of_few_units_vs_oracle(port_kernels, tag, dtype, kind, B, N, H, Mc):
    """At most 32 units: forward pass and train step run as one launch each.  Sizes around the blocks of 32 inputs, the
    stages of 64 and 128 samples, one to eight samples per block, and 8, 16 and 32 units."""
    import oracle
    import streambrain_b200 as B200
    hp = dict(taupdt=0.05, khalf=-100.0, pmin=0.05, taubdt=0.02, density=0.5)
    rs = np.random.RandomState(B + N)
    init = (0.5, 1 / Mc, 0.5 / Mc)
    np.random.seed(0)
    if kind == "dense":
        dev = B200.DenseLayer(N, H, Mc, hp["taupdt"], init, dtype=dtype)
    else:
        dev = B200.StructuralPlasticityLayer(N, H, Mc, hp["taupdt"], hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"],
                                             16, init, dtype=dtype)
    np.random.seed(0)
    ref = oracle.OracleLayer(port_kernels, kind, N, H, Mc, hp["taupdt"], init, dtype,
                             **({} if kind == "dense" else {k: hp[k] for k in ("khalf", "pmin", "taubdt", "density")}))
    tol = TOL[np.dtype(dtype)]
    for step in range(3):
        x = rs.rand(B, N).astype(dtype)
        a_ref, a_dev = ref.compute_activation(x), dev.compute_activation(x)
        assert rel_inf(a_dev, a_ref) < tol, step
        if kind == "dense":
            t = np.eye(H * Mc, dtype=dtype)[rs.randint(0, H * Mc, B)]
            ref.train_step(x, t)
            dev.train_step(x, t)
        else:
            ref.train_step(x, a_ref, None)
            dev.train_step(x, a_ref, None)
        for name in ("Ci", "Cj", "Cij", "bias"):
            assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, (name, step)
        assert weight_err(dev.weights, ref.weights) < 10 * tol, step
        for name in ("weights", "bias", "Ci", "Cj", "Cij"):
            setattr(dev, name, getattr(ref, name))


def _forward_and_launches(port_kernels, dtype, B, N, H, Mc):
    """A dense layer's forward pass within the tolerance of the oracle's in float64; returns the kernels it launched."""
    import streambrain_b200 as B200
    from streambrain_b200._lib import lib
    rs = np.random.RandomState(B + N + Mc)
    init = (0.5, 1 / Mc, 0.5 / Mc)
    dev = B200.DenseLayer(N, H, Mc, 0.1, init, dtype=dtype)
    ref = oracle.OracleLayer(port_kernels, "dense", N, H, Mc, 0.1, init, np.float64)
    weights, bias = (rs.randn(N, H * Mc) / np.sqrt(N)).astype(dtype), (0.1 * rs.randn(H * Mc)).astype(dtype)
    x = rs.rand(B, N).astype(dtype)
    for layer in (dev, ref):
        layer.weights, layer.bias = weights.astype(layer.dtype), bias.astype(layer.dtype)
    launches = lib.sbb_kernel_launches()
    got = dev.compute_activation(x)
    launches = lib.sbb_kernel_launches() - launches
    assert rel_inf(got, ref.compute_activation(x.astype(np.float64))) < TOL[np.dtype(dtype)]
    return launches


@pytest.mark.parametrize("B,N,H,Mc,one_launch", [
    (8, 20000, 1, 10, True), (256, 32768, 1, 7, True), (257, 600, 1, 7, False), (64, 8192, 1, 8, True), (65, 8192, 1, 8, False),
    (128, 8192, 2, 5, True), (129, 8192, 2, 5, False), (131, 5000, 1, 11, True), (132, 5000, 1, 11, False), (8, 9001, 3, 5, True),
    (64, 8192, 7, 2, True), (64, 8193, 7, 2, False), (65, 2016, 1, 13, True), (65, 2017, 1, 13, False), (8, 640, 2, 8, False)])
def test_float64_forward_of_few_units_on_both_sides_of_its_rule(port_kernels, B, N, H, Mc, one_launch):
    """One launch where the kernel for layers of few units is the faster one, a product in tiles and a softmax elsewhere."""
    launches = _forward_and_launches(port_kernels, np.float64, B, N, H, Mc)
    assert (launches == 1) == one_launch, launches


@pytest.mark.parametrize("tag,dtype", DTYPES)
@pytest.mark.parametrize("B,N,H,Mc", [(1, 4096, 1, 10), (18, 4097, 2, 5), (5, 8191, 1, 7), (19, 4100, 1, 3), (18, 2048, 1, 8),
                                      (37, 2049, 3, 3), (18, 1024, 1, 9), (38, 1024, 1, 10), (74, 1027, 5, 2), (74, 9001, 1, 7),
                                      (75, 5000, 1, 9), (18, 1023, 1, 10), (17, 5000, 1, 32), (36, 2050, 2, 16), (40, 1025, 4, 5)])
def test_forward_of_few_units_in_clusters(port_kernels, tag, dtype, B, N, H, Mc):
    """Eight, four or two blocks share the inputs of a sample, whole and ragged parts; one block where samples or inputs are
    one too many or too few."""
    launches = _forward_and_launches(port_kernels, dtype, B, N, H, Mc)
    assert launches == 1 or (tag == "f64" and H * Mc > 11), launches


@pytest.mark.parametrize("B,N,H,Mc,general,tensor", [
    (400, 206, 1, 32, False, False), (297, 512, 2, 12, False, False), (400, 128, 3, 8, False, True), (593, 512, 3, 3, False, False),
    (593, 448, 3, 3, True, True), (400, 512, 1, 12, False, True), (200, 300, 1, 31, True, True), (201, 300, 1, 31, False, False),
    (201, 300, 4, 7, False, True), (1024, 64, 1, 32, True, True), (1023, 64, 8, 4, False, False), (1023, 64, 7, 4, False, True),
    (2000, 300, 4, 2, True, True), (80, 1535, 3, 7, True, True), (80, 1792, 3, 7, False, False)])
def test_float32_steps_of_few_units_on_both_sides_of_their_rule(port_kernels, contraction_path, B, N, H, Mc, general, tensor):
    """A float32 layer that learns from its own activations: two launches a step where the kernels for layers of few units
    are the faster ones, which depends on what the other way is; the same step either way."""
    import streambrain_b200 as B200
    from streambrain_b200._lib import lib
    hp = dict(khalf=-100.0, pmin=0.05, taubdt=0.02, density=0.5)
    init = (0.5, 1 / Mc, 0.5 / Mc)
    np.random.seed(5)
    dev = B200.StructuralPlasticityLayer(N, H, Mc, 0.02, hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"], 16, init, dtype=np.float32)
    ref = oracle.OracleLayer(port_kernels, "plastic", N, H, Mc, 0.02, init, np.float32, **hp)
    ref.wmask = dev.wmask
    rs = np.random.RandomState(B + N)
    dev.weights = (0.05 * rs.randn(N, H * Mc)).astype(np.float32)
    for name in ("weights", "bias"):
        setattr(ref, name, getattr(dev, name))
    x = rs.rand(B, N).astype(np.float32)
    tol = TOL[np.dtype(np.float32)]
    launches = lib.sbb_kernel_launches()
    y = dev.compute_activation(x)
    dev.train_step(x, y, None)
    launches = lib.sbb_kernel_launches() - launches
    assert (launches == 2) == (tensor if contraction_path == "tensor" else general), launches
    assert rel_inf(y, ref.compute_activation(x)) < 10 * tol
    ref.train_step(x, y, None)
    for name in ("Ci", "Cj", "Cij", "bias"):
        assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, name
    assert weight_err(dev.weights, ref.weights) < 10 * tol


@pytest.mark.parametrize("B,N,H,Mc,scale", [(1, 128, 3, 12, 1.0), (16, 256, 2, 128, 1.0), (255, 260, 4, 65, 1.0),
                                            (256, 516, 33, 8, 1.0), (257, 252, 7, 36, 1e-5), (300, 600, 1, 260, 300.0),
                                            (2049, 132, 3, 88, 1.0), (40, 140, 80, 4, 1.0), (530, 257, 3, 40, 1.0)])
def test_tensor_core_train_step_vs_oracle(port_kernels, B, N, H, Mc, scale):
    """The float32 train step: one and several accumulation chains, ragged row and column tiles, operands with and without
    one-box loads, hypercolumns wider and narrower than a 32-column group and more of them than a mask word holds, inputs
    far from one, and a shape that takes the general kernels."""
    import streambrain_b200 as B200
    hp = dict(taupdt=0.1, khalf=-100.0, pmin=0.05, taubdt=0.02, density=0.5)
    rs = np.random.RandomState(B + N)
    init = (0.5 * scale, 1 / Mc, 0.5 * scale / Mc)
    np.random.seed(0)
    dev = B200.StructuralPlasticityLayer(N, H, Mc, hp["taupdt"], hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"], 16, init,
                                         dtype=np.float32)
    np.random.seed(0)
    ref = oracle.OracleLayer(port_kernels, "plastic", N, H, Mc, hp["taupdt"], init, np.float32, **{
        k: hp[k] for k in ("khalf", "pmin", "taubdt", "density")})
    tol = TOL[np.dtype(np.float32)]
    for step in range(2):
        x = (scale * rs.rand(B, N) * (rs.rand(B, N) > 0.3)).astype(np.float32)
        y = rs.dirichlet(np.ones(Mc), size=(B, H)).reshape(B, H * Mc).astype(np.float32)
        ref.train_step(x, y, None)
        dev.train_step(x, y, None)
        for name in ("Ci", "Cj", "Cij", "bias", "kbi"):
            assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, (name, step)
        assert weight_err(dev.weights, ref.weights) < 10 * tol, step
        off = np.repeat(ref.wmask == 0, Mc, axis=1)
        assert not dev.weights[off].any()
        for name in ("weights", "bias", "Ci", "Cj", "Cij", "kbi"):
            setattr(dev, name, getattr(ref, name))


@pytest.mark.parametrize("n,m", [(64, 256), (5461, 3), (8193, 8), (65537, 4), (2048, 1024), (1399, 1499)])
def test_state_round_trip_through_the_copy_slots(n, m):
    """Host arrays of 64 kB up to several pinned slots, whole and ragged, from two threads at once."""
    import threading
    import streambrain_b200 as B200
    np.random.seed(1)
    layers = [B200.DenseLayer(n, 1, m, 0.1, (1, 1, 1), dtype=np.float32) for _ in range(2)]
    values = [np.random.rand(n, m).astype(np.float32) for _ in range(2)]
    bad = []

    def turn(layer, value):
        for _ in range(3):
            layer.weights = value
            if not np.array_equal(layer.weights, value):
                bad.append(value.shape)
    threads = [threading.Thread(target=turn, args=a) for a in zip(layers, values)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("tag,dtype", DTYPES)
@pytest.mark.parametrize("B", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("N,H,Mc", [(1, 1, 33), (17, 3, 37), (1568, 30, 100), (4096, 2, 256), (4097, 5, 64), (700, 13, 4), (333, 2, 300),
                                    (260, 1, 1024), (9001, 3, 7), (3000, 150, 4), (300, 75, 251)])
def test_forward_of_few_samples_vs_oracle(port_kernels, tag, dtype, B, N, H, Mc):
    """One to four samples take a kernel of their own: vector and scalar columns, one and many hypercolumns per block, wide
    hypercolumns, inputs that do and do not divide into ranges, ranges whose weights stream, and the first sizes that do not
    take it."""
    import streambrain_b200 as B200
    np.random.seed(2)
    args = (N, H, Mc, 0.01, -100.0, 0.05, 0.02, 0.5, 16, (0.5, 1 / Mc, 0.5 / Mc))
    dev = B200.StructuralPlasticityLayer(*args, dtype=dtype)
    ref = oracle.OracleLayer(port_kernels, "plastic", N, H, Mc, 0.01, (0.5, 1 / Mc, 0.5 / Mc), dtype, khalf=-100.0, pmin=0.05,
                             taubdt=0.02, density=0.5)
    for name in ("weights", "bias"):
        setattr(ref, name, getattr(dev, name))
    x = np.random.rand(B, N).astype(dtype)
    want = ref.compute_activation(x)
    for _ in range(2):
        assert rel_inf(dev.compute_activation(x), want) < TOL[np.dtype(dtype)]


def test_forward_of_few_samples_with_several_fills_of_shared_memory(port_kernels):
    """Ranges of more inputs than the streaming form holds at a time."""
    import streambrain_b200 as B200
    N, H, Mc = 1030, 149, 129
    rs = np.random.RandomState(3)
    dev = B200.DenseLayer(N, H, Mc, 0.01, (0.5, 1 / Mc, 0.5 / Mc), dtype=np.float64)
    x = rs.rand(3, N)
    support = x @ dev.weights + dev.bias
    e = np.exp(support.reshape(3, H, Mc) - support.reshape(3, H, Mc).max(axis=2, keepdims=True))
    want = (e / e.sum(axis=2, keepdims=True)).reshape(3, H * Mc)
    assert rel_inf(dev.compute_activation(x), want) < TOL[np.dtype(np.float64)]


@pytest.mark.parametrize("tag,dtype", DTYPES)
@pytest.mark.parametrize("B,N,H,Mc", [(5, 1, 1, 33), (33, 31, 5, 13), (97, 65, 7, 19), (128, 129, 3, 43), (131, 1601, 8, 63),
                                      (257, 2051, 11, 127), (1025, 517, 27, 39), (64, 1600, 47, 64), (320, 1602, 19, 33)])
def test_contractions_of_odd_rows_vs_oracle(port_kernels, tag, dtype, B, N, H, Mc):
    """Rows of any length: small and large output tiles and their edges, one slab and many, one k-split and several, 8-byte
    and 16-byte copies of float64, one deep block per SM and several."""
    import streambrain_b200 as B200
    init = (0.5, 1 / Mc, 0.5 / Mc)
    np.random.seed(4)
    dev = B200.StructuralPlasticityLayer(N, H, Mc, 0.1, -100.0, 0.05, 0.02, 0.5, 16, init, dtype=dtype)
    ref = oracle.OracleLayer(port_kernels, "plastic", N, H, Mc, 0.1, init, dtype, khalf=-100.0, pmin=0.05, taubdt=0.02, density=0.5)
    rs = np.random.RandomState(B + N)
    dev.weights = (0.05 * rs.randn(N, H * Mc)).astype(dtype)
    for name in ("weights", "bias", "wmask"):
        setattr(ref, name, getattr(dev, name))
    x = rs.rand(B, N).astype(dtype)
    tol = TOL[np.dtype(dtype)]
    assert rel_inf(dev.compute_activation(x), ref.compute_activation(x)) < 10 * tol
    y = rs.dirichlet(np.ones(Mc), size=(B, H)).reshape(B, H * Mc).astype(dtype)
    ref.train_step(x, y, None)
    dev.train_step(x, y, None)
    for name in ("Ci", "Cj", "Cij", "bias"):
        assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, name
    assert weight_err(dev.weights, ref.weights) < 10 * tol


@pytest.mark.parametrize("tag,dtype", DTYPES)
@pytest.mark.parametrize("kind,B,N,H,Mc", [("plastic", 512, 128, 2, 48), ("plastic", 1500, 88, 2, 66), ("plastic", 1030, 207, 5, 9),
                                           ("plastic", 2049, 65, 3, 13), ("plastic", 700, 260, 1, 300), ("plastic", 5000, 129, 40, 1),
                                           ("plastic", 600, 104, 1, 9), ("plastic", 1025, 300, 2, 16), ("dense", 1024, 300, 1, 10),
                                           ("dense", 2050, 1100, 1, 30), ("dense", 513, 2300, 1, 3)])
def test_long_batches_of_few_outputs_vs_oracle(port_kernels, tag, dtype, kind, B, N, H, Mc):
    """Batches whose trace step is few tiles are cut into parts whose sums a second launch adds up; layers of few units share
    a batch over a cluster of two, four or eight blocks: whole and ragged parts, vector and scalar rows, masks with many
    hypercolumns to a row, units on both sides of the limits."""
    import streambrain_b200 as B200
    hp = dict(khalf=-100.0, pmin=0.05, taubdt=0.02, density=0.5)
    init = (0.5, 1 / Mc, 0.5 / Mc)
    np.random.seed(5)
    if kind == "dense":
        dev = B200.DenseLayer(N, H, Mc, 0.1, init, dtype=dtype)
        ref = oracle.OracleLayer(port_kernels, kind, N, H, Mc, 0.1, init, dtype)
    else:
        dev = B200.StructuralPlasticityLayer(N, H, Mc, 0.1, hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"], 16, init, dtype=dtype)
        ref = oracle.OracleLayer(port_kernels, kind, N, H, Mc, 0.1, init, dtype, **hp)
        ref.wmask = dev.wmask
    rs = np.random.RandomState(B + N)
    dev.weights = (0.05 * rs.randn(N, H * Mc)).astype(dtype)
    for name in ("weights", "bias"):
        setattr(ref, name, getattr(dev, name))
    tol = TOL[np.dtype(dtype)]
    for step in range(2):   # the tickets are zero again after a launch
        x = rs.rand(B, N).astype(dtype)
        y = rs.dirichlet(np.ones(Mc), size=(B, H)).reshape(B, H * Mc).astype(dtype)
        assert rel_inf(dev.compute_activation(x), ref.compute_activation(x)) < 10 * tol, step
        for layer in (ref, dev):
            layer.train_step(x, y, *(() if kind == "dense" else (None,)))
        for name in ("Ci", "Cj", "Cij", "bias"):
            assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, (name, step)
        assert weight_err(dev.weights, ref.weights) < 10 * tol, step
        if kind == "plastic":
            assert not dev.weights[np.repeat(ref.wmask == 0, Mc, axis=1)].any()
        for name in ("weights", "bias", "Ci", "Cj", "Cij"):
            setattr(dev, name, getattr(ref, name))


@pytest.mark.parametrize("B", [1, 4, 5, 8, 9, 16, 17])
@pytest.mark.parametrize("N,H,Mc", [(131, 3, 11), (33, 1, 33), (1025, 37, 9), (66, 1, 301), (5003, 5, 31), (7, 90, 33)])
def test_train_steps_of_few_samples_of_odd_rows_vs_oracle(port_kernels, N, H, Mc, B):
    """A float32 train step of up to 16 samples on rows that no 16-byte copy can address: every number of samples a kernel is
    built for, rows and columns that fill their warps and that do not, four to thirty-two rows a warp, inputs that never
    fire (no weights there), masks with one and many hypercolumns to a row."""
    import streambrain_b200 as B200
    hp = dict(khalf=-100.0, pmin=0.05, taubdt=0.02, density=0.5)
    init = (0.5, 1 / Mc, 0.5 / Mc)
    np.random.seed(5)
    dev = B200.StructuralPlasticityLayer(N, H, Mc, 0.1, hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"], 16, init, dtype=np.float32)
    ref = oracle.OracleLayer(port_kernels, "plastic", N, H, Mc, 0.1, init, np.float32, **hp)
    ref.wmask = dev.wmask
    Ci = dev.Ci
    Ci[N // 2:N // 2 + 3] = 1e-12   # below the threshold, and stays there
    dev.Ci = Ci
    for name in ("weights", "bias", "Ci", "Cj", "Cij"):
        setattr(ref, name, getattr(dev, name))
    rs = np.random.RandomState(B + N)
    tol = TOL[np.dtype(np.float32)]
    for step in range(2):
        x = rs.rand(B, N).astype(np.float32)
        x[:, N // 2:N // 2 + 3] = 0
        y = rs.dirichlet(np.ones(Mc), size=(B, H)).reshape(B, H * Mc).astype(np.float32)
        for layer in (ref, dev):
            layer.train_step(x, y, None)
        for name in ("Ci", "Cj", "Cij", "bias"):
            assert rel_inf(getattr(dev, name), getattr(ref, name)) < tol, (name, step)
        assert weight_err(dev.weights, ref.weights) < 10 * tol, step
        assert not dev.weights[np.repeat(ref.wmask == 0, Mc, axis=1)].any()
        assert not dev.weights[N // 2:N // 2 + 3].any()


def _twins(kind, N, H, Mc, dtype):
    """Two layers of the same state, and a long batch's inputs and outputs on the device."""
    import torch
    import streambrain_b200 as B200
    init = (0.5, 1 / Mc, 0.5 / Mc)
    twins = []
    for _ in range(2):
        np.random.seed(5)
        twins.append(B200.DenseLayer(N, H, Mc, 0.1, init, dtype=dtype) if kind == "dense" else
                     B200.StructuralPlasticityLayer(N, H, Mc, 0.1, -100.0, 0.05, 0.02, 0.5, 16, init, dtype=dtype))
    t = torch.float32 if dtype is np.float32 else torch.float64

    def batch(B, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.rand((B, N), generator=g, device="cuda", dtype=t)
        y = torch.softmax(torch.rand((B, H, Mc), generator=g, device="cuda", dtype=t), dim=2).reshape(B, H * Mc)
        return x, y
    return twins, batch


def _assert_same_step(a, b, dtype):
    tol = TOL[np.dtype(dtype)]
    for name in ("Ci", "Cj", "bias"):   # (not of the contraction: the same launch in both)
        assert np.array_equal(getattr(a, name), getattr(b, name)), name
    assert rel_inf(a.Cij, b.Cij) < tol
    assert weight_err(a.weights, b.weights) < 10 * tol


@pytest.mark.parametrize("tag,dtype,B,N,M", [("f32", np.float32, 782, 915, 2782), ("f64", np.float64, 1088, 1752, 1030),
                                             ("f32", np.float32, 8196, 1268, 928)])
def test_long_batch_without_room_for_the_products_of_its_parts(tag, dtype, B, N, M):
    """The parts of a long batch want some 50 MB; on a device with less than that left the step is done in one piece, the
    layer is as it would have been, and the steps after it know nothing of the failed allocation."""
    import torch
    from streambrain_b200._lib import lib
    (roomy, tight), batch = _twins("plastic", N, 1, M, dtype)
    x0, y0 = batch(16, 0)
    x, y = batch(B, 1)
    for layer in (roomy, tight):   # (what the kernels' code takes of the device is there before it is filled)
        layer.train_step(x0, y0, None)
    launches = lib.sbb_kernel_launches()
    roomy.train_step(x, y, None)
    split = lib.sbb_kernel_launches() - launches
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hogs, size = [], torch.cuda.mem_get_info()[0]
    while size >= 16 << 20:
        try:
            hogs.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size //= 2
    try:
        launches = lib.sbb_kernel_launches()
        tight.train_step(x, y, None)
        whole = lib.sbb_kernel_launches() - launches
        torch.cuda.synchronize()
    finally:
        hogs.clear()
        torch.cuda.empty_cache()
    assert whole == 2 and split >= whole   # (vectors, and the trace update in one launch)
    _assert_same_step(tight, roomy, dtype)
    for layer in (roomy, tight):
        layer.train_step(x, y, None)
    torch.cuda.synchronize()
    _assert_same_step(tight, roomy, dtype)


@pytest.mark.parametrize("tag,dtype", DTYPES)
@pytest.mark.parametrize("kind,B,N,H,Mc", [("plastic", 1500, 88, 2, 66), ("plastic", 2049, 65, 3, 13), ("dense", 1024, 300, 1, 40)])
def test_first_long_batch_of_a_layer_inside_a_capture(tag, dtype, kind, B, N, H, Mc):
    """A captured step may not allocate: without the workspace of a split batch it is recorded in one piece."""
    import torch
    (eager, captured), batch = _twins(kind, N, H, Mc, dtype)
    x, y = batch(B, 1)
    step = (lambda layer: layer.train_step(x, y)) if kind == "dense" else (lambda layer: layer.train_step(x, y, None))
    before = captured.Cij
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step(captured)
    assert np.array_equal(captured.Cij, before)
    for _ in range(2):
        step(eager)
        graph.replay()
        torch.cuda.synchronize()
        _assert_same_step(captured, eager, dtype)
    del graph


@pytest.mark.parametrize("tag,dtype", DTYPES)
def test_an_allocation_that_fails_is_reported_once(B200, tag, dtype):
    """A layer larger than any device is refused; the next call on another layer does not fail for it half way."""
    from streambrain_b200 import _lib
    np.random.seed(0)
    layer = B200.DenseLayer(60, 1, 40, 0.1, (0.5, 0.025, 0.0125), dtype=dtype)
    x, y = np.random.rand(7, 60).astype(dtype), np.eye(40, dtype=dtype)[:7]
    desc = _lib.LayerDesc(_lib.dtype_code(dtype), _lib.DENSE, 1 << 28, 1, 1 << 20, 0.1, 0.0, 0.0, 0.0, 0)
    handle = ctypes.c_void_p()
    assert _lib.lib.sbb_layer_create(ctypes.byref(desc), ctypes.byref(handle)) == 2
    assert b"emory" in _lib.lib.sbb_last_error() and not handle.value
    before = layer.Ci
    layer.train_step(x, y)
    assert not np.array_equal(layer.Ci, before)
    net = B200.Network(dtype)
    net.add_layer(layer)
    assert _lib.lib.sbb_layer_create(ctypes.byref(desc), ctypes.byref(handle)) == 2
    net.fit(x, y, 7, [(0, 1)])
    assert np.isfinite(layer.weights).all()


@pytest.mark.parametrize("tag,dtype", DTYPES)
@pytest.mark.parametrize("kind,B,N,H,Mc", [("plastic", 1500, 88, 2, 66), ("plastic", 2049, 65, 3, 13), ("plastic", 40, 700, 3, 100)])
def test_captured_step_after_a_larger_batch(tag, dtype, kind, B, N, H, Mc):
    """The workspaces that a captured step uses outlive their replacement by larger ones: the graph runs as before after the
    layer has taken a batch of four times the size, and other memory is left alone."""
    import torch
    (eager, captured), batch = _twins(kind, N, H, Mc, dtype)
    x, y = batch(B, 1)
    large, large_y = batch(4 * B + 1, 2)

    def step(layer):
        a = layer.compute_activation(x)
        layer.train_step(x, y, None)
        return a
    for layer in (eager, captured):
        step(layer)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(captured)
    for layer in (eager, captured):
        layer.compute_activation(large)
        layer.train_step(large, large_y, None)
    torch.cuda.synchronize()
    bystanders = [torch.full((n,), 7, dtype=torch.uint8, device="cuda") for n in (1 << 21, 1 << 22, 1 << 23) for _ in range(4)]
    for _ in range(2):
        want = step(eager)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        _assert_same_step(captured, eager, dtype)
        assert np.array_equal(captured.Cij, eager.Cij)
    assert all(bool((b == 7).all()) for b in bystanders)
    del graph
