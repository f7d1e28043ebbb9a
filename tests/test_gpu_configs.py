"""Parity at the shapes of the benchmark configurations that the small fuzz cases do not reach:

* the wide hidden layer (1568 -> 100 x 300, batch 1024, float32): three teacher-forced steps, two of
  them with a mask update, against the CPU oracle at the full shape.  Mc = 300 puts hypercolumn
  boundaries inside most column tiles of the tensor-core trace update and takes the softmax through
  its widest register cache;
* the STL-10-shaped layer (55296 -> 30 x 100, batch 256) started from traces with finite plasticity
  scores: the full-size mask update against the oracle's, float32 (tie-aware) and float64 (identical);
* classifier argmax predictions on 10 000 held-out synthetic samples, float32 and float64.
"""
import numpy as np
import pytest

from conftest import TOL, mask_mismatch_is_a_tie, rel_inf, weight_err

import oracle

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("contraction_path")]

PLASTIC_STATE = ("weights", "bias", "Ci", "Cj", "Cij", "kbi", "wmask")


@pytest.fixture(scope="module")
def B200():
    import streambrain_b200
    return streambrain_b200


def _plastic_pair(B200, kernels, hp, dtype, seed=0, with_oracle=True):
    np.random.seed(seed)
    dev = B200.StructuralPlasticityLayer(hp["in_features"], hp["hypercolumns"], hp["minicolumns"], hp["taupdt"],
                                         hp["khalf"], hp["pmin"], hp["taubdt"], hp["density"], 16,
                                         hp["initial_counters"], dtype=dtype)
    if not with_oracle:
        return dev, None
    np.random.seed(seed)
    ref = oracle.OracleLayer(kernels, "plastic", hp["in_features"], hp["hypercolumns"], hp["minicolumns"],
                             hp["taupdt"], hp["initial_counters"], dtype, khalf=hp["khalf"], pmin=hp["pmin"],
                             taubdt=hp["taubdt"], density=hp["density"])
    return dev, ref


@pytest.fixture(scope="module")
def wide_oracle_run(port_kernels):
    """The oracle's trajectory at the wide configuration, computed once for both contraction paths:
    per step the state before, the batch, the activation, the hypercolumn and the state after."""
    from streambrain_b200 import synthetic
    p = synthetic.layer_params("wide_f32")
    hp = p["hidden"]
    np.random.seed(0)
    ref = oracle.OracleLayer(port_kernels, "plastic", hp["in_features"], hp["hypercolumns"], hp["minicolumns"],
                             hp["taupdt"], hp["initial_counters"], np.float32, khalf=hp["khalf"], pmin=hp["pmin"],
                             taubdt=hp["taubdt"], density=hp["density"])
    B = p["batch"]
    x, _ = synthetic.make_inputs(3 * B, p["n_pixels"], p["sparsity"], np.float32)
    ref.Ci, ref.Cj, ref.Cij = synthetic.steady_state_traces(p, x[:B])
    steps = []
    for s, h in enumerate((None, hp["hypercolumns"] - 1, 37)):
        xb = np.ascontiguousarray(x[s * B:(s + 1) * B])
        before = ref.state()
        act = ref.compute_activation(xb)
        ref.train_step(xb, act, h)
        steps.append(dict(before=before, x=xb, act=act, h=h, after=ref.state()))
    return p, steps


def test_wide_layer_teacher_forced_vs_oracle_at_shape(B200, wide_oracle_run):
    p, steps = wide_oracle_run
    hp = p["hidden"]
    Mc = hp["minicolumns"]
    tol = TOL[np.dtype(np.float32)]
    dev, _ = _plastic_pair(B200, None, hp, np.float32, with_oracle=False)
    for s, rec in enumerate(steps):
        for name in PLASTIC_STATE:
            setattr(dev, name, rec["before"][name])
        act = dev.compute_activation(rec["x"])
        assert rel_inf(act, rec["act"]) < tol, s
        assert np.allclose(act.reshape(-1, hp["hypercolumns"], Mc).sum(axis=2), 1.0, atol=1e-5)
        dev.train_step(rec["x"], rec["act"], rec["h"])
        after = rec["after"]
        for name in ("Ci", "Cj", "Cij", "kbi", "bias"):
            assert rel_inf(getattr(dev, name), after[name]) < tol, (s, name)
        got = dev.wmask
        h = rec["h"]
        if h is None:
            assert np.array_equal(got, after["wmask"]), s
        else:
            assert mask_mismatch_is_a_tie(got, after["wmask"], h, rec["before"]["wmask"], after, hp["taupdt"] / 2,
                                          Mc, 1e-5), s
            assert (got[:, h] != rec["before"]["wmask"][:, h]).sum() > 0, "the mask step moved nothing"
        if np.array_equal(got, after["wmask"]):
            W = dev.weights
            assert weight_err(W, after["weights"]) < 10 * tol, s
            assert np.array_equal(W == 0, after["weights"] == 0), s


def _oracle_mask_update(port_kernels, dev, hp, h, mask_before):
    """The oracle's mask update for hypercolumn h from the device layer's own post-update traces.  The
    oracle reads only hypercolumn h's columns of the weights (the freshly recomputed, un-masked ones), so
    only those columns of a zero matrix are filled, by the oracle's own weight recompute."""
    N, H, Mc = hp["in_features"], hp["hypercolumns"], hp["minicolumns"]
    Ci, Cj, Cij = dev.Ci, dev.Cj, dev.Cij
    cthr = hp["taupdt"] / 2
    cols = slice(h * Mc, (h + 1) * Mc)
    w_h = port_kernels.recompute_weights(np.zeros((N, Mc), dtype=Cij.dtype), Ci, np.ascontiguousarray(Cj[cols]),
                                         np.ascontiguousarray(Cij[:, cols]), cthr)
    W = np.zeros((N, H * Mc), dtype=Cij.dtype)
    W[:, cols] = w_h
    want = port_kernels.update_mask(mask_before.copy(), W, Ci, Cj, Cij, cthr, H, Mc, h, 16)
    return want, {"Ci": Ci, "Cj": Cj, "Cij": Cij}


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_stl10_full_size_mask_update_vs_oracle(B200, port_kernels, contraction_path, dtype):
    """55296 input rows: the lists from some 860 blocks of 64 rows, from finite scores (the start state
    of the benchmark), must pick the connections the oracle picks from the same traces."""
    from streambrain_b200 import synthetic
    if dtype == np.float64 and contraction_path == "tensor":
        pytest.skip("float64 always takes the general-shape kernels: covered by the other parametrisation")
    p = synthetic.layer_params("stl10_f32")
    hp = p["hidden"]
    N, H, Mc, B = hp["in_features"], hp["hypercolumns"], hp["minicolumns"], p["batch"]
    dev, _ = _plastic_pair(B200, None, hp, dtype, with_oracle=False)
    x, _ = synthetic.make_inputs(B, p["n_pixels"], 0.0, dtype)
    Ci, Cj, Cij = synthetic.steady_state_traces(dict(p, dtype=np.dtype(dtype)), x)
    dev.Ci, dev.Cj, dev.Cij = Ci, Cj, Cij
    del Cij
    y = dev.compute_activation(x)
    for h in (3, H - 1):
        before = dev.wmask
        dev.train_step(x, y, h)
        got = dev.wmask
        want, ref_state = _oracle_mask_update(port_kernels, dev, hp, h, before)
        moved = int((want[:, h] != before[:, h]).sum())
        assert moved > 0, "the oracle moved no connection: the start state does not exercise the search"
        if dtype == np.float64:
            assert np.array_equal(got, want), (h, int((got != want).sum()))
        else:
            assert mask_mismatch_is_a_tie(got, want, h, before, ref_state, hp["taupdt"] / 2, Mc, 1e-5), \
                (h, int((got != want).sum()), moved)
        # the weights of hypercolumn h follow the NEW mask: silent connections carry none
        W = dev.weights
        assert (W[:, h * Mc:(h + 1) * Mc][got[:, h] == 0] == 0).all()
        del W, ref_state


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_argmax_predictions_on_10000_held_out_samples(B200, port_kernels, dtype):
    """Hidden layer and classifier hold the oracle's state (teacher-forced training); the class predicted
    for each of 10 000 held-out samples must be the oracle's.  In float32 a prediction may differ only
    where the oracle's own two best classes lie closer than the float32 rounding of the support."""
    from streambrain_b200 import synthetic
    p = synthetic.layer_params("mnist_f32" if dtype == np.float32 else "mnist_f64")
    hp, op, B = p["hidden"], p["out"], p["batch"]
    dev, ref = _plastic_pair(B200, port_kernels, hp, dtype)
    np.random.seed(1)
    dev_out = B200.DenseLayer(op["in_features"], 1, 10, op["taupdt"], op["initial_counters"], dtype=dtype)
    np.random.seed(1)
    ref_out = oracle.OracleLayer(port_kernels, "dense", op["in_features"], 1, 10, op["taupdt"],
                                 op["initial_counters"], dtype)
    x, lab = synthetic.make_inputs(8 * B, p["n_pixels"], p["sparsity"], dtype)
    for s in range(8):
        xb, lb = x[s * B:(s + 1) * B], lab[s * B:(s + 1) * B]
        a = ref.compute_activation(xb)
        ref.train_step(xb, a, None)
        ref_out.train_step(a, lb)
    ref_out.train_finalize()
    for name in PLASTIC_STATE:
        setattr(dev, name, getattr(ref, name))
    for name in ("weights", "bias", "Ci", "Cj", "Cij"):
        setattr(dev_out, name, getattr(ref_out, name))
    xt, _ = synthetic.make_inputs(10000, p["n_pixels"], p["sparsity"], dtype, seed=synthetic.DATA_SEED + 99)
    hidden_ref = ref.compute_activation(xt)
    out_ref = ref_out.compute_activation(hidden_ref)
    out_dev = dev_out.compute_activation(dev.compute_activation(xt))
    want, got = np.argmax(out_ref, axis=1), np.argmax(out_dev, axis=1)
    if dtype == np.float64:
        assert np.array_equal(got, want)
        return
    wrong = np.flatnonzero(got != want)
    # class probabilities of the oracle's own two best classes at the samples that differ
    top2 = np.sort(out_ref[wrong].astype(np.float64), axis=1)[:, -2:]
    assert ((top2[:, 1] - top2[:, 0]) <= 1e-5 * top2[:, 1]).all(), (len(wrong), top2[:4])
    assert len(wrong) <= 10, len(wrong)
