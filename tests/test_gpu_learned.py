"""The learned PPE warm start and preconditioner scale on the GPU.

* the FP32 training kernels' loss and gradient equal the numpy FP64 oracle's;
* tensor-core inference (BF16 operands, FP32 accumulation) equals the oracle run with
  the same BF16 roundings;
* training on samples the FP64 CG generates lowers the loss;
* the learned solve reaches the requested residual (the FP64 true residual judges it)
  without the FP64 fallback, matches the plain solution, and its iteration count is
  compared with the same solve driven by a zero network.
"""
import numpy as np
import pytest

from helpers import rel_err
from oracle import mlp
from openmps_gb300 import _abi as abi
from openmps_gb300 import learned, scenes
from openmps_gb300.computer import Computer, mlp_infer, mlp_loss_grad, mlp_train

pytestmark = pytest.mark.gpu


def _random_case(seed, n):
    rng = np.random.default_rng(seed)
    mu = rng.standard_normal(16) * 0.2
    sd = 0.5 + rng.random(16)
    blob = mlp.init_blob(mu, sd, seed=seed)
    samples = np.concatenate([mu + sd * rng.standard_normal((n, 16)), rng.standard_normal((n, 2))], axis=1)
    return blob, samples.astype(np.float32)


@pytest.mark.parametrize("n", [1, 63, 64, 1000, 5003])
def test_gradient_matches_oracle(gpu_lib, n):
    blob, samples = _random_case(11 + n, n)
    loss, grad = mlp_loss_grad(blob, samples)
    loss_o, grad_o = mlp.loss_grad(blob.astype(np.float64), samples.astype(np.float64))
    assert abs(loss - loss_o) <= 1e-5 * abs(loss_o)
    assert np.all(grad[:32] == 0.0)
    err = np.linalg.norm(grad - grad_o) / np.linalg.norm(grad_o)
    assert err < 1e-4, err


@pytest.mark.parametrize("n", [4096, 8192, 16384, 32768])
def test_gradient_of_large_batches_sums_148_parts(gpu_lib, n):
    # A batch's gradient is its tiles' (64 samples) in at most 148 FP32 sums of tiles 148
    # apart, then FP64 over those (each eighth one in one of eight sums, even and odd ones
    # apart): composed here from the gradients of the tiles by themselves.  n / 64 is a power
    # of two, so 1 / 64 against 1 / n scales every term exactly, and the bits are the same.
    blob, samples = _random_case(3, n)
    _, got = mlp_loss_grad(blob, samples)
    tiles = [mlp_loss_grad(blob, samples[k:k + 64])[1] for k in range(0, n, 64)]
    parts = []
    for p in range(min(148, len(tiles))):
        g = np.zeros_like(got)
        for k in range(p, len(tiles), 148):
            g = g + tiles[k]
        parts.append(g.astype(np.float64))
    zero = np.zeros(got.size)
    warps = [sum(parts[w::16], zero) + sum(parts[w + 8::16], zero) for w in range(8)]
    total = ((warps[0] + warps[1]) + (warps[2] + warps[3])) + ((warps[4] + warps[5]) + (warps[6] + warps[7]))
    np.testing.assert_array_equal(got, (total * (64.0 / n)).astype(np.float32))


@pytest.mark.parametrize("n,batch", [(1, 4), (31, 31), (33, 64), (64, 64), (130, 64), (5000, 4900)])
def test_training_steps_match_oracle(gpu_lib, n, batch):
    # Three epochs of the same minibatches in FP64 (the shuffle by SplitMix64 and Fisher-Yates).
    # An entry moves by about lr a step whatever its gradient's size, so one whose gradient is
    # at the FP32 sums' rounding (1e-6 of the largest) may move the other way: a few in a
    # thousand of them, hence the bound of 2 % of the movement in the 2-norm.
    blob, samples = _random_case(5 + n, n)
    lr, epochs, seed = 1e-3, 3, 9
    got, losses = mlp_train(blob, samples, epochs=epochs, batch=batch, lr=lr, seed=seed)
    w = blob.astype(np.float64)
    m, v = np.zeros_like(w), np.zeros_like(w)
    mask = (1 << 64) - 1
    state, step, expect = seed, 0, []
    for _ in range(epochs):
        perm = list(range(n))
        for i in range(n - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        total = 0.0
        for at in range(0, n, batch):
            part = samples[perm[at:at + batch]].astype(np.float64)
            loss, grad = mlp.loss_grad(w, part)
            total += loss * len(part)
            step += 1
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad * grad
            w = w - lr * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        expect.append(total / n)
    assert np.array_equal(got[:32], blob[:32])
    moved = lr * step * np.sqrt(w.size)
    assert np.linalg.norm(got - w) <= 0.02 * moved
    np.testing.assert_allclose(losses, expect, rtol=1e-3)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 20000])
def test_tensor_core_inference_matches_oracle(gpu_lib, n):
    blob, samples = _random_case(7 + n, n)
    feats = samples[:, :16]
    out = mlp_infer(blob, feats)
    ref = mlp.forward(blob, feats.astype(np.float64), bf16_path=True)
    scale = max(np.max(np.abs(ref)), 1e-3)
    # same BF16 roundings, FP32 accumulation in a different order: rare one-ulp flips of
    # a BF16 activation bound the difference
    assert np.max(np.abs(out - ref)) <= 2e-2 * scale, np.max(np.abs(out - ref))
    assert np.mean(np.abs(out - ref)) <= 1e-3 * scale
    full = mlp.forward(blob, feats.astype(np.float64))
    assert np.max(np.abs(out - full)) <= 5e-2 * max(np.max(np.abs(full)), 1e-3)


def test_training_lowers_loss(gpu_lib):
    rng = np.random.default_rng(1)
    x = rng.standard_normal((6000, 16)).astype(np.float32)
    y = np.tanh(x[:, 0] - 0.5 * x[:, 3]) + 0.1 * x[:, 7]
    g = y / (1.0 + 0.2 * np.tanh(x[:, 5]))  # reachable: s = 1 + 0.2 tanh(x5)
    samples = np.concatenate([x, y[:, None], g[:, None]], axis=1).astype(np.float32)
    blob = learned.init_weights(samples, seed=2)
    l0, _ = mlp_loss_grad(blob, samples)
    trained, losses = mlp_train(blob, samples, epochs=15, batch=512, lr=3e-3, seed=4)
    l1, _ = mlp_loss_grad(trained, samples)
    assert losses[-1] < losses[0]
    assert l1 < 0.3 * l0, (l0, l1)
    # deterministic: same seed, same weights
    again, _ = mlp_train(blob, samples, epochs=15, batch=512, lr=3e-3, seed=4)
    np.testing.assert_array_equal(trained, again)


@pytest.fixture(scope="module")
def small_weights(gpu_lib):
    data = learned.collect(n_scenes=6, target=30000, steps=24, every=4, seed=77)
    assert data.shape[0] > 10000 and np.all(np.isfinite(data))
    blob, losses = learned.train(data, epochs=12, batch=2048, lr=2e-3, seed=5)
    assert losses[-1] < losses[0]
    return blob


def _dam(seed_k):
    s = learned.training_scene(seed_k, seed=991)
    return s


def zero_network():
    """The network with zero output: s = 1 and the warm start one preconditioned step."""
    blob = np.zeros(abi.MLP_BLOB_FLOATS, dtype=np.float32)
    blob[16:32] = 1.0
    return blob


def _run(s, solver, blob=None, steps=12):
    c = Computer(s.params(solver=solver, criterion=abi.CRIT_RHS, eps=1e-8))
    if blob is not None:
        c.learned_set_weights(blob)
    c.add_scene(s)
    its = []
    for _ in range(steps):
        c.forward_time(s.meta["dt"])
        st = c.stats()
        assert st["cg_true_relres"] <= 1e-8
        assert st["fallback"] == 0
        its.append(st["cg_iterations"])
    return c.particles(), np.array(its)


def test_learned_solve_matches_plain_cg(small_weights):
    s = _dam(3)
    P64, it64 = _run(s, abi.SOLVER_CG64)
    Pmg, itmg = _run(s, abi.SOLVER_MIXED_MG)
    Pl, itl = _run(s, abi.SOLVER_LEARNED, small_weights)
    Pz, itz = _run(s, abi.SOLVER_LEARNED, zero_network())
    for P in (Pmg, Pl, Pz):
        assert rel_err(P["p"], P64["p"]) < 1e-5
        assert rel_err(P["x"], P64["x"], scale=s.l0) < 1e-6
    # what the trained network gains over the same solve without it (zero network)
    print("iterations over %d steps: CG64 %d, MIXED_MG %d, zero network %d, trained network %d"
          % (len(it64), it64.sum(), itmg.sum(), itz.sum(), itl.sum()))
    assert itz.sum() <= itmg.sum()
    assert itl.sum() <= 1.05 * itz.sum()
    assert itl.sum() * 2 < it64.sum()


def test_learned_requires_weights(gpu_lib):
    s = _dam(0)
    c = Computer(s.params(solver=abi.SOLVER_LEARNED, criterion=abi.CRIT_RHS, eps=1e-8))
    c.add_scene(s)
    with pytest.raises(Exception) as e:
        c.forward_time(s.meta["dt"])
    assert getattr(e.value, "code", None) == abi.MPS_ERR_STATE


def test_collected_samples_are_consistent(gpu_lib):
    # y is the error the coarse correction misses, in units of sigma: solving from
    # x0 + c + sigma y gives the solution, so the samples are exact on the solved step
    s = _dam(1)
    c = Computer(s.params(solver=abi.SOLVER_CG64, criterion=abi.CRIT_RHS, eps=1e-12))
    c.add_scene(s)
    for _ in range(3):
        c.forward_time(s.meta["dt"])
    c.learned_collect(True)
    c.forward_time(s.meta["dt"])
    smp, act = c.learned_samples()
    assert act.sum() > 0.5 * s.count
    a = smp[act != 0]
    assert np.all(np.isfinite(a))
    # the Jacobi feature (8, in units of sigma) has unit RMS over the active rows
    assert abs(np.sqrt(np.mean(a[:, 8].astype(np.float64) ** 2)) - 1.0) < 1e-3
    np.testing.assert_allclose(a[:, 17], a[:, 8], rtol=1e-6, atol=1e-7)
