"""The network's products at the edges of their tiles: batches and widths of
one tile, odd multiples of 64, and sizes on both sides of the rule that picks
64 x 64 over 32 x 32 tiles (148 CTAs); forward, weight-gradient and
input-gradient products (both operand layouts) through the gradient, rows
around the padding granularity and the 1024-row chunk through predict, and
training across graph and pass boundaries.

Tolerances as in test_mlp.py: 2e-3 relative L2 against the oracle with
bfloat16 rounding at the same points, 1e-4 on the loss."""
from __future__ import annotations

import numpy as np
import pytest

import rfsyn_b200 as rb
from oracle.mlp_oracle import MlpOracle

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


# (batch, n_in, width, depth, n_out): the largest two reach 64 x 64 tiles in
# the forward and input-gradient products, and in the weight gradients
@pytest.mark.parametrize("shape", [(64, 1, 64, 1, 64), (64, 65, 128, 2, 192), (192, 54, 320, 3, 64),
                                   (448, 130, 192, 1, 448), (1024, 54, 640, 1, 128), (64, 54, 832, 2, 832)],
                         ids=lambda s: "x".join(map(str, s)))
def test_gradient_matches_oracle(shape):
    B, n_in, width, depth, n_out = shape
    rng = np.random.default_rng(B + width)
    X, Y = rng.uniform(-1, 1, (B, n_in)), rng.normal(0, 1, (B, n_out))
    net = rb.Mlp(n_in, width, depth, n_out, seed=21)
    orc = MlpOracle(n_in, width, depth, n_out)
    p = net.params().astype(np.float64)
    loss, g = net.grad(X, Y)
    loss_o, g_o = orc.loss_grad(p, X, Y, bf16=True)
    assert abs(loss - loss_o) <= 1e-4 * abs(loss_o)
    o = 0
    for i, n in orc.shapes:
        k = n * i + n
        assert _rel(g[o:o + k].astype(np.float64), g_o[o:o + k]) < 2e-3
        o += k
    net.close()


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 1023, 1025])
def test_predict_rows(rows):
    rng = np.random.default_rng(rows)
    X = rng.uniform(-1, 1, (rows, 54))
    net = rb.Mlp(54, 128, 2, 128, seed=22)
    orc = MlpOracle(54, 128, 2, 128)
    want = orc.predict(net.params().astype(np.float64), X, bf16=True)
    first = net.predict(X)
    assert _rel(first.astype(np.float64), want) < 2e-3
    # rows left over from a larger call change nothing
    net.predict(rng.uniform(-1, 1, (1024, 54)))
    assert np.array_equal(net.predict(X), first)
    net.close()


def test_training_is_one_sequence():
    """7, 8 and 9 steps (one step of the smaller graph, one replay of the
    larger, both) and passes that end inside a graph's reach: the same data,
    seed and schedule give the same weights on a fresh network, on one that
    trained before (kept graphs) and after its data were set again."""
    rng = np.random.default_rng(3)
    X, Y = rng.uniform(-1, 1, (640, 54)), rng.normal(0, 1, (640, 64))
    used = rb.Mlp(54, 64, 2, 64, seed=23)
    p0 = used.params()
    used.set_data(X[:128], Y[:128])
    used.train(11, batch=64, seed=9)
    used.set_data(X, Y)
    for steps in (7, 8, 9, 23):
        fresh = rb.Mlp(54, 64, 2, 64, seed=23)
        fresh.set_data(X, Y)
        want_loss = fresh.train(steps, batch=64, seed=4)
        used.set_params(p0)
        assert used.train(steps, batch=64, seed=4) == want_loss
        assert np.array_equal(used.params(), fresh.params())
        fresh.close()
    used.close()


@pytest.mark.parametrize("gemm", ["mma", "tcgen05"])
def test_launches_of_replayed_steps_count(gemm, monkeypatch):
    """Every call counts the launches of its steps, also where it replays
    graphs that an earlier call captured."""
    monkeypatch.setenv("RFSYN_FDTD_MLP_GEMM", gemm)
    rng = np.random.default_rng(5)
    net = rb.Mlp(64, 128, 2, 128, seed=29)
    net.set_data(rng.uniform(-1, 1, (512, 64)), rng.normal(0, 1, (512, 128)))
    counts = []
    for _ in range(3):
        net.train(9, batch=128, seed=1)
        counts.append((net.lib.fdtd_b200_mlp_launch_count(net.h), net.tensor_core_launches()))
    (l0, t0), (l1, t1), (l2, t2) = counts
    assert l1 - l0 == l2 - l1 > 0 and (l1 - l0) % 9 == 0
    assert t1 - t0 == t2 - t1 == t0 and (t0 > 0) == (gemm == "tcgen05") and t0 % 9 == 0
    net.close()
