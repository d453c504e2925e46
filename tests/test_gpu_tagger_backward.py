"""The tagger's backward kernel (GPU) at the edges of its rounds: a gradient over n samples is
the sum of those over two parts of them, and the float64 oracle's up to bfloat16 ties."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _magnitudes(params, X, y, pos_weight):
    """Sums over the samples of the gradient terms' magnitudes (parameter layout)."""
    from oracle import mlp

    w = mlp.unpack(params)
    z, c = mlp.forward(params, X)
    d3 = np.abs(np.where(y > 0.5, pos_weight, 1.0) * (1.0 / (1.0 + np.exp(-z)) - y))
    d2 = np.where(c["z2"] > 0.0, d3[:, None] * np.abs(c["round"](w["W3"]))[None, :], 0.0)
    d1 = d2 @ np.abs(c["round"](w["W2"]))
    out = np.zeros(mlp.PARAMS)
    out[mlp.SLICES["W1"]] = (d1.T @ np.abs(c["x"])).ravel()
    out[mlp.SLICES["b1"]] = d1.sum(axis=0)
    out[mlp.SLICES["W2"]] = (d2.T @ c["h1"]).ravel()
    out[mlp.SLICES["b2"]] = d2.sum(axis=0)
    out[mlp.SLICES["W3"]] = d3 @ c["h2"]
    out[mlp.SLICES["b3"]] = d3.sum()
    return out


# 64 samples a round, 148 blocks: one sample, a part of a round, one more than a round, one
# more than a round of every block, several rounds a block
@pytest.mark.parametrize("n", [1, 63, 64, 65, 148 * 64 + 1, 30000])
def test_gradients_add_up_and_match_the_oracle(n):
    from oracle import mlp
    from wellbalanced_b200.tagger import LearnedTagger

    rng = np.random.default_rng(n)
    tagger = LearnedTagger(seed=4)
    X = rng.standard_normal((n, 16)).astype(np.float32)
    y = (rng.uniform(size=n) < 0.2).astype(np.float32)
    Xd, yd = torch.from_numpy(X).cuda(), torch.from_numpy(y).cuda()
    loss, grad = tagger.gradient(Xd, yd, pos_weight=5.0)
    params = tagger.params.cpu().numpy()
    got = grad.cpu().numpy().astype(np.float64)
    # float32 sums of at most 64 + rounds + blocks additions in a row
    size = _magnitudes(params, X, y, 5.0)
    rounding = (64 + n // (148 * 64) + 148 + 32) * 2.0**-24 * size
    if n > 1:
        k = n // 3 + 1
        parts = [tagger.gradient(Xd[s], yd[s], pos_weight=5.0) for s in (slice(0, k), slice(k, n))]
        both = sum(g.cpu().numpy().astype(np.float64) for _, g in parts)
        assert np.all(np.abs(got - both) <= 2.0 * rounding)
        assert abs(loss - sum(part for part, _ in parts)) <= 1e-12 * max(loss, 1.0)
    want_loss, want = mlp.loss_and_gradients(params, X, y, 5.0)
    # a hidden value next to a bfloat16 tie may round the other way: half a unit in 2^-8
    assert np.all(np.abs(got - want) <= rounding + 2.0**-8 * size)
    assert abs(loss - want_loss) <= 2.0**-8 * want_loss
    # gradients added to what is there, at any alignment
    flat = torch.ones(mlp.PARAMS + 1, device="cuda")
    total = torch.zeros(1, dtype=torch.float64, device="cuda")
    from wellbalanced_b200 import _lib

    _lib.call("wb_mlp_backward", Xd.data_ptr(), yd.data_ptr(), n, tagger.params.data_ptr(), 5.0, flat.data_ptr() + 4,
              total.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert float(flat[0]) == 1.0
    assert np.all(np.abs(flat[1:].cpu().numpy() - 1.0 - got) <= 2.0 * rounding + 150 * 2.0**-24 * (1.0 + size))
