"""The one-pass pruner + compressor (vnm_sparsify_magnitude) and the candidate search of the pruner, bit for bit against the
CPU oracle's exhaustive search followed by the mask-based compressor."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (M, K, V, m): one quadruple; padded tiles; m not a multiple of four; m = 8, 16, 32 (compiled sizes); V above 128; the smallest m that scores;
# the last m of the task lists and the first beyond; enough blocks for the small CTAs
SHAPES = [(64, 64, 32, 4), (128, 96, 32, 16), (128, 160, 64, 20), (64, 70, 32, 7), (192, 72, 64, 8), (128, 48, 128, 16), (64, 96, 32, 32), (256, 64, 256, 16),
          (64, 45, 32, 5), (64, 62, 64, 31), (32, 66, 32, 33), (2048, 640, 32, 8)]


def _weights(kind, M, K, V, m, seed):
    rng = np.random.default_rng(seed)
    w = rng.normal(0, 0.02, (M, K)).astype(np.float16)
    if kind == "ties":                 # few distinct magnitudes: candidate lists overflow into the exhaustive search
        w = (np.round(w.astype(np.float32) * 100) / 100).astype(np.float16)
    elif kind == "near":               # many candidates that the integer scores cannot tell apart
        w = (0.02 * (1 + 1e-3 * rng.normal(size=(M, K)))).astype(np.float16)
    elif kind == "zeros":              # blocks that keep nothing, rows with fewer than two entries
        w[:V] = 0
        w[V:, :m] = 0
        w[-1, 1:] = 0
    return w


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["normal", "ties", "near", "zeros"])
@pytest.mark.parametrize("half", [True, False])
def test_sparsify_equals_prune_then_compress(oracle, shape, kind, half):
    import torch
    from venom_b200 import capi
    M, K, V, m = shape
    w = _weights(kind, M, K, V, m, seed=M + K + m)
    omask, ocols = oracle.prune(np.abs(w.astype(np.float32)), V, m)
    wd = torch.from_numpy(w).cuda()
    if not half:
        wd = wd.float()
    values, meta, cols, bad = capi.sparsify_magnitude(wd, V, m)
    mask2, cols2 = capi.prune_magnitude(wd, V, m)
    assert np.array_equal(cols.cpu().numpy().view(np.uint32), ocols) and torch.equal(cols, cols2)
    mask2 = mask2.cpu().numpy()
    # which of two equal entries of a row is kept is the implementation's choice: the same magnitude is kept in every row
    a = np.abs(w.astype(np.float64))
    assert np.array_equal((a * mask2).sum(1), (a * omask).sum(1)) and np.array_equal(mask2.sum(1), omask.sum(1))
    ov, om, obad = oracle.compress((w * mask2).astype(np.float16), ocols, V, m, mask=mask2)
    assert np.array_equal(values.cpu().numpy().reshape(-1), ov.reshape(-1))
    assert np.array_equal(meta.cpu().numpy().view(np.uint32), om)
    assert bad == obad


def test_sparsify_leaves_other_shapes_to_the_two_step_path():
    import torch
    from venom_b200 import capi
    from venom_b200.nmv import MagnitudeSparsifier
    w = torch.randn((128, 200), device="cuda").half()
    assert capi.sparsify_magnitude(w, 32, 100) is None                # m > 64
    t = MagnitudeSparsifier(2, 100, 32)(w)
    assert t.violations == 0 and int((t.to_dense() != 0).sum()) == 128 * 4
