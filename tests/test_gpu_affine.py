"""adain_affine's one pass over the chunk statistics: rows where a pass relative to the first mean could go wrong."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _two_pass(stats, gb, l):
    """Mean and variance in float64, two passes (numpy's own NaN and infinity rules)."""
    c, n, _ = stats.shape
    st = stats.astype(np.float64)
    cols = np.full(n, 128.0)
    cols[-1] = l - (n - 1) * 128
    with np.errstate(invalid="ignore", over="ignore"):
        mean = (st[..., 0] * cols).sum(1) / l
        var = (st[..., 1] + cols * (st[..., 0] - mean[:, None]) ** 2).sum(1) / l
        return np.stack([mean, (1 + gb[:c].astype(np.float64)) / np.sqrt(var + 1e-5), gb[c:]])


@pytest.mark.parametrize("l", [1, 128, 129, 4097, 131072, 131073, 300001])
def test_one_pass_is_the_two_pass_result(cuda, l):
    from lokinfer_b200 import ops
    c, n = 8, -(-l // 128)
    r = np.random.default_rng(l)
    stats = np.stack([r.standard_normal((c, n)), r.uniform(0, 200, (c, n))], axis=2).astype(np.float32)
    stats[1, :, 0] = 3.0                       # constant means
    stats[2, :, :] = (1e4, 0.0)                # a constant row far from 0
    stats[3, 0, 0], stats[3, 1:, 0] = 1e5, 0   # the first mean far from the others
    stats[4, n // 2, 0] = np.inf
    stats[5, 0, 0] = np.inf
    stats[6, 0, 0] = np.nan
    stats[7, :, 1] = 0
    gb = r.standard_normal(2 * c).astype(np.float32)
    got = ops.adain_affine_f32_cuda(torch.from_numpy(stats).to(cuda), torch.from_numpy(gb).to(cuda), l).cpu().numpy()
    # float32 results of float64 sums whose error is n * 2^-53 of the mean square: half a unit, and the square root's and divide's
    np.testing.assert_allclose(got, _two_pass(stats, gb, l), rtol=4e-7, atol=1e-7)
