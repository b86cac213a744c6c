"""The order statistics against numpy: both ranks of a quantile on few, equal,
negative and widely spread values, at the edges of the select's blocks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 3, 20, 21, 1023, 1024, 1025, 200003])
@pytest.mark.parametrize("kind", ["spread", "equal", "two", "negative", "signed", "narrow"])
def test_percentile(gpu, dtype, n, kind):
    from tensorsph_b200.particle_shifting import estimate_reference_concentration
    rng = np.random.default_rng(n)
    x = {"spread": lambda: 10.0 ** rng.uniform(-30, 30, n), "equal": lambda: np.full(n, 0.7),
         "two": lambda: rng.integers(0, 2, n).astype(float), "negative": lambda: -rng.random(n),
         "signed": lambda: rng.normal(size=n), "narrow": lambda: 1.0 + 1e-6 * rng.random(n)}[kind]().astype(dtype)
    for q in (0.0, 50.0, 95.0, 100.0):
        got = estimate_reference_concentration(torch.from_numpy(x).to(gpu), q)
        s = np.sort(x).astype(np.float64)
        pos = q / 100.0 * (n - 1)
        lo, hi = s[int(np.floor(pos))], s[int(np.ceil(pos))]
        w = pos - np.floor(pos)
        want = lo + w * (hi - lo) if w < 0.5 else hi - (hi - lo) * (1.0 - w)
        assert got == pytest.approx(want, rel=1e-15, abs=0.0), (q, got, want)
