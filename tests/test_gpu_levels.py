"""The extrema reduction on the GPU."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 5, 31, 511, 8191, 8193, 3_000_001])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_extrema_at_any_alignment(n, offset, dtype):
    import torch

    import waltz_b200
    rng = np.random.default_rng(n + offset)
    a = rng.standard_normal(n + offset).astype(dtype)
    view = torch.from_numpy(a).cuda()[offset:]
    assert waltz_b200.extrema(view) == (float(a[offset:].min()), float(a[offset:].max()))
    if n > 2:  # a NaN is passed over, infinities are not
        a[offset], a[offset + 1] = np.nan, -np.inf
        view = torch.from_numpy(a).cuda()[offset:]
        assert waltz_b200.extrema(view) == (-np.inf, float(np.nanmax(a[offset:])))
