"""Level kernels at the sizes where their tiles and windows end, and the
extrema reduction, on the GPU."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from tests import patterns as P
from tests.test_gpu_parity import gpu_compress, gpu_decompress, gpu_transform

pytestmark = pytest.mark.gpu

# (nx, ny, nz), dyadic. Strips of 32 x start at 28 mod 32, Z windows hold 16
# planes, Y windows 8 rows; the finest level's half row is a multiple of 4
# (the staged kernels) except in the last two (the register marches).
LEVEL_SHAPES = [(24, 9, 9), (40, 15, 16), (24, 17, 15), (72, 31, 17), (32, 40, 23), (136, 33, 34), (64, 65, 66),
                (37, 33, 35), (66, 47, 41)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nxyz", LEVEL_SHAPES)
def test_levels_bit_exact_at_their_edges(nxyz, dtype):
    rng = np.random.default_rng(sum(nxyz))
    a = rng.standard_normal(P.zyx(nxyz)).astype(dtype)
    f = gpu_transform(a, inverse=False)
    assert f.tobytes() == O.transform(a, inverse=False).tobytes()
    assert gpu_transform(f, inverse=True).tobytes() == O.transform(f, inverse=True).tobytes()
    # 1e-1 on noise leaves many samples to repair, 1e-4 few
    for eb in (float(np.float32(1e-1)), float(np.float32(1e-4))):
        expect = O.compress(a, eb)
        assert gpu_compress(a, eb) == expect
        assert gpu_decompress(expect, a.shape, dtype).tobytes() == O.decompress(expect, a.shape, dtype).tobytes()


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


@pytest.mark.parametrize("form", ["matrix-tf32", "matrix-bf16", "matrix-exact"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_matrix_repairs_with_a_partial_last_warp(form, dtype):
    """612 columns: the last warp of the matrix synthesis holds four of them.
    The repairs recorded are exactly the samples whose synthesis without
    repairs misses the bound, each with its error; every sample meets the
    bound and the decode repeats."""
    import waltz_b200
    from waltz_b200 import synthetic as S
    a = S.power_law_field((33, 18, 34), 6, dtype=dtype)
    eb = float(np.float32(1e-3))
    archive = waltz_b200.compress(a, abs_error=eb, form=form)
    wzp, = np.frombuffer(archive[16:24], np.uint64)
    count, outliers = np.frombuffer(archive[24:32], np.uint32)
    assert count > 0, "the field has repairs"
    at = 32 + (int(wzp) + 7) // 8 * 8
    values = at + (4 * int(count) + 7) // 8 * 8
    rest = values + (a.itemsize * int(count) + 7) // 8 * 8
    # the same archive without its repair section
    bare = archive[:4] + bytes(4) + archive[8:24] + bytes(4) + archive[28:at] + archive[rest:]
    raw = waltz_b200.decompress(bare, shape=a.shape, dtype=dtype)
    err = (raw - a).ravel()
    missed = np.flatnonzero(np.abs(err) > dtype(eb))
    index = np.frombuffer(archive[at:at + 4 * count], np.uint32)
    assert np.array_equal(index, missed)
    assert np.array_equal(np.frombuffer(archive[values:values + a.itemsize * count], dtype), err[missed])
    assert (index % 612 >= 608).any(), "some of them in the last warp"
    out = waltz_b200.decompress(archive, shape=a.shape, dtype=dtype)
    assert np.abs(out.astype(np.float64) - a.astype(np.float64)).max() <= eb
    assert waltz_b200.decompress(archive, shape=a.shape, dtype=dtype).tobytes() == out.tobytes()
    assert waltz_b200.compress(a, abs_error=eb, form=form) == archive


_ROUND_TRIP = """
import ctypes as C, sys, torch
from waltz_b200 import _lib
z, y, x = 1040, 2048, 2056
assert z * y * x > 1 << 32
a = torch.empty((z, y, x), device="cuda").normal_(generator=torch.Generator("cuda").manual_seed(3))
b = a.clone()
for inverse in (0, 1):
    _lib.checked(_lib.lib().waltz_b200_transform(C.c_void_p(b.data_ptr()), 4, x, y, z, inverse,
                                                 C.c_void_p(torch.cuda.current_stream().cuda_stream)))
worst = max(float((p - q).abs().max()) for p, q in zip(a.split(40), b.split(40)))
print("worst", worst)
sys.exit(worst > 1e-3)
"""


def test_transform_of_more_than_2_to_the_32_samples():
    """The transform entry takes any size: forward and inverse of 4.4e9 samples
    give the field back (rounding alone: about 1e-5 of samples of order one).
    In a process of its own, whose scratch ends with it."""
    import subprocess
    import sys

    import torch
    if torch.cuda.mem_get_info()[0] < 110 << 30:
        pytest.skip("needs 110 GiB of device memory")
    r = subprocess.run([sys.executable, "-c", _ROUND_TRIP], capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stdout + r.stderr
