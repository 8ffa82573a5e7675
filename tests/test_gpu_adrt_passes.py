"""The multi-level ADRT passes (adrt_fwd_pass / adrt_adj_pass: up to four levels per pass, bands of rows with a halo)
against the oracle, bit for bit: integers exactly, floating point because the additions and their order are the
reference's. Sizes cover every split of the levels into passes (1 to 3 passes), every band height and ragged last bands."""

import numpy as np
import pytest

from oracle import adrt_np as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
@pytest.mark.parametrize("dtype", ["int32", "int64", "float32", "float64"])
def test_passes_match_oracle(pkg, n, dtype):
    import torch

    N, B = 1 << n, 3 if n < 9 else 1
    rng = np.random.default_rng(n)
    x = rng.integers(-99, 256, (B, N, N)).astype(dtype)
    b = rng.integers(-99, 256, (B, 4, 2 * N - 1, N)).astype(dtype)
    f = pkg.adrtcore.adrt(n, torch.from_numpy(x).cuda(), dtype=dtype).cpu().numpy()
    t = pkg.adrtcore.adrt_T(n, torch.from_numpy(b).cuda(), dtype=dtype).cpu().numpy()
    for i in {0, B - 1}:
        # whole numbers below 2^24 throughout for the forward (256 N <= 2^18), so FP32 sums are exact too
        assert np.array_equal(f[i].astype(np.float64), A.adrt(n, x[i].astype(np.float64)))
        ref = A.adrt_T(n, b[i].astype(np.float64))
        if dtype == "float32":  # |R^T b| <= 4 N 256 stays below 2^24 up to N = 1024
            assert np.abs(ref).max() < 2 ** 24
        assert np.array_equal(t[i].astype(np.float64), ref)


@pytest.mark.parametrize("n", [5, 8])
def test_floating_sums_keep_their_order(pkg, n):
    N = 1 << n
    rng = np.random.default_rng(n)
    x, b = rng.standard_normal((N, N)), rng.standard_normal((4, 2 * N - 1, N))
    assert np.array_equal(pkg.adrtcore.adrt(n, x), A.adrt(n, x))
    assert np.array_equal(pkg.adrtcore.adrt_T(n, b), A.adrt_T(n, b))


def test_entries_outside_the_domain_stay_unread(pkg):
    """The transpose never uses the structurally zero entries h < -s of a sinogram: NaNs there change nothing."""
    n, N = 7, 128
    b = np.random.default_rng(3).standard_normal((4, 2 * N - 1, N))
    dirty = np.where(pkg.adrtcore.mask_full(n), b, np.nan)
    out = pkg.adrtcore.adrt_T(n, dirty)
    assert np.array_equal(out, pkg.adrtcore.adrt_T(n, np.where(pkg.adrtcore.mask_full(n), b, 0.0)))


def test_largest_size_adjoint_identity(pkg):
    """N = 4096 (n = 12, three passes of four levels): <R x, y> = <x, R^T y> and row sums of a constant image."""
    import torch

    n, N = 12, 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((N, N), dtype=torch.float64, device="cuda", generator=g)
    y = torch.randn((4, 2 * N - 1, N), dtype=torch.float64, device="cuda", generator=g)
    y *= torch.from_numpy(pkg.adrtcore.mask_full(n)).cuda()
    lhs = float((pkg.adrtcore.adrt(n, x) * y).sum())
    rhs = float((x * pkg.adrtcore.adrt_T(n, y)).sum())
    assert abs(lhs - rhs) < 1e-9 * float(y.norm() * x.norm()) * N ** 0.5
    r = pkg.adrtcore.adrt(n, torch.ones((N, N), dtype=torch.int32, device="cuda"), dtype="int32")
    assert torch.equal(r.sum(dim=1), torch.full((4, N), N * N, dtype=r.sum(dim=1).dtype, device="cuda"))
