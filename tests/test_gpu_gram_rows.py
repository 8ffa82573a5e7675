"""The Gram rows (rows_gram_kernel, one M = B^* B over all levels) through gram.gram_freq at every size and at batches
around the images-per-item split, against the oracle's butterflies. Norm-wise tolerances: FP64 1e-12 (as the row kernels);
FP32 2e-6: 2 n <= 22 levels of FP32 multiply-adds and FP32 twiddles, each about 1e-7 of the row."""

import numpy as np
import pytest

from oracle import oblique_np as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", range(1, 12))
def test_gram_rows_match_oracle(pkg, n):
    import torch

    N, rows = 1 << n, 6 if n > 8 else 11
    rng = np.random.default_rng(n)
    omega = rng.uniform(-np.pi, np.pi, rows)
    omega[:2] = 0.0, np.pi
    z = np.exp(1j * omega)
    for B in (1, 2, 5, 9):
        a = rng.standard_normal((B, rows, N)) + 1j * rng.standard_normal((B, rows, N))
        ref = np.stack([O.bflyT(n, z, O.bfly(n, z, a[i])) for i in range(B)])
        got = pkg.gram.gram_freq(torch.from_numpy(a).cuda(), torch.from_numpy(omega)).cpu().numpy()
        assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-12
        w32 = omega.astype(np.float32)
        z32 = np.exp(1j * w32.astype(np.float64))
        a32 = a.astype(np.complex64)
        ref32 = np.stack([O.bflyT(n, z32, O.bfly(n, z32, a32[i].astype(complex))) for i in range(B)])
        got = pkg.gram.gram_freq(torch.from_numpy(a32).cuda(), torch.from_numpy(w32)).cpu().numpy()
        err = np.linalg.norm(got - ref32, axis=-1) / np.linalg.norm(ref32, axis=-1)
        assert err.max() < 2e-6, (B, err.max())


def test_gram_rows_many_images_per_row(pkg):
    """Enough rows and images that a group keeps its twiddles for four images, with a ragged last chunk: every image as
    the same rows alone."""
    import torch

    n, N, B = 6, 64, 23
    a = torch.randn((B, 4096, N), dtype=torch.complex64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    w = torch.linspace(-3.1, 3.1, 4096)
    full = pkg.gram.gram_freq(a, w)
    for i in (0, 3, 4, 20, 22):
        assert torch.equal(full[i], pkg.gram.gram_freq(a[i], w))
