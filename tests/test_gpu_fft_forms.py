"""The offset FFTs' two forms (few points per thread for small launches, many for large ones) against each other over their
line: the first images of a batch that takes the large form, against the same images in batches that take the small one.
Tolerance: at most 2 x 10 radix-2 levels there and back, each about one unit roundoff of a complex multiply-add (2 u), so
40 u norm-wise: 2.4e-6 in FP32, 4.5e-15 in FP64."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n", [("fp32", 8), ("fp64", 3), ("fp64", 4), ("fp64", 5), ("fp64", 6), ("fp64", 7),
                                         ("fp64", 8), ("fp64", 9)])
def test_small_and_large_form_agree(pkg, precision, n):
    import numpy as np
    import torch

    N = 1 << n
    line = max(1, 512 >> n)                                # images of the largest small launch (N = 512: one)
    plan = pkg.Plan("hybrid", n, np.full(2 * N, 4.0), outer=(1.0, 2.0, 3))
    x = torch.randn((line + 1, N, N), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))

    def there_and_back(a):
        pipe = pkg.Pipeline(plan, len(a), precision)
        pipe.pack(a, sino=False)
        spectrum = pipe.Y.clone()
        pipe.packed_image(a, [])                           # no row operator: the transforms alone
        out = torch.empty_like(a)
        pipe.sum_parts(out)
        return spectrum, out

    large = there_and_back(x)
    tol = 40 * 2.0 ** (-24 if precision == "fp32" else -53)
    for B in {1, line}:
        for got, ref in zip(there_and_back(x[:B].contiguous()), large):
            assert float((got - ref[:B]).norm() / ref[:B].norm()) < tol, B
