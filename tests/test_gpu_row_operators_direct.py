"""The one-output-per-thread row operators (N = 64, and N = 128 in FP64) against the FP64 polynomial and dense rows: single and
odd batches (a frequency's last CTA half empty, the self-conjugate frequencies with half the vectors), and both sides of the
FP32 line to the tiled kernel at N = 64. Tolerances, norm-wise: FP64 1e-12, as the row kernels; FP32 5e-7: two rounded
phases and sums of 32 rounded products."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batches", [(6, (1, 2, 5, 40, 41)), (7, (1, 2, 5))])
@pytest.mark.parametrize("method,p,cap", [("lp", 16, 12), ("hybrid", 32, 16)])
@pytest.mark.parametrize("kind", ["G", "BP"])
def test_direct_operators_match_rows(pkg, kind, method, p, cap, n, batches):
    import torch
    from adrt_pinv_gb300.device import RowTables, _op_lists

    plan = pkg.Plan(method, n, pkg.power_lam_max(n, 1 if method == "lp" else 2), deg_cap=p, dense_cap=cap)
    ops = _op_lists(plan)[kind]
    N = 1 << n
    dev = torch.device("cuda")
    ref_t = RowTables(plan, torch.float64, dev)
    ref_t.row_ops = False
    cases = [(RowTables(plan, torch.float64, dev), torch.complex128, 1e-12)]
    if n == 6:
        cases.append((RowTables(plan, torch.float32, dev), torch.complex64, 5e-7))
    g = torch.Generator(device="cuda").manual_seed(n)
    for B in batches:
        Y = torch.randn((B, 4 * N, N), dtype=torch.complex128, device="cuda", generator=g)
        ref = Y.clone()
        ref_t.run(ref, ops)
        for tables, dtype, tol in cases:
            assert tables.row_ops
            got = Y.to(dtype, copy=True)  # run works in place
            tables.run(got, ops)
            assert float((got.to(torch.complex128) - ref).norm() / ref.norm()) < tol, (B, dtype)
