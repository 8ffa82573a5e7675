"""Row operators (adrt_rows_operator: a packed pass as one real matrix pair per frequency) against the FP64 polynomial and
dense rows of the row engine on random packed rows.

Tolerances, norm-wise over all rows: FP64 1e-12, as the row kernels are held to; FP32 1e-6: two half-shift phases, the
sums over N/2 <= 256 terms of rounded products (about sqrt(256) eps = 1e-6 at worst, norm-wise less) and FP32 matrices."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plans(pkg):
    cache = {}

    def get(method, n, p, cap):
        key = (method, n, p, cap)
        if key not in cache:
            lam = pkg.power_lam_max(n, 1 if method == "lp" else 2)
            cache[key] = pkg.Plan(method, n, lam, deg_cap=p, dense_cap=cap)
        return cache[key]

    return get


def _tables(plan, real, ops):
    import torch
    from adrt_pinv_gb300.device import RowTables

    t = RowTables(plan, real, torch.device("cuda"))
    assert t.row_ops
    t.row_ops = ops
    return t


# batches around the kernels' tiles: one image, the few-vector kernel, its limit (2 VT / 4 vectors), ragged tiles
@pytest.mark.parametrize("n,batches", [(6, (1, 3, 16, 17, 37)), (7, (1, 3, 4, 8, 9, 33)), (8, (1, 2, 4, 5, 13)), (9, (1, 2, 3, 7))])
@pytest.mark.parametrize("method,p,cap", [("lp", 16, 12), ("hybrid", 32, 16), ("hybrid", 8, None)])
@pytest.mark.parametrize("kind", ["G", "BP"])
def test_row_operators_match_rows(pkg, plans, kind, method, p, cap, n, batches):
    import torch
    from adrt_pinv_gb300.device import _op_lists

    plan = plans(method, n, p, cap)
    ops = _op_lists(plan)[kind]
    N = 1 << n
    g = torch.Generator(device="cuda").manual_seed(n)
    ref_t, op64, op32 = (_tables(plan, torch.float64, False), _tables(plan, torch.float64, True),
                         _tables(plan, torch.float32, True))
    for B in batches:
        Y = torch.randn((B, 4 * N, N), dtype=torch.complex128, device="cuda", generator=g)
        ref = Y.clone()
        ref_t.run(ref, ops)
        got = Y.clone()
        op64.run(got, ops)
        assert float((got - ref).norm() / ref.norm()) < 1e-12, B
        y32 = Y.to(torch.complex64)
        op32.run(y32, ops)
        assert float((y32.to(torch.complex128) - ref).norm() / ref.norm()) < 1e-6, B
        # every frequency, the largest error of any row against the largest row
        rows = (y32.to(torch.complex128) - ref).norm(dim=-1).amax() / ref.norm(dim=-1).amax()
        assert float(rows) < 1e-6, B
        assert op32.count == op64.count == ref_t.count
        if n >= 7:
            # both forms of the FP32 operators at every batch, the tensor cores to the same bound
            for form in (True, False):
                op32.op_mma = form
                y32 = Y.to(torch.complex64)
                op32.run(y32, ops)
                op32.raise_if_error()
                assert float((y32.to(torch.complex128) - ref).norm() / ref.norm()) < 1e-6, (B, form)
            op32.op_mma = None
            op32.count = ref_t.count


@pytest.mark.parametrize("n", [7, 8, 9])
def test_tensor_core_form_keeps_range_and_accuracy(pkg, plans, n):
    """Vectors of very different magnitude (1e-30 .. 1e30) in one batch each keep their own scale, zero rows stay zero, a
    row with a wide dynamic range keeps the accuracy of its largest values, and non-finite rows touch no other row."""
    import torch
    from adrt_pinv_gb300.device import _op_lists

    plan = plans("hybrid", n, 32, 16)
    ops, N, B = _op_lists(plan)["G"], 1 << n, 9
    ref_t, t = _tables(plan, torch.float64, True), _tables(plan, torch.float32, True)
    t.op_mma = True
    g = torch.Generator(device="cuda").manual_seed(5)
    Y = torch.randn((B, 4 * N, N), dtype=torch.complex128, device="cuda", generator=g)
    mag = torch.randint(-30, 31, (B, 4 * N, 1), device="cuda", generator=g).double()
    Y *= 10.0 ** mag
    Y[2] = 0
    Y[3] *= torch.exp(-20.0 * torch.rand((4 * N, N), device="cuda", generator=g, dtype=torch.float64))
    y32 = Y.to(torch.complex64)
    ref = y32.to(torch.complex128)
    ref_t.run(ref, ops)
    got = y32.clone()
    t.run(got, ops)
    t.raise_if_error()
    err = (got.to(torch.complex128) - ref).norm(dim=-1)
    assert not got[2].any()
    assert bool((err <= 2e-6 * ref.norm(dim=-1)).all())
    bad = y32.clone()
    bad[4, 7, 5] = float("nan")
    bad[5, 9, 1] = float("inf")
    t.run(bad, ops)
    rows = torch.isfinite(torch.view_as_real(bad)).all(dim=-1).all(dim=-1)
    assert not rows[4, 7] and not rows[5, 9] and int(rows.sum()) == rows.numel() - 2
    rows = rows.clone()
    assert torch.equal(bad[rows], got[rows])


def test_row_operators_need_symmetric_plans(pkg, plans):
    """A plan whose bounds or degrees differ between k and -k, or that asked for no operator memory, keeps the polynomial
    rows; so do sizes outside the operators' range."""
    from adrt_pinv_gb300.device import row_operators_for

    plan = plans("hybrid", 6, 8, None)
    assert row_operators_for(plan)
    lam, deg = plan.lam_max.copy(), plan.deg.copy()
    deg[3] += 1
    assert not row_operators_for(pkg.Plan("hybrid", 6, lam, deg=deg))
    lam[5] *= 1.5
    assert not row_operators_for(pkg.Plan("hybrid", 6, lam, raw_lam=True))
    assert not row_operators_for(pkg.Plan("hybrid", 6, plan.lam_max, deg_cap=8, dense_cap=4, high_rows="ff"))
    assert not row_operators_for(pkg.Plan("lp", 5, np.full(64, 4.0))) and not row_operators_for(
        pkg.Plan("lp", 10, np.full(2048, 4.0)))


def test_row_operators_row_stride_and_errors(pkg, plans):
    """Rows of a longer image stride are left alone, and bad arguments are refused."""
    import torch

    plan = plans("lp", 6, 16, 12)
    C = pkg._lib
    t = _tables(plan, torch.float32, True)
    T, N = t.op_table("G"), 64
    Y = torch.randn((3, 4 * N + 2, N), dtype=torch.complex64, device="cuda")
    want = Y[:, :4 * N].clone()
    t.run_operators(want, "G", T)
    got = Y.clone()
    st = C.stream_handle()
    C.call("adrt_rows_operator", C.F32, 6, 3, 0, C.ptr(T), C.ptr(got), (4 * N + 2) * N, C.ptr(t._roots8), st)
    assert torch.equal(got[:, :4 * N], want) and torch.equal(got[:, 4 * N:], Y[:, 4 * N:])
    for args in ((C.I32, 6, 3, 0, C.ptr(T)), (C.F32, 5, 3, 0, C.ptr(T)), (C.F32, 10, 3, 0, C.ptr(T)),
                 (C.F32, 6, -1, 0, C.ptr(T)), (C.F32, 6, 3, 2, C.ptr(T)), (C.F32, 6, 3, 0, None)):
        with pytest.raises(RuntimeError):
            C.call("adrt_rows_operator", *args, C.ptr(got), 4 * N * N, C.ptr(t._roots8), st)
