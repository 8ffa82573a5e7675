"""The tiled outer step (float-float state, G_1 preconditioner; chosen by size and batch when no band is given) against the
clustered register-resident form (any explicit band): the same arithmetic in the same order, so the new states are equal
bit for bit. Batches lie on both sides of every line of the dispatch; degrees up to the halo and beyond it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batches", [(6, (1, 76, 77)), (7, (1, 19, 20, 38, 39)), (8, (1, 4, 5, 25, 26)), (9, (1, 2, 5))])
@pytest.mark.parametrize("deg", [1, 2, 14, 16, 17])
def test_tiles_equal_clusters(pkg, n, batches, deg):
    import torch

    N = 1 << n
    if deg != 14:
        batches = batches[:2]
    plan = pkg.Plan("hybrid", n, np.full(2 * N, 4.0), precond="g1", g1_deg=deg, outer=(1.0, 2.0, 3))
    for B in batches:
        pipe = pkg.Pipeline(plan, B, "fp32")
        assert pipe.ff_state
        g = torch.Generator(device="cuda").manual_seed(n + B)
        pipe.parts.normal_(generator=g)
        y = torch.randn((B, N, N), dtype=torch.float32, device="cuda", generator=g)
        x, xp = (torch.randn((B, 2, N, N), dtype=torch.float32, device="cuda", generator=g) for _ in range(2))
        x[:, 1] *= 1e-8
        xp[:, 1] *= 1e-8
        om = torch.rand((B, 2), dtype=torch.float64, device="cuda", generator=g)
        outs = []
        for band in (0, 32):
            pipe.band = band
            a, b, c = (torch.full_like(x, 7.0) for _ in range(3))
            pipe.fused_outer_step(y, True, x, xp, a, 0.7, 0.3, 0.0)
            pipe.fused_outer_step(y, True, x, xp, b, 0.0, 0.0, 0.0, om_img=om)
            pipe.fused_outer_step(y, False, None, None, c, 0.0, 0.0, 0.37)
            outs.append((a, b, c))
        for u, v in zip(*outs):
            assert torch.equal(u, v), (B, deg)
