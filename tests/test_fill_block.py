"""Single blocks of the boundary operator at the edges of the fill tiles (32 columns, 128 rows for a
block of its own): any rows and columns, in any order, against the assembled operator."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 31, 127, 128, 129, 300])
@pytest.mark.parametrize("n", [1, 32, 33, 300])
def test_block_of_any_rows_and_columns(m, n):
    import torch
    import spinfemx_b200 as spx
    X, T = spx.kuhn_box(11, 9, 4, 2.0)
    g = spx.BoundaryGeometry(X, T)
    jump = torch.as_tensor(spx.geometry.boundary_data(X, T)["omega_sum"] / (4 * np.pi) - 1.0, device="cuda")
    B = g.dense_B() - torch.diag(jump)
    rng = np.random.default_rng(m + 1000 * n)
    r, c = (torch.as_tensor(rng.permutation(g.Nb)[:k].astype(np.int32), device="cuda") for k in (m, n))
    ref = B[r.long()][:, c.long()]
    # tens of terms an entry, in another order in another tile: rounding of entries below one
    assert float((g.fill_block(r, c) - ref).abs().max()) < 1e-13
