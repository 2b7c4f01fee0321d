"""The exact cell inverses of A at the edges of their CTAs (kInvCells cells: 64, 25, 16, 9, 7, 5 at
degrees 1 to 6) and with a last row without a partner (odd (P+1)^2): A (A^{-1} v) = v and
A^{-1} (A v) = v to 1e-11 for a density that varies by 30 % inside the cells, on distorted cells."""
import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
CELLS = {1: 64, 2: 25, 3: 16, 4: 9, 5: 7, 6: 5}


@pytest.mark.parametrize("P", sorted(CELLS))
@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_inverse_at_cta_edges(P, extra):
    from atmospheric_flows_b200.operator import EULEROperator
    sc = M.Scaling()
    for nx, nz in ((CELLS[P] + extra, 1), (1, 2 * CELLS[P] + extra), (1, 1)):
        m = M.jitter_mesh(M.box_mesh(nx, nz, 0.0, 50.0 * nx, 0.0, 40.0 * nz), 0.15, 3)
        op = EULEROperator(m, P, sc.Ma, sc.Fr, 0.5)
        rng = np.random.default_rng(nx + 7 * nz)
        n = op.n_dofs(1)
        rho = torch.from_numpy(1.0 + 0.3 * rng.uniform(-1, 1, n)).cuda()
        v = torch.from_numpy(rng.standard_normal(2 * n)).cuda()
        op.set_rho_for_fixed(rho)
        op.set_NS_stage(3)
        x, y = torch.empty_like(v), torch.empty_like(v)
        for a, b in ((op.vmult_inverse, op.vmult), (op.vmult, op.vmult_inverse)):
            a(x, v)
            b(y, x)
            op.synchronize()
            assert float((y - v).norm() / v.norm()) < 1e-11, (nx, nz)
