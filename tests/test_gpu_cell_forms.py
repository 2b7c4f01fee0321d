"""The general form of the explicit right-hand sides (radial gravity or the sponge) at the edges of the
tiles that its kernels use: 32 cells at degree 1, 9 at degree 3, and the smaller counts of fused stage
2 (8 at degree 3, 12 at degree 4).  The plain form at these sizes and both forms at the other degrees:
test_gpu_cell_tiles.py.  Oracle, 1e-12 relative L2 as there."""
import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("P,cb", [(1, 32), (3, 9), (3, 8), (4, 12)])
@pytest.mark.parametrize("form", ["sponge", "radial"])
def test_general_form_at_tile_edges(P, cb, form):
    from atmospheric_flows_b200.operator import EULEROperator
    from oracle.oracle import OracleOperator
    sc = M.Scaling()
    for k, (nx, nz, per) in enumerate([(cb - 1, 3, True), (cb, 2, True), (cb + 1, 3, False), (3, cb, True)]):
        m = M.annulus_mesh(nx, nz) if form == "radial" else M.jitter_mesh(M.hill_mesh(nx, nz, periodic_x=per), 0.1, 27 + k)
        g, o = EULEROperator(m, P, sc.Ma, sc.Fr, 0.5), OracleOperator(m, P, sc.Ma, sc.Fr, 0.5)
        if form == "sponge":
            for q in (g, o):
                q.set_sponge(8000.0, 16000.0, 0.02, -20000.0, 20000.0, 6000.0, 0.01, 10.0)
        st = [M.random_state(m, P, 19 * k + j) for j in range(4)]
        full = [a for s in st for a in (s.rho, s.u, s.p)]
        for stage in (1, 2, 3):
            src = full[:3 * stage] + [st[3].rho, st[3].u]
            d = [torch.from_numpy(a).cuda() for a in src]
            out = [torch.empty_like(d[0]), torch.empty_like(d[1]), torch.empty_like(d[0])]
            g.set_HYPERBOLIC_stage(stage)
            o.set_HYPERBOLIC_stage(stage)
            g.vmult_rhs_fused(*out, d)
            g.synchronize()
            want = [o.vmult_rhs_rho_update([x for j in range(stage) for x in src[3 * j:3 * j + 2]]),
                    o.vmult_rhs_velocity_fixed(src[:3 * stage] + (src[3 * stage:3 * stage + 1] if stage < 3 else [])),
                    o.vmult_rhs_pressure(src)]
            for got, w in zip(out, want):
                assert rel(got.cpu().numpy(), w) < 1e-12, (nx, nz, per, stage)
