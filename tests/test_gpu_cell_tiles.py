"""The cell kernel at the edges of its tiles: CTAs of consecutive cells that end inside a row,
span several short rows, hold a whole periodic row or its two ends, and partial or odd last CTAs
(the non-bulk staging and stores), for every degree; all stages, with one, two and three face
groups, and both compiled forms of the explicit right-hand sides (vertical gravity alone; radial
gravity or the sponge).  Oracle, 1e-12 relative L2 (velocity 1e-12 as in the other parity tests)."""
import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

TOL = 1e-12
# cells per CTA of the FP64 right-hand sides per degree
CELLS = {1: 42, 2: 24, 3: 18, 4: 14, 5: 11, 6: 8}


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def shapes(P):
    cb = CELLS[P]
    return [(cb, 2, True), (cb - 1, 3, True), (cb + 1, 3, False), (3, cb // 2, True), (2 * cb + 1, 1, True),
            (cb // 2 + 1, 5, True)]


@pytest.mark.parametrize("P", sorted(CELLS))
@pytest.mark.parametrize("form", ["plain", "sponge", "radial"])
def test_rhs_at_tile_edges(P, form):
    from atmospheric_flows_b200.operator import EULEROperator
    from oracle.oracle import OracleOperator
    sc = M.Scaling()
    for k, (nx, nz, per) in enumerate(shapes(P)):
        m = M.annulus_mesh(max(nx, 3), nz) if form == "radial" else M.jitter_mesh(
            M.hill_mesh(nx, nz, periodic_x=per), 0.1, 7 + k)
        g, o = EULEROperator(m, P, sc.Ma, sc.Fr, 0.5), OracleOperator(m, P, sc.Ma, sc.Fr, 0.5)
        if form == "sponge":
            for q in (g, o):
                q.set_sponge(8000.0, 16000.0, 0.02, -20000.0, 20000.0, 6000.0, 0.01, 10.0)
        st = [M.random_state(m, P, 11 * k + j) for j in range(4)]
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
                assert rel(got.cpu().numpy(), w) < TOL, (nx, nz, per, stage)


@pytest.mark.parametrize("P", sorted(CELLS))
def test_range_launches_at_any_cell(P):
    """The host-buffer call launches the kernel on ranges of rows: odd row lengths give ranges that
    start at cells off the tile grid.  Bit-identical to the whole-mesh launch."""
    from atmospheric_flows_b200.operator import EULEROperator
    sc = M.Scaling()
    for nx, nz in ((CELLS[P] + 2, 40), (7, 33)):
        m = M.hill_mesh(nx, nz, periodic_x=True)
        g = EULEROperator(m, P, sc.Ma, sc.Fr, 0.5)
        st, s2 = M.random_state(m, P, 3), M.random_state(m, P, 4)
        src = [st.rho, st.u, st.p, s2.rho, s2.u]
        g.set_HYPERBOLIC_stage(1)
        d = [torch.from_numpy(a).cuda() for a in src]
        out = [torch.empty_like(d[0]), torch.empty_like(d[1]), torch.empty_like(d[0])]
        g.vmult_rhs_fused(*out, d)
        g.synchronize()
        host = [np.empty(t.numel()) for t in out]
        g.vmult_rhs_fused_host(*host, src)
        for a, b in zip(out, host):
            assert np.array_equal(a.cpu().numpy(), b)


# cells per CTA of the fused right-hand sides where they differ from the sizes above: the degree's own
# count, and the smaller one of stage 2 that lets one more CTA share an SM
@pytest.mark.parametrize("P,cb", [(1, 32), (3, 9), (3, 8), (4, 12)])
def test_rhs_at_small_tile_edges(P, cb):
    from atmospheric_flows_b200.operator import EULEROperator
    from oracle.oracle import OracleOperator
    sc = M.Scaling()
    for k, (nx, nz, per) in enumerate([(cb, 2, True), (cb + 1, 3, False), (3, cb, True), (2 * cb - 1, 1, True)]):
        m = M.jitter_mesh(M.hill_mesh(nx, nz, periodic_x=per), 0.1, 17 + k)
        g, o = EULEROperator(m, P, sc.Ma, sc.Fr, 0.5), OracleOperator(m, P, sc.Ma, sc.Fr, 0.5)
        st = [M.random_state(m, P, 13 * k + j) for j in range(4)]
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
                assert rel(got.cpu().numpy(), w) < TOL, (nx, nz, per, stage)
