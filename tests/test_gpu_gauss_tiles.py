"""The Gauss-point smoother at the edges of its 32-cell tiles: fewer cells than a tile, one tile
exactly, one cell more, rows that cross tiles, columns of single cells, and the polynomial degrees
whose last step adds one or two directions to x (degree 1: no step).  Compared with the nodal
smoother (reduced_quadrature = 1: the same polynomial; FP32 rounding, amplified by the recurrence:
2e-5 up to degree 5, as for degree 2 on the 16x8 mesh, the condition being smaller on fewer cells),
and a chain of applications of a small mesh, whose kernels overlap, must repeat bit for bit."""
import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def setup(nx, nz, P, per, degree, rq, dt=0.5):
    from atmospheric_flows_b200.operator import EULEROperator
    from atmospheric_flows_b200.schur import SchurSolver
    sc = M.Scaling()
    m = M.hill_mesh(nx, nz, periodic_x=per)
    op = EULEROperator(m, P, sc.Ma, sc.Fr, dt)
    op.set_stream(torch.cuda.current_stream())
    op.set_HYPERBOLIC_stage(1)
    st = M.hill_state(m, P, modes=4)
    op.set_rho_for_fixed(torch.from_numpy(st.rho).cuda())
    op.set_pres_fixed(torch.from_numpy(st.p).cuda())
    s = SchurSolver(op, "cheb_fp32", poly_degree=degree, reduced_quadrature=rq)
    s.setup()
    return s, m.n_cells * (P + 1) ** 2


@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("nx,nz,per", [(5, 3, True), (31, 1, False), (8, 4, True), (11, 3, False), (1, 33, True),
                                       (21, 5, True), (32, 2, True)])
def test_smoother_at_tile_edges(P, nx, nz, per):
    for degree in (1, 2, 3, 4, 5):
        z = {}
        for rq in (1, 2):
            s, n = setup(nx, nz, P, per, degree, rq)
            b = torch.from_numpy(np.random.default_rng(5).standard_normal(n)).cuda()
            z[rq] = torch.zeros_like(b)
            s.precondition(z[rq], b)
            torch.cuda.synchronize()
        assert rel(z[2].cpu().numpy(), z[1].cpu().numpy()) < 2e-5, degree


@pytest.mark.parametrize("P", [2, 4, 6])
def test_overlapping_applications_repeat(P):
    s, n = setup(20, 11, P, True, 16, 2)
    b = torch.from_numpy(np.random.default_rng(5).standard_normal(n)).cuda()
    out = [torch.empty_like(b) for _ in range(40)]
    for o in out:
        s.precondition(o, b)
    torch.cuda.synchronize()
    for o in out[1:]:
        assert torch.equal(o, out[0])


def both(nx, nz, P, per, degree, dt):
    z = {}
    for rq in (1, 2):
        s, n = setup(nx, nz, P, per, degree, rq, dt)
        b = torch.from_numpy(np.random.default_rng(5).standard_normal(n)).cuda()
        z[rq] = torch.zeros_like(b)
        s.precondition(z[rq], b)
        torch.cuda.synchronize()
    return z[2].cpu().numpy(), z[1].cpu().numpy()


# more tiles than the device holds at once (148 SMs, 5 to 12 CTAs each): a launch per half step; the same
# Courant number, hence condition, as the 16x8 mesh above, and the tolerance of up to five steps
@pytest.mark.parametrize("P,nx,nz", [(1, 301, 200), (2, 199, 201), (3, 161, 150), (4, 141, 137), (5, 121, 119), (6, 99, 97)])
def test_smoother_of_large_meshes(P, nx, nz):
    got, want = both(nx, nz, P, True, 5, 0.5 * min(16 / nx, 8 / nz))
    assert rel(got, want) < 2e-5


# one launch takes 64 steps: 64, 65 and 129 steps; rounding grows with their number (2e-5 for five)
@pytest.mark.parametrize("P", [1, 4, 6])
@pytest.mark.parametrize("degree", [65, 66, 130])
def test_many_steps(P, degree):
    got, want = both(21, 5, P, True, degree, 0.5)
    assert rel(got, want) < 2e-5 * degree / 5


def test_waits_between_tiles_are_bounded():
    from atmospheric_flows_b200.operator import AF_TIMEOUT, AFError
    s, n = setup(20, 11, 4, True, 8, 2)
    b = torch.from_numpy(np.random.default_rng(5).standard_normal(n)).cuda()
    want, got = torch.zeros_like(b), torch.zeros_like(b)
    s.precondition(want, b)
    s.op.synchronize()
    s.op.set_stage_wait_test(64)
    s.precondition(got, b)
    with pytest.raises(AFError) as e:
        s.op.synchronize()
    assert e.value.status == AF_TIMEOUT
    s.op.set_stage_wait_test(0)
    s.precondition(got, b)
    s.op.synchronize()
    assert torch.equal(got, want)
