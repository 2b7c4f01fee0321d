"""The two routes of the Gauss-point polynomial: all steps in one cooperative launch (meshes whose tiles
are resident together) and one launch per half step (the others)."""
import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a - b).norm() / b.norm())


def setup(nx, nz, P, per, degree, rq=2, dt=0.5):
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
    b = torch.from_numpy(np.random.default_rng(5).standard_normal(m.n_cells * (P + 1) ** 2)).cuda()
    return s, b


@pytest.mark.parametrize("degree", [8, 130])  # one launch; three, of which the first gives up
def test_given_up_wait_leaves_the_output_unwritten(degree):
    from atmospheric_flows_b200.operator import AF_TIMEOUT, AFError
    s, b = setup(20, 11, 4, True, degree)
    want = torch.zeros_like(b)
    s.precondition(want, b)
    s.op.synchronize()
    got = torch.full_like(b, 12345.0)
    s.op.set_stage_wait_test(64)
    s.precondition(got, b)
    with pytest.raises(AFError) as e:
        s.op.synchronize()
    assert e.value.status == AF_TIMEOUT
    assert bool((got == 12345.0).all())
    s.op.set_stage_wait_test(0)
    s.precondition(got, b)
    s.op.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("degree,launches", [(1, 2), (8, 3), (65, 3), (66, 4), (130, 5)])
def test_launch_count_of_the_one_launch_route(degree, launches):
    """Entry and exit, and one launch per 64 of the degree - 1 steps."""
    s, b = setup(20, 11, 4, True, degree)
    out, before = torch.empty_like(b), s.op.launch_count()
    s.precondition(out, b)
    assert s.op.launch_count() - before == launches


def pair(s, b):
    """One application by the pair of kernels, which the launch count confirms."""
    s.set_one_launch(False)
    out, before = torch.empty_like(b), s.op.launch_count()
    s.precondition(out, b)
    assert s.op.launch_count() - before == 2 + 2 * (s.options.poly_degree - 1)
    return out


# As the one-launch route at the edges of its tiles (tolerance: FP32 rounding of up to five steps against the
# nodal smoother, 2e-5); steps that leave x, add two directions and, at the last odd step, one
@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 6])
def test_pair_at_tile_edges(P):
    for nx, nz, per in [(5, 3, True), (31, 1, False), (8, 4, True), (11, 3, False), (1, 33, True), (21, 5, True),
                        (32, 2, True)]:
        for degree in (1, 2, 3, 4, 5):
            s, b = setup(nx, nz, P, per, degree)
            nodal, _ = setup(nx, nz, P, per, degree, rq=1)
            want = torch.empty_like(b)
            nodal.precondition(want, b)
            assert rel(pair(s, b), want) < 2e-5, (nx, nz, per, degree)


# consecutive launches overlap; a load moved above the wait for the kernel before shows on small meshes
@pytest.mark.parametrize("P", [2, 4, 6])
@pytest.mark.parametrize("degree", [16, 17])
def test_overlapping_pairs_repeat(P, degree):
    s, b = setup(20, 11, P, True, degree)
    out = [pair(s, b) for _ in range(40)]
    torch.cuda.synchronize()
    for o in out[1:]:
        assert torch.equal(o, out[0])


# more tiles than are resident at once, with walls; an odd and an even number of steps
@pytest.mark.parametrize("P,nx,nz", [(1, 301, 200), (2, 199, 201), (3, 161, 150), (4, 141, 137), (5, 121, 119), (6, 99, 97)])
@pytest.mark.parametrize("degree", [4, 5])
def test_large_walled_meshes(P, nx, nz, degree):
    dt = 0.5 * min(16 / nx, 8 / nz)
    s, b = setup(nx, nz, P, False, degree, dt=dt)
    nodal, _ = setup(nx, nz, P, False, degree, rq=1, dt=dt)
    got, want, before = torch.empty_like(b), torch.empty_like(b), s.op.launch_count()
    s.precondition(got, b)
    assert s.op.launch_count() - before == 2 + 2 * (degree - 1)
    nodal.precondition(want, b)
    assert rel(got, want) < 2e-5
