"""The Gauss-point smoother takes the weights 1/JxW and the face normals from FP64 geometry.

Cells sheared until their two edges are nearly parallel (area 6e-5 of the product of the edges): a
determinant formed in FP32 cancels and is off by 4.3e-4 here (a difference of two rounded products).
Tolerances: the polynomial of degree 1 is D^{-1} b / theta, four contractions of P+1 terms and a few
products in FP32, (4 (P+1) + 6) 2^-24 times the condition of the change of basis (about 10): 2e-5.
Further steps against the nodal smoother (the same polynomial for constant coefficients): FP32
rounding as at the tile edges (2e-5 up to degree 5), times 5 for the anisotropy: 1e-4."""
import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a - b).norm() / b.norm())


def sheared(nx, nz):
    a, d = np.array([830.0, 557.0]), 2.0 ** -14
    c = 0.77 * a + d * np.array([-a[1], a[0]])
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(nz + 1))
    v = i[..., None] * a + j[..., None] * c
    return M.Mesh(nx, nz, np.ascontiguousarray(v), False, 0)


def operator(P, nx=9, nz=7):
    from atmospheric_flows_b200.operator import EULEROperator
    sc = M.Scaling()
    m = sheared(nx, nz)
    n = m.n_cells * (P + 1) ** 2
    op = EULEROperator(m, P, sc.Ma, sc.Fr, 1e-3)
    op.set_stream(torch.cuda.current_stream())
    op.set_HYPERBOLIC_stage(1)
    for f in (op.set_rho_for_fixed, op.set_pres_fixed):
        f(torch.full((n,), 1.1, dtype=torch.float64, device="cuda"))
    b = torch.from_numpy(np.random.default_rng(3).standard_normal(n)).cuda()
    return op, b


@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 6])
def test_inverse_of_a_sheared_cell(P):
    from atmospheric_flows_b200.schur import SchurSolver
    op, b = operator(P)
    s = SchurSolver(op, "cheb_fp32", poly_degree=1)
    s.setup()
    hi = 1.2 * s.levels()[0]
    theta = 0.5 * (hi + min(0.9, hi / s.options.smoothing_range))
    got, want = torch.zeros_like(b), torch.zeros_like(b)
    s.precondition(got, b)
    op.set_NS_stage(6)
    op.vmult_inverse(want, b)
    torch.cuda.synchronize()
    assert rel(got, want / theta) < 2e-5


@pytest.mark.parametrize("P", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("degree", [2, 3])
def test_steps_on_sheared_cells(P, degree):
    from atmospheric_flows_b200.schur import SchurSolver
    op, b = operator(P)
    z = []
    for rq in (1, 2):
        s = SchurSolver(op, "cheb_fp32", poly_degree=degree, reduced_quadrature=rq)
        s.setup()
        z.append(torch.zeros_like(b))
        s.precondition(z[-1], b)
    torch.cuda.synchronize()
    assert rel(z[1], z[0]) < 1e-4
