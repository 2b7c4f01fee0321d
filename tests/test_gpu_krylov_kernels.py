"""The Krylov basis kernels against host sums (tests/cpp/krylov_test.cpp), and FGMRES on vectors that
take every block of them several trips: its iterates minimise the residual over the preconditioned
Krylov space, restated with torch in FP64 from the solver's own preconditioner and the operator's own
apply."""
import os
import subprocess

import numpy as np
import pytest

from atmospheric_flows_b200 import mesh as M

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_kernels_against_host_sums(tmp_path):
    lib = os.path.join(ROOT, "atmospheric_flows_b200")
    exe = tmp_path / "krylov_test"
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(lib, "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "krylov_test.cpp"), "-o", str(exe), "-L", lib, "-laf_gpu",
                    "-L", "/usr/local/cuda/lib64", "-lcudart", f"-Wl,-rpath,{lib}",
                    "-Wl,-rpath,/usr/local/cuda/lib64"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("precond", ["jacobi", "cheb_fp32"])
def test_iterates_on_long_vectors(precond):
    """478975 unknowns (more than 444 chunks of 1024, odd).  Residuals to 1e-9 of |b|, iterates to 1e-8
    (rounding of 1e-13 in the basis times a condition of the small least squares problem below 1e4)."""
    from atmospheric_flows_b200.operator import EULEROperator
    from atmospheric_flows_b200.schur import SchurSolver
    P, sc = 4, M.Scaling()
    m = M.hill_mesh(161, 119, periodic_x=True)
    st = M.hill_state(m, P, modes=4)
    op = EULEROperator(m, P, sc.Ma, sc.Fr, 0.05)
    op.set_stream(torch.cuda.current_stream())
    op.set_schur_mode(1)
    op.set_HYPERBOLIC_stage(1)
    op.set_rho_for_fixed(torch.from_numpy(st.rho).cuda())
    op.set_pres_fixed(torch.from_numpy(st.p).cuda())
    n = op.n_dofs(1)
    assert n > 444 * 1024 and n % 1024
    b = torch.from_numpy(np.random.default_rng(7).standard_normal(n)).cuda()
    s = SchurSolver(op, precond, restart=24)
    s.setup()
    steps = 12
    ld = n + n % 2
    V, Z = (torch.zeros(steps + 1, ld, dtype=torch.float64, device="cuda") for _ in range(2))
    H = torch.zeros(steps + 1, steps, dtype=torch.float64, device="cuda")
    op.set_NS_stage(2)
    beta = b.norm()
    V[0, :n] = b / beta
    for j in range(steps):
        s.precondition(Z[j, :n], V[j, :n])
        w = torch.empty(n, dtype=torch.float64, device="cuda")
        op.vmult(w, Z[j, :n])
        for _ in range(2):
            h = V[:j + 1, :n] @ w
            w -= h @ V[:j + 1, :n]
            H[:j + 1, j] += h
        H[j + 1, j] = w.norm()
        V[j + 1, :n] = w / H[j + 1, j]
    for k in (1, 3, 4, 5, steps):
        rhs = torch.zeros(k + 1, 1, dtype=torch.float64, device="cuda")
        rhs[0] = beta
        y = torch.linalg.lstsq(H[:k + 1, :k], rhs).solution
        res = float((H[:k + 1, :k] @ y - rhs).norm())
        if res <= 1e-15 * float(beta):  # solved to the tolerance asked for: there is no further iterate
            break
        want = (Z[:k, :n].T @ y)[:, 0]
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        q = s.solve(x, b, rel_tol=1e-15, max_iterations=k, raise_on_failure=False)
        assert q["iterations"] == k
        assert abs(q["initial_residual"] - float(beta)) < 1e-12 * float(beta)
        assert abs(q["final_residual"] - res) < 1e-9 * float(beta)
        assert float((x - want).norm() / want.norm()) < 1e-8
        # stopped by the tolerance at the same iteration
        x.zero_()
        q = s.solve(x, b, rel_tol=1.0001 * res / float(beta), max_iterations=steps)
        assert q["iterations"] == k


@pytest.mark.parametrize("restart", [1, 2, 3, 5])
def test_short_restarts_never_lose_ground(restart):
    """Each cycle minimises the residual from where the last one ended: the true residual, by the
    operator's own apply, is what the solver reports (1e-10 of |b|) and does not grow with the cap."""
    from atmospheric_flows_b200.operator import EULEROperator
    from atmospheric_flows_b200.schur import SchurSolver
    P, sc = 4, M.Scaling()
    m = M.hill_mesh(40, 26, periodic_x=True)
    st = M.hill_state(m, P, modes=4)
    op = EULEROperator(m, P, sc.Ma, sc.Fr, 0.25)
    op.set_stream(torch.cuda.current_stream())
    op.set_schur_mode(1)
    op.set_HYPERBOLIC_stage(1)
    op.set_rho_for_fixed(torch.from_numpy(st.rho).cuda())
    op.set_pres_fixed(torch.from_numpy(st.p).cuda())
    b = torch.from_numpy(np.random.default_rng(7).standard_normal(op.n_dofs(1))).cuda()
    s = SchurSolver(op, "jacobi", restart=restart)
    s.setup()
    last = float(b.norm())
    for cap in (1, 2, 4, 7, 12, 20):
        x, r = torch.zeros_like(b), torch.empty_like(b)
        q = s.solve(x, b, rel_tol=1e-10, max_iterations=cap, raise_on_failure=False)
        op.set_NS_stage(2)
        op.vmult(r, x)
        true = float((b - r).norm())
        assert abs(true - q["final_residual"]) < 1e-10 * float(b.norm())
        assert true <= last * (1 + 1e-10)
        last = true
    assert last < float(b.norm())
