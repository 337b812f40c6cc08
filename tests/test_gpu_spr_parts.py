"""The linear-response solver over parts of a system (spr.cu, k_spr_res): one
part and many, parts with a last slice that is not full, every place its data
can live (all in shared memory; the matrix in global memory; the vectors too;
the kernel for systems beyond it), against a dense solve.

Bound: the solver stops at ||r|| <= 1e-12 ||b||, so the solution is off by at
most 1e-12 cond(K) relatively; these networks have cond(K) < 1e5."""
import numpy as np
import pytest

import network_relaxation_gb300 as nr

pytestmark = pytest.mark.gpu


def _dense(h, kb, mu, compr, shear):
    a = h.arrays()
    n = len(a["points"])
    r, c, v = nr.spr_assemble(h, 1.0, kb, mu)
    K = np.zeros((2 * n, 2 * n))
    K[r, c] = v
    K[c, r] = v
    y = a["points"][:, 1]
    lo, hi = y.min(), y.max()
    bc = np.zeros((n, 2))
    bc[:, 0] = shear * (y - lo) / (hi - lo)
    bc[:, 1] = compr * (lo - y) / (hi - lo)
    free = np.repeat((y >= lo + 1e-10) & (y <= hi - 1e-10), 2)
    u = bc.reshape(-1).copy()
    rhs = -(K @ u)[free]
    u[free] += np.linalg.solve(K[np.ix_(free, free)], rhs)
    return u.reshape(n, 2)


@pytest.mark.parametrize("smem", [None, 40000, 12000, 1])
@pytest.mark.parametrize("nx,ny", [(5, 4), (9, 8), (31, 29)])
def test_parts_match_dense_solve(cuda, monkeypatch, smem, nx, ny):
    if smem is not None:
        monkeypatch.setenv("NR_SPR_SMEM", str(smem))
    h = nr.HostNetwork.lattice(nx, ny, 0.85, 0.0, 7).get_triples()
    spr = nr.Spr(h, 1.0, 1e-2, 0.1)
    assert spr.solve(affine=True, tol=1e-12) == nr.NR_OK
    assert max(spr.info().rel_residual) <= 1e-12
    for compr, shear in ((0.02, 0.0), (-0.01, 0.03)):
        rec, u = spr.point(compr, shear)
        ref = _dense(h, 1e-2, 0.1, compr, shear)
        assert np.abs(u - ref).max() <= 1e-7 * np.abs(ref).max()
    first = spr.point(0.02, 0.01)[1].copy()
    spr.solve(affine=True, tol=1e-12)
    assert np.array_equal(first, spr.point(0.02, 0.01)[1])


def test_parts_iteration_limit(cuda):
    spr = nr.Spr(nr.HostNetwork.lattice(31, 29, 0.85, 0.0, 7).get_triples(), 1.0, 1e-2, 0.1)
    assert spr.solve(affine=True, tol=1e-12, max_iter=5) == nr.NR_NOT_CONVERGED
    assert list(spr.info().iterations) == [5, 5]
    assert spr.solve(affine=True, tol=1e-12, max_iter=0) == nr.NR_NOT_CONVERGED
