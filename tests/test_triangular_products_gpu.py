"""The FP64 products that use a triangle or a symmetry (R3 R2 R1 of the QR stage,
V^T V of the mixed engine's re-orthogonalisation), at widths of one to six
64-column tiles with and without a remainder.

A wrong or missing tile in R shows in U S V^T - A, one in V^T V in
V^T V - I.  Both to 1e-12 n, the orthogonality bound of the path's other
tests (a reconstruction is off by at most the factors' departures).
"""
import numpy as np
import pytest

import jsvd
import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["precond", "mixed"])
@pytest.mark.parametrize("n", [63, 64, 65, 128, 193, 321])
def test_factors_at_tile_edges(engine, n):
    m = n + 70
    a = workloads.spectrum_matrix(m, n, workloads.geometric_sigma(n, 1e-4), n)
    r = jsvd.svd(a, engine, jsvd.default_config(epsilon=1e-14))
    for x in (r.u, r.v):
        assert np.linalg.norm(x.T @ x - np.eye(n)) <= 1e-12 * n
    assert np.linalg.norm((r.u * r.sigma) @ r.v.T - a) <= 1e-12 * n * r.sigma[0]
