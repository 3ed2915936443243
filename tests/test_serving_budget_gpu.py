"""The memory that a resident trajectory takes of a server's budget: its
coordinates and node grids (34 bytes a frame at d = 3), which leaves room for its
jobs in a budget of 46 bytes a frame."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,m", [(40, 3000), (12, 10000)])
def test_jobs_fit_beside_a_resident_trajectory(N, m):
    from netsci_gb300 import serving, synthetic
    X, _ = synthetic.protein_trajectory(N, m, seed=3)
    with serving.Server(budget_bytes=46 * N * m, max_m=16384) as srv:
        t = srv.register_trajectory(X, 3)
        gc = srv.wait(srv.submit_gc(t, N, 6), timeout=20.0)
    assert gc.shape == (N * (N - 1) // 2,) and np.isfinite(gc).all()
