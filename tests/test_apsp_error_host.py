"""Results of a shortest-path call that fails are zeros, as fresh arrays are,
not what their storage held before. Without a CUDA device every solve fails
after its results were given their shape."""
import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.usefixtures("nsg_lib"),
              pytest.mark.skipif(torch.cuda.is_available(), reason="the solve would succeed")]


def _arrays(n, L):
    from netsci_gb300 import cuarray
    A, H, P = cuarray.FloatCuArray(), cuarray.FloatCuArray(), cuarray.IntCuArray()
    A.fromNumpy2D(np.ones((n, n), np.float32))
    H.fromNumpy2D(np.full((n, n), 7.0, np.float32))
    P.fromNumpy2D(np.full((1, n * L * n), 7, np.int32))
    return A, H, P


@pytest.mark.parametrize("entry", ["lengths", "paths", "all"])
@pytest.mark.parametrize("n", [3, 40])
def test_failed_solve_leaves_zeros(entry, n):
    from netsci_gb300 import netcalc
    L = 4
    A, H, P = _arrays(n, L)
    with pytest.raises(Exception):
        if entry == "lengths":
            netcalc.hedetniemiAllShortestPathLengthsGpu(A, H, L)
        elif entry == "paths":
            netcalc.hedetniemiAllShortestPathsGpu(A, H, P, 1e-4, L)
        else:
            netcalc.hedetniemiAllShortestPaths(A, H, P, L, 1e-4)
    assert not H.toNumpy2D().any()
    if entry != "lengths":
        assert P.toNumpy1D().shape == (n * L * n,) and not P.toNumpy1D().any()
    assert (A.toNumpy2D() == 1).all()
