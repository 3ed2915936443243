"""A CuArray initialised to the size it has keeps its storage: contents start
over, other sizes and other arrays are as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.usefixtures("nsg_lib")


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 5), (64, 1000)])
def test_same_size_starts_over(rows, cols):
    from netsci_gb300 import cuarray
    a, b = cuarray.FloatCuArray(), cuarray.FloatCuArray()
    values = np.arange(rows * cols, dtype=np.float32).reshape(rows, cols) + 1
    a.fromNumpy2D(values)
    b.fromNumpy2D(values)
    kept = np.array(a.toNumpy2D())
    a.init(rows, cols)
    assert not a.toNumpy2D().any()
    assert np.array_equal(kept, values) and np.array_equal(b.toNumpy2D(), values)
    a.fromNumpy2D(-values)
    assert np.array_equal(a.toNumpy2D(), -values)
    a.init(cols, rows + 1)
    assert (a.m(), a.n()) == (cols, rows + 1) and not a.toNumpy2D().any()
    a.init(rows, cols)
    assert (a.m(), a.n()) == (rows, cols) and not a.toNumpy2D().any()
