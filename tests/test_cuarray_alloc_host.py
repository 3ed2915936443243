"""A deep copy whose allocation fails leaves the array as it was: its storage,
and what it knows of that storage's size (init() to the same size keeps it)."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.usefixtures("nsg_lib")
ROOT = Path(__file__).resolve().parent.parent

CHILD = """
import resource
import numpy as np
from netsci_gb300 import cuarray

rows, cols = 1000, 3000  # 12 MB: below the size of page-locked storage
big, small = cuarray.FloatCuArray(), cuarray.FloatCuArray()
big.fromNumpy2D(np.full((rows, cols), 2.0, np.float32))
values = np.arange(6, dtype=np.float32).reshape(2, 3)
small.fromNumpy2D(values)
soft, hard = resource.getrlimit(resource.RLIMIT_AS)
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (2 << 20), hard))
try:
    small.fromCuArray(big, 0, rows - 1, rows, cols)
    failed = ""
except Exception as e:
    failed = str(e)
finally:
    resource.setrlimit(resource.RLIMIT_AS, (soft, hard))
assert "alloc" in failed, failed
assert np.array_equal(small.toNumpy2D(), values)
small.init(rows, cols)
assert not small.toNumpy2D().any()
assert (big.toNumpy2D() == 2.0).all()
print("ok")
"""


def test_failed_deep_copy_leaves_the_array(tmp_path):
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr[-2000:])
