"""Device memory that an FP32 search of many rows takes for its partial lists:
one list per row and a block of them per resident CTA, not two per row."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import torch
from manifoldann_gb300 import _lib
lib = _lib.load()
k, nq, n, d = 128, 100_000, 3_000, 8
x, q = torch.rand((n, d), device="cuda"), torch.rand((nq, d), device="cuda")
ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
dist = torch.empty((nq, k), device="cuda")
def search(rows):
    _lib.check(lib.mann_knn_device(_lib.params(1, k, 0), x.data_ptr(), n, q.data_ptr(), rows, d, ids.data_ptr(),
                                   dist.data_ptr(), None, None))
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
before = search(100)
print("taken", before - search(nq))
"""


def test_partial_lists_of_many_rows(gpu_lib):
    out = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    taken = int(out.stdout.split("taken")[1])
    one = 100_000 * 128 * 8
    # 304 CTAs of 64 rows more, allocations of 2 MB
    assert one <= taken + (64 << 20) and taken <= one + 304 * 64 * 128 * 8 + (8 << 20), taken
