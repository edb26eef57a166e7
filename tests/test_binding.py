"""The Python binding of the products (host code; no GPU needed): what tensors throw comes back as a Python exception."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# in a process of its own: an exception that leaves the binding ends the process
CALL = """
import torch
from mask_b200 import _lib
spmm = _lib.binding().spmm
def call(ids):
    return spmm(0, 16, 16, ids, None, None, None, 0, torch.zeros(16, 16), None, 0, True)
try:
    {}
except RuntimeError as e:
    print("RuntimeError:", str(e).splitlines()[0])
"""


@pytest.mark.parametrize("make", ["call(torch.zeros(16, 16).to_sparse())", "torch.func.vmap(call)(torch.zeros(3, 16, dtype=torch.int32))"])
def test_tensors_without_an_address_raise(make):
    r = subprocess.run([sys.executable, "-c", CALL.format(make)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-500:]
    assert r.stdout.startswith("RuntimeError:"), (r.stdout, r.stderr[-500:])


def test_host_tensors_are_refused():
    import torch
    from mask_b200 import _lib
    with pytest.raises(RuntimeError, match="dense must be a CUDA tensor"):
        _lib.binding().spmm(0, 16, 16, None, None, None, None, 0, torch.zeros(16, 16), None, 0, True)
    with pytest.raises(RuntimeError, match="12 arguments"):
        _lib.binding().spmm(0)
