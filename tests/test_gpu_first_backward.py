"""A process whose first backward call finds all its memory cached: autograd's thread has made no CUDA call by then."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import torch
from natten_mps_b200 import _cabi, functional as F
def t(*s): return torch.randn(*s, device="cuda").to(torch.float16).requires_grad_(True)
q, k, v, do = t(2, 200, 4, 64), t(2, 200, 4, 64), t(2, 200, 4, 64), t(2, 200, 4, 64).detach()
_cabi.set_force("tc")
out = F.na1d(q, k, v, kernel_size=15)
torch.autograd.grad(out, [q, k, v], do)
print(_cabi.last_path())
"""


def test_first_backward_of_a_process_on_the_tensor_cores():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split()[-1] == "tcgen05", r.stderr[-2000:]
