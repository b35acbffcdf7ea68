"""What the collectives' call path (src/python/fastcall.cpp) refuses before anything is launched.  No GPU is needed:
the checks come first.  Each snippet runs in a process of its own, since a missing check ends the process."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

PRELUDE = """
import torch
import allreduce_proto_b200 as ar
from allreduce_proto_b200 import _native
fast = _native.fast()
host = lambda n=8: torch.ones(n)
"""


def outcome(snippet):
    """Name of the exception that `snippet` ends with, and its text."""
    code = PRELUDE + "try:\n    " + snippet.replace("\n", "\n    ") + "\n    print('nothing')\nexcept Exception as e:\n    print(type(e).__name__, e)\n"
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.PIPE, text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stderr[-2000:])
    return p.stdout.strip()


@pytest.mark.parametrize("call", [
    "ar.ops.copy_scale(host(), host())",
    "fast.emu_allreduce(0, 2, [host()] * 2, [host()] * 2, 1, 1.0, -1, 0, None, 0)",
    "fast.emu_rsag(0, 2, 0, [host(16)] * 2, [host()] * 2, 1.0, 0)",
    "fast.allreduce(0, host(), host(), 1, 1.0, -1, None, 2)",
])
def test_host_tensors_are_refused(call):
    assert outcome(call) == "IbcommError [ibcomm error 1] tensors must live on the GPU"


FAKE = """from torch._subclasses.fake_tensor import FakeTensorMode
with FakeTensorMode():
    t = torch.ones(8, device="cuda")
    """


@pytest.mark.parametrize("call", [
    "ar.ops.copy_scale(t, t)",
    "fast.emu_allreduce(0, 2, [t] * 2, [t] * 2, 1, 1.0, -1, 0, None, 0)",
    "fast.emu_rsag(0, 2, 0, [t] * 2, [t] * 2, 1.0, 0)",
    "fast.allreduce(0, t, t, 1, 1.0, -1, None, 2)",
])
def test_exceptions_of_torch_become_python_exceptions(call):
    # A tensor that claims to be on the GPU and has no memory; without a driver its stream cannot be had either.
    assert outcome(FAKE + call).split()[0] in ("RuntimeError", "AcceleratorError", "IbcommError")
