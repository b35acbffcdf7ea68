"""What the collectives' call path (src/python/fastcall.cpp) refuses before anything is launched.  No GPU is needed:
the checks come first.  The calls run in a process of their own, since a missing check ends the process."""
import json
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

# `t`: a tensor that claims to be on the GPU and has no memory.
RUNNER = """
import json, sys
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
import allreduce_proto_b200 as ar
from allreduce_proto_b200 import _native
fast = _native.fast()
host = torch.ones(8)
with FakeTensorMode():
    t, other = torch.ones(8, device="cuda:0"), torch.ones(8, device="cuda:1")
got = []
for call in json.loads(sys.argv[1]):
    try:
        eval(call)
        got.append("nothing")
    except Exception as e:
        got.append(type(e).__name__ + " " + str(e))
print(json.dumps(got))
"""


def outcomes(calls):
    """Per call, the exception that it ends with."""
    p = subprocess.run([sys.executable, "-c", RUNNER, json.dumps(calls)], cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.PIPE,
                       text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stderr[-2000:])
    return dict(zip(calls, json.loads(p.stdout.strip().splitlines()[-1])))


def test_host_tensors_are_refused():
    for call, got in outcomes([
        "ar.ops.copy_scale(host, host)",
        "fast.emu_allreduce(0, 2, [host] * 2, [host] * 2, 1, 1.0, -1, 0, None, 0)",
        "fast.emu_rsag(0, 2, 0, [host] * 2, [host[:4]] * 2, 1.0, 0)",
        "fast.allreduce(0, host, host, 1, 1.0, -1, None, 2)",
    ]).items():
        assert got == "IbcommError [ibcomm error 1] tensors must live on the GPU", (call, got)


def test_exceptions_of_torch_become_python_exceptions():
    # Without a driver there is no stream to be had; with one, the tensors' missing memory stops the call.
    for call, got in outcomes([
        "ar.ops.copy_scale(t, t)",
        "fast.emu_allreduce(0, 2, [t] * 2, [t] * 2, 1, 1.0, -1, 0, None, 0)",
        "fast.emu_rsag(0, 2, 0, [t] * 2, [t[:4]] * 2, 1.0, 0)",
        "fast.allreduce(0, t, t, 1, 1.0, -1, None, 2)",
    ]).items():
        assert got.split()[0] in ("RuntimeError", "AcceleratorError", "IbcommError"), (call, got)


def test_tensors_that_do_not_fit_are_refused():
    dst = "dst must hold every element of src, on the same GPU"
    ranks = "the ranks' tensors must match in dtype and live on one GPU"
    shorter = "every rank's tensors must match in dtype and hold as many elements as the first"
    blocks = "every rank's tensors must match in dtype and hold a block, or a block per rank"
    cases = {
        "ar.ops.copy_scale(t, t[:7])": dst,
        "ar.ops.copy_scale(t, other)": dst,
        "fast.allreduce(0, t, other, 1, 1.0, -1, None, 2)": "sendbuf and recvbuf must live on the same GPU",
        "fast.allreduce(0, t, t, 1, 1.0, -1, 0, 2)": "tensors must have memory",
        "fast.emu_allreduce(0, 2, [t, t[:7]], [t, t], 1, 1.0, -1, 0, None, 0)": shorter,
        "fast.emu_allreduce(0, 2, [t, t], [t, t[:7]], 1, 1.0, -1, 0, None, 0)": shorter,
        "fast.emu_allreduce(0, 2, [t, t], [t.half(), t.half()], 1, 1.0, -1, 0, None, 0)": shorter,
        "fast.emu_allreduce(0, 2, [t, t.half()], [t, t], 1, 1.0, -1, 0, None, 0)": ranks,
        "fast.emu_allreduce(0, 2, [t, other], [t, t], 1, 1.0, -1, 0, None, 0)": ranks,
        "fast.emu_rsag(0, 2, 0, [t, t[:7]], [t[:4], t[:4]], 1.0, 0)": blocks,
        "fast.emu_rsag(0, 2, 0, [t, t], [t[:4], t[:3]], 1.0, 0)": blocks,
        "fast.emu_rsag(0, 2, 1, [t[:4], t[:3]], [t, t], 1.0, 0)": blocks,
        "fast.emu_rsag(0, 2, 1, [t[:4], t[:4]], [t, t[:7]], 1.0, 0)": blocks,
        # Longer ones are taken, as prefixes: what stops this call is the handle.
        "fast.emu_allreduce(0, 2, [t[:7], t], [t, t], 1, 1.0, -1, 0, 0, 0)": "The handle is null",
    }
    for call, got in outcomes(list(cases)).items():
        assert got.startswith("IbcommError [ibcomm error 1] ") and cases[call] in got, (call, got)
