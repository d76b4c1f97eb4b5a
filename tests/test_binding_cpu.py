"""Argument errors of the compiled binding that show without a GPU: fake CUDA tensors (a device, no memory) get a call as
far as the unwrapping of its arguments."""
import subprocess
import sys

from conftest import ROOT

PROGRAM = """
import sys
sys.path.insert(0, {root!r})
import numpy as np
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
import __graft_entry__ as entry

native = entry.load_package()._native()
with FakeTensorMode(allow_non_fake_inputs=True):
    x, strided = torch.empty(4, 64, device="cuda"), torch.empty(4, 2, device="cuda")[:, 0]
cpu = torch.zeros(4)
for call in {calls!r}:
    try:
        eval(call)
        print("no error")
    except BaseException as e:
        print(type(e).__name__)
"""


def errors(calls):
    """The exceptions of the calls, in a process of its own: what is tested for is an error in place of the process' end."""
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT, calls=calls)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-2000:])
    return r.stdout.split()


def test_four_six_rowwise_amax_error():
    """The amax is unwrapped, and refused, before the GIL is released."""
    calls = ["native.four_six_rowwise_f32(x, %s)" % amax for amax in ("cpu", "strided", "7")]
    assert errors(calls) == ["AssertionError", "AssertionError", "TypeError"]


def test_truth_value_error():
    """A flag without a truth value is an error, not a false."""
    calls = ["native.quantize_new(x, None, np.zeros(2), True, False)", "native.quantize_new(x, None, True, np.zeros(2), False)"]
    assert errors(calls) == ["ValueError", "ValueError"]


def test_binding_of_another_torch_or_python_is_another_file(pkg, monkeypatch):
    """The file the package loads is the one the build makes, and neither is taken over from another torch or Python."""
    import sysconfig

    import torch

    import __graft_entry__ as entry

    script = entry._load_build_script()
    assert script.binding_path() == pkg.BINDING_PATH
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0.1")
        assert script.binding_path() != pkg.BINDING_PATH
    with monkeypatch.context() as m:
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-00")
        assert script.binding_path() != pkg.BINDING_PATH
