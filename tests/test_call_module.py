"""The call module and the library that reads torch's tensors: the module loads without torch, the library belongs to one torch and is not taken
for another, a torch without CUDA (or one that nothing was built for) goes without."""
import subprocess
import sys
from types import SimpleNamespace

import pytest

from chatokf_b200 import _lib, build

ROOT = build.PKG.parent


def python(code):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return r.stdout


def test_the_module_links_against_nothing(lib_built):
    out = python(f"""
import importlib.util
spec = importlib.util.spec_from_file_location("_okfcall", {str(_lib.CALL_PATH)!r})
spec.loader.exec_module(importlib.util.module_from_spec(spec))
print([l for l in open("/proc/self/maps") if "libtorch" in l or "libc10" in l])
""")
    assert out.strip() == "[]"


@pytest.mark.parametrize("setting", ["torch.version.cuda = None", "torch.__version__ = '0.0.1'", "torch.version.git_version = 'another'"])
def test_without_a_library_for_this_torch(lib_built, setting):
    """The package loads, what needs no device works, and tensors are read by look-ups."""
    out = python(f"""
import torch
{setting}
from chatokf_b200 import _lib
lib = _lib.load()
assert lib.okf_row_bytes(8, 64) == 68
print([l for l in open("/proc/self/maps") if "_okftensor" in l])
from types import SimpleNamespace as N
from chatokf_b200.enc import GGUFTensor
from chatokf_b200.gguf_types import GGUFType
enc, w, t = N(ctx=N(_addr=0), stream=N(cuda_stream=0)), N(_addr=0), GGUFTensor("w", (64, 4), GGUFType.Q8_0)
x, out = torch.zeros(64), torch.zeros(4)
print(_lib.call.gemm(enc, 0, t, x, out, w, 1))  # no context: OKF_E_ARG
try:
    _lib.call.gemm(enc, 0, t, x.double(), out, w, 1)
except KeyError as e:
    print(e)
""")
    assert out.split() == ["[]", "-1", "torch.float64"]


def test_one_library_a_torch(lib_built, monkeypatch):
    import torch

    mine = _lib.tensor_path(torch)
    assert mine is not None and mine.exists() and not build.needs_build()
    version = SimpleNamespace(cuda=torch.version.cuda, git_version=torch.version.git_version)
    other = SimpleNamespace(__version__="9.9", version=version)
    assert _lib.tensor_path(other) not in (None, mine)
    assert _lib.tensor_path(SimpleNamespace(__version__=torch.__version__, version=SimpleNamespace(cuda=version.cuda, git_version="0" * 40))) not in (None, mine)
    assert _lib.tensor_path(SimpleNamespace(__version__=torch.__version__, version=SimpleNamespace(cuda=None, git_version=version.git_version))) is None
    monkeypatch.setattr(build, "_torch", lambda: other)
    assert build.needs_build()
    monkeypatch.setattr(build, "_torch", lambda: None)
    assert not build.needs_build()
