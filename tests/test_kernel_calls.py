"""The Python side of the kernel calls, without a GPU: importing before a build, and the two ways a call is made."""
import subprocess
import sys
from pathlib import Path

import pytest

from spbitnet_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent


def _run(code):
    return subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)


def test_import_needs_no_library():
    res = _run("import spbitnet_b200._lib as l, pathlib; l.LIB_PATH = pathlib.Path('/nonexistent/lib.so')\n"
               "import spbitnet_b200.kernels as K\n"
               "try:\n    K.softmax_gpu(1, 1, 1, 1, stream=0)\n"
               "except ImportError as e:\n    assert 'missing' in str(e)\n"
               "else:\n    raise AssertionError")
    assert res.returncode == 0, res.stderr


def test_import_needs_no_cuda_in_torch():
    """A torch without the CUDA symbols that look up the current stream: calls that name their stream still work."""
    res = _run("import torch\ndel torch._C._cuda_getCurrentRawStream\n"
               "import spbitnet_b200.kernels as K\nK.softmax_gpu(None, 0, 4, 4, stream=0)")
    assert res.returncode == 0, res.stderr


def _both():
    module, plain = _lib.calls(), _lib.CtypesCalls(_lib.load())
    return [pytest.param(c, id=type(c).__name__) for c in (module, plain)]


@pytest.mark.parametrize("calls", _both())
def test_conversion_and_errors(calls):
    calls.spb_softmax(None, 0, 4, 4, 0)  # nothing to do
    calls.spb_rms_norm(None, None, None, 0, 1e-5, 0)
    with pytest.raises(_lib.SpbError):
        calls.spb_softmax(None, 1, 4, 4, 0)
    with pytest.raises(_lib.SpbError):
        calls.spb_softmax(64, 1, 4, 5, 0)
    with pytest.raises(TypeError):
        calls.spb_softmax(None, 0, 4, 0)
    with pytest.raises((TypeError, AttributeError)):
        calls.spb_softmax("scores", 1, 4, 4, 0)
