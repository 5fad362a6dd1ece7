"""The native host path takes torch's tensors apart with the code of the headers that it was compiled with: it serves no other
torch, and is compiled anew for one."""
import torch

from shflbw_sparse_nn_b200 import _cabi, build


def test_native_calls_serve_the_torch_they_were_compiled_for(monkeypatch):
    build.build_native()
    assert build.native_is_current(str(torch.__version__))
    assert not build.native_is_current("0.0.0") and not build.native_is_current(str(torch.__version__)[:-1])
    monkeypatch.setattr(_cabi, "_native_of", None)           # bound anew
    monkeypatch.setattr(_cabi, "_native", None)
    assert _cabi.native() is not None
    monkeypatch.setattr(_cabi, "_native_of", None)
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert _cabi.native() is None                            # ctypes and the modules' Python code run
