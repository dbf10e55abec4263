"""The native host module's file and its loading: one per torch and interpreter, from several threads at once (no GPU needed)."""
import subprocess
import sys
import textwrap
import types

import pytest
import torch

from nanopysche_b200 import build
from nanopysche_b200.ops import _lib

built = pytest.mark.skipif(not (_lib.LIB_PATH.exists() and build.host_path().exists()), reason="the library is not built here")


def test_the_file_belongs_to_one_torch_and_interpreter(monkeypatch):
    import sysconfig

    here = build.host_path()
    assert torch.__version__ in here.name and sysconfig.get_config_var("SOABI") in here.name
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert build.host_path() != here


@built
def test_the_kernel_library_does_not_need_it(monkeypatch):
    monkeypatch.setattr(build, "host_path", lambda: _lib.LIB_PATH.with_name("absent.so"))
    monkeypatch.setattr(build, "build_extension", lambda *a: pytest.fail("built"))
    monkeypatch.setattr(_lib, "_LIB", None)
    assert _lib.lib().np_sumsq_parts() > 0


@built
def test_a_module_that_does_not_load_is_named_with_the_command(monkeypatch, tmp_path):
    bad = tmp_path / "npb200_host.other.so"
    bad.write_bytes(b"not a library")
    monkeypatch.setattr(build, "host_path", lambda: bad)
    monkeypatch.setattr(_lib, "_HOST", None)
    with pytest.raises(_lib.KernelError, match="npb200_host.other.so.*python -m nanopysche_b200.build"):
        _lib.host()
    made = types.SimpleNamespace(done=0)
    monkeypatch.setattr(build, "host_path", lambda: tmp_path / "absent.so")
    monkeypatch.setattr(build, "build_host", lambda: setattr(made, "done", 1))
    with pytest.raises(_lib.KernelError):
        _lib.host()
    assert made.done == 1


@built
@pytest.mark.skipif(not hasattr(torch._C, "_cuda_getCurrentRawStream"), reason="a torch without CUDA never loads it")
def test_several_threads_may_load_it():
    code = textwrap.dedent("""
        import sys, threading
        from nanopysche_b200.ops import _lib
        sys.setswitchinterval(1e-6)
        gate, got = threading.Barrier(8), []
        def load():
            gate.wait()
            try:
                got.append(_lib.host())
            except Exception as e:
                got.append(e)
        ts = [threading.Thread(target=load) for _ in range(8)]
        [t.start() for t in ts], [t.join() for t in ts]
        assert len({id(g) for g in got}) == 1 and hasattr(got[0], "linear"), got
    """)
    for _ in range(3):
        p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True)
        assert p.returncode == 0, p.stderr[-2000:]
