"""Loading of the native host module (no GPU needed)."""
import subprocess
import sys
import textwrap

import pytest
import torch

from nanopysche_b200 import build
from nanopysche_b200.ops import _lib

built = pytest.mark.skipif(not (_lib.LIB_PATH.exists() and build.HOST_PATH.exists()), reason="the library is not built here")


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
