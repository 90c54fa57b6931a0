"""The package imports, and reads the current stream, with a torch that has no raw reader of it (torch built without
CUDA, or one that names it otherwise)."""

import subprocess
import sys

from conftest import ROOT

SCENARIO = r'''
import sys
sys.path.insert(0, sys.argv[1])
import torch
if hasattr(torch._C, "_cuda_getCurrentRawStream"):
    del torch._C._cuda_getCurrentRawStream
from stdgpu_gb300 import containers, server
class stream:
    cuda_stream = 41
torch.cuda.current_device = lambda: 0
torch.cuda.current_stream = lambda device=None: stream
assert containers._stream(None) == 41 and containers._stream(stream) == 41
print("OK")
'''


def test_package_imports_without_the_raw_stream_reader():
    r = subprocess.run([sys.executable, "-c", SCENARIO, str(ROOT)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
