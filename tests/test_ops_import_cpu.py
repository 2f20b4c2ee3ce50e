"""The operator module with a torch that was built without CUDA."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_import_without_cuda_bindings():
    code = ("import torch\n"
            "for name in [n for n in dir(torch._C) if n.startswith('_cuda_')]: delattr(torch._C, name)\n"
            "from insignia_b200 import ops\n"
            "assert ops.PRO['plain'] == 0\n"
            "torch.cuda.current_stream = lambda: type('Stream', (), {'cuda_stream': 77})\n"
            "assert ops._stream() == 77\n")
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
