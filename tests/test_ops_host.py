"""The kernel wrappers where no GPU is."""
import subprocess
import sys


def test_the_wrappers_import_and_refuse_under_a_torch_without_cuda():
    """A torch built for the CPU has no CUDA names in its C module: the package imports all the same and says what is missing."""
    code = ("import torch\n"
            "for name in [n for n in dir(torch._C) if n.startswith('_cuda_')]:\n"
            "    delattr(torch._C, name)\n"
            "from llm_infer_rust_b200.kernels import ops\n"
            "try:\n"
            "    ops.rms_norm(torch.ones(2, 8), torch.ones(8), 1e-6)\n"
            "except ops.KernelError as e:\n"
            "    assert 'CUDA tensors only' in str(e)\n"
            "else:\n"
            "    raise SystemExit('accepted')\n")
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
