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


def test_which_prompts_of_the_further_forms_take_the_tcgen05_kernel():
    """The rule's decisions at the sizes that were measured on both kernels (148 SMs)."""
    from llm_infer_rust_b200.kernels.ops import shaped_prompt_on_tcgen05

    def taken(tokens, nh, nkv, rows=1, cached=0, capped=False, limit=0):
        return shaped_prompt_on_tcgen05(tokens, nh // nkv, nkv, rows, cached + tokens, capped, 148, limit)
    for capped in (False, True):
        assert not taken(64, 16, 8, capped=capped) and not taken(64, 32, 8, capped=capped) and not taken(16, 16, 1, capped=capped)
        assert taken(128, 16, 8, capped=capped) and taken(2048, 16, 8, capped=capped) and taken(256, 16, 8, 4, capped=capped)
        assert taken(64, 32, 8, cached=2000, capped=capped) and taken(16, 16, 1, cached=300, capped=capped)
        assert not taken(64, 16, 8, cached=8000, capped=capped)             # one tile of query vectors a KV head
        assert not taken(128, 16, 8, 16, capped=capped) and not taken(200, 16, 8, 16, capped=capped)       # waves of one or two blocks
        assert taken(300, 16, 8, 4, capped=capped) and taken(512, 16, 8, 16, capped=capped)
    assert taken(300, 16, 8, 16) and not taken(300, 16, 8, 16, capped=True)
    assert taken(100, 32, 8) and taken(400, 32, 8, 16, capped=True) and not taken(400, 16, 8, 16, capped=True)
    # windows and blocks: a query that sees few keys leaves a CTA little behind its first block
    assert not taken(2000, 16, 8, limit=64 + 64) and not taken(1000, 16, 8, 8, limit=128 + 64) and not taken(1000, 16, 8, 8, limit=128)
    assert taken(2000, 16, 8, limit=128 + 64) and taken(200, 32, 8, 4, capped=True) and not taken(200, 16, 8, 8, capped=True)
    assert taken(500, 16, 8, limit=128) and taken(1000, 16, 8, 8, limit=512) and taken(2048, 16, 8, limit=1024)
