"""What the kernels do before their dependency wait.  A writer that releases its dependents at once and writes late (late_writer.cu)
stands for an engine's own kernel: everything but the weights that B200_OPT_STABLE_WEIGHTS covers must come out as it wrote it.  And
with that option on, every path gives the bits that it gives with the option off."""
import ctypes as C
import os
import subprocess
import numpy as np
import pytest
import torch

from util import pkg

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LATE_US = 300                                        # far longer than the host needs to enqueue the launches after the writer


def late_copy(dst, src):
    path = os.path.join(ROOT, 'tests', 'cpp', 'liblate_writer.so')
    if not os.path.exists(path):
        subprocess.check_call(['make', '-C', os.path.join(ROOT, 'glm-5.3-flash-cuda-server_b200'), 'gate'])
    f = C.CDLL(path).late_copy
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_uint, C.c_void_p]
    assert src.numel() * src.element_size() == dst.numel() * dst.element_size()
    assert f(dst.data_ptr(), src.data_ptr(), dst.numel() * dst.element_size(), LATE_US, torch.cuda.current_stream().cuda_stream) == 0


class stable_weights:
    def __enter__(self):
        pkg().set_option(pkg().OPT_STABLE_WEIGHTS, 1)

    def __exit__(self, *a):
        pkg().set_option(pkg().OPT_STABLE_WEIGHTS, 0)


@pytest.mark.parametrize('N,K,M', [(144, 4096, 1), (64, 2048, 4), (2048, 4096, 8)])
def test_a_bf16_matrix_is_no_stable_weight(N, K, M):
    """The option is a promise about NVFP4 weights.  A plain bf16 matrix written by the kernel before is read as it was written."""
    P = pkg()
    g = torch.Generator(device='cuda').manual_seed(N + M)
    old, new = [torch.randn((N, K), generator=g, device='cuda').to(torch.bfloat16) for _ in range(2)]
    x = torch.randn((M, K), generator=g, device='cuda')
    want = P.gemm(new, x)
    W, y = old.clone(), torch.empty_like(want)
    with stable_weights():
        for _ in range(5):
            W.copy_(old)
            P.gemm(W, x, y)
            late_copy(W, new)
            P.gemm(W, x, y)
            assert torch.equal(y, want)
