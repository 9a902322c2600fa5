"""A launch that the CUDA runtime refuses is reported once, by the call that made it, and leaves no error behind for the
next launch to find."""
import ctypes

import pytest
import torch

import iris_b200 as iris
from iris_b200.ops import attention as A
from iris_b200.ops import elementwise as E
from iris_b200.ops import gemm as G
from iris_b200.utils.bench import memset_tensor

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)


def _bf16(*shape):
    return torch.randn(shape, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("call", ["rmsnorm", "attention", "gemm"])
def test_launch_that_would_join_a_capture(call):
    """On the legacy default stream while a stream that synchronises with it is being captured: refused by the runtime."""
    cudart = ctypes.CDLL([line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line][0])
    x, w = _bf16(4, 256), _bf16(256)
    qkv, out = _bf16(128, 384), _bf16(128, 128)
    flags = torch.zeros(8, dtype=torch.int32, device="cuda")
    ctx = iris.iris(64 << 20)
    op = G.gemm_all_scatter(ctx, [_bf16(64, 128)], [_bf16(256, 128)])
    assert op.local
    calls = {"rmsnorm": lambda: E.rmsnorm(x, w, x, stream=0),
             "attention": lambda: A.attention_fwd(qkv, out, 1, 128, 1, stream=0), "gemm": lambda: op(stream=0)}
    calls[call]()
    torch.cuda.synchronize()
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert cudart.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert cudart.cudaStreamBeginCapture(stream, 0) == 0
    try:
        with pytest.raises(RuntimeError):
            calls[call]()
    finally:
        cudart.cudaStreamEndCapture(stream, ctypes.byref(graph))
        cudart.cudaStreamDestroy(stream)
        cudart.cudaGetLastError()          # PyTorch's runtime is another instance than the library's
    memset_tensor(flags, 7)      # its launch check looks for the runtime's last error
    assert flags.tolist() == [7] * 8
    calls[call]()
    op.check()
    op.close(), ctx.close()
