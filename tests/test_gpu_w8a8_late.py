"""W8A8 linears that have started early behind a kernel that runs for longer than their own waits may take: the limit on a wait (2 s) counts from
the end of what came before, so nothing is reported and the result is the usual one."""
import ctypes
import subprocess

import pytest

from tests._util import capi
from tests.test_gpu_w8a8_split import on_device

pytestmark = pytest.mark.gpu

# one thread that lets its successors start at once and ends after `ns` nanoseconds
LATE = r"""
__global__ void late_kernel(unsigned long long ns)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do
    {
        __nanosleep(100000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    } while (t - t0 < ns);
}
extern "C" int late(unsigned long long ns, void* stream)
{
    late_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(ns);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def late(tmp_path_factory):
    top = tmp_path_factory.mktemp("late")
    (top / "late.cu").write_text(LATE)
    so = str(top / "late.so")
    subprocess.check_call(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "shared", "-Xcompiler", "-fPIC",
                           "-o", so, str(top / "late.cu")])
    f = ctypes.CDLL(so).late
    f.argtypes = [ctypes.c_ulonglong, ctypes.c_void_p]
    return f


# the pairs of one and of two feature tiles, the persistent ones, the k slices; with a scale that is given, and one that is found
@pytest.mark.parametrize("form", [1, 2, 3, 4])
@pytest.mark.parametrize("scale", [0.0, 0.02])
def test_a_late_predecessor_is_no_timeout(late, form, scale):
    import torch

    c, N, M, K = capi(), 1000, 100, 4096
    (W,), X = on_device([N], K, M)
    want, got = (torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert c.gemm_w8a8_bf16(W, 0.01, X, scale, want, N, M, K, flags=form << 8) == 0 and c.check_error("alone") == 0
    torch.cuda.synchronize()
    assert late(2_300_000_000, torch.cuda.current_stream().cuda_stream) == 0
    assert c.gemm_w8a8_bf16(W, 0.01, X, scale, got, N, M, K, flags=1 | form << 8) == 0
    assert c.check_error("late") == 0
    assert torch.equal(got, want) and want.abs().sum() > 0
