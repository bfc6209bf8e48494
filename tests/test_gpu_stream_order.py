"""What a GEMM sees of the kernels before it in its stream, without a synchronisation in between."""

import numpy as np
import pytest
import torch

import tuna_b200
from tests.gpu_util import make_case, stream_ptr
from tuna_b200 import _lib

pytestmark = pytest.mark.gpu

# Lets its dependents start at once, writes only some 50 us later.
LATE_WRITER = """
extern "C" __global__ void late_writer(unsigned char *dst, const unsigned char *src, int n, float *cdst, const float *csrc)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long t0 = clock64();
    while (clock64() - t0 < 100000) { }
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
    if (threadIdx.x < 16) cdst[threadIdx.x] = csrc[threadIdx.x];
}
"""


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("m,k,n", [(512, 256, 65), (520, 264, 100), (264, 96, 300), (256, 2048, 256)])
def test_weights_and_codebook_of_the_kernel_before(m, k, n, graph):
    """Above 64 tokens weights and codebook follow ordinary stream order, whatever the kernel before does about its dependents."""
    (x, q, absmax, code), (xd, qd, sd, cd) = make_case(m, n, k, seed=m + n)
    out, ref = (torch.empty((n, m), dtype=torch.float16, device="cuda") for _ in range(2))
    tuna_b200.matmul(xd, qd, sd, cd, ref, m, n, k)
    q2, c2 = torch.zeros_like(qd), torch.zeros_like(cd)
    writer = torch.cuda._compile_kernel(LATE_WRITER, "late_writer")

    def calls():
        writer(grid=(1, 1, 1), block=(256, 1, 1), args=[q2, qd, q2.numel(), c2, cd])
        tuna_b200.matmul(xd, q2, sd, c2, out, m, n, k)

    if graph:
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            tuna_b200.matmul(xd, qd, sd, cd, out, m, n, k)  # the stream's workspace
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                calls()
        calls = g.replay
    for _ in range(3):
        torch.cuda.synchronize()
        q2.zero_(), c2.zero_(), out.fill_(float("nan"))
        torch.cuda.synchronize()
        calls()
        torch.cuda.synchronize()
        assert torch.equal(out, ref)
    assert _lib.load().tuna_check_device_status(stream_ptr()) == 0
    assert np.isfinite(ref.float().cpu().numpy()).all()
