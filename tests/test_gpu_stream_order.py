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


# (m, n, k) of GEMMs that each read their activations from the output before: both sides of every change of kernel, tiles cut
# along K and uncut ones
CHAIN = [(2048, 300, 512), (4096, 16, 4096), (11000, 43, 1024), (768, 16, 4096), (520, 8, 1536), (4096, 1, 4096), (8192, 100, 40), (1032, 65, 8192),
         (4096, 24, 2048), (2048, 25, 3072), (512, 129, 264)]


class Chain:
    def __init__(self):
        lib = _lib.load()
        self.steps = []
        need = 0
        gen = torch.Generator(device="cuda").manual_seed(11)
        for i, (m, n, k) in enumerate(CHAIN):
            _, (x, q, s, c) = make_case(m, n, k, seed=40 + i)
            s = s * (8.0 / k ** 0.5) / s.mean() / 4  # outputs of the size of the inputs
            self.steps.append((m, n, k, q, s.contiguous(), c, torch.empty((n, m), dtype=torch.float16, device="cuda")))
            self.x = x if i == 0 else self.x
            need = max(need, lib.tuna_matmul_workspace_bytes(m, n, k))
        last = self.steps[-1][-1]
        self.w = torch.randn((1024, 2048), device="cuda", generator=gen).half() * 2048 ** -0.5
        self.o_quantized = torch.empty((32, 1024), dtype=torch.float16, device="cuda")
        self.x_quantized = last.view(-1)[:32 * 2048].view(32, 2048)
        m, n, k = 256, 16, 512
        per = [make_case(m, n, k, seed=70 + i)[1] for i in range(4)]
        self.q4, self.s4 = torch.stack([p[1] for p in per]), torch.stack([p[2] for p in per])
        self.o4 = torch.empty((4, n, m), dtype=torch.float16, device="cuda")
        self.x4 = self.o_quantized.view(-1)[:4 * n * k].view(4, n, k)
        self.code = per[0][3]
        self.seq_out = [torch.empty((t, 512), dtype=torch.float16, device="cuda") for t in (9, 70, 33)]
        weights = [make_case(512, 16, 64, seed=90 + i)[1] for i in range(3)]
        flat, first, gemms = self.o4.view(-1), 0, []
        for out, (_, q, s, c) in zip(self.seq_out, weights):
            t = out.shape[0]
            gemms.append((flat[first:first + t * 64].view(t, 64), q, s, out, 512, t, 64))
            first += t * 64
        self.ws = torch.zeros(max(need, 64 << 20), dtype=torch.uint8, device="cuda")  # one workspace for all of them
        self.seq = tuna_b200.MatmulSequence(gemms, self.code, workspace=self.ws)

    def outputs(self):
        return [st[-1] for st in self.steps] + [self.o_quantized, self.o4] + self.seq_out

    def run(self, between=lambda: None):
        x = self.x
        for m, n, k, q, s, c, o in self.steps:
            tuna_b200.matmul(x.view(-1)[:n * k].view(n, k), q, s, c, o, m, n, k, workspace=self.ws)
            between()
            x = o
        q, (absmax, code) = tuna_b200.quantize(self.w)  # weights, scales and codebook of the next call
        between()
        tuna_b200.matmul(self.x_quantized, q, absmax, code, self.o_quantized, 1024, 32, 2048, workspace=self.ws)
        between()
        tuna_b200.matmul_batched(self.x4, self.q4, self.s4, self.code, self.o4, 256, 16, 512, workspace=self.ws)
        between()
        self.seq.run()
        between()


def test_chain_of_dependent_calls_on_one_workspace():
    """Calls that follow one another without a synchronisation, each reading what the one before wrote: the same bits as with one."""
    chain = Chain()
    for m, n, k in CHAIN[1:]:
        i = CHAIN.index((m, n, k))
        assert n * k <= CHAIN[i - 1][0] * CHAIN[i - 1][1]  # the output before holds that many activations
    chain.run(torch.cuda.synchronize)
    ref = [o.clone() for o in chain.outputs()]
    for o in ref:
        assert torch.isfinite(o).all() and float(o.float().std()) > 1e-3

    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            chain.run()
            chain.run()
    for run in (chain.run, lambda: (chain.run(), chain.run()), g.replay):
        for _ in range(5):
            torch.cuda.synchronize()
            for o in chain.outputs():
                o.fill_(float("nan"))
            run()
            torch.cuda.synchronize()
            for o, r in zip(chain.outputs(), ref):
                assert torch.equal(o, r)
    assert _lib.load().tuna_check_device_status(stream_ptr()) == 0
    assert int(chain.ws[_lib.load().tuna_workspace_scratch_bytes():].sum()) == 0


# Takes SMs away for a while: its shared memory leaves no room for another CTA beside it.
OCCUPIER = """
extern "C" __global__ void occupier(long long *out, int clocks)
{
    extern __shared__ unsigned char smem[];
    const long long t0 = clock64();
    while (clock64() - t0 < clocks) { }
    if (threadIdx.x == 0) { smem[0] = 1; out[blockIdx.x] = clock64() - t0 + smem[0]; }
}
"""


def _late_start_calls(kind):
    if kind == "sequence" or kind == "reduce":
        shapes = [(1032, 8, 520), (520, 16, 2048), (264, 5, 1000), (1024, 16, 512)] * 6
    else:
        shapes = [(4096, 16, 4096), (520, 3, 8192), (1024, 24, 2048), (2048, 50, 1024), (512, 200, 4096)]
    gemms = []
    for i, (m, n, k) in enumerate(shapes):
        _, (x, q, s, c) = make_case(m, n, k, seed=200 + i)
        gemms.append((x, q, s, torch.empty((n, m), dtype=torch.float16, device="cuda"), m, n, k))
    if kind == "matmul":
        def run():
            for x, q, s, o, m, n, k in gemms:
                tuna_b200.matmul(x, q, s, c, o, m, n, k)
    elif kind == "sequence":
        run = tuna_b200.MatmulSequence(gemms, c).run
    else:
        exchange = tuna_b200.Exchange(tuna_b200.ReduceSequence.exchange_bytes([g[4:] for g in gemms], 1), "cuda:0")
        run = tuna_b200.ReduceSequence(gemms, c, exchange).run
    return run, [g[3] for g in gemms]


@pytest.mark.parametrize("kind", ["matmul", "sequence", "reduce"])
def test_ctas_that_start_late(kind):
    """With all but a few SMs taken, CTAs that share a tile run one after another instead of side by side, so the one that
    arrives last - and adds the partial sums up - is another one than usual: the same bits."""
    occupier = torch.cuda._compile_kernel(OCCUPIER, "occupier")
    occupier.set_shared_memory_config(200 << 10)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    times = torch.zeros(sms, dtype=torch.int64, device="cuda")
    work, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(work):
        run, outs = _late_start_calls(kind)
        run()
        torch.cuda.synchronize()
        ref = [o.clone() for o in outs]
        for free in (2, 10, 74):
            for o in outs:
                o.fill_(float("nan"))
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                occupier(grid=(sms - free, 1, 1), block=(32, 1, 1), args=[times, 1000000], shared_mem=200 << 10)
            run()
            torch.cuda.synchronize()
            for o, r in zip(outs, ref):
                assert torch.equal(o, r)
        assert _lib.load().tuna_check_device_status(work.cuda_stream) == 0
