"""The device quantizer against the oracle (bit-exact) and the torch-CPU golden fixture."""

import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
import torch

import tuna_b200
from oracle import tuna_oracle as orc
from tests.gpu_util import check_parity

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).parent / "golden"


def _quantize_gpu(w: np.ndarray):
    q, (absmax, code) = tuna_b200.quantize(torch.from_numpy(w).cuda())
    torch.cuda.synchronize()
    return q.cpu().numpy(), absmax.cpu().numpy(), code.cpu().numpy()


def test_fixture_from_the_reference_expression():
    d = np.load(GOLDEN / "quantizer_torch_cpu.npz")
    q, absmax, _ = _quantize_gpu(d["w_bits"].view(np.float16).copy())
    assert np.array_equal(absmax, d["absmax"])
    assert np.array_equal(q, d["q"])


@pytest.mark.parametrize("m,k", [(16, 8), (64, 256), (136, 80), (1024, 4096), (4096, 1000)])
def test_bit_exact_against_the_oracle(m, k):
    rng = np.random.default_rng(m * 131 + k)
    w = (rng.standard_normal((m, k)) * 0.05).astype(np.float16)
    w[m // 2] = 0
    q, absmax, _ = _quantize_gpu(w)
    q_ref, a_ref, _ = orc.quantize_blockwise_dynamic_4bit(w)
    assert np.array_equal(absmax, a_ref)
    assert np.array_equal(q, q_ref)


def test_quantize_then_matmul_matches_the_fp16_product():
    # the reference's own smoke check (test.py:81-88): quantized GEMM next to x @ w.T
    m, n, k = 2048, 16, 4096
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((n, k), device="cuda", generator=g).half() * 0.1
    w = torch.randn((m, k), device="cuda", generator=g).half() * 0.05
    q, (absmax, code) = tuna_b200.quantize(w)
    out = torch.empty((n, m), dtype=torch.float16, device="cuda")
    tuna_b200.matmul(x, q, absmax, code, out, m, n, k)
    torch.cuda.synchronize()
    # exact check against the oracle on the quantized weights ...
    ref = orc.matmul_ref(x.cpu().numpy(), q.cpu().numpy(), absmax.cpu().numpy(), code.cpu().numpy(), m, n, k)
    check_parity(out.cpu().numpy(), ref, 1e-2)
    # ... and the quantization error itself stays at the 4-bit level
    dense = (x.float() @ w.float().t()).cpu().numpy()
    rel = np.abs(out.cpu().numpy().astype(np.float32) - dense).max() / np.abs(dense).max()
    assert rel < 0.15


def test_rejects_bad_arguments():
    with pytest.raises(ValueError):
        tuna_b200.quantize(torch.zeros((8, 8), dtype=torch.float32, device="cuda"))
    with pytest.raises(tuna_b200.TunaError):
        tuna_b200.quantize(torch.zeros((12, 8), dtype=torch.float16, device="cuda"))


# one CTA per row group up to 4096 columns, clusters above, the two-pass kernels beyond 111488; rows of every kind
@pytest.mark.parametrize("m,k", [(16, 8), (32, 4088), (16, 4096), (16, 4104), (48, 10008), (8, 28672), (16, 32776), (16, 111488), (16, 111496), (8, 112000), (16, 112008)])
@pytest.mark.parametrize("book", ["nf4", "unsorted", "close", "duplicate"])
def test_every_share_and_codebook_is_bit_exact(m, k, book):
    rng = np.random.default_rng(m + k)
    w = (rng.standard_normal((m, k)) * 0.05).astype(np.float16)
    w[1] = 0
    w[2] *= np.float16(1e-3)           # 63 / absmax overflows fp16: the literal expression
    w[3] = rng.integers(-8, 9, k) / 8  # exact midpoints and end points
    w[4, 0] = 60000
    w[5, k - 1] = np.float16(-6e-8)
    code = orc.NF4_CODE.copy()
    if book == "unsorted":             # sign-magnitude order
        code = np.array([0.01, 0.1, 0.2, 0.3, 0.45, 0.6, 0.8, 1, -0.02, -0.1, -0.2, -0.3, -0.45, -0.6, -0.8, -1.5], dtype=np.float32)
    elif book == "close":              # two thresholds in one bucket
        code[8] = 0.001
    elif book == "duplicate":
        code[8] = 0.0
    q, (absmax, c) = tuna_b200.quantize(torch.from_numpy(w).cuda(), None if book == "nf4" else torch.from_numpy(code).cuda())
    q_ref, a_ref, _ = orc.quantize_blockwise_dynamic_4bit(w, code)
    assert np.array_equal(c.cpu().numpy(), code)
    assert np.array_equal(absmax.cpu().numpy(), a_ref)
    assert np.array_equal(q.cpu().numpy(), q_ref)


# two thresholds in one of 64 buckets but not in one of 128, in one of 128 only, in one of either
@pytest.mark.parametrize("codes", [(0.0, 0.04, 0.05), (0.0, 0.021, 0.0213), (0.04, 0.0402, 0.0404)])
@pytest.mark.parametrize("m,k", [(16, 1000), (16, 4104)])
def test_codes_whose_thresholds_share_buckets(codes, m, k):
    w = (np.random.default_rng(k).standard_normal((m, k)) * 0.05).astype(np.float16)
    w[1, : k // 2] = (np.arange(k // 2) / 2048).astype(np.float16)
    w[1, 0] = 1
    code = orc.NF4_CODE.copy()
    code[7:10] = codes
    q, (absmax, _) = tuna_b200.quantize(torch.from_numpy(w).cuda(), torch.from_numpy(code).cuda())
    q_ref, a_ref, _ = orc.quantize_blockwise_dynamic_4bit(w, code)
    assert np.array_equal(absmax.cpu().numpy(), a_ref)
    assert np.array_equal(q.cpu().numpy(), q_ref)


@pytest.mark.parametrize("m,k", [(2048, 8), (4096, 8), (4096, 64), (4096, 136), (8192, 128), (8192, 256)])
@pytest.mark.parametrize("book", ["nf4", "unsorted"])
def test_narrow_rows_on_both_sides_of_the_two_pass_line(m, k, book):
    rng = np.random.default_rng(m + k)
    w = (rng.standard_normal((m, k)) * 0.05).astype(np.float16)
    w[1] = 0
    w[2] *= np.float16(1e-3)
    w[3] = rng.integers(-8, 9, k) / 8
    code = orc.NF4_CODE if book == "nf4" else np.ascontiguousarray(np.roll(orc.NF4_CODE, 5))
    q, (absmax, c) = tuna_b200.quantize(torch.from_numpy(w).cuda(), None if book == "nf4" else torch.from_numpy(code).cuda())
    q_ref, a_ref, _ = orc.quantize_blockwise_dynamic_4bit(w, code)
    assert np.array_equal(c.cpu().numpy(), code)
    assert np.array_equal(absmax.cpu().numpy(), a_ref)
    assert np.array_equal(q.cpu().numpy(), q_ref)


def test_widest_single_pass_rows():
    """The widest rows whose staged share and tables fit a CTA of the largest cluster; 8 columns more take two passes."""
    for k in (111488, 111496):
        w = (np.random.default_rng(k).standard_normal((16, k)) * 0.05).astype(np.float16)
        q, (absmax, _) = tuna_b200.quantize(torch.from_numpy(w).cuda())
        q_ref, a_ref, _ = orc.quantize_blockwise_dynamic_4bit(w)
        assert np.array_equal(absmax.cpu().numpy(), a_ref)
        assert np.array_equal(q.cpu().numpy(), q_ref)


FIRST_CALL_CAPTURED = """
import numpy as np, torch, tuna_b200
from oracle import tuna_oracle as orc
w = (np.random.default_rng(5).standard_normal((64, 4104)) * 0.05).astype(np.float16)
wd, code = torch.zeros(w.shape, dtype=torch.float16, device="cuda"), torch.from_numpy(orc.NF4_CODE).cuda()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    q, (absmax, c) = tuna_b200.quantize(wd, {codebook})
wd.copy_(torch.from_numpy(w))
g.replay()
q_ref, a_ref, _ = orc.quantize_blockwise_dynamic_4bit(w)
assert np.array_equal(q.cpu().numpy(), q_ref) and np.array_equal(absmax.cpu().numpy(), a_ref)
assert np.array_equal(c.cpu().numpy(), orc.NF4_CODE)
assert tuna_b200._lib.load().tuna_check_device_status(torch.cuda.current_stream().cuda_stream) == 0
"""


@pytest.mark.parametrize("codebook", ["None", "code"])
def test_first_call_of_a_process_can_be_captured(codebook):
    r = subprocess.run([sys.executable, "-c", FIRST_CALL_CAPTURED.format(codebook=codebook)], capture_output=True, text=True, timeout=300,
                       cwd=GOLDEN.parents[1])
    assert r.returncode == 0, r.stderr[-2000:]
