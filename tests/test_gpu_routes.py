"""tuna_matmul without a configuration on both sides of the lines where its kernel, tile and split change: uncut tiles,
whole segments per tile, tiles cut anywhere; ragged rows and columns."""

import ctypes

import pytest
import torch

from oracle import tuna_oracle as orc
from tests.gpu_util import check_parity, make_case, run_matmul, stream_ptr
from tuna_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 16, 17, 32, 33, 64, 65, 129])
@pytest.mark.parametrize("m,k", [(8, 8), (136, 136), (512, 128), (520, 2048), (4104, 1032), (1024, 8192), (18952, 264)])
def test_default_route_matches_the_oracle(m, k, n):
    host, dev = make_case(m, n, k, seed=m + n)
    st, out, holder = run_matmul(dev, m, n, k)
    assert st == 0
    assert _lib.load().tuna_check_device_status(stream_ptr()) == 0, "a bounded wait ran out"
    check_parity(out.cpu().numpy(), orc.matmul_ref(*host, m, n, k), 1e-2)
    assert holder.guards_intact()


@pytest.mark.parametrize("m,k,n", [(520, 2048, 20), (520, 2048, 43), (512, 512, 100), (4104, 1032, 200), (1024, 8192, 300)])
def test_looked_up_configuration_gives_the_same_bits(m, k, n):
    _, dev = make_case(m, n, k, seed=3)
    cfg = _lib.TunaConfig()
    assert _lib.load().tuna_lookup_config(m, n, k, ctypes.byref(cfg)) == 0
    st0, by_default, _ = run_matmul(dev, m, n, k)
    st1, by_config, _ = run_matmul(dev, m, n, k, cfg=cfg)
    assert st0 == 0 and st1 == 0
    assert torch.equal(by_default, by_config)


# cut tiles that are added up by four tokens (more than four segments, one round of the CTA's warps) and by eight, with a last group alone
@pytest.mark.parametrize("m,n,k", [(640, 12, 1408), (1152, 11, 3328), (1792, 12, 4224), (888, 2, 8104), (4096, 16, 4096), (2688, 18, 7296), (768, 15, 2304)])
def test_cut_tiles_added_up_by_four_and_by_eight_tokens(m, n, k):
    host, dev = make_case(m, n, k, seed=m + n)
    st, out, holder = run_matmul(dev, m, n, k)
    assert st == 0
    check_parity(out.cpu().numpy(), orc.matmul_ref(*host, m, n, k), 1e-2)
    assert holder.guards_intact()
    again = run_matmul(dev, m, n, k)[1]
    assert torch.equal(out, again)
