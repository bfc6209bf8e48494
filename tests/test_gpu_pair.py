"""The two-SM tcgen05 kernel at the edges of its tiles, stages and work split, against the oracle."""

import numpy as np
import pytest
import torch

from oracle import tuna_oracle as orc
from tuna_b200 import _lib
from tests.gpu_util import check_parity, make_case, run_matmul, stream_ptr

pytestmark = pytest.mark.gpu
TOL = 1e-2  # max relative error budget of the GEMM (fp32 accumulation on both sides)


def _run(m, n, k, seed=0, **cfgd):
    host, dev = make_case(m, n, k, seed)
    cfg = _lib.TunaConfig(path=_lib.PATH_UMMA, **cfgd)
    st, out, holder = run_matmul(dev, m, n, k, cfg=cfg)
    assert st == 0, _lib.load().tuna_status_string(st)
    assert _lib.load().tuna_check_device_status(stream_ptr()) == 0, "a bounded wait ran out"
    check_parity(out.cpu().numpy(), orc.matmul_ref(*host, m, n, k), TOL)
    assert holder.guards_intact()
    return out.cpu().numpy().view(np.uint16)


# token tiles of 32 .. 256, the last one full, ragged or a few tokens; stages of 64 and 128 columns
@pytest.mark.parametrize("n", [1, 33, 65, 96, 127, 130, 161, 200, 224, 255, 257, 300, 513])
def test_token_counts(n):
    _run(384, n, 320, seed=n)


# every token tile, two full ones and a remainder: 16 dequant warps and the wide table up to 192 tokens, 8 and the compact one above
@pytest.mark.parametrize("tile_tok", [32, 64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("m,k", [(512, 576), (264, 1000)])
def test_token_tiles(tile_tok, m, k):
    _run(m, 2 * tile_tok + 7, k, seed=tile_tok, tile_tok=tile_tok)


# short tiles (8 dequant warps) and long ones (16 up to 192 tokens), several per pair
@pytest.mark.parametrize("tile_tok", [32, 64, 96, 128, 160, 192, 224])
@pytest.mark.parametrize("k", [136, 640, 5128])
def test_short_and_long_tiles(tile_tok, k):
    _run(1032, tile_tok + 9, k, seed=tile_tok + k, tile_tok=tile_tok, ctas=6)


# few and many segments of a tile, added up in pieces of 8 and of 16 columns, with tokens and rows left over
@pytest.mark.parametrize("ctas", [4, 10, 34, 148])
@pytest.mark.parametrize("n,tile_tok", [(20, 32), (32, 32), (60, 64), (96, 96), (100, 64), (190, 192), (250, 256)])
def test_segments_of_cut_tiles(n, tile_tok, ctas):
    _run(264, n, 8200, seed=n + ctas, tile_tok=tile_tok, ctas=ctas)


# m and k of every weight view: 5-D runs, 3-D boxes (k % 32 == 0), 2-D boxes (any k); fewer rows than a tile, row remainders
@pytest.mark.parametrize("m,k", [(8, 8), (256, 64), (264, 96), (520, 136), (1032, 1000), (2048, 2112)])
@pytest.mark.parametrize("n", [70, 250])
def test_shapes(m, k, n):
    _run(m, n, k, seed=m + n)


# one pair walking several whole tiles; tiles cut over two, three and many pairs with and without whole waves before and after
@pytest.mark.parametrize("ctas", [2, 4, 6, 16, 148])
@pytest.mark.parametrize("m,n,k", [(1280, 600, 2048), (512, 100, 8192)])
def test_work_splits_are_deterministic(m, n, k, ctas):
    first = _run(m, n, k, seed=5, ctas=ctas)
    for _ in range(3):
        assert np.array_equal(first, _run(m, n, k, seed=5, ctas=ctas))


@pytest.mark.parametrize("m,k,n", [(2048, 512, 100), (512, 512, 200), (520, 264, 200)])
def test_one_hot_activations_reproduce_the_weights(m, k, n):
    """Row j of x selects column 7 j mod k: any permutation of rows, columns or tokens shows."""
    (x, q, absmax, code), dev = make_case(m, n, k, seed=9)
    x = np.zeros((n, k), dtype=np.float16)
    cols = (7 * np.arange(n)) % k
    x[np.arange(n), cols] = 1
    dev = (torch.from_numpy(x).cuda(),) + tuple(dev[1:])
    st, out, _ = run_matmul(dev, m, n, k, cfg=_lib.TunaConfig(path=_lib.PATH_UMMA))
    assert st == 0
    w = orc.dequant_ref(q, np.ones(m, np.float32), code, m, k).astype(np.float32)  # fp16 codes
    ref = (w[:, cols] * absmax[:, None]).astype(np.float16).T
    assert np.array_equal(out.cpu().numpy().view(np.uint16), ref.view(np.uint16))
