"""tuna_dequant where its work split can go wrong: row groups cut across warps, warps that walk several row groups,
passes that end inside a row; small matrices and narrow rows."""

import numpy as np
import pytest
import torch

from oracle import tuna_oracle as orc
from tests.gpu_util import Guarded, make_case, stream_ptr
from tuna_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(40000, 264), (8, 40008), (32, 8200), (33328, 256), (30016, 520),
                                 # both sides of the line between the two kernels, and the smallest and narrowest
                                 (8, 131072), (8, 131080), (32, 40008), (4096, 256), (4104, 256), (57344, 128), (57344, 136), (57344, 8), (8, 8), (520, 136)])
def test_dequant_work_split_is_exact(m, k):
    lib = _lib.load()
    (x, q, absmax, code), (xd, qd, sd, cd) = make_case(m, 1, k, seed=m + k)
    code[5], code[9] = -0.0, np.inf  # entries whose bit patterns have to survive
    cd = torch.from_numpy(code).cuda()
    out = Guarded(m * k * 2, torch.float16, (m, k))
    assert lib.tuna_dequant(qd.data_ptr(), sd.data_ptr(), cd.data_ptr(), out.view.data_ptr(), m, k, stream_ptr()) == 0
    torch.cuda.synchronize()
    ref = orc.dequant_ref(q, absmax, code, m, k)
    assert np.array_equal(out.view.cpu().numpy().view(np.uint16), ref.view(np.uint16))
    assert out.guards_intact()
