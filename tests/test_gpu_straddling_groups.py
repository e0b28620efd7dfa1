"""Groups that are odd multiples of 64 straddle the 128-k stages of the tensor-core kernels."""
import numpy as np
import pytest
import torch

from oracle import qf_oracle as O
from qfactory import QLinear

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2, 40, 130])
@pytest.mark.parametrize("GS", [192, 320])
def test_groups_that_straddle_stages(M, GS):
    x, q, s, z = O.make_case(M, 256, 4 * GS, 4, GS, False, seed=GS + M)
    layer = QLinear.init(M, 4 * GS, 256, 4, q.cuda(), GS, s.cuda(), z.cuda())
    y = layer(x.cuda())
    _, yex = O.reference_forward(x, q, s, z, 4)
    assert np.abs(y.float().cpu().numpy() - yex).max() <= 1e-2 * np.abs(yex).max()
