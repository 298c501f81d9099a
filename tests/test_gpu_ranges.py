"""Kernel variants at the edges of their ranges: the sizes where a launch changes shape, remainders of its
tiles, and the smallest and largest of what it takes, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import adamas_ref as ref
from test_gpu_parity import DEV, State, _assert_attn_close, _mods, _randn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hk", [(32, 32), (28, 4), (3, 1)])
@pytest.mark.parametrize("seq", [1, 2, 4735, 4737, 4739])   # several tokens per block from 4736 on, with remainders
def test_rope_token_groups(seq, hq, hk):
    _, K, U = _mods()
    q, k = _randn((seq, hq, 128), 1 + seq, torch.float16), _randn((seq, hk, 128), 2 + seq, torch.float16)
    qd, kd = q.to(DEV), k.to(DEV)
    U.apply_rope_in_place(qd, kd, 100, rope_scale=8.0)
    # the reference's tolerance for this operator (adamas/tests/test_rope.py:10-15)
    torch.testing.assert_close(qd.cpu().float(), ref.rope(q, 100, 8.0).float(), rtol=5e-3, atol=5e-3)
    torch.testing.assert_close(kd.cpu().float(), ref.rope(k, 100, 8.0).float(), rtol=5e-3, atol=5e-3)
