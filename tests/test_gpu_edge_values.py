"""Arguments and values at the edge of what the operators take."""
import pytest
import torch

from test_gpu_parity import DEV, _mods

pytestmark = pytest.mark.gpu


def test_flag_that_has_no_truth_value():
    """A flag that refuses to be a truth value raises its own error."""
    _, K, _ = _mods()
    x = torch.zeros(2, 128, dtype=torch.float16, device=DEV)
    with pytest.raises(RuntimeError, match="[Bb]oolean value"):
        K.hadamard_transform(x, inplace=torch.zeros(2))
