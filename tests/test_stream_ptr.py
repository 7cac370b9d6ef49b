"""A tensor that is not on a GPU meets torch's own error for the stream it lacks."""
import pytest
import torch

from lattica_b200.ntt import _stream_ptr


def test_cpu_tensor_error_is_torchs():
    t = torch.zeros(4, dtype=torch.int32)
    with pytest.raises(Exception) as want:
        torch.cuda.current_stream(t.device)
    with pytest.raises(type(want.value)) as got:
        _stream_ptr(t)
    assert str(got.value) == str(want.value)
