"""Host-side checks of the MLP's native calls: what would make a kernel read a
bad address is refused before any launch (no GPU needed: the tensors stay in
host memory, which is one of the things refused)."""
import pytest
import torch

from eulersr_b200.warmstart.mlp import MLP, _array


def _network(n):
    """An MLP whose flat vectors lie in host memory (its constructor wants a GPU)."""
    net = MLP.__new__(MLP)
    net.offsets, off = {}, 0
    for name, shape in MLP.SHAPES:
        net.offsets[name] = (off, shape)
        off += torch.Size(shape).numel()
    net.n_params = off
    net.p, net.pb, net.g = torch.zeros(n or off), torch.zeros(n or off, dtype=torch.bfloat16), torch.zeros(n or off)
    return net


def test_native_calls_refuse_host_tensors():
    net = _network(None)
    with pytest.raises(ValueError, match="CUDA tensor"):
        net._net()
    with pytest.raises(ValueError, match="CUDA tensor"):
        net._addresses(net.g)
    with pytest.raises(ValueError, match="CUDA tensor"):
        _array([torch.zeros(128, 256, dtype=torch.bfloat16)] * 4)
    assert _array(None) is None


def test_native_calls_refuse_short_flat_vectors():
    net = _network(1000)
    with pytest.raises(ValueError, match="cannot hold"):
        net._net()
    with pytest.raises(ValueError, match="cannot hold"):
        net._addresses(net.g)
