"""The native host path of linear layers and experts (native/host.cpp) against the oracle: inputs that it takes, inputs that
it hands back, and a layer whose tensors are replaced or that is copied between calls."""
import copy

import pytest
import torch

from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, random_layer
from tests.test_gpu_parity import make_expert

DEV = torch.device("cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("shape, dtype, strided", [
    ((256,), torch.bfloat16, False), ((3, 256), torch.bfloat16, False), ((2, 3, 256), torch.bfloat16, False),
    ((2, 3, 256), torch.float16, False), ((4, 256), torch.bfloat16, True)])
def test_linear_and_expert_inputs(shape, dtype, strided):
    od, g = random_layer(128, 256, 4, 64, seed=1), torch.Generator().manual_seed(2)
    ods = tuple(random_layer(n, k, 2, 16, seed=3 + i) for i, (n, k) in enumerate(((512, 256), (256, 512), (512, 256))))
    x = torch.randn(*shape, generator=g).to(dtype)
    xd = torch.stack([x, x], -1).to(DEV)[..., 0] if strided else x.to(DEV)
    for module, want in ((layer_from_oracle(od, DEV), O.linear(x.to(torch.bfloat16).reshape(-1, 256), od)),
                         (make_expert(256, 512, ods), O.expert_ffn(x.to(torch.bfloat16).reshape(-1, 256), *ods))):
        for _ in range(2):
            y = module(xd)
            assert y.shape[:-1] == x.shape[:-1] and y.dtype == dtype
            assert O.rel_err(y.cpu().reshape(want.shape), want) < 1e-2


@pytest.mark.gpu
def test_layer_with_new_tensors_and_copied_layer():
    a, b = (random_layer(128, 256, 4, 64, seed=s) for s in (1, 2))
    x = torch.randn(1, 256, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    layer, other = layer_from_oracle(a, DEV), layer_from_oracle(b, DEV)
    layer(x.to(DEV)), other(x.to(DEV))
    layer.W_q, layer.meta = other.W_q, copy.copy(other.meta)
    assert O.rel_err(layer(x.to(DEV)).cpu(), O.linear(x, b)) < 1e-2
    assert copy.deepcopy(layer._plan) is None
    with pytest.raises(RuntimeError):
        layer(x)
