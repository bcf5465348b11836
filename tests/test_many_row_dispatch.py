"""Which many-row calls go to the tensor-core kernel, and what happens to those that do not: formats, workspaces and inputs at
the edges of its range, against the oracle."""
import pytest
import torch

from mixtral_offloading_b200 import _cabi
from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, random_layer

DEV = torch.device("cuda:0")
# bf16 results: 2^-9 / sqrt(3) for a rounding that is uniform in the last place, and the kernels' 16-bit factors under it
TOL = 4e-3


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,group,N,K", [(4, 512, 1024, 256), (2, 512, 2048, 256), (4, 256, 1024, 256)])
@pytest.mark.parametrize("M", [5, 64])
def test_groups_of_more_than_256_rows(nbits, group, N, K, M):
    """Tensor maps are encoded up to groups of 256; larger ones go to the shape-agnostic kernel at every row count."""
    od = random_layer(N, K, nbits, group, seed=group)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16)
    y = layer_from_oracle(od, DEV)(x.to(DEV))
    assert O.rel_err(y.cpu(), O.linear(x, od)) < TOL
    assert _cabi.lib().hqm_device_error() == 0
