"""csrc/gemv_rows.cu fills its stages under the kernel in front and then waits for it; what bounds its waits is its own work."""
import pytest
import torch

from mixtral_offloading_b200 import _cabi
from tests.helpers import layer_from_oracle, random_layer, random_layer_fast
from tests.test_gpu_parity import make_expert

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def test_expert_behind_many_rows():
    """A launch of some 10 ms lets its successor start at once; its last tiles leave SMs to it one after the other."""
    layer = layer_from_oracle(random_layer_fast(14336, 4096, 2, 16, seed=1), DEV)
    ods = tuple(random_layer(n, k, 2, 16, seed=i) for i, (n, k) in enumerate(((3072, 512), (512, 3072), (3072, 512))))
    expert = make_expert(512, 3072, ods)
    g = torch.Generator(device=DEV).manual_seed(1)
    many = torch.randn(65536, 4096, generator=g, device=DEV, dtype=torch.bfloat16)
    for M in (1, 3, 8):
        x = torch.randn(M, 512, generator=g, device=DEV, dtype=torch.bfloat16)
        alone = expert(x)
        torch.cuda.synchronize()
        layer(many)
        assert torch.equal(expert(x), alone), M
    assert _cabi.lib().hqm_device_error() == 0
