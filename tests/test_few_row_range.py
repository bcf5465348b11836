"""The ends of the number range through csrc/gemv_rows.cu and csrc/gemv_lists.cu: scales with which x * s leaves fp16, infinities."""
import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, _cabi
from tests.helpers import layer_from_oracle, random_layer, random_layer_fast
from tests.test_few_row_kernel import reference
from tests.test_gpu_parity import Cfg, make_expert
from tests.test_many_row_precision import weight64

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def layers(hidden, ffn, std):
    """Gate and up of the given size, with down projections that bring h back."""
    return tuple(random_layer(n, k, 2, 16, seed=i, std=s) for i, (n, k, s) in enumerate(((ffn, hidden, std), (hidden, ffn, 0.02), (ffn, hidden, std))))


def rows(M, hidden, std, seed):
    return (torch.randn(M, hidden, generator=torch.Generator().manual_seed(seed)) / std).to(torch.bfloat16).to(DEV)


# scales (about 1.2 std) on both sides of 2048, where x * s leaves fp16 with x just below 32
@pytest.mark.parametrize("std", [1e3, 2e3, 1e4])
@pytest.mark.parametrize("M", [5, 8])
def test_large_scales_of_an_expert(std, M):
    expert = make_expert(512, 3072, layers(512, 3072, std))
    x = rows(M, 512, std, M)
    y, want = expert(x), reference(expert, x)
    assert ((y.double() - want).norm() / want.norm()).item() < 6e-3          # as in test_few_row_kernel: relative, so whatever std is


@pytest.mark.parametrize("std", [1e3, 2e3, 1e4])
@pytest.mark.parametrize("tokens", [2, 8, 9])
def test_large_scales_of_a_block(std, tokens):
    experts = [make_expert(512, 3072, layers(512, 3072, std)) for _ in range(4)]
    gate = torch.nn.Linear(512, 4, bias=False, dtype=torch.bfloat16, device=DEV)
    gate.weight.data = torch.randn(4, 512, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    moe = ResidentMoe(Cfg(512, 3072, 4), 0, gate, experts)
    x = rows(tokens, 512, std, tokens)
    y, logits = moe(x.view(1, tokens, 512))
    p = torch.softmax(logits.view(tokens, 4).float(), 1).topk(2, 1).values
    p = (p / p.sum(1, keepdim=True)).to(torch.bfloat16).double()
    want = reference(experts[0], x) * p.sum(1, keepdim=True)                  # (the experts are alike)
    assert ((y.view(tokens, 512).double() - want).norm() / want.norm()).item() < 7e-3
    assert _cabi.lib().hqm_device_error() == 0


@pytest.mark.parametrize("std", [1e-6, 1e-4, 3e-3])
@pytest.mark.parametrize("tokens", [2, 8])
def test_small_h_of_a_block(std, tokens):
    """h of 1e-10 to 1e-3: as fp16 without a factor of its row, and times a scale, below fp16's smallest."""
    experts = [make_expert(512, 3072, layers(512, 3072, std)) for _ in range(4)]
    gate = torch.nn.Linear(512, 4, bias=False, dtype=torch.bfloat16, device=DEV)
    gate.weight.data = (torch.randn(4, 512, generator=torch.Generator().manual_seed(1)) * 0.1).to(torch.bfloat16).to(DEV)
    moe = ResidentMoe(Cfg(512, 3072, 4), 0, gate, experts)
    x = rows(tokens, 512, 1.0, tokens)
    y, logits = moe(x.view(1, tokens, 512))
    p = torch.softmax(logits.view(tokens, 4).float(), 1).topk(2, 1).values
    p = (p / p.sum(1, keepdim=True)).to(torch.bfloat16).double()
    want = reference(experts[0], x) * p.sum(1, keepdim=True)                  # (the experts are alike)
    assert ((y.view(tokens, 512).double() - want).norm() / want.norm()).item() < 7e-3


@pytest.mark.parametrize("N,K", [(14336, 4096), (4096, 14336)])
@pytest.mark.parametrize("value", [float("inf"), -float("inf")])
def test_an_infinite_x_has_the_sign_of_the_weight(N, K, value):
    layer = layer_from_oracle(random_layer_fast(N, K, 2, 16, seed=3), DEV)
    W = weight64(layer)
    x = torch.randn(5, K, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).to(DEV)
    want = x.double() @ W.t()
    x[3, 777] = value
    y = layer(x)
    w = W[:, 777]
    clear = w.abs() > 1e-3 * w.abs().max()                   # (a weight of zero makes NaN)
    assert clear.float().mean().item() > 0.9
    assert torch.equal(y[3].double()[clear], (value * w)[clear])
    others = [0, 1, 2, 4]
    assert ((y[others].double() - want[others]).norm() / want[others].norm()).item() < 2.5e-3       # as in test_few_row_kernel
    x[3, 778] = -value                                       # both signs: NaN where the weights' signs agree
    both = layer(x)[3]
    clear &= W[:, 778].abs() > 1e-3 * w.abs().max()
    assert torch.equal(torch.isnan(both)[clear], (torch.sign(w) == torch.sign(W[:, 778]))[clear])


def test_a_nan_stays_in_its_row():
    expert = make_expert(512, 3072, layers(512, 3072, 0.02))
    for M in (2, 4, 5, 8):
        x = rows(M, 512, 1.0, M)
        clean = expert(x)
        x[1, 5] = float("nan")
        y = expert(x)
        assert bool(torch.isnan(y[1]).all())
        others = [m for m in range(M) if m != 1]
        assert torch.equal(y[others], clean[others])
