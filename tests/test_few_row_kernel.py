"""csrc/gemv_rows.cu through an expert (up to 8 rows) or a layer (up to 5), and csrc/gemv_lists.cu through a block: the remainders of their units and
shares, every number of rows, layers they leave to the other kernels, rows outside the range of fp16."""
import ctypes as C

import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, _cabi
from tests.helpers import layer_from_oracle, random_layer, random_layer_fast
from tests.test_gpu_parity import Cfg, make_expert
from tests.test_many_row_precision import weight64
from tests.test_tma_mode import kernels_of

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def reference(expert, x):
    w1, w2, w3 = (weight64(layer) for layer in (expert.w1, expert.w2, expert.w3))
    x = x.double()
    return (torch.nn.functional.silu(x @ w1.t()) * (x @ w3.t())) @ w2.t()


@pytest.mark.parametrize("hidden,ffn", [
    (128, 4096),                 # one step to a unit; down: two residues of a unit's 16
    (512, 3072),                 # fp16 values repeat after 3 residues
    (512, 7168), (1024, 7168),   # after 7; units cut between CTAs
    (512, 11264),                # after 11: not taken
    (256, 768)])                 # their rows are no multiple of 128: not taken
def test_units_and_shares(hidden, ffn):
    ods = tuple(random_layer(n, k, 2, 16, seed=i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
    expert = make_expert(hidden, ffn, ods)
    for M in range(1, 10):
        x = torch.randn(M, hidden, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
        y, want = expert(x), reference(expert, x)
        # bf16 roundings (1.7e-3 of the value each) of gate, activation, up, h and the result: 3.8e-3; 7e-4 for the 16-bit
        # factors of either layer; and half as much again for the scatter of 128 results
        assert ((y.double() - want).norm() / want.norm()).item() < 6e-3, M
        assert torch.equal(y, expert(x)), M                  # pieces of a unit are added in a fixed order
    assert _cabi.lib().hqm_device_error() == 0


@pytest.mark.parametrize("M", [5, 8])
@pytest.mark.parametrize("scale", [1e-7, 3e5])
def test_rows_outside_the_range_of_fp16(M, scale):
    """From five rows on a row carries a power of two; its neighbours are not affected.  (Such rows make h = silu(a) * b very small
    or, with weights this small, large but inside bf16.)"""
    hidden, ffn = 512, 3072
    ods = tuple(random_layer(n, k, 2, 16, seed=i, std=0.02 if scale < 1 else 1e-3)
                for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
    expert = make_expert(hidden, ffn, ods)
    x = torch.randn(M, hidden, generator=torch.Generator().manual_seed(M))
    x[M // 2] *= scale
    x = x.to(torch.bfloat16).to(DEV)
    y, want = expert(x).double(), reference(expert, x)
    for m in range(M):
        assert ((y[m] - want[m]).norm() / want[m].norm()).item() < 6e-3, m


@pytest.mark.parametrize("hidden,ffn,n_exp", [(512, 3072, 8), (128, 4096, 3), (1024, 7168, 32)])
@pytest.mark.parametrize("tokens", [2, 5, 8, 9, 30, 36, 37])
def test_lists_of_every_length(hidden, ffn, n_exp, tokens):
    """A block's lists: empty ones, up to 4, 5 to 8 and more rows in one call, units cut between CTAs, fewer steps than CTAs."""
    ods = [tuple(random_layer(n, k, 2, 16, seed=10 * e + i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
           for e in range(min(n_exp, 4))]
    gate = torch.nn.Linear(hidden, n_exp, bias=False, dtype=torch.bfloat16, device=DEV)
    g = torch.Generator().manual_seed(tokens)
    gate.weight.data = (torch.randn(n_exp, hidden, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    gate.weight.data[1] = -4.0 * gate.weight.data[0]         # lists of very different lengths
    experts = [make_expert(hidden, ffn, ods[e % len(ods)]) for e in range(n_exp)]
    moe = ResidentMoe(Cfg(hidden, ffn, n_exp), 0, gate, experts)
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16).to(DEV)
    y, logits = moe(x.view(1, tokens, hidden))
    y = y.view(tokens, hidden)
    p, idx = torch.softmax(logits.view(tokens, n_exp).float(), 1).topk(2, 1)
    p = (p / p.sum(1, keepdim=True)).to(torch.bfloat16).double()
    want = torch.zeros(tokens, hidden, dtype=torch.float64, device=DEV)
    for e in range(n_exp):
        t = (idx == e).any(1).nonzero().flatten()
        if len(t):
            want[t] += (p * (idx == e)).sum(1)[t].unsqueeze(1) * reference(experts[e], x[t])
    # 5.9e-3 for the experts with more than 16 rows (bf16 weights), 4e-3 for the others, and a rounding each (1.7e-3) of the weighted
    # outputs and of their sum: 6.4e-3; twice that for any single token, whose two outputs may partly cancel
    error, size = (y.double() - want).norm(dim=1), want.norm(dim=1)
    assert (error.norm() / size.norm()).item() < 7e-3
    assert (error / size).max().item() < 1.3e-2
    assert torch.equal(y, moe(x.view(1, tokens, hidden))[0].view(tokens, hidden))
    assert _cabi.lib().hqm_device_error() == 0


@pytest.mark.parametrize("n_exp,tokens,few", [(2, 8, True), (2, 9, False), (3, 12, True), (3, 13, False), (4, 16, True), (4, 17, False),
                                              (8, 36, True), (8, 37, False), (32, 144, True), (32, 145, False)])
def test_which_blocks_have_short_lists(n_exp, tokens, few):
    """Up to nine entries per list on average, up to eight with four experts or less."""
    hidden, ffn = 128, 4096
    ods = tuple(random_layer(n, k, 2, 16, seed=i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
    gate = torch.nn.Linear(hidden, n_exp, bias=False, dtype=torch.bfloat16, device=DEV)
    gate.weight.data = (torch.randn(n_exp, hidden, generator=torch.Generator().manual_seed(1)) * 0.1).to(torch.bfloat16).to(DEV)
    expert = make_expert(hidden, ffn, ods)
    moe = ResidentMoe(Cfg(hidden, ffn, n_exp), 0, gate, [expert] * n_exp)
    x = torch.randn(1, tokens, hidden, generator=torch.Generator().manual_seed(tokens)).to(torch.bfloat16).to(DEV)
    assert ("gemv_lists_kernel" in kernels_of(lambda: moe(x))) == few
    y, logits = moe(x)
    p = torch.softmax(logits.view(tokens, n_exp).float(), 1).topk(2, 1).values
    p = (p / p.sum(1, keepdim=True)).to(torch.bfloat16).double()
    want = reference(expert, x[0]) * p.sum(1, keepdim=True)                   # (the experts are alike)
    assert ((y[0].double() - want).norm() / want.norm()).item() < 7e-3        # as in test_lists_of_every_length
    assert _cabi.lib().hqm_device_error() == 0


@pytest.mark.parametrize("N,K,few", [(14336, 4096, True), (4096, 14336, True), (14336, 14336, True), (14336, 3072, False)])
def test_large_linear_layers(N, K, few):
    """Two to five rows of layers with three steps or more for every SM (one with less, which the other kernels keep); with less
    workspace than that wants, and a bias."""
    steps = -(-N // 16 // 4 // 16) * (K // 128)
    assert few == (steps >= 3 * torch.cuda.get_device_properties(0).multi_processor_count)
    layer = layer_from_oracle(random_layer_fast(N, K, 2, 16, seed=3), DEV)
    layer.bias = torch.randn(N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    lib, d, W = _cabi.lib(), layer.descriptor(), weight64(layer)
    for M in (1, 2, 4, 5, 6):
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
        want = x.double() @ W.t() + layer.bias.double()
        need, wanted = lib.hqm_linear_scratch_bytes(M, C.byref(d)), lib.hqm_linear_scratch_preferred(M, C.byref(d))
        assert wanted >= need
        header = lib.hqm_scratch_header_bytes()                  # (where nothing is needed the buffer still has one)
        for size in sorted({need, max(need, wanted - 1), wanted}):
            ws = torch.full((wanted + 4096,), 7, dtype=torch.uint8, device=DEV)
            _cabi.check(lib.hqm_scratch_init(_cabi.ptr(ws), _cabi.stream_ptr(DEV)))
            y = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
            run = lambda: _cabi.check(lib.hqm_linear(_cabi.ptr(y), _cabi.ptr(x), M, C.byref(d), _cabi.ptr(layer.bias), _cabi.ptr(ws), size,
                                                     _cabi.stream_ptr(DEV)))
            assert ("gemv_rows_kernel" in kernels_of(run)) == (few and 2 <= M <= 5 and size == wanted), (M, size)
            assert bool((ws[max(size, header):] == 7).all())
            # a rounding to bf16 (1.7e-3) and 16-bit factors (1e-3)
            assert ((y.double() - want).norm() / want.norm()).item() < 2.5e-3, (M, size)


def test_what_the_factors_add():
    """Five rows, one of them with a bias that takes its value away, so that the rounding of the result is small: what is left are
    the roundings to fp16 of a scale (3.0e-4: of byte - zero and of the product) and of x * s (2.1e-4), 3.7e-4 together.  (These
    layers with the same roundings in 64 bits: 3.65e-4.)  Zeros of 11 bits have two more, relative to z, which is 1.7 times q - z:
    6.2e-4."""
    layer = layer_from_oracle(random_layer(14336, 4096, 2, 16, seed=3), DEV)
    x = torch.randn(5, 4096, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).to(DEV)
    want = x.double() @ weight64(layer).t()
    layer.bias = (-want[0]).to(torch.bfloat16)
    y = layer(x)[0].double() - layer.bias.double()
    assert ((y - want[0]).norm() / want[0].norm()).item() < 4.5e-4
