"""csrc/gemm_grouped.cu at the sizes where it can go wrong: remainders of tiles, column blocks and row chunks, both ways
of dequantising, lists of every size in one launch."""
import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, _cabi
from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, random_layer, random_layer_fast
from tests.test_gpu_parity import Cfg, make_expert

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
TOL = 4e-3          # bf16 results of 16-bit factors with fp32 sums


@pytest.mark.parametrize("nbits,group,N,K,std", [
    (2, 16, 512, 512, 0.02), (2, 16, 192, 192, 0.02),        # an odd number of tile parts and of column blocks
    (2, 16, 320, 704, 2.0),                                  # scales beyond the range of the denormal fields
    (2, 32, 256, 320, 0.02), (4, 32, 256, 512, 0.02),
    (4, 64, 256, 320, 0.02), (4, 64, 1024, 1024, 30.0),
    (3, 64, 512, 128, 0.02), (3, 64, 1024, 320, 0.02), (3, 64, 2560, 192, 0.02), (3, 64, 5120, 256, 30.0)])
def test_linear_edges(nbits, group, N, K, std):
    od = random_layer(N, K, nbits, group, seed=nbits + group, std=std)
    layer = layer_from_oracle(od, DEV)
    W = layer.dequantize(torch.float32).double()
    for M in (2, 5, 16, 17, 64, 65, 128, 129, 256, 257, 530):
        x = (torch.randn(M, K, generator=torch.Generator().manual_seed(M)) * 10.0 ** (M % 7 - 3)).to(torch.bfloat16).to(DEV)
        y = layer(x)
        want = x.double() @ W.t()
        assert ((y.double() - want).norm() / want.norm()).item() < TOL, M
        assert torch.equal(y, layer(x)), M                   # pieces of a tile are added in a fixed order
    assert _cabi.lib().hqm_device_error() == 0


@pytest.mark.parametrize("nbits,group,N,K,rows", [(2, 16, 13312, 512, (299, 512)), (4, 64, 13312, 512, (300,)), (3, 64, 11264, 1024, (400,))])
def test_whole_tiles_that_the_ctas_do_not_divide(nbits, group, N, K, rows):
    """416 and 440 tiles in shares of three: the last CTA has fewer."""
    layer = layer_from_oracle(random_layer_fast(N, K, nbits, group, seed=nbits), DEV)
    W = layer.dequantize(torch.float32).double()
    for M in rows:
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
        y, want = layer(x), x.double() @ W.t()
        assert ((y.double() - want).norm() / want.norm()).item() < TOL, M
        # and no row or column of a tile is worse than the rest: three times the bound, as a column has some hundred values
        assert ((y.double() - want).norm(dim=0) / want.norm(dim=0)).max().item() < 3 * TOL, M
        assert torch.equal(y, layer(x)), M
    assert _cabi.lib().hqm_device_error() == 0


@pytest.mark.parametrize("nbits,group", [(2, 16), (3, 64), (4, 64)])
def test_fp16_rows_stay_fp16(nbits, group):
    layer = layer_from_oracle(random_layer(1024, 512, nbits, group, seed=nbits), DEV)
    x = torch.randn(33, 512, generator=torch.Generator().manual_seed(1)).to(torch.float16).to(DEV)
    want = x.double() @ layer.dequantize(torch.float32).double().t()
    y = layer(x)
    assert y.dtype == torch.float16 and ((y.double() - want).norm() / want.norm()).item() < 2e-3


@pytest.mark.parametrize("tokens", [2, 3, 17, 70, 300])
def test_moe_block_of_many_tokens(tokens):
    hidden, ffn, n_exp = 256, 768, 4
    ods = [tuple(random_layer(n, k, 2, 16, seed=10 * e + i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
           for e in range(n_exp)]
    gate = torch.nn.Linear(hidden, n_exp, bias=False, dtype=torch.bfloat16, device=DEV)
    g = torch.Generator().manual_seed(tokens)
    gate.weight.data = (torch.randn(n_exp, hidden, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    gate.weight.data[1] = -10.0 * gate.weight.data[0]        # an expert that is often without a token
    moe = ResidentMoe(Cfg(hidden, ffn, n_exp), 0, gate, [make_expert(hidden, ffn, o) for o in ods])
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16)
    y, logits = moe(x.to(DEV).view(1, tokens, hidden))
    want, want_logits = O.moe_forward(x, gate.weight.data.cpu(), ods)
    assert O.rel_err(y.cpu().view(tokens, hidden), want) < 1e-2
    assert O.rel_err(logits.cpu(), want_logits) < 1e-2
    assert torch.equal(y, moe(x.to(DEV).view(1, tokens, hidden))[0])
    assert _cabi.lib().hqm_device_error() == 0
