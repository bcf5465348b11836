"""hqm_greedy_advance: lengths around the vector width, equal values, signed zeros, infinities and NaN."""
import pytest
import torch

from mixtral_offloading_b200.decoder import greedy_advance

DEV = torch.device("cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("vocab", [1, 7, 8, 1000, 32000, 32003])
@pytest.mark.parametrize("kind", ["random", "equal", "zeros", "negative", "inf", "nan"])
def test_argmax_and_position(vocab, kind):
    x = torch.randn(1, vocab, generator=torch.Generator().manual_seed(vocab)).to(torch.bfloat16)
    if kind == "equal":
        x = x.clamp(max=0.5)
    elif kind == "zeros":
        x = torch.where(x > 0, 0.0, -0.0).to(torch.bfloat16)
    elif kind == "negative":
        x = -x.abs() - 1
    elif kind in ("inf", "nan"):
        x[0, vocab // 2] = float(kind)
    v = x[0].float()
    want = int(v.isnan().nonzero()[0]) if kind == "nan" else int((v == v.max()).nonzero()[0])
    token, position = torch.full((1,), -1, device=DEV), torch.full((1,), 4, dtype=torch.int32, device=DEV)
    greedy_advance(x.to(DEV), token, position)
    assert token.item() == want and position.item() == 5
