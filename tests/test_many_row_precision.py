"""The many-row kernel against 64 bits: what its 16-bit factors add to the rounding of the result."""
import pytest
import torch

from tests.helpers import layer_from_oracle, random_layer

DEV = torch.device("cuda:0")


def weight64(layer):
    """The weight that the layer's tensors stand for, in 64 bits."""
    m = layer.meta
    (N, K), nbits = m["shape"], m["nbits"]

    def decode(q, mm):
        return ((q.reshape(-1, mm["scale"].numel()).double() - mm["zero"].double().view(1, -1)) * mm["scale"].double().view(1, -1)).view(1, -1)

    shifts = {2: (6, 4, 2, 0), 3: tuple(3 * (9 - i) for i in range(10)), 4: (4, 0)}[nbits]
    codes = torch.stack([(layer.W_q >> s) & (2 ** nbits - 1) for s in shifts], 1).reshape(-1, K)[:N].reshape(m["group_size"], -1)
    return ((codes.double() - decode(m["zero_q"], m["meta_zero"])) * decode(m["scale_q"], m["meta_scale"])).reshape(N, K)


def errors(y, want):
    """Relative error of y, and that of the wanted values rounded to y's type."""
    return tuple(((t.double() - want).norm() / want.norm()).item() for t in (y, want.to(y.dtype)))


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,group,bound", [(2, 16, 6e-4), (3, 64, 7e-4), (4, 64, 7e-4)])
@pytest.mark.parametrize("M", [5, 16, 64, 200])
def test_factors_of_16_bits(nbits, group, bound, M):
    """A weight (c - z) s is formed as c s + T, T = -z s, in fp16.  A rounding to fp16 is 2^-11 / sqrt(3) of half the binade
    on average, 2.1e-4 of the value: of the weight, and of T, which is 1.7 (2 bit) to 2.4 times as large for min / max
    quantised normal weights: 4.2e-4 and 5.5e-4, with a sixth to a quarter on top for the 8-bit decoding of s.  (Forming z in
    fp16 instead adds two roundings of T's size: 7e-4 and 9.5e-4.)"""
    layer = layer_from_oracle(random_layer(1024, 2048, nbits, group, seed=nbits), DEV)
    x = torch.randn(M, 2048, generator=torch.Generator().manual_seed(M)).to(torch.float16).to(DEV)
    err, rounding = errors(layer(x), x.double() @ weight64(layer).t())
    assert (err ** 2 - rounding ** 2) ** 0.5 < bound
