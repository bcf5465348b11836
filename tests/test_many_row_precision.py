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


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,group,N,K,Ms", [
    (3, 64, 5120, 256, (2, 4)),                              # more members than the 3-bit streaming kernel takes
    (2, 64, 512, 256, (5, 17)), (2, 48, 384, 256, (5, 17)), (4, 128, 1024, 256, (5, 64)), (4, 16, 256, 256, (5, 64)),
    (2, 16, 192, 192, (5, 17)), (2, 16, 320, 704, (17,)), (4, 32, 192, 256, (17,))])
def test_formats_that_only_the_fp32_kernel_takes(nbits, group, N, K, Ms):
    """Weights, products and sums in fp32: what is left is the rounding of the result (and 2^-24 sqrt(K) of the sums)."""
    layer = layer_from_oracle(random_layer(N, K, nbits, group, seed=group), DEV)
    for M in Ms:
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
        err, rounding = errors(layer(x), x.double() @ weight64(layer).t())
        assert err < 1.002 * rounding, M
        # fp16 rows through bf16 would be 2^-9 / sqrt(3) off twice, 2.3e-3
        half = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.float16).to(DEV)
        err, rounding = errors(layer(half), half.double() @ weight64(layer).t())
        assert M < 5 and nbits != 3 or err < 1e-3, M


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,group,N,K", [(2, 16, 256, 320), (4, 64, 256, 320), (4, 64, 1024, 192)])
def test_odd_column_blocks_and_tile_parts(nbits, group, N, K):
    """From 17 rows on: K an odd number of 64-column blocks, some of a tile's parts beyond the last residue."""
    layer = layer_from_oracle(random_layer(N, K, nbits, group, seed=N), DEV)
    for M in (17, 130, 257):
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
        err, rounding = errors(layer(x), x.double() @ weight64(layer).t())
        assert rounding < err < 1.25 * rounding, M           # (and not the fp32 kernel's)
