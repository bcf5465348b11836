"""hqm_dequantize against the oracle, bit for bit: groups that fill a storage word or not, columns that four divides or not."""
import pytest
import torch

from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, random_layer

DEV = torch.device("cuda:0")


@pytest.mark.gpu
@pytest.mark.parametrize("nbits, group, N, K", [
    (2, 16, 64, 256), (2, 16, 1024, 1024), (2, 8, 48, 256), (4, 64, 192, 512), (4, 64, 1024, 512), (4, 32, 256, 128),
    (3, 64, 448, 512), (3, 64, 1792, 256)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_exact(nbits, group, N, K, dtype):
    od = random_layer(N, K, nbits, group, seed=5)
    assert torch.equal(layer_from_oracle(od, DEV).dequantize(dtype).cpu(), O.dequantize(od).to(dtype))


@pytest.mark.gpu
@pytest.mark.parametrize("group, N, K, std", [(16, 192, 64, 0.02), (16, 64, 1088, 3e4), (48, 384, 256, 1e-6), (5, 20, 512, 0.02)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_table_of_four_values(group, N, K, std, dtype):
    """2 bit into 16-bit types: K of few columns and no multiple of a CTA's, values beyond fp16 and below its normal range."""
    od = random_layer(N, K, 2, group, seed=7, std=std)
    assert torch.equal(layer_from_oracle(od, DEV).dequantize(dtype).cpu(), O.dequantize(od).to(dtype))


@pytest.mark.gpu
def test_tensors_off_the_vector_alignment():
    od = random_layer(128, 256, 2, 16, seed=6)
    layer = layer_from_oracle(od, DEV)
    storage = torch.empty(layer.W_q.numel() + 1, dtype=torch.uint8, device=DEV)
    storage[1:] = layer.W_q.reshape(-1)
    layer.W_q = storage[1:].view(layer.W_q.shape)
    assert torch.equal(layer.dequantize(torch.float32).cpu(), O.dequantize(od))
