"""The shape-agnostic linear (csrc/linear_generic.cu) at its remainders, against 64 bits: rows, members and columns that do not
fill a tile, meta vectors that wrap in the middle of a lane's columns, rows at odd addresses, gathered rows, a bias."""
import ctypes as C

import pytest
import torch

from mixtral_offloading_b200 import HQQLinearTritonSavable, _cabi
from oracle import hqq_oracle as O
from tests.helpers import fill_layer, quant_config
from tests.test_many_row_precision import errors, weight64

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _layer(nbits, group, N, K, meta_group, seed=1, meta_zero=None):
    W = (torch.randn(N, K, generator=torch.Generator().manual_seed(seed)) * 0.02).to(torch.bfloat16)
    cfg = quant_config(nbits, group)
    cfg["scale_quant_params"]["group_size"], cfg["zero_quant_params"]["group_size"] = meta_group, meta_zero or meta_group
    layer = HQQLinearTritonSavable(None, cfg, HQQLinearTritonSavable.get_hqq_meta((K, N), cfg))
    return fill_layer(layer, O.quantize(W, nbits, group, meta_group, meta_zero), DEV)


@pytest.mark.parametrize("nbits,group,N,K,meta_group", [
    (2, 12, 48, 36, 12), (2, 12, 36, 1028, 4), (2, 5, 60, 132, 4),           # whole bytes and G = 3, 12; groups of 12 and 5
    (4, 20, 80, 36, 8), (4, 6, 18, 1156, 4), (4, 128, 512, 260, 16),         # G = 4, 3; a group of 128 in 8 chunks
    (3, 7, 35, 40, 8), (3, 64, 640, 132, 24), (3, 17, 34, 2052, 8),          # the last word not full; one member too many
    (2, 16, 64, 30, 8), (4, 32, 64, 33, 2), (3, 16, 48, 18, 2)])             # K no multiple of 4: element by element
@pytest.mark.parametrize("M", [1, 4, 5, 8, 19])
def test_remainders(nbits, group, N, K, meta_group, M):
    layer = _layer(nbits, group, N, K, meta_group)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
    want = x.double() @ weight64(layer).t()
    bias = torch.randn(N, generator=torch.Generator().manual_seed(7)).to(torch.bfloat16).to(DEV)
    odd = torch.empty(x.numel() + 1, dtype=torch.bfloat16, device=DEV)[1:].view(M, K).copy_(x)
    for rows in (x, odd):
        # weights, products and sums in fp32: 2^-24 sqrt(K) of the result at most, beside its rounding
        err, rounding = errors(layer(rows), want)
        assert err < 1.002 * rounding + 1e-5
    layer.bias = bias
    err, rounding = errors(layer(x), want + bias.double())
    assert err < 1.002 * rounding + 1e-5
    assert _cabi.lib().hqm_device_error() == 0


def test_scale_and_zero_of_different_groups():
    layer = _layer(4, 64, 256, 256, 256, meta_zero=64)
    x = torch.randn(3, 256, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    err, rounding = errors(layer(x), x.double() @ weight64(layer).t())
    assert err < 1.002 * rounding + 1e-5


def test_gathered_rows():
    """An expert whose layers only this kernel takes, on rows picked by index."""
    hidden, ffn = 96, 160
    layers = [_layer(4, 16, ffn, hidden, 32, 1), _layer(4, 16, hidden, ffn, 32, 2), _layer(4, 16, ffn, hidden, 32, 3)]
    x = torch.randn(20, hidden, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    idx = torch.tensor([3, 19, 0, 7, 11, 12], dtype=torch.int32, device=DEV)
    d1, d2, d3 = (C.byref(lyr.descriptor()) for lyr in layers)
    lib = _cabi.lib()
    need = lib.hqm_expert_ffn_scratch_bytes(len(idx), d1, d2, d3)
    ws = torch.zeros(need, dtype=torch.uint8, device=DEV)
    out = torch.zeros_like(x)
    _cabi.check(lib.hqm_expert_ffn(_cabi.ptr(out), _cabi.ptr(x), len(idx), _cabi.ptr(idx), None, 0, d1, d2, d3, _cabi.ptr(ws), need,
                                   _cabi.stream_ptr(DEV)))
    a, b, xs = weight64(layers[0]), weight64(layers[2]), x[idx.long()].double()
    want = (torch.nn.functional.silu(xs @ a.t()) * (xs @ b.t())) @ weight64(layers[1]).t()
    assert ((out[idx.long()].double() - want).norm() / want.norm()).item() < 1e-2      # (h and its factors are bf16)
    rest = torch.ones(20, dtype=torch.bool, device=DEV)
    rest[idx.long()] = False
    assert not out[rest].any()
