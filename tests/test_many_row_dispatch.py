"""Which many-row calls go to the tensor-core kernel, and what happens to those that do not: formats, workspaces and inputs at
the edges of its range, against the oracle."""
import ctypes as C

import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, _cabi
from mixtral_offloading_b200.custom_layers import linear_group
from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, random_layer, random_layer_fast
from tests.test_gpu_parity import Cfg, make_expert

DEV = torch.device("cuda:0")
# of the largest result: half a unit in the last place of bf16 (2^-9), and as much again for the kernels' 16-bit factors
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


def _in_scratch(d, x, size, y):
    """hqm_linear with exactly `size` bytes of scratch; the bytes behind them stay as they are."""
    lib, guard = _cabi.lib(), 1 << 16
    ws = torch.full((size + guard,), 7, dtype=torch.uint8, device=DEV)
    _cabi.check(lib.hqm_scratch_init(_cabi.ptr(ws), _cabi.stream_ptr(DEV)))
    rc = lib.hqm_linear(_cabi.ptr(y), _cabi.ptr(x), x.shape[0], C.byref(d), None, _cabi.ptr(ws), size, _cabi.stream_ptr(DEV))
    assert bool((ws[size:] == 7).all()) and int(ws[:lib.hqm_scratch_header_bytes()].max()) == 0
    return rc


@pytest.mark.gpu
@pytest.mark.parametrize("nbits,group,N,K,Ms", [
    (2, 16, 4096, 14336, (17, 32, 100)), (2, 16, 14336, 4096, (5, 17, 34)), (4, 64, 4096, 4096, (64, 100)),
    (4, 64, 1024, 4096, (5, 100, 400)), (3, 64, 1024, 4096, (5, 100))])
def test_little_scratch(nbits, group, N, K, Ms):
    """Calls whose fp32 sums fit a fixed workspace work in it: the built-in one of 2 MiB, and one of the size that
    hqm_linear_scratch_bytes names (narrow chunks, few CTAs, several passes); with a byte less they are refused."""
    lib = _cabi.lib()
    layer = layer_from_oracle(random_layer_fast(N, K, nbits, group, seed=nbits), DEV)
    d, W = layer.descriptor(), layer.dequantize(torch.float32).double()
    for M in Ms:
        x = torch.randn(M, K, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16).to(DEV)
        want, y = x.double() @ W.t(), torch.empty((M, N), dtype=torch.bfloat16, device=DEV)

        def right():
            return ((y.double() - want).abs().max() / want.abs().max()).item() < TOL

        need = lib.hqm_linear_scratch_bytes(M, C.byref(d))
        if nbits != 3:
            assert need <= lib.hqm_static_scratch_capacity()
            assert lib.hqm_linear_static_scratch(_cabi.ptr(y.fill_(7.0)), _cabi.ptr(x), M, C.byref(d), None, _cabi.stream_ptr(DEV)) == 0
            assert right(), M
        for size in (need, (need + lib.hqm_linear_scratch_preferred(M, C.byref(d))) // 512 * 256):
            y.fill_(7.0)
            assert _in_scratch(d, x, size, y) == 0 and right(), (M, size)
        assert _in_scratch(d, x, need - 1, y) == _cabi.HQM_ERR_SCRATCH
    assert lib.hqm_device_error() == 0


@pytest.mark.gpu
def test_builtin_scratch_takes_a_layer_too_wide_for_it():
    """16 staged rows of 65536 columns are more than 2 MiB; the sums of 20 rows are not."""
    N, K, M = 128, 65536, 20
    layer = layer_from_oracle(random_layer_fast(N, K, 4, 64, seed=1), DEV)
    x = torch.randn(M, K, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    y = torch.empty((M, N), dtype=torch.bfloat16, device=DEV)
    assert _cabi.lib().hqm_linear_static_scratch(_cabi.ptr(y), _cabi.ptr(x), M, C.byref(layer.descriptor()), None,
                                                 _cabi.stream_ptr(DEV)) == 0
    want = x.double() @ layer.dequantize(torch.float32).double().t()
    assert ((y.double() - want).abs().max() / want.abs().max()).item() < TOL


def _at_odd_address(t):
    """t in memory that starts 2 bytes behind a 16-byte boundary."""
    room = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
    out = room[1:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == 2
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 3, 5, 40, 30000])
def test_expert_on_unaligned_rows(M):
    """The layers then run one after the other, in the workspace that hqm_expert_ffn_scratch_bytes names (30000 rows: their
    outputs alone are larger than what the fused launches need)."""
    hidden, ffn = 256, 768
    ods = tuple(random_layer(n, k, 2, 16, seed=i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
    expert = make_expert(hidden, ffn, ods)
    few = torch.randn(min(M, 64), hidden, generator=torch.Generator().manual_seed(M)).to(torch.bfloat16)
    x = _at_odd_address(few.repeat(-(-M // few.shape[0]), 1)[:M].to(DEV))
    d1, d2, d3 = (C.byref(lyr.descriptor()) for lyr in (expert.w1, expert.w2, expert.w3))
    lib = _cabi.lib()
    need, guard = lib.hqm_expert_ffn_scratch_bytes(M, d1, d2, d3), 1 << 20
    ws = torch.full((need + guard,), 7, dtype=torch.uint8, device=DEV)
    _cabi.check(lib.hqm_scratch_init(_cabi.ptr(ws), _cabi.stream_ptr(DEV)))
    out = torch.empty(M, hidden, dtype=torch.bfloat16, device=DEV)
    _cabi.check(lib.hqm_expert_ffn(_cabi.ptr(out), _cabi.ptr(x), M, None, None, 0, d1, d2, d3, _cabi.ptr(ws), need,
                                   _cabi.stream_ptr(DEV)))
    assert bool((ws[need:] == 7).all())
    want, last = O.expert_ffn(few, *ods), M % few.shape[0] or few.shape[0]
    assert O.rel_err(out[:few.shape[0]].cpu(), want) < 1e-2 and O.rel_err(out[-last:].cpu(), want[:last]) < 1e-2
    assert lib.hqm_device_error() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("tokens", [3, 33])
def test_moe_block_and_group_on_unaligned_rows(tokens):
    hidden, ffn, n_exp = 256, 768, 4
    ods = [tuple(random_layer(n, k, 2, 16, seed=10 * e + i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
           for e in range(n_exp)]
    g = torch.Generator().manual_seed(tokens)
    gate = torch.nn.Linear(hidden, n_exp, bias=False, dtype=torch.bfloat16, device=DEV)
    gate.weight.data = (torch.randn(n_exp, hidden, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16)
    xd = _at_odd_address(x.to(DEV))
    y, _ = ResidentMoe(Cfg(hidden, ffn, n_exp), 0, gate, [make_expert(hidden, ffn, o) for o in ods])(xd.view(1, tokens, hidden))
    assert O.rel_err(y.cpu().view(tokens, hidden), O.moe_forward(x, gate.weight.data.cpu(), ods)[0]) < 1e-2
    layers = [random_layer(n, hidden, 4, 64, seed=n) for n in (512, 256)]
    for y, od in zip(linear_group([layer_from_oracle(od, DEV) for od in layers], xd), layers):
        assert O.rel_err(y.cpu(), O.linear(x, od)) < TOL
