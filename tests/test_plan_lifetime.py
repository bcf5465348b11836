"""The native plan of a layer (native/host.cpp) lives as long as the layer's own descriptor, and a call holds the plans it uses."""
import pytest
import torch

from mixtral_offloading_b200 import HQQLinearTritonSavable, _cabi, custom_layers
from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, quant_config, random_layer
from tests.test_gpu_parity import make_expert

DEV = torch.device("cuda:0")


def _host_layer(od):
    """A layer on the CPU with the tensors of an oracle layer."""
    return layer_from_oracle(od, torch.device("cpu"))


def test_loading_a_state_dict_drops_the_plan():
    layer, other = (_host_layer(random_layer(128, 256, 4, 64, seed=s)) for s in (1, 2))
    layer._plan = layer._desc = object()
    layer.load_state_dict(other.state_dict())
    assert layer._desc is None and "_plan" not in layer.__dict__


@pytest.mark.gpu
def test_repacking_drops_the_plan():
    od = random_layer(128, 256, 4, 64, seed=1)
    layer = _host_layer(od)
    layer.W_q = torch.from_numpy(O.PACK[4](od["codes"].reshape(64, -1)))        # packed over (group_size, G * K)
    layer._plan = layer._desc = object()
    layer.W_q = layer.W_q.to(DEV)
    layer.repack()
    assert layer._desc is None and "_plan" not in layer.__dict__


@pytest.mark.gpu
def test_quantizing_again_drops_the_plan():
    """A layer quantized again in another format into blocks of the same size: 4-bit (N, K) and 2-bit (2 N, K) have tensors
    of equal sizes, which the allocator hands back."""
    layer = HQQLinearTritonSavable(None, quant_config(4, 64), HQQLinearTritonSavable.get_hqq_meta((256, 512), quant_config(4, 64)))
    g = torch.Generator(device=DEV).manual_seed(1)
    x = torch.randn(7, 256, generator=g, device=DEV).to(torch.bfloat16)
    for i in range(6):
        nbits, group, N = ((4, 64, 512), (2, 128, 1024))[i % 2]
        W = (torch.randn(N, 256, generator=g, device=DEV) * 0.02).to(torch.bfloat16)
        layer.quantize(W, **quant_config(nbits, group))
        assert "_plan" not in layer.__dict__
        y = layer(x)
        want = x.double() @ layer.dequantize(torch.float32).double().t()
        assert y.shape == (7, N) and ((y.double() - want).norm() / want.norm()).item() < 1e-2


@pytest.mark.gpu
def test_plan_is_not_used_without_the_descriptor():
    """The same addresses with another format behind them, the descriptor dropped from outside."""
    a, b = random_layer(512, 256, 4, 64, seed=1), random_layer(1024, 256, 2, 128, seed=2)
    la, lb = layer_from_oracle(a, DEV), layer_from_oracle(b, DEV)
    x = torch.randn(3, 256, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16)
    la(x.to(DEV))
    assert la._plan is not None

    def into(dst, src):                                      # src's values in dst's memory
        return dst.view(-1).copy_(src.reshape(-1)).view(src.shape)

    meta = dict(lb.meta)
    meta["scale_q"], meta["zero_q"] = into(la.meta["scale_q"], lb.meta["scale_q"]), into(la.meta["zero_q"], lb.meta["zero_q"])
    for name in ("meta_scale", "meta_zero"):
        meta[name] = dict(lb.meta[name], **{k: into(la.meta[name][k], lb.meta[name][k]) for k in ("scale", "zero")})
    la.W_q, la.meta, la._desc = into(la.W_q, lb.W_q), meta, None
    y = la(x.to(DEV))
    assert y.shape == (3, 1024) and O.rel_err(y.cpu(), O.linear(x, b)) < 1e-2


@pytest.mark.gpu
def test_layer_replaced_while_its_workspace_grows():
    """The workspace grows through Python code, which may drop the plan that the call works with."""
    od = random_layer(512, 256, 4, 64, seed=1)
    ods = tuple(random_layer(n, k, 2, 16, seed=3 + i) for i, (n, k) in enumerate(((512, 256), (256, 512), (512, 256))))
    layer, expert = layer_from_oracle(od, DEV), make_expert(256, 512, ods)
    x = torch.randn(40, 256, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)
    layer(x[:1].to(DEV)), expert(x[:1].to(DEV))
    grow, calls = custom_layers._scratch, []

    def dropping(device, nbytes):
        for lyr in (layer, expert.w1, expert.w2, expert.w3):
            lyr._drop_descriptor()
        calls.append([bytes(4096) for _ in range(64)])       # whatever was freed is written over
        return grow(device, nbytes)

    host = _cabi.host()
    old = dict(custom_layers._SCRATCH)
    try:
        host.setup(custom_layers._SCRATCH, dropping)
        custom_layers._SCRATCH.clear()
        y = layer(x.to(DEV))
        custom_layers._SCRATCH.clear()
        z = expert(x.to(DEV))
    finally:
        host.setup(custom_layers._SCRATCH, grow)
        custom_layers._SCRATCH.update(old)
    assert len(calls) == 2
    assert O.rel_err(y.cpu(), O.linear(x, od)) < 1e-2
    assert O.rel_err(z.cpu(), O.expert_ffn(x, *ods)) < 1e-2
