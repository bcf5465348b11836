"""ResidentMoe computes with the experts as they are at the call: replaced, of different formats, at odd addresses; and with a
gate of any strides."""
import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, _cabi
from oracle import hqq_oracle as O
from tests.helpers import layer_from_oracle, random_layer
from tests.test_gpu_parity import Cfg, make_expert

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
HIDDEN, FFN, EXPERTS = 256, 768, 4
SHAPES = ((FFN, HIDDEN), (HIDDEN, FFN), (FFN, HIDDEN))


def _oracle_expert(seed, nbits=2, group=16):
    return tuple(random_layer(n, k, nbits, group, seed=10 * seed + i) for i, (n, k) in enumerate(SHAPES))


class _Block:
    def __init__(self):
        self.ods = [_oracle_expert(e) for e in range(EXPERTS)]
        self.gate = torch.nn.Linear(HIDDEN, EXPERTS, bias=False, dtype=torch.bfloat16, device=DEV)
        self.gate.weight.data = (torch.randn(EXPERTS, HIDDEN, generator=torch.Generator().manual_seed(1)) * 0.1).to(torch.bfloat16).to(DEV)
        self.moe = ResidentMoe(Cfg(HIDDEN, FFN, EXPERTS), 0, self.gate, [make_expert(HIDDEN, FFN, o) for o in self.ods])

    def check(self):
        for tokens in (1, 2, 40):
            x = torch.randn(tokens, HIDDEN, generator=torch.Generator().manual_seed(tokens)).to(torch.bfloat16)
            want, logits = O.moe_forward(x, self.gate.weight.data.cpu().contiguous(), self.ods)
            y, got = self.moe(x.to(DEV).view(1, tokens, HIDDEN))
            assert O.rel_err(y.cpu().view(tokens, HIDDEN), want) < 1e-2, tokens
            assert O.rel_err(got.cpu(), logits) < 1e-2, tokens
        assert _cabi.lib().hqm_device_error() == 0


def _ffn(expert):
    return ResidentMoe._ffn(expert)


@pytest.mark.parametrize("how", ["tensors", "layer", "expert"])
def test_replaced_expert(how):
    block = _Block()
    block.check()
    block.ods[2] = _oracle_expert(7)
    ffn = _ffn(block.moe._experts[2])
    if how == "expert":
        block.moe._experts[2] = make_expert(HIDDEN, FFN, block.ods[2])
    for name, od in zip(("w1", "w2", "w3"), block.ods[2]):
        if how == "tensors":                                 # the layer does not learn of it
            fresh, layer = layer_from_oracle(od, DEV), getattr(ffn, name)
            layer.W_q, layer.meta = fresh.W_q, fresh.meta
        elif how == "layer":
            setattr(ffn, name, layer_from_oracle(od, DEV))
    block.check()


def test_expert_of_another_format_in_the_same_memory():
    """2-bit groups of 32 in memory that held groups of 16; the layer has been used, and so has a descriptor, in between."""
    block = _Block()
    block.check()
    ods = _oracle_expert(9, 2, 32)
    for name, od in zip(("w1", "w2", "w3"), ods):
        layer, fresh = getattr(_ffn(block.moe._experts[0]), name), layer_from_oracle(od, DEV)

        def into(dst, src):
            return dst.view(-1)[:src.numel()].copy_(src.reshape(-1)).view(src.shape)

        meta = dict(fresh.meta, scale_q=into(layer.meta["scale_q"], fresh.meta["scale_q"]), zero_q=into(layer.meta["zero_q"], fresh.meta["zero_q"]))
        for m in ("meta_scale", "meta_zero"):
            meta[m] = dict(fresh.meta[m], **{k: into(layer.meta[m][k], fresh.meta[m][k]) for k in ("scale", "zero")})
        layer.W_q, layer.meta, layer._desc = into(layer.W_q, fresh.W_q), meta, None
        layer.descriptor()
        x = torch.randn(3, od["K"], generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
        assert O.rel_err(layer(x.to(DEV)).cpu(), O.linear(x, od)) < 1e-2
    block.ods[0] = ods
    block.check()


@pytest.mark.parametrize("nbits,group", [(4, 64), (2, 32)])
def test_experts_of_different_formats(nbits, group):
    block = _Block()
    block.ods[1] = _oracle_expert(1, nbits, group)
    for name, od in zip(("w1", "w2", "w3"), block.ods[1]):
        setattr(_ffn(block.moe._experts[1]), name, layer_from_oracle(od, DEV))
    assert block.moe.scratch_bytes(1) == block.moe.scratch_bytes(40) == 0
    block.check()
    block.ods[1] = _oracle_expert(8)
    for name, od in zip(("w1", "w2", "w3"), block.ods[1]):
        setattr(_ffn(block.moe._experts[1]), name, layer_from_oracle(od, DEV))
    assert block.moe.scratch_bytes(40) > 0
    block.check()


def test_expert_at_an_odd_address():
    block = _Block()
    layer = _ffn(block.moe._experts[3]).w2
    room = torch.empty(layer.W_q.numel() + 4, dtype=torch.uint8, device=DEV)
    layer.W_q = room[4:].copy_(layer.W_q.view(-1)).view(layer.W_q.shape)
    assert block.moe.scratch_bytes(1) == block.moe.scratch_bytes(40) == 0
    block.check()


def test_gate_with_other_strides():
    block = _Block()
    wide = torch.zeros(HIDDEN, EXPERTS + 3, dtype=torch.bfloat16, device=DEV)
    wide[:, :EXPERTS] = block.gate.weight.data.t()
    block.gate.weight.data = wide[:, :EXPERTS].t()
    assert not block.gate.weight.is_contiguous()
    block.check()
