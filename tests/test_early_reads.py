"""What a kernel may read before it waits for the launch in front (include/hqq_moe.h, hqm_set_overlap): the tensors of quantized
weights only.  Router and norm weights may be the output of that launch, as where a host keeps its gate in another type."""
import os
import re

import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, SparseMoeWrapper, _cabi
from oracle import hqq_oracle as O
from tests.helpers import random_layer
from tests.test_gpu_parity import Cfg, make_expert

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mixtral_offloading_b200", "csrc")
DEV = torch.device("cuda:0")


def kernels_with_wait(name):
    """{kernel: its body up to the wait, comments removed} of a source file."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    found = {}
    for part in text.split("__global__")[1:]:
        if "grid_dependency_wait()" in part:
            head = part[:part.index("grid_dependency_wait()")]
            found[re.search(r"(\w+_kernel)\s*\(", head).group(1)] = head[head.index("{"):]
    return found


@pytest.mark.parametrize("kernel", ["router_short_rows_kernel", "router_logits_top2_kernel", "router_lists_kernel"])
def test_router_reads_nothing_early(kernel):
    assert not re.search(r"__ldg|__ldcg|\*reinterpret_cast|\b(gate_w|x|topk_idx)\[", kernels_with_wait("router.cu")[kernel])


@pytest.mark.parametrize("kernel", ["add_rmsnorm_kernel", "add_rmsnorm_rows_vec_kernel"])
def test_norm_reads_nothing_early(kernel):
    assert not re.search(r"__ldg|__ldcg|\*reinterpret_cast|\b(h|w|delta)\[", kernels_with_wait("decode_attn.cu")[kernel])


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("tokens", [1, 3, 33])
def test_gate_in_another_type(dtype, tokens):
    """The gate is converted right in front of the router's launch."""
    hidden, ffn, n_exp = 256, 768, 4
    ods = [tuple(random_layer(n, k, 2, 16, seed=10 * e + i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
           for e in range(n_exp)]
    g = torch.Generator().manual_seed(tokens)
    gate = torch.nn.Linear(hidden, n_exp, bias=False, dtype=dtype, device=DEV)
    experts = [make_expert(hidden, ffn, o) for o in ods]
    moe = ResidentMoe(Cfg(hidden, ffn, n_exp), 0, gate, experts)
    router = SparseMoeWrapper(Cfg(hidden, ffn, n_exp), 0, gate, expert_cache=None)
    for _ in range(4):                                       # new weights for every call: an old conversion would show
        gate.weight.data.copy_((torch.randn(n_exp, hidden, generator=g) * 0.1).to(torch.bfloat16))
        x = torch.randn(tokens, hidden, generator=g).to(torch.bfloat16)
        want, want_logits = O.moe_forward(x, gate.weight.data.cpu().to(torch.bfloat16), ods)
        y, logits = moe(x.to(DEV).view(1, tokens, hidden))
        assert O.rel_err(y.cpu().view(tokens, hidden), want) < 1e-2
        assert O.rel_err(logits.cpu(), want_logits) < 1e-2
        assert O.rel_err(router.route(x.to(DEV))[0].cpu(), want_logits) < 1e-2
    assert _cabi.lib().hqm_device_error() == 0
