"""Tokens whose logits are not finite: still two different experts (a block finds a token's two outputs by its entries in two row
lists), weights that are NaN as softmax makes them, and no effect on the other tokens."""
import pytest
import torch

from mixtral_offloading_b200 import ResidentMoe, SparseMoeWrapper, _cabi
from tests.helpers import random_layer
from tests.test_few_row_kernel import reference
from tests.test_gpu_parity import Cfg, make_expert

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
NOT_FINITE = (float("nan"), float("inf"), -float("inf"))


def gate_of(hidden, n_exp, seed=0):
    gate = torch.nn.Linear(hidden, n_exp, bias=False, dtype=torch.bfloat16, device=DEV)
    gate.weight.data = (torch.randn(n_exp, hidden, generator=torch.Generator().manual_seed(seed)) * 0.1).to(torch.bfloat16).to(DEV)
    return gate


@pytest.mark.parametrize("n_exp,hidden", [(2, 128), (8, 4096), (8, 4104), (32, 256)])          # the three kernels
def test_two_experts_whatever_the_logits(n_exp, hidden):
    router = SparseMoeWrapper(Cfg(hidden, 2 * hidden, n_exp), 0, gate_of(hidden, n_exp), None)
    x = torch.randn(9, hidden, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    clean = [t.clone() for t in router.route(x)[:3]]
    for i, v in enumerate(NOT_FINITE):
        x[2 * i + 1, 5 * i] = v
    logits, w, idx, meta, token_idx, token_w = router.route(x)
    bad = ~torch.isfinite(logits.float()).all(1)
    assert bad[1::2][:3].all() and not bad[0::2].any()
    assert bool((idx[:, 0] != idx[:, 1]).all()) and bool(((idx >= 0) & (idx < n_exp)).all())
    assert bool(torch.isnan(w[bad]).all())
    for got, want in zip((logits, w, idx), clean):
        assert torch.equal(got[~bad], want[~bad])
    counts = meta[:n_exp]
    assert torch.equal(counts, torch.bincount(idx.flatten().long(), minlength=n_exp).int())
    for e in range(n_exp):
        lo = int(meta[n_exp + e])
        assert token_idx[lo:lo + int(counts[e])].tolist() == [t for t in range(9) if e in idx[t].tolist()]


@pytest.mark.parametrize("hidden,ffn", [(512, 3072), (256, 768)])              # with the few-row kernel, without
@pytest.mark.parametrize("tokens", [1, 2, 8, 9, 37])
def test_block_with_a_token_of_nan(hidden, ffn, tokens):
    ods = [tuple(random_layer(n, k, 2, 16, seed=10 * e + i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
           for e in range(4)]
    experts = [make_expert(hidden, ffn, od) for od in ods]
    moe = ResidentMoe(Cfg(hidden, ffn, 4), 0, gate_of(hidden, 4), experts)
    x = torch.randn(tokens, hidden, generator=torch.Generator().manual_seed(tokens)).to(torch.bfloat16).to(DEV)
    x[tokens // 2, 3] = float("nan")
    y, logits = moe(x.view(1, tokens, hidden))
    y, others = y.view(tokens, hidden), [t for t in range(tokens) if t != tokens // 2]
    assert bool(torch.isnan(y[tokens // 2]).all())
    p, idx = torch.softmax(logits.view(tokens, 4).float(), 1).topk(2, 1)
    p = (p / p.sum(1, keepdim=True)).to(torch.bfloat16).double()
    outs = [reference(e, x) for e in experts]
    for t in others:
        want = sum(p[t, j] * outs[int(idx[t, j])][t] for j in range(2))
        assert ((y[t].double() - want).norm() / want.norm()).item() < 1.3e-2, t            # of a single token: see test_few_row_kernel
    assert _cabi.lib().hqm_device_error() == 0
