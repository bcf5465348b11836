"""hqm_set_tma_mode: which kernel takes the single-row launches of an expert and of a block, and that all three agree."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from mixtral_offloading_b200 import ResidentMoe, _cabi
from tests.helpers import random_layer
from tests.test_gpu_parity import Cfg, make_expert
from tests.test_many_row_precision import weight64

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
KERNELS = {0: "gemv_stream_kernel", 1: "gemv_rows_kernel", 2: "gemv_tma_kernel"}


def kernels_of(run):
    run()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    return {k for k in (*KERNELS.values(), "gemv_lists_kernel") if k in names}


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_who_takes_a_single_row(mode):
    hidden, ffn = 512, 3072
    ods = tuple(random_layer(n, k, 2, 16, seed=i) for i, (n, k) in enumerate(((ffn, hidden), (hidden, ffn), (ffn, hidden))))
    x = torch.randn(3, hidden, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).to(DEV)
    gate = torch.nn.Linear(hidden, 4, bias=False, dtype=torch.bfloat16, device=DEV)
    lib = _cabi.lib()
    prev = lib.hqm_set_tma_mode(mode)
    try:
        expert = make_expert(hidden, ffn, ods)
        moe = ResidentMoe(Cfg(hidden, ffn, 4), 0, gate, [make_expert(hidden, ffn, ods) for _ in range(4)])
        one = x[:1].contiguous()
        assert kernels_of(lambda: expert(one)) == {KERNELS[mode]}
        assert kernels_of(lambda: moe(one.view(1, 1, hidden))) == {KERNELS[mode]}
        w1, w2, w3 = (weight64(layer) for layer in (expert.w1, expert.w2, expert.w3))
        want = (torch.nn.functional.silu(x.double() @ w1.t()) * (x.double() @ w3.t())) @ w2.t()
        for y in (expert(one), moe(one.view(1, 1, hidden))[0].view(1, hidden)):            # (the block's experts are alike)
            assert ((y.double() - want[:1]).norm() / want[:1].norm()).item() < 7e-3        # as in test_few_row_kernel
        assert kernels_of(lambda: expert(x)) == {"gemv_rows_kernel"}
        assert lib.hqm_device_error() == 0
    finally:
        lib.hqm_set_tma_mode(prev)
