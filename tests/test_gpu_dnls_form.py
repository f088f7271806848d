"""DNLS: which form a chain's linear sub-steps take (real-space stencil or transforms) follows from its time
step and length alone, so that a chain's bits are the same in an ensemble of any size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,tier", [(28, 5), (32, 3), (36, 5), (48, 3), (64, 5)])
def test_form_and_bits_do_not_depend_on_copies(gpu, n, tier):
    import torch
    dt, steps = 0.1, 6
    rng = np.random.default_rng(n)
    chain = torch.from_numpy(rng.standard_normal((1, n, 2))).cuda()
    out = []
    for copies in (1, 3072, 5000):   # few chains, and around and above 3 2^15 sites
        plan = gpu.Plan(gpu.Model("DNLS", n, copies, dt, beta=1.0))
        assert plan.shape()["tier"] == tier, copies
        state = chain.repeat(copies, 1, 1).contiguous()
        torch.cuda.synchronize()
        plan.move(state.data_ptr(), steps)
        torch.cuda.synchronize()
        assert torch.equal(state, state[:1].expand_as(state))
        out.append(state[:1].clone())
        plan.close()
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
