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


# radix 4 only, with a 2, 3, 5 and 7 (direct) pass, padded; warp teams and blocks.  7000 chains fill the
# schedulers, so the transforms' first additions run on the integer pipes, as 5 chains' do not
@pytest.mark.parametrize("n", [16, 28, 32, 60, 64, 96, 256, 500, 512, 1009])
@pytest.mark.parametrize("zeros", [False, True])
def test_fourier_form_bits_do_not_depend_on_copies(gpu, n, zeros):
    import torch
    few, many = 5, 7000
    psi = np.random.default_rng(n).standard_normal((few, n, 2))
    if zeros:   # sums that the integer pipes do not take
        psi[:, n // 3:] = 0.
    base = torch.from_numpy(psi).cuda()
    out = []
    for copies in (few, many):
        plan = gpu.Plan(gpu.Model("DNLS", n, copies, 0.02, beta=1.0, flags=gpu.FLAG_DNLS_FOURIER))
        assert plan.shape()["tier"] == 3
        state = base.repeat(copies // few, 1, 1).contiguous()
        torch.cuda.synchronize()
        plan.move(state.data_ptr(), 4)
        torch.cuda.synchronize()
        out.append(state)
        plan.close()
    assert torch.equal(out[1], out[0].repeat(many // few, 1, 1))
