"""The windowed tiers' second state buffer: an ensemble larger than it is advanced a part of its chains at
a time, so that a plan takes little memory beside the caller's state, and every chain's bits are those
of an ensemble that fits at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n,copies,kw", [
    ("FPUT", 7000, 20000, dict(dt=0.05, alpha=0.25, beta=1.0)),
    ("DNKG", 20000, 7001, dict(dt=0.05, m=1.0, beta=1.0)),
    ("DNLS", 9000, 15011, dict(dt=0.1, beta=1.0)),
])
def test_large_ensembles_need_no_second_state(gpu, name, n, copies, kw):
    import torch
    few, state_bytes = 37, n * copies * 16
    assert state_bytes > 2 << 30
    rng = np.random.default_rng(n)
    base = torch.from_numpy(0.3 * rng.standard_normal((few, n, 2))).cuda()
    dt = kw.pop("dt")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = gpu.Plan(gpu.Model(name, n, copies, dt, flags=gpu.FLAG_NO_TUNE, **kw))
    taken = before - torch.cuda.mem_get_info()[0]
    assert plan.shape()["tier"] in (4, 6)
    assert taken < 1.25 * 2 ** 30, f"the plan took {taken / 2 ** 30:.2f} GiB beside a state of {state_bytes / 2 ** 30:.2f}"
    state = base.repeat((copies + few - 1) // few, 1, 1)[:copies].contiguous()
    torch.cuda.synchronize()
    small = gpu.Plan(gpu.Model(name, n, few, dt, flags=gpu.FLAG_NO_TUNE, **kw))
    for steps in (23, 1):   # several launches a pass, and one with a copy back
        small.move(base.data_ptr(), steps)
        plan.move(state.data_ptr(), steps)
    torch.cuda.synchronize()
    for first in range(0, copies, few):
        part = state[first:first + few]
        assert torch.equal(part, base[:len(part)]), f"chains from {first} on"
    plan.close()
    small.close()
