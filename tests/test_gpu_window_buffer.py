"""The windowed tiers' second state buffer: an ensemble larger than it is advanced a part of its chains at
a time, so that a plan takes little memory beside the caller's state, and every chain's bits are those
of an ensemble that fits at once."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def bytes_of_a_plan(name, n, copies, dt, kw):
    """Device memory that a plan takes, in a process of its own (this one's pool may have memory to spare)."""
    script = f'''
import sys
sys.path.insert(0, {ROOT!r})
import torch
import nlchains_gb300 as nlc
nlc.Plan(nlc.Model("FPUT", 16, 4, 0.05, alpha=0.25, beta=1.0)).close()
before = torch.cuda.mem_get_info()[0]
plan = nlc.Plan(nlc.Model({name!r}, {n}, {copies}, {dt}, flags=nlc.FLAG_NO_TUNE, **{kw!r}))
print(before - torch.cuda.mem_get_info()[0])
'''
    out = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    return int(out.stdout.split()[-1])


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
    kw = dict(kw)
    dt = kw.pop("dt")
    plan = gpu.Plan(gpu.Model(name, n, copies, dt, flags=gpu.FLAG_NO_TUNE, **kw))
    assert plan.shape()["tier"] in (4, 6)
    taken = bytes_of_a_plan(name, n, copies, dt, kw)
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


@pytest.mark.parametrize("name,limit,kw", [("DNKG", 8192, dict(m=1.0, beta=1.0)), ("FPUT", 6144, dict(alpha=0.25, beta=0.5)),
                                           ("Toda", 6144, dict(alpha=0.5)), ("dDNKG", 4096, dict(beta=1.0))])
def test_longest_chain_of_a_block(gpu, name, limit, kw):
    """The longest chain that a block holds, and one site more, which runs in windows: bit for bit the oracle's."""
    import oracle as O
    copies, steps = 2, 3
    flags = gpu.FLAG_CANONICAL_SHAPE | gpu.FLAG_NO_TUNE | (gpu.FLAG_FP64_PROJECTION if name == "dDNKG" else 0)
    for n, tier in ((limit, 2), (limit + 1, 4)):
        state = 0.3 * np.random.default_rng(n).standard_normal((copies, n, 2))
        if name == "dDNKG":
            kw = dict(kw, masses=np.random.default_rng(n + 1).uniform(1.0, 3.0, n))
        model = gpu.Model(name, n, copies, 0.05, flags=flags, **kw)
        plan = gpu.Plan(model)
        assert plan.shape()["tier"] == tier
        plan.close()
        ctx = gpu.Context(0)
        job = ctx.job(model, steps)
        job.upload(state)
        job.advance(steps)
        out = job.download()
        job.close()
        ctx.close()
        exp = O.advance(O.Model(name, n, copies, 0.05, **kw), state.copy(), steps, steps)
        assert np.array_equal(np.asarray(out), np.asarray(exp).reshape(out.shape)), n
