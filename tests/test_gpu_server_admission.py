"""Admission counts what a plan holds: two dDNKG requests whose projection splits its tiles (and so holds the
parts' sums) run one after the other under a budget that has room for one."""
import numpy as np
import pytest

from nlchains_gb300 import ic

pytestmark = pytest.mark.gpu


def test_projection_parts_are_counted(gpu):
    # 72 MB each: slices 22, parked sums 16 and parts' sums 16, eigenvectors 8, state 4, partial rows and tables 5;
    # without the parts and the parked sums of more than whole tiles 44
    n, copies, budget = 1024, 256, 100 << 20
    model = gpu.Model("dDNKG", n, copies, 0.05, masses=ic.masses_uniform(n, seed=1), beta=1.0)
    state = 0.3 * np.random.default_rng(2).standard_normal((copies, n, 2))
    srv = gpu.Server(0, hbm_budget_bytes=budget)
    ids = [srv.submit(model, 1000, 10000, state) for _ in range(2)]
    for rid in ids:
        srv.wait(rid)
    first, second = (srv.poll(rid) for rid in ids)
    srv.close()
    assert second["start_ms"] >= first["finish_ms"]
