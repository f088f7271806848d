"""The integrators' integer-pipe operations (nlc_intfp.cuh) at operands where they can go wrong: bit for
bit against the oracle, whose operations are the FP64 unit's.  Each ensemble mixes chains at rest, one
excited site, exact nodes and equal neighbours (sums of zero, deep cancellation), dyadic values (ties),
neighbours 2^40 apart, subnormal and very small values, and amplitudes beyond the squares' range."""
import os

import numpy as np
import pytest

import oracle as O
from nlchains_gb300 import ic

pytestmark = pytest.mark.gpu


def edge_states(n, seed):
    r = np.random.RandomState(seed)
    s = np.arange(n)
    rows = []

    def add(phi, pi=None):
        rows.append(np.stack((phi, np.zeros(n) if pi is None else pi), 1))

    add(np.zeros(n))
    add(np.where(s == n // 3, 0.3, 0.0))
    add(-np.zeros(n), np.where(s == 0, -0.25, -0.0))
    add(0.5 * np.sin(2 * np.pi * s / n), 0.1 * np.cos(2 * np.pi * s / n))
    add(np.where(s % 4 == 0, 0.5, 0.0), np.where(s % 2 == 0, 0.25, -0.25))
    add(r.randint(-8, 9, n) / 8.0, r.randint(-8, 9, n) / 16.0)
    add(np.where(s % 2 == 0, 0.7, 0.7 * 2.0 ** -40) * r.uniform(0.5, 1, n))
    add(0.3 + 1e-9 * r.standard_normal(n))
    add(0.3 * (1 + 2.0 ** -52 * r.randint(0, 4, n)))
    add(1e-310 * r.standard_normal(n), 1e-308 * r.standard_normal(n))
    add(1e-200 * r.standard_normal(n), 1e-150 * r.standard_normal(n))
    add(2.5 * r.standard_normal(n), r.standard_normal(n))
    add(r.standard_normal(n) * 10.0 ** -r.randint(0, 30, n), r.standard_normal(n) * 10.0 ** -r.randint(0, 30, n))
    add(0.4 * r.standard_normal(n), 0.4 * r.standard_normal(n))
    return np.array(rows)


# one site per lane, in a warp and in a block, two; then from four on: one warp with full lanes and short ones, up to and beyond a batch of 8, several
# chains per warp, a block
SHAPES = [(16, 16), (64, 64), (256, 256), (5, 4), (200, 128), (4, 1), (8, 1), (9, 1), (16, 1), (61, 8), (64, 8), (128, 16), (100, 8), (500, 32), (512, 64), (1000, 128)]
MODELS = [("DNKG", dict(m=1.0, beta=1.0)), ("DNKG", dict(m=0.0, beta=1.0)), ("DNKG", dict(m=-2.5, beta=1.0)), ("DNKG", dict(m=-2.0, beta=1.0)),
          ("DNKG", dict(m=0.3, beta=0.7)), ("dDNKG", dict(beta=1.0)), ("FPUT", dict(alpha=0.0, beta=1.0)),
          ("FPUT", dict(alpha=0.25, beta=0.5)), ("Toda", dict(alpha=0.5)), ("Toda", dict(alpha=0.75))]


@pytest.mark.parametrize("n,lanes", SHAPES)
@pytest.mark.parametrize("model,params", MODELS, ids=lambda v: v if isinstance(v, str) else "-".join(map(str, v.values())))
def test_bits_at_edge_operands(gpu, monkeypatch, model, params, n, lanes):
    monkeypatch.setenv("NLC_FORCE_LANES", str(lanes))
    masses = ic.masses_uniform(n, seed=n) if model == "dDNKG" else None
    if masses is not None:
        masses[n // 2] = -1.0   # an addend of 1 among those of 3 to 5
    state = edge_states(n, n)
    copies = len(state)
    ctx = gpu.Context(0)
    job = ctx.job(gpu.Model(model, n, copies, 0.05, masses=masses, **params), 4)
    job.upload(state)
    job.advance(8)
    out = job.download()
    job.close()
    ctx.close()
    exp = O.advance(O.Model(model, n, copies, 0.05, masses=masses, **params), state, 8, 4, order=O.ORDER_DEVICE)
    exp = exp.reshape(copies, n, 2)
    finite = np.isfinite(exp)
    assert np.array_equal(finite, np.isfinite(out))
    bad = (out.view(np.uint64) != exp.view(np.uint64)) & finite
    assert not bad.any(), f"rows {np.unique(np.nonzero(bad)[0])}: {np.count_nonzero(bad)} values differ"


# lanes of one, two and three sites take the integer pipes too from a few warps per scheduler on: the same
# chains, many times over
@pytest.mark.parametrize("n,lanes", [(16, 16), (64, 64), (5, 4), (200, 128), (23, 8)])
@pytest.mark.parametrize("model,params", MODELS, ids=lambda v: v if isinstance(v, str) else "-".join(map(str, v.values())))
def test_bits_of_few_sites_per_lane_in_large_ensembles(gpu, monkeypatch, model, params, n, lanes):
    monkeypatch.setenv("NLC_FORCE_LANES", str(lanes))
    masses = ic.masses_uniform(n, seed=n) if model == "dDNKG" else None
    rows = edge_states(n, n)
    reps = -(-4 * 128 * 160 // (lanes * len(rows)))   # over 4 warps for each of 160 x 4 schedulers
    copies = reps * len(rows)
    ctx = gpu.Context(0)
    job = ctx.job(gpu.Model(model, n, copies, 0.05, masses=masses, **params), 4)
    job.upload(np.tile(rows, (reps, 1, 1)))
    job.advance(4)
    out = job.download().reshape(reps, len(rows), n, 2)
    job.close()
    ctx.close()
    exp = O.advance(O.Model(model, n, len(rows), 0.05, masses=masses, **params), rows, 4, 4, order=O.ORDER_DEVICE)
    exp = exp.reshape(len(rows), n, 2)
    finite = np.isfinite(exp)
    for r in (0, reps // 2, reps - 1):
        assert np.array_equal(finite, np.isfinite(out[r]))
        bad = (out[r].view(np.uint64) != exp.view(np.uint64)) & finite
        assert not bad.any(), f"rows {np.unique(np.nonzero(bad)[0])}: {np.count_nonzero(bad)} values differ"


# sites per lane 1 .. 16 (rows over several chains of a warp, one chain of a warp, a block), every radius, and
# windows
@pytest.mark.parametrize("n,dt,sites,window", [(16, 0.01, 0, 0), (33, 0.01, 1, 0), (64, 0.01, 2, 0), (24, 0.05, 12, 0),
                                               (100, 0.05, 8, 0), (250, 0.01, 1, 0), (515, 0.01, 16, 0),
                                               (1021, 0.05, 4, 0), (1300, 0.01, 0, 64), (2100, 0.05, 0, 96),
                                               (28, 0.1, 0, 0), (200, 0.15, 4, 0), (501, 0.1, 8, 0), (2100, 0.1, 0, 96)])
def test_dnls_bits_at_edge_operands(gpu, monkeypatch, n, dt, sites, window):
    """The DNLS stencil form on the same states (phi + i pi as psi: real, imaginary and zero sites, angles on
    both sides of 2^-4 within a warp)."""
    if sites:
        monkeypatch.setenv("NLC_DNLS_SITES", str(sites))
    if window:
        monkeypatch.setenv("NLC_FORCE_WINDOW", str(window))
    state = edge_states(n, n)
    copies, steps = len(state), 2
    shape = gpu.Plan(gpu.Model("DNLS", n, copies, dt, beta=1.0)).shape()
    assert shape["tier"] == (6 if window else 5) and (not sites or shape["sites_per_lane"] == sites)
    ctx = gpu.Context(0)
    job = ctx.job(gpu.Model("DNLS", n, copies, dt, beta=1.0), steps)
    job.upload(state)
    job.advance(2 * steps)
    out = job.download()
    job.close()
    ctx.close()
    exp = O.advance(O.Model("DNLS", n, copies, dt, beta=1.0), state, 2 * steps, steps, order=O.ORDER_STENCIL)
    exp = exp.reshape(copies, n, 2)
    assert np.isfinite(exp).all()
    bad = out.view(np.uint64) != exp.view(np.uint64)
    assert not bad.any(), f"rows {np.unique(np.nonzero(bad)[0])}: {np.count_nonzero(bad)} values differ"


@pytest.mark.parametrize("model,params", [("DNKG", dict(m=1.0, beta=1.0)), ("DNKG", dict(m=0.3, beta=0.7)),
                                          ("dDNKG", dict(beta=1.0)), ("FPUT", dict(alpha=0.25, beta=0.5)),
                                          ("Toda", dict(alpha=0.5))], ids=lambda v: v if isinstance(v, str) else "")
@pytest.mark.parametrize("n,lanes", [(2049, 256), (2500, 512), (3600, 256)])
def test_chains_moved_to_windows_equal_one_block(gpu, monkeypatch, model, params, n, lanes):
    """Lengths that a block would hold but that run in windows for few chains: the same bits as on a block,
    over an odd and an even number of launches, in one batch and in several."""
    if model == "dDNKG":
        n, lanes = n // 4, 64
        monkeypatch.setenv("NLC_FORCE_WINDOW", "64")
    masses = ic.masses_uniform(n, seed=n) if model == "dDNKG" else None
    r = np.random.RandomState(n)
    state = 0.3 * r.standard_normal((3, n, 2))
    state[1, ::3] = 0.0

    def advance(batching, steps):
        ctx = gpu.Context(0)
        job = ctx.job(gpu.Model(model, n, 3, 0.05, masses=masses, **params), batching)
        job.upload(state)
        job.advance(steps)
        out = job.download()
        job.close()
        ctx.close()
        return out

    assert gpu.Plan(gpu.Model(model, n, 3, 0.05, masses=masses, **params)).shape()["tier"] == 4
    windows = [advance(b, 24) for b in (24, 8, 3)]
    monkeypatch.delenv("NLC_FORCE_WINDOW", raising=False)
    monkeypatch.setenv("NLC_FORCE_LANES", str(lanes))
    for b, w in zip((24, 8, 3), windows):
        assert np.array_equal(w.view(np.uint64), advance(b, 24).view(np.uint64)), b
