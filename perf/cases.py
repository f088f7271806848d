"""The work that a user of this engine has it do, as cases to be timed.

A production run is the reference's main loop: batches of `kernel_batching` Yoshida steps of a whole
ensemble, a diagnostics sample (linear-mode energies and the two entropies) after each, and at the
start a seeded ensemble.  Every case calls the public Python binding of the C ABI as such a program
does, on state that the caller keeps on the GPU (or, for `job`, through the job API with its
read-back).  Kinds of case:

  job     one loop iteration through the job API: the batch and its sample replayed as one graph,
          the mode energies, the entropies and the state read back to the host
  step    one loop iteration through the operators: nlc_move, then nlc_linenergies
  move    the batch alone (loops that sample rarely)
  sample  the diagnostics alone (post-processing of stored ensembles, sampling every few steps)
  seed    a seeded initial ensemble and the energy of each of its chains

States are partly thermalised ensembles: most of the energy in the lowest modes, every mode excited.
"""
import math
import os

import numpy as np
import torch

import nlchains_gb300 as nlc

# launch shapes that the engine's tuner measures are kept beside the library they were measured on
os.environ.setdefault("NLC_TUNE_CACHE", os.path.join(os.path.dirname(nlc.__file__), "_build", "shapes.tsv"))


def _case(name, kind, model, n, copies, steps=0, dt=0.05, m=0.0, alpha=0.0, beta=0.0):
    return {"name": name, "kind": kind, "model": model, "n": n, "copies": copies, "steps": steps, "dt": dt, "m": m,
            "alpha": alpha, "beta": beta}


def listed():
    return [
        # the smallest runs: a first look at a parameter set, where latency and launches count
        _case("fput_job_64x96", "job", "FPUT", 64, 96, 10, 0.1, beta=1.0),
        # FPUT-beta recurrence studies: short chains, a thousand realisations, a sample per 100 steps
        _case("fput_step_64x1024", "step", "FPUT", 64, 1024, 100, 0.1, beta=1.0),
        # the production ensemble: nonlinear Klein-Gordon, 65536 realisations
        _case("dnkg_move_128x65536", "move", "DNKG", 128, 65536, 100, m=1.0, beta=1.0),
        # Toda, whose exponential dominates
        _case("toda_step_128x16384", "step", "Toda", 128, 16384, 100, alpha=0.5),
        # disordered Klein-Gordon: per-site masses, eigenbasis projection at every sample
        _case("ddnkg_step_256x4096", "step", "dDNKG", 256, 4096, 100, beta=1.0),
        # DNLS wave turbulence at its usual small time step
        _case("dnls_step_1024x8192", "step", "DNLS", 1024, 8192, 10, 0.01, beta=1.0),
        # DNLS at a large time step, a length that is not a power of two
        _case("dnls_step_500x1024_dt0.1", "step", "DNLS", 500, 1024, 20, 0.1, beta=1.0),
        # an odd length with both nonlinearities and a ragged number of copies
        _case("fput_step_459x3001_alpha", "step", "FPUT", 459, 3001, 50, 0.05, alpha=0.25, beta=0.5),
        # few very long chains
        _case("dnkg_step_20000x96", "step", "DNKG", 20000, 96, 50, m=1.0, beta=1.0),
        # diagnostics of the production ensemble
        _case("dnkg_sample_128x65536", "sample", "DNKG", 128, 65536, m=1.0, beta=1.0),
        # diagnostics of long disordered chains: the one dense contraction
        _case("ddnkg_sample_1024x4096", "sample", "dDNKG", 1024, 4096, beta=1.0),
        # setting up a production ensemble on the device and checking its energies
        _case("fput_seed_128x65536", "seed", "FPUT", 128, 65536, alpha=0.25, beta=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("job", "step", "step", "step", "move", "sample", "sample", "seed"))
    model = rng.choice(("DNKG", "FPUT", "Toda", "dDNKG", "DNLS"))
    n = _log_int(rng, 16, 1024 if model == "dDNKG" else 20000)
    if kind == "job":   # its state goes to the host: small ensembles
        n = min(n, 2048)
    copies = max(1, min(65536, _log_int(rng, 4096, 1 << (18 if kind == "job" else 23)) // n))
    steps = 0 if kind in ("sample", "seed") else rng.randint(1, 100)
    c = {"kind": kind, "model": model, "n": n, "copies": copies, "steps": steps, "dt": 0.05, "m": 0.0, "alpha": 0.0,
         "beta": 0.0}
    if model == "DNKG":
        c.update(m=rng.choice((0.0, 0.5, 1.0)), beta=rng.choice((0.5, 1.0)))
    elif model == "FPUT":
        c.update(dt=rng.choice((0.05, 0.1)), alpha=rng.choice((0.0, 0.25)), beta=rng.choice((0.5, 1.0)))
    elif model == "Toda":
        c.update(alpha=rng.choice((0.5, 0.75)))
    elif model == "dDNKG":
        c.update(beta=rng.choice((0.5, 1.0)))
    else:
        c.update(dt=rng.choice((0.01, 0.02, 0.1)), beta=1.0)
    # no more work than the production batch, with room for the lengths whose transforms cost most
    most = 0.2 * work(listed()[2])["flops"]
    while steps > 1 and work(c)["flops"] > most:
        steps = c["steps"] = steps // 2
    return c


# ---------------------------------------------------------------------------------------------------------------------


def _omega(c, device="cpu"):
    s = 2 * torch.sin(torch.arange(c["n"], dtype=torch.float64) * (math.pi / c["n"]))
    w2 = s * s + (c["m"] if c["model"] == "DNKG" else 0.0)
    return (w2 if c["model"] == "DNLS" else w2.sqrt()).to(device)


def _masses(c, seed):
    return np.random.RandomState(seed % (1 << 31)).uniform(1.0, 3.0, c["n"]) if c["model"] == "dDNKG" else None


def _state(c, seed):
    """[copies, n, 2]: (phi, pi), or psi as (re, im)."""
    n, copies = c["n"], c["copies"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.minimum(torch.arange(n), n - torch.arange(n)).to("cuda", torch.float64)
    weight = torch.where(k <= max(1.0, 0.05 * n), 1.0, 0.05)
    z = torch.randn(copies, n, 2, dtype=torch.float64, device="cuda", generator=g)
    if c["model"] == "DNLS":
        psi = torch.fft.ifft(torch.view_as_complex(z) * weight)
        return torch.view_as_real(psi * psi.abs().square().mean().rsqrt()).contiguous()
    w = torch.fft.fft(z, dim=1) * weight[:, None]
    om = _omega(c, "cuda") if c["model"] != "dDNKG" else torch.full((n,), 1.5, dtype=torch.float64, device="cuda")
    w[:, :, 0] *= torch.where(om > 0, 1 / om.clamp(min=1e-300), 0.0)   # phi_k = (momentum-like amplitude) / omega_k
    s = torch.fft.ifft(w, dim=1).real
    return (s * (0.4 * s[:, :, 1].square().mean().rsqrt())).contiguous()


def _seed_modes(c):
    n = c["n"]
    if c["model"] == "dDNKG":
        return list(range(max(2, n // 12)))
    kmax = max(1, min(int(0.04 * n), (n - 1) // 2))
    return [k for k in sorted({0} | set(range(1, kmax + 1)) | {n - k for k in range(1, kmax + 1)})
            if c["model"] == "DNLS" or c["m"] > 0 or k]


def prepare(case, seed):
    c = case
    model = nlc.Model(c["model"], c["n"], c["copies"], c["dt"], m=c["m"], alpha=c["alpha"], beta=c["beta"],
                      masses=_masses(c, seed))
    s = {"case": c, "seed": seed}
    if c["kind"] == "job":
        s["ctx"] = nlc.Context(0)
        s["job"] = s["ctx"].job(model, c["steps"])
        s["job"].upload(_state(c, seed).cpu().numpy())
        return s
    s["plan"] = nlc.Plan(model)
    if c["kind"] == "seed":
        s["state"] = torch.empty(c["copies"], c["n"], 2, dtype=torch.float64, device="cuda")
        s["energies"] = torch.empty(c["copies"], dtype=torch.float64, device="cuda")
        s["modes"] = np.array(_seed_modes(c), dtype=np.uint32)
        return s
    s["state"] = _state(c, seed)
    s["lin"] = torch.empty(c["n"], dtype=torch.float64, device="cuda")
    s["entropies"] = torch.empty(2, dtype=torch.float64, device="cuda")
    torch.cuda.current_stream().synchronize()
    return s


def run(state):
    s, kind = state, state["case"]["kind"]
    if kind == "job":
        s["job"].step_async(0, copy_state=True)
        lin, wt, inf, x = s["job"].sample_wait(0, with_state=True)
        return {"state": x, "lin": lin, "entropies": np.array([wt, inf])}
    stream = torch.cuda.current_stream().cuda_stream
    plan, x = s["plan"], s["state"]
    if kind == "seed":
        plan.initial_state(x.data_ptr(), s["seed"], 0.5, s["modes"], stream=stream)
        plan.energies(x.data_ptr(), s["energies"].data_ptr(), stream=stream)
        return {"state": x, "energies": s["energies"]}
    if kind != "sample":
        plan.move(x.data_ptr(), s["case"]["steps"], stream=stream)
        if kind == "move":
            return {"state": x}
    plan.linenergies(x.data_ptr(), s["lin"].data_ptr(), s["entropies"].data_ptr(), stream=stream)
    out = {"lin": s["lin"], "entropies": s["entropies"]}
    return out if kind == "sample" else {"state": x, **out}


# floating-point operations of a site's step in the reference's algorithm: 7 sub-steps of a drift, the force and a kick
# (an exponential counts as 8); a DNLS sub-step is a phase rotation and two transforms
_FLOPS = {"DNKG": 70, "dDNKG": 70, "FPUT": 91, "Toda": 112}


def work(case):
    c, n, copies = case, case["n"], case["copies"]
    sites, lg = n * copies, math.log2(n)
    flops, bytes_ = 0.0, 0.0
    if c["steps"]:
        per = _FLOPS[c["model"]] if c["model"] != "DNLS" else 7 * (10 * lg + 16)
        flops += float(sites) * c["steps"] * per
        bytes_ += 32.0 * sites
    if c["kind"] in ("job", "step", "sample"):
        flops += float(sites) * (4 * n + 4 if c["model"] == "dDNKG" else 5 * lg + 10)
        bytes_ += 8.0 * n + 16 + (8.0 * n * n if c["model"] == "dDNKG" else 0.0)
        if c["kind"] == "sample":
            bytes_ += 16.0 * sites
    if c["kind"] == "seed":
        flops += float(sites) * ((4 * len(_seed_modes(c)) if c["model"] == "dDNKG" else 5 * lg + 10) + 10)
        bytes_ += 16.0 * sites + 8.0 * copies
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------------------------------------------------
# the same results from plain torch and numpy

# H. Yoshida, Phys. Lett. A 150 (1990) 262, sixth order, solution A, drift and kick coefficients as the reference has them
_C = (0.392256805238780, 0.510043411918458, -0.471053385409757, 0.068753168252518, 0.068753168252518,
      -0.471053385409757, 0.510043411918458, 0.392256805238780)
_D = (0.784513610477560, 0.235573213359357, -1.177679984178870, 1.315186320683906, -1.177679984178870,
      0.235573213359357, 0.784513610477560)


def _exact_move(c, s, masses):
    dt, n = c["dt"], c["n"]
    if c["model"] == "DNLS":
        psi, om = torch.view_as_complex(s.contiguous()), _omega(c, s.device)
        lin = [torch.polar(torch.ones_like(om), -dt * d * om) for d in _D]

        def rotate(v, coef):
            return v * torch.polar(torch.ones_like(v.real), -c["beta"] * dt * coef * v.abs().square())

        for i in range(c["steps"]):
            for k in range(7):
                psi = rotate(psi, _C[k] * (2 if i and not k else 1))
                psi = torch.fft.ifft(torch.fft.fft(psi) * lin[k])
        return torch.view_as_real(rotate(psi, _C[7]))
    x, p = s[:, :, 0].contiguous(), s[:, :, 1].contiguous()
    m = c["m"] if masses is None else torch.from_numpy(masses).to(s.device)
    for i in range(c["steps"]):
        for k in range(7):
            x += dt * _C[k] * (2 if i and not k else 1) * p
            if c["model"] in ("DNKG", "dDNKG"):
                f = torch.roll(x, 1, 1) + torch.roll(x, -1, 1) - x * (m + 2 + c["beta"] * x * x)
            else:
                d = torch.roll(x, -1, 1) - x
                g = (torch.exp(2 * c["alpha"] * d) / (2 * c["alpha"]) if c["model"] == "Toda"
                     else d * (1 + d * (c["alpha"] + c["beta"] * d)))
                f = g - torch.roll(g, 1, 1)
            p += dt * _D[k] * f
    x += dt * _C[7] * p
    return torch.stack((x, p), 2)


def _eigensystem(masses):
    n = len(masses)
    h = np.diag(masses + 2.0)
    for i in range(n):
        h[i, (i + 1) % n] -= 1.0
        h[(i + 1) % n, i] -= 1.0
    w2, v = np.linalg.eigh(h)
    return np.sqrt(w2), v


def _exact_sample(c, s, masses):
    n, copies = c["n"], c["copies"]
    a0is0 = c["model"] != "dDNKG" and not (c["model"] == "DNKG" and c["m"])
    if c["model"] == "dDNKG":
        om, v = (torch.from_numpy(a).to(s.device) for a in _eigensystem(masses))
        lin = ((om * (s[:, :, 0] @ v)).square() + (s[:, :, 1] @ v).square()).sum(0) * (0.5 / copies)
    elif c["model"] == "DNLS":
        lin = _omega(c, s.device) * torch.fft.fft(torch.view_as_complex(s.contiguous())).abs().square().sum(0) / (copies * n)
    else:
        z = _omega(c, s.device) * torch.fft.fft(s[:, :, 0]) + 1j * torch.fft.fft(s[:, :, 1])
        lin = z.abs().square().sum(0) * (0.5 / (copies * n))
    if a0is0:
        lin[0] = 0.0
    e = lin[1:] if a0is0 else lin
    r = e * (len(e) / e.sum())
    return lin, torch.stack((-r.log().sum(), (r * r.log()).sum()))


def _splitmix(x):
    z = x + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _exact_seed(c, seed, masses):
    """The documented recipe of nlc_initial_state (include/nlchains.h), and the energy of each chain."""
    n, copies, eps = c["n"], c["copies"], 0.5
    modes = np.array(_seed_modes(c))
    stream = {"DNLS": 2, "dDNKG": 3}.get(c["model"], 1)
    key = _splitmix(np.array([(seed * 0xD1B54A32D192ED03 + stream) & (2 ** 64 - 1)], dtype=np.uint64))
    index = np.arange(copies, dtype=np.uint64)[:, None] * np.uint64(n) + modes[None, :].astype(np.uint64)
    theta = 2 * np.pi * ((_splitmix(key + index) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53)
    if c["model"] == "dDNKG":
        return None   # an eigenvector's sign is the solver's choice
    z = torch.zeros(copies, n, dtype=torch.complex128)
    phase = torch.polar(torch.ones(theta.shape, dtype=torch.float64), torch.from_numpy(theta))
    if c["model"] == "DNLS":
        z[:, modes] = math.sqrt(n * n * eps / len(modes)) * phase
        return torch.view_as_real(torch.fft.ifft(z.cuda()))
    om = _omega(c)
    z[:, modes] = math.sqrt(2 * n * eps * n / len(modes)) * phase
    z = z.cuda()
    zc = torch.roll(z.flip(1), 1, 1).conj()
    om = om.cuda()
    phi = torch.where(om > 0, (z + zc) / (2 * om.clamp(min=1e-300)), 0)
    return torch.stack((torch.fft.ifft(phi).real, torch.fft.ifft((z - zc) / 2j).real), 2)


def _exact_energies(c, s, masses):
    d = torch.roll(s, -1, 1) - s
    if c["model"] == "DNLS":
        return (d.square().sum(2) + c["beta"] / 2 * s.square().sum(2).square()).sum(1)
    q, p, d = s[:, :, 0], s[:, :, 1], d[:, :, 0]
    e = p.square() / 2
    if c["model"] == "Toda":
        x = 2 * c["alpha"] * d
        return (e + (torch.expm1(x) - x) / (4 * c["alpha"] ** 2)).sum(1)
    if c["model"] == "FPUT":
        return (e + d ** 2 / 2 + c["alpha"] * d ** 3 / 3 + c["beta"] * d ** 4 / 4).sum(1)
    m = c["m"] if masses is None else torch.from_numpy(masses).to(s.device)
    return (e + d ** 2 / 2 + m * q ** 2 / 2 + c["beta"] * q ** 4 / 4).sum(1)


def exact(case, seed):
    c, masses = case, _masses(case, seed)
    if c["kind"] == "seed":
        s = _exact_seed(c, seed, masses)
        return {"state": s, "energies": None if s is None else _exact_energies(c, s, masses)}
    s = _state(c, seed)
    out = {}
    if c["steps"]:
        s = out["state"] = _exact_move(c, s, masses)
    if c["kind"] != "move":
        lin, ent = _exact_sample(c, s, masses)
        out.update(lin=lin, entropies=ent)
    return out
