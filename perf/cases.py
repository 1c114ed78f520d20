"""The work that a user of glac_b200 has it do, as cases that can be timed and checked.

Every case is one pass through the package's public entry points (`Lattice`,
`Ensemble`, `ProposalNet`) on fields of the kind that lattice runs hold: SU(3)
links with a plaquette of about 0.6 (a thermalised field at beta = 6.0-6.2 has
0.59-0.61), hidden by a random gauge transformation so that single links look
Haar distributed.  Fields come from the seed alone.

Kinds of pass:
  flow      gradient flow of a copy of the chain's field, n RK3 steps, with the
            plaquette / charge / energy after every step or without
  sweeps    Metropolis sweeps of the chain, by the fixed spread or the learned one
  measure   plaquette / charge / energy of the chain's field
  weinberg  the same with the Weinberg operator
  load      a configuration from host memory: upload, flow, download
  ensemble  uneven lattices together: sweeps, then the flow of their copies
  train     Adam steps of the learned proposal spread
  forward   spreads of many rows by the network
  esj       training rows (expected squared jumps) from a chain's field

Results of a single-precision context are returned in single precision: that
is what they hold.
"""
import math

import numpy as np
import torch

import glac_b200
from glac_b200.ensemble import Ensemble, draw_ensemble
from glac_b200.learned import DEFAULT_GRID, ProposalNet

SPREAD = 0.31  # width of the links about 1 before the gauge transformation: plaquette about 0.6


def listed():
    return [
        # Scale-setting flow at the benchmark's lattice: every step measured.
        dict(name="flow_fp32_32x64", kind="flow", dims="32,32,32,64", precision="fp32", steps=6, measured=True),
        # The same in double precision (the default) at the middle lattice of a continuum series.
        dict(name="flow_fp64_24x48", kind="flow", dims="24,24,24,48", precision="fp64", steps=3, measured=True),
        # A short flow on a lattice of a test run: launches and latency.
        dict(name="flow_fp32_8x16", kind="flow", dims="8,8,8,16", precision="fp32", steps=20, measured=True),
        # Flow to a fixed time between topological-charge samples, extents that no block size divides.
        dict(name="flow_fp32_ragged", kind="flow", dims="18,20,22,42", precision="fp32", steps=8, measured=False),
        # Updates between measurements, the bulk of a production chain in single precision.
        dict(name="sweeps_fp32_24x48", kind="sweeps", dims="24,24,24,48", precision="fp32", sweeps=2, learned=False),
        # The default, double precision, at a lattice of a quick study.
        dict(name="sweeps_fp64_16x32", kind="sweeps", dims="16,16,16,32", precision="fp64", sweeps=4, learned=False),
        # Updates with the network's spreads.
        dict(name="sweeps_learned_24x48", kind="sweeps", dims="24,24,24,48", precision="fp32", sweeps=2, learned=True),
        # The measurement that a chain takes after every sweep.
        dict(name="measure_fp64_24x48", kind="measure", dims="24,24,24,48", precision="fp64"),
        dict(name="measure_fp32_32x64", kind="measure", dims="32,32,32,64", precision="fp32"),
        # Flow of a stored configuration: host array in, flowed host array out.
        dict(name="load_fp64_12x24", kind="load", dims="12,12,12,24", precision="fp64", steps=10),
        # Twelve lattices of a coupling scan advanced together.
        dict(name="ensemble_fp32_12", kind="ensemble", lattices=12, draw=7, precision="fp32", sweeps=4, steps=6),
        # Fit of the proposal network to collected rows.
        dict(name="train_8192", kind="train", rows=131072, batch=8192, steps=100),
    ]


def draw(rng):
    kind = rng.choice(("flow", "flow", "flow", "sweeps", "sweeps", "measure", "weinberg", "load", "ensemble", "train",
                       "forward", "esj"))
    if kind == "ensemble":
        return dict(kind=kind, lattices=rng.randint(2, 16), draw=rng.randint(1, 10**6), precision="fp32",
                    sweeps=rng.randint(1, 4), steps=rng.randint(1, 6))
    if kind == "train":
        batch = int(2 ** rng.uniform(8, 15))
        return dict(kind=kind, rows=batch * rng.randint(1, 12) + rng.randint(0, 99), batch=batch,
                    steps=rng.randint(10, 100))
    if kind == "forward":
        return dict(kind=kind, rows=int(2 ** rng.uniform(10, 21)))
    precision = rng.choice(("fp32", "fp64"))
    # volumes spread over their logarithm, 4^3 x 8 to 32^3 x 64 (in double precision to half of that)
    top = {"flow": 21.0, "sweeps": 20.0, "measure": 21.0, "weinberg": 19.0, "load": 16.0, "esj": 20.0}[kind]
    volume = 2 ** rng.uniform(9.5, top - (precision == "fp64"))
    dims = []
    for k in range(4):
        side = volume ** 0.25 * 2 ** rng.uniform(-0.5, 0.5) if k < 3 else volume / math.prod(dims)
        dims.append(min(128, max(4, 2 * round(side / 2))))
    while math.prod(dims) > volume * 1.1 and dims[3] > 4:
        dims[3] -= 2
    case = dict(kind=kind, dims=",".join(map(str, dims)), precision=precision)
    if kind == "flow":
        case.update(steps=rng.randint(1, 6), measured=rng.random() < 0.7)
    elif kind == "sweeps":
        case.update(sweeps=rng.randint(1, 2), learned=precision == "fp32" and rng.random() < 0.4)
    elif kind == "load":
        case.update(steps=rng.randint(1, 10))
    elif kind == "esj":
        case.update(stride=rng.choice((16, 64)), trials=rng.randint(1, 4))
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dims(case):
    return tuple(int(x) for x in case["dims"].split(","))


def _su3(m):
    """The SU(3) matrix of the first two rows of m (..., 3, 3): orthonormal rows, the third their conjugate cross product."""
    a = m[..., 0, :]
    a = a / torch.linalg.vector_norm(a, dim=-1, keepdim=True)
    b = m[..., 1, :]
    b = b - (a.conj() * b).sum(-1, keepdim=True) * a
    b = b / torch.linalg.vector_norm(b, dim=-1, keepdim=True)
    return torch.stack((a, b, torch.linalg.cross(a, b).conj()), dim=-2)


def _shift(u, mu, by):
    """u at n + by e_mu, for fields (Nt, Nz, Ny, Nx, ...)."""
    return torch.roll(u, -by, 3 - mu)


def _links(dims, seed):
    """(4, V, 18) float64 links on the GPU."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    shape = (dims[3], dims[2], dims[1], dims[0], 3, 3)

    def gauss():
        return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=gen)

    one = torch.eye(3, dtype=torch.complex128, device="cuda")
    g = _su3(gauss())
    out = torch.empty((4,) + shape, dtype=torch.complex128, device="cuda")
    for mu in range(4):
        out[mu] = g @ _su3(one + SPREAD * gauss()) @ _shift(g, mu, 1).mH
    return torch.view_as_real(out).reshape(4, -1, 18)


def _params(rng):
    """Network parameters as a training run starts from: He-normal layers, a small output layer."""
    p = np.zeros(glac_b200.MLP_NPARAMS, np.float32)
    p[0:256] = rng.standard_normal(256) * math.sqrt(2 / 8)
    p[288:1312] = rng.standard_normal(1024) * math.sqrt(2 / 32)
    p[1344:1376] = rng.standard_normal(32) * 0.05
    s = (0.24 - DEFAULT_GRID[0]) / (DEFAULT_GRID[-1] - DEFAULT_GRID[0])
    p[1376] = math.log(s / (1 - s))
    return p


def _rows(rows, seed):
    """Features and expected squared jumps with the ranges that collected rows have."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    f = torch.randn((rows, 8), device="cuda", generator=gen) * 0.3
    f[:, 0] += 2.0
    f[:, 6].mul_(0.2).add_(0.13)
    f[:, 7] = 0.03
    grid = torch.as_tensor(DEFAULT_GRID, dtype=torch.float32, device="cuda")
    peak = 0.25 * torch.exp(0.4 * f[:, 1:2])
    esj = grid * grid * torch.exp(-grid / peak) * (1 + 0.2 * torch.rand((rows, len(grid)), device="cuda", generator=gen))
    return f.contiguous(), (esj / esj.mean()).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(int(seed))
    if kind == "train":
        net = ProposalNet()
        features, esj = _rows(case["rows"], seed)
        return dict(case, net=net, params=_params(rng), features=features, esj=esj)
    if kind == "forward":
        net = ProposalNet()
        net.params = _params(rng)
        return dict(case, net=net, features=_rows(case["rows"], seed)[0])
    if kind == "ensemble":
        dims, betas = draw_ensemble(case["draw"], case["lattices"])
        E = Ensemble(dims, betas, precision=case["precision"], seed=int(seed))
        for i, d in enumerate(dims):
            E.set_links(i, _links(d, 1000 * int(seed) + i).cpu().numpy())
        return dict(case, ensemble=E)
    dims = _dims(case)
    links = _links(dims, seed)
    if kind == "load":
        return dict(case, flow=glac_b200.Lattice(dims, beta=6.0, precision=case["precision"]), links=links.cpu().numpy())
    L = glac_b200.Lattice(dims, beta=6.0, precision=case["precision"], seed=int(seed))
    torch.cuda.synchronize()
    L.set_links_device(links.data_ptr())
    L.sync()
    s = dict(case, chain=L, stream=torch.cuda.ExternalStream(L.stream))
    if kind == "flow":
        F = glac_b200.Lattice(dims, beta=6.0, precision=case["precision"])
        s.update(flow=F, stream=torch.cuda.ExternalStream(F.stream), links=links)
    elif kind == "sweeps":
        s.update(links=links)
        if case["learned"]:
            L.set_option("su2_sign_flips", 0)
            L.set_proposal_net(_params(rng), DEFAULT_GRID[0], DEFAULT_GRID[-1])
    elif kind == "esj":
        n = L.esj_rows(case["stride"])
        s.update(features=torch.empty((n, 8), device="cuda"), esj=torch.empty((n, len(DEFAULT_GRID)), device="cuda"))
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _field(L, s):
    """The lattice's links in the state's buffer, in the precision of the lattice."""
    L.get_links_device(s["links"].data_ptr())
    out = s["links"]
    if s["precision"] == "fp32":
        with torch.cuda.stream(s["stream"]):
            out = out.float()
    L.sync()
    return out


def _obs(s, obs):
    return obs.astype(np.float32) if s["precision"] == "fp32" else obs


def run(s):
    kind = s["kind"]
    if kind == "flow":
        F = s["flow"]
        F.copy_from(s["chain"])
        obs = F.flow(s["steps"], measure=s["measured"])
        links = _field(F, s)
        return {"links": links, "obs": _obs(s, obs)} if s["measured"] else {"links": links}
    if kind == "sweeps":
        acceptance = s["chain"].metropolis(s["sweeps"])
        return {"links": _field(s["chain"], s), "acceptance": acceptance}
    if kind == "measure":
        return {"obs": _obs(s, s["chain"].measure())}
    if kind == "weinberg":
        return {"obs": _obs(s, s["chain"].measure_weinberg())}
    if kind == "load":
        F = s["flow"]
        F.set_links(s["links"])
        obs = F.flow(s["steps"])
        return {"links": _obs(s, F.get_links()), "obs": _obs(s, obs)}
    if kind == "ensemble":
        acceptance, obs, _ = s["ensemble"].run(s["sweeps"], s["steps"])
        return {"acceptance": acceptance.astype(np.float32), "obs": [_obs(s, o) for o in obs]}
    if kind == "train":
        net = s["net"]
        net.params = s["params"]
        losses = net.train(s["features"], s["esj"], DEFAULT_GRID, s["steps"], s["batch"], 2e-3)
        return {"losses": losses.astype(np.float32), "params": net.params}
    if kind == "forward":
        return {"spreads": s["net"].forward(s["features"], DEFAULT_GRID[0], DEFAULT_GRID[-1])}
    s["chain"].esj_data_ptr(DEFAULT_GRID, s["trials"], s["stride"], 3, s["features"].data_ptr(), s["esj"].data_ptr(),
                            None, s["features"].shape[0])
    return {"features": s["features"], "esj": s["esj"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# Multiply-adds: a complex 3x3 product 108, one of which only the traceless
# anti-Hermitian part is wanted 90.
FULL, PART = 108, 90
# An RK3 stage per site: per plane two two-link products, three loops for the forces of its four links
# (one base corner is shared); per link the exponential's polynomial and the link update.
STAGE = 6 * (3 * FULL + 3 * PART) + 4 * (150 + FULL)
# A measurement per site: per plane the plaquette's four loops; six traces.
CLOVER = 6 * (4 * FULL + 4 * PART) + 9 * 10
# A Metropolis link update: the staple (half of its products shared at best), ten hits of a proposal matrix,
# two random-number blocks and one trace.
STAPLE, HIT = 6 * 2 * FULL, 45 + 6 * 12 + 18 + 40


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = min(case["batch"], case["rows"]) * case["steps"]
        return {"bytes": rows * (8 + 16) * 4.0, "flops": 6.0 * rows * (8 * 32 + 32 * 32 + 32)}
    if kind == "forward":
        return {"bytes": case["rows"] * 36.0, "flops": 2.0 * case["rows"] * (8 * 32 + 32 * 32 + 32)}
    real = 8 if case["precision"] == "fp64" else 4
    if kind == "ensemble":
        V = sum(math.prod(d) for d in draw_ensemble(case["draw"], case["lattices"])[0])
    else:
        V = math.prod(_dims(case))
    links = 4.0 * 18 * real * V
    force = 4.0 * 8 * real * V

    def flow(steps):
        return steps * (6 * links + 4 * force), 2.0 * V * steps * 3 * STAGE

    def sweeps(n):  # a sub-sweep of one direction and parity reads all four directions about it once
        return n * 8 * (1.125 * links), 2.0 * 4 * V * n * (STAPLE + 10 * HIT)

    b = f = 0.0
    if kind == "flow":
        b, f = flow(case["steps"])
        b += links + 4 * 18 * 8 * V
        f += 2.0 * V * CLOVER * (case["steps"] + 1) * case["measured"]
    elif kind == "sweeps":
        b, f = sweeps(case["sweeps"])
        b += links + 4 * 18 * 8 * V
    elif kind in ("measure", "weinberg"):
        b, f = links, 2.0 * V * CLOVER
    elif kind == "load":
        b, f = flow(case["steps"])
        b += 4 * 4 * 18 * 8.0 * V + 2 * links
        f += 2.0 * V * CLOVER * (case["steps"] + 1)
    elif kind == "ensemble":
        b, f = (x + y for x, y in zip(sweeps(case["sweeps"]), flow(case["steps"])))
        f += 2.0 * V * CLOVER * (case["steps"] + 1)
    elif kind == "esj":
        rows = 4.0 * V / case["stride"]
        b, f = min(links, rows * 19 * 18 * real) + rows * 96, 2.0 * rows * (STAPLE + 16 * case["trials"] * 10 * HIT)
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# the values in 64 bits
# ---------------------------------------------------------------------------
def _observables(U, weinberg=False):
    """[plaq, topc, energy, topct[Nt]] (or [plaq, topc, energy, weinberg, topct, weinbergt]) of (4, Nt, Nz, Ny, Nx, 3, 3) links."""
    V = U[0, ..., 0, 0].numel()
    F, plaq = {}, 0.0
    for mu in range(4):
        for nu in range(mu + 1, 4):
            A, B = U[mu], U[nu]
            Bm, An = _shift(B, mu, 1), _shift(A, nu, 1)
            P = A @ Bm @ An.mH @ B.mH
            plaq = plaq + torch.diagonal(P, dim1=-2, dim2=-1).sum().real
            # the plaquette's loops about its other corners, moved to the site they start at
            C = P + _shift(Bm @ An.mH @ B.mH @ A, mu, -1) + _shift(B.mH @ A @ Bm @ An.mH, nu, -1) \
                + _shift(_shift(An.mH @ B.mH @ A @ Bm, mu, -1), nu, -1)
            D = C - C.mH
            D = D - torch.diagonal(D, dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * torch.eye(3, device=U.device, dtype=U.dtype)
            F[mu, nu], F[nu, mu] = D, -D

    def tr(x, y):  # per time slice
        return (x * y.transpose(-1, -2)).sum((1, 2, 3, 4, 5)).real

    q = -sum(tr(F[0, n], F[n % 3 + 1, (n + 1) % 3 + 1]) for n in (1, 2, 3)) / (256 * math.pi ** 2)
    e = sum(tr(F[m, n], F[m, n]).sum() for m in range(4) for n in range(m + 1, 4)) / V
    out = [plaq / (18 * V), q.sum(), e]
    if not weinberg:
        return torch.cat([torch.stack(out), q]).cpu().numpy()
    w = 0.0
    for n in (1, 2, 3):
        acc = sum(F[0, m] @ F[n, m] for m in (1, 2, 3) if m != n)
        w = w - tr(acc, F[n % 3 + 1, (n + 1) % 3 + 1])
    w = w * 2 * 64 / (3 * 16 ** 3)
    return torch.cat([torch.stack(out + [w.sum()]), q, w]).cpu().numpy()


def _force(U, mu):
    """The traceless anti-Hermitian part of U_mu times its staples, with the flow's sign."""
    A = torch.zeros_like(U[mu])
    for nu in range(4):
        if nu != mu:
            B, Bm = U[nu], _shift(U[nu], mu, 1)
            A += Bm @ _shift(U[mu], nu, 1).mH @ B.mH
            A += _shift(Bm.mH @ U[mu].mH @ B, nu, -1)
    X = U[mu] @ A
    D = X.mH - X
    return 0.5 * (D - torch.diagonal(D, dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * torch.eye(3, device=U.device, dtype=U.dtype))


def _expm(M):
    one = torch.eye(3, device=M.device, dtype=M.dtype)
    E = one + M / 16
    for k in range(15, 0, -1):
        E = one + M @ E / k
    return E


def _flow_step(U, eps):
    Z0 = torch.stack([_force(U, mu) for mu in range(4)])
    W1 = torch.stack([_expm(eps / 4 * Z0[mu]) @ U[mu] for mu in range(4)])
    M1 = torch.stack([8 / 9 * eps * _force(W1, mu) - 17 / 36 * eps * Z0[mu] for mu in range(4)])
    del Z0
    W2 = torch.stack([_expm(M1[mu]) @ W1[mu] for mu in range(4)])
    del W1
    return torch.stack([_expm(0.75 * eps * _force(W2, mu) - M1[mu]) @ W2[mu] for mu in range(4)])


def exact(case, seed):
    if case["kind"] not in ("flow", "load", "measure", "weinberg"):
        return None  # accept decisions and rounded operands: no value in 64 bits
    dims = _dims(case)
    if math.prod(dims) * (1 + 6 * case.get("steps", 0)) > 1e8:
        return None
    U = _links(dims, seed)
    U = torch.view_as_complex(U.reshape(4, dims[3], dims[2], dims[1], dims[0], 3, 3, 2))
    if case["kind"] == "measure":
        return {"obs": _observables(U)}
    if case["kind"] == "weinberg":
        return {"obs": _observables(U, True)}
    measured = case.get("measured", True)
    obs = [_observables(U)] if measured else []
    for _ in range(case["steps"]):
        U = _flow_step(U, 0.01)
        if measured:
            obs.append(_observables(U))
    out = {"links": torch.view_as_real(U).reshape(4, -1, 18)}
    if case["kind"] == "load":
        out["links"] = out["links"].cpu().numpy()
    if measured:
        out["obs"] = np.stack(obs)
    return out
