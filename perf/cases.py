"""The work that programs have this framework do, as cases that can be timed.

A case is a dict of plain values.  ``prepare`` makes what the program holds before the
call (states, operators, ensembles, chains), ``run`` makes one pass through the public
entry points and returns its outputs, ``work`` counts what the pass cannot do without and
``exact`` gives the outputs in 64 bits where they follow from the inputs alone.
"""
import numpy as np
import torch

import rbmongpu_gb300 as rg
from rbmongpu_gb300.autograd import energy

FLOPS_F = 44         # the rational log-cosh of one complex angle
FLOPS_PROPOSAL = 43  # one hidden unit of a Metropolis proposal


def listed():
    return [
        # a first run on a small chain: energy and gradient over every configuration
        dict(name="exact_gradient_12", kind="exact_gradient", N=12, M=24),
        # projecting one imaginary- or real-time step on a trial state, over every configuration
        dict(name="exact_distance_16", kind="exact_distance", N=16, M=32),
        # one training step of an RBM on the 8 x 8 Ising model: sweeps, energy, gradient
        dict(name="rbm_step_8x8", kind="rbm_step", N=64, M=128, lattice="square", walkers=4096, rows=20, therm=20),
        # a ragged, smaller training step on a chain (M is not a multiple of the warp)
        dict(name="rbm_step_30", kind="rbm_step", N=30, M=75, lattice="chain", walkers=1000, rows=8, therm=10),
        # a long production run: persistent walkers, sweeps and the energies of every row
        dict(name="chain_rows_100", kind="chain_rows", N=100, M=400, walkers=16384, rows=4, sweeps=2),
        # the same with the learned cluster-flip proposal, trained online and then frozen
        dict(name="learned_rows_100", kind="learned_rows", N=100, M=400, walkers=16384, rows=2, steps=20, train=4,
             train_walkers=4096),
        # measuring a Heisenberg chain in a fixed magnetisation sector
        dict(name="sector_samples_36", kind="sector_samples", N=36, M=75, walkers=2048, rows=4, therm=20),
        # energies and amplitudes of configurations that the program already has
        dict(name="configurations_75", kind="configurations", N=75, M=150, count=10007),
        # one training step of a deep net through torch.autograd
        dict(name="deep_step_100", kind="deep_step", N=100, layers="200,100,50", walkers=8192, therm=3),
        # the reference's own gradient estimator of a small deep net
        dict(name="deep_gradient_20", kind="deep_gradient", N=20, layers="40,20,10", walkers=512, therm=5),
        # the covariance matrix of stochastic reconfiguration
        dict(name="s_matrix_32", kind="s_matrix", N=32, M=60, walkers=4096, therm=10),
        # many networks of uneven sizes served together
        dict(name="serving_64", kind="serving", instances=64, largest=144, per_spin=16),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["exact_gradient", "exact_distance", "rbm_step", "rbm_step", "chain_rows", "learned_rows",
                       "sector_samples", "configurations", "deep_step", "deep_gradient", "s_matrix", "serving"])
    if kind == "exact_gradient":
        N = rng.randint(6, 16)
        return dict(kind=kind, N=N, M=_log(rng, N, 6 * N))
    if kind == "exact_distance":
        N = rng.randint(6, 16)
        return dict(kind=kind, N=N, M=_log(rng, 8, 2 * N))
    if kind == "rbm_step":
        if rng.random() < 0.5:
            side = rng.randint(3, 8)
            N, lattice = side * side, "square"
        else:
            N, lattice = rng.randint(10, 64), "chain"
        return dict(kind=kind, N=N, M=_log(rng, N, min(256, 4 * N)), lattice=lattice, walkers=_log(rng, 100, 4096),
                    rows=rng.randint(2, 12), therm=rng.randint(0, 20))
    if kind == "chain_rows":
        N = rng.randint(20, 140)
        return dict(kind=kind, N=N, M=_log(rng, N, min(576, 4 * N)), walkers=_log(rng, 512, 16384),
                    rows=rng.randint(1, 4), sweeps=rng.randint(1, 3))
    if kind == "learned_rows":
        N = rng.randint(20, 110)
        return dict(kind=kind, N=N, M=_log(rng, N, 4 * N), walkers=_log(rng, 1024, 16384), rows=rng.randint(1, 2),
                    steps=rng.randint(5, 20), train=rng.randint(0, 3), train_walkers=512)
    if kind == "sector_samples":
        N = 2 * rng.randint(5, 30)
        return dict(kind=kind, N=N, M=_log(rng, N, 3 * N), walkers=_log(rng, 128, 4096), rows=rng.randint(1, 4),
                    therm=rng.randint(5, 20))
    if kind == "configurations":
        N = rng.randint(10, 140)
        return dict(kind=kind, N=N, M=_log(rng, 16, min(4 * N, 400)), count=_log(rng, 1, 12000))
    if kind == "deep_step":
        N = rng.randint(20, 100)
        layers = [_log(rng, 16, 200), _log(rng, 16, 100)] + ([_log(rng, 8, 50)] if rng.random() < 0.7 else [])
        return dict(kind=kind, N=N, layers=",".join(map(str, layers)), walkers=_log(rng, 256, 4096),
                    therm=rng.randint(1, 3))
    if kind == "deep_gradient":
        N = rng.randint(8, 28)
        layers = [_log(rng, 10, 48), _log(rng, 6, 24)] + ([_log(rng, 4, 12)] if rng.random() < 0.5 else [])
        return dict(kind=kind, N=N, layers=",".join(map(str, layers)), walkers=_log(rng, 64, 512),
                    therm=rng.randint(2, 6))
    if kind == "s_matrix":
        N = rng.randint(8, 32)
        return dict(kind=kind, N=N, M=_log(rng, N, 2 * N), walkers=_log(rng, 512, 4096), therm=rng.randint(2, 10))
    return dict(kind=kind, instances=rng.randint(4, 48), largest=8 * rng.randint(4, 16), per_spin=rng.choice([4, 8, 16]))


# ------------------------------------------------------------------ inputs
def _rng(seed, tag):
    return np.random.Generator(np.random.PCG64([int(seed) & 0x7FFFFFFF, tag]))


def _rbm(g, N, M, sigma=0.05):
    b = g.normal(0, sigma, M) + 1j * g.normal(0, sigma, M)
    W = g.normal(0, sigma, (N, M)) + 1j * g.normal(0, sigma, (N, M))
    return b, W


def _psi(b, W):
    N = W.shape[0]
    return rg.Psi(np.zeros(N), np.zeros(N), b, W)


def _deep(g, N, layers):
    """Dense layers, complex Normal(0, 0.1 / fan_in) weights and biases, final weights 1."""
    b, conn, W, fan = [], [], [], N
    for m in layers:
        sd = np.sqrt(0.1 / fan / 2)
        b.append(g.normal(0, sd, m) + 1j * g.normal(0, sd, m))
        conn.append(np.repeat(np.arange(fan)[:, None], m, axis=1))
        W.append(g.normal(0, sd, (fan, m)) + 1j * g.normal(0, sd, (fan, m)))
        fan = m
    return rg.PsiDeep(np.zeros(N), np.zeros(N), b, conn, W, np.ones(layers[-1]))


def _layers(case):
    return [int(x) for x in case["layers"].split(",")]


def _spins(g, count, N):
    """count configurations as uint64 words."""
    up = g.integers(0, 2, (count, N)).astype(bool)
    w = np.zeros((count, (N + 63) // 64), np.uint64)
    for i in range(N):
        w[:, i // 64] |= up[:, i].astype(np.uint64) << np.uint64(i % 64)
    return w, up


def _distance_inputs(case, seed):
    """A state, a nearby state and the operator 1 - i dt H of a short time step."""
    g = _rng(seed, 2)
    b, W = _rbm(g, case["N"], case["M"])
    db, dW = _rbm(g, case["N"], case["M"], 0.02)
    coef, types, idx = rg.operators.tfim_chain(case["N"], 1.0, 1.0)
    coef = np.concatenate([[1.0], -0.05j * coef])
    types = np.concatenate([np.zeros((1, types.shape[1]), np.int32), types])
    idx = np.concatenate([-np.ones((1, idx.shape[1]), np.int32), idx])
    return (b, W), (b + db, W + dW), (coef, types, idx)


def _batch_shapes(case):
    """(N, M, h) of a batch's networks: the same for every seed."""
    g = _rng(105, 6)
    for i in range(case["instances"]):
        N = int(g.choice(np.arange(16, case["largest"] + 1, 8)))
        yield N, int(g.choice([1, 2, 4])) * N, float(g.uniform(0.5, 2.0))


def prepare(case, seed):
    kind, s = case["kind"], dict(kind=case["kind"])
    g = _rng(seed, 1)
    N = case.get("N")
    s["ev"] = rg.ExpectationValue()
    if kind == "exact_gradient":
        s["psi"] = _psi(*_rbm(g, N, case["M"]))
        s["op"] = rg.Operator(*rg.operators.tfim_chain(N, 1.0, 1.0))
        s["ens"] = rg.ExactSummation(N)
        s["psi"].normalize(s["ens"])
    elif kind == "exact_distance":
        p, q, op = _distance_inputs(case, seed)
        s["psi"], s["prime"], s["op"] = _psi(*p), _psi(*q), rg.Operator(*op)
        s["ens"] = rg.ExactSummation(N)
        s["hsd"] = rg.HilbertSpaceDistance(N, s["psi"].num_params)
    elif kind == "rbm_step":
        side = int(round(N ** 0.5))
        op = rg.operators.tfim_square(side, 1.0, 3.0) if case["lattice"] == "square" else rg.operators.tfim_chain(N)
        s["psi"], s["op"] = _psi(*_rbm(g, N, case["M"])), rg.Operator(*op)
        s["ens"] = rg.MonteCarloLoop(case["walkers"] * case["rows"], 1, case["therm"], case["walkers"], seed=seed)
        # the parameters as a torch program trains them: single precision, on the GPU
        s["params"] = torch.tensor(s["psi"].params, dtype=torch.complex64, device="cuda").requires_grad_()
    elif kind == "chain_rows":
        s["psi"], s["op"] = _psi(*_rbm(g, N, case["M"])), rg.Operator(*rg.operators.tfim_chain(N))
        s["chain"] = rg.Chain(s["psi"], case["walkers"], seed=seed)
        s["sweeps"], s["rows"], s["stream"] = case["sweeps"], case["rows"], torch.cuda.Stream()
        s["eloc"] = torch.empty((case["rows"], case["walkers"], 2), dtype=torch.float64, device="cuda")
        s["chain"].sweep_async(s["psi"], None, 5, 1, 0, s["stream"].cuda_stream)
    elif kind == "learned_rows":
        s["psi"], s["op"] = _psi(*_rbm(g, N, case["M"])), rg.Operator(*rg.operators.tfim_chain(N))
        s["chain"] = rg.Chain(s["psi"], case["walkers"], seed=seed)
        s["net"] = rg.Proposal(N, seed=seed)
        s.update({k: case[k] for k in ("rows", "steps", "train", "train_walkers")}, stream=torch.cuda.Stream())
        s["eloc"] = torch.empty((case["rows"], case["walkers"], 2), dtype=torch.float64, device="cuda")
        s["chain"].sweep_async(s["psi"], None, 5, 1, 0, s["stream"].cuda_stream)
        s["chain"].learned_async(s["psi"], None, s["net"], 10, min(512, case["walkers"]), 1, 0,
                                 s["stream"].cuda_stream)
    elif kind == "sector_samples":
        s["psi"], s["op"] = _psi(*_rbm(g, N, case["M"])), rg.Operator(*rg.operators.heisenberg_chain(N))
        s["ens"] = rg.MonteCarloLoop(case["walkers"] * case["rows"], 1, case["therm"], case["walkers"], seed=seed)
        s["ens"].set_total_z_symmetry(0)
    elif kind == "configurations":
        s["psi"], s["op"] = _psi(*_rbm(g, N, case["M"])), rg.Operator(*rg.operators.tfim_chain(N))
        s["spins"] = _spins(g, case["count"], N)[0]
    elif kind == "deep_step":
        s["psi"], s["op"] = _deep(g, N, _layers(case)), rg.Operator(*rg.operators.tfim_chain(N))
        s["ens"] = rg.MonteCarloLoop(case["walkers"], 1, case["therm"], case["walkers"], seed=seed)
        s["params"] = torch.tensor(s["psi"].params, dtype=torch.complex64, device="cuda").requires_grad_()
    elif kind == "deep_gradient":
        s["psi"], s["op"] = _deep(g, N, _layers(case)), rg.Operator(*rg.operators.tfim_chain(N))
        s["ens"] = rg.MonteCarloLoop(case["walkers"], 1, case["therm"], case["walkers"], seed=seed)
    elif kind == "s_matrix":
        s["psi"] = _psi(*_rbm(g, N, case["M"]))
        s["ens"] = rg.MonteCarloLoop(case["walkers"], 1, case["therm"], case["walkers"], seed=seed)
    elif kind == "serving":
        inst = []
        for i, (n, m, h) in enumerate(_batch_shapes(case)):
            inst.append((_psi(*_rbm(g, n, m)), rg.Operator(*rg.operators.tfim_chain(n, 1.0, h)),
                         case["per_spin"] * n, seed + i))
        s["batch"] = rg.Batch(inst)
        s["batch"].run(10, 1)
        s["batch"].autotune(sweeps=1, reps=2)
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind in ("exact_gradient", "deep_gradient"):
        grad, E = s["ev"].gradient(s["psi"], s["op"], s["ens"])
        return dict(energy=np.complex128(E), gradient=grad)
    if kind == "exact_distance":
        grad, d = s["hsd"].gradient(s["psi"], s["prime"], s["op"], True, s["ens"])
        return dict(distance=d, gradient=grad)
    if kind in ("rbm_step", "deep_step"):
        s["params"].grad = None
        E = energy(s["params"], s["psi"], s["op"], s["ens"])
        E.backward()
        return dict(energy=E.detach(), gradient=s["params"].grad)
    if kind == "chain_rows":
        n = s["rows"] * s["sweeps"]
        s["chain"].sweep_async(s["psi"], s["op"], n, s["sweeps"], s["eloc"].data_ptr(), s["stream"].cuda_stream)
        c = s["chain"].checkpoint()
        return dict(eloc=s["eloc"], spins=c["spins"].view(np.int64), accepts=c["accepts"].view(np.int64))
    if kind == "learned_rows":
        st = s["stream"].cuda_stream
        if s["train"]:
            s["chain"].learned_async(s["psi"], None, s["net"], s["train"], s["train_walkers"], 1, 0, st)
        s["chain"].learned_async(s["psi"], s["op"], s["net"], s["rows"] * s["steps"], 0, s["steps"],
                                 s["eloc"].data_ptr(), st)
        c = s["chain"].checkpoint()
        return dict(eloc=s["eloc"], spins=c["spins"].view(np.int64), accepts=c["accepts"].view(np.int64),
                    network=s["net"].params)
    if kind == "sector_samples":
        spins, log_psi, eloc = s["ens"].samples(s["psi"], s["op"])
        return dict(spins=spins.view(np.int64), log_psi=log_psi, eloc=eloc)
    if kind == "configurations":
        return dict(eloc=rg.local_energies(s["psi"], s["op"], s["spins"]), log_psi=s["psi"].log_psi_batch(s["spins"]))
    if kind == "s_matrix":
        return rg.get_S_matrix(s["psi"], s["ens"], centered=True)
    s["batch"].run(0, 1)
    got = [s["batch"].result(i) for i in range(len(s["batch"].instances))]
    return dict(energies=np.array([e for e, _, _ in got]), gradients=np.concatenate([g for _, g, _ in got]))


# ------------------------------------------------------------------ what a pass cannot do without
def _rbm_flops(N, M, sweeps, samples, offdiag, gradient):
    f = sweeps * (N * M * FLOPS_PROPOSAL + 2 * N * M)
    f += samples * (2 * N * M + FLOPS_F * M + offdiag * M * (FLOPS_F + 8))
    if gradient:  # the tanh of every flipped angle from its denominator, and the sums over samples
        f += samples * (offdiag * M * 52 + (N + 1) * M * 22)
    return f


def _deep_macs(N, layers):
    later = sum(a * b for a, b in zip(layers, layers[1:]))
    return N * layers[0] + later, later


def work(case):
    kind, N, M = case["kind"], case.get("N", 0), case.get("M", 0)
    P = 2 * N + M + N * M
    if kind == "exact_gradient":
        n = 1 << N
        return dict(bytes=32 * P, flops=_rbm_flops(N, M, 0, n, N, True))
    if kind == "exact_distance":
        n = 1 << N
        return dict(bytes=48 * P, flops=n * (4 * N * M + 3 * FLOPS_F * M + N * M * (FLOPS_F + 8) + (N + 1) * M * 8))
    if kind == "rbm_step":
        w = case["walkers"]
        return dict(bytes=16 * P, flops=_rbm_flops(N, M, w * (case["rows"] + case["therm"]), w * case["rows"], N, True))
    if kind == "chain_rows":
        w = case["walkers"]
        return dict(bytes=16 * P + w * (16 * case["rows"] + 8 * ((N + 63) // 64) + 8),
                    flops=_rbm_flops(N, M, w * case["rows"] * case["sweeps"], w * case["rows"], N, False))
    if kind == "learned_rows":
        w, n, O = case["walkers"], case["rows"] * case["steps"], N + 8
        net = 2 * (N * 256 + 256 * 256 + 256 * O)
        return dict(bytes=16 * P + 4 * net + w * (16 * case["rows"] + 24),
                    flops=w * (n + case["train"]) * (net + FLOPS_PROPOSAL * M) + w * case["rows"] * N * M * 52
                    + case["train"] * case["train_walkers"] * (2 * net + N * 8 * M * 41))
    if kind == "sector_samples":
        w = case["walkers"]
        return dict(bytes=16 * P + w * case["rows"] * 40,
                    flops=_rbm_flops(N, M, w * (case["rows"] + case["therm"]), w * case["rows"], 2 * N, False))
    if kind == "configurations":
        n = case["count"]
        return dict(bytes=16 * P + n * (8 * ((N + 63) // 64) + 32),
                    flops=n * (4 * N * M + 2 * FLOPS_F * M + N * M * (FLOPS_F + 8)))
    if kind in ("deep_step", "deep_gradient"):
        L, w = _layers(case), case["walkers"]
        macs, later = _deep_macs(N, L)
        unit = 50 * sum(L)
        proposal = 8 * (L[0] + later) + unit
        adjoint = 8 * macs + N * proposal + (N + 1) * (8 * later + 8 * macs + unit)
        params = macs + sum(L) + L[-1]
        return dict(bytes=32 * params, flops=w * ((case["therm"] + 1) * (8 * macs + N * proposal) + adjoint))
    if kind == "s_matrix":
        K, w = M + N * M, case["walkers"]
        return dict(bytes=16 * (K * K + P), flops=_rbm_flops(N, M, w * (case["therm"] + 1), 0, 0, False) + 4 * w * K * K)
    b = f = 0
    for n, m, _ in _batch_shapes(case):
        w = case["per_spin"] * n
        b += 32 * (m + n * m)
        f += _rbm_flops(n, m, w, w, n, True)
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------ the same in 64 bits
def _t(a):
    return torch.as_tensor(np.asarray(a, np.complex128), device="cuda")


def _lc(z):
    """The rational log-cosh f and its derivative, for sign(Re z) z."""
    s = torch.where(z.real > 0, 1.0, -1.0).to(torch.float64)
    u = s * z
    D = 9.19376335670885 + u * (10.2180213465 + u * (7.771429504240965 + u * (3.746646023906276 + u)))
    dD = 10.2180213465 + u * (2 * 7.771429504240965 + u * (3 * 3.746646023906276 + u * 4))
    n = 5.49914721954 - 2.16564366435 * u
    return 0.9003320053750442 * u + n / D - 0.598139, s * (0.9003320053750442 + (-2.16564366435 * D - n * dD) / (D * D))


def _enumerated(N):
    x = torch.arange(1 << N, device="cuda")
    return x, (((x[:, None] >> torch.arange(N, device="cuda")) & 1) * 2 - 1).to(torch.complex128)


def exact(case, seed):
    kind, N = case["kind"], case.get("N")
    if kind == "exact_gradient":
        b, W = map(_t, _rbm(_rng(seed, 1), N, case["M"]))
        x, s = _enumerated(N)
        f, T = _lc(b + s @ W)
        lp = f.sum(1)
        w = torch.softmax(2 * lp.real, 0)
        diag = -(s * s.roll(-1, 1)).sum(1)
        O = lambda q: torch.cat([T[q], (s[q][:, :, None] * T[q][:, None, :]).reshape(len(q), -1)], 1)  # noqa: E731
        E = diag.clone()
        for i in range(N):
            E -= torch.exp(lp[x ^ (1 << i)] - lp)
        mean = (w * E).sum()
        # sum_s w_s E_k(s) = sum_s O(s) c(s), each string's neighbour collected at its own index
        c = w * diag
        for i in range(N):
            c = c - (w * torch.exp(lp[x ^ (1 << i)] - lp))[x ^ (1 << i)]
        grad = 0
        for q in x.split(4096):
            Oq = O(q)
            grad = grad + (w[q] * (E[q] - 2 * mean)) @ Oq.conj() + (c[q] @ Oq).conj()
        return dict(energy=np.complex128(complex(mean)),
                    gradient=np.concatenate([np.zeros(2 * N, np.complex128), grad.cpu().numpy()]))
    if kind == "exact_distance":
        p, q, (coef, _, _) = _distance_inputs(case, seed)
        x, s = _enumerated(N)
        lp = _lc(_t(p[0]) + s @ _t(p[1]))[0].sum(1)
        f2, T = _lc(_t(q[0]) + s @ _t(q[1]))
        dl = f2.sum(1) - lp
        w = torch.softmax(2 * lp.real, 0)
        E = complex(coef[0]) + complex(coef[1]) * (s * s.roll(-1, 1)).sum(1)
        for i in range(N):
            E = E + complex(coef[-1]) * torch.exp(lp[x ^ (1 << i)] - lp)
        om, pr, nn = torch.exp(dl.conj()) * E, torch.exp(2 * dl.real), E.abs() ** 2
        Om, PR, NN = (w * om).sum(), (w * pr).sum(), (w * nn).sum()
        u, v = Om.abs() ** 2, NN * PR
        d = torch.sqrt(1 - u / v)
        c = w * (Om.conj() * om * v - u * NN * pr) / (v * v * d)
        grad = 0
        for k in x.split(4096):
            O = torch.cat([T[k], (s[k][:, :, None] * T[k][:, None, :]).reshape(len(k), -1)], 1)
            grad = grad - c[k] @ O.conj()
        return dict(distance=float(d), gradient=np.concatenate([np.zeros(2 * N, np.complex128), grad.cpu().numpy()]))
    if kind == "configurations":
        g = _rng(seed, 1)
        b, W = map(_t, _rbm(g, N, case["M"]))
        s = _t(2.0 * _spins(g, case["count"], N)[1] - 1)
        th = b + s @ W
        f = _lc(th)[0]
        E = -(s * s.roll(-1, 1)).sum(1)
        for i in range(N):
            E = E - torch.exp((_lc(th - 2 * s[:, i:i + 1] * W[i])[0] - f).sum(1))
        return dict(eloc=E.cpu().numpy(), log_psi=f.sum(1).cpu().numpy())
    return None  # the outputs follow a Markov chain of 32-bit decisions
