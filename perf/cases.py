"""The workloads whose speed is measured: what a user of this package has it do.

A case is a dict of plain values; ``listed()`` gives the fixed ones and ``draw()`` further ones of
the same ranges.  Four kinds:

* ``network``: a run of the integrator from given phases to t1 (``Network``): stored adjacency in
  float32 or int8, the regenerated volcano coupling, or an ensemble of trajectories that share one
  adjacency on the tensor cores.  Returns r(t) of every trajectory and, at dense level 1 and 2,
  the phases and couplings of every record;
* ``multi``: independent networks of uneven size in one call (``MultiNetworks``), r(t) of each;
* ``train`` / ``predict``: the surrogate MLP's training and its evaluation (``MLP``).

``exact()`` restates each of them in 64 bits with plain torch.
"""
import numpy as np
import torch

import kuramoto_gb300 as kg

VOLCANO, WEIGHTED = "volcano", "weighted"  # the adjacency: the reference's rule, or a user's own weights


# ---------------------------------------------------------------- the cases
def network(name=None, n=1000, k=5, batch=1, coupling="dense", adjacency=VOLCANO, storage="f32", engine="auto",
            freq="cauchy", init=np.pi, c0=3.0, c1=3.0, t1=0.25, dt=0.0625, level=0, rtol=0.0, fixed=False, steps=0):
    case = dict(kind="network", n=n, k=k, batch=batch, coupling=coupling, adjacency=adjacency, storage=storage,
                engine=engine, freq=freq, init=float(init), c0=c0, c1=c1, t1=t1, dt=dt, level=level, rtol=rtol,
                fixed=fixed, steps=steps)
    return dict(case, name=name) if name else case


def listed():
    return [
        # a small stored network with its phases and couplings written out (-D 2): every kernel interval is latency
        network("dense-997-D2", n=997, k=6, level=2, steps=60),
        # the reference program's defaults: N=5000, Cauchy frequencies, all phases zero at the start
        network("dense-5000", n=5000, k=5, init=0.0, t1=0.5, dt=0.125, steps=80),
        # one trajectory of the shared-adjacency ensemble on the plain float32 path: 17 GB of adjacency per RHS
        network("dense-65536", n=65536, t1=0.03125, dt=0.0078125, steps=8),
        # the same network rule with N*A stored as int8, at a size that is no multiple of the kernels' tiles
        network("dense-int8-40009", n=40009, k=7, storage="i8", level=1, t1=0.125, dt=0.03125, steps=18),
        # -A on a small network: nothing stored, one trajectory
        network("volcano-1000", n=1000, coupling="volcano", level=1, t1=0.5, dt=0.125, steps=110),
        # -A on the large network, the five couplings of a sweep as one batch
        network("volcano-200000x5", n=200000, batch=5, coupling="volcano", freq="normal", c0=1.0, c1=5.0,
                t1=10.0, dt=1.0, steps=40),
        # a small ensemble: the adjacency is a few megabytes
        network("ensemble-3000x24", n=3000, batch=24, steps=50),
        # an ensemble over a user's own weighted network (-R), which takes two BF16 parts to hold
        network("ensemble-6007x64-weighted", n=6007, batch=64, adjacency=WEIGHTED, freq="normal", c0=1.0, c1=2.0, t1=4.0,
                dt=0.5, steps=14),
        # the shared-adjacency ensemble the throughput metric is quoted on
        network("ensemble-65536x128", n=65536, batch=128, t1=0.125, dt=0.03125, steps=20),
        # a sweep's networks: uneven sizes, ranks and couplings, each with its own step
        dict(name="multi-64", kind="multi", count=64, nmin=1000, nmax=20000, cauchy=0.1, t1=2.0, dt=0.25, steps=30),
        # the surrogate's training: 20000 samples, minibatches of 512, two epochs
        dict(name="mlp-train-20000", kind="train", hidden=256, batch=512, samples=20000, epochs=2),
        # the surrogate evaluated on a sweep's candidate couplings
        dict(name="mlp-predict-64", kind="predict", hidden=256, batch=512, samples=64),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))

    what = rng.choice(["dense", "dense", "int8", "volcano", "volcano", "ensemble", "ensemble", "multi", "mlp"])
    freq = rng.choice(["cauchy", "normal"])
    t1, dt = rng.choice([(2.0, 0.5), (4.0, 0.5), (4.0, 1.0)] if freq == "normal" else [(0.125, 0.03125), (0.25, 0.0625)])
    steps = int(4 + 3 * t1) if freq == "normal" else int(8 + 120 * t1)
    common = dict(freq=freq, init=rng.choice([0.0, np.pi]) if freq == "cauchy" else np.pi,
                  c0=round(rng.uniform(0.5, 2.0 if freq == "normal" else 3.0), 2), t1=t1, dt=dt, steps=steps)
    last = round(rng.uniform(0.5, 2.0 if freq == "normal" else 3.0), 2)  # the coupling of a batch's last trajectory
    if what == "dense":
        n = log(200, 40000)
        own = n <= 6000 and rng.random() < 0.3
        return network(n=n, k=rng.randint(2, 8), adjacency=WEIGHTED if own else VOLCANO, c1=common["c0"],
                       level=rng.choice([0, 0, 1, 2]) if n <= 10000 else 0, rtol=rng.choice([0.0, 0.0, 0.0, 1e-6]), **common)
    if what == "int8":
        return network(n=log(1000, 65536), k=rng.randint(2, 8), storage="i8", c1=common["c0"], **common)
    if what == "volcano":
        n = log(300, 300000)
        return network(n=n, k=rng.choice([2, 4, 5, 6, 8, 12]), batch=rng.choice([1, 1, 1, 2, 5, 8]), coupling="volcano", c1=last,
                       level=rng.choice([0, 0, 1, 2]) if n <= 10000 else 0, rtol=rng.choice([0.0, 0.0, 0.0, 1e-6]),
                       fixed=rng.random() < 0.1, **common)
    if what == "ensemble":
        n = log(500, 40000)
        own = n <= 6000 and rng.random() < 0.3
        return network(n=n, k=rng.randint(2, 8), batch=log(2, 128), adjacency=WEIGHTED if own else VOLCANO, c1=last, **common)
    if what == "multi":
        return dict(kind="multi", count=log(2, 128), nmin=log(300, 2000), nmax=log(3000, 20000),
                    cauchy=rng.choice([0.0, 0.1]), t1=rng.choice([1.0, 2.0]), dt=0.25, steps=30)
    hidden, batch = rng.choice([64, 128, 256]), rng.choice([256, 512, 1024])
    if rng.random() < 0.5:
        return dict(kind="train", hidden=hidden, batch=batch, samples=log(2000, 20000), epochs=rng.randint(1, 2))
    return dict(kind="predict", hidden=hidden, batch=batch, samples=log(16, 20000))


# ---------------------------------------------------------------- inputs
def frequencies(rng, n, freq):
    w = rng.standard_cauchy(n) if freq == "cauchy" else rng.standard_normal(n)
    return w.astype(np.float32)


def weighted_adjacency(n, seed):
    """A sparse directed network of weights in [0.5, 1.5], about one link in ten, rows of unit mean sum."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    a = torch.rand(n, n, generator=g, device="cuda") + 0.5
    a *= torch.rand(n, n, generator=g, device="cuda") < 0.1
    return a * (1.0 / (0.1 * n))


def network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    omega = frequencies(rng, case["n"], case["freq"])
    thetas = (rng.random((case["batch"], case["n"])) * case["init"]).astype(np.float32)
    cs = np.linspace(case["c0"], case["c1"], case["batch"]).astype(np.float32)
    return omega, thetas, cs, case["dt"] / (16 if case["fixed"] else 100)


def multi_inputs(case, seed):
    rng = np.random.default_rng(seed)
    count = case["count"]
    ns = np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), count)).astype(int)
    ks, cs = rng.integers(2, 9, count), rng.uniform(0.0, 4.0, count).astype(np.float32)
    seeds = rng.integers(1, 1 << 30, count)
    # the Cauchy networks are the first ones: their number does not change with the seed
    family = ["cauchy" if i < round(case["cauchy"] * count) else "normal" for i in range(count)]
    omega = [frequencies(rng, n, f) for n, f in zip(ns, family)]
    theta = [(rng.random(n) * np.pi).astype(np.float32) for n in ns]
    return ns, ks, seeds, cs, omega, theta


IN, OUT = 14, 2  # the surrogate's features and targets


def mlp_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((case["samples"], IN)).astype(np.float32)
    y = np.stack([np.tanh(x[:, 0] + 0.5 * x[:, 1]), np.exp(-x[:, 2] ** 2) * x[:, 3]], 1).astype(np.float32)
    dims = [IN, case["hidden"], case["hidden"], case["hidden"], OUT]
    params = []
    for i, o in zip(dims, dims[1:]):
        params += [rng.uniform(-1, 1, i * o) * np.sqrt(6.0 / (i + o)), rng.uniform(-0.1, 0.1, o)]
    return x, y, np.concatenate(params).astype(np.float32)


# ---------------------------------------------------------------- what a program has in hand, and one pass
def prepare(case, seed):
    if case["kind"] == "multi":
        ns, ks, seeds, cs, omega, theta = multi_inputs(case, seed)
        nets = kg.MultiNetworks(ns, ks, seeds, cs, case["t1"], case["dt"])
        return dict(case=case, nets=nets, omega=np.concatenate(omega), theta=np.concatenate(theta))
    if case["kind"] in ("train", "predict"):
        x, y, params = mlp_inputs(case, seed)
        net = kg.MLP(IN, OUT, hidden=case["hidden"], batch=case["batch"], seed=1)
        net.set_params(params)
        return dict(case=case, net=net, x=x, y=y, params=params, seed=seed)
    omega, thetas, cs, h0 = network_inputs(case, seed)
    dense = case["coupling"] == "dense"
    engine = {"auto": kg.ENGINE_AUTO, "persistent": kg.ENGINE_PERSISTENT, "tensor": kg.ENGINE_TENSOR}[case["engine"]]
    net = kg.Network(case["n"], k=case["k"], coupling=kg.COUPLING_DENSE if dense else kg.COUPLING_VOLCANO,
                     batch=case["batch"], seed=1 + seed % 1000, rtol=case["rtol"], fixed_step=case["fixed"],
                     dense_level=case["level"], engine=engine,
                     adj_storage=kg.ADJ_I8 if case["storage"] == "i8" else kg.ADJ_F32)
    net.set_frequencies(omega)
    if dense and case["adjacency"] == VOLCANO:
        net.generate_adjacency()
    elif dense:
        net.set_adjacency(weighted_adjacency(case["n"], seed).cpu().numpy())
    for b, c in enumerate(cs):
        net.set_coupling(b, c)
    return dict(case=case, net=net, thetas=thetas, h0=h0)


def run(state):
    case = state["case"]
    if case["kind"] == "multi":
        return state["nets"].integrate(state["omega"], state["theta"], want_theta=False)[0]
    net = state["net"]
    if case["kind"] == "predict":
        return net.forward(state["x"])
    if case["kind"] == "train":
        net.set_params(state["params"])
        losses, _ = net.train(state["x"], state["y"], case["epochs"], lr=2e-3, lr_final=1e-4, seed=1 + state["seed"])
        return losses, net.params()
    for b, theta in enumerate(state["thetas"]):
        net.set_state(b, theta, 0.0, state["h0"])
    net.set_horizon(case["t1"], case["dt"], True)
    out = {}
    if case["level"]:
        records = []
        net.run(on_output=lambda b, i, t, r, theta, coup: records.append((b, theta, coup)))
        records.sort(key=lambda q: q[0])  # by trajectory, in the order of time
        out["thetas"] = np.stack([q[1] for q in records])
        if case["level"] > 1:
            out["couplings"] = np.stack([q[2] for q in records])
    else:
        net.run()
    out["order"] = np.stack([net.order(b) for b in range(case["batch"])])
    return out


# ---------------------------------------------------------------- the work of one pass
def work(case):
    """The steps a run takes depend on its inputs: ``steps`` is their number for typical ones."""
    if case["kind"] == "multi":
        mean = (case["nmax"] - case["nmin"]) / np.log(case["nmax"] / case["nmin"])
        osc = case["count"] * mean
        return {"bytes": osc * 8 + case["count"] * 4 * (case["t1"] / case["dt"] + 1), "flops": osc * case["steps"] * 6 * 100}
    if case["kind"] in ("train", "predict"):
        h, m = case["hidden"], case["samples"]
        weights = IN * h + 2 * h * h + h * OUT
        if case["kind"] == "predict":
            return {"bytes": m * 4 * (IN + OUT) + 2 * weights, "flops": 2 * m * weights}
        m = m // case["batch"] * case["batch"] * case["epochs"]
        return {"bytes": m * 4 * (IN + OUT) + m // case["batch"] * 24 * weights, "flops": 6 * m * weights}
    n, b = case["n"], case["batch"]
    rhs = 6 * case["steps"] + 1
    records = case["t1"] / case["dt"] + 1
    state = 4 * n * (1 + b) + 12 * n + 4 * n * b * records * [0, 1, 3][case["level"]]
    if case["coupling"] == "volcano":
        return {"bytes": state, "flops": n * b * rhs * (60 + 8 * case["k"])}
    # every RHS reads the stored adjacency once for the whole batch
    entry = 1 if case["storage"] == "i8" else 4 if b == 1 else 2
    return {"bytes": state + rhs * entry * n * n, "flops": rhs * b * (4.0 * n * n + 60 * n)}


# ---------------------------------------------------------------- the same in 64 bits
A = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
     [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
     [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
     [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
E = [-71 / 57600, 0, 71 / 16695, -71 / 1920, 17253 / 339200, -22 / 525, 1 / 40]
P = [[1.0, -8048581381 / 2820520608, 8663915743 / 2820520608, -12715105075 / 11282082432], [0.0] * 4,
     [0, 131558114200 / 32700410799, -68118460800 / 10900136933, 87487479700 / 32700410799],
     [0, -1754552775 / 470086768, 14199869525 / 1410260304, -10690763975 / 1880347072],
     [0, 127303824393 / 49829197408, -318862633887 / 49829197408, 701980252875 / 199316789632],
     [0, -282668133 / 205662961, 2019193451 / 616988883, -1453857185 / 822651844],
     [0, 40617522 / 29380423, -110615467 / 29380423, 69997945 / 29380423]]


def factor(seed, n, k):
    """The volcano factor, +1 or -1: the low bit of word m*n + i of the Philox4x32-10 stream (Salmon et al. 2011)."""
    if k == 0:
        return torch.zeros(0, n, dtype=torch.float64, device="cuda")
    low = 0xFFFFFFFF

    def mul(a, c):  # the high and the low word of a 32-bit product, in int64
        p0, p1 = (a & 0xFFFF) * c, (a >> 16) * c
        return (p1 + (p0 >> 16)) >> 16, (a * c) & low

    q = torch.arange(n * k, dtype=torch.int64, device="cuda")
    x = [(q >> 2) & low, q >> 34, torch.zeros_like(q), torch.zeros_like(q)]
    k0, k1 = seed & low, (seed >> 32) & low
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
        h0, l0 = mul(x[0], 0xD2511F53)
        h1, l1 = mul(x[2], 0xCD9E8D57)
        x = [h1 ^ x[1] ^ k0, l1, h0 ^ x[3] ^ k1, l0]
    word = torch.stack(x, 1).gather(1, (q & 3)[:, None])[:, 0]
    return ((word & 1) * 2 - 1).to(torch.float64).reshape(k, n)


class Integrator:
    """dp45 with its dense output, every trajectory of a batch with its own step."""

    def __init__(self, omega, cs, matrix=None, u=None, atol=1e-6, rtol=0.0, fixed=False):
        self.omega = torch.tensor(omega, dtype=torch.float64, device="cuda")
        self.c = torch.tensor(np.asarray(cs, np.float64), device="cuda")[:, None]
        self.matrix, self.u, self.atol, self.rtol, self.fixed = matrix, u, atol, rtol, fixed
        if u is not None:
            self.sign = torch.tensor([1.0 - 2 * (m % 2) for m in range(u.shape[0])], dtype=torch.float64, device="cuda")
        self.n = self.omega.numel()

    def couplings(self, theta):
        c, s = torch.cos(theta), torch.sin(theta)
        if self.matrix is not None:
            return c @ self.matrix.T, s @ self.matrix.T, c, s
        fc, fs = ((x @ self.u.T * (self.sign / self.n)) @ self.u for x in (c, s))
        return fc, fs, c, s

    def rhs(self, theta):
        fc, fs, c, s = self.couplings(theta)
        return self.omega + self.c * (s * fc - c * fs)

    def run(self, theta0, t1, dt, h0):
        """r [B, records] and the phases of every record."""
        y = torch.tensor(theta0, dtype=torch.float64, device="cuda")
        B = y.shape[0]
        dtf, t1f = np.float32(dt), np.float32(t1)
        grid = [float(dtf * np.float32(i)) for i in range(1, int(t1f / dtf) + 1)]
        col = lambda v: torch.tensor(v, dtype=torch.float64, device="cuda")[:, None]  # noqa: E731
        t, h, nxt = [0.0] * B, [h0] * B, [0] * B
        k1 = self.rhs(y)
        rec = [[y[b].clone()] for b in range(B)]
        while True:
            live = [t[b] < t1 for b in range(B)]
            if not any(live):
                break
            hc, ks = col(h), [k1]
            for s in range(1, 7):
                arg = y + hc * sum(a * kk for a, kk in zip(A[s], ks) if a)
                ks.append(self.rhs(arg))
            y7 = arg
            if self.fixed:
                norm = [0.0] * B
            else:
                err = hc * sum(e * kk for e, kk in zip(E, ks) if e)
                tol = self.atol + self.rtol * torch.maximum(y.abs(), y7.abs())
                norm = ((err / tol).square().sum(1).sqrt() / np.sqrt(self.n)).tolist()
            take = [False] * B
            for b in range(B):
                if not live[b]:
                    continue
                fac = 0.9 * norm[b] ** -0.2 if norm[b] > 0 else 10.0
                if not norm[b] < 1.0:
                    h[b] *= max(min(fac, 1.0), 0.2)
                    continue
                take[b] = True
                new = t[b] + h[b]
                while nxt[b] < len(grid) and new >= grid[nxt[b]]:
                    x = (grid[nxt[b]] - t[b]) / h[b]
                    w = [h[b] * (((p[3] * x + p[2]) * x + p[1]) * x * x + p[0] * x) for p in P]
                    rec[b].append(y[b] + sum(wj * kk[b] for wj, kk in zip(w, ks) if wj))
                    nxt[b] += 1
                t[b] = new
                if not self.fixed:
                    h[b] *= min(fac, 10.0)
            mask = torch.tensor(take, device="cuda")[:, None]
            y = torch.where(mask, y7, y)
            k1 = torch.where(mask, ks[6], k1)
        r = torch.tensor([[float(torch.hypot(torch.cos(q).mean(), torch.sin(q).mean())) for q in rec[b]] for b in range(B)],
                         dtype=torch.float64)
        return r, rec


def exact_network(case, seed):
    n, b = case["n"], case["batch"]
    omega, thetas, cs, h0 = network_inputs(case, seed)
    matrix = u = None
    if case["adjacency"] == WEIGHTED:
        matrix = weighted_adjacency(n, seed).double()
    else:
        u = factor(1 + seed % 1000, n, case["k"])
    sim = Integrator(omega, cs, matrix, u, rtol=case["rtol"], fixed=case["fixed"])
    r, rec = sim.run(thetas, case["t1"], case["dt"], h0)
    out = {"order": r}
    if case["level"]:
        every = torch.stack([q for one in rec for q in one])
        out["thetas"] = every
        if case["level"] > 1:
            fc, fs, _, _ = sim.couplings(every)
            out["couplings"] = torch.stack([fc, fs], 2).reshape(every.shape[0], 2 * n)
    return out


def exact_multi(case, seed):
    if case["count"] > 64:
        return None  # one network after another: too long
    ns, ks, seeds, cs, omega, theta = multi_inputs(case, seed)
    rows = []
    for n, k, s, c, om, th in zip(ns, ks, seeds, cs, omega, theta):
        sim = Integrator(om, [c], u=factor(int(s), int(n), int(k)))
        rows.append(sim.run(th[None], case["t1"], case["dt"], case["dt"] / 100)[0][0])
    return torch.stack(rows)


def exact_mlp(case, seed):
    x, y, params = mlp_inputs(case, seed)
    x, y = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (x, y))
    h = case["hidden"]
    dims, at, w = [IN, h, h, h, OUT], 0, []
    for i, o in zip(dims, dims[1:]):
        for shape in ((o, i), (o,)):
            size = int(np.prod(shape))
            w.append(torch.tensor(params[at:at + size], dtype=torch.float64, device="cuda").reshape(shape))
            at += size

    def forward(v):
        for l in range(4):
            v = v @ w[2 * l].T + w[2 * l + 1]
            v = v * torch.sigmoid(v) if l < 3 else v
        return v

    if case["kind"] == "predict":
        return forward(x)
    for p in w:
        p.requires_grad_(True)
    m, bt = case["samples"], case["batch"]
    per, mask, s = m // bt, (1 << 64) - 1, 1 + seed
    total, step, losses = per * case["epochs"], 0, []
    first, second = [torch.zeros_like(p) for p in w], [torch.zeros_like(p) for p in w]
    for _ in range(case["epochs"]):
        perm = list(range(m))
        for i in range(m - 1, 0, -1):  # Fisher-Yates on the splitmix64 stream
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        rows = torch.tensor(perm, device="cuda")
        sums = 0.0
        for q in range(per):
            at = rows[q * bt:(q + 1) * bt]
            loss = (forward(x[at]) - y[at]).square().mean()
            grads = torch.autograd.grad(loss, w)
            sums += float(loss.detach())
            lr = 2e-3 + (1e-4 - 2e-3) * (step / (total - 1) if total > 1 else 0.0)
            step += 1
            with torch.no_grad():
                for p, g, a, b in zip(w, grads, first, second):
                    a.mul_(0.9).add_(0.1 * g)
                    b.mul_(0.999).add_(0.001 * g * g)
                    p -= lr * (a / (1 - 0.9 ** step)) / ((b / (1 - 0.999 ** step)).sqrt() + 1e-8)
        losses.append(sums / per)
    return torch.tensor(losses, dtype=torch.float64), torch.cat([p.detach().reshape(-1) for p in w])


def exact(case, seed):
    if case["kind"] == "multi":
        return exact_multi(case, seed)
    if case["kind"] in ("train", "predict"):
        return exact_mlp(case, seed)
    return exact_network(case, seed)
