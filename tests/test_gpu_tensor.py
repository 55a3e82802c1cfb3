"""The shared-adjacency ensemble on tcgen05 tensor cores against the FP64 oracle.

The adjacency enters the GEMM as N*A in BF16 (exact integers for the volcano rule; a
general adjacency as BF16 hi + lo), the phases as BF16 hi + lo of (cos, sin), with FP32
accumulation.  Couplings therefore agree with the oracle to about 2^-16 of their
magnitude, and whole runs to the tolerances of the other parity tests.
"""
import numpy as np
import pytest

from helpers import cauchy_inputs, normal_inputs

pytestmark = pytest.mark.gpu
DENSE = 0
TENSOR = 2


def make(native, n, k, thetas, omega, cs, seed=1, t1=10.0, dt=1.0, adj=None, atol=1e-6, h0=None):
    B = len(thetas)
    net = native.Network(n, k=k, coupling=DENSE, batch=B, seed=seed, atol=atol, dense_level=0, engine=TENSOR)
    net.set_frequencies(omega)
    if adj is None:
        net.generate_adjacency()
    else:
        net.set_adjacency(adj)
    for b in range(B):
        net.set_coupling(b, cs[b])
        net.set_state(b, thetas[b], 0.0, dt / 100 if h0 is None else h0)
    net.set_horizon(t1, dt, True)
    return net


@pytest.mark.parametrize("n,k", [(100, 5), (300, 300), (1000, 6)])
def test_tensor_adjacency_bit_exact(native, oracle_lib, n, k):
    _, om = normal_inputs(n, 1)
    net = make(native, n, k, [om * 0] * 16, om, [1.0] * 16, seed=9)
    a = net.adjacency()
    ref = oracle_lib.volcano_adjacency(9, n, k, fp64=False)
    assert np.array_equal(a.view(np.uint32), ref.view(np.uint32))
    net.close()


# (25600, 128): 200 two-tile units on 152 SMs, so the GEMM runs its last rows as one-tile units
@pytest.mark.parametrize("n,batch,k", [(130, 16, 5), (700, 40, 5), (384, 128, 300), (25600, 128, 5)])
def test_tensor_rhs_matches_oracle(native, oracle_lib, n, batch, k):
    th, om = cauchy_inputs(n, 3)
    thetas = [(th + 0.1 * b).astype(np.float32) for b in range(batch)]
    net = make(native, n, k, thetas, om, [2.5] * batch, seed=3)
    for b in (0, batch // 2, batch - 1):
        f, cp = net.rhs(b, thetas[b])
        # the rank-K form builds the same matrix as the stored volcano adjacency
        fr, cpr = oracle_lib.rhs(thetas[b], om, k=k, c1=2.5, seed=3, fp64=True, onthefly=n > 4096)
        scale = np.max(np.abs(cpr)) + 1e-3
        assert np.max(np.abs(cp - cpr)) <= 3e-5 * scale + 1e-7, np.max(np.abs(cp - cpr))
        assert np.all(np.abs(f - fr) <= 1e-4 * scale + 1e-6 * np.abs(fr))
    net.close()


# units of one and of two row tiles, clusters of 1 to 8 CTAs along K, part-filled tiles, several
# waves of clusters, every column width; the tolerance is the test's above
@pytest.mark.parametrize("n,batch", [(1, 2), (127, 3), (129, 16), (500, 17), (1000, 32), (3001, 64), (3001, 128),
                                     (6100, 33), (12700, 11), (20000, 128), (38000, 2)])
def test_tensor_split_gemm_matches_oracle(native, oracle_lib, n, batch):
    th, om = cauchy_inputs(n, 4)
    thetas = [(th + 0.1 * b).astype(np.float32) for b in range(batch)]
    net = make(native, n, 5, thetas, om, [2.5] * batch, seed=3)
    for b in (0, batch - 1):
        f, cp = net.rhs(b, thetas[b])
        fr, cpr = oracle_lib.rhs(thetas[b], om, k=5, c1=2.5, seed=3, fp64=True, onthefly=n > 4096)
        scale = np.max(np.abs(cpr)) + 1e-3
        assert np.max(np.abs(cp - cpr)) <= 3e-5 * scale + 1e-7, np.max(np.abs(cp - cpr))
        assert np.all(np.abs(f - fr) <= 1e-4 * scale + 1e-6 * np.abs(fr))
    net.close()


# the A_lo pass inside the split GEMM's K loop; N*A = hi + lo holds 16 significant bits of an entry
@pytest.mark.parametrize("n,batch", [(130, 2), (1500, 40), (2100, 128)])
def test_tensor_split_gemm_general_adjacency(native, oracle_lib, n, batch):
    rng = np.random.default_rng(n)
    adj = (rng.random((n, n)) * (rng.random((n, n)) < 0.2) / (0.1 * n)).astype(np.float32)
    th, om = normal_inputs(n, 5)
    thetas = [(th + 0.1 * b).astype(np.float32) for b in range(batch)]
    net = make(native, n, 5, thetas, om, [2.0] * batch, adj=adj)
    for b in (0, batch - 1):
        _, cp = net.rhs(b, thetas[b])
        x = np.stack([np.cos(thetas[b].astype(np.float64)), np.sin(thetas[b].astype(np.float64))], 1)
        ref = adj.astype(np.float64) @ x
        # relative errors per term: 2^-17 of the entry, 2^-17 of (cos, sin), 2^-16 of the dropped
        # lo * lo part and the sums, on the absolute row sums
        bound = 3 * 2.0**-16 * np.abs(adj.astype(np.float64)).sum(1)
        assert np.all(np.abs(cp.reshape(n, 2) - ref) <= bound[:, None])
    net.close()


@pytest.mark.parametrize("amp", [0.1, 1e-2, 1e-4, 1e-6])
@pytest.mark.parametrize("n,batch", [(130, 3), (1000, 24)])
def test_tensor_small_phases_keep_their_digits(native, n, batch, amp):
    """Phases around 0: the sums of sin are small, each term with its own relative error."""
    rng = np.random.default_rng(n)
    om = np.zeros(n, np.float32)
    th = (amp * rng.standard_normal(n)).astype(np.float32)
    net = make(native, n, 5, [th] * batch, om, [1.0] * batch, seed=3)
    a = np.rint(net.adjacency().astype(np.float64) * n) / n
    _, cp = net.rhs(batch - 1, th)
    x = np.sin(th.astype(np.float64))
    err = cp.reshape(n, 2)[:, 1] - a @ x
    # per term 2^-18 of it, the error of the two parts of sin, independent of one another; the sums in
    # float32 are 2^-24 of themselves off per step of 16 columns, always less than the terms' share
    assert np.sqrt(np.mean(err**2)) <= 2.0**-18 * np.sqrt(np.mean((a * a) @ (x * x)))
    net.close()


@pytest.mark.parametrize("general", [False, True])
def test_tensor_couplings_to_two_f16_parts(native, general):
    """One K step of 64: per term 2^-21 of (cos, sin) and, of a general weight, 2^-22 of it and 2^-20 of
    what is left out (half a step of X_lo times 2^-11), independent of one another and evenly spread
    (1 / sqrt 3); four additions per column and part, 2^-23 each: 2^-20 of the terms' root sum square.  BF16
    parts are 2^-18.5 off here."""
    n, batch = 64, 16
    rng = np.random.default_rng(8)
    thetas = [rng.uniform(0, 2 * np.pi, n).astype(np.float32) for _ in range(batch)]
    adj = (rng.standard_normal((n, n)) / n).astype(np.float32) if general else None
    net = make(native, n, 5, thetas, np.zeros(n, np.float32), [1.0] * batch, adj=adj)
    a = adj.astype(np.float64) if general else np.rint(net.adjacency().astype(np.float64) * n) / n
    err = []
    for b in range(batch):
        x = np.stack([np.cos(thetas[b].astype(np.float64)), np.sin(thetas[b].astype(np.float64))], 1)
        err.append(net.rhs(b, thetas[b])[1].reshape(n, 2) - a @ x)
    assert np.sqrt(np.mean(np.square(err))) <= 2.0**-20 * np.sqrt(np.mean((a * a).sum(1)))
    if general:
        # 11 + 11 bits of an entry, and the roundings of N A, 1/N and the product
        assert np.all(np.abs(net.adjacency().astype(np.float64) - a) <= (2.0**-22 + 3 * 2.0**-24) * np.abs(a) + 2.0**-38 * np.abs(a).max())
    net.close()


@pytest.mark.parametrize("n,batch", [(130, 3), (1500, 24)])
def test_tensor_rows_of_wide_range(native, n, batch):
    """Rows whose entries span 2^40, rows of tiny entries and of zeros: every entry of N A is held in two
    BF16 parts, in what is given back and in the couplings."""
    def bf16(x):  # to nearest, ties to even
        u = x.view(np.uint32)
        return ((u + np.uint32(0x7FFF) + ((u >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)).view(np.float32)

    def held(a):
        na = a * np.float32(n)
        hi = bf16(na)
        return (hi + bf16(na - hi)) * (np.float32(1) / np.float32(n))

    rng = np.random.default_rng(n)
    adj = ((rng.random((n, n)) + 0.5) / n).astype(np.float32)
    adj[::2] *= np.exp2(-rng.integers(0, 41, (len(adj[::2]), n))).astype(np.float32)
    adj[5] *= np.float32(1e-25)
    adj[:, 7] = 1.0  # the largest entry of its row, at a phase of 0
    adj[3] = 0
    adj[9] = adj[11] * np.float32(1e-30)
    om = np.zeros(n, np.float32)
    th = (rng.random(n) * np.pi).astype(np.float32)
    th[7] = 0
    net = make(native, n, 5, [th] * batch, om, [1.0] * batch, adj=adj)
    assert np.array_equal(net.adjacency(), held(adj))
    _, cp = net.rhs(batch - 1, th)
    # the sums of sin, to which the largest entries give nothing: 2^-17 of an entry, 2^-17 of (cos, sin),
    # 2^-16 of the dropped lo * lo part and the sums
    x = np.sin(th.astype(np.float64))
    bound = 3 * 2.0**-16 * np.abs(adj.astype(np.float64)) @ np.abs(x)
    assert np.all(np.abs(cp.reshape(n, 2)[:, 1] - adj.astype(np.float64) @ x) <= bound)
    # the engine goes back and forth between the two forms
    for a in (((rng.random((n, n)) + 0.5) / n).astype(np.float32), adj):
        net.set_adjacency(a)
        back = net.adjacency()
        if a is adj:
            assert np.array_equal(back, held(adj))
        else:
            assert np.all(np.abs(back.astype(np.float64) - a) <= 2.0**-17 * np.abs(a.astype(np.float64)))
        _, cp = net.rhs(0, th)
        ref = a.astype(np.float64) @ np.stack([np.cos(th.astype(np.float64)), x], 1)
        assert np.all(np.abs(cp.reshape(n, 2) - ref) <= 3 * 2.0**-16 * np.abs(a.astype(np.float64)).sum(1)[:, None])
    net.close()


def test_tensor_weights_that_are_not_finite(native):
    """They reach their own row's couplings and no other row's."""
    n, batch = 200, 2
    rng = np.random.default_rng(2)
    adj = ((rng.random((n, n)) + 0.5) / n).astype(np.float32)
    adj[11, 20], adj[60, 3] = np.inf, np.nan
    th = (rng.random(n)).astype(np.float32)
    net = make(native, n, 5, [th] * batch, np.zeros(n, np.float32), [1.0] * batch, adj=adj)
    _, cp = net.rhs(1, th)
    cp = cp.reshape(n, 2)
    rest = np.delete(np.arange(n), [11, 60])
    assert not np.isfinite(cp[[11, 60]]).any() and np.isfinite(cp[rest]).all()
    ref = adj[rest].astype(np.float64) @ np.stack([np.cos(th.astype(np.float64)), np.sin(th.astype(np.float64))], 1)
    assert np.all(np.abs(cp[rest] - ref) <= 3 * 2.0**-16 * adj[rest].astype(np.float64).sum(1)[:, None])
    net.close()


@pytest.mark.parametrize("n,batch", [(300, 5), (3000, 24)])
def test_tensor_phase_that_is_not_finite(native, n, batch):
    """A NaN phase reaches every coupling of its own trajectory and none of the others'."""
    rng = np.random.default_rng(2)
    om = rng.standard_normal(n).astype(np.float32)
    thetas = [rng.uniform(-3, 3, n).astype(np.float32) for _ in range(batch)]
    net = make(native, n, 5, thetas, om, [1.0] * batch, seed=2)
    good = [net.rhs(b, thetas[b])[0] for b in range(batch)]
    bad = thetas[1].copy()
    bad[n // 2] = np.nan
    assert np.isnan(net.rhs(1, bad)[0]).all()
    net.set_state(1, bad, 0.0, 0.01)
    assert np.array_equal(net.rhs(0, thetas[0])[0], good[0])
    net.set_state(1, thetas[1], 0.0, 0.01)
    for b in range(batch):
        assert np.array_equal(net.rhs(b, thetas[b])[0], good[b])
    net.close()


def test_tensor_general_adjacency_split(native, oracle_lib):
    n, batch = 200, 16
    rng = np.random.default_rng(5)
    adj = (rng.standard_normal((n, n)) / n).astype(np.float32)
    th, om = normal_inputs(n, 4)
    thetas = [(th + 0.2 * b).astype(np.float32) for b in range(batch)]
    net = make(native, n, 5, thetas, om, [1.5] * batch, adj=adj)
    back = net.adjacency()
    # N*A stored as BF16 hi + lo: 16 significant bits, about 2^-16 relative per entry
    assert np.all(np.abs(back - adj) <= 2.0 ** -15 * np.abs(adj) + 1e-12)
    f, cp = net.rhs(3, thetas[3])
    fr, cpr = oracle_lib.rhs(thetas[3], om, k=5, c1=1.5, adj=adj.astype(np.float64), fp64=True)
    assert np.max(np.abs(cp - cpr)) <= 3e-5 * np.max(np.abs(cpr))
    net.close()


@pytest.mark.parametrize("n,batch", [(256, 16), (1000, 24)])
def test_tensor_runs_match_fp64(native, oracle_lib, n, batch):
    _, om = normal_inputs(n, 11)
    thetas = [normal_inputs(n, 100 + b, init=2 * np.pi)[0] for b in range(batch)]
    cs = [1.0 + 0.25 * (b % 9) for b in range(batch)]
    net = make(native, n, 5, thetas, om, cs, seed=2, t1=10.0, dt=1.0)
    net.run()
    st = net.stats()
    assert st["accepted"] > 0
    for b in (0, batch // 3, batch - 1):
        r = net.order(b)
        ref = oracle_lib.run(thetas[b], om, k=5, c1=cs[b], seed=2, fp64=True, t1=10.0, dt=1.0)
        r32 = oracle_lib.run(thetas[b], om, k=5, c1=cs[b], seed=2, fp64=False, t1=10.0, dt=1.0)
        assert r.size == ref.order.size == 11
        env = np.abs(r32.order - ref.order)
        assert np.all(np.abs(r - ref.order) <= 1e-4 + 4 * env), (b, np.max(np.abs(r - ref.order)))
    th_end, t_end, _ = net.state(0)
    assert t_end >= 10.0
    net.close()


def test_tensor_batch_128_long_horizon(native, oracle_lib):
    n, batch = 512, 128
    _, om = normal_inputs(n, 21)
    thetas = [normal_inputs(n, 200 + b, init=2 * np.pi)[0] for b in range(batch)]
    cs = [3.0] * batch
    net = make(native, n, 5, thetas, om, cs, seed=4, t1=40.0, dt=1.0)
    net.run()
    for b in (0, 63, 127):
        r = net.order(b)
        ref = oracle_lib.run(thetas[b], om, k=5, c1=3.0, seed=4, fp64=True, t1=40.0, dt=1.0)
        assert abs(r.mean() - ref.order.mean()) < 1e-3
    net.close()


@pytest.mark.parametrize("n,batch", [(130, 2), (257, 16), (1000, 7), (1021, 24), (2500, 3)])
def test_tensor_operands_from_the_gemm_match_fp64(native, oracle_lib, n, batch):
    """Sizes whose attempts make the stages' operands in the GEMM's epilogue: ragged last tiles and
    groups of four rows, padded columns, one and several CTAs per tile.  The bound is the other
    runs': 1e-4 plus four times what float32 arithmetic itself is off."""
    _, om = normal_inputs(n, 21)
    thetas = [normal_inputs(n, 300 + b, init=2 * np.pi)[0] for b in range(batch)]
    cs = [1.0 + 0.5 * (b % 4) for b in range(batch)]
    net = make(native, n, 5, thetas, om, cs, seed=2, t1=5.0, dt=0.5)
    net.run()
    for b in (0, batch - 1):
        r = net.order(b)
        ref = oracle_lib.run(thetas[b], om, k=5, c1=cs[b], seed=2, fp64=True, t1=5.0, dt=0.5)
        r32 = oracle_lib.run(thetas[b], om, k=5, c1=cs[b], seed=2, fp64=False, t1=5.0, dt=0.5)
        assert r.size == ref.order.size == 11
        assert np.all(np.abs(r - ref.order) <= 1e-4 + 4 * np.abs(r32.order - ref.order)), b
    net.close()


@pytest.mark.parametrize("c,fixed,t1,dt,h0", [(0.0, False, 50.0, 0.1, 0.001), (1.0, True, 8.0, 0.01, 1.0),
                                              (1.0, True, 5.0, 1.0 / 33, 1.0)])
@pytest.mark.parametrize("n,batch", [(64, 3), (700, 7)])
def test_tensor_step_over_many_output_times(native, n, batch, c, fixed, t1, dt, h0):
    """Steps that cross up to hundreds of output times, 33 among them: every record is there, also when
    budgets of attempts end between them.  Without coupling the phases are exact in both engines and r is a
    float32 sum (5e-6); with it the bound is the other runs'."""
    _, om = normal_inputs(n, 21)
    thetas = [normal_inputs(n, 300 + b, init=2 * np.pi)[0] for b in range(batch)]

    def net_of(engine):
        net = native.Network(n, k=5, coupling=DENSE, batch=batch, seed=2, engine=engine, fixed_step=fixed)
        net.set_frequencies(om)
        net.generate_adjacency()
        for b in range(batch):
            net.set_coupling(b, c)
            net.set_state(b, thetas[b], 0.0, h0 * (1 + 0.5 * b) if not fixed else h0)
        net.set_horizon(t1, dt, True)
        return net

    out = []
    for engine in (native.ENGINE_PERSISTENT, TENSOR):
        net = net_of(engine)
        net.run()
        out.append([net.order(b) for b in range(batch)])
        net.close()
    net = net_of(TENSOR)
    rec = [[] for _ in range(batch)]
    while net.advance(4, on_output=lambda b, i, t, r, theta, cp: rec[b].append((i, r)) and False):
        pass
    net.close()
    for b in range(batch):
        assert out[0][b].size == out[1][b].size == int(np.float32(t1) / np.float32(dt)) + 1
        assert np.max(np.abs(out[0][b] - out[1][b])) < (5e-6 if c == 0 else 1e-4)
        assert [q[0] for q in rec[b]] == list(range(-1, out[1][b].size - 1))
        assert np.array_equal(np.array([q[1] for q in rec[b]], np.float32), out[1][b])


def test_tensor_engine_reused_over_horizons(native):
    """One engine over horizons that grow, shrink and grow again (kept buffers, kept graph), with a state
    that is replaced before its upload is over, gives the records of a fresh engine each time."""
    n, batch = 700, 5
    rng = np.random.default_rng(3)
    om = (1.8 * rng.standard_cauchy(n)).astype(np.float32)
    cs = [1.0 + 0.5 * b for b in range(batch)]
    net = None
    for t1, dt in ((2.0, 0.5), (2.0, 0.5), (1.0, 0.25), (1.0, 0.5), (6.0, 0.1), (2.0, 0.5)):
        thetas = [rng.uniform(-3, 3, n).astype(np.float32) for _ in range(batch)]
        fresh = make(native, n, 3, thetas, om, cs, t1=t1, dt=dt)
        fresh.run()
        if net is None:
            net = make(native, n, 3, thetas, om, cs, t1=t1, dt=dt)
        else:
            for b in range(batch):
                scratch = rng.uniform(-3, 3, n).astype(np.float32)
                net.set_state(b, scratch, 0.0, 0.3)
                scratch[:] = thetas[b]
                net.set_state(b, scratch, 0.0, dt / 100)
                scratch[:] = np.nan  # the caller's buffer is its own again
            net.set_horizon(t1, dt, True)
        net.run()
        for b in range(batch):
            np.testing.assert_array_equal(net.order(b), fresh.order(b))
            np.testing.assert_array_equal(net.state(b)[0], fresh.state(b)[0])


def test_tensor_engine_reused_over_adjacencies(native):
    """A new adjacency of another form (volcano: one part; general: two) on an engine that has run."""
    n, batch, k = 300, 3, 3
    rng = np.random.default_rng(5)
    om = rng.standard_normal(n).astype(np.float32)
    cs = [1.0, 2.0, 3.0]
    adjs = [None, rng.standard_normal((n, n)).astype(np.float32) / n, None]
    net = None
    for adj in adjs:
        thetas = [rng.uniform(-3, 3, n).astype(np.float32) for _ in range(batch)]
        fresh = make(native, n, k, thetas, om, cs, t1=2.0, dt=0.5, adj=adj)
        fresh.run()
        if net is None:
            net = make(native, n, k, thetas, om, cs, t1=2.0, dt=0.5, adj=adj)
        else:
            if adj is None:
                net.generate_adjacency()
            else:
                net.set_adjacency(adj)
            for b in range(batch):
                net.set_state(b, thetas[b], 0.0, 0.005)
            net.set_horizon(2.0, 0.5, True)
        net.run()
        for b in range(batch):
            np.testing.assert_array_equal(net.order(b), fresh.order(b))
            np.testing.assert_array_equal(net.state(b)[0], fresh.state(b)[0])


def test_tensor_rejects_unsupported(native):
    with pytest.raises(native.KuraError):
        native.Network(100, k=5, coupling=1, batch=16, engine=TENSOR)  # volcano coupling
    with pytest.raises(native.KuraError):
        native.Network(100, k=5, coupling=DENSE, batch=16, engine=TENSOR, dense_level=1)


def test_auto_engine_choice(native):
    """KURA_ENGINE_AUTO: the tensor engine (it reports grid 0) for a dense batch of two or more
    that keeps only r, and for any dense batch above 8; the persistent kernel for one trajectory,
    for per-step records (dense level >= 1), for the int8 adjacency and for the -A coupling."""
    def grid(**kw):
        net = native.Network(300, k=5, **kw)
        g = net.stats()["grid"]
        net.close()
        return g
    assert grid(coupling=DENSE, batch=2, dense_level=0) == 0
    assert grid(coupling=DENSE, batch=16, dense_level=0) == 0
    assert grid(coupling=DENSE, batch=1, dense_level=0) > 0
    assert grid(coupling=DENSE, batch=4, dense_level=1) > 0
    assert grid(coupling=DENSE, batch=4, dense_level=0, adj_storage=native.ADJ_I8) > 0
    assert grid(coupling=1, batch=4, dense_level=0) > 0
