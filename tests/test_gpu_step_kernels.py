"""The steppers' stages, error estimates and solutions against the device-op
layer: one step of every solver restated with torque(), Madd and Normalize.

Both forms of the step are covered: small meshes form the next stage (and the
error estimate) inside the torque kernel, large ones in kernels of their own.
Every operation is rounded the same way in all of them, so the results are
equal bit for bit.

And what run() queues ahead of what it knows changes nothing, nor does the
compaction of an ensemble's batch.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

GAMMA = 1.7595e11
DT = 2e-14
SMALL = (37, 21, 3)       # odd sizes: scalar paths, partial blocks
TILED = (64, 30, 2)       # TMA tiles, partial blocks
LARGE = (1028, 1020, 3)   # separate stage and error kernels, 16-byte loads
LARGE_ODD = (1031, 1021, 3)  # the same, scalar loads


def make(N, solver, regions, geom):
    from umagnus_b200 import engine
    rng = np.random.default_rng(3)
    kw = {}
    if regions:
        kw["regions"] = rng.integers(0, 3, N[::-1]).astype(np.uint8)
    if geom:
        g = np.ones(N[::-1], np.float32)
        g[:, : N[1] // 3, : N[0] // 3] = 0
        kw["geom"] = g
    return engine.Simulation(N, (3e-9, 3e-9, 4e-9), 8e5, 1.3e-11, 0.1, Ku1=2e4, B_ext=(0.01, 0.0, 0.02),
                             solver=solver, FixDt=DT, demag=False, **kw)


def one_step(sim, probe, m, solver, vol):
    """What the solver makes of state m: (new state, error torque, last torque)."""
    from umagnus_b200 import opencl
    h = np.float32(DT * GAMMA)

    def torque(x):
        probe.restore_m(x)
        return probe.torque()

    def stage(cs, ks, base=m, normalize=True):
        out = torch.empty_like(m)
        opencl.Madd(out, [base] + ks, [1.0] + [float(np.float32(np.float32(c) * h)) for c in cs])
        if normalize:
            opencl.Normalize(out, vol) if vol is not None else opencl.Normalize(out)
        return out

    k1 = torque(m)
    if solver == 2:
        y = stage([1.0], [k1], normalize=False)
        k2 = torque(y)
        return stage([0.5, -0.5], [k2, k1], base=y), (k1 - k2), k2
    if solver == 4:
        k2 = torque(stage([1 / 2], [k1]))
        k3 = torque(stage([1 / 2], [k2]))
        k4 = torque(stage([1.0], [k3]))
        return stage([1 / 6, 1 / 3, 1 / 3, 1 / 6], [k1, k2, k3, k4]), (k1 - k4), k4
    if solver == 3:
        k2 = torque(stage([1 / 2], [k1]))
        k3 = torque(stage([3 / 4], [k2]))
        y = stage([2 / 9, 1 / 3, 4 / 9], [k1, k2, k3])
        k4 = torque(y)
        e = torch.empty_like(m)
        opencl.Madd(e, [k1, k2, k3, k4], [5 / 72, -1 / 12, -1 / 9, 1 / 8])
        return y, e, k4
    ks = [k1]
    for cs in ([1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
               [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
               [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656]):
        ks.append(torque(stage(cs, ks)))
    y = stage([35 / 384, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84], [ks[0]] + ks[2:])
    k7 = torque(y)
    e = torch.empty_like(m)
    opencl.Madd(e, [ks[0]] + ks[2:] + [k7], [71 / 57600, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40])
    return y, e, k7


@pytest.mark.parametrize("solver", [2, 3, 4, 5])
@pytest.mark.parametrize("N,regions,geom", [(SMALL, False, False), (SMALL, True, True), (TILED, False, True),
                                            (LARGE, False, False), (LARGE_ODD, True, False)],
                         ids=["small", "small-regions-geom", "tiled-geom", "large", "large-odd-regions"])
def test_step_equals_device_ops(solver, N, regions, geom):
    from umagnus_b200 import opencl
    sim, probe = make(N, solver, regions, geom), make(N, solver, regions, geom)
    m = torch.randn((3,) + N[::-1], device="cuda", generator=torch.Generator("cuda").manual_seed(7))
    sim.set_m(m)
    m = sim.get_m()
    vol = (m != 0).any(0).float().contiguous() if geom else None
    want, err, last = one_step(sim, probe, m, solver, vol)
    sim.steps(1)
    assert torch.equal(sim.get_m(), want)
    st = sim.state()
    assert st["nsteps"] == 1 and st["status"] == 0
    # float32 maxima of squared norms: equal up to the rounding of the square root
    h = float(np.float32(DT * GAMMA))
    assert st["last_err"] == pytest.approx(opencl.MaxVecNorm(err) * h, rel=1e-6)
    assert st["last_torque"] == pytest.approx(opencl.MaxVecNorm(last), rel=1e-6)
    # a second step starts from the swapped buffers
    want2, _, _ = one_step(sim, probe, want, solver, vol)
    sim.steps(1)
    assert torch.equal(sim.get_m(), want2)
    sim.free()
    probe.free()


@pytest.mark.parametrize("chunk", [1, 3, 16, 64, 1000])
def test_run_does_not_depend_on_the_block_size(chunk):
    """run() queues steps ahead of what it knows; steps past the stop time change nothing."""
    from umagnus_b200 import engine

    def start():
        s = engine.Simulation((40, 24, 1), (4e-9, 4e-9, 3e-9), 8e5, 1.3e-11, 0.1, B_ext=(0, 0, 0.01))
        s.set_m(torch.randn((3, 1, 24, 40), device="cuda", generator=torch.Generator("cuda").manual_seed(9)))
        return s

    a, b = start(), start()
    T = 8e-12
    a.run(T, chunk=chunk)
    b.run(T)
    assert a.state() == b.state() and a.state()["status"] == 0
    assert a.state()["time"] >= T * (1 - 1e-12)
    assert torch.equal(a.get_m(), b.get_m())
    # bounded: exactly max_steps attempts
    c = start()
    c.run(1.0, chunk=chunk, max_steps=21)
    st = c.state()
    assert st["nsteps"] + st["nundone"] == 21
    d = start()
    d.steps(21)
    assert torch.equal(c.get_m(), d.get_m())
    a.run(T, chunk=chunk)  # a second run restarts from the stop time
    assert a.state()["time"] >= 2 * T * (1 - 1e-12)
    for s in (a, b, c, d):
        s.free()


def test_ensemble_compacts_long_runs():
    """Stiff instances among soft ones run several hundred steps longer, enough for a smaller batch: all still
    equal their single runs."""
    from umagnus_b200 import engine
    insts = [dict(N=(32, 32, 1), cell=(4e-9, 4e-9, 3e-9), Msat=8e5, Aex=2e-11 if i in (1, 6) else 2e-12, alpha=0.1,
                  B_ext=(0.0, 0.0, 0.01 * i)) for i in range(9)]
    rng = np.random.default_rng(4)
    m0 = [rng.standard_normal((3, 1, 32, 32)).astype(np.float32) for _ in insts]
    T = 1e-10
    ens = engine.Ensemble(insts)
    for i, m in enumerate(m0):
        ens.set_m(i, m)
    ens.run(T)
    n = [ens.state(i)["nsteps"] for i in range(9)]
    assert max(n) - sorted(n)[6] > 128, n  # seven finish while the others have far to go
    for i, d in enumerate(insts):
        sim = engine.Simulation(d["N"], d["cell"], d["Msat"], d["Aex"], d["alpha"], B_ext=d["B_ext"])
        sim.set_m(m0[i])
        sim.run(T)
        assert ens.state(i) == sim.state()
        assert np.array_equal(np.asarray(ens.get_m(i)), sim.get_m().cpu().numpy()), i
        sim.free()
    ens.free()
