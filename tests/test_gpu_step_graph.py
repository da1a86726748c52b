"""Steps in one call against steps one at a time, bit for bit: long calls run
in a graph of several steps (for NVE and Langevin the final half of a step and
the initial half of the next in one kernel).  Engines below 100,000 atoms launch
the chain as programmatic dependents and run the scalar updates in the last
block of the atom passes; larger ones have them as kernels and the list build
in conditional nodes.  One item per system, several, systems of uneven size in
one engine, both cell sorts, with and without PME."""
import numpy as np
import pytest

KEYS = ("x", "y", "z", "vx", "vy", "vz", "fx", "fy", "fz")


def _same(a, b):
    (fa, sa), (fb, sb) = a, b
    for k in KEYS:
        assert np.array_equal(fa[k], fb[k]), k
    for k in ("energy", "kinetic", "conserved", "nh_xi", "step", "rebuilds", "list_pairs"):
        assert sa[k] == sb[k], k
    assert np.array_equal(sa["stress"], sb["stress"])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("thermostat", [0, 1, 2])
@pytest.mark.parametrize("n", [255, 257, 2047])
def test_long_calls_equal_single_steps(atvb, ctx, precision, thermostat, n):
    from atomiverse_b200 import workloads as W
    ncell = int(np.ceil((n / 4) ** (1 / 3)))
    desc, frame = W.lj_fcc(ncell=ncell, n_keep=n, seed=n, precision=precision,
                           thermostat=thermostat)
    desc.update(stress_required=1, tau=50.0)
    one, many = (atvb.System(ctx, desc, frame) for _ in range(2))
    for s in (one, many):
        s.compute_forces()
    for _ in range(67):
        one.step(1)
    many.step(30)        # the longer graph stands after the first steps
    many.step(37)
    _same(one.download(), many.download())
    assert np.array_equal(one.history(67), many.history(67))


@pytest.mark.gpu
@pytest.mark.parametrize("thermostat", [0, 1, 2])
def test_a_first_long_call_runs_the_longer_graph(atvb, ctx, thermostat):
    from atomiverse_b200 import workloads as W
    desc, frame = W.lj_fcc(ncell=6, seed=4, thermostat=thermostat)
    desc.update(tau=50.0)
    one, many, short = (atvb.System(ctx, desc, frame) for _ in range(3))
    for s in (one, many, short):
        s.compute_forces()
    for _ in range(70):
        one.step(1)
    per_step = one.launch_count()
    many.step(70)
    # 8 launches of eight steps, a pass less between two steps of each where
    # no sum of the whole system stands between the halves
    merged = 0 if thermostat == 1 else 8 * 7
    assert many.launch_count() == 70 * per_step - merged
    short.step(20)  # too short to pay for the capture
    assert short.launch_count() == 20 * per_step
    _same(one.download(), many.download())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nose_hoover", [False, True])
def test_uneven_batch_equals_single_steps(atvb, ctx, precision, nose_hoover):
    # one Nose-Hoover system keeps every system's half steps apart
    from atomiverse_b200 import workloads as W
    items = [W.lj_fcc(ncell=c, seed=c, precision=precision, thermostat=c % 2 * 2)
             for c in (4, 9, 13)]
    items.append(W.rocksalt_melt(ncell=8, rc=9.0, grid=(24, 24, 24), precision=precision))
    if not nose_hoover:
        items[-1][0].update(thermostat=2, damp=100.0, seed=5)
    one, many = (atvb.Batch(ctx, items) for _ in range(2))
    for b in (one, many):
        b.compute_forces()
    for _ in range(44):
        one.step(1)
    per_step = one.launch_count()
    many.step(25)
    many.step(19)
    assert many.launch_count() == 19 * per_step - (0 if nose_hoover else 2 * 7)
    for k in range(len(items)):
        _same(one.download(k), many.download(k))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sizes", [
    (70000,),        # the cell sort of several kernels, as programmatic launches
    (70000, 4000),   # and beside the sort in one cluster
    (108000,),       # scalar kernels, conditional list build
    (70000, 33000),  # the same with both sorts
])
@pytest.mark.parametrize("thermostat", [0, 1, 2])
def test_large_engines_equal_single_steps(atvb, ctx, precision, sizes, thermostat):
    from atomiverse_b200 import workloads as W
    items = []
    for n in sizes:
        desc, frame = W.lj_fcc(ncell=int(np.ceil((n / 4) ** (1 / 3))), n_keep=n, seed=n,
                               precision=precision, thermostat=thermostat)
        desc.update(tau=50.0, stress_required=1)
        items.append((desc, frame))
    one, many = (atvb.Batch(ctx, items) for _ in range(2))
    for b in (one, many):
        b.compute_forces()
    for _ in range(57):
        one.step(1)
    per_step = one.launch_count()
    many.step(57)
    if thermostat != 1:  # seven launches of eight steps; a scalar kernel less too
        assert many.launch_count() == 57 * per_step - 7 * 7 * (2 if sum(sizes) >= 100000 else 1)
    for k in range(len(items)):
        a, b = one.download(k), many.download(k)
        assert a[1]["rebuilds"] >= 3
        _same(a, b)
    one.close()
    many.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ncell", [12, 48])
@pytest.mark.parametrize("thermostat", [0, 2])
def test_merged_halves_with_pme_equal_single_steps(atvb, ctx, precision, ncell, thermostat):
    from atomiverse_b200 import workloads as W
    K = 32 if ncell == 12 else 96
    desc, frame = W.rocksalt_melt(ncell=ncell, rc=9.0, grid=(K, K, K), precision=precision)
    desc.update(thermostat=thermostat, damp=100.0, seed=3, dt=4.0)
    one, many = (atvb.System(ctx, desc, frame) for _ in range(2))
    for s in (one, many):
        s.compute_forces()
    for _ in range(53):
        one.step(1)
    per_step = one.launch_count()
    many.step(53)
    assert many.launch_count() == 53 * per_step - 6 * 7 * (1 if ncell == 12 else 2)
    a, b = one.download(), many.download()
    assert a[1]["rebuilds"] >= 2
    _same(a, b)


@pytest.mark.gpu
def test_stop_on_nan_inside_a_long_call(atvb, ctx):
    # atoms at rest, further apart than the list reaches, but for one that
    # flies at its neighbour; the force when the two come within the cutoff
    # takes its velocity out of range at a step known beforehand, well inside
    # the second long call (in the middle of a graph of eight steps).  The step
    # it stops at and the state it leaves do not depend on how the steps were
    # called
    m, sp, rc, dt, vz = 6, 4.0, 2.5, 0.05, 0.53
    g = (np.arange(m) + 0.5) * sp
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    n = len(pos)
    frame = dict(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(),
                 vx=np.zeros(n), vy=np.zeros(n), vz=np.zeros(n), mass=np.full(n, 1e-9))
    frame["vz"][7] = vz  # towards atom 8
    desc = dict(n_atoms=n, box=(m * sp,) * 3, nl_cutoff=rc, nl_skin=0.3, lj_enabled=1,
                lj_epsilon=3e306, lj_sigma=1.0, lj_cutoff=rc, dt=dt)
    contact = int(np.floor((sp - rc) / (vz * dt))) + 1
    assert 31 + 16 < contact < 31 + 32 and (contact - 31) % 8 not in (0, 7)
    got = []
    for calls in ([1] * 70, [30, 40]):
        s = atvb.System(ctx, desc, frame)
        s.step(1)
        s.set_stop_on_nan(True)
        for c in calls:
            try:
                s.step(c)
            except atvb.PhysicsError:
                break
        sc = s.scalars(check=False)
        assert sc["halted"] and sc["status_bits"] & 8
        # the force of step `contact` is applied by its final half, and the
        # drift of the step after it finds the velocity
        assert sc["step"] == contact + 1
        got.append((sc, s.download(check=False)[0]))
    (sa, fa), (sb, fb) = got
    assert sa["status_bits"] == sb["status_bits"] and sa["rebuilds"] == sb["rebuilds"]
    for k in KEYS:
        assert np.array_equal(fa[k], fb[k], equal_nan=True), k
    bad = ~np.isfinite(fa["vz"])
    assert bad[7] and bad.sum() == 2  # the pair, and nothing else
