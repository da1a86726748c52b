"""Steps in one call against steps one at a time, bit for bit: a small engine
runs long calls in a graph of several steps (programmatic launches across
steps; for NVE and Langevin the final half of a step and the initial half of
the next in one kernel), and the scalar updates run in the last block of the
atom passes -- one item per system, several, and systems of uneven size in
one engine."""
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
def test_uneven_batch_equals_single_steps(atvb, ctx, precision):
    from atomiverse_b200 import workloads as W
    items = [W.lj_fcc(ncell=c, seed=c, precision=precision, thermostat=2) for c in (4, 9, 13)]
    items.append(W.rocksalt_melt(ncell=8, rc=9.0, grid=(24, 24, 24), precision=precision))
    one, many = (atvb.Batch(ctx, items) for _ in range(2))
    for b in (one, many):
        b.compute_forces()
    for _ in range(44):
        one.step(1)
    many.step(25)
    many.step(19)
    for k in range(len(items)):
        _same(one.download(k), many.download(k))


@pytest.mark.gpu
def test_stop_on_nan_inside_a_long_call(atvb, ctx):
    # a pair driven together overflows some steps in: the halting step and the
    # state it leaves do not depend on how the steps were called
    from atomiverse_b200 import workloads as W
    desc, frame = W.lj_fcc(ncell=5, seed=3)
    frame = {k: v.copy() for k, v in frame.items()}
    frame["vx"][7] = 1e308
    got = []
    for calls in ([1] * 40, [26, 14]):
        s = atvb.System(ctx, desc, frame)
        s.step(1)
        s.clear_status()
        s.set_stop_on_nan(True)
        for c in calls:
            try:
                s.step(c)
            except atvb.PhysicsError:
                break
        sc = s.scalars(check=False)
        got.append((sc["halted"], sc["step"], sc["status_bits"]))
    assert got[0] == got[1]
