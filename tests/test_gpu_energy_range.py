"""Energies and virials of atoms that nearly coincide: the pair kernels sum
them in fixed point, and a sum beyond one word's 2^31 eV must neither wrap to
an ordinary value nor lose the ordinary shares beside it."""
import numpy as np
import pytest

from conftest import oracle_system

EPS, SIG, RC, SP, M = 0.0104, 3.4, 8.5, 5.0, 8


def _frame(gap, pairs, charge=0.0):
    """A cubic lattice of M^3 atoms; `pairs` of them, spread over the box,
    brought to `gap` sigma from a neighbour."""
    g = (np.arange(M) + 0.5) * SP
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    pos += np.random.default_rng(pairs).uniform(-0.2, 0.2, size=pos.shape)
    for k in range(pairs):
        i = (k * (M ** 3 // pairs)) // 2 * 2
        pos[i + 1] = pos[i] + gap * SIG * np.array([0.48, 0.6, 0.64])
    q = np.full(len(pos), charge)
    return dict(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(),
                mass=np.ones(len(pos)), charge=q)


def _desc(precision, **over):
    d = dict(n_atoms=M ** 3, box=(M * SP,) * 3, precision=precision, nl_cutoff=RC, nl_skin=1.0,
             lj_enabled=1, lj_epsilon=EPS, lj_sigma=SIG, lj_cutoff=RC, dt=1.0, stress_required=1)
    d.update(over)
    return d


# relative error of a term in r^-12 (r^-14 times components for the virial):
# 12 (14) times that of r.  FP64: a few 2^-53 of the coordinates (20 A) over r
# = 0.34 A, 1e-13.  Mixed: the 32-bit fixed-point quantum 40 / 2^32 A of each
# coordinate over 0.34 A, 3e-8 per axis, 14 x 2 of it 8e-7, and some 20
# roundings of 6e-8
TOL = {0: 1e-11, 1: 4e-6}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("types", [False, True])
@pytest.mark.parametrize("pairs", [1, 37])
def test_overlapping_atoms(atvb, ctx, orc, precision, types, pairs):
    desc, frame = _desc(precision), _frame(0.1, pairs)
    o = oracle_system(orc, desc, frame)
    opts = {}
    if types:  # the general pair kernel
        opts["lj_types"] = [(0, 0, EPS, SIG)]
        frame["type"] = np.zeros(M ** 3, np.int32)
        o.set_lj_types(opts["lj_types"], frame["type"])
    o.build_list()
    o.compute_forces()
    want = o.scalars()
    assert want["e_lj"] > 2.0 ** 31 * pairs  # above the range of one word
    s = atvb.System(ctx, desc, frame, **opts)
    s.compute_forces()
    got = s.scalars(check=False)
    assert abs(got["energy_lj"] / want["e_lj"] - 1.0) < TOL[precision]
    assert np.allclose(got["stress"], want["virial"], rtol=TOL[precision],
                       atol=TOL[precision] * np.abs(want["virial"]).max())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_wide_shares_leave_the_others_exact(atvb, ctx, orc, precision):
    # a gap that gives shares just above the line at which they leave the
    # columns: the sum stays that of FP64
    desc, frame = _desc(precision), _frame(0.36, 20)
    o = oracle_system(orc, desc, frame)
    o.build_list()
    o.compute_forces()
    want = o.scalars()
    assert 512.0 * 20 < want["e_lj"] < 2.0 ** 31
    s = atvb.System(ctx, desc, frame)
    s.compute_forces()
    got = s.scalars()
    assert abs(got["energy_lj"] / want["e_lj"] - 1.0) < TOL[precision]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("charge", [0.0, 1.0])
@pytest.mark.parametrize("gap", [1e-3, 1e-6])
def test_energies_beyond_any_range_stay_large(atvb, ctx, precision, charge, gap):
    # 1e34 eV and more (infinite or not a number in FP32): cut off, not wrapped
    over = dict(coul_enabled=1, coul_alpha=0.3, coul_cutoff=RC) if charge else {}
    s = atvb.System(ctx, _desc(precision, **over), _frame(gap, 5, charge))
    s.compute_forces()
    got = s.scalars(check=False)
    assert np.isfinite(got["energy"]) and got["energy"] > 2.0 ** 40
    if charge:
        assert np.isfinite(got["energy_coul"])
