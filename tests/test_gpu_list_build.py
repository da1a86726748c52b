"""The neighbour build where its cell sort, screen and warp shares can go
wrong, against the oracle's pair set: pairs placed within FP32 rounding of
cutoff + skin on both sides, boxes small enough for the minimum image inside
the screen, cells split over several warps or holding more atoms than one
pass, sparse long cells, cell counts at and across the scan's chunks, and rows
pinned at the longest row's exact length."""
import numpy as np
import pytest

from conftest import oracle_system


def _pairs(i, j):
    return set(zip(np.minimum(i, j).tolist(), np.maximum(i, j).tolist()))


def _check(atvb, ctx, orc, pos, box, rc, skin):
    n = len(pos)
    desc = dict(n_atoms=n, box=tuple(box), nl_cutoff=rc, nl_skin=skin, lj_enabled=1,
                lj_epsilon=1e-3, lj_sigma=0.3, lj_cutoff=rc, dt=0.01)
    frame = dict(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), mass=np.ones(n))
    o = oracle_system(orc, desc, frame)
    o.build_list()
    want = _pairs(*o.pairs())
    for precision in (0, 1):
        s = atvb.System(ctx, dict(desc, precision=precision), frame)
        got = _pairs(*s.pairs())
        assert s.scalars()["list_pairs"] == len(want)
        s.close()
        assert got == want


@pytest.mark.gpu
@pytest.mark.parametrize("cells,jitter", [(6, 0.0), (7, 3e-8), (13, 2e-7), (13, 1e-6)])
def test_pairs_at_the_edge_of_the_list(atvb, ctx, orc, cells, jitter):
    # a cubic lattice of spacing 1 with cutoff + skin = 2: six partners per
    # atom at 2 +- the jitter, inside the screen's error band
    g = np.arange(cells) + 0.25
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(cells)
    pos = pos + jitter * rng.uniform(-1, 1, size=pos.shape)
    _check(atvb, ctx, orc, pos, (cells,) * 3, 1.75, 0.25)


@pytest.mark.gpu
@pytest.mark.parametrize("n,box,rc", [
    (40, (5.7, 5.9, 30.0), 2.5),      # two cells across: minimum image in the screen
    (3000, (9.0, 9.5, 10.0), 4.0),    # dense cells, several warps and passes per cell
    (900, (30.0, 31.0, 33.0), 1.2),   # sparse, reach 1
    (8193, (21.0, 22.0, 23.0), 2.2),  # long cells; more atoms than the sort's threads
    (49152, (40.0, 41.0, 43.0), 0.9),  # the largest sort in one cluster
    (49153, (40.0, 41.0, 43.0), 0.9),  # and the smallest in several kernels
    (65537, (40.0, 41.0, 43.0), 0.9),
    (20000, (20.48, 20.48, 81.92), 1.0),  # several scan chunks
])
def test_random_positions(atvb, ctx, orc, n, box, rc):
    rng = np.random.default_rng(n)
    pos = rng.uniform(size=(n, 3)) * np.array(box)
    _check(atvb, ctx, orc, pos, box, rc, 0.3)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("cells", [6, 13])
@pytest.mark.parametrize("special", [False, True])
def test_rows_pinned_at_their_exact_length(atvb, ctx, orc, cells, precision, special):
    # the lattice stretched so that about one in eight of the six partners at
    # cutoff + skin is listed, the others in the screen's error band but out:
    # rows hold 26 to about 30 entries out of 32 candidates, in any order
    g = np.arange(cells) + 0.25
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) * (1.0 + 5e-7)
    pos += 1e-6 * np.random.default_rng(cells).uniform(-1, 1, size=pos.shape)
    n, L = len(pos), cells * (1.0 + 5e-7)
    desc = dict(n_atoms=n, box=(L,) * 3, nl_cutoff=1.75, nl_skin=0.25, lj_enabled=1,
                lj_epsilon=1e-3, lj_sigma=0.3, lj_cutoff=1.75, dt=0.01, precision=precision)
    frame = dict(x=pos[:, 0].copy(), y=pos[:, 1].copy(), z=pos[:, 2].copy(), mass=np.ones(n))
    opts = {}
    if special:  # entries carry a class
        t = np.arange(1, n, 3)
        opts["special_bonds"] = dict(lj=(0.0, 0.5, 0.5), coul=(0.0, 0.5, 0.5),
                                     bonds=np.stack([t, t + 1], 1))
    o = oracle_system(orc, desc, frame)
    o.build_list()
    want = _pairs(*o.pairs())
    row = np.zeros(n, int)
    np.add.at(row, np.array(sorted(want)).ravel(), 1)
    longest = int(row.max())
    assert 26 <= row.min() and longest < 32
    free = atvb.System(ctx, desc, frame, **opts)
    free.compute_forces()
    assert free.scalars()["max_neighbors"] == longest
    s = atvb.System(ctx, desc, frame, **opts)
    s.set_capacity(row_capacity=longest)
    assert _pairs(*s.pairs()) == want
    sc = s.scalars()
    assert sc["list_pairs"] == len(want) and sc["max_neighbors"] == longest
    s.compute_forces()
    (fa, sa), (fb, sb) = free.download(), s.download()
    for k in fa:
        assert np.array_equal(fa[k], fb[k]), k
    assert sa["energy"] == sb["energy"]
    for cut in range(26, longest):
        # some true pair has no place: flagged, with the length it needs
        s.set_capacity(row_capacity=cut)
        sc = s.scalars(check=False)
        assert sc["status_bits"] & 1 and sc["max_neighbors"] == longest
        # and what a cut row holds are listed pairs, none of them twice
        i, j = s.pairs()
        assert len(_pairs(i, j)) == len(i) and _pairs(i, j) <= want
        with pytest.raises(atvb.AtvbError):
            s.compute_forces()
        s.clear_status()
