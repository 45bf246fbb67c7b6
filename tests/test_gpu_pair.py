"""The pair kernel at the edges of its tiles and tables, against the FP64
oracle: atom counts around multiples of the 32-atom tile, single-copy,
orthorhombic and tilted minimum images, one and several atom types (more than
32 take another type test), listed exclusions with and without scales, forces
with and without energies, the exact form, and any split of the entries into
work items."""

import threading

import numpy as np
import pytest

import heddle_b200 as hb
import oracle as O
from heddle_b200 import HeddleError
from heddle_b200 import systems as S
from heddle_b200 import units as U

pytestmark = pytest.mark.gpu


def system(n, edge_A, tilt, n_types, scaled, seed=3):
    """n charged Lennard-Jones atoms on jittered lattice sites, chained by
    exclusions (1-2 excluded, 1-3 scaled when `scaled`)."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    L = U.angstrom_au(edge_A)
    sites = np.array([(i, j, k) for i in range(side) for j in range(side) for k in range(side)])
    sites = sites[rng.permutation(len(sites))[:n]]
    f = (sites + 0.5 + rng.uniform(-0.1, 0.1, size=(n, 3))) / side - 0.5
    box = np.array([L, L, L] + [t * L for t in tilt])
    h = np.array([[L, box[3], box[4]], [0.0, L, box[5]], [0.0, 0.0, L]])
    q = rng.uniform(-0.6, 0.6, size=n)
    types = rng.integers(0, n_types, size=n).astype(np.uint32)
    rc = U.angstrom_au(6.0)
    sg = U.angstrom_au(2.0 + rng.uniform(0.0, 0.4, size=(n_types, n_types)))
    ep = U.energy_au_kj_per_mol(rng.uniform(0.2, 0.8, size=(n_types, n_types)))
    ep[0, :] = ep[:, 0] = 0.0 if n_types > 1 else ep[0, 0]  # a type without the term
    sg, ep = 0.5 * (sg + sg.T), 0.5 * (ep + ep.T)
    adj = [{} for _ in range(n)]
    for i in range(n):
        for d, s in ((1, (0.0, 0.0)), (2, (0.5, 0.8) if scaled else (0.0, 0.0))):
            if i + d < n and i % 7 + d < 7:
                adj[i][i + d] = adj[i + d][i] = s
    off = np.concatenate([[0], np.cumsum([len(a) for a in adj])]).astype(np.uint32)
    part = np.array([j for a in adj for j in sorted(a)], dtype=np.uint32)
    sc = np.array([a[j] for a in adj for j in sorted(a)]).reshape(-1, 2)
    return S.SystemSpec(
        name="pairs", positions=f @ h.T, velocities=np.zeros((n, 3)), masses=np.full(n, 1.0e4),
        charges=q, types=types, box=box, n_types=n_types, lj_sigma=sg, lj_epsilon=ep,
        lj_cutoff=np.full((n_types, n_types), rc), lj_switch=np.full((n_types, n_types), 0.9 * rc),
        alpha=2.6 / rc, r_cut_coul=rc, grid=None, excl_offsets=off, excl_partners=part,
        excl_lj=sc[:, 0].copy(), excl_coul=sc[:, 1].copy(), r_skin=U.angstrom_au(0.6))


def off(F, R):
    """RMS error over its bound: 1e-5 of the RMS force (single precision and
    the erfc polynomial's 1.5e-7, with cancellation in an atom's sum) plus
    one unit, 2^-30 hartree/bohr, of the fixed-point pair forces, which is
    what the far pairs of a nearly force-free atom are rounded to."""
    err, size = (float(np.sqrt((x ** 2).sum(axis=1).mean())) for x in (F - R, R))
    return err / (1e-5 * size + 2.0 ** -30)


SMALL = [(9, 1, False), (31, 1, True), (33, 3, False), (64, 40, True), (65, 64, False), (97, 3, True), (161, 33, False)]
CASES = ([("ortho", 13.6, (0.0, 0.0, 0.0), *c) for c in SMALL]
         + [("tilted", 14.6, (0.12, -0.07, 0.1), *c) for c in SMALL]
         + [("single", e, (0.0, 0.0, 0.0), *c) for e, c in ((30.0, (641, 33, False)), (33.0, (993, 1, False)),
                                                              (40.0, (2000, 3, True)))])


@pytest.mark.parametrize("form,edge,tilt,n,n_types,scaled", CASES, ids=[f"{c[0]}-{c[3]}-{c[4]}" for c in CASES])
def test_forces_match_oracle(ctx, form, edge, tilt, n, n_types, scaled):
    spec = system(n, edge, tilt, n_types, scaled)
    sys_ = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(sys_, spec)
    ff.step(scalars=False)
    F = sys_.forces()
    Fo, _, _, _ = O.forces(spec, sys_.positions())
    _, Ep, _, Tp = O.forces(spec, sys_.positions(), poly_erfc=True)
    assert off(F, Fo) <= 1.0, off(F, Fo)
    ff.step(scalars=True)
    assert off(sys_.forces(), Fo) <= 1.0
    e, _ = ff.per_atom()
    # energies: the same, with 2^-28 hartree units and up to 64 pairs an atom
    assert np.abs(e - Ep).max() <= 1e-5 * np.abs(Ep).max() + 64 * 2.0 ** -29
    for chunk in (1, 2, 7, 64):
        ff.set_launch(pair_chunk=chunk)
        ff.step(scalars=False)
        assert np.array_equal(sys_.forces(), F), chunk
    ff.close()
    ff = hb.ForceField.from_spec(sys_, spec, exact_pairs=True)
    ff.step(scalars=False)
    Fx = sys_.forces()
    assert off(Fx, Fo) <= 1.0
    ff.step(scalars=True)
    assert off(sys_.forces(), Fo) <= 1.0
    ff.close()
    sys_.close()


def test_sums_at_the_guard_do_not_wrap(ctx):
    """32 atoms at one point and one atom 4 bohr from them, at the minimum's
    side of sigma = r, where a pair's virial is 24 eps exactly: with eps at and
    around 1 / 48 each of the 32 pairs gives the single atom a half of 0.25
    hartree, 2^26 units, and 32 of those are 2^31."""
    n, L = 33, U.angstrom_au(13.6)
    rc = U.angstrom_au(6.0)
    pos = np.zeros((n, 3))
    pos[32, 0] = 4.0
    types = np.zeros(n, dtype=np.uint32)
    types[32] = 1
    for k in range(-4, 5):
        eps = np.zeros((2, 2))
        eps[0, 1] = eps[1, 0] = (0.5 + k * 2.0 ** -25) / 24.0
        spec = S.SystemSpec(
            name="guard", positions=pos, velocities=np.zeros((n, 3)), masses=np.full(n, 1.0e4),
            charges=np.zeros(n), types=types, box=np.array([L, L, L, 0.0, 0.0, 0.0]), n_types=2,
            lj_sigma=np.full((2, 2), 4.0), lj_epsilon=eps, lj_cutoff=np.full((2, 2), rc),
            lj_switch=np.full((2, 2), rc), alpha=None, r_cut_coul=None, grid=None, excl_offsets=None,
            excl_partners=None, excl_lj=None, excl_coul=None, r_skin=U.angstrom_au(0.6))
        sys_ = hb.System.from_spec(ctx, spec)
        ff = hb.ForceField.from_spec(sys_, spec)
        ff.step(scalars=True)
        _, w = ff.per_atom()
        ff.close()
        sys_.close()
        # 2^-28 units; rsqrt's 2^-22 in sr^12 makes 3e-6 of 0.25 at most
        assert np.abs(w[:32] - 0.25).max() <= 5e-6, (k, w[:32])
        assert abs(w[32] - 8.0) <= 32 * 5e-6, (k, w[32])


def test_two_threads_with_tables_of_different_sizes(ctx):
    """Type tables of more than 28 types need more shared memory than a kernel
    has by default, and that limit belongs to the process: two contexts in two
    threads, one with the largest table and one with a smaller, evaluate at
    the same time without lowering it under each other."""
    specs = [system(97, 13.6, (0.0, 0.0, 0.0), t, False) for t in (64, 40)]
    want, errors = [], []
    for spec in specs:
        sys_ = hb.System.from_spec(ctx, spec)
        ff = hb.ForceField.from_spec(sys_, spec)
        ff.step()
        want.append(sys_.forces())
        ff.close()
        sys_.close()

    def work(k):
        try:
            own = hb.Context(0)
            own.timing(True)  # every evaluation launches its kernels one by one
            sys_ = hb.System.from_spec(own, specs[k])
            ff = hb.ForceField.from_spec(sys_, specs[k])
            for _ in range(1000):
                ff.step()
            assert np.array_equal(sys_.forces(), want[k])
            for o in (ff, sys_, own):
                o.close()
        except Exception as e:
            errors.append((k, e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_launch_defaults_can_be_restored(ctx):
    """0 gives the pair kernel's work item and residency back to the rules by
    size and form; values that are out of range stay refused."""
    spec = system(161, 13.6, (0.0, 0.0, 0.0), 3, False)
    sys_ = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(sys_, spec)
    ff.step()
    F = sys_.forces()
    for kw in (dict(pair_chunk=16), dict(pair_blocks_per_sm=3), dict(pair_chunk=0),
               dict(pair_blocks_per_sm=0)):
        ff.set_launch(**kw)
        ff.step()
        assert np.array_equal(sys_.forces(), F), kw
    for kw in (dict(pair_chunk=-1), dict(pair_chunk=65), dict(pair_blocks_per_sm=-1),
               dict(pair_blocks_per_sm=9)):
        with pytest.raises(HeddleError):
            ff.set_launch(**kw)
    ff.close()
    sys_.close()
