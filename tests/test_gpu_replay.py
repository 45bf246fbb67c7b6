"""Evaluations from the fourth of a kind on replay a captured graph: what they
give is what a fresh force field gives eagerly, byte for byte (where both have
built their list from the same positions), on unchanged positions, on frames displaced beyond the skin (the rebuild is the graph's
conditional node), in a scaled and in a sheared cell, after the list's buffers
were replaced and after a change of launch shape, with and without energies,
with the reciprocal part (positions gathered after the rebuild) and without
(copied by the displacement check)."""

import numpy as np
import pytest

import heddle_b200 as hb
import oracle as O
from heddle_b200 import systems as S

pytestmark = pytest.mark.gpu

SCALARS = ("lj", "coulomb_real", "recip", "potential", "virial")


def fresh(ctx, spec, box, pos, reciprocal, scalars):
    """Forces and scalars of a first, eager evaluation."""
    sys_ = hb.System.from_spec(ctx, spec)
    sys_.set_box(box)
    sys_.set_state_f32(pos)
    ff = hb.ForceField.from_spec(sys_, spec, reciprocal=reciprocal)
    ff.step(scalars=scalars)
    out = sys_.forces(), ff.scalars() if scalars else None
    ff.close()
    sys_.close()
    return out


@pytest.mark.parametrize("reciprocal", [True, False], ids=["spme", "pairs"])
@pytest.mark.parametrize("scalars", [False, True], ids=["forces", "energies"])
def test_replay_equals_eager(ctx, reciprocal, scalars):
    spec = S.spc_water(343, r_cut_A=7.0, skin_A=1.0, seed=3)
    L = spec.box[0]
    cell = np.array([L, L, L, 0.0, 0.0, 0.0])
    start = spec.positions.astype(np.float32)
    other = S.spc_water(343, r_cut_A=7.0, skin_A=1.0, seed=4).positions.astype(np.float32)
    rng = np.random.default_rng(9)
    near = (start + rng.uniform(-0.02, 0.02, size=start.shape)).astype(np.float32)
    wide = cell * 1.04
    shear = wide + np.array([0.0, 0.0, 0.0, 0.08 * L, -0.05 * L, 0.06 * L])
    sys_ = hb.System.from_spec(ctx, spec)
    sys_.set_state_f32(start)
    ff = hb.ForceField.from_spec(sys_, spec, reciprocal=reciprocal)

    def check(pos, box, rebuilt, change=None):
        if change is not None:
            change()
        before = ff.stats()["rebuilds"]
        sys_.set_state_f32(pos)
        ff.step(scalars=scalars)
        F = sys_.forces()
        assert (ff.stats()["rebuilds"] != before) == rebuilt
        Fe, se = fresh(ctx, spec, box, pos, reciprocal, scalars)
        if pos is near:
            # the list of an earlier frame: atoms shifted next to other tiles'
            # centres round their positions (6e-8) otherwise
            assert np.sqrt(((F - Fe) ** 2).sum() / (Fe ** 2).sum()) <= 2e-6
            return F
        assert np.array_equal(F, Fe)
        if scalars:
            sc = ff.scalars()
            assert all(sc[k] == se[k] for k in SCALARS), (sc, se)
        return F

    for _ in range(5):  # three eager, the capture, a replay
        F = check(start, cell, False)
    if reciprocal:
        Fo, _, _, _ = O.forces(spec, start.astype(np.float64))
        assert np.sqrt(((F - Fo) ** 2).sum() / (Fo ** 2).sum()) <= 1e-5
    check(near, cell, False)      # within the skin: no rebuild
    check(other, cell, True)      # a rebuild inside the replay
    check(start, cell, True)
    check(start, cell, False)
    check(start, wide, True, lambda: sys_.set_box(wide))
    check(other, wide, True)
    check(other, shear, True, lambda: sys_.set_box(shear))
    check(start, shear, True)
    check(start, cell, True, lambda: sys_.set_box(cell))
    # new list buffers: eager again, captured anew
    slab = ff.capacity()["slab"]
    check(start, cell, False, lambda: ff.set_launch(nl_slab=slab + 5))
    for pos, rebuilt in ((start, False), (other, True), (other, False), (start, True), (near, False)):
        check(pos, cell, rebuilt)
    # launch shapes are baked into the graph
    check(start, cell, False, lambda: ff.set_launch(pair_chunk=3))
    for pos, rebuilt in ((other, True), (other, False), (start, True), (start, False), (other, True)):
        check(pos, cell, rebuilt)
    ff.close()
    sys_.close()


def test_kinds_interleaved_and_two_force_fields(ctx):
    """The two kinds' graphs and two force fields of one system take turns."""
    spec = S.spc_water(216, r_cut_A=6.5, skin_A=0.8, seed=5)
    frames = [S.spc_water(216, r_cut_A=6.5, skin_A=0.8, seed=s).positions.astype(np.float32) for s in (5, 6)]
    want = {(k, sc): fresh(ctx, spec, spec.box, frames[k], True, sc) for k in (0, 1) for sc in (False, True)}
    sys_ = hb.System.from_spec(ctx, spec)
    sys_.set_state_f32(frames[0])
    ffs = [hb.ForceField.from_spec(sys_, spec) for _ in range(2)]
    for k in range(24):
        ff, frame, sc = ffs[k % 2], (k // 2) % 2, k % 3 == 0
        sys_.set_state_f32(frames[frame])
        ff.step(scalars=sc)
        F, s = want[(frame, sc)]
        assert np.array_equal(sys_.forces(), F), k
        if sc:
            assert all(ff.scalars()[q] == s[q] for q in SCALARS), k
    for ff in ffs:
        ff.close()
    sys_.close()


@pytest.mark.parametrize("n", [5450, 5803, 9000])
def test_list_rebuilt_in_a_replay_matches_oracle(ctx, n):
    """The graph's rebuild on both sides of the candidate sweep by groups of
    32 tiles (512 tiles), pair for pair."""
    spec = S.spc_water(n, r_cut_A=6.0, skin_A=1.0, seed=2)
    frames = [spec.positions.astype(np.float32),
              S.spc_water(n, r_cut_A=6.0, skin_A=1.0, seed=7).positions.astype(np.float32)]
    sys_ = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(sys_, spec, reciprocal=False)
    for k in range(6):
        sys_.set_state_f32(frames[k % 2])
        ff.step()
    before = ff.stats()["rebuilds"]
    sys_.set_state_f32(frames[0])
    ff.step()
    assert ff.stats()["rebuilds"] != before
    pairs, dup = ff.neighbor_pairs()
    pos = sys_.positions().astype(np.float32)
    rc = max(float(np.max(spec.lj_cutoff[spec.lj_epsilon != 0])), spec.r_cut_coul or 0.0)
    ref = O.neighbor_pairs_f32(pos, spec.box.astype(np.float32), np.float32(rc + spec.r_skin))
    ff.close()
    sys_.close()
    assert dup == 0
    assert np.array_equal(pairs, ref)
