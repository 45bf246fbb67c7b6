"""The packed list's candidate sweep and refinement against the oracle's pair
list, pair for pair: sizes on both sides of the sweep by groups of 32 tiles
(512 tiles), a last tile and a last group that are nearly empty, tilted cells
(tiles pruned along the face normals), cells too small for a single periodic
copy, and a slab with vacuum (tiles of very different extents)."""

import numpy as np
import pytest

import heddle_b200 as hb
import oracle as O
from heddle_b200 import systems as S

pytestmark = pytest.mark.gpu


def tilted(spec, t):
    L = spec.box[0]
    spec.box = np.array([L, L, L] + [x * L for x in t])
    h = np.array([[L, spec.box[3], spec.box[4]], [0.0, L, spec.box[5]], [0.0, 0.0, L]])
    spec.positions = (spec.positions / L) @ h.T
    spec.excl_offsets = None  # the shear bends the molecules: atoms only
    return spec


def slab(n, L_z):
    spec = S.spc_water(n, r_cut_A=7.0, skin_A=1.5, seed=4)
    spec.box = spec.box * np.array([1.0, 1.0, L_z, 1.0, 1.0, 1.0])
    return spec


CASES = {
    "511-tiles": lambda: S.spc_water(5450, r_cut_A=6.0, skin_A=1.2, seed=2),
    "513-tiles-1-atom": lambda: S.lj_argon(n_atoms=512 * 32 + 1, n_side=26, box_m=9.2e-9, skin_frac=0.1),
    "545-tiles": lambda: S.spc_water(5803, r_cut_A=6.0, skin_A=1.2, seed=2),
    "tilted-small": lambda: tilted(S.spc_water(400, r_cut_A=7.0, skin_A=1.0, seed=5), (0.11, -0.07, 0.09)),
    "tilted-large": lambda: tilted(S.spc_water(5803, r_cut_A=6.0, skin_A=1.0, seed=5), (0.3, 0.25, -0.28)),
    "small-cell": lambda: S.spc_water(300, r_cut_A=8.0, skin_A=1.5, seed=6),
    "slab": lambda: slab(6000, 2.2),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_pair_set_matches_oracle(ctx, case):
    spec = CASES[case]()
    sys_ = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(sys_, spec, reciprocal=False)
    pairs, dup = ff.neighbor_pairs()
    pos = sys_.positions().astype(np.float32)
    rc = max(float(np.max(spec.lj_cutoff[spec.lj_epsilon != 0])), spec.r_cut_coul or 0.0)
    ref = O.neighbor_pairs_f32(pos, spec.box.astype(np.float32), np.float32(rc + spec.r_skin))
    ff.close()
    sys_.close()
    assert dup == 0
    assert np.array_equal(pairs, ref)


def test_candidate_capacities_of_two_force_fields(ctx):
    """Cut-offs that reach more than 640 tiles take more shared memory in the
    tile build than its first size: a second force field with fewer
    candidates leaves the first one's rebuild as it was."""
    specs = [S.spc_water(30000, r_cut_A=40.0, skin_A=4.0, seed=1),
             S.spc_water(20000, r_cut_A=36.0, skin_A=3.6, seed=1)]
    systems = [hb.System.from_spec(ctx, spec) for spec in specs]
    ffs = [hb.ForceField.from_spec(s, spec, reciprocal=False) for s, spec in zip(systems, specs)]
    entries = [ff.stats()["entries"] for ff in ffs]
    for ff, e in zip(ffs, entries):
        assert ff.pre_step(force=True)
        assert ff.stats()["entries"] == e
    for o in ffs + systems:
        o.close()
