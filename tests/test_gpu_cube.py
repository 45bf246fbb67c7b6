"""The one-cluster transform of small cubic grids: every size against the
FP64 oracle and the line passes, with and without energies, in orthorhombic
and tilted cells; the charge grid comes back cleared (a second evaluation
gives the same bytes)."""

import numpy as np
import pytest

import heddle_b200 as hb
import oracle as O
from heddle_b200 import _native as N
from heddle_b200 import systems as S

pytestmark = pytest.mark.gpu


def rms(F, R):
    return float(np.sqrt(((F - R) ** 2).sum() / (R ** 2).sum()))


@pytest.mark.parametrize("n", [16, 20, 24, 25, 27, 30, 32])
@pytest.mark.parametrize("tilt", [False, True], ids=["ortho", "tilted"])
def test_cube_matches_oracle_and_line_passes(ctx, n, tilt):
    spec = S.spc_water(216, r_cut_A=7.0, skin_A=0.8, seed=n)
    spec.grid = (n, n, n)
    if tilt:
        L = spec.box[0]
        spec.box = np.array([L, L, L, 0.11 * L, -0.07 * L, 0.09 * L])
    sys_ = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(sys_, spec)
    ff.step(scalars=False)
    F0 = sys_.forces()
    ff.step(scalars=True)
    F1, sc = sys_.forces(), ff.scalars()
    ff.step(scalars=False)
    assert np.array_equal(sys_.forces(), F0)
    Fo, _, _, _ = O.forces(spec, sys_.positions())
    _, _, _, T = O.forces(spec, sys_.positions(), poly_erfc=True)
    assert rms(F0, Fo) <= 1e-5 and rms(F1, Fo) <= 1e-5
    assert abs(sc["recip"] - T["recip"]) <= 1e-5 * abs(T["recip"])
    N.check(ff.lib.hb_forcefield_set_launch(ff.h, N.HB_LAUNCH_FFT_PLANE, 0))
    ff.step(scalars=True)
    Fl, sl = sys_.forces(), ff.scalars()
    # both transforms round in single precision: log2(n^3) stages of 6e-8
    # on reciprocal forces no larger than the total
    assert rms(F1, Fl) <= 2e-6
    assert abs(sc["recip"] - sl["recip"]) <= 1e-6 * abs(sl["recip"])
    assert abs(sc["virial_recip"] - sl["virial_recip"]) <= 2e-6 * abs(sl["virial_recip"]) + 1e-6 * abs(sl["recip"])
    ff.close()
    sys_.close()


@pytest.mark.parametrize("grid", [(72, 75, 81), (90, 100, 108), (120, 125, 135), (144, 150, 180)])
def test_compiled_line_sizes_match_oracle(ctx, grid):
    spec = S.spc_water(216, r_cut_A=7.0, skin_A=0.8, seed=5)
    spec.grid = grid
    sys_ = hb.System.from_spec(ctx, spec)
    ff = hb.ForceField.from_spec(sys_, spec)
    ff.step(scalars=True)
    F, sc, pos = sys_.forces(), ff.scalars(), sys_.positions()
    ff.close()
    sys_.close()
    Fo, _, _, _ = O.forces(spec, pos)
    _, _, _, T = O.forces(spec, pos, poly_erfc=True)
    assert rms(F, Fo) <= 1e-5
    assert abs(sc["recip"] - T["recip"]) <= 1e-5 * abs(T["recip"])
