"""The kernel shape of a handle whose tile shape nobody set: 10x10 tiles with
programmatically dependent launches on small grids. In exact precision every
shape computes the same float operations, so the default's states equal those
of an explicitly set shape bit for bit; the sizes are the rule's edges (444
tiles of 10x10 on 148 SMs), ragged tiles, and grids below one tile row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(rn, s, tile, calls, precision="exact"):
    g = rn.GPUSolver(s.Nx, s.Nr)
    g.setPrecision(precision)
    if tile:
        g.setTile(tile)
    g.setGeometry(s.geo)
    init = s.initialState()
    g.setState(init["A"], init["B"])
    for n in calls:
        g.step(n, s.P)
    out = g.readAll(), g.readStepInfo()
    g.close()
    return out


@pytest.mark.parametrize("kind,Nx,Nr", [("viscous_plume", 96, 17), ("plain_small", 101, 38), ("viscous_plume", 203, 77),
                                        ("viscous_plume", 370, 120), ("viscous_plume", 370, 121),
                                        ("plain_small", 371, 120)])
def test_default_shape_matches_set_shape(rn, kind, Nx, Nr):
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(getattr(configs, kind)(Nx, Nr)[0])
    # single launches, graph replays of either parity, a remainder
    calls = (1, 13, 4, 4, 15)
    a, b = run(rn, s, None, calls), run(rn, s, "16x16", calls)
    assert np.array_equal(a[0]["A"], b[0]["A"]) and np.array_equal(a[0]["B"], b[0]["B"])
    assert np.array_equal(a[1], b[1])


def test_resize_follows_the_default_shape(rn):
    """A resized handle with an unset shape steps the new grid as a new handle does."""
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(configs.viscous_plume(512, 192)[0])
    g = rn.GPUSolver(128, 48)
    g.resize(s.Nx, s.Nr)
    g.setPrecision("exact")
    g.setGeometry(s.geo)
    init = s.initialState()
    g.setState(init["A"], init["B"])
    g.step(7, s.P)
    ref = run(rn, s, None, (7,))
    out = g.readAll()
    assert np.array_equal(out["A"], ref[0]["A"]) and np.array_equal(out["B"], ref[0]["B"])
    g.close()
