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


@pytest.mark.parametrize("kind", ["viscous_plume", "plain_small"])
@pytest.mark.parametrize("tile", ["16x15", "16x16", "16x8", "32x15", None])
def test_cell_classes_follow_the_geometry(rn, oracle, kind, tile):
    """The step kernels take uncut cells' volumes, areas and turbulence lengths
    from the cell classes instead of the geometry planes. A geometry with
    values off the grid's own in single cells and faces (each class bit on and
    off, alone and together, at tile and grid edges, zeros of either sign) steps
    bit for bit as the 14x16 shape steps it in exact precision, which reads the
    planes, and as the oracle but for the wall functions' pow (last bits, 6e-8
    of a wall cell's terms in each of 9 steps: 1e-6); so does the grid's own
    geometry set after it."""
    from helpers import state_rel_l2
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(getattr(configs, kind)(77, 33)[0])
    Nx, Nr = s.Nx, s.Nr
    rng = np.random.default_rng(11)
    geo = dict(s.geo)
    gA, gG, gM = (np.array(geo[k], np.float32) for k in ("geoA", "geoG", "geoM"))
    gA, gG, gM = gA.reshape(Nr + 1, Nx + 1, 4), gG.reshape(Nr, Nx, 4), gM.reshape(Nr, Nx, 4)
    pick = lambda p, sh: rng.uniform(size=sh) < p  # noqa: E731
    for k in (2, 3):
        gA[..., k] = np.where(pick(0.05, gA.shape[:2]), gA[..., k] * np.float32(0.9), gA[..., k])
        gA[..., k] = np.where(pick(0.05, gA.shape[:2]), -gA[..., k], gA[..., k])
    for k in (0, 1):
        gG[..., k] = np.where(pick(0.05, (Nr, Nx)), gG[..., k] * np.float32(1.1), gG[..., k])
    for k in (2, 3):
        gG[..., k] = np.where(pick(0.02, (Nr, Nx)), np.float32(0.2), gG[..., k])
        gG[..., k] = np.where(pick(0.05, (Nr, Nx)) & (gG[..., k] == 0), np.float32(-0.0), gG[..., k])
    gM[..., 3] = np.where(pick(0.1, (Nr, Nx)), np.float32(0.25), gM[..., 3])
    gM[..., 2] = np.where(pick(0.05, (Nr, Nx)) & (gM[..., 2] == 0), np.float32(16.0), gM[..., 2])
    geo.update(geoA=gA.reshape(-1), geoG=gG.reshape(-1), geoM=gM.reshape(-1))
    init = s.initialState()
    g, ref = rn.GPUSolver(Nx, Nr), rn.GPUSolver(Nx, Nr)
    for h in (g, ref):
        h.setPrecision("exact")
    if tile:
        g.setTile(tile)
    ref.setTile("14x16")
    for planes in (geo, s.geo):
        o = oracle.OracleSolver(Nx, Nr)
        for h in (g, ref, o):
            h.setGeometry(planes)
            h.setState(init["A"], init["B"])
            h.step(9, s.P)
        a, b = g.readAll(), ref.readAll()
        assert np.array_equal(a["A"], b["A"]) and np.array_equal(a["B"], b["B"])
        assert max(state_rel_l2(a, o.readAll()).values()) <= 1e-6
    g.close()
    ref.close()


@pytest.mark.parametrize("Nx,Nr", [(128, 48), (300, 61), (512, 130)])
def test_spray_steps_on_each_default_shape(rn, oracle, Nx, Nr):
    """Spray steps (the parcel step and the apply by cell classes, dependent
    launches after the apply) against the oracle in exact precision, through
    single launches and graph replays, on grids of the small shape and of 14x16
    with up to two and up to three blocks an SM. Bar of the exact precision's
    spray cases: only pow, exp, log, sin and cos may differ, in the last bit."""
    from helpers import state_rel_l2
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(configs.injector_spray(Nx, Nr)[0])
    PA, PB, head = configs.prepopulated_parcels(s, 5000)
    init = s.initialState()
    g = rn.GPUSolver(Nx, Nr)
    g.setPrecision("exact")
    g.setGeometry(s.geo)
    g.setState(init["A"], init["B"])
    rn.GPUSpray(g).resize()
    g.spray.setInjector(s.injector)
    g.spray.setParcels(PA, PB, head)
    o = oracle.OracleSolver(Nx, Nr)
    o.setGeometry(s.geo)
    o.setState(init["A"], init["B"])
    o.setInjector(s.injector)
    o.setParcels(PA, PB, head)
    for n in (1, 2, 9, 8):
        g.step(n, s.P)
        o.step(n, s.P)
    assert max(state_rel_l2(g.readAll(), o.readAll()).values()) <= 1e-5
    alive = lambda p: np.asarray(p).reshape(-1, 4)[:, 1] > 0  # noqa: E731
    assert np.array_equal(alive(g.spray.readParcels()["PB"]), alive(o.readParcels()["PB"]))
    g.close()


@pytest.mark.parametrize("kind,Nx,Nr,precision", [("plain_small", 101, 38, "fast"), ("viscous_plume", 128, 48, "fast"),
                                                  ("viscous_plume", 128, 48, "exact"), ("injector_spray", 192, 72, "exact")])
def test_uncut_cells_round_as_the_general_path(rn, kind, Nx, Nr, precision):
    """Uncut cells take their net fluxes from their four faces directly where
    the general path sums a cut-cell group; both round every product and sum
    alike, in fast precision too (but for the oxidiser's scalar sums, which the
    compiler contracts as it likes: sprays in exact precision). A wall vector of
    1e-7 in every uncut cell (below the 1e-6 at which a wall counts) sends the
    same flow through the general path: the states are equal, values below the
    smallest normal float apart (fast precision flushes those to zero or not,
    as an operation comes packed or alone)."""
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(dict(getattr(configs, kind)(Nx, Nr)[0], startMode="burst"))
    init = s.initialState()
    gG = np.array(s.geo["geoG"], np.float32).reshape(-1, 4)
    gG[:, 2] = np.where((gG[:, 2] == 0) & (gG[:, 3] == 0), np.float32(1e-7), gG[:, 2])
    outs = []
    for geo in (s.geo, dict(s.geo, geoG=gG.reshape(-1))):
        g = rn.GPUSolver(s.Nx, s.Nr)
        g.setPrecision(precision)
        g.setTile("16x15")
        g.setGeometry(geo)
        g.setState(init["A"], init["B"])
        if s.injector is not None:
            rn.GPUSpray(g).resize()
            g.spray.setInjector(s.injector)
        g.step(60, s.P)
        outs.append(g.readAll())
        g.close()
    for k in ("A", "B"):
        a, b = (np.where(np.abs(o[k]) < np.finfo(np.float32).tiny, 0, o[k]) for o in outs)
        assert np.array_equal(a, b), (k, np.abs(a - b).max(), (a != b).sum())


def longest_list(geoM, Nx, Nr, TX, TY):
    """Most cells outside one TX x TY tile that belong to a group with a cell inside it."""
    gM = np.asarray(geoM).reshape(Nr, Nx, 4)
    lists = {}
    for j, i in zip(*np.nonzero(gM[..., 2])):
        bits = int(gM[j, i, 2]) & 15
        group = [(j, i)] + [(j + dj, i + di) for b, dj, di in ((1, 0, -1), (2, 0, 1), (4, -1, 0), (8, 1, 0)) if bits & b]
        for a in group:
            t = (a[0] // TY, a[1] // TX)
            lists.setdefault(t, set()).update(c for c in group if (c[0] // TY, c[1] // TX) != t)
    return max(map(len, lists.values()), default=0)


CHANNEL = ((16.4, 40, 16.4, 31.6), (12, 14.6, 12, 36), (12, 40, 12, 14.6), (12, 40, 33.4, 36))
POCKET = ((20, 76, 5, 14.7), (20, 76, 30.3, 40), (20, 31.7, 18, 26))


def blocks_setup(Nx, Nr, blocks):
    """Fluid around solid blocks (x0, x1, r0, r1), in cells. CHANNEL leaves a
    channel one cell and two slivers wide along three sides of the 16 x 16 tile
    at (16, 16): each channel cell and its outer sliver are members outside that
    tile of a group with a sliver inside it. POCKET has slivers just outside the
    32 x 15 tile at (32, 15) merged into it: 32 below, 32 above, 8 on the left."""
    from types import SimpleNamespace
    from rocket_nozzle_cfd_solver_b200 import cutcell
    contour = SimpleNamespace(xe=-1.0, xt=0.0, Rt=0.0, radiusAt=lambda x: 0.0)
    inp = {"Nx": Nx, "Nr": Nr, "dx": 1.0, "contour": contour, "tw": 0.0, "base": False, "xBase": 0.0, "bodyR": 0.0,
           "solids": [dict(zip(("x0", "x1", "r0", "r1"), b)) for b in blocks]}
    return {"cutInput": inp, "contour": contour, "rinCol": np.zeros(Nx, np.float32), "iExit": 0, "dx": 1.0,
            "geo": cutcell.build_cut_geometry(inp)}


def test_lists_too_long_for_the_small_shape(rn):
    """An unset handle takes a geometry whose lists fit its named shape (14x16)
    but not the 10x10 one its size would run: 72 members outside the 10x10
    tile at (10, 10), where a tile may list 64."""
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(configs.plain_small(96, 36)[0])
    Nx, Nr = s.Nx, s.Nr
    rows = np.arange(Nr + 1, dtype=np.float32)[:, None]
    gA, gG, gM = np.zeros((Nr + 1, Nx + 1, 4), np.float32), np.zeros((Nr, Nx, 4), np.float32), np.zeros((Nr, Nx, 4), np.float32)
    gA[..., 2], gA[..., 3] = rows + 0.5, rows
    gA[Nr, :, 2] = gA[:, Nx, 3] = 0
    gG[..., 0], gG[..., 1], gM[..., 3] = rows[:Nr] + 0.5, 1, 0.17
    groups = [((9, j), (10, j), (8, j)) for j in range(10, 20)] + [((20, j), (19, j), (21, j)) for j in range(10, 20)]
    groups += [((i, 9), (i, 10), (i, 8)) for i in range(11, 19)] + [((i, 20), (i, 19), (i, 21)) for i in range(11, 19)]
    bit = {(-1, 0): 1, (1, 0): 2, (0, -1): 4, (0, 1): 8}
    for (hi, hj), *slaves in groups:
        for i, j in slaves:
            gM[hj, hi, 2] += bit[i - hi, j - hj]
            gM[j, i, :2] = hi - i, hj - j
        cells = [(hi, hj)] + slaves
        total = sum(gG[j, i].copy() for i, j in cells)
        for i, j in cells:
            gG[j, i] = total
    assert longest_list(gM, Nx, Nr, 10, 10) > 64 >= longest_list(gM, Nx, Nr, 14, 16)
    geo = dict(s.geo, mask=np.zeros(Nx * Nr, np.uint8), geoA=gA.reshape(-1), geoG=gG.reshape(-1), geoM=gM.reshape(-1))
    init = s.initialState()
    outs = []
    for tile in (None, "14x16"):
        g = rn.GPUSolver(Nx, Nr)
        g.setPrecision("exact")
        if tile:
            g.setTile(tile)
        g.setGeometry(geo)
        g.setState(init["A"], init["B"])
        g.step(9, s.P)
        outs.append(g.readAll())
        g.setGeometry(s.geo)                     # and back to one that fits the small shape
        g.setState(init["A"], init["B"])
        g.step(9, s.P)
        outs.append(g.readAll())
        g.close()
    for a, b in zip(outs[:2], outs[2:]):
        assert np.array_equal(a["A"], b["A"]) and np.array_equal(a["B"], b["B"])


@pytest.mark.parametrize("build", [False, True])
def test_lists_too_long_for_16x16(rn, build):
    """An unset handle whose size runs 16x16 tiles takes a geometry whose lists
    fit 16x15 only, uploaded or built on the device."""
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(configs.plain_small(1024, 287)[0])
    c = blocks_setup(s.Nx, s.Nr, CHANNEL)
    assert longest_list(c["geo"]["geoM"], s.Nx, s.Nr, 16, 16) > 64 >= longest_list(c["geo"]["geoM"], s.Nx, s.Nr, 16, 15)
    init = s.initialState()
    outs = []
    for tile in (None, "16x15"):
        g = rn.GPUSolver(s.Nx, s.Nr)
        g.setPrecision("exact")
        if tile:
            g.setTile(tile)
        if build:
            g.buildGeometry(c)
        else:
            g.setGeometry(c["geo"])
        g.setState(init["A"], init["B"])
        g.step(5, s.P)
        outs.append(g.readAll())
        g.close()
    assert np.array_equal(outs[0]["A"], outs[1]["A"]) and np.array_equal(outs[0]["B"], outs[1]["B"])


def test_refused_built_geometry_leaves_the_handle_as_it_was(rn):
    """rn_build_geometry of a geometry that the set tile shape cannot hold fails
    and changes nothing: the planes read back as before, and the handle steps
    as one that was never asked (its classes, lists and planes go together)."""
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(configs.viscous_plume(96, 45)[0])
    c = blocks_setup(s.Nx, s.Nr, POCKET)
    assert longest_list(c["geo"]["geoM"], s.Nx, s.Nr, 32, 15) > 64
    init = s.initialState()
    outs = []
    for ask in (False, True):
        g = rn.GPUSolver(s.Nx, s.Nr)
        g.setPrecision("exact")
        g.setTile("32x15")
        g.setGeometry(s.geo)
        g.setState(init["A"], init["B"])
        g.step(3, s.P)
        if ask:
            before = g.readGeometry()
            with pytest.raises(rn.solver.RnError):
                g.buildGeometry(c)
            after = g.readGeometry()
            assert all(np.array_equal(before[k], after[k]) for k in before)
        g.step(5, s.P)
        outs.append(g.readAll())
        g.close()
    assert np.array_equal(outs[0]["A"], outs[1]["A"]) and np.array_equal(outs[0]["B"], outs[1]["B"])


def test_batch_shape_follows_its_members_geometry(rn):
    """A batch whose shape nobody set runs 16x16 tiles for these grids (2 waves
    of blocks against 3). A member's new geometry whose lists fit 16x15 only is
    taken all the same, uploaded or built, as is one set after leaving the batch
    under the name 16x15; every member steps as a handle of its own."""
    from rocket_nozzle_cfd_solver_b200 import configs
    ss = [rn.build_sim_setup(configs.plain_small(*sz)[0]) for sz in ((1024, 287), (128, 48))]
    big, small = ss
    c = blocks_setup(big.Nx, big.Nr, CHANNEL)

    def make(s, tile=None):
        g = rn.GPUSolver(s.Nx, s.Nr)
        g.setPrecision("exact")
        if tile:
            g.setTile(tile)
        init = s.initialState()
        g.setGeometry(s.geo)
        g.setState(init["A"], init["B"])
        return g

    def same(a, b):
        x, y = a.readAll(), b.readAll()
        return np.array_equal(x["A"], y["A"]) and np.array_equal(x["B"], y["B"])
    for build in (True, False):
        batch = rn.SolverBatch()
        members, alone = [make(s) for s in ss], [make(s, "16x15") for s in ss]
        take = (lambda g: g.buildGeometry(c)) if build else (lambda g: g.setGeometry(c["geo"]))
        for g, s in zip(members, ss):
            batch.add(g, s.P)
        batch.step(7)
        for g, s in zip(alone, ss):
            g.step(7, s.P)
        take(members[0])                         # in the batch
        take(alone[0])
        batch.step(7)
        for g, s in zip(alone, ss):
            g.step(7, s.P)
        assert all(same(g, h) for g, h in zip(members, alone))
        batch.close()
        for g in members + alone:
            g.close()
    batch = rn.SolverBatch()
    g, h = make(big), make(big, "16x15")
    batch.add(g, big.P)
    batch.step(3)
    batch.remove(g)
    h.step(3, big.P)
    assert g.tile == "16x15"
    g.step(2, big.P)
    h.step(2, big.P)
    g.buildGeometry(c)                           # after leaving
    h.buildGeometry(c)
    g.step(3, big.P)
    h.step(3, big.P)
    assert same(g, h)
    batch.close()
    g.close()
    h.close()


@pytest.mark.parametrize("kind", ["plain_small", "viscous_plume", "injector_spray"])
def test_a_members_bits_do_not_depend_on_its_companions(rn, kind):
    """A batch whose shape nobody set moves from 16x16 tiles (the first member
    alone) to 16x15 (with the second, which leaves no wave to save) between its
    steps. In fast precision too each member ends with the bits of a handle set
    to 16x15, values below the smallest normal float apart (flushed to zero or
    not, as an operation comes packed or alone)."""
    from rocket_nozzle_cfd_solver_b200 import configs
    ss = [rn.build_sim_setup(dict(getattr(configs, kind)(*sz)[0], startMode="burst"))
          for sz in ((1024, 287), (1024, 384))]

    def make(s, tile=None):
        g = rn.GPUSolver(s.Nx, s.Nr)
        if tile:
            g.setTile(tile)
        init = s.initialState()
        g.setGeometry(s.geo)
        g.setState(init["A"], init["B"])
        if s.injector is not None:
            rn.GPUSpray(g).resize()
            g.spray.setInjector(s.injector)
        return g

    batch = rn.SolverBatch()
    members, alone = [make(s) for s in ss], [make(s, "16x15") for s in ss]
    for k, s in enumerate(ss):
        batch.add(members[k], s.P)
        batch.step(15)
        for h, t in list(zip(alone, ss))[:k + 1]:
            h.step(15, t.P)
    for g, h in zip(members, alone):
        x, y = g.readAll(), h.readAll()
        for p in ("A", "B"):
            a, b = (np.where(np.abs(v[p]) < np.finfo(np.float32).tiny, 0, v[p]) for v in (x, y))
            assert np.array_equal(a, b), (p, np.abs(a - b).max(), (a != b).sum())
    batch.close()
    for g in members + alone:
        g.close()


def test_autotune_sets_the_shape_it_names(rn):
    """After rn_autotune on a small unset handle the kernels run the shape it
    returned: resized, the handle steps with the bits of one set to that name
    (fast precision, where an unset handle's of the larger grid are others)."""
    from rocket_nozzle_cfd_solver_b200 import configs
    small, s = (rn.build_sim_setup(configs.viscous_plume(*sz)[0]) for sz in ((128, 48), (1024, 287)))
    outs = []
    g = rn.GPUSolver(small.Nx, small.Nr)
    g.setGeometry(small.geo)
    init = small.initialState()
    g.setState(init["A"], init["B"])
    chosen = g.autotune(small.P, steps=120)
    assert g.tile == chosen
    g.resize(s.Nx, s.Nr)
    h = rn.GPUSolver(s.Nx, s.Nr)
    h.setTile(chosen)
    init = s.initialState()
    for q in (g, h):
        assert q.tile == chosen
        q.setGeometry(s.geo)
        q.setState(init["A"], init["B"])
        q.step(40, s.P)
        outs.append(q.readAll())
        q.close()
    assert np.array_equal(outs[0]["A"], outs[1]["A"]) and np.array_equal(outs[0]["B"], outs[1]["B"])


def test_unset_name_follows_a_resize(rn):
    """An unset handle is named by its present grid's size, a set one as set."""
    g = rn.GPUSolver(128, 48)
    for Nx, Nr in ((1024, 384), (128, 48), (2048, 512)):
        h = rn.GPUSolver(Nx, Nr)
        g.resize(Nx, Nr)
        assert g.tile == h.tile, (Nx, Nr)
        h.close()
    g.setTile("16x8")
    g.resize(128, 48)
    assert g.tile == "16x8"
    g.close()


@pytest.mark.parametrize("done", [0, 1, 2])
@pytest.mark.parametrize("batched", [False, True])
def test_autotune_leaves_the_turbulence_fields(rn, done, batched):
    """The fields formed from the last step's stage-1 state (turbulence and
    mixing rate) are the same before and after the trials of an autotuner, whose
    steps are odd in number, on a spray handle that has taken no, an odd and an
    even number of steps (the stage-1 slot alternates with the steps' parity)."""
    from rocket_nozzle_cfd_solver_b200 import configs, solver
    s = rn.build_sim_setup(dict(configs.injector_spray(192, 72)[0], startMode="burst"))
    init = s.initialState()
    g = rn.GPUSolver(s.Nx, s.Nr)
    g.setGeometry(s.geo)
    g.setState(init["A"], init["B"])
    rn.GPUSpray(g).resize()
    g.spray.setInjector(s.injector)
    if done:
        g.step(done, s.P)
    specs = [solver.derived_spec(s, f) for f in (9, 13)]
    before = [g.derived(sp, s.P).copy() for sp in specs]
    if batched:
        batch = rn.SolverBatch()
        batch.add(g, s.P)
        batch.autotune(steps=5)
    else:
        g.autotune(s.P, steps=5)
    after = [g.derived(sp, s.P) for sp in specs]
    assert all(np.array_equal(a, b) for a, b in zip(before, after))
    if batched:
        batch.close()
    g.close()


@pytest.mark.parametrize("kind,Nx,Nr", [("plain_small", 512, 192), ("plain_small", 640, 224), ("viscous_plume", 640, 224),
                                        ("plain_small", 1024, 287), ("viscous_plume", 1024, 287),
                                        ("plain_small", 4700, 64)])
def test_larger_default_shapes_match_set_shapes(rn, kind, Nx, Nr):
    """Unset handles beyond the 10x10 sizes, exact precision, against set 16x8
    tiles: 14x16 with two to three blocks an SM, inviscid (both stage kernels
    are dependent launches there); 16x16 by a wave saved (2 to 1, 3 to 2) and by
    tiles saved; and, at viscous 1024x287, 16x15 again for its long lists."""
    from rocket_nozzle_cfd_solver_b200 import configs
    s = rn.build_sim_setup(getattr(configs, kind)(Nx, Nr)[0])
    if (Nx, Nr) == (1024, 287):
        assert (longest_list(s.geo["geoM"], Nx, Nr, 16, 16) > 4) == (kind == "viscous_plume")
    calls = (1, 13, 4, 4, 15)
    a, b = run(rn, s, None, calls), run(rn, s, "16x8", calls)
    assert np.array_equal(a[0]["A"], b[0]["A"]) and np.array_equal(a[0]["B"], b[0]["B"])
    assert np.array_equal(a[1], b[1])
