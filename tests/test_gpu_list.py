"""The particle-list timestep kernel at the sizes where it can go wrong:
region edges and ragged rows, tiles split because their particles do not fit
the list, more reaction candidates than its list holds, species ids past a
list entry's, and the species counts taken in it.  Everything is compared bit
for bit with the oracle."""
import numpy as np
import pytest

from lattice_microbes_b200 import configs
from tests.cases import oracle_tables
from tests.oracle_lib import oracle_counts, oracle_run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(gpu):
    from lattice_microbes_b200.solver import Context
    c = Context(0)
    yield c
    c.close()


def _run(ctx, spec, n, tile=(0, 0), lattice=None, records=1, tables=None):
    from lattice_microbes_b200 import _lib as L
    from lattice_microbes_b200.solver import Lattice, Model
    t = tables or oracle_tables(spec)
    src = spec.lattice if lattice is None else lattice
    model = Model.from_tables(ctx, t)
    lat = Lattice(ctx, spec.X, spec.Y, spec.Z, spec.slots, spec.bytes_per_slot)
    lat.set_schedule(L.LMB_SCHEDULE_FUSED, *tile)
    lat.set_native(src, spec.sites)
    step, rc, split = 0, 0, 0
    for _ in range(records):
        rc, st, counts = lat.run_counts(model, 11, step, n, spec.ns, check=False)
        step += n
        split += lat.tile_lists()[0]
        if rc:
            break
    out, _ = lat.get_native()
    ref, rc_ref, st_ref = oracle_run(t, src, spec.sites, 11, 0, n * records)
    assert rc == rc_ref
    assert np.array_equal(out, ref)
    if rc == 0:
        assert np.array_equal(counts, oracle_counts(t, ref))
    lat.close()
    model.close()
    return st_ref, split


VARIANTS = [(4, 1), (8, 1), (16, 1), (4, 4), (8, 4), (16, 4)]


@pytest.mark.parametrize("slots,bps", VARIANTS)
@pytest.mark.parametrize("shape,tile", [((1, 6, 4), (2, 2)), ((2, 3, 5), (3, 1)), ((3, 1, 8), (1, 4)),
                                        ((4, 4, 4), (4, 4)), ((12, 16, 1), (16, 1)), ((30, 6, 9), (3, 3)),
                                        ((36, 10, 6), (5, 2)), ((48, 16, 16), (16, 4)), ((64, 8, 12), (4, 6)),
                                        ((160, 6, 6), (2, 3))])
def test_regions_vs_oracle(ctx, shape, tile, slots, bps):
    spec = configs.random_problem(sum(shape) + slots, X=shape[0], Y=shape[1], Z=shape[2], slots=slots,
                                  bytes_per_slot=bps, density=0.15 * slots, zeroth=slots == 8)
    _run(ctx, spec, 5, tile, records=2)


@pytest.mark.parametrize("slots,bps", VARIANTS)
def test_crowded_corner_splits_its_tile(ctx, slots, bps):
    """Every particle of the lattice in one corner, sites full: the mean
    density sizes a list far too short for that corner's tile."""
    spec = configs.random_problem(5 + slots, X=64, Y=48, Z=32, slots=slots, bytes_per_slot=bps, density=0.02,
                                  zeroth=False)
    N = spec.X * spec.Y * spec.Z
    rng = np.random.default_rng(3)
    z, y, x = np.meshgrid(np.arange(10), np.arange(14), np.arange(64), indexing="ij")
    at = (x + y * spec.X + z * spec.X * spec.Y).reshape(-1)
    lat = np.zeros_like(spec.lattice)
    for k in range(slots - 1):  # one slot free: the first timesteps overflow only a little
        sp = rng.integers(1, spec.ns + 1, at.size).astype(np.uint32)
        here = rng.random(at.size) < (0.9 if k < slots // 2 else 0.35)
        if bps == 1:
            lat[(k // 4) * N + at[here]] |= sp[here] << np.uint32(8 * (k % 4))
        else:
            lat[k * N + at[here]] = sp[here]
    _, split = _run(ctx, spec, 3, lattice=lat, records=2)
    assert split > 0


@pytest.mark.parametrize("slots,bps", [(8, 1), (16, 4)])
def test_more_reaction_candidates_than_listed(ctx, slots, bps):
    """Rates so high that most occupied sites may react in a timestep."""
    spec = configs.random_problem(21, X=64, Y=16, Z=16, slots=slots, bytes_per_slot=bps, density=0.6, zeroth=False)
    spec.K = spec.K * 40.0
    # One timestep of two tiles, worked whole: one of them had more.
    st, split = _run(ctx, spec, 1, (16, 8))
    assert st.reactions > 2 * 512 and split == 0
    st, _ = _run(ctx, spec, 4, (16, 8))
    assert st.reactions > 4 * 512


@pytest.mark.parametrize("X,slots", [(32, 8), (128, 16)])
def test_species_past_a_list_entry(ctx, X, slots):
    """Species ids above 4095: the dense kernel, or the per-phase kernels
    where only the particle-list kernel could hold the tile."""
    spec = configs.random_problem(31, X=X, Y=8, Z=8, slots=slots, bytes_per_slot=4, ns=3, nst=2, nr=3, density=0.4,
                                  zeroth=False)
    # The three species renamed to ids up to 5000.
    ids = np.array([0, 17, 4097, 5000], dtype=np.uint32)
    big = configs.ModelSpec(**{**spec.__dict__, "ns": 5000,
                               "S": np.zeros((5000, spec.nr), np.int32), "D": np.zeros((5000, spec.nr), np.uint32),
                               "DF": np.zeros((2, 2, 5000)), "lattice": ids[spec.lattice]})
    for s in range(3):
        big.S[ids[s + 1] - 1], big.D[ids[s + 1] - 1] = spec.S[s], spec.D[s]
        big.DF[:, :, ids[s + 1] - 1] = spec.DF[:, :, s]
    _run(ctx, big, 3, (4, 4) if X == 128 else (2, 2))


@pytest.mark.parametrize("slots,bps,density", [(8, 1, 2.6), (8, 1, 4.2), (16, 1, 9.6), (4, 4, 1.7), (16, 4, 9.6)])
@pytest.mark.parametrize("schedule", ["fused", "phases"])
def test_many_overflows_in_a_timestep(ctx, slots, bps, density, schedule):
    """From tens to more overflows than a block has threads in one timestep,
    many of them into the same sites: the insertions made together equal the
    oracle's, made one after another."""
    from lattice_microbes_b200 import _lib as L
    from lattice_microbes_b200.solver import Lattice, Model
    spec = configs.random_problem(61, X=64, Y=16, Z=16, slots=slots, bytes_per_slot=bps, density=density, nst=2,
                                  zeroth=False)
    t = oracle_tables(spec)
    model = Model.from_tables(ctx, t)
    lat = Lattice(ctx, spec.X, spec.Y, spec.Z, slots, bps)
    lat.set_schedule(L.LMB_SCHEDULE_FUSED if schedule == "fused" else L.LMB_SCHEDULE_PHASES)
    lat.set_native(spec.lattice, spec.sites)
    rc, st = lat.run(model, 5, 0, 4, check=False)
    ref, rc_ref, st_ref = oracle_run(t, spec.lattice, spec.sites, 5, 0, 4)
    assert rc == rc_ref
    assert st_ref.overflows > 40
    assert st.overflows == st_ref.overflows
    out, _ = lat.get_native()
    assert np.array_equal(out, ref)
    lat.close()
    model.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("counted", [1, 3])
def test_counts_of_fewer_species_than_overflow(ctx, counted, mode):
    """Species totals asked for up to a species below those the overflow
    resolution puts back in the counted timestep."""
    from lattice_microbes_b200.solver import Lattice, Model
    spec = configs.random_problem(61, X=64, Y=16, Z=16, slots=8, bytes_per_slot=1, density=2.6, nst=2, zeroth=False)
    t = oracle_tables(spec)
    model = Model.from_tables(ctx, t)
    lat = Lattice(ctx, spec.X, spec.Y, spec.Z, 8, 1)
    lat.set_native(spec.lattice, spec.sites)
    ref, rc_ref, st_ref = oracle_run(t, spec.lattice, spec.sites, 5, 0, 1, mode)
    assert rc_ref == 0 and st_ref.overflows > 40
    rc, st, counts = lat.run_counts(model, 5, 0, 1, counted, mode)
    assert st.overflows == st_ref.overflows
    assert np.array_equal(counts, oracle_counts(t, ref)[: counted + 1])
    lat.close()
    model.close()


@pytest.mark.parametrize("slots,bps", [(8, 1), (16, 4)])
def test_zeroth_order_rate_switched_on_between_runs(ctx, slots, bps):
    """A source whose rate is 0 for 64 timesteps (a captured graph) and
    positive for the next 64: empty sites produce from then on, however the
    run is cut."""
    from lattice_microbes_b200.solver import Lattice, Model
    spec = configs.random_problem(71, X=32, Y=16, Z=16, slots=slots, bytes_per_slot=bps, density=0.01)
    src = [j for j in range(spec.nr) if spec.rtype[j] == configs.ZEROTH]
    spec.RL[src] = 1
    on = spec.K.copy()
    on[src] *= 0.1
    spec.K[src] = 0.0
    off = oracle_tables(spec)
    spec.K = on
    lit = oracle_tables(spec)
    assert not off.qp0.any() and lit.qp0.all()
    mid, rc, _ = oracle_run(off, spec.lattice, spec.sites, 13, 0, 64)
    ref, rc2, st_ref = oracle_run(lit, mid, spec.sites, 13, 64, 64)
    assert rc == rc2 == 0 and st_ref.reactions > 1000
    for piece in (64, 16):
        spec.K = on.copy()
        spec.K[src] = 0.0
        model = Model.from_spec(ctx, spec)
        lat = Lattice(ctx, spec.X, spec.Y, spec.Z, slots, bps)
        lat.set_native(spec.lattice, spec.sites)
        for t in range(0, 128, piece):
            if t == 64:
                for j in src:
                    model.set_reaction_rate(j, float(on[j]))
            lat.run(model, 13, t, piece)
        out, _ = lat.get_native()
        assert np.array_equal(out, ref), piece
        lat.close()
        model.close()


def _tiles(lat):
    _, Ty, Tz = lat.schedule()
    return (lat.Y // Ty) * (lat.Z // Tz)


def test_lists_follow_a_lattice_that_fills_up(ctx):
    """An empty lattice with sources: its tiles start with the shortest
    lists and are split as it fills, and the lists are sized anew from what
    the split tiles held, not from the count of 0."""
    from lattice_microbes_b200.solver import Lattice, Model
    spec = configs.random_problem(81, X=64, Y=32, Z=32, density=0.0)
    spec.K = np.where(spec.rtype == configs.ZEROTH, 0.004 * spec.nsites, 0.0)
    spec.RL[:] = 1
    t = oracle_tables(spec)
    model = Model.from_tables(ctx, t)
    lat = Lattice(ctx, spec.X, spec.Y, spec.Z, 8, 1)
    lat.set_native(spec.lattice, spec.sites)
    seen = []
    for k in range(10):
        assert lat.run(model, 3, 16 * k, 16)[0] == 0
        seen.append(lat.tile_lists())
    ref, rc, _ = oracle_run(t, spec.lattice, spec.sites, 3, 0, 160)
    assert rc == 0
    assert np.array_equal(lat.get_native()[0], ref)
    density = np.count_nonzero(ref.view(np.uint8)) / spec.nsites
    assert max(s for s, _ in seen) > 0, seen
    assert seen[-1][0] * 8 <= 16 * _tiles(lat), seen
    assert density / 2 < seen[-1][1] <= 8, (density, seen)
    lat.close()
    model.close()


@pytest.mark.parametrize("slots,bps", [(8, 1), (16, 4)])
@pytest.mark.parametrize("tile", [None, (0, 0), (8, 8)])
def test_lists_of_a_crowded_corner_stay_bounded(ctx, slots, bps, tile):
    """Full sites in one corner, in the lattice's own schedule and plan, in the
    fused schedule's own plan and in a tile that cannot hold them: the figure
    the lists are sized for is a measured one, however many runs split tiles,
    and an autotuner's trials leave none that is not."""
    from lattice_microbes_b200 import _lib as L
    from lattice_microbes_b200.solver import Lattice, Model
    spec = configs.random_problem(82, X=64, Y=64, Z=64, slots=slots, bytes_per_slot=bps, density=0.0, nr=0, nst=1,
                                  qmax=0.002)
    N = spec.nsites
    rng = np.random.default_rng(4)
    z, y, x = np.meshgrid(np.arange(6), np.arange(24), np.arange(64), indexing="ij")
    at = (x + y * spec.X + z * spec.X * spec.Y).reshape(-1)
    lattice = np.zeros_like(spec.lattice)
    for k in range(slots - 2):
        sp = rng.integers(1, spec.ns + 1, at.size).astype(np.uint32)
        if bps == 1:
            lattice[(k // 4) * N + at] |= sp << np.uint32(8 * (k % 4))
        else:
            lattice[k * N + at] = sp
    t = oracle_tables(spec)
    model = Model.from_tables(ctx, t)
    lat = Lattice(ctx, spec.X, spec.Y, spec.Z, slots, bps)
    if tile:
        lat.set_schedule(L.LMB_SCHEDULE_FUSED, *tile)
    lat.set_native(lattice, spec.sites)
    seen = []
    for k in range(12):
        assert lat.run(model, 3, 2 * k, 2)[0] == 0
        seen.append(lat.tile_lists())
    ref, rc, _ = oracle_run(t, lattice, spec.sites, 3, 0, 24)
    assert rc == 0
    assert np.array_equal(lat.get_native()[0], ref)
    assert max(s for s, _ in seen) > 0, seen
    assert all(d <= slots for _, d in seen), seen
    if tile != (8, 8):
        assert seen[-1][0] == 0, seen
    # Crowded contents of an IntLattice go to the per-phase kernels when the
    # schedule is the lattice's own; even contents come back to the tiles.
    _, _, launches = lat.run_profiled(model, 3, 24, 2)
    assert (launches[5] == 0) == (tile is None and bps == 4)
    even = np.zeros_like(lattice)
    even[::37] = 1
    lat.set_native(even, spec.sites)
    assert lat.run_profiled(model, 3, 26, 2)[2][5] == 2
    assert np.array_equal(lat.get_native()[0], oracle_run(t, even, spec.sites, 3, 26, 2)[0])
    lat.set_native(lattice, spec.sites)
    lat.autotune(model, 3, 24, 4)
    lat.set_schedule(L.LMB_SCHEDULE_FUSED)
    assert lat.tile_lists()[1] <= slots
    lat.close()
    model.close()
