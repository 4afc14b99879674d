"""Ragged sizes of the device kernels against the CPU oracle (1e-12 relative,
max-norm): particle counts around the edges of a thread's run, a warp and a
CTA, wall runs whose absorbed particles move to the end of the sorted order, and
periodic 1D grids with every kind of divisor."""
import numpy as np
import pytest

import apic
import pyoracle as po
from common import rel_max

pytestmark = pytest.mark.gpu
TOL = 1e-12
SPECIES = [(-1.0, 1.0, 0.05), (1.0, 50.0, 0.05)]


def _particles(n, dims, length, seed):
    rng = np.random.default_rng(seed)
    pos = np.zeros((3, n))
    for a in range(dims):
        pos[a] = rng.uniform(0.0, length[a], n)
    return pos, rng.standard_normal((3, n))


@pytest.mark.parametrize("dims,B", [(2, (0.0, 0.0, 0.0)), (2, (0.1, 0.2, 0.3)), (3, (0.1, 0.2, 0.3))])
@pytest.mark.parametrize("count", [1, 2, 3, 31, 33, 65, 511, 513, 1025])
def test_push_of_ragged_counts(dims, B, count):
    n, length = ((8, 4), (4.0, 2.0)) if dims == 2 else ((8, 4, 4), (4.0, 2.0, 3.0))
    dev = apic.SimulationND(apic.config_nd(dims=dims, n=n, length=length, dt=0.1, magnetic_field=B, sort_interval=2,
                                           species=[(q, m, w, count) for q, m, w in SPECIES]))
    ora = po.SimND(dims, n, length, 0.1, 1.0, B, SPECIES)
    for k in range(2):
        pos, v = _particles(count, dims, length, 10 * count + k)
        dev.load(k, pos, v)
        ora.load(k, pos, v, v)
    dev.initialize()
    ora.initialize()
    dev.step(5)
    ora.step(5)
    for k in range(2):
        for x, y in zip(dev.particles(k), ora.particles(k)):
            assert rel_max(x[:dims], y[:dims]) < TOL
    for x, y in zip(dev.fields(), ora.fields()):
        assert rel_max(x, y) < TOL


@pytest.mark.parametrize("count", [1, 2, 65, 513, 1025])
@pytest.mark.parametrize("sort", [1, 3, 1000])
def test_walls_of_ragged_counts(count, sort):
    """Positions, the dead flags and the loss counts in load order, however
    often the particles are sorted."""
    n, length, B = (8, 9), (4.0, 2.0), (0.0, 0.0, 0.2)
    wall, pot, pb = (0, 1), (0.0, 0.0, 0.0, 1.5), (0, 0, 1, 2)
    dev = apic.SimulationND(apic.config_nd(dims=2, n=n, length=length, dt=0.1, magnetic_field=B, sort_interval=sort,
                                           species=[(q, m, w, count) for q, m, w in SPECIES],
                                           walls=(wall, pot, [3 if b == 0 else b for b in pb])))
    ora = po.SimND(2, n, length, 0.1, 1.0, B, SPECIES)
    ora.set_walls(wall, pot, pb)
    for k in range(2):
        pos, v = _particles(count, 2, length, 10 * count + k)
        dev.load(k, pos, v)
        ora.load(k, pos, v, v)
    dev.initialize()
    ora.initialize()
    dev.step(6)
    ora.step(6)
    for k in range(2):
        alive, losses = ora.alive_losses(k)
        assert np.array_equal(dev.alive(k), alive)
        assert np.array_equal(dev.boundary_losses(k), np.asarray(losses)[:4])
        keep = np.asarray(alive) == 1
        if keep.any():
            for x, y in zip(dev.particles(k)[::2], ora.particles(k)[::2]):  # positions, v_half
                assert rel_max(x[:2][:, keep], y[:2][:, keep]) < TOL
    for x, y in zip(dev.fields(), ora.fields()):
        assert rel_max(x, y) < TOL


@pytest.mark.parametrize("B", [(0.0, 0.0, 0.0), (0.1, 0.2, 0.3), "profile"])
@pytest.mark.parametrize("n,walls", [((64, 32), None), ((64, 33), (0, 1)), ((33, 65), (1, 1)), ((32, 16, 8), None),
                                     ((17, 33, 9), (1, 1, 1))])
@pytest.mark.parametrize("count", [113_665, 113_920, 170_001])
def test_two_particles_a_thread_give_the_bits_of_one(n, walls, B, count):
    """A species of more particles than the one-a-thread push takes against the same particles
    as two species below that (the density is one sum of integers): counts that end inside a
    thread, a warp and a CTA, periodic and with absorbing and reflecting walls."""
    dims = len(n)
    length = (4.0, 2.0, 3.0)[:dims]
    rng = np.random.default_rng(count)
    pos, v = _particles(count, dims, length, count)
    profile = (0, [0.0, 1.0, 4.0], rng.standard_normal((3, 3))) if B == "profile" else None
    got = []
    for split in (1, 2):
        parts = np.array_split(np.arange(count), split)
        dev = apic.SimulationND(apic.config_nd(
            dims=dims, n=n, length=length, dt=0.05, magnetic_field=(0.0, 0.0, 0.0) if profile else B,
            magnetic_field_profile=profile, sort_interval=3, species=[(-1.0, 1.0, 2.0 ** -12, len(i)) for i in parts],
            walls=(walls, [0.0] * 4 if dims == 2 else None,
                   [(1 if k % 2 else 2) if walls[k // 2] else 3 for k in range(2 * dims)]) if walls else None))
        for k, i in enumerate(parts):
            dev.load(k, pos[:, i], v[:, i])
        dev.initialize()
        dev.step(8)
        out = [dev.particles(k) for k in range(split)]
        got.append([np.concatenate([o[c] for o in out], axis=1) for c in range(3)] + list(dev.fields()) +
                   ([np.concatenate([dev.alive(k) for k in range(split)])] if walls else []))
        dev.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("nx", [3, 4, 5, 12, 37, 64, 97, 100, 127, 255, 256, 1022, 1024, 1999, 2048])
def test_periodic_1d_solve(nx):
    """Two-step transforms (even and odd extents, squares, primes)."""
    rng = np.random.default_rng(nx)
    xs = [rng.uniform(0.0, 2.0, 3000), rng.uniform(0.0, 2.0, 3000)]
    args = (nx, 2.0, 1.3, 0.0, 0.0, [-1.0, 1.5], [0.1, 0.1], xs)
    rho, phi, E = apic.deposit_solve_gather_1d(apic.PERIODIC, *args)[:3]
    dx = 2.0 / nx
    want = np.zeros(nx)
    for q, x in zip((-0.1, 0.15), xs):
        g = x / dx
        i = np.floor(g).astype(int)
        f = g - i
        want += np.bincount(i % nx, q / dx * (1 - f), nx) + np.bincount((i + 1) % nx, q / dx * f, nx)
    assert rel_max(rho, want) < TOL
    hat = np.fft.fft(rho - rho.mean())
    k = 2 * np.pi * np.fft.fftfreq(nx, dx)
    k[0] = 1.0
    ph = hat / (1.3 * k * k)
    ek = -1j * k * ph
    ph[0] = ek[0] = 0.0
    assert rel_max(phi, np.fft.ifft(ph).real) < TOL
    assert rel_max(E, np.fft.ifft(ek).real) < TOL


@pytest.mark.parametrize("mcc", [False, True])
@pytest.mark.parametrize("count,leaving", [(1, 0.0), (1023, 0.3), (1025, 0.3), (4097, 0.9), (100_003, 0.6), (100_003, 0.98)])
def test_1d_heavy_wall_losses(mcc, count, leaving):
    """Survivors keep their order through tiles that lose some, most or nearly
    all of their particles (and so read their next tile from many short ranges)."""
    from apic import workloads as W
    from common import load_device, load_oracle, oracle_config
    wl = W.ccp_helium(particles_per_cell=1, cells=32, seed=2, table_rows=256)
    if not mcc:
        wl.models = []
    rng = np.random.default_rng(count)
    for s in wl.species:
        s.weight *= 1e-6
        s.capacity = 2 * count + 4096
        s.x = rng.uniform(0.0, wl.length, count)
        s.v, s.vy, s.vz = (s.thermal * rng.standard_normal(count) for _ in range(3))
        go = rng.random(count) < leaving  # these cross the gap in one of the first three steps
        s.v[go] = rng.choice([-1.0, 1.0], go.sum()) * wl.length / wl.dt / rng.integers(1, 4, go.sum())
        if mcc:  # fast enough to leave, slow enough for the models' frequency bound: move them to the walls instead
            s.v[go] = s.thermal * np.abs(rng.standard_normal(go.sum())) * -1.0
            s.x[go] = np.abs(s.v[go]) * wl.dt * rng.uniform(0.2, 2.5, go.sum())
    cfg, tabs = W.to_device_config(wl, seed=77)
    dev = apic.Simulation1D(cfg, tabs)
    load_device(dev, wl)
    dev.initialize()
    T = po.TableSet()
    ora = po.Sim1D(oracle_config(wl, T), 1, 77)
    load_oracle(ora, wl)
    ora.initialize()
    for steps in (1, 2, 3):
        dev.step(steps)
        ora.step(steps)
        for k in range(2):
            a, b = dev.particles(k), ora.particles(k)
            assert len(a["x"]) == len(b["x"])
            for c in ("x", "vh", "v", "vy", "vz"):
                assert rel_max(a[c], b[c]) < 1e-11
        for x, y in zip(dev.fields(), ora.fields()):
            assert rel_max(x, y) < 1e-11


@pytest.mark.parametrize("precision", [apic.FP64, apic.FP32_STORAGE])
@pytest.mark.parametrize("vdim", [1, 3])
@pytest.mark.parametrize("cells,count", [(40, 40_960), (40, 41_985), (1500, 66_000), (1500, 66_561), (3299, 70_001)])
def test_collision_passes_give_the_same_bits(cells, count, vdim, precision):
    """Around the tiles (81, or 129 of a wide mesh) from which a discharge takes the pass of
    small CTAs: the same run with the electric-work ledger, which always takes the other pass."""
    from apic import workloads as W
    from common import load_device
    wl = W.ccp_helium(particles_per_cell=1, cells=cells, seed=4, table_rows=256, te_ev=8.0, vdim=vdim)
    rng = np.random.default_rng(count)
    for s in wl.species:
        s.weight *= cells / count
        s.capacity = count + 20_000
        s.x = rng.uniform(0.0, wl.length, count)
        v = s.thermal * rng.standard_normal((3, count))
        s.v, s.vy, s.vz = v[0], *((v[1], v[2]) if vdim == 3 else (None, None))
    got = []
    for ledger in (False, True):
        cfg, tabs = W.to_device_config(wl, seed=21, precision=precision)
        dev = apic.Simulation1D(cfg, tabs)
        load_device(dev, wl)
        if ledger:
            dev.enable_power_transfer()
        dev.initialize()
        dev.step(7)
        t = dev.collision_totals()
        assert t.candidates > count // 20
        out = [np.array([t.candidates, t.null_collisions] + [c for m in t.channel_collisions for c in m])]
        for k in range(2):
            p, b = dev.particles(k), dev.boundary_losses(k)
            out += [np.array([b.absorbed_left, b.absorbed_right])] + [p[c] for c in ("x", "v", "vh", "vy", "vz")]
        got.append(out + list(dev.fields()))
        dev.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_reloads_across_the_collision_passes():
    """A run that is loaded again with many, few and many particles, with steps still under way,
    is each time the run of a new handle."""
    from apic import workloads as W
    from common import load_device
    wl = W.ccp_helium(particles_per_cell=1, cells=40, seed=4, table_rows=256, te_ev=8.0)
    for s in wl.species:
        s.capacity = 100_000
        s.weight *= 40 / 60_000  # the deck's density at the larger counts

    def load(count):
        rng = np.random.default_rng(count)
        for s in wl.species:
            s.x = rng.uniform(0.0, wl.length, count)
            s.v, s.vy, s.vz = s.thermal * rng.standard_normal((3, count))

    def state(dev):
        return [dev.particles(k)[c] for k in range(2) for c in ("x", "v", "vh", "vy", "vz")] + list(dev.fields())

    cfg, tabs = W.to_device_config(wl, seed=21)
    dev = apic.Simulation1D(cfg, tabs)
    for count in (60_000, 1500, 60_001):
        load(count)
        load_device(dev, wl)
        dev.initialize()
        dev.step(6)
        fresh = apic.Simulation1D(*W.to_device_config(wl, seed=21))
        load_device(fresh, wl)
        fresh.initialize()
        fresh.step(6)
        for a, b in zip(state(dev), state(fresh)):
            assert np.array_equal(a, b)
        dev.step(40)  # under way at the next load
        fresh.close()


@pytest.mark.parametrize("n,axis", [((4, 3), 0), ((3, 4), 1), ((8, 34), 0), ((35, 16), 1), ((1024, 40), 0),
                                    ((4, 4002), 0), ((4, 4003), 0), ((4100, 8), 1)])
def test_mixed_solve_sizes(n, axis):
    """Odd row counts (a pair with one row), one interior row, the longest
    column kept in shared memory and longer ones."""
    rng = np.random.default_rng(sum(n))
    rho = rng.standard_normal((n[1], n[0]))
    phi, E = apic.field_solve_mixed_2d(n, (2.0, 3.0), axis, 1.3, 0.7, -1.1, rho)
    pr, Er = po.solve_mixed_2d(rho, n, (2.0, 3.0), axis, 1.3, 0.7, -1.1)
    # the oracle's own column solve has a condition number of about (rows / pi)^2
    rows = n[1] if axis == 0 else n[0]
    tol = max(TOL, 2.2e-16 * (rows / np.pi) ** 2)
    assert rel_max(phi, pr) < tol
    assert rel_max(E, Er) < 10 * tol


@pytest.mark.parametrize("n", [(3, 3), (5, 3), (3, 513), (513, 9), (3, 5, 9), (17, 3, 3), (33, 65, 17), (129, 33), (9, 129, 65),
                               (129, 33, 65), (65, 129, 33), (33, 65, 129), (33, 33, 17)])
def test_dirichlet_solve_sizes(n):
    """The discrete equation at every interior node: eps Laplacian(phi) = -rho."""
    rng = np.random.default_rng(sum(n))
    dims = len(n)
    length = (2.0, 3.0, 1.5)[:dims]
    shape = tuple(reversed(n))
    rho = rng.standard_normal(shape)
    sides = (0.3, -0.2, 1.0, 0.5) if dims == 2 else None
    phi, E = apic.field_solve_dirichlet_nd(n, length, 1.3, rho, sides)
    p = phi.reshape(shape)
    lap, scale = 0.0, 0.0
    inner = tuple(slice(1, -1) for _ in range(dims))
    for a in range(dims):
        ax, h = dims - 1 - a, length[a] / (n[a] - 1)
        up = tuple(slice(2, None) if b == ax else slice(1, -1) for b in range(dims))
        dn = tuple(slice(0, -2) if b == ax else slice(1, -1) for b in range(dims))
        lap = lap + (p[up] - 2 * p[inner] + p[dn]) / h ** 2
        scale += 4.0 / h ** 2
        e = E[a].reshape(shape)
        assert rel_max(e[inner], -(p[up] - p[dn]) / (2 * h)) < TOL
    # the residual's rounding is that of the largest term of the Laplacian
    assert np.max(np.abs(1.3 * lap + rho[inner])) < 1e-13 * scale * 1.3 * np.max(np.abs(p))
    if dims == 2:
        assert np.all(p[1:-1, 0] == 0.3) and np.all(p[1:-1, -1] == -0.2)
        assert np.all(p[0, 1:-1] == 1.0) and np.all(p[-1, 1:-1] == 0.5)
        assert p[0, 0] == 0.65 and p[-1, -1] == 0.15
    else:
        assert np.all(p[0] == 0.0) and np.all(p[:, :, -1] == 0.0)


@pytest.mark.parametrize("n", [(64, 32), (1024, 1024), (64, 128, 128)])
def test_fields_read_back(n):
    """Small reads (one copy after another) and large ones (threads): every
    component in its place."""
    dims = len(n)
    length = tuple(float(k) for k in n)
    count = 20011
    dev = apic.SimulationND(apic.config_nd(dims=dims, n=n, length=length, dt=0.1,
                                           species=[(q, m, w, count) for q, m, w in SPECIES]))
    for k in range(2):
        pos, v = _particles(count, dims, length, 5 + k)
        dev.load(k, pos, v)
    dev.initialize()
    for _ in range(2):
        dev.step(1)
        rho, phi, E = dev.fields()
        p2, E2 = apic.field_solve_periodic_nd(dims, n, length, 1.0, rho)
        assert rel_max(phi, p2) < TOL
        assert rel_max(E, E2) < TOL


def test_fields_into_any_destination():
    """Large reads of some or all fields, into pageable and page-locked memory, before and after
    the run's first read of the field."""
    import torch
    n = (128, 128, 128)
    N = int(np.prod(n))
    dev = apic.SimulationND(apic.config_nd(dims=3, n=n, length=(1.0, 2.0, 3.0), dt=0.1,
                                           species=[(q, m, w, 5000) for q, m, w in SPECIES]))
    for k in range(2):
        dev.load(k, *_particles(5000, 3, (1.0, 2.0, 3.0), 5 + k))
    dev.initialize()
    L, sizes = apic._bind_nd(), (N, N, 3 * N)

    def read(which, locked):
        out = [torch.full((s,), np.nan, dtype=torch.float64, pin_memory=k in locked).numpy() if k in which else None
               for k, s in enumerate(sizes)]
        apic._check_nd(L.apic_simnd_read_fields(dev.h, *[apic.dptr(a) for a in out]), dev.h)
        return out

    first = [read((0, 1), ()), read((0, 1, 2), ())]
    want = [a.ravel() for a in dev.fields()]
    calls = first + [read(w, l) for w, l in (((0, 1), ()), ((0, 1, 2), ()), ((0, 1, 2), (0, 1, 2)), ((0, 2), (2,)),
                                               ((1, 2), (1,)), ((2,), ()), ((1,), (1,)))]
    for out in calls:
        for a, b in zip(out, want):
            assert a is None or np.array_equal(a, b)


@pytest.mark.parametrize("precision", [apic.FP64, apic.FP32])
@pytest.mark.parametrize("particles,steps_per_launch", [(1, 7), (1023, 1), (1025, 60), (2500, 129), (2500, 300)])
def test_fixed_swarm_alone_and_beside_a_branching_run(precision, particles, steps_per_launch):
    """Alone, a fixed population's steps run inside one kernel; beside a branching
    run, step by step.  Both give the same bits."""
    from apic import workloads as W
    spec = W.swarm_c5(particles=particles, steps=260, burn_in_steps=100, seed=7)
    branch = W.swarm_c5(particles=500, steps=260, burn_in_steps=100, seed=8, branching=True)
    _, gas, keep = W.to_device_swarm(spec, precision=precision)
    got = []
    for beside in (False, True):
        srv = apic.SwarmServer(gas, 64 << 20, max_runs=4, precision=precision, steps_per_launch=steps_per_launch)
        rid = srv.submit(W.swarm_request(spec, 300.0, seed=5))
        if beside:
            srv.submit(W.swarm_request(branch, 50.0, seed=6))
        r = None
        while r is None:
            srv.advance()
            r = srv.poll(rid)
        got.append([getattr(r, k) for k in ("status", "steps_done", "mean_velocity_x", "mean_energy_ev",
                                            "diffusion_longitudinal", "diffusion_transverse", "max_observed_energy_ev",
                                            "ionization_rate", "net_rate", "candidates", "null_collisions")]
                   + list(r.channel_collisions) + list(r.channel_rate) + list(r.channel_rate_se))
        srv.close()
    assert got[0][0] == 0 and got[0][1] == 260
    assert got[0] == got[1]


def _plasma3d_run(n, count, pos, v, split, B=(0.005, 0.1, 0.2), steps=1, sort=2, weight=0.01):
    """One electron species of at least 64 particles a cell (tiled push), or the same
    particles as `split` species of fewer each (few tiles: the untiled push)."""
    length = tuple(float(k) for k in n)
    parts = np.array_split(np.arange(count), split)
    dev = apic.SimulationND(apic.config_nd(dims=3, n=n, length=length, dt=0.2, magnetic_field=B, precision=apic.FP32,
                                           sort_interval=sort, species=[(-1.0, 1.0, weight, len(i)) for i in parts]))
    for k, i in enumerate(parts):
        dev.load(k, pos[:, i], v[:, i])
    dev.initialize()
    dev.step(steps)
    out = [dev.particles(k) for k in range(split)]
    return [np.concatenate([o[c] for o in out], axis=1) for c in range(3)], dev.fields()[0]


@pytest.mark.parametrize("steps", [1, 5])
@pytest.mark.parametrize("n,ppc,spread", [((8, 8, 8), 64.1, 1.0), ((16, 8, 32), 77.3, 1.0), ((32, 16, 8), 65.9, 4.0),
                                          ((8, 16, 8), 96.0, 30.0)])
def test_tiled_push_gives_the_untiled_bits(n, ppc, spread, steps):
    """Gather, push and deposit through a tile's shared memory against the kernels
    without it, from thermal particles to ones that cross several tiles a step."""
    rng = np.random.default_rng(int(10 * ppc))
    count = int(ppc * np.prod(n)) | 1
    pos = np.stack([rng.uniform(0.0, k, count) for k in n])
    v = spread * rng.standard_normal((3, count))
    # cells of volume 1 and a weight of 2^-7: a density is an integer times 2^-30, exact in
    # FP64 however many accumulators it is summed from, so both runs see the same field
    a, ra = _plasma3d_run(n, count, pos, v, 1, steps=steps, weight=2.0 ** -7)
    b, rb = _plasma3d_run(n, count, pos, v, 4, steps=steps, weight=2.0 ** -7)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert np.array_equal(ra, rb)


def test_tiled_push_with_crowded_nodes():
    """More weight on a node than one 32-bit word of a tile's box holds (and several work items
    of one tile): the charge stays exact."""
    n, count = (16, 8, 8), 70000
    rng = np.random.default_rng(3)
    pos = np.stack([rng.uniform(0.0, k, count) for k in n])
    crowd = rng.random(count) < 0.8
    pos[:, crowd] = np.array([[5.25], [3.5], [2.125]])
    (px, _, _), rho = _plasma3d_run(n, count, pos, np.zeros((3, count)), 1, steps=2, sort=1)
    i = np.floor(px).astype(int)
    f = px - i
    want = np.zeros(int(np.prod(n)))
    for c in range(8):
        o = np.array([[c & 1], [c >> 1 & 1], [c >> 2]])
        g = (i + o) % np.array(n)[:, None]
        w = np.prod(np.where(o == 1, f, 1.0 - f), axis=0)
        want += np.bincount((g[2] * n[1] + g[1]) * n[0] + g[0], -0.01 * w, want.size)
    # weights are multiples of 2^-23, offsets 24-bit floats
    assert rel_max(rho, want) < 1e-6


@pytest.mark.parametrize("n", [(128, 64), (64, 128), (32, 128), (512, 32), (16, 128), (64, 64, 64), (128, 32, 16), (32, 64, 128)])
def test_periodic_solve_of_every_line_length(n):
    """Register transforms of 32 to 256 points along contiguous and strided axes, mixed
    with the shared-memory tiles."""
    rng = np.random.default_rng(sum(n))
    dims = len(n)
    length = (2.0, 3.0, 1.5)[:dims]
    shape = tuple(reversed(n))
    rho = rng.standard_normal(shape)
    phi, E = apic.field_solve_periodic_nd(dims, n, length, 1.3, rho)
    hat = np.fft.fftn(rho)
    k = [2 * np.pi * np.fft.fftfreq(n[a], length[a] / n[a]).reshape([-1 if dims - 1 - b == a else 1 for b in range(dims)])
         for a in range(dims)]
    k2 = sum(q * q for q in k) * np.ones(shape)
    k2.flat[0] = 1.0
    ph = hat / (1.3 * k2)
    ph.flat[0] = 0.0
    assert rel_max(phi.reshape(shape), np.fft.ifftn(ph).real) < TOL
    for a in range(dims):
        assert rel_max(E[a].reshape(shape), np.fft.ifftn(-1j * k[a] * ph).real) < TOL


@pytest.mark.parametrize("dims", [2, 3])
def test_walls_until_most_particles_are_absorbed(dims):
    """The push skips the particles that a sort moved behind the living; counts, flags and
    positions stay those of runs that are never sorted; a second load starts over."""
    n, length = ((9, 17), (4.0, 2.0)) if dims == 2 else ((9, 9, 17), (4.0, 2.0, 3.0))
    wall, pb = (1,) * dims, (1,) * (2 * dims)
    sims = []
    for sort in (3, 10 ** 6):
        dev = apic.SimulationND(apic.config_nd(dims=dims, n=n, length=length, dt=0.1, magnetic_field=(0.0, 0.0, 0.2),
                                               sort_interval=sort, species=[(q, m, w, 3001) for q, m, w in SPECIES],
                                               walls=(wall, [0.0] * 4 if dims == 2 else None, pb)))
        sims.append(dev)
    for attempt in range(2):
        for dev in sims:
            for k in range(2):
                pos, v = _particles(3001, dims, length, 40 + k + 10 * attempt)
                dev.load(k, pos, v)
            dev.initialize()
        for steps in (4, 30, 40):
            for dev in sims:
                dev.step(steps)
            for k in range(2):
                assert np.array_equal(sims[0].alive(k), sims[1].alive(k))
                assert np.array_equal(sims[0].boundary_losses(k), sims[1].boundary_losses(k))
                for x, y in zip(sims[0].particles(k)[::2], sims[1].particles(k)[::2]):
                    assert np.array_equal(x, y)
            assert np.array_equal(sims[0].fields()[0], sims[1].fields()[0])
        assert sims[0].alive(0).mean() < 0.5


@pytest.mark.parametrize("dims", [2, 3])
def test_walls_loaded_on_the_device(dims):
    """A species loaded on the device between absorbing walls is alive, also when it replaces
    one that was sorted and absorbed: the same run as its read-back loaded from the host."""
    n, length = ((9, 17), (4.0, 2.0)) if dims == 2 else ((9, 9, 17), (4.0, 2.0, 3.0))
    count = 3001
    cfg = lambda: apic.config_nd(dims=dims, n=n, length=length, dt=0.1, sort_interval=3,
                                 species=[(q, m, w, count) for q, m, w in SPECIES],
                                 walls=((1,) * dims, [0.0] * 4 if dims == 2 else None, (1,) * (2 * dims)))
    dev = apic.SimulationND(cfg())
    before = np.zeros((2, 2 * dims), np.int64)
    for attempt in range(2):
        host = apic.SimulationND(cfg())
        for k in range(2):
            dev.load_maxwellian(k, count, 11 + k + 10 * attempt, 1.0)
            assert dev.alive(k).all()
            pos, v, vh = dev.particles(k)
            host.load(k, pos, v, vh)
        for sim in (dev, host):
            sim.initialize()
        for steps in (0, 1, 40):
            for sim in (dev, host):
                sim.step(steps)
            for k in range(2):
                assert np.array_equal(dev.alive(k), host.alive(k))
                assert np.array_equal(dev.boundary_losses(k).astype(np.int64) - before[k], host.boundary_losses(k))
                for x, y in zip(dev.particles(k)[::2], host.particles(k)[::2]):
                    assert np.array_equal(x, y)
            assert np.array_equal(dev.fields()[0], host.fields()[0])
        assert 0.0 < dev.alive(0).mean() < 0.7
        before = np.array([dev.boundary_losses(k) for k in range(2)], np.int64)


@pytest.mark.parametrize("ppc,sorts", [(255, 2), (256, 0)])
def test_crowded_walls_are_counted_as_they_run(ppc, sorts):
    """2D runs with walls of 256 particles a node and more are not sorted, and no sort is counted."""
    n = (8, 9)
    count = ppc * n[0] * n[1]
    dev = apic.SimulationND(apic.config_nd(dims=2, n=n, length=(4.0, 2.0), dt=1e-3, sort_interval=2,
                                           species=[(q, m, w, count) for q, m, w in SPECIES],
                                           walls=((0, 1), [0.0] * 4, (3, 3, 2, 2))))
    for k in range(2):
        dev.load_maxwellian(k, count, 3 + k, 1.0)
    dev.initialize()
    dev.step(4)
    # density, forward, sweep, inverse, field; a push per species; five launches per sorted species
    assert dev.launch_count() == 4 * (5 + 2) + sorts * 2 * 5


@pytest.mark.parametrize("n,wall", [((9, 8), (1, 0)), ((9, 17), (1, 1)), ((9, 9, 17), (1, 1, 1))])
def test_velocities_of_absorbed_particles(n, wall):
    """v is read in load order: an absorbed particle keeps the v of the last read before its loss
    and nobody else's, however often the run was sorted; kinetic energy and a second
    initialize() take the same v."""
    dims, count = len(n), 2001
    length = (4.0, 2.0, 3.0)[:dims]
    sims = [apic.SimulationND(apic.config_nd(
        dims=dims, n=n, length=length, dt=0.1, magnetic_field=(0.0, 0.1, 0.2), sort_interval=sort,
        species=[(q, m, w, count) for q, m, w in SPECIES],
        walls=(wall, [0.0] * 4 if dims == 2 else None, [1 if wall[k // 2] else 3 for k in range(2 * dims)])))
        for sort in (2, 10 ** 6)]
    for dev in sims:
        for k in range(2):
            dev.load(k, *_particles(count, dims, length, 60 + k))
        dev.initialize()
    last = [None, None]
    for steps in (1, 5, 5, -1, 7, 20):
        for dev in sims:
            dev.step(steps) if steps > 0 else dev.initialize()
        for k in range(2):
            a, b = (dev.particles(k) for dev in sims)
            for x, y in zip(a, b):
                assert np.array_equal(x, y)
            if last[k] is not None:
                dead = last[k][0] == 0
                assert np.array_equal(a[1][:, dead], last[k][1][:, dead])
            last[k] = sims[0].alive(k), a[1]
        assert 0 < (last[0][0] == 0).sum() < count
        e = [dev.sample() for dev in sims]
        for k in range(2):
            assert abs(e[0].kinetic_by_species[k] - e[1].kinetic_by_species[k]) < TOL * e[1].kinetic_by_species[k]


def _narrow_table(centre_ev, span, rows, seed):
    """Cross sections that jump between 0 and 1 from row to row of a narrow table."""
    from apic import workloads as W
    e = centre_ev * W.E_CHARGE * np.linspace(1.0, 1.0 + span, rows)
    sigma = 1e-20 * np.random.default_rng(seed).integers(0, 2, rows)
    density, vmax = 1e21, np.sqrt(2.0 * e[-1] / W.M_E)
    return e, sigma, density, 1.001 * density * 1e-20 * vmax


@pytest.mark.parametrize("centre_ev,span,rows", [(11.5, 4.3e-4, 256), (11.5, 4.3e-4, 8192), (1000.0, 0.01, 8192),
                                                 (11.5, 1e-6, 3), (1.0, 5.0, 64)])
def test_collisions_on_a_narrow_table(centre_ev, span, rows):
    """A resonance of a few meV: the bracket of every energy is the oracle's, however fine the
    rows are against the single-precision log of the bracket index."""
    from apic import workloads as W
    e, sigma, density, numax = _narrow_table(centre_ev, span, rows, 5)
    rng = np.random.default_rng(6)
    n, dt = 3000, 1.5 / numax
    speed = np.sqrt(2.0 * (e[0] + (e[-1] - e[0]) * rng.uniform(0.0, 1.0, n)) / W.M_E)
    v = rng.standard_normal((n, 3))
    v *= (speed / np.linalg.norm(v, axis=1))[:, None]
    tabs, keep = apic.Tables(), po.TableSet()
    model = apic.mcc_model(0, [tabs.channel(W.ELASTIC, e, sigma)], density, numax)
    got, stats = apic.collide3(model, W.M_E, v, dt, seed=(7 << 32) | 9, step=3, stream=0)
    col = (po.C.c_byte * 8192)()
    om = po.make_model(0, [keep.channel(W.ELASTIC, e, sigma)], density, numax)
    assert po.oracle().ora_collider_init(col, po.C.byref(om), W.M_E) == 0
    hits = 0
    for i in range(n):
        r, st = po.Rng(), po.CollideStats()
        r.kind, r.key[0], r.key[1] = 1, 9, 7
        r.ctr[0], r.ctr[1], r.ctr[2] = i, 3, 0
        w = np.ascontiguousarray(v[i])
        assert po.oracle().ora_collide3(col, po.dptr(w), dt, po.C.byref(r), po.C.byref(st)) == 0
        assert stats[i].candidates == st.candidates and stats[i].null_collisions == st.null_collisions
        assert stats[i].channel_collisions[0] == st.channel_collisions[0]
        assert rel_max(got[i], w) < TOL
        hits += st.channel_collisions[0]
    assert hits > n // 4


def test_fp32_collisions_on_a_narrow_table():
    """The FP32 form on 8192 rows within 1 %: no rate above the majorant (a wrong row
    extrapolates past it), and the accepted collisions of the table's mean."""
    from apic import workloads as W
    e, sigma, density, numax = _narrow_table(1000.0, 0.01, 8192, 5)
    rng = np.random.default_rng(6)
    n, p = 200_000, 0.1
    energy = e[0] + (e[-1] - e[0]) * rng.uniform(0.0, 1.0, n)
    v = rng.standard_normal((3, n))
    v *= np.sqrt(2.0 * energy / W.M_E) / np.linalg.norm(v, axis=0)
    tabs = apic.Tables()
    model = apic.mcc_model(0, [tabs.channel(W.ELASTIC, e, sigma)], density, numax)
    dev = apic.Simulation1D(apic.config1d(boundary=apic.DIRICHLET, velocity_dimensions=3, units=apic.SI, nx=65, length=1.0,
                                          dt=p / numax, species=[(-W.E_CHARGE, W.M_E, 1e-3, n)], models=[model],
                                          precision=apic.FP32), tabs)
    dev.load(0, rng.uniform(0.4, 0.6, n), v[0], None, v[1], v[2])
    dev.initialize()
    dev.step(1)
    dev.synchronize()
    t = dev.collision_totals()
    rate = p * np.interp(energy, e, sigma) * np.sqrt(2.0 * energy / W.M_E) * density / numax
    assert abs(t.candidates - n * p) < 5 * np.sqrt(n * p)
    assert abs(t.channel_collisions[0][0] - rate.sum()) < 5 * np.sqrt(rate.sum())
    dev.close()
