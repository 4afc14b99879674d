"""Failure detection of the 1D step, injected from the host: inputs that make
the reference throw (src/Collision.cpp:620-623, :680-684, :910-916, :938-943,
src/Simulation.cpp:941-964) set the device error word, which the next
synchronising call returns as the matching status with the reference's
message.  Nothing here traps, faults or spins on the device: the kernels flag
and drop the offending particle or product, and the host's wait on the
stream is bounded."""
import numpy as np
import pytest

import apic
from apic import workloads as W
from common import load_device

pytestmark = pytest.mark.gpu

ERR_CAPACITY, ERR_MAJORANT, ERR_CANDIDATES, ERR_NONFINITE, ERR_TIMEOUT = 3, 4, 5, 6, 7


def _deck(te_ev=1.0):
    return W.ccp_helium(particles_per_cell=32, cells=64, seed=11, table_rows=1024, te_ev=te_ev)


def _run(wl, steps, precision=apic.FP64):
    cfg, tabs = W.to_device_config(wl, seed=99, precision=precision)
    dev = apic.Simulation1D(cfg, tabs)
    load_device(dev, wl)
    dev.initialize()
    dev.step(steps)
    with pytest.raises(apic.ApicError) as e:
        dev.synchronize()
    return dev, e.value


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_max_frequency_below_the_rate_bound(precision):
    wl = _deck(te_ev=20.0)
    wl.models[0].max_frequency *= 0.02  # far below the electrons' total collision rate
    dev, err = _run(wl, 3, apic.FP64 if precision == "fp64" else apic.FP32)
    assert err.status == ERR_MAJORANT, err
    assert "exceeds configured max_frequency" in str(err)
    dev.close()


def test_candidate_limit():
    wl = _deck()
    m = wl.models[1]  # ions in a gas 200x denser: many candidates per particle per step
    m.neutral_density *= 200.0
    m.max_frequency *= 200.0
    m.max_candidates = 1
    dev, err = _run(wl, 2)
    assert err.status == ERR_CANDIDATES, err
    assert "candidate limit" in str(err)
    dev.close()


def test_capacity_too_small_for_ionization_products():
    wl = _deck(te_ev=40.0)
    for s in wl.species:
        s.capacity = len(s.x)  # no room for a single product
    dev, err = _run(wl, 20)
    assert err.status == ERR_CAPACITY, err
    assert "max_particles_per_species" in str(err)
    dev.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_non_finite_velocity_loaded_from_the_host(precision):
    wl = _deck()
    wl.species[0].v[17] = np.nan
    dev, err = _run(wl, 2, apic.FP64 if precision == "fp64" else apic.FP32)
    assert err.status == ERR_NONFINITE, err
    assert "non-finite" in str(err)
    dev.close()


@pytest.mark.parametrize("what", ["position", "velocity"])
@pytest.mark.parametrize("n,wall", [((9, 8), (1, 0)), ((8, 9), (0, 1)), ((9, 17), (1, 1)), ((5, 9, 17), (1, 1, 1))])
def test_non_finite_coordinate_between_walls(n, wall, what):
    """A NaN on a wall axis (reflecting on both sides, so that nothing absorbs it)
    counts at the lower wall: every index stays inside the mesh, the charge stays whole
    and the other particles stay finite, sorted every step."""
    dims, count = len(n), 700
    length = (4.0, 2.0, 3.0)[:dims]
    axis = wall.index(1)
    rng = np.random.default_rng(5)
    dev = apic.SimulationND(apic.config_nd(
        dims=dims, n=n, length=length, dt=0.1, sort_interval=1, species=[(-1.0, 1.0, 0.05, count)],
        walls=(wall, [0.0] * 4 if dims == 2 else None, [2 if wall[k // 2] else 3 for k in range(2 * dims)])))
    pos = np.stack([rng.uniform(0.0, L, count) for L in length])
    v = rng.standard_normal((3, count))
    (pos if what == "position" else v)[axis, 17] = np.nan
    dev.load(0, pos, v)
    dev.initialize()
    # node volumes: half cells at the walls
    volume = np.ones(())
    for a in range(dims):
        w = np.full(n[a], length[a] / (n[a] - wall[a]))
        if wall[a]:
            w[[0, -1]] *= 0.5
        volume = np.multiply.outer(w, volume)
    for _ in range(4):
        charge = np.sum(dev.fields()[0] * volume.ravel())
        assert abs(charge + 0.05 * count) < 1e-9 * 0.05 * count
        dev.step(1)
    x, _, vh = dev.particles(0)
    others = np.arange(count) != 17
    assert np.isfinite(x[:dims, others]).all() and np.isfinite(vh[:, others]).all()
    assert np.isnan(x[axis, 17])
    dev.close()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("n,items", [((16, 32), 1), ((16, 32), 2), ((16, 32), 4), ((8, 8, 4), 1), ((8, 8, 4), 2),
                                     ((8, 8, 4), 4), ((8, 16, 8), 0)])
def test_non_finite_particle_of_the_fp32_form(n, items, bad):
    """A particle of non-finite velocity deposits nothing from its first step on, in every
    kernel of the FP32 push (the last mesh goes through its tiles); the others go on."""
    dims, count = len(n), (8 if items else 64) * int(np.prod(n)) + 1
    rng = np.random.default_rng(3)
    dev = apic.SimulationND(apic.config_nd(
        dims=dims, n=n, length=[float(k) for k in n], dt=0.1, magnetic_field=(0.1, 0.0, 0.2), precision=apic.FP32,
        sort_interval=2, push_items=items, species=[(-1.0, 1.0, 0.01, count)]))
    pos = np.stack([rng.uniform(0.0, k, count) for k in n])
    v = rng.standard_normal((3, count))
    v[0, 100] = bad
    dev.load(0, pos, v)
    dev.initialize()
    for _ in range(4):
        dev.step(1)
        charge = dev.fields()[0].sum() / -0.01  # in particles; 2^dims weights of 2^-23 units each
        assert abs(charge - (count - 1)) < count * 2 ** dims * 2.0 ** -22
    x, _, vh = dev.particles(0)
    others = np.arange(count) != 100
    assert np.isfinite(x[:dims, others]).all() and np.isfinite(vh[:, others]).all()
    dev.close()


@pytest.mark.parametrize("precision", [apic.FP64, apic.FP32])
@pytest.mark.parametrize("dims,axis", [(2, 0), (2, 1), (3, 2)])
def test_positions_outside_the_table_of_a_field_profile(dims, axis, precision):
    """B tabulated along an axis, particles loaded outside the domain: the table's end brackets
    (a uniform B here) hold there, and a NaN position (FP32: it deposits nothing) reads none
    past them."""
    n, length, B, count = (8, 16, 8)[:dims], (4.0, 2.0, 3.0)[:dims], (0.1, 0.2, 0.3), 900
    rng = np.random.default_rng(8)
    pos = np.stack([rng.uniform(-0.9 * L, 1.9 * L, count) for L in length])
    v = rng.standard_normal((3, count))
    if precision == apic.FP32:
        pos[axis, 17] = np.nan
    got = []
    for profile in (None, (axis, [0.0, 0.4, length[axis]], [B] * 3)):
        dev = apic.SimulationND(apic.config_nd(
            dims=dims, n=n, length=length, dt=0.05, precision=precision, species=[(-1.0, 1.0, 0.01, count)],
            magnetic_field=(0.0, 0.0, 0.0) if profile else B, magnetic_field_profile=profile))
        dev.load(0, pos, v)
        dev.initialize()
        dev.step(3)
        got.append([a[:, np.arange(count) != 17] for a in dev.particles(0)])
        dev.close()
    for a, b in zip(*got):
        assert np.isfinite(b).all()
        assert np.max(np.abs(a - b)) < (1e-12 if precision == apic.FP64 else 1e-6) * np.max(np.abs(a))


def test_bounded_wait_gives_up_and_a_later_wait_completes():
    """A wait limit far below the time of the enqueued steps ends the
    synchronising call with APIC_ERR_TIMEOUT; the work itself runs on, and a
    synchronise with a normal limit then succeeds with the run intact."""
    wl = W.ccp_helium(particles_per_cell=256, cells=256, seed=5, table_rows=1024)
    cfg, tabs = W.to_device_config(wl, seed=3)
    dev = apic.Simulation1D(cfg, tabs)
    load_device(dev, wl)
    dev.initialize()
    dev.synchronize()
    dev.set_wait_limit(1e-5)
    dev.step(400)
    with pytest.raises(apic.ApicError) as e:
        dev.synchronize()
    assert e.value.status == ERR_TIMEOUT
    dev.set_wait_limit(120.0)
    dev.synchronize()
    assert dev.sample().step == 400
    dev.close()
