"""The C ABI library loads and exports every entry point include/*.h declares;
host-side behaviour that needs no GPU."""
import ctypes as C
import os
import re

import numpy as np
import pytest

import apic
from apic import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    names = set()
    inc = os.path.join(ROOT, "include")
    for fn in os.listdir(inc):
        if fn.endswith(".h"):
            text = open(os.path.join(inc, fn)).read()
            names |= set(re.findall(r"APIC_EXPORT\s+[\w\s\*]+?\b(apic_\w+)\s*\(", text))
    return sorted(names)


def test_library_exports_every_declared_symbol():
    lib = apic.lib()
    names = declared_symbols()
    assert len(names) >= 20
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, missing


def test_overlapping_1d_kernels_load_coherently():
    """The kernels of a 1D step are resident while the one before them still writes
    (programmatic launches), so the sources that hold them use no non-coherent load:
    none by intrinsic or PTX, and no kernel of a step has a const __restrict__ argument."""
    for name in ("pic1d.cu", "pic1d_c32.cuh"):
        text = open(os.path.join(ROOT, "aurora-pic_b200", "csrc", name)).read()
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)
        assert "grid_wait" in code
        assert not re.findall(r"__ldg|ld\.global\.nc", code), name
        for args in re.findall(r"__global__[^(]*(?:__launch_bounds__\([^{;]*?\)\s*)?k_\w+\(([^)]*)\)", code):
            assert not (args.startswith("Params1D") and "__restrict__" in args), args


def test_status_strings_and_version():
    lib = apic.lib()
    assert b"sm_100a" in lib.apic_version()
    for code in range(11):
        assert lib.apic_status_string(code)


@pytest.mark.skipif(apic.lib().apic_device_count() > 0, reason="checks the no-device path")
def test_create_without_device_fails_loudly():
    wl = W.two_stream(particles_per_beam=64, nx=16)
    cfg, tabs = W.to_device_config(wl)
    with pytest.raises(apic.ApicError) as e:
        apic.Simulation1D(cfg, tabs)
    assert e.value.status == 10  # APIC_ERR_NO_DEVICE, never a CPU fallback


def test_workload_shapes():
    wl = W.ccp_helium()
    assert wl.nx == 513 and len(wl.species) == 2
    assert all(len(s.x) == 262144 for s in wl.species)
    assert abs(wl.dt - 1.0 / (400 * 13.56e6)) < 1e-24
    # max_frequency * dt stays well below 1 (the reference requires <= 0.1 for swarms)
    for m in wl.models:
        assert m.max_frequency * wl.dt < 0.1
    ts = W.two_stream()
    assert ts.nx == 256 and sum(len(s.x) for s in ts.species) == 32768
    assert np.all((ts.species[0].x >= 0) & (ts.species[0].x < ts.length))


def test_ctypes_structs_match_the_c_header(tmp_path):
    """Every struct the Python binding passes across the ABI has the C size."""
    names = {"apic_mcc_channel": apic.McChannel, "apic_mcc_model": apic.MccModel, "apic_config1d": apic.Config1D,
             "apic_config_nd": apic.ConfigND, "apic_sample_nd": apic.SampleND,
             "apic_swarm_config": apic.SwarmConfig, "apic_swarm_result": apic.SwarmResult,
             "apic_swarm_request": apic.SwarmRequest, "apic_swarm_server_config": apic.SwarmServerConfig}
    src = tmp_path / "sizes.c"
    body = "".join(f'    printf("{n} %zu\\n", sizeof({n}));\n' for n in names)
    src.write_text('#include <stdio.h>\n#include "aurorapic_b200.h"\nint main(void) {\n' + body + "    return 0;\n}\n")
    exe = tmp_path / "sizes"
    import subprocess
    subprocess.run(["gcc", "-I", os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    got = dict(zip(out[0::2], map(int, out[1::2])))
    for n, cls in names.items():
        assert got[n] == C.sizeof(cls), (n, got[n], C.sizeof(cls))


def test_swarm_request_validation_on_cpu():
    """Server creation needs a device; its absence is reported, never hidden."""
    spec = W.swarm_c5(particles=1000, steps=100, burn_in_steps=50)
    cfg, gas, tabs = W.to_device_swarm(spec)
    if apic.lib().apic_device_count() > 0:
        pytest.skip("checks the no-device path")
    with pytest.raises(apic.ApicError):
        apic.swarm_run(cfg, gas, [10.0])


def build_facade_check(tmp_path):
    import subprocess
    exe = tmp_path / "facade_check"
    subprocess.run(["g++", "-std=c++20", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "facade_check.cpp"), "-L", os.path.dirname(apic.library_path()),
                    "-laurorapic_b200", "-Wl,-rpath," + os.path.dirname(apic.library_path()), "-o", str(exe)],
                   check=True)
    return exe


def test_cpp20_facade_compiles_and_maps_errors(tmp_path):
    """The C++20 facade (include/aurorapic_b200.hpp) builds against the
    library; without a device, creation raises runtime_error and a bad
    configuration keeps the reference's invalid_argument."""
    import subprocess
    if apic.lib().apic_device_count() > 0:
        pytest.skip("checks the no-device path")
    out = subprocess.run([str(build_facade_check(tmp_path))], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "invalid_argument: simulation dt must be positive and finite" in out.stdout


@pytest.mark.parametrize("walls,msg", [
    (((1, 1, 0), None, (0,) * 6), "3D meshes are periodic or Dirichlet on every axis"),
    (((1, 1, 1), (0.0, 1.0, 0.0, 0.0), (0,) * 6), "3D Dirichlet walls are grounded"),
    (((1, 1, 1), None, (0, 0, 0, 0, 0, 7)), "unknown particle boundary"),
])
def test_3d_wall_configuration_checks(walls, msg):
    """A 3D mesh is periodic or Dirichlet as a whole, with grounded walls
    (Simulation3DConfig's single field boundary, src/Mesh3D.cpp:37-48,
    src/FieldSolver.cpp:351-372); create rejects anything else before it looks
    for a device."""
    cfg = apic.config_nd(dims=3, n=(9, 9, 9), length=(1.0, 1.0, 1.0), dt=0.1,
                         species=[(-1.0, 1.0, 1.0, 16)], walls=walls)
    with pytest.raises(apic.ApicError) as e:
        apic.SimulationND(cfg)
    assert msg in str(e.value)


@pytest.mark.parametrize("bgk,models,msg", [
    ((-1.0, 1.0), False, "collision frequency must be non-negative and finite"),
    ((float("nan"), 1.0), False, "collision frequency must be non-negative and finite"),
    ((1.0, -2.0), False, "neutral_temperature_velocity must be non-negative and finite"),
    ((1.0e8, 1.0e5), True, "named collision models cannot be combined with the legacy collision model"),
])
def test_bgk_configuration_checks(bgk, models, msg):
    """The legacy BGK model's checks (src/Simulation.cpp:95-100, :388-392) run
    in create before it looks for a device."""
    from apic import workloads as W
    wl = W.ccp_helium(particles_per_cell=2, cells=8, seed=1, steps=1, table_rows=16, bgk=bgk)
    if models:
        wl.models = W.ccp_helium(particles_per_cell=2, cells=8, seed=1, steps=1, table_rows=16).models
    cfg, tabs = W.to_device_config(wl)
    with pytest.raises(apic.ApicError) as e:
        apic.Simulation1D(cfg, tabs)
    assert msg in str(e.value)


CELLS_CHECK = r"""
#include <cstdio>
#include <random>
#include "apic_common.cuh"
int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    long long bad = 0, n = 0;
    auto check = [&](double x, double d, double rd) {
        ++n;
        if (!(x >= 0.0)) return;
        const double q = apic::cells_of(x, d, rd), want = x / d;
        // below 2^-960 the remainder leaves the normal range: the cell is the same
        const bool same = x < 0x1p-960 ? std::floor(q) == std::floor(want) && std::fabs(q - want) <= 0x1p-900 : q == want;
        if (!same && bad++ < 5) std::printf("%a / %a\\n", x, d);
    };
    for (int c = 0; c < 4000; ++c) {
        const int cells = 2 + (int)(rng() % 4096);
        // lengths of every size, some of them exact multiples of the cells
        const double L = c % 3 == 0 ? cells * std::ldexp(1.0, (int)(rng() % 60) - 50) : std::exp2(60.0 * u(rng) - 50.0);
        const double d = L / cells, rd = apic::reciprocal_spacing(d);
        for (int k = 0; k < 400; ++k) {
            const int i = (int)(rng() % (unsigned)(cells + 1));
            double edge[2] = {i * d, L * ((double)i / cells)};
            for (double e : edge) {
                check(e, d, rd);
                double lo = e, hi = e;
                for (int s = 0; s < 3; ++s) {
                    check(lo = std::nextafter(lo, 0.0), d, rd);
                    check(hi = std::nextafter(hi, 2.0 * L), d, rd);
                }
            }
            check(L * u(rng), d, rd);
        }
    }
    for (double d : {1e-300, 1e300, 1e-310}) check(0.7 * d, d, apic::reciprocal_spacing(d));
    std::printf("%lld of %lld quotients differ\\n", bad, n);
    return bad != 0;
}
"""


def test_cell_quotients_are_the_division(tmp_path):
    """cells_of (a product and a correction in place of the division) gives the bits of x / d at
    the multiples of the spacing, next to them and anywhere in the domain: cell indices and
    fractions are the reference's (the fraction of a position below 2^-960 within 2^-900)."""
    import shutil
    import subprocess
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc on this host")
    src, exe = tmp_path / "cells.cu", tmp_path / "cells"
    src.write_text(CELLS_CHECK)
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "aurora-pic_b200", "csrc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
