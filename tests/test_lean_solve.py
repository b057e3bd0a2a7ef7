"""The engine's lean implicit solve, W inversion and torus functions
(koral-zig_b200/csrc/kc_implicit_lean.cuh, kc_u2p_lean.cuh, kc_init_lean.cuh)
against the plain restatement of the reference (include/koral), and its parallel
ordered fold (kc_fold.cuh) against the serial sum, bit for bit, on the host: the same source as the kernels, compiled by g++ with lean_check.cpp."""
import os
import subprocess

import numpy as np
import pytest

from tests.kgold import load_kgld

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lean_binary(tmp_path_factory):
    exe = tmp_path_factory.mktemp("lean") / "lean_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wno-unknown-pragmas", "-o", str(exe),
                    os.path.join(HERE, "lean_check.cpp")], check=True)
    return str(exe)


@pytest.fixture(scope="module")
def cells(tmp_path_factory):
    """The reference's 336 implicit records, and copies with the density, the
    energies, the fields and the step moved over decades; some field-free, at
    rest, or with a broken state."""
    rec = load_kgld("rad/rad_implicit")[0][:, :37]
    rng = np.random.default_rng(7)
    out = [rec]
    for k in range(4):
        c = rec.copy()
        n = len(c)
        c[:, 23] *= 10.0 ** rng.uniform(-4, 4, n)            # dt
        c[:, 24] *= 10.0 ** rng.uniform(-3, 3, n)            # rho
        c[:, 25] *= 10.0 ** rng.uniform(-3, 3, n)            # u_int
        c[:, 33] *= 10.0 ** rng.uniform(-4, 4, n)            # E
        c[:, 30:33] *= 10.0 ** rng.uniform(-2, 1, (n, 1))    # B
        c[: n // 8, 30:33] = 0.0
        c[n // 8: n // 4, 26:29] = 0.0
        c[n // 4: n // 3, 34:37] = 0.0
        c[-3, 25], c[-2, 33], c[-1, 24] = -1e-9, 0.0, np.nan
        out.append(c)
    a = np.ascontiguousarray(np.concatenate(out))
    path = tmp_path_factory.mktemp("cells") / "cells.bin"
    a.tofile(path)
    return str(path), len(a)


@pytest.mark.parametrize("variant", range(12))
def test_lean_solve_is_bitwise_the_plain_solve(lean_binary, cells, variant):
    """Each option that changes the solve's path (lean_check.cpp's variants:
    bisection off, unscaled Jacobian, lagged opacities, no ceiling and no entropy
    fallback, damped levels, opacity channels, another adiabatic index, tight
    convergence), with every rung of the ladder reached."""
    path, n = cells
    r = subprocess.run([lean_binary, path, str(n), str(variant)], check=True, capture_output=True, text=True)
    bad, bad_w, ok, failed, *rungs = (int(x) for x in r.stdout.split())
    assert bad == 0 and bad_w == 0, r.stderr
    assert ok > 0 and failed > 0 and ok + failed == n and sum(1 for x in rungs if x) >= 3


@pytest.mark.parametrize("variant", [12, 15])
def test_ladder_without_rungs_fails_every_cell(lean_binary, cells, variant):
    """A negative radimp_opdamp_maxlevels leaves the ladder no rung: every cell fails
    at once with its state untouched, as in the plain solve."""
    path, n = cells
    r = subprocess.run([lean_binary, path, str(n), str(variant)], check=True, capture_output=True, text=True, timeout=120)
    bad, bad_w, ok, failed, *rungs = (int(x) for x in r.stdout.split())
    assert bad == 0 and bad_w == 0, r.stderr
    assert ok == 0 and failed == n


@pytest.mark.parametrize("spin", [0.0, 0.5, -0.3, 0.95])
def test_torus_functions_are_bitwise_the_plain_ones(lean_binary, spin):
    r = subprocess.run([lean_binary, "init", str(spin)], check=True, capture_output=True, text=True)
    bad, n = (int(x) for x in r.stdout.split())
    assert bad == 0 and n > 100


def test_parallel_fold_is_bitwise_the_serial_sum(lean_binary):
    r = subprocess.run([lean_binary, "fold"], check=True, capture_output=True, text=True)
    bad, mapped = (int(x) for x in r.stdout.split())
    assert bad == 0 and mapped > 10000
