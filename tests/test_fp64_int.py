"""The integer forms of FP64 operations (csrc/fp64_int.cuh): the FP64 results, bit for bit."""
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_integer_forms_equal_fp64_on_the_cpu(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-o", exe,
                    os.path.join(ROOT, "tests", "drivers", "fp64_int_check.cpp")], check=True)
    cases, bad = map(int, subprocess.run([exe, "3000000"], check=True, capture_output=True, text=True).stdout.split())
    assert cases > 1000000 and bad == 0


def states(q, n, kind, rng):
    """Populations around the limits within which the integer forms apply."""
    w = O.equilibrium(q, 0, 0, 0, 1.0)
    f = []
    for _ in range(n):
        u = rng.uniform(-1, 1, 3) * (1, 1, q == 19)
        rho = 1 + rng.normal(0, 0.02)
        if kind == "rest":
            u, rho = u * 0, 1.0
        elif kind == "tiny":
            u = u * 10.0 ** rng.uniform(-300, -3)
        elif kind == "mach":
            u = u * 0.17
        elif kind == "fast":
            u = u * 0.5
        elif kind == "dense":
            u, rho = u * 0.1, rng.choice([0.3, 0.49, 0.51, 0.99, 1.0, 1.01, 1.9, 2.1, 40.0])
        else:
            u = u * 0.06
        g = O.equilibrium(q, *u, rho)
        if kind == "noise":
            g = g + rng.normal(0, 1, q) * 10.0 ** rng.uniform(-9, -1)
        elif kind == "dyadic":
            g = np.round(g * 2.0 ** 12) / 2.0 ** 12
        elif kind == "mach":
            g = g + rng.normal(0, 1e-4, q)
        elif kind == "holes":
            g = g * rng.choice([0.0, 1e-3, 1.0, 1.0, 1.0], q) - (rng.random(q) < 0.05) * w
        f.append(g)
    return np.concatenate(f)


@pytest.mark.gpu
@pytest.mark.parametrize("q,shape", [(9, (67, 31, 1)), (19, (17, 11, 7))])
@pytest.mark.parametrize("op", [1, 2, 3, 4])
@pytest.mark.parametrize("kind", ["rest", "tiny", "mach", "fast", "dense", "noise", "dyadic", "holes"])
def test_fp64_collision_at_the_limits_of_the_integer_forms(q, shape, op, kind):
    """One collision and a few steps of states inside, at and outside the ranges in which the exact path uses
    integer arithmetic, mixed among the lanes of a warp: the oracle's bits."""
    import erlbm_gb300 as E
    if q == 19 and op == 2:
        pytest.skip("MRT is a D2Q9 operator")
    n = int(np.prod(shape))
    f = states(q, n, kind, np.random.default_rng(100 * q + op))
    tnh = 1.0 if op == 3 else 0.65
    for steps in (1, 4):
        ref = O.Lattice(q, *shape, None, 0.55, tnh, op)
        ref.set(f)
        ref.step(steps)
        with E.Lattice(q, *shape, None, 0.55, tnh, op, E.FP64) as lat:
            lat.set_populations(f)
            lat.step(steps)
            got = lat.get_populations(E.STAGE_POST_COLLISION)
        want = ref.get(1)
        fine = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fine) and np.array_equal(got[fine], want[fine])


@pytest.mark.gpu
@pytest.mark.parametrize("q,shape", [(9, (131, 83, 1)), (9, (211, 157, 1)), (19, (29, 23, 17)), (19, (41, 32, 26))])
@pytest.mark.parametrize("kind", ["rest", "mach", "dense", "noise", "dyadic", "holes"])
def test_fp64_collision_of_larger_lattices(q, shape, kind):
    """The same for lattices past the sizes of four lanes a node, and past those of FP64 sums."""
    import erlbm_gb300 as E
    n = int(np.prod(shape))
    f = states(q, n, kind, np.random.default_rng(n))
    for op in (3, 4):
        ref = O.Lattice(q, *shape, None, 0.52, 0.65, op)
        ref.set(f)
        ref.step(3)
        with E.Lattice(q, *shape, None, 0.52, 0.65, op, E.FP64) as lat:
            lat.set_populations(f)
            lat.step(3)
            got = lat.get_populations(E.STAGE_POST_COLLISION)
        want = ref.get(1)
        fine = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), fine) and np.array_equal(got[fine], want[fine])


@pytest.mark.gpu
@pytest.mark.parametrize("q,nx,ny", [(9, 16, 16), (9, 24, 23), (9, 33, 31), (19, 12, 10), (19, 16, 17), (19, 21, 20)])
@pytest.mark.parametrize("kind", ["mach", "fast", "dense", "noise"])
def test_batched_fp64_runs_of_states_mixed_among_the_lanes(q, nx, ny, kind):
    """Batched runs (one, two and four nodes a thread) whose warps have lanes in and out of the ranges of the integer
    forms: the greatest density of four steps, bit for bit."""
    import erlbm_gb300 as E
    n, limit = nx * ny, 1e6
    runs, blocks, want = [], [], []
    for k, op in enumerate((3, 4, 1)):
        f = states(q, n, kind, np.random.default_rng(10 * n + k))
        tnh = 1.0 if op == 3 else 0.65
        ref = O.Lattice(q, nx, ny, 1, None, 0.6, tnh, op)
        ref.set(f)
        most = 0.0
        for _ in range(4):
            ref.step(1)
            most = max(most, ref.max_abs_density(1)[0])
        runs.append(dict(op=op, tau=0.6, tau_nh=tnh, u0=0.0, n_steps=4, aos_offset=k * f.size))
        blocks.append(f)
        want.append(most / limit)
    got = E.batch_run(q, nx, ny, runs, precision=E.FP64, init=E.INIT_AOS, aos=np.concatenate(blocks),
                      density_check=True, density_limit=limit)
    assert [g["margin"] for g in got] == want
