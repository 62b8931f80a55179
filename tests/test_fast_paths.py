"""Forms of the single-lattice path that are chosen by size: they give the general path's bits."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def flow(q, nx, ny, nz, seed, amp=0.03):
    """A smooth random flow with noise, as AoS populations."""
    rng = np.random.default_rng(seed)
    n = nx * ny * nz
    f = np.concatenate([O.equilibrium(q, *(rng.normal(0, amp, 3) * (1, 1, q == 19)), 1 + rng.normal(0, 0.01))
                        for _ in range(n)])
    return f + rng.normal(0, 1e-4, f.size)


@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 3), (16, 16), (257, 1), (61, 67), (256, 40)])
@pytest.mark.parametrize("kind", ["flow", "rest", "uniform", "mixed", "nan"])
def test_energy_sum_keeps_the_serial_order_and_rounding(nx, ny, kind):
    """kinetic_energy up to 65536 nodes is the reference's serial sum, bit for bit: equal terms (ties at every
    add), zeros, terms over twenty binades, a term that is not a number."""
    import erlbm_gb300 as E
    n = nx * ny
    rng = np.random.default_rng(n)
    if kind == "rest":
        f = np.tile(O.equilibrium(9, 0, 0, 0, 1.0), n)
    elif kind == "uniform":
        f = np.tile(O.equilibrium(9, 0.25, 0.5, 0, 1.0), n)
    elif kind == "mixed":
        f = np.concatenate([O.equilibrium(9, 0.3 * 2.0 ** -rng.integers(0, 30), 0, 0, 1.0) for _ in range(n)])
    else:
        f = flow(9, nx, ny, 1, n)
        if kind == "nan":
            f[9 * (n // 2)] = np.nan
    ref = O.Lattice(9, nx, ny, 1, None, 0.6, 0.65, 4)
    ref.set(f)
    with E.Lattice(9, nx, ny, 1, None, 0.6, 0.65, 4, E.FP64) as lat:
        lat.set_populations(f)
        a, b = lat.kinetic_energy(E.STAGE_POST_STREAM), ref.kinetic_energy(0)
        assert a == b or (np.isnan(a) and np.isnan(b))


@pytest.mark.parametrize("nx,ny", [(32, 8), (33, 9), (61, 17), (128, 19), (132, 16), (190, 31), (1001, 24), (644, 70),
                                   (1996, 401)])
@pytest.mark.parametrize("steps", [2, 3, 6, 73])
def test_periodic_steps_of_any_box_equal_their_cpu_restatement(nx, ny, steps):
    """Two- and three-step strips chosen by the engine, on boxes whose sides leave remainders of the strips,
    chunks and row pairs; leftover steps; graph blocks (73 steps)."""
    import erlbm_gb300 as E
    if nx * ny * steps > 6e6:
        steps = 7
    op = (1, 3, 4, 2)[(nx + ny + steps) % 4]
    f = flow(9, nx, min(ny, 40), 1, nx)
    f = np.resize(f.reshape(-1, 9), (nx * ny, 9)).reshape(-1)
    tnh = 1.0 if op == 3 else 0.65
    with E.Lattice(9, nx, ny, 1, None, 0.53, tnh, op, E.FP32_SHIFTED) as lat:
        lat.set_populations(f)
        lat.step(steps)
        got = lat.get_populations(E.STAGE_POST_COLLISION)
    assert np.array_equal(got, O.fp32_periodic_d2q9(nx, ny, op, 0.53, tnh, f, steps))


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 3), (129, 3, 2), (31, 33, 5), (127, 2, 7), (16, 16, 1)])
@pytest.mark.parametrize("op", [1, 3, 4])
def test_periodic_d3q19_of_any_box_equals_its_cpu_restatement(shape, op):
    import erlbm_gb300 as E
    f = flow(19, *shape, seed=sum(shape))
    tnh = 1.0 if op == 3 else 0.65
    with E.Lattice(19, *shape, None, 0.53, tnh, op, E.FP32_SHIFTED) as lat:
        lat.set_populations(f)
        lat.step(5)
        got = lat.get_populations(E.STAGE_POST_COLLISION)
    assert np.array_equal(got, O.fp32_periodic_d3q19(*shape, op, 0.53, tnh, f, 5))


def test_run_without_density_checks_takes_the_stepping_path():
    """run() with energy checks steps as step() does: the same populations, and the checks of the oracle's loop."""
    import erlbm_gb300 as E
    nx, ny = 132, 20
    f = flow(9, nx, ny, 1, 3)
    with E.Lattice(9, nx, ny, 1, None, 0.56, 0.65, 4, E.FP32_SHIFTED) as a, \
            E.Lattice(9, nx, ny, 1, None, 0.56, 0.65, 4, E.FP32_SHIFTED) as b:
        a.set_populations(f)
        b.set_populations(f)
        r = a.run(250, energy_every=100, energy_factor=50.0)
        b.step(250)
        assert r["label"] == 0 and r["steps_done"] == 250
        assert np.array_equal(a.get_populations(), b.get_populations())


@pytest.mark.parametrize("nx,ny,op", [(1000, 250, 4), (1003, 211, 3), (701, 300, 2), (1536, 1024, 4), (1660, 922, 1)])
@pytest.mark.parametrize("planes", ["channel", "open", "density", "solids"])
def test_three_steps_per_launch_with_planes_equal_single_steps(nx, ny, op, planes):
    """Boxes with walls, an obstacle, scattered solids (also on the seams) and boundary planes take three steps per
    launch in calls of many steps; calls of one step run one at a time.  The same bits, through graph blocks, single
    launches and leftover steps."""
    import erlbm_gb300 as E
    rng = np.random.default_rng(nx + ny)
    s = np.zeros((ny, nx), np.uint8)
    if planes in ("channel", "density"):
        s[0] = s[-1] = s[:, 0] = s[:, -1] = 1
    if planes != "open":
        y, x = np.mgrid[0:ny, 0:nx]
        s[(x - nx // 3) ** 2 + (y - ny // 2) ** 2 <= (ny // 10) ** 2] = 1
        s[rng.integers(0, ny, 30), rng.integers(0, nx, 30)] = 1
        s[ny // 2, nx - 1] = s[0, nx // 2] = 1
    bc = {"channel": dict(inlet_x=1, inlet_kind=E.INLET_PARABOLIC, parabolic_L=ny - 2, u_in=0.05, outlet_x=nx - 2,
                          outlet_kind=E.OUTLET_CONVECTIVE),
          "density": dict(inlet_x=1, u_in=0.04, outlet_x=nx - 2),
          "open": dict(inlet_x=0, u_in=0.03, outlet_x=nx - 1, outlet_kind=E.OUTLET_OPEN, open_y=ny - 1),
          "solids": None}[planes]
    with E.Lattice(9, nx, ny, 1, s.reshape(-1) if s.any() else None, 0.55, 1.0 if op == 3 else 0.7, op,
                   E.FP32_SHIFTED) as a, \
            E.Lattice(9, nx, ny, 1, s.reshape(-1) if s.any() else None, 0.55, 1.0 if op == 3 else 0.7, op,
                      E.FP32_SHIFTED) as b:
        w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
        f = (w[None, :] * (1.0 + 0.03 * rng.standard_normal((a.n_fluid, 9)))).ravel()
        a.set_populations(f)
        b.set_populations(f)
        a.step(200, bc)
        for _ in range(200):
            b.step(1, bc)
        assert np.array_equal(a.get_populations(E.STAGE_POST_COLLISION), b.get_populations(E.STAGE_POST_COLLISION))
        assert np.array_equal(a.get_populations(), b.get_populations())


@pytest.mark.parametrize("nx,ny", [(16, 16), (8, 8), (32, 2), (2, 32), (24, 24), (32, 32), (12, 12), (16, 15)])
@pytest.mark.parametrize("op", [1, 3, 4])
def test_mirrored_taylor_green_runs_equal_the_general_map_kernel(nx, ny, op):
    """FP32 Taylor-Green runs keep 14 of the 19 populations (the others are mirror images in z): every result of
    the restatement of the general kernel, bit for bit, stable and unstable runs, and shapes left to the latter."""
    import erlbm_gb300 as E
    runs = [dict(op=op, tau=tau, tau_nh=0.65, u0=u0, n_steps=n)
            for tau, u0, n in ((0.6, 0.05, 250), (0.5003, 0.2, 400), (0.5001, 0.55, 1000), (0.53, 0.01, 0), (0.53, 0.01, 1))]
    got = E.batch_run(19, nx, ny, runs, precision=E.FP32_SHIFTED, energy_every=40, energy_factor=2.0, init=E.INIT_TG_MAP)
    block = ((nx * ny + 1) // 2 + 31) // 32 * 32
    for r, g in zip(runs, got):
        want = O.fp32_batch_run(19, nx, ny, op, r["tau"], r["tau_nh"], r["u0"], r["n_steps"], block, 2, energy_every=40,
                                energy_factor=2.0, init=1)
        for k in want:
            assert g[k] == want[k] or (g[k] != g[k] and want[k] != want[k]), (k, r, g, want)
