"""Three steps per launch with solids and boundary planes: when they are set up, and that they give single steps' bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)


def geometry(nx, ny, seed, scattered=30):
    rng = np.random.default_rng(seed)
    s = np.zeros((ny, nx), np.uint8)
    s[0] = s[-1] = s[:, 0] = s[:, -1] = 1
    y, x = np.mgrid[0:ny, 0:nx]
    s[(x - nx // 3) ** 2 + (y - ny // 2) ** 2 <= (ny // 10) ** 2] = 1
    s[rng.integers(0, ny, scattered), rng.integers(0, nx, scattered)] = 1
    return s.reshape(-1)


def planes(E, nx, ny, kind):
    return {"channel": dict(inlet_x=1, inlet_kind=E.INLET_PARABOLIC, parabolic_L=ny - 2, u_in=0.05, outlet_x=nx - 2,
                            outlet_kind=E.OUTLET_CONVECTIVE),
            "density": dict(inlet_x=1, u_in=0.04, outlet_x=nx - 2),
            "open": dict(inlet_x=1, u_in=0.03, outlet_x=nx - 2, outlet_kind=E.OUTLET_OPEN, open_y=ny - 2),
            "solids": None}[kind]


def pair(E, nx, ny, solid, op=4):
    """Two lattices of the same state: for long calls, and for calls of single steps."""
    tnh = 1.0 if op == 3 else 0.7
    a, b = (E.Lattice(9, nx, ny, 1, solid, 0.55, tnh, op, E.FP32_SHIFTED) for _ in range(2))
    f = (W[None, :] * (1.0 + 0.03 * np.random.default_rng(nx).standard_normal((a.n_fluid, 9)))).ravel()
    a.set_populations(f)
    b.set_populations(f)
    a.step(1)
    b.step(1)
    return a, b


def step_both(a, b, n, bc):
    a.step(n, bc)
    for _ in range(n):
        b.step(1, bc)
    assert b.launch_form() == (1, False)


def same(E, a, b):
    return np.array_equal(a.get_populations(E.STAGE_POST_COLLISION), b.get_populations(E.STAGE_POST_COLLISION))


@pytest.mark.parametrize("nx,ny,op,steps", [(1003, 511, 3, 745), (1101, 703, 2, 230), (1660, 922, 1, 92),
                                            (1536, 1024, 4, 481), (1664, 1203, 4, 151)])
@pytest.mark.parametrize("kind", ["channel", "density", "open", "solids"])
def test_long_calls_go_by_threes_and_equal_single_steps(nx, ny, op, steps, kind):
    import erlbm_gb300 as E
    a, b = pair(E, nx, ny, geometry(nx, ny, nx), op)
    with a, b:
        step_both(a, b, steps, planes(E, nx, ny, kind))
        assert a.launch_form()[0] == 3
        assert same(E, a, b)


@pytest.mark.parametrize("other,want", [("open", [1, 1, 1, 1, 3, 1, 3, 1, 3, 3, 1]),
                                        ("density", [1, 1, 3, 3, 3, 3, 3, 3, 3, 3, 1])])
def test_calls_in_a_row_add_up_and_a_change_of_planes_starts_again(other, want):
    """86 steps pay on this machine: calls with the same planes add up to them, calls with planes elsewhere start the count
    again, and neither undoes a set-up that stands.  Planes of another kind at the same places share it.  Every call
    gives the single steps' bits."""
    import erlbm_gb300 as E
    nx, ny = 1660, 922
    a, b = pair(E, nx, ny, geometry(nx, ny, 5))
    forms = []
    with a, b:
        for kind, n in (("channel", 40), (other, 40), ("channel", 40), ("channel", 40), ("channel", 70),
                        (other, 50), ("channel", 9), (other, 50), (other, 50), ("channel", 100), ("solids", 7)):
            step_both(a, b, n, planes(E, nx, ny, kind))
            forms.append(a.launch_form()[0])
            assert same(E, a, b), (kind, forms)
    assert forms == want


def test_new_parameters_between_long_calls():
    import erlbm_gb300 as E
    nx, ny = 1660, 922
    a, b = pair(E, nx, ny, geometry(nx, ny, 6))
    with a, b:
        for tau, op in ((0.55, 4), (0.61, 4), (0.58, 2), (0.7, 1)):
            a.set_params(tau, 0.7, op)
            b.set_params(tau, 0.7, op)
            step_both(a, b, 100, planes(E, nx, ny, "channel"))
            assert a.launch_form()[0] == 3 and same(E, a, b)


def test_boxes_full_of_solids_keep_single_steps():
    """More than a quarter of the nodes near a solid: no set-up, and nothing kept of the attempt."""
    import torch

    import erlbm_gb300 as E
    nx, ny = 1003, 700
    a, b = pair(E, nx, ny, geometry(nx, ny, 7, scattered=20000))
    with a, b:
        a.sync()
        before = torch.cuda.mem_get_info()[0]
        step_both(a, b, 400, planes(E, nx, ny, "channel"))
        assert a.launch_form() == (1, False) and same(E, a, b)
        assert before - torch.cuda.mem_get_info()[0] < 4 * nx * ny


@pytest.mark.parametrize("nx,ny", [(132, 20), (100, 31), (256, 33)])
@pytest.mark.parametrize("steps", [2, 3, 5, 71])
def test_launch_shapes_asked_for_on_boxes_of_any_size(nx, ny, steps):
    """set_launch on boxes that its multi-step shapes do not take: the engine's strips or single steps, same bits."""
    import erlbm_gb300 as E
    from oracle import oracle as O
    f = (W[None, :] * (1.0 + 0.02 * np.random.default_rng(ny).standard_normal((nx * ny, 9)))).ravel()
    want = O.fp32_periodic_d2q9(nx, ny, 4, 0.55, 0.7, f, steps)
    for shape in (dict(), dict(two_step=True), dict(three_step=True), dict(three_step=True, wide_strips=True)):
        with E.Lattice(9, nx, ny, 1, None, 0.55, 0.7, 4, E.FP32_SHIFTED) as lat:
            lat.set_launch(128, **shape)
            lat.set_populations(f)
            lat.step(steps)
            assert np.array_equal(lat.get_populations(E.STAGE_POST_COLLISION), want), shape


def test_set_ups_do_not_wait_for_the_servers_resident_loops():
    """While a server works through a long request: a set-up, one that replaces it and one that is refused."""
    import erlbm_gb300 as E
    nx, ny = 1660, 922
    a, b = pair(E, nx, ny, geometry(nx, ny, 8))
    c, d = pair(E, 1003, 700, geometry(1003, 700, 9, scattered=20000))
    with a, b, c, d, E.Server(hbm_budget_bytes=1 << 30) as srv:
        def run(steps):
            return srv.submit(E.REQ_TG3D, E.FP64, E.OP_EXTREG, L=64, tau=0.55, tau_nh=0.65, u0=0.05, n_steps=steps)
        srv.wait(run(2))
        ticket = run(30000)  # some seconds
        for kind in ("channel", "open"):
            a.step(100, planes(E, nx, ny, kind))
            a.sync()
            assert a.launch_form()[0] == 3
        c.step(400, planes(E, 1003, 700, "channel"))
        c.sync()
        assert c.launch_form() == (1, False)
        assert srv.poll(ticket) is None  # still running
        for kind in ("channel", "open"):
            for _ in range(100):
                b.step(1, planes(E, nx, ny, kind))
        b.sync()
        assert srv.wait(ticket)["status"] == 0
        assert same(E, a, b)
