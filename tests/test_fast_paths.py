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
