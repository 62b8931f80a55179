"""The serial energy sum around the lengths at which it changes its form: the oracle's bits."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 255, 511, 512, 513, 640, 1023, 1024, 1025, 2048, 2049])
def test_energy_sum_at_the_lengths_of_its_forms(n):
    """The plain loop, the first chunk, whole chunks and one term more."""
    import erlbm_gb300 as E
    rng = np.random.default_rng(n)
    f = np.concatenate([O.equilibrium(9, *(rng.normal(0, 0.05, 2)), 0, 1 + rng.normal(0, 0.01)) for _ in range(n)])
    ref = O.Lattice(9, n, 1, 1, None, 0.6, 0.65, 4)
    ref.set(f)
    with E.Lattice(9, n, 1, 1, None, 0.6, 0.65, 4, E.FP64) as lat:
        lat.set_populations(f)
        assert lat.kinetic_energy(E.STAGE_POST_STREAM) == ref.kinetic_energy(0)
