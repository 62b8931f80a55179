"""Step calls on a stream that the caller is recording into a CUDA graph of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def channel(E, nx, ny):
    s = np.zeros((ny, nx), np.uint8)
    s[0] = s[-1] = s[:, 0] = s[:, -1] = 1
    return s.reshape(-1), dict(inlet_x=1, inlet_kind=E.INLET_PARABOLIC, parabolic_L=ny - 2, u_in=0.05, outlet_x=nx - 2,
                               outlet_kind=E.OUTLET_CONVECTIVE)


@pytest.mark.parametrize("steps", [7, 50, 70, 199])
@pytest.mark.parametrize("nx,ny,planes,before", [(100, 60, False, 0), (256, 64, False, 0), (256, 64, False, 200),
                                                 (2000, 600, True, 0), (2000, 600, True, 400), (2048, 800, True, 0),
                                                 (2048, 800, True, 400)])
def test_recorded_steps_replay_as_the_steps_they_stand_for(nx, ny, planes, before, steps):
    """Periodic boxes and channels, before and after long calls that are not recorded: the replayed graph gives the
    populations of the same steps taken directly."""
    import torch

    import erlbm_gb300 as E
    torch.cuda.set_device(0)
    solid, bc = channel(E, nx, ny) if planes else (None, None)
    got, f = [], None
    for recorded in (False, True):
        with E.Lattice(9, nx, ny, 1, solid, 0.56, 0.7, E.OP_EXTREG, E.FP32_SHIFTED) as lat:
            stream = torch.cuda.Stream()
            lat.set_stream(stream.cuda_stream)
            if f is None:
                w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
                f = (w[None, :] * (1 + 0.01 * np.random.default_rng(nx).standard_normal((lat.n_fluid, 9)))).ravel()
            lat.set_populations(f)
            lat.step(1 + before, bc)
            lat.sync()
            if recorded:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.stream(stream):
                    graph.capture_begin()
                    lat.step(steps, bc)
                    graph.capture_end()
                    graph.replay()
                stream.synchronize()
            else:
                lat.step(steps, bc)
            got.append(lat.get_populations(E.STAGE_POST_COLLISION))
            lat.set_stream(None)
    assert np.array_equal(*got)
