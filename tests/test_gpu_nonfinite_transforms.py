"""A NaN or an infinity in the input of a whole-array transform reaches every
output that it has a weight in, the middle ones (whose weight on odd modes is
zero, and 0 * NaN is NaN) included, as the full contraction has it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("shape", [(17,), (33, 65), (19, 21, 35), (16, 32, 64)])
@pytest.mark.parametrize("odd", [0, 1])
def test_dct_pair(shape, odd, value):
    import torch
    from spectral_galerkin_heat_b200 import kernels
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.standard_normal(shape)).cuda()
    x[tuple(2 + odd for _ in shape)] = value
    for f in (kernels.DCT_II, kernels.IDCT_II):
        y = f(x).cpu().numpy()
        assert not np.isfinite(y).any()


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("mode", [(1, 0, 0), (0, 3, 0), (0, 0, 5), (2, 2, 2), (1, 3, 5)])
@pytest.mark.parametrize("nx,ny,nz", [(32, 16, 8), (33, 18, 7)])
def test_node_field(nx, ny, nz, mode, value):
    import torch
    from spectral_galerkin_heat_b200 import B200SpectralSolver, SimulationContext, kernels, workloads
    s = B200SpectralSolver(None, SimulationContext.from_dict(workloads.straight_track(nx, ny, nz)[0]))
    s.initialize()
    a = torch.from_numpy(np.random.default_rng(6).standard_normal((nz, ny, nx))).cuda()
    a[mode] = value
    T = kernels.reconstruct_temperature_DCT(a, s.state).cpu().numpy()
    assert not np.isfinite(T).any()
    s.finalize()
