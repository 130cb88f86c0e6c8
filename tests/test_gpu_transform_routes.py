"""Long axes of few columns, on both sides of the rule that sends a pass to the
halved or to the full contraction (sym::fills): DCT pairs against scipy, node
fields in both axis orders against the oracle, to the 1e-12 these are held to
elsewhere."""
import ctypes as C

import numpy as np
import pytest
import scipy.fft

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(129, 65), (300, 17), (17, 300, 5), (257, 640), (400, 400), (20, 20, 600)])
def test_dct_pair(shape):
    import torch
    from spectral_galerkin_heat_b200 import kernels as K
    x = np.random.default_rng(sum(shape)).standard_normal(shape)
    xd = torch.as_tensor(x, device="cuda")
    assert rel_l2(K.DCT_II(xd).cpu().numpy(), scipy.fft.dctn(x, type=2, norm="ortho")) < 1e-12
    assert rel_l2(K.IDCT_II(xd).cpu().numpy(), scipy.fft.dctn(x, type=3, norm="ortho")) < 1e-12


@pytest.mark.parametrize("nx,ny,nz", [(300, 9, 10), (9, 301, 10), (8, 9, 300), (129, 12, 7), (258, 131, 3), (200, 150, 90)])
def test_node_field(nx, ny, nz):
    import torch
    from oracle.sgh_oracle import nodal_temperature
    from spectral_galerkin_heat_b200 import _lib, kernels as K
    size = (2e-3, 1.1e-3, 0.4e-3)
    a = np.random.default_rng(nx).standard_normal((nz, ny, nx))
    ad = torch.as_tensor(a, device="cuda")

    class State:
        pass

    st = State()
    st.size = size
    got = K.reconstruct_temperature_DCT(ad, st)
    assert rel_l2(got.cpu().numpy(), nodal_temperature(a, size)) < 1e-12
    out = torch.empty((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device="cuda")
    nb = C.c_uint64()
    L = _lib.lib()
    _lib.check("ws", L.sgh_nodal_workspace_bytes(nx, ny, nz, C.byref(nb)))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    _lib.check("nodal", L.sgh_nodal_temperature(nx, ny, nz, *size, C.c_void_p(ad.data_ptr()),
                                                C.c_void_p(out.data_ptr()), C.c_void_p(ws.data_ptr()), nb.value, None))
    torch.cuda.synchronize()
    assert np.array_equal(out.permute(2, 1, 0).contiguous().cpu().numpy(), got.cpu().numpy())
