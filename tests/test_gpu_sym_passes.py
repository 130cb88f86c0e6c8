"""The halved cosine passes (sgh_sym.cuh) at the edges of their tiles: axis
lengths around the 16-slice stages and the 32-pair tiles, odd lengths with a
middle sample, odd column counts (8-byte copies), columns that end inside a
tile, several stages. Against scipy and the oracle to 1e-12, the bound the
transforms and the output field are held to elsewhere."""
import numpy as np
import pytest
import scipy.fft

from conftest import rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(15,), (16,), (17,), (33,), (1030,), (31, 64), (64, 31), (65, 66), (16, 17, 18), (33, 70, 47), (66, 34, 129),
          (5, 130, 260)]


@pytest.mark.parametrize("shape", SHAPES)
def test_dct_pair_matches_scipy(shape):
    import torch
    from spectral_galerkin_heat_b200 import kernels as K
    x = np.random.default_rng(sum(shape)).standard_normal(shape)
    xd = torch.as_tensor(x, device="cuda")
    f = K.DCT_II(xd)
    assert rel_l2(f.cpu().numpy(), scipy.fft.dctn(x, type=2, norm="ortho")) < 1e-12
    assert rel_l2(K.IDCT_II(xd).cpu().numpy(), scipy.fft.dctn(x, type=3, norm="ortho")) < 1e-12
    # a view that starts off a 16-byte boundary
    flat = torch.empty(x.size + 1, dtype=torch.float64, device="cuda")[1:]
    v = flat.view(shape)
    v.copy_(xd)
    assert np.array_equal(K.DCT_II(v).cpu().numpy(), f.cpu().numpy())


@pytest.mark.parametrize("shape", [(2, 3, 4), (15, 16, 17), (33, 31, 64), (70, 65, 34), (9, 130, 66)])
def test_node_field_matches_oracle_in_both_axis_orders(shape):
    import ctypes as C
    import torch
    from oracle.sgh_oracle import nodal_temperature
    from spectral_galerkin_heat_b200 import _lib, kernels as K
    nz, ny, nx = shape
    size = (2e-3, 1.1e-3, 0.4e-3)
    a = np.random.default_rng(nx).standard_normal(shape)
    ad = torch.as_tensor(a, device="cuda")

    class State:
        pass

    st = State()
    st.size = size
    want = nodal_temperature(a, size)
    got = K.reconstruct_temperature_DCT(ad, st)
    assert tuple(got.shape) == (nx + 1, ny + 1, nz + 1)
    assert rel_l2(got.cpu().numpy(), want) < 1e-12
    out = torch.empty((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device="cuda")
    nb = C.c_uint64()
    L = _lib.lib()
    _lib.check("ws", L.sgh_nodal_workspace_bytes(nx, ny, nz, C.byref(nb)))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    _lib.check("nodal", L.sgh_nodal_temperature(nx, ny, nz, *size, C.c_void_p(ad.data_ptr()),
                                                C.c_void_p(out.data_ptr()), C.c_void_p(ws.data_ptr()), nb.value, None))
    torch.cuda.synchronize()
    assert np.array_equal(out.permute(2, 1, 0).contiguous().cpu().numpy(), got.cpu().numpy())
