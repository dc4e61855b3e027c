"""The FAST form at the bounds of its compile-time geometries: every (k-steps, angle tiles) pair up to m = 64, odd mode
counts (the odd classes one mode short), the 64-mode third-fold kernel at fewer modes, the one-warp kernel with more
tiles than resident warps, and point counts around the 8-point tiles.  Against pocketfft products on the reference's
grid; rel-L2 <= 1e-12, the bar of the FP64 forms."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu
TOL = 1e-12
SIZES = [1, 3, 8, 9, 11, 12, 16, 17, 22, 23, 24, 25, 31, 32, 33, 40, 41, 43, 44, 48, 49, 54, 55, 56, 57, 63, 64, 65]


def _pad(m):
    return max(1, (3 * m) // 2)


@pytest.mark.parametrize("m", SIZES)
@pytest.mark.parametrize("kind", ["cross", "dot", "prod", "svect", "tensor"])
def test_products_at_geometry_bounds(kind, m):
    _, n1, n2, _ = sf.KINDS[kind]
    for npts in (9, 24):
        V1, V2 = R.synthetic_field(npts, n1, m, 0.2, 3 * m), R.synthetic_field(npts, n2, m, 0.2, 3 * m + 1)
        ref = R.fft_par(kind, V1, V2, _pad(m))
        out = sf.product(sf.KINDS[kind][0], sf.to_device(V1), sf.to_device(V2), m_max_pad=_pad(m), algo=sf.ALGO_FAST)
        assert R.rel_l2(sf.to_host(out), ref) <= TOL


@pytest.mark.parametrize("npts,m", [(30011, 4), (30000, 13), (29999, 16)])
@pytest.mark.parametrize("kind", ["cross", "prod"])
def test_one_warp_kernel_over_many_tiles(kind, npts, m):
    _, n1, n2, _ = sf.KINDS[kind]
    V1, V2 = R.synthetic_field(npts, n1, m, 0.2, 7), R.synthetic_field(npts, n2, m, 0.2, 8)
    ref = R.fft_par(kind, V1, V2, _pad(m))
    a, b = sf.to_device(V1), sf.to_device(V2)
    out = sf.product(sf.KINDS[kind][0], a, b, m_max_pad=_pad(m), algo=sf.ALGO_FAST)
    assert R.rel_l2(sf.to_host(out), ref) <= TOL
    if kind == "cross":  # in place
        sf.product(sf.OP_CROSS, a, b, out=a, m_max_pad=_pad(m), algo=sf.ALGO_FAST)
        assert np.array_equal(sf.to_host(a), sf.to_host(out))


@pytest.mark.parametrize("m", [3, 9, 16, 21, 30, 37, 45, 59, 63])
def test_adjoint_identity_at_geometry_bounds(m):
    npts, k = 37, 2
    u, w = (sf.to_device(R.synthetic_field(npts, 6, m, 0.2, 90 + i)) for i in range(2))
    v = np.asfortranarray(np.stack([R.synthetic_field(npts, 12, m, 0.2, 95 + i) for i in range(k)], -1))
    c = np.asfortranarray(np.stack([R.synthetic_field(npts, 6, m, 0.2, 97 + i) for i in range(k)], -1))
    jv = sf.to_host(sf.cross_jvp(u, w, sf.to_device(v), m_max_pad=_pad(m)))
    jc = sf.to_host(sf.cross_vjp(u, w, sf.to_device(c), m_max_pad=_pad(m)))
    for t in range(k):
        ref = R.fft_par("cross", np.asfortranarray(v[:, :6, :, t]), sf.to_host(w), _pad(m)) + R.fft_par(
            "cross", sf.to_host(u), np.asfortranarray(v[:, 6:, :, t]), _pad(m))
        assert R.rel_l2(jv[..., t], ref) <= TOL
        lhs, rhs = float((jv[..., t] * c[..., t]).sum()), float((v[..., t] * jc[..., t]).sum())
        scale = np.linalg.norm(jv[..., t]) * np.linalg.norm(c[..., t])
        assert abs(lhs - rhs) <= TOL * scale


@pytest.mark.parametrize("waves", [1.6, 1.7, 1.74, 1.8, 2.0, 2.1])
@pytest.mark.parametrize("m", [25, 28, 29, 32])
def test_dot_products_around_the_waves_of_the_one_warp_kernel(m, waves):
    torch = pytest.importorskip("torch")
    npts = int(8 * 12 * torch.cuda.get_device_properties(0).multi_processor_count * waves) - 3
    V1, V2 = R.synthetic_field(npts, 6, m, 0.2, 7), R.synthetic_field(npts, 6, m, 0.2, 8)
    out = sf.product(sf.OP_DOT, sf.to_device(V1), sf.to_device(V2), m_max_pad=_pad(m), algo=sf.ALGO_FAST)
    assert R.rel_l2(sf.to_host(out), R.fft_par("dot", V1, V2, _pad(m))) <= TOL
