"""The programs that take several operands through one launch (the cross product's VJP, the linearised MHD pair and its
transpose, the MHD bundle) over the mode counts that their kernel serves and their neighbours, odd and even point
counts, one and several batch entries.  Against pocketfft products; rel-L2 <= 1e-12, the bar of the FP64 forms, and the
transposes against <J v, c> = <v, J^T c> to 1e-12."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu
TOL = 1e-12
SIZES = [8, 9, 12, 16, 17, 22, 23, 32, 33, 43, 44, 49, 55, 63, 64, 65]


def _pad(m):
    return (3 * m) // 2


def _field(npts, nslot, m, seed):
    return R.synthetic_field(npts, nslot, m, 0.2, seed)


@pytest.mark.parametrize("npts", [7, 24])
@pytest.mark.parametrize("m", SIZES)
def test_bundle(npts, m):
    f = [_field(npts, 6, m, 50 + i) for i in range(5)]
    refs = R.mhd_bundle(*f, _pad(m), engine=lambda op, x, y: R.fft_par(op, x, y, _pad(m)))
    outs = sf.bundle_mhd(*[sf.to_device(x) for x in f], m_max_pad=_pad(m), algo=sf.ALGO_FAST)
    for o, r in zip(outs, refs):
        assert R.rel_l2(sf.to_host(o), r) <= TOL


@pytest.mark.parametrize("npts,k", [(7, 1), (24, 3)])
@pytest.mark.parametrize("m", SIZES)
def test_linearised_pair_and_transposes(npts, k, m):
    cross = lambda x, y: R.fft_par("cross", np.asfortranarray(x), np.asfortranarray(y), _pad(m))  # noqa: E731
    u, w, b = (_field(npts, 6, m, 60 + i) for i in range(3))
    v = np.asfortranarray(np.stack([_field(npts, 18, m, 70 + i) for i in range(k)], -1))
    c = np.asfortranarray(np.stack([_field(npts, 12, m, 80 + i) for i in range(k)], -1))
    base = [sf.to_device(x) for x in (u, w, b)]
    jv = sf.to_host(sf.mhd_jvp(*base, sf.to_device(v), m_max_pad=_pad(m)))
    jc = sf.to_host(sf.mhd_vjp(*base, sf.to_device(c), m_max_pad=_pad(m)))
    c1 = np.asfortranarray(c[:, :6])
    jc1 = sf.to_host(sf.cross_vjp(base[0], base[1], sf.to_device(c1), m_max_pad=_pad(m)))
    for t in range(k):
        du, dw, db = (v[:, 6 * i:6 * i + 6, :, t] for i in range(3))
        ref = np.concatenate([cross(du, w) + cross(u, dw), cross(du, b) + cross(u, db)], 1)
        assert R.rel_l2(jv[..., t], ref) <= TOL
        scale = np.linalg.norm(jv[..., t]) * np.linalg.norm(c[..., t])
        assert abs(float((jv[..., t] * c[..., t]).sum() - (v[..., t] * jc[..., t]).sum())) <= TOL * scale
        lhs = float(((cross(du, w) + cross(u, dw)) * c1[..., t]).sum())
        assert abs(lhs - float((v[:, :12, :, t] * jc1[..., t]).sum())) <= TOL * scale
