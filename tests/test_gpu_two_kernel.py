"""The two-kernel form on the programs that run it (bundle and conservative advection from m = 108, tensor from m = 87): the
whole grid with an odd and an even number of angle tiles, the grid's residue classes (m = 256, 384, 512), each number of
classes, and workspaces of many point chunks.  Against pocketfft products; rel-L2 <= 1e-12, the bar of the FP64 forms."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _pad(m):
    return 3 * m // 2


def _check_bundle(npts, m):
    f = [R.synthetic_field(npts, 6, m, 0.05, 500 + i) for i in range(5)]
    refs = R.mhd_bundle(*f, _pad(m), engine=lambda op, x, y: R.fft_par(op, x, y, _pad(m)))
    for o, r in zip(sf.bundle_mhd(*[sf.to_device(x) for x in f], m_max_pad=_pad(m), algo=sf.ALGO_FAST), refs):
        assert R.rel_l2(sf.to_host(o), r) <= TOL


def _check_tensor(npts, m):
    a, b = (R.synthetic_field(npts, 6, m, 0.05, 510 + i) for i in range(2))
    out = sf.product(sf.OP_TENSOR, sf.to_device(a), sf.to_device(b), m_max_pad=_pad(m), algo=sf.ALGO_FAST)
    assert R.rel_l2(sf.to_host(out), R.fft_par("tensor", a, b, _pad(m))) <= TOL


@pytest.mark.parametrize("npts,m", [(19, 108), (24, 128), (9, 255), (19, 256), (8, 384), (5, 512)])
def test_bundle(npts, m):
    _check_bundle(npts, m)


@pytest.mark.parametrize("npts,m", [(19, 87), (24, 96), (19, 97), (16, 128), (11, 256), (5, 511)])
def test_tensor(npts, m):
    _check_tensor(npts, m)


@pytest.mark.parametrize("residues", [0, 3, 6, 12])
def test_residue_classes_in_point_chunks(residues):
    assert sf.lib().sfnl_test_large_residues(residues) == 0 and sf.lib().sfnl_test_large_workspace_cap(4 << 20) == 0
    try:
        _check_bundle(150, 256)
        _check_tensor(131, 256)
    finally:
        sf.lib().sfnl_test_large_residues(0)
        sf.lib().sfnl_test_large_workspace_cap(0)


@pytest.mark.parametrize("m", [112, 256])
def test_conservative_advection(m):
    torch = pytest.importorskip("torch")
    from sfemans_b200.profile_case import p2_rectangle

    mesh = p2_rectangle(3, 2)
    dmesh = {k: torch.from_numpy(np.ascontiguousarray(mesh[k].T)).cuda().permute(*range(mesh[k].ndim - 1, -1, -1))
             for k in ("jj", "ww", "dw", "rr")}
    modes = torch.arange(m, dtype=torch.int32, device="cuda")
    heat = torch.linspace(0.5, 2.0, mesh["me"], device="cuda", dtype=torch.float64)
    v, c = (sf.to_device(R.synthetic_field(mesh["np"], s, m, 0.05, 520 + s)) for s in (6, 2))
    kw = dict(heat=heat, conservative=True)
    g, w, d, hc = (sf.to_host(x) for x in sf.gauss_operands(sf.GAUSS_ADVECT, v, dmesh, modes, v2=c, **kw))
    out = sf.to_host(sf.ugradc_gauss(v, c, dmesh, modes, m_max_pad=_pad(m), **kw))
    assert R.rel_l2(out, R.fft_par("dot", g, w, _pad(m)) + R.fft_par("prod", d, hc, _pad(m))) <= TOL
