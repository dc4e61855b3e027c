"""Every kernel family on operands that start 8 bytes off a 16-byte boundary, at odd and even point counts, and with points
that are not finite.  Where the copies are made differently the arithmetic is the same, and points do not mix: both are
exact comparisons with the plain call."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# kind, modes: one-warp, class-split, third-fold and run-time kernels, residue grids of 64 and 128 angles, the caller's grid
PRODUCTS = [("cross", 8, sf.ALGO_FAST), ("svect", 16, sf.ALGO_FAST), ("prod", 30, sf.ALGO_FAST), ("dot", 24, sf.ALGO_FAST),
            ("dot", 32, sf.ALGO_FAST), ("tensor", 20, sf.ALGO_FAST), ("cross", 40, sf.ALGO_FAST), ("cross", 60, sf.ALGO_FAST),
            ("tensor", 72, sf.ALGO_FAST), ("cross", 72, sf.ALGO_FAST), ("svect", 200, sf.ALGO_FAST), ("dot", 300, sf.ALGO_FAST),
            ("cross", 20, sf.ALGO_GRID), ("prod", 33, sf.ALGO_GRID), ("tensor", 9, sf.ALGO_GRID), ("div", 20, sf.ALGO_AUTO),
            ("svdiv", 33, sf.ALGO_AUTO), ("tension", 12, sf.ALGO_AUTO), ("cross", 16, "split"), ("cross", 40, "split")]
LINEAR = {"cross_jvp": (2, 12), "cross_vjp": (2, 6), "mhd_jvp": (3, 18), "mhd_vjp": (3, 12)}
PROGRAMS = [("bundle", 20), ("bundle", 64), ("bundle", 72), ("cross_jvp", 66), ("cross_vjp", 20), ("cross_vjp", 60),
            ("mhd_jvp", 20), ("mhd_jvp", 64), ("mhd_vjp", 33), ("mhd_vjp", 72), ("mhd_jvp", 260)]


def _pad(m):
    return (3 * m + 1) // 2


def _inputs(kind, npts, m):
    if kind == "bundle":
        slots = [6] * 5
    elif kind in LINEAR:
        slots = [6] * LINEAR[kind][0] + [LINEAR[kind][1]]
    else:
        slots = list(sf.KINDS[kind][1:3])
    f = [R.synthetic_field(npts, s, m, 0.1, 10 * i + m) for i, s in enumerate(slots)]
    if kind in ("div", "svdiv"):
        f[1] *= 0.05
        f[1][:, 0, 0] = 3.0
    return [sf.to_device(x) for x in f]


def _run(kind, f, algo=None):
    m = f[0].shape[2]
    if kind == "bundle":
        out = sf.bundle_mhd(*f, m_max_pad=_pad(m))
    elif kind in LINEAR:
        out = getattr(sf, kind)(*f[:-1], f[-1][..., None], m_max_pad=_pad(m))
    else:
        kw = {"split": sf.SPLIT_BF16X3} if algo == "split" else {"algo": algo}
        out = sf.product(sf.KINDS[kind][0], *f, m_max_pad=_pad(m), **kw)
    return [sf.to_host(o) for o in (out if isinstance(out, tuple) else (out,))]


def _shifted(t):
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    return buf[1:].as_strided(t.shape, t.stride()).copy_(t)


CASES = [(k, m, a) for k, m, a in PRODUCTS] + [(k, m, None) for k, m in PROGRAMS]


@pytest.mark.parametrize("npts", [29, 40])
@pytest.mark.parametrize("kind,m,algo", CASES)
def test_operands_off_a_16_byte_boundary(kind, m, algo, npts):
    f = _inputs(kind, npts, m)
    want = _run(kind, f, algo)
    for moved in [set(range(len(f)))] + [{i} for i in range(len(f))]:
        got = _run(kind, [_shifted(x) if i in moved else x for i, x in enumerate(f)], algo)
        assert all(np.array_equal(g, w) for g, w in zip(got, want)), moved


@pytest.mark.parametrize("kind,m,algo", CASES)
def test_non_finite_points_stay_alone(kind, m, algo):
    npts, bad = 29, [3, 26]
    f = _inputs(kind, npts, m)
    want = _run(kind, f, algo)
    f[0][bad[0], 0, 1] = float("nan")
    f[-1][bad[1], 0, 2] = float("nan" if kind in ("div", "svdiv") else "inf")  # a quotient by infinity is zero
    keep = np.ones(npts, bool)
    keep[bad] = False
    for g, w in zip(_run(kind, f, algo), want):
        g, w = (np.moveaxis(x, 1, 0) if kind in ("tensor", "tension") else x for x in (g, w))
        assert np.array_equal(g[keep], w[keep])
    got = _run(kind, f, algo)
    hit = [any(not np.isfinite(np.moveaxis(g, 1, 0)[p] if kind in ("tensor", "tension") else g[p]).all() for g in got)
           for p in bad]
    assert all(hit)


@pytest.mark.parametrize("kind,m,algo", CASES + [("bundle", 128, None), ("bundle", 256, None), ("tensor", 256, None)])
def test_the_sine_of_mode_0_is_not_read(kind, m, algo):
    f = _inputs(kind, 21, m)
    algo = sf.ALGO_FAST if kind == "tensor" else algo
    want = _run(kind, f, algo)
    for x in f:
        x[:, 1::2, 0] = float("nan")
    assert all(np.array_equal(g, w) for g, w in zip(_run(kind, f, algo), want))


@pytest.mark.parametrize("npts", [29, 40])
@pytest.mark.parametrize("nslot,m", [(2, 20), (6, 33), (4, 9)])
def test_synthesis(nslot, m, npts):
    v = sf.to_device(R.synthetic_field(npts, nslot, m, 0.1, m))
    want, most = sf.to_host(sf.synthesis(v)), sf.max_vel(v, _pad(m))
    assert np.array_equal(sf.to_host(sf.synthesis(_shifted(v))), want) and sf.max_vel(_shifted(v), _pad(m)) == most
    v[3, 0, 1] = float("nan")
    got = sf.to_host(sf.synthesis(v))
    keep = np.arange(npts) != 3
    assert np.array_equal(got[..., keep], want[..., keep]) and not np.isfinite(got[:, 0, 3]).all()


@pytest.mark.parametrize("m", [17, 33, 64])
def test_split_programs_over_many_tiles(m):
    # tiles of 8 points, more of them than CTAs: the next tile's operands are written during a tile's last analysis
    npts, pad = 2501, _pad(m)
    f = [R.synthetic_field(npts, 6, m, 0.3, 40 + i) for i in range(5)]
    d = [sf.to_device(x) for x in f]
    refs = R.mhd_bundle(*f, pad, engine=lambda op, x, y: R.fft_par(op, x, y, pad))
    for split, bar in ((sf.SPLIT_BF16X3, 1e-7), (sf.SPLIT_BF16X2, 1e-4)):  # the bars of the two split forms
        for o, r in zip(sf.bundle_mhd(*d, m_max_pad=pad, split=split), refs):
            assert R.rel_l2(sf.to_host(o), r) <= bar
    for kind, nslot in (("mhd_jvp", 18), ("mhd_vjp", 12)):
        x = sf.to_device(R.synthetic_field(npts, nslot, m, 0.3, 60 + nslot)[..., None])
        want = sf.to_host(getattr(sf, kind)(*d[:3], x, m_max_pad=pad))
        assert R.rel_l2(sf.to_host(getattr(sf, kind)(*d[:3], x, m_max_pad=pad, split=sf.SPLIT_BF16X3)), want) <= 1e-7
