"""The tiled kernels of the caller's grid (GRID products, synthesis, maxima) at the edges of their tiles: point
counts around the 8- and 16-point tiles, odd counts (8-byte copies), modes around the k-steps of 4 and the output
tiles of 8, grids of odd and even length (an even one has a second angle that is its own mirror), and sizes on both
sides of the shared-memory limit beyond which the one-warp-per-point kernel runs.  Compared with dense Fourier sums
in numpy's long double; rel-L2 <= 1e-12, the bar of the FP64 forms (the divisor stays away from zero)."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _values(V, N):
    """(np, ncomp, N) long-double values at 2 pi j / N."""
    m = V.shape[2]
    th = 2 * np.pi * np.longdouble(1) * (np.outer(np.arange(m), np.arange(N)) % N) / N
    a, b = V[:, 0::2].astype(np.longdouble), V[:, 1::2].astype(np.longdouble).copy()
    b[:, :, 0] = 0
    return a @ np.cos(th) + b @ np.sin(th)


def _analyse(f, m):
    N = f.shape[-1]
    th = 2 * np.pi * np.longdouble(1) * (np.outer(np.arange(N), np.arange(m)) % N) / N
    w = np.full(m, np.longdouble(2) / N)
    w[0] = np.longdouble(1) / N
    out = np.zeros((f.shape[0], 2 * f.shape[1], m))
    out[:, 0::2] = (f @ np.cos(th)) * w
    out[:, 1::2] = (f @ np.sin(th)) * w
    return out


def _field(npts, nslot, m, seed):
    v = R.synthetic_field(npts, nslot, m, 0.3, seed)
    return 0.1 * v


GRID_CASES = [(1, 1, 1), (7, 3, 8), (8, 4, 11), (9, 5, 14), (16, 8, 23), (17, 9, 26), (31, 31, 95), (33, 33, 98),
              (15, 64, 191), (10, 96, 287), (6, 160, 479), (4, 220, 659)]


@pytest.mark.parametrize("npts,m,N", GRID_CASES)
@pytest.mark.parametrize("kind", ["cross", "svdiv", "div", "tension"])
def test_grid_products_at_tile_edges(kind, npts, m, N):
    if kind == "tension" and m > 160:
        pytest.skip("beyond the shared memory of every GRID kernel")
    op, n1, n2, _ = sf.KINDS[kind]
    V1, V2 = _field(npts, n1, m, 11 + m), _field(npts, n2, m, 12 + m)
    V2[:, 0::2, 0] += 3.0  # positive on the whole circle
    x, y = _values(V1, N), _values(V2, N)
    if kind == "cross":
        ref = _analyse(np.stack([x[:, 1] * y[:, 2] - x[:, 2] * y[:, 1], x[:, 2] * y[:, 0] - x[:, 0] * y[:, 2],
                                 x[:, 0] * y[:, 1] - x[:, 1] * y[:, 0]], 1), m)
    elif kind == "tension":
        nrm = np.sqrt((y ** 2).sum(1))
        ref = np.stack([_analyse(x[:, k:k + 1] * y / (nrm + 1e-14)[:, None] - np.eye(3)[k][None, :, None] * nrm[:, None], m)
                        for k in range(3)])
    else:
        ref = _analyse(x / y, m)
    out = sf.to_host(sf.product(op, sf.to_device(V1), sf.to_device(V2), m_max_pad=max(m, (N + 1) // 2), n_theta=N,
                                algo=sf.ALGO_GRID))
    assert R.rel_l2(out, ref.astype(np.float64)) <= TOL


@pytest.mark.parametrize("nslot", [2, 4, 6, 12])
@pytest.mark.parametrize("npts,m,N", [(1, 1, 1), (7, 3, 5), (8, 4, 8), (9, 5, 14), (17, 9, 26), (33, 33, 65),
                                      (66, 64, 190), (5, 130, 259), (3, 300, 2001)])
def test_synthesis_and_maximum_at_tile_edges(npts, m, N, nslot):
    V = _field(npts, nslot, m, 5 + m)
    f = _values(V, N)
    got = sf.to_host(sf.synthesis(sf.to_device(V), n_theta=N))
    assert R.rel_l2(got, f.transpose(2, 1, 0).astype(np.float64)) <= TOL
    pad = 3 * m // 2 + 1
    f = _values(V, 2 * pad - 1)[:, :3 if nslot == 6 else 1]
    ref = float(np.sqrt((f ** 2).sum(1)).max())
    assert abs(sf.max_vel(sf.to_device(V), pad) - ref) <= TOL * ref
