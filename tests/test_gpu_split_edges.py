"""The split kernel at the bounds of its register classes (8, 16, 32 modes per class: m = 16 | 17, 32 | 33), its
second k-step (the even classes only at m = 33) and its chunk counts, with more tiles than resident CTAs so that a
CTA prepares its next tile while the last chunk of the current one is analysed.  Bars of the split forms: rel-L2
<= 1e-7 with three slices, <= 1e-4 with two."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu


def _call(kind, V1, V2, split):
    m = V1.shape[2]
    return sf.to_host(sf.product(sf.KINDS[kind][0], sf.to_device(V1), sf.to_device(V2), m_max_pad=max(1, 3 * m // 2),
                                 split=split))


@pytest.mark.parametrize("kind", ["cross", "svect", "prod"])
@pytest.mark.parametrize("npts,m", [(15, 4), (4753, 16), (2407, 17), (2393, 22), (17, 23), (2407, 32), (4801, 33),
                                    (2383, 43), (33, 44), (2399, 64)])
def test_split_products_at_class_bounds(kind, npts, m):
    _, n1, n2, _ = sf.KINDS[kind]
    V1, V2 = R.synthetic_field(npts, n1, m, 0.3, 31 + m), R.synthetic_field(npts, n2, m, 0.3, 32 + m)
    ref = R.fft_par(kind, V1, V2, max(1, 3 * m // 2))
    assert R.rel_l2(_call(kind, V1, V2, sf.SPLIT_BF16X3), ref) <= 1e-7
    assert R.rel_l2(_call(kind, V1, V2, sf.SPLIT_BF16X2), ref) <= 1e-4


@pytest.mark.parametrize("m", [16, 64])
def test_a_non_finite_point_stays_alone(m):
    npts = 40
    V1, V2 = R.synthetic_field(npts, 6, m, 0.3, 1), R.synthetic_field(npts, 6, m, 0.3, 2)
    good = _call("cross", V1, V2, sf.SPLIT_BF16X3)
    V1[7, 2, 1], V1[23, 0, 3] = np.nan, np.inf
    got = _call("cross", V1, V2, sf.SPLIT_BF16X3)
    keep = np.ones(npts, bool)
    keep[[7, 23]] = False
    assert np.array_equal(got[keep], good[keep])
    assert not np.isfinite(got[7]).all() and not np.isfinite(got[23]).all()
