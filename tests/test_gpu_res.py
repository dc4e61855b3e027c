"""The FAST form on residue grids (m = 65 .. 512) at the bounds of its residue counts and grid lengths: 64 angles up to
m = 256, 128 beyond; each number of residues from both; mode counts that fill the last residue block or leave it nearly
empty; point counts that are no multiple of the 8-point tiles; and a small workspace, which splits points and batch
entries into several chunks.  Against pocketfft products; rel-L2 <= 1e-12, the bar of the FP64 forms."""
import numpy as np
import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu
TOL = 1e-12
SIZES = [65, 72, 73, 86, 87, 107, 108, 128, 129, 150, 171, 192, 200, 214, 235, 256, 257, 299, 300, 384, 385, 470, 512]


def _pad(m):
    return (3 * m + 1) // 2


def _field(npts, nslot, m, seed):
    return R.synthetic_field(npts, nslot, m, 0.05, seed)


@pytest.mark.parametrize("m", SIZES)
@pytest.mark.parametrize("kind", ["cross", "dot", "prod", "svect"])
def test_products(kind, m):
    _, n1, n2, _ = sf.KINDS[kind]
    for npts in (5, 16):
        V1, V2 = _field(npts, n1, m, 21 + m), _field(npts, n2, m, 22 + m)
        out = sf.product(sf.KINDS[kind][0], sf.to_device(V1), sf.to_device(V2), m_max_pad=_pad(m), algo=sf.ALGO_FAST)
        assert R.rel_l2(sf.to_host(out), R.fft_par(kind, V1, V2, _pad(m))) <= TOL


@pytest.mark.parametrize("cap", [0, 1 << 20])
@pytest.mark.parametrize("m", [65, 73, 129, 200, 256, 257, 400])
def test_linearised_programs(m, cap):
    npts, k = 21, 3
    cross = lambda x, y: R.fft_par("cross", np.asfortranarray(x), np.asfortranarray(y), _pad(m))  # noqa: E731
    u, w, b = (_field(npts, 6, m, 31 + i) for i in range(3))
    v = np.asfortranarray(np.stack([_field(npts, 18, m, 41 + i) for i in range(k)], -1))
    c = np.asfortranarray(np.stack([_field(npts, 12, m, 51 + i) for i in range(k)], -1))
    base = [sf.to_device(x) for x in (u, w, b)]
    v12, c1 = np.asfortranarray(v[:, :12]), np.asfortranarray(c[:, :6])
    assert sf.lib().sfnl_test_large_workspace_cap(cap) == 0
    try:
        jv, jc = (sf.to_host(f(*base, sf.to_device(x), m_max_pad=_pad(m))) for f, x in ((sf.mhd_jvp, v), (sf.mhd_vjp, c)))
        jv1 = sf.to_host(sf.cross_jvp(*base[:2], sf.to_device(v12), m_max_pad=_pad(m)))
        jc1 = sf.to_host(sf.cross_vjp(*base[:2], sf.to_device(c1), m_max_pad=_pad(m)))
    finally:
        sf.lib().sfnl_test_large_workspace_cap(0)
    for t in range(k):
        du, dw, db = (v[:, 6 * i:6 * i + 6, :, t] for i in range(3))
        ref1 = cross(du, w) + cross(u, dw)
        ref = np.concatenate([ref1, cross(du, b) + cross(u, db)], 1)
        assert R.rel_l2(jv[..., t], ref) <= TOL and R.rel_l2(jv1[..., t], ref1) <= TOL
        scale = np.linalg.norm(ref) * np.linalg.norm(c[..., t])
        assert abs(float((ref * c[..., t]).sum() - (v[..., t] * jc[..., t]).sum())) <= TOL * scale
        assert abs(float((ref1 * c1[..., t]).sum() - (v12[..., t] * jc1[..., t]).sum())) <= TOL * scale


@pytest.mark.parametrize("m", [72, 96])
def test_captured_calls_without_a_workspace(m):
    # a graph is captured on a stream that has no workspace yet: sizes that the fused kernels hold run on them
    torch = pytest.importorskip("torch")
    npts = 19
    f = [_field(npts, 6, m, 61 + i) for i in range(3)]
    c = _field(npts, 12, m, 71)
    u, w, b, cd = (sf.to_device(x) for x in (*f, c))
    eager = sf.product(sf.OP_CROSS, u, w, m_max_pad=_pad(m)), sf.mhd_vjp(u, w, b, cd, m_max_pad=_pad(m))
    outs = [torch.zeros_like(x) for x in eager]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        sf.product(sf.OP_CROSS, u, w, out=outs[0], m_max_pad=_pad(m))
        sf.mhd_vjp(u, w, b, cd, out=outs[1], m_max_pad=_pad(m))
    g.replay()
    torch.cuda.synchronize()
    for o, e in zip(outs, eager):
        assert R.rel_l2(sf.to_host(o), sf.to_host(e)) <= TOL


def test_a_workspace_leaves_memory_to_the_caller():
    # with 4 GiB free the buffer may take a quarter: at m = 72 the fused kernels run instead, at m = 200 shorter chunks
    torch = pytest.importorskip("torch")
    G = 1 << 30
    u, w, b = (sf.to_device(_field(7000, 6, 72, 81 + i)) for i in range(3))
    cot = sf.to_device(np.stack([_field(7000, 12, 72, 85 + i) for i in range(4)], -1))
    x, y = (sf.to_device(_field(30_000, 6, 200, 91 + i)) for i in range(2))
    calls = [lambda out: sf.mhd_vjp(u, w, b, cot, m_max_pad=_pad(72), out=out),
             lambda out: sf.product(sf.OP_CROSS, x, y, m_max_pad=_pad(200), out=out)]
    outs = [sf.fortran_empty(7000, 18, 72, 4), sf.fortran_empty(30_000, 6, 200)]
    wants = [f(torch.empty_like(o)) for f, o in zip(calls, outs)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    sf.lib().sfnl_finalize()
    for f, o in zip(calls, outs):  # tables and kernels are loaded; small calls, small buffers
        f(o)
    torch.cuda.synchronize()
    sf.lib().sfnl_finalize()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - 4 * G, dtype=torch.uint8, device="cuda")
    for f, o, w_, most in zip(calls, outs, wants, (G // 8, G + G // 8)):  # tables of a few MB beside the buffer
        before = torch.cuda.mem_get_info()[0]
        f(o.zero_())
        torch.cuda.synchronize()
        assert before - torch.cuda.mem_get_info()[0] <= most
        assert float((o - w_).norm() / w_.norm()) <= TOL
    del filler


@pytest.mark.parametrize("kind,nbase,nin,nout,launches", [("cross_jvp", 2, 12, 6, (1, 2)), ("cross_vjp", 2, 6, 12, (2, 2)),
                                                          ("mhd_jvp", 3, 18, 12, (2, 4)), ("mhd_vjp", 3, 12, 18, (3, 4))])
@pytest.mark.parametrize("m", [73, 86, 87, 107])
def test_captured_linearised_programs(m, kind, nbase, nin, nout, launches):
    # to m = 86 a sum of two cross products is one launch of a captured call, beyond two
    torch = pytest.importorskip("torch")
    cudart = pytest.importorskip("cuda.bindings.runtime")
    npts, k = 13, 2
    f = [sf.to_device(_field(npts, 6, m, 61 + i)) for i in range(nbase)]
    x = sf.to_device(np.stack([_field(npts, nin, m, 71 + i) for i in range(k)], -1))
    call = lambda out: getattr(sf, kind)(*f, x, m_max_pad=_pad(m), out=out)  # noqa: E731
    want, out = call(sf.fortran_empty(npts, nout, m, k)), sf.fortran_empty(npts, nout, m, k)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call(out)
    err, _, count = cudart.cudaGraphGetNodes(g.raw_cuda_graph(), 0)
    assert int(err) == 0 and count == launches[m > 86]
    g.instantiate()
    g.replay()
    torch.cuda.synchronize()
    assert R.rel_l2(sf.to_host(out), sf.to_host(want)) <= TOL


@pytest.mark.parametrize("kind", ["cross", "bundle"])
def test_a_graph_keeps_its_buffer(kind):
    # captured after a call of its size; a larger call on the same stream grows the stream's buffer before the replay
    torch = pytest.importorskip("torch")
    m, st = 128, torch.cuda.Stream()

    def problem(npts):
        f = [sf.to_device(_field(npts, 6, m, 31 + i)) for i in range(2 if kind == "cross" else 5)]
        outs = [sf.fortran_empty(npts, s, m) for s in ((6,) if kind == "cross" else (6, 6, 6, 2))]
        if kind == "cross":
            return lambda: sf.product(sf.OP_CROSS, *f, out=outs[0], m_max_pad=_pad(m)), outs
        return lambda: sf.bundle_mhd(*f, m_max_pad=_pad(m), outs=tuple(outs)), outs

    (small, outs), (large, _) = problem(40), problem(5000)
    torch.cuda.synchronize()
    sf.lib().sfnl_finalize()
    with torch.cuda.stream(st):
        small()
    torch.cuda.synchronize()
    wants = [o.clone() for o in outs]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        small()
    with torch.cuda.stream(st):
        large()
    torch.cuda.synchronize()
    for _ in range(3):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            g.replay()
            large()
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o, w in zip(outs, wants))
