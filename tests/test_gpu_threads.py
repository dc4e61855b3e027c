"""Entry points from several host threads at once: on one stream, and on cudaStreamPerThread, one handle that names
another stream in every thread.  From m = 65 a call takes several launches through a workspace of its stream.  Every
result has to be the one that the call gives alone, bit for bit."""
import threading

import pytest

import sfemans_b200 as sf
from oracle import ref_fft as R

pytestmark = pytest.mark.gpu
PER_THREAD = 2  # the value of cudaStreamPerThread
CALLS = 150


def _problem(kind, npts, m, seed):
    """A call into a given output on a given stream, its own result, and outputs for CALLS calls."""
    torch = pytest.importorskip("torch")
    pad = (3 * m + 1) // 2
    if kind == "cross":
        a, b = (sf.to_device(R.synthetic_field(npts, 6, m, 0.05, seed + i)) for i in range(2))
        call = lambda out, st: sf.product(sf.OP_CROSS, a, b, out=out, m_max_pad=pad, stream=st)  # noqa: E731
        shape = (npts, 6, m)
    elif kind == "bundle":
        f = [sf.to_device(R.synthetic_field(npts, 6, m, 0.05, seed + i)) for i in range(5)]
        rest = [sf.fortran_empty(npts, s, m) for s in (6, 6, 2)]
        call = lambda out, st: sf.bundle_mhd(*f, m_max_pad=pad, outs=(out, *rest), stream=st)[0]  # noqa: E731
        shape = (npts, 6, m)
    else:
        f = [sf.to_device(R.synthetic_field(npts, s, m, 0.05, seed + i)) for i, s in enumerate((6, 6, 6, 12))]
        call = lambda out, st: sf.mhd_vjp(*f, m_max_pad=pad, out=out, stream=st)  # noqa: E731
        shape = (npts, 18, m)
    want = call(sf.fortran_empty(*shape), 0)
    outs = [sf.fortran_empty(*shape) for _ in range(CALLS)]
    torch.cuda.synchronize()
    return call, want, outs


@pytest.mark.parametrize("stream", [0, PER_THREAD])
@pytest.mark.parametrize("first,second", [(("cross", 301, 72), ("cross", 777, 72)), (("cross", 301, 72), ("mhd_vjp", 205, 200)),
                                          (("mhd_vjp", 150, 96), ("cross", 1201, 200)), (("bundle", 150, 128), ("bundle", 410, 128))])
def test_two_threads(stream, first, second):
    torch = pytest.importorskip("torch")
    problems = [_problem(*p, 11 + 100 * i) for i, p in enumerate((first, second))]
    sf.lib().sfnl_finalize()  # the buffers of both threads are allocated, and grown, side by side
    start, errors = threading.Barrier(2), []

    def work(call, outs):
        try:
            start.wait()
            for out in outs:
                call(out, stream)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(call, outs)) for call, _, outs in problems]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    for _, want, outs in problems:
        assert all(torch.equal(out, want) for out in outs)


@pytest.mark.parametrize("legacy", [False, True])
@pytest.mark.parametrize("m", [72, 200])
def test_a_capture_in_another_thread_goes_on(m, legacy):
    # a first and a growing call allocate their workspace while another thread captures a graph on its own stream
    torch = pytest.importorskip("torch")
    pad, sizes = (3 * m + 1) // 2, (150, 900)
    f = [[sf.to_device(R.synthetic_field(n, 6, m, 0.05, 7 + i)) for i in range(2)] for n in sizes]
    wants = [sf.product(sf.OP_CROSS, *ab, m_max_pad=pad, stream=0) for ab in f]
    outs, side, errors = [torch.empty_like(w) for w in wants], 0 if legacy else torch.cuda.Stream(), []
    x = torch.ones(64, device="cuda")
    torch.cuda.synchronize()

    def work():
        try:
            for (a, b), out in zip(f, outs):
                sf.product(sf.OP_CROSS, a, b, out=out, m_max_pad=pad, stream=side)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.mul_(2.0)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        x.add_(1.0)
    g.replay()
    torch.cuda.synchronize()
    assert not errors and bool((x == 3.0).all())
    assert all(torch.equal(o, w) for o, w in zip(outs, wants))


def test_a_new_stream_with_an_old_handle():
    # streams made and destroyed one after the other, their work still pending, mostly share one handle
    torch = pytest.importorskip("torch")
    cudart = pytest.importorskip("cuda.bindings.runtime")
    (a, b), (c, d) = ([sf.to_device(R.synthetic_field(n, 6, 72, 0.05, n + i)) for i in range(2)] for n in (4000, 700))
    wants = [sf.product(sf.OP_CROSS, x, y, m_max_pad=108, stream=0) for x, y in ((a, b), (c, d))]
    outs = [[torch.empty_like(w) for _ in range(20)] for w in wants]
    torch.cuda.synchronize()
    for pair in zip(*outs):
        for (x, y), out in zip(((a, b), (c, d)), pair):
            err, st = cudart.cudaStreamCreateWithFlags(1)  # not blocking
            assert int(err) == 0
            sf.product(sf.OP_CROSS, x, y, out=out, m_max_pad=108, stream=int(st))
            assert int(cudart.cudaStreamDestroy(st)[0]) == 0
    torch.cuda.synchronize()
    for want, group in zip(wants, outs):
        assert all(torch.equal(out, want) for out in group)
