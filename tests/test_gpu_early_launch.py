"""Small launches may begin before the previous kernel of their stream has ended (they wait for it
inside): chains of dependent calls, with other kernels between them, on a side stream and replayed
from a captured graph, give what the calls one at a time give.  Launches of 74, 148 and more CTAs, and
transforms of which one pass is small enough to begin early and the other is not."""
import numpy as np
import pytest

from conftest import load_package, rand_elems
from gpu_util import from_dev, to_dev, torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def glc():
    g = load_package()
    ctx = g.Context.create()
    yield g
    ctx.destroy()


def chain(glc, d, log_n, cols, n, other=False):
    """Forward on a coset, bit reversal twice, back: the input again; `other` adds 0 between the calls."""
    for _ in range(10):
        glc.ntt.batch_ntt_in_place(d, log_n, cols, 0, n, False, False, 1, 1)
        if other:
            d.add_(0)
        glc.ops_complex.bit_reverse_in_place(d, n, cols)
        glc.ops_complex.bit_reverse_in_place(d, n, cols)
        if other:
            d.add_(0)
        glc.ntt.batch_ntt_in_place(d, log_n, cols, 0, n, True, True, 1, 1)


@pytest.mark.parametrize("log_n,cols", [(1, 1), (9, 3), (10, 5), (10, 148), (10, 149), (13, 2), (13, 8), (16, 1), (16, 2),
                                        (17, 1), (17, 2)])
def test_chains(glc, oracle, log_n, cols):
    T = torch()
    n = 1 << log_n
    x = rand_elems(cols * n, log_n)
    for other in (False, True):
        d = to_dev(x)
        chain(glc, d, log_n, cols, n, other)
        assert (from_dev(d) == x).all()
    side = T.cuda.Stream()
    d = to_dev(x)
    side.wait_stream(T.cuda.current_stream())
    with T.cuda.stream(side):
        chain(glc, d, log_n, cols, n)
        idx = T.arange(n - 1, -1, -1, dtype=T.int32, device="cuda")
        rows = T.zeros(cols * n, dtype=T.int64, device="cuda")
        glc.GLHasher.gather_rows(idx, 0, d, n, cols, rows, n, cols)
    side.synchronize()
    assert (from_dev(d) == x).all()
    assert (from_dev(rows).reshape(cols, n) == x.reshape(cols, n)[:, ::-1]).all()
    graph = T.cuda.CUDAGraph()
    with T.cuda.graph(graph):
        chain(glc, d, log_n, cols, n)
        glc.ntt.batch_ntt_in_place(d, log_n, cols, 0, n, False, False, 0, 0)
    want = x
    for _ in range(3):
        graph.replay()
        want = oracle.batch_ntt(np.ascontiguousarray(want), log_n, cols, n, n, 0, 0, 0, 0)
    assert (from_dev(d) == want).all()
