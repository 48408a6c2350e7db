"""The NTT passes on the tensor cores against the oracle: every split of the stages into rounds,
column groups with remainders, in place and out of place, offsets and strides that forbid the wide
stores, at and just above the sizes from which batches take this path, and on both sides of those between
which 2^16 and 2^17 rows leave it."""
import numpy as np
import pytest

from conftest import canon, load_package, rand_elems
from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def glc():
    g = load_package()
    ctx = g.Context.create()
    yield g
    ctx.destroy()


@pytest.mark.parametrize("log_n,cols", [(12, 256), (12, 513), (12, 5000), (16, 16), (16, 19), (16, 20), (16, 21),
                                        (16, 26), (16, 27), (16, 67), (17, 8), (17, 9), (17, 10), (17, 11), (17, 13),
                                        (17, 14), (17, 16), (18, 8), (19, 5), (20, 2), (21, 1), (22, 1), (23, 1), (23, 2)])
@pytest.mark.parametrize("bitrev,inverse,log_ext,coset", [(False, False, 0, 0), (False, True, 0, 0), (True, False, 0, 0),
                                                          (True, True, 0, 0), (False, False, 3, 5)])
def test_against_oracle(glc, oracle, log_n, cols, bitrev, inverse, log_ext, coset):
    n = 1 << log_n
    # 12 x 513: odd offset and stride; 16 x 67: even, not a multiple of 4
    off, gap = {(12, 513): (1, 3), (16, 67): (2, 6), (18, 8): (3, 4)}.get((log_n, cols), (0, 0))
    stride = n + gap
    x = rand_elems(cols * stride, log_n * 1000 + cols, noncanonical=True)
    want = np.full(cols * stride, 7, dtype=np.uint64)
    packed = np.ascontiguousarray(x.reshape(cols, stride)[:, off:off + n])
    want.reshape(cols, stride)[:, off:off + n] = oracle.batch_ntt(packed.reshape(-1), log_n, cols, n, n, int(bitrev),
                                                                  int(inverse), log_ext, coset).reshape(cols, n)
    src, out = to_dev(x), to_dev(np.full(cols * stride, 7, dtype=np.uint64))
    glc.ntt.batch_ntt_out_of_place(src, out, log_n, cols, off, off, stride, stride, bitrev, inverse, log_ext, coset)
    assert (from_dev(src) == x).all()
    assert (from_dev(out) == want).all()
    glc.ntt.batch_ntt_in_place(src, log_n, cols, off, stride, bitrev, inverse, log_ext, coset)
    got = from_dev(src).reshape(cols, stride)
    assert (got[:, off:off + n] == want.reshape(cols, stride)[:, off:off + n]).all()
    assert (got[:, :off] == x.reshape(cols, stride)[:, :off]).all()
    assert (got[:, off + n:] == x.reshape(cols, stride)[:, off + n:]).all()
    assert glc.commit.fused_timeouts() == 0


@pytest.mark.parametrize("bitrev,inverse,log_ext,coset", [(False, False, 0, 0), (False, True, 0, 0), (True, False, 0, 0),
                                                          (True, True, 0, 0), (False, False, 3, 5)])
def test_largest_rows(glc, oracle, bitrev, inverse, log_ext, coset):
    """2^24 rows, whose strided tiles hold one element a row: 17 columns, each against the same column alone,
    which the register passes transform, and one against the oracle."""
    import torch
    torch.cuda.empty_cache()
    n, cols = 1 << 24, 17
    x = torch.randint(-(2**63), 2**63 - 1, (cols, n), device="cuda", generator=torch.Generator("cuda").manual_seed(24))
    out, one = torch.zeros_like(x), torch.zeros(n, dtype=torch.int64, device="cuda")
    glc.ntt.batch_ntt_out_of_place(x, out, 24, cols, 0, 0, n, n, bitrev, inverse, log_ext, coset)
    for c in range(cols):
        glc.ntt.batch_ntt_out_of_place(x[c], one, 24, 1, 0, 0, n, n, bitrev, inverse, log_ext, coset)
        assert torch.equal(out[c], one), c
    want = oracle.batch_ntt(from_dev(x[16]), 24, 1, n, n, int(bitrev), int(inverse), log_ext, coset)
    assert (from_dev(out[16]) == want).all()
    glc.ntt.batch_ntt_in_place(x, 24, cols, 0, n, bitrev, inverse, log_ext, coset)
    assert torch.equal(x, out)
    assert glc.commit.fused_timeouts() == 0


def test_column_groups_past_the_grid(glc, oracle):
    """More column groups than one launch's grid holds (65535 groups of 16 columns)."""
    cols, n = 16 * 65535 + 35, 1 << 12
    import torch
    torch.cuda.empty_cache()  # what other tests' tensors left cached
    free, _ = torch.cuda.mem_get_info()
    if free < 9 * cols * n:
        pytest.skip("needs %d GB" % (9 * cols * n >> 30))
    x = torch.randint(0, 2**62, (cols, n), device="cuda")
    keep = [0, 15, 16, 16 * 65535 - 1, 16 * 65535, cols - 1]
    before = x[keep].cpu().numpy().view(np.uint64)
    glc.ntt.batch_ntt_in_place(x, 12, cols, 0, n, False, True, 0, 0)
    got = x[keep].cpu().numpy().view(np.uint64)
    want = oracle.batch_ntt(np.ascontiguousarray(before).reshape(-1), 12, len(keep), n, n, 0, 1, 0, 0)
    assert (canon(got.reshape(-1)) == want).all()
