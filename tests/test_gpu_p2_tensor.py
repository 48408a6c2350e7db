"""Leaf and node hashing with the partial rounds on the tensor cores (from 2^18 leaves or nodes on),
against the oracle: partial tiles, rows per leaf, checkpoints, installed round constants, commitments
alone and in a batch, calls that follow the installation of their tables at once."""
import numpy as np
import pytest

from conftest import load_package, rand_elems
from gpu_util import from_dev, to_dev, zeros_dev

pytestmark = pytest.mark.gpu
N = 1 << 18


@pytest.fixture(scope="module")
def glc(round_constants):
    g = load_package()
    ctx = g.Context.create()
    g.poseidon2.set_round_constants(round_constants)
    yield g
    ctx.destroy()


@pytest.mark.parametrize("count", [N - 1, N, N + 1, 2 * N + 77])
@pytest.mark.parametrize("cols,log_rows", [(1, 0), (8, 0), (11, 0), (3, 2)])
def test_leaves(glc, oracle, count, cols, log_rows):
    x = rand_elems((cols * count) << log_rows, count + cols, noncanonical=True)
    out = zeros_dev(4 * count)
    glc.GLHasher.compute_leaf_hashes(to_dev(x), out, log_rows, False, False)
    assert (from_dev(out) == oracle.leaves(x, 4 * count, log_rows)).all()
    assert glc.commit.fused_timeouts() == 0


def test_checkpointed_leaves(glc, oracle):
    count = N + 130
    x = rand_elems(13 * count, 4, noncanonical=True)
    out = zeros_dev(4 * count)
    glc.GLHasher.compute_leaf_hashes(to_dev(x[:8 * count]), out, 0, False, True)
    glc.GLHasher.compute_leaf_hashes(to_dev(x[8 * count:]), out, 0, True, False)
    assert (from_dev(out) == oracle.leaves(x, 4 * count)).all()


@pytest.mark.parametrize("count,shift", [(N, 0), (N + 5, 0), (2 * N, 1)])
def test_nodes(glc, oracle, count, shift):
    x = rand_elems(8 * count, count, noncanonical=True)
    d = to_dev(np.concatenate([np.zeros(shift, dtype=np.uint64), x]))
    out = zeros_dev(4 * count)
    glc.GLHasher.compute_node_hashes(d[shift:], out)
    assert (from_dev(out) == oracle.nodes(x)).all()


def test_installed_constants(glc, oracle, round_constants):
    other = [int(v) for v in rand_elems(360, 9)]
    x = rand_elems(16 * N, 8)
    out = zeros_dev(4 * N)
    try:
        glc.poseidon2.set_round_constants(other)
        oracle.set_round_constants(other)
        glc.GLHasher.compute_leaf_hashes(to_dev(x), out, 0, False, False)
        assert (from_dev(out) == oracle.leaves(x, 4 * N)).all()
    finally:
        glc.poseidon2.set_round_constants(round_constants)
        oracle.set_round_constants(round_constants)


def test_tables_are_there_when_the_call_returns(glc, oracle, round_constants):
    """Work enqueued at once on a non-blocking stream, which waits for no copy that is still under way."""
    import torch
    x, y = rand_elems(8 * N, 3), rand_elems(N, 4)
    d, side = to_dev(x), torch.cuda.Stream()
    out, ntt = zeros_dev(4 * N), zeros_dev(4 * N)
    want = oracle.batch_ntt(y, 18, 1, N, N, 0, 1, 0, 0)
    try:
        for seed in range(3):
            other = [int(v) for v in rand_elems(360, 20 + seed)]
            oracle.set_round_constants(other)
            ntt.copy_(to_dev(np.tile(y, 4)))
            torch.cuda.synchronize()
            glc.Context.create()
            with torch.cuda.stream(side):
                glc.ntt.batch_ntt_in_place(ntt, 18, 4, 0, N, False, True, 0, 0)
            glc.poseidon2.set_round_constants(other)
            with torch.cuda.stream(side):
                glc.GLHasher.compute_node_hashes(d, out)
            side.synchronize()
            assert (from_dev(out) == oracle.nodes(x)).all()
            assert (from_dev(ntt).reshape(4, N) == want).all()
    finally:
        glc.poseidon2.set_round_constants(round_constants)
        oracle.set_round_constants(round_constants)


@pytest.mark.parametrize("log_n,cols", [(11, 8), (12, 9), (13, 3), (18, 9)])
def test_commitment_alone_and_in_a_batch(glc, oracle, log_n, cols):
    """The leaves' form follows what hashes beside them: nothing, the other coset, other jobs."""
    log_lde, log_cap = 1, 4
    ev = rand_elems(cols << log_n, 5)
    _, lde, trees, cap = oracle.commit(ev, log_n, cols, log_lde, log_cap)
    sz = glc.CommitJob.sizes(log_n, cols, log_lde, log_cap)
    jobs = [glc.CommitJob(to_dev(ev), log_n, cols, log_lde, log_cap, zeros_dev(sz["lde"]), zeros_dev(sz["trees"]),
                          zeros_dev(sz["cap"])) for _ in range(6)]
    glc.commit.commit(jobs[0])
    glc.commit.commit_batch(jobs[1:2])
    glc.commit.commit_batch(jobs[2:4])
    glc.commit.commit_batch(jobs[4:], n_streams=1)
    for j in jobs:
        assert (from_dev(j.cap) == cap).all()
        assert (from_dev(j.trees) == trees).all()
        assert (from_dev(j.lde) == lde).all()
