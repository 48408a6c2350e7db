"""Leaf and node hashing with the partial rounds on the tensor cores (from 2^18 leaves or nodes on),
against the oracle: partial tiles, rows per leaf, checkpoints, installed round constants, commitments
alone and in a batch."""
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


def test_commitment_alone_and_in_a_batch(glc, oracle):
    log_n, cols, log_lde, log_cap = 18, 9, 1, 4
    ev = rand_elems(cols << log_n, 5)
    _, lde, trees, cap = oracle.commit(ev, log_n, cols, log_lde, log_cap)
    sz = glc.CommitJob.sizes(log_n, cols, log_lde, log_cap)
    jobs = [glc.CommitJob(to_dev(ev), log_n, cols, log_lde, log_cap, zeros_dev(sz["lde"]), zeros_dev(sz["trees"]),
                          zeros_dev(sz["cap"])) for _ in range(3)]
    glc.commit.commit(jobs[0])
    glc.commit.commit_batch(jobs[1:])
    for j in jobs:
        assert (from_dev(j.cap) == cap).all()
        assert (from_dev(j.trees) == trees).all()
        assert (from_dev(j.lde) == lde).all()
