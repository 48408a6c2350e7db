"""Leaf and node hashing around the counts where the lanes per permutation change (2048 and 8192),
with partial warps and CTAs, against the oracle."""
import numpy as np
import pytest

from conftest import load_package, rand_elems
from gpu_util import from_dev, to_dev, zeros_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def glc():
    g = load_package()
    ctx = g.Context.create()
    yield g
    ctx.destroy()


@pytest.mark.parametrize("count", [1, 3, 17, 2047, 2048, 2049, 8191, 8192, 8193])
@pytest.mark.parametrize("cols,log_rows", [(8, 0), (13, 0), (3, 2)])
def test_leaves(glc, oracle, round_constants, count, cols, log_rows):
    glc.poseidon2.set_round_constants(round_constants)
    x = rand_elems((cols * count) << log_rows, count + cols, noncanonical=True)
    d, out = to_dev(x), zeros_dev(4 * count)
    glc.GLHasher.compute_leaf_hashes(d, out, log_rows, False, False)
    assert (from_dev(out) == oracle.leaves(x, 4 * count, log_rows)).all()


@pytest.mark.parametrize("count", [5, 2048, 8192])
def test_checkpointed_leaves(glc, oracle, round_constants, count):
    glc.poseidon2.set_round_constants(round_constants)
    x = rand_elems(21 * count, count, noncanonical=True)
    out = zeros_dev(4 * count)
    glc.GLHasher.compute_leaf_hashes(to_dev(x[:16 * count]), out, 0, False, True)
    glc.GLHasher.compute_leaf_hashes(to_dev(x[16 * count:]), out, 0, True, False)
    assert (from_dev(out) == oracle.leaves(x, 4 * count)).all()


@pytest.mark.parametrize("count", [1, 2, 31, 2047, 2048, 2049, 8192, 8193])
@pytest.mark.parametrize("shift", [0, 1])
def test_nodes(glc, oracle, round_constants, count, shift):
    glc.poseidon2.set_round_constants(round_constants)
    x = rand_elems(8 * count, count, noncanonical=True)
    d = to_dev(np.concatenate([np.zeros(shift, dtype=np.uint64), x]))  # shift 1: not 16-byte aligned
    out = zeros_dev(4 * count)
    glc.GLHasher.compute_node_hashes(d[shift:], out)
    assert (from_dev(out) == oracle.nodes(x)).all()


@pytest.mark.parametrize("log_leaves", [1, 2, 4, 5, 6, 11, 12, 13, 14, 15])
@pytest.mark.parametrize("log_cap", [0, 1, 4])
def test_trees(glc, oracle, round_constants, log_leaves, log_cap):
    if log_cap > log_leaves:
        pytest.skip("cap larger than the tree")
    glc.poseidon2.set_round_constants(round_constants)
    leaves, layers = 1 << log_leaves, log_leaves - log_cap + 1
    x = rand_elems(5 * leaves, log_leaves)
    out = zeros_dev(8 * leaves)
    glc.GLHasher.build_merkle_tree(to_dev(x), out, 0, layers_count=layers)
    assert (from_dev(out) == oracle.build_merkle_tree(x, 8 * leaves, 0, layers)).all()
