"""A wait for the tensor cores that gives up: every thread of it is counted, the kernel ends with its
products finished and its TMEM freed, a served request that it may have been part of fails, and the calls
after it are whole.  The wait is one on a barrier that nothing completes (glc_expired_wait_probe).  Each
check runs in a process of its own, as the count stays for the life of the process."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import canon, load_package, load_synthetic, rand_elems
from gpu_util import from_dev, to_dev, torch, zeros_dev

THREADS = 128


def expire(glc, polls):
    glc._lib.call("glc_expired_wait_probe", polls, None)
    torch().cuda.synchronize()


def every_thread_counts(glc, oracle):
    assert glc.context.expired_waits() == 0
    for i, polls in enumerate((0, 1, 20)):
        expire(glc, polls)
        assert glc.context.expired_waits() == glc.commit.fused_timeouts() == (i + 1) * THREADS
    with pytest.raises(glc.GlcError):
        glc._lib.call("glc_expired_wait_probe", 50001, None)


def kernels_after_it_are_whole(glc, oracle):
    for _ in range(40):
        glc._lib.call("glc_expired_wait_probe", 0, None)
    n, cols = 1 << 16, 18
    x = rand_elems(cols * n, 1)
    d = to_dev(x)
    glc.ntt.batch_ntt_in_place(d, 16, cols, 0, n, False, True, 0, 0)
    assert (from_dev(d) == oracle.batch_ntt(x, 16, cols, n, n, 0, 1, 0, 0)).all()
    v, out = rand_elems(8 << 18, 2), zeros_dev(4 << 18)
    glc.GLHasher.compute_leaf_hashes(to_dev(v), out, 0, False, False)
    assert (from_dev(out) == oracle.leaves(v, 4 << 18, 0)).all()
    assert glc.context.expired_waits() == 40 * THREADS


def server_fails_the_request(glc, oracle):
    log_n, cols, log_lde, log_cap = 12, 8, 1, 4
    ev = load_synthetic().random_field_elements("expired", cols << log_n)
    _, _, _, want = oracle.commit(ev, log_n, cols, log_lde, log_cap)

    def served(srv):
        cap, _ = srv.wait(srv.submit(ev, log_n, cols, log_lde, log_cap))
        return (canon(np.asarray(cap)) == want).all()

    for _ in range(2):
        with glc.serve.Server(hbm_budget_bytes=1 << 30, max_inflight=2, streams=2) as srv:
            assert served(srv)
            expire(glc, 1)
            with pytest.raises(glc.GlcError) as e:
                served(srv)
            assert e.value.status == 909  # cudaErrorTimeout
            assert served(srv)


@pytest.mark.gpu
@pytest.mark.parametrize("check", ["every_thread_counts", "kernels_after_it_are_whole", "server_fails_the_request"])
def test_expired_wait(check):
    p = subprocess.run([sys.executable, os.path.abspath(__file__), check], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr


if __name__ == "__main__":
    import conftest
    import oracle as O
    constants = conftest.load_constants_module()
    rc = constants.env_round_constants() or constants.grain_lfsr_round_constants()
    O.build()
    O.set_round_constants(rc)
    package = load_package()
    package.Context.create(15, 15)
    package.poseidon2.set_round_constants(rc)
    globals()[sys.argv[1]](package, O)
