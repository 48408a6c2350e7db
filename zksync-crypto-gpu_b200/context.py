"""Per-device twiddle/power tables: the counterpart of boojum-cuda's context::Context
(crates/boojum-cuda/src/context.rs:157-297)."""
from __future__ import annotations

import ctypes as C

from ._lib import call

OMEGA_LOG_ORDER = 30


def expired_waits() -> int:
    """Bounded waits of kernels on this device that gave up since load (glc_expired_waits): 0 unless
    something is wrong.  NTT, hash and commitment calls are asynchronous and cannot report one; results
    are sound if this did not grow over a synchronisation after them.  Synchronous."""
    v = C.c_uint64()
    call("glc_expired_waits", C.byref(v))
    return v.value


class Context:
    """Tables of the current device.  Context.create(...) mirrors Context::create (context.rs:171);
    destroy() mirrors Context::destroy (context.rs:284).  One per device, like the reference's
    __constant__ descriptors."""

    def __init__(self, w_coarse_log: int, g_coarse_log: int):
        self.w_coarse_log = w_coarse_log
        self.g_coarse_log = g_coarse_log
        self._alive = True

    @classmethod
    def create(cls, powers_of_w_coarse_log_count: int = 15, powers_of_g_coarse_log_count: int = 15) -> "Context":
        call("glc_context_create", powers_of_w_coarse_log_count, powers_of_g_coarse_log_count)
        return cls(powers_of_w_coarse_log_count, powers_of_g_coarse_log_count)

    def destroy(self) -> None:
        if self._alive:
            call("glc_context_destroy")
            self._alive = False
