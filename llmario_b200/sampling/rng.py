"""xoshiro256** seeded through splitmix64: one stream per request, one ``next_f64`` per sampled
token, never advanced by greedy decoding (crates/engine/decode/src/rng.rs:14-52).  The streams
advance in ``csrc/host/rng_core.cpp``."""
from __future__ import annotations

import ctypes
from typing import Optional, Sequence

from ..csrc.build import load_host_library

_M = (1 << 64) - 1
_State = ctypes.c_uint64 * 4
_lib: Optional[ctypes.CDLL] = None


def _native() -> ctypes.CDLL:
    global _lib
    if _lib is None:
        lib = load_host_library()
        lib.llm_rng_next.restype = ctypes.c_uint64
        lib.llm_rng_next.argtypes = [ctypes.c_void_p]
        lib.llm_rng_uniforms.restype = None
        lib.llm_rng_uniforms.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
        _lib = lib
    return _lib


class Xoshiro256StarStar:
    __slots__ = ("s",)

    def __init__(self, seed: int):
        state = seed & _M
        self.s = _State()
        for i in range(4):
            state = (state + 0x9E3779B97F4A7C15) & _M
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M
            self.s[i] = z ^ (z >> 31)

    def next_u64(self) -> int:
        return _native().llm_rng_next(ctypes.addressof(self.s))

    def next_f64(self) -> float:
        """Uniform in [0, 1) from the top 53 bits."""
        return (self.next_u64() >> 11) * (1.0 / (1 << 53))


def next_uniforms(streams: Sequence[Optional[Xoshiro256StarStar]], out: int) -> None:
    """The next ``next_f64`` of every stream, in order, as float64 values at the host address
    ``out``; 0 where there is no stream."""
    n = len(streams)
    where = (ctypes.c_uint64 * n)(*[0 if r is None else ctypes.addressof(r.s) for r in streams])
    _native().llm_rng_uniforms(where, n, out)
