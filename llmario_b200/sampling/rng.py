"""xoshiro256** seeded through splitmix64: one stream per request, one ``next_f64`` per sampled
token, never advanced by greedy decoding (crates/engine/decode/src/rng.rs:14-52).  The streams
advance in ``csrc/host/rng_core.cpp``."""
from __future__ import annotations

import ctypes
from array import array
from typing import List, Optional, Sequence

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
    """``next_u64``, ``next_f64``; ``s`` is the state, a list of four integers that may be read, set
    and changed in place.  Until somebody asks for it, it is kept as four 64-bit words."""

    def __init__(self, seed: int):
        state = seed & _M
        self._words: Optional[ctypes.Array] = _State()
        self._list: Optional[List[int]] = None
        self._at = ctypes.addressof(self._words)      # 0 when the state is a list
        for i in range(4):
            state = (state + 0x9E3779B97F4A7C15) & _M
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M
            self._words[i] = z ^ (z >> 31)

    @property
    def s(self) -> List[int]:
        if self._words is not None:
            self._list, self._words, self._at = list(self._words), None, 0
        return self._list

    @s.setter
    def s(self, value: List[int]) -> None:
        self._list, self._words, self._at = value, None, 0

    def __getstate__(self):
        return {"s": self.s}

    def __setstate__(self, state) -> None:
        self.s = state["s"]

    def next_u64(self) -> int:
        if self._at:
            return _native().llm_rng_next(self._at)
        words = _State(*self._list)
        result = _native().llm_rng_next(ctypes.addressof(words))
        self._list[:] = words
        return result

    def next_f64(self) -> float:
        """Uniform in [0, 1) from the top 53 bits."""
        return (self.next_u64() >> 11) * (1.0 / (1 << 53))


def next_uniforms(streams: Sequence[Optional[Xoshiro256StarStar]], out: int) -> None:
    """The next ``next_f64`` of every stream, in order, as float64 values at the host address
    ``out``; 0 where there is no stream.  Streams that keep their words advance in one call; a stream
    whose ``s`` is a list, or of another class, is asked for its number."""
    at = [r._at if type(r) is Xoshiro256StarStar else 0 for r in streams]
    where = array("Q", at)
    _native().llm_rng_uniforms(where.buffer_info()[0], len(at), out)
    if 0 in at:
        for i in [i for i, a in enumerate(at) if not a and streams[i] is not None]:
            ctypes.c_double.from_address(out + 8 * i).value = streams[i].next_f64()
