// The random streams of requests (xoshiro256**; crates/engine/decode/src/rng.rs:14-52): a stream is
// four 64-bit words that its owner holds.  A draw for 64 requests took some 60 us in Python, whose
// integers have no fixed width; here it is one call.
#include <cstdint>

namespace {
uint64_t rotl(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }

uint64_t next(uint64_t* s) {
  const uint64_t result = rotl(s[1] * 5, 7) * 9;
  const uint64_t t = s[1] << 17;
  s[2] ^= s[0];
  s[3] ^= s[1];
  s[1] ^= s[2];
  s[0] ^= s[3];
  s[2] ^= t;
  s[3] = rotl(s[3], 45);
  return result;
}
}  // namespace

extern "C" {

uint64_t llm_rng_next(uint64_t* state) { return next(state); }

// out[i] = the next uniform in [0, 1) of stream i, from the top 53 bits; 0 for a null stream
void llm_rng_uniforms(uint64_t* const* states, int n, double* out) {
  for (int i = 0; i < n; ++i) out[i] = states[i] ? (double)(next(states[i]) >> 11) * (1.0 / 9007199254740992.0) : 0.0;
}

}  // extern "C"
