// Parities in a ring of operand stages (host and device; no CUDA headers).
#pragma once
#include <cstdint>
#if defined(__CUDACC__)
#define TNNB_HD __host__ __device__
#else
#define TNNB_HD
#endif

namespace tnnb {

// A ring's copies go into stages 0, 1, ..., each turn into all of them; the last one went into `stage` in a turn of parity
// `phase`. Parity to wait for so that the newest copy into stage `s` has landed: this turn's up to `stage`, the turn before's
// behind it. Before the first turn that is a phase which a fresh barrier counts as complete.
TNNB_HD constexpr uint32_t ring_parity(int s, int stage, uint32_t phase) { return s <= stage ? phase : phase ^ 1u; }

}  // namespace tnnb
