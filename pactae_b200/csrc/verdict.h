// verdict.h -- what the precheck tells a host that waits for it, in one word of
// pinned memory: the number of the solve it belongs to, and the verdict.  A
// solve that fails after its precheck is enqueued does not wait for it, so the
// word of an earlier solve may arrive during a later one; it counts for nothing
// there.
#pragma once

#include <cstdint>

namespace smpb200 {

enum Verdict : uint32_t { kVerdictNone = 0, kVerdictQuery = 1, kVerdictPerfect = 2, kVerdictOther = 3 };

constexpr uint32_t verdict_word(uint32_t solve, Verdict v) { return (solve << 2) | v; }

// kVerdictNone unless the word is this solve's.
constexpr Verdict verdict_of(uint32_t word, uint32_t solve) {
  return (word >> 2) == ((solve << 2) >> 2) ? static_cast<Verdict>(word & 3u) : kVerdictNone;
}

}  // namespace smpb200
