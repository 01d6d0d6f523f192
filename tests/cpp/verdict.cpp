// The precheck's verdict word: a word of another solve is no verdict.
#include <cstdio>
#include <initializer_list>

#include "verdict.h"

using namespace smpb200;

int main() {
  int bad = 0;
  const uint32_t last = 0xFFFFFFFFu;  // solve numbers wrap
  for (uint32_t solve : {1u, 2u, 77u, 0x3FFFFFFFu, 0x40000000u, last}) {
    for (Verdict v : {kVerdictQuery, kVerdictPerfect, kVerdictOther}) {
      const uint32_t word = verdict_word(solve, v);
      bad += verdict_of(word, solve) != v;
      bad += verdict_of(word, solve + 1) != kVerdictNone;  // late, from the solve before
      bad += verdict_of(word, solve + 2) != kVerdictNone;
    }
    bad += verdict_of(0u, solve) != kVerdictNone;  // before the first
  }
  std::printf("%s %d\n", bad ? "BAD" : "VERDICT_OK", bad);
  return bad != 0;
}
