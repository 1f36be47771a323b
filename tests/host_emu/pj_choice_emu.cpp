/*
 * pj_choice_emu.cpp — TEST INFRASTRUCTURE. The choice of the parse kernel for streams of several models. tests/test_mixed_choice.py drives it.
 */
#include "pj_choice.h"

static pj::NdChoice g;
extern "C" void mixed_choice_reset() { g = pj::NdChoice(); g.several = g.items = true; }
extern "C" int mixed_choice_note(unsigned long long len, float ms, unsigned long long records, unsigned long long fast, unsigned long long dense) {
  pj::note_call(g, len, ms, records, 0, fast, dense, 400);
  return g.items;
}
