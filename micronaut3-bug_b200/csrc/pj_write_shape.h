/*
 * pj_write_shape.h — how many records a tile of the writer takes, and how much shared memory: from the sizes of the columns.
 */
#ifndef PJ_WRITE_SHAPE_H
#define PJ_WRITE_SHAPE_H

#include <stdint.h>

namespace pj {

struct WriteShapeIn {
  uint64_t n;           /* records */
  uint64_t rows[3];     /* rows of the models' tables */
  uint64_t arena_bytes; /* of all string arenas */
  uint64_t strs, objs;  /* elements of the lists of strings / of objects */
  uint32_t sms;
};
struct WriteShape { uint32_t recs, smem; };

/* A tile holds the pieces of the columns it reads, a running sum per list element and a window for its text, which goes in rounds. Names,
 * punctuation and numbers are taken at their usual length. Blocks share an SM as WtT<> says (pj_write_tile.cuh): two of 512 threads for Pets and
 * mixed streams, three of 256 for Orders and Users. Records per tile, 400 k records, us of the kernel: Orders 128 / 192 / 256: 84 / 72 / 62
 * (look-back and the way of the columns to shared memory cost as much for few records as for many), Users 128 / 192 / 256: 109 / 97 / 100; 600 k Pets
 * in windows of 128, 128 / 256 to a tile: 240 / 224 (one window for all 256, one block per SM: 307). Long records, 300 MB, with at least four (two) to a
 * tile and what was left for a window / so that a window holds one: Users of 16 KB 900 / 395, Pets with 100 strings of 400 bytes 2650 /
 * 385, with 600 of 60 bytes 2850 / 525. A record that would need more than a block's share goes to the general road at once, unless it is long for its
 * lists: one to a staged tile / 32 to one on that road, Users of 30 KB 520 / 450, of 48 KB 695 / 340, Pets of 43 KB 610 / 315, 100 strings of 400 bytes
 * 385 / 1000. */
inline WriteShape write_shape(const WriteShapeIn& in, uint32_t max_recs, uint32_t max_smem) {
  const double n = in.n ? (double)in.n : 1.0;
  /* columns: 36 bytes of a Pet, 32 of an Order, 38 of a User, 8 and 17 of the lists' elements with their sums */
  const double staged = (36.0 * (double)in.rows[0] + 32.0 * (double)in.rows[1] + 38.0 * (double)in.rows[2] + (double)in.arena_bytes + 8.0 * (double)in.strs + 17.0 * (double)in.objs) / n;
  const double text = (130.0 * (double)in.rows[0] + 150.0 * (double)in.rows[1] + 125.0 * (double)in.rows[2] + (double)in.arena_bytes + 3.0 * (double)in.strs + 40.0 * (double)in.objs) / n;
  const bool several = (in.rows[0] > 0) + (in.rows[1] > 0) + (in.rows[2] > 0) > 1;
  const double room = (several || in.rows[0] ? 100.0 : 64.0) * 1024.0;
  uint32_t recs = several || in.rows[0] || in.rows[1] ? 256u : 192u;
  const uint32_t round = !several && in.rows[0] ? 128u : recs;
  if (recs > max_recs) recs = max_recs;
  while (recs > 32u && in.n < (uint64_t)recs * in.sms) recs -= 32u;
  /* the window holds a record, and one half as long again: what does not fit it is written from global memory */
  const double one = 1.5 * text + 256.0;
  const bool lists = (double)(in.strs + in.objs) > 16.0 * n; /* (whose elements the lanes of a staged tile write side by side) */
  double smem;
  if (staged * 1.04 + 1024.0 + one > (lists ? (double)max_smem : room)) { /* not even one: the general road, whose long strings and lists are the warps' */
    recs = 32u;
    while (recs > 1u && in.n < (uint64_t)recs * in.sms * 2u) recs /= 2u;
    smem = 16384.0;
  } else if (!lists) {
    while (recs > 32u && staged * recs > 0.55 * room) recs -= 32u;
    while (recs > 4u && staged * recs > 0.9 * room) recs /= 2u;
    while (recs > 1u && staged * recs * 1.04 + 1024.0 + one > room) recs = recs > 4u ? recs / 2u : recs - 1u;
    const double pieces = staged * recs * 1.04 + 1024.0, left = room - pieces > 8192.0 ? room - pieces : 8192.0;
    const double window = text * (recs < round ? recs : round) * 1.06;
    smem = pieces + (window < left ? (window > one ? window : one) : left);
  } else { /* long lists differ much from record to record: few records in much room, two blocks to an SM, so that (almost) no tile outgrows it */
    if (recs > 16u) recs = 16u;
    while (recs > 2u && staged * recs > 0.25 * room) recs -= 2u;
    smem = 100.0 * 1024.0;
    while (recs > 1u && staged * recs * 1.04 + 1024.0 + one > smem) --recs;
    if (staged * recs * 1.04 + 1024.0 + one > smem) smem = staged * recs * 1.04 + 1024.0 + one;
  }
  if (smem < 8192.0) smem = 8192.0;
  if (smem > (double)max_smem) smem = (double)max_smem;
  WriteShape s;
  s.recs = recs;
  s.smem = ((uint32_t)smem + 127u) & ~127u;
  return s;
}

}  // namespace pj
#endif
