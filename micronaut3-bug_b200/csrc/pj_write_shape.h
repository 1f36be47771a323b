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

/* A tile holds the pieces of the columns it reads, a running sum per list element and its text. Names, punctuation and numbers are taken at
 * their usual length; text that does not fit goes in rounds. Three blocks of 256 threads share an SM (80 registers a thread), 70 KB each.
 * Records per tile, 400 k records, us of the kernel: Orders 128 / 192 / 256: 84 / 72 / 62 (their tiles are short, and look-back and the way of the
 * columns to shared memory cost as much for few records as for many), Users 128 / 192: 109 / 97, Pets 128 / 192 (two blocks): 164 / 191. */
inline WriteShape write_shape(const WriteShapeIn& in, uint32_t max_recs, uint32_t max_smem) {
  const double n = in.n ? (double)in.n : 1.0;
  /* columns: 36 bytes of a Pet, 32 of an Order, 38 of a User, 8 and 17 of the lists' elements with their sums */
  const double staged = (36.0 * (double)in.rows[0] + 32.0 * (double)in.rows[1] + 38.0 * (double)in.rows[2] + (double)in.arena_bytes + 8.0 * (double)in.strs + 17.0 * (double)in.objs) / n;
  const double text = (130.0 * (double)in.rows[0] + 150.0 * (double)in.rows[1] + 125.0 * (double)in.rows[2] + (double)in.arena_bytes + 3.0 * (double)in.strs + 40.0 * (double)in.objs) / n;
  const double room = 64.0 * 1024.0;
  uint32_t recs = (in.rows[0] > 0) + (in.rows[1] > 0) + (in.rows[2] > 0) > 1 ? 192u : (in.rows[0] ? 128u : (in.rows[1] ? 256u : 192u));
  if (recs > max_recs) recs = max_recs;
  while (recs > 32u && in.n < (uint64_t)recs * in.sms) recs -= 32u;
  double smem;
  if ((double)(in.strs + in.objs) <= 16.0 * n) {
    while (recs > 32u && staged * recs > 0.5 * room) recs -= 32u;
    while (recs > 4u && staged * recs > 1.4 * room) recs /= 2u;
    const double window = text * recs * 1.06;
    smem = staged * recs * 1.04 + (window < 0.75 * room ? window : 0.75 * room) + 1024.0;
  } else { /* long lists differ much from record to record: few records in much room, two blocks to an SM, so that (almost) no tile outgrows it */
    if (recs > 16u) recs = 16u;
    while (recs > 2u && staged * recs > 0.4 * room) recs -= 2u;
    smem = 100.0 * 1024.0;
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
