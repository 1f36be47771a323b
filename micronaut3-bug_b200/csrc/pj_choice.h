/*
 * pj_choice.h — which of the two parse kernels an NDJSON call takes. Host only.
 */
#ifndef PJ_CHOICE_H
#define PJ_CHOICE_H

#include <stdint.h>

namespace pj {

static constexpr uint64_t ND_LONG = 16384; /* bytes per record */

/* Which kernel a schema's next call takes, and what note_call() remembers of the calls before. */
struct NdChoice {
  bool items = false;           /* k_parse_items, else k_parse_stream */
  bool several = false;         /* records of several models */
  bool handed_back = false;     /* the last change was back, because the text was all in one compact spelling */
  uint32_t clean = 0, wait = 1; /* such calls in a row, and how many it takes */
  double ns[2] = {0, 0};        /* per input byte, of the last timed call with k_parse_stream / k_parse_items, */
  uint64_t len[2] = {0, 0};     /* that call's bytes */
  uint64_t per[2] = {0, 0};     /* and its records' */
  uint32_t runs = 0;            /* timed calls with k_parse_stream */
  bool again = false;           /* its first one lost narrowly: this call is its second */
  uint32_t aside = 0;           /* several: calls in a row that k_parse_items put aside because of their long records */
  double tried = 0;             /* what k_parse_stream takes for the text that k_parse_items was last slower on, */
  uint32_t spared = 0;          /* and calls on such text since */
};
/* Which kernel parses the next NDJSON call. A record per thread (k_parse_stream) is the faster one as long as its lockstep pass takes
 * them; with 2 % of the records left to the exact parser every warp has one that the others wait for, and with most of them left to the
 * word-at-a-time tokeniser its threads go separate ways. k_parse_items is then often the faster one, but not always (100k Users, us:
 * blanks 195 / 89, an unknown string in each 344 / 130, names in another script 84 / 114, 10 % with a nested unknown value 355 / 590, all of
 * them 340 / 740), so it is tried, and of two calls of like size one with each kernel the time per byte decides. It hands back what its
 * strict walk took at 99 %, at once the first time, after twice as many such calls each time the text turned out to change its spelling.
 * Streams of several models start with k_parse_items and stay with it: it sorts a tile's lines by model, where a warp of the other one runs the
 * three models' code one after the other (300k records, us: compact 312 / 250, 1 % malformed 371 / 283); only text that leaves its records to
 * the exact parser has the other one tried, and then the time decides.
 * Records of 16 KB leave its blocks too little to do side by side: they are not tried (300 Pets of 40 KB: 0.5 / 15.6 ms), and such calls on
 * streams of several models are put aside when a look at some of their bytes shows them (pj_index.cuh). Their times are only compared between
 * calls of like record length; one model's are by bytes alone, so that a call on longer records finds its way back (it is not put aside). The
 * first timed call of a handle takes up to 0.15 ms more than the next ones (50 k Users with nested unknown values: k_parse_stream 255, then 113 us,
 * k_parse_items 172): where k_parse_items wins by less than 0.2 ms, the other one has a second call. The result does not depend on the choice. */
inline void note_call(NdChoice& k, uint64_t len, float ms, uint64_t records, uint64_t errors, uint64_t fast, uint64_t dense, uint32_t max_rec) {
  if (records < 16 && len < (1u << 16)) return;
  const uint64_t per = len / (records ? records : 1);
  if (k.several && per >= ND_LONG) { /* says nothing of usual records, which have k_parse_items again */
    k.items = false;
    return;
  }
  k.aside = 0;
  const bool timed = len >= (1u << 18); /* below, a call's time is not its text's */
  const int now = k.items ? 1 : 0, other = 1 - now;
  if (timed) { k.ns[now] = ms * 1e6 / (double)len; k.len[now] = len; k.per[now] = per; k.runs += k.items ? 0u : 1u; }
  const bool alike = timed && k.len[other] && k.len[other] / 2 <= len && len / 2 <= k.len[other] && (!k.several || (k.per[other] / 2 <= per && per / 2 <= k.per[other])); /* the two can be compared */
  const bool lost = alike && k.ns[other] < k.ns[now];
  const uint64_t good = records - errors;
  const bool again = k.again;
  k.again = false;
  if (!k.items) {
    if (!k.several && fast * 100 >= good * 98 && dense * 2 >= good) return;
    if (per >= ND_LONG) return;
    if ((k.handed_back || again) && alike && !lost) k.tried = k.ns[0];
    /* text as that which k_parse_items was slower on; every 64th such call tries all the same */
    if (timed && k.ns[0] < k.tried * 1.25 && k.ns[0] > k.tried * 0.8 && ++k.spared < 64) return;
    k.spared = 0;
    if (k.handed_back && k.wait < 64) k.wait *= 2;
    k.items = true; k.handed_back = false; k.clean = 0;
  } else if (lost) {
    k.tried = k.ns[0];
    k.items = k.handed_back = false;
  } else if (!k.several && alike && k.runs == 1 && (k.ns[0] - k.ns[1]) * (double)len < 0.2e6) {
    k.items = false; k.again = true;
  } else if (k.several && timed && !alike && fast * 100 < good * 98) {
    k.items = false; k.handed_back = true;
  } else if (!k.several && dense * 100 >= good * 99 && max_rec <= 1024) {
    if (++k.clean >= k.wait) { k.items = false; k.handed_back = true; }
  } else k.clean = 0;
}
/* ... and when a call was put aside: the second in a row takes the next one to k_parse_stream at once. */
inline void note_aside(NdChoice& k) {
  if (++k.aside >= 2) k.items = false;
}

}  // namespace pj
#endif
