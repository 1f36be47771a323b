/*
 * pj_item_shape.h — how k_parse_items cuts a call's input into tiles, and what a tile gets of shared memory. Host only. The result
 * of a call does not depend on it.
 */
#ifndef PJ_ITEM_SHAPE_H
#define PJ_ITEM_SHAPE_H

#include "pj_item.cuh"

namespace pj {

struct ItemShapeIn {
  uint64_t len;       /* bytes of the longest launch of the call */
  double avg;         /* bytes per record of the context's last call on the schema; 0: there was none */
  double guess;       /* without one: of records as the workload generator writes them */
  uint32_t longest;   /* bytes of the longest record of that call; 0: not known */
  uint32_t strs_per_kb; /* strings per 1024 bytes of its tile with the most; 0: not known */
  uint32_t tile_opt;  /* pj_options.tile_bytes; 0: ours to choose */
  uint32_t stride;    /* words per row (ItStride) */
  uint32_t sms;
};
struct ItemShape { uint32_t tile_bytes, win_bytes, str_words, row_cap; };

/* dynamic shared memory a block may take so that `blocks` of them share an SM (1 KB of each is the system's) */
inline uint32_t item_room(uint32_t blocks) {
  const uint32_t room = (228u * 1024u) / blocks - 1024u - (uint32_t)sizeof(ItemShared) - 256u;
  return room < IT_MAX_DYN_SMEM ? room : IT_MAX_DYN_SMEM;
}
inline ItemShape item_shape(const ItemShapeIn& in) {
  const double avg = in.avg > 0 ? in.avg : in.guess;
  /* Room behind the tile for its last record: a quarter more than the longest one of the call before, or 13 average records, which
     reach the longest ones of lists whose lengths are zipf(1.2) distributed. */
  const uint64_t longest = in.longest ? (uint64_t)in.longest + in.longest / 4 + 64 : (uint64_t)(avg * 13);
  const uint32_t slack = (longest < 4096 ? 4096u : (longest > 28672 ? 28672u : (uint32_t)longest)) & ~15u;
  /* what the block indexes in one step, or so that most tiles have fewer than three quarters of the lines they may have (a first
     call's records may be shorter than the guess) */
  const uint64_t most = (uint64_t)(avg * (in.avg > 0 ? IT_MAX_LINES * 47 / 64 : IT_MAX_LINES * 9 / 16));
  uint64_t tile = avg * 4 > IT_STEP ? IT_STEP / 2 : IT_STEP - (uint64_t)(2 * avg);
  if (tile > most) tile = most;
  /* lists of short strings: 4096 of them are a tile's limit, and each wants its word. (50k Pets of 40 strings of 4 bytes in an array:
     8.1 ms when their tiles did not fit; records as the generator writes them have 45 to 75 in 1024 bytes.) */
  if (in.strs_per_kb) {
    const uint64_t fit = (uint64_t)(IT_MAX_STRS * 7u / 8u) * 1024u / in.strs_per_kb;
    if (tile + slack > fit) tile = fit > slack + ST_MIN_TILE_BYTES ? fit - slack : ST_MIN_TILE_BYTES;
  }
  /* few tiles: one for every block that can be resident (one more would be a wave of its own: 20 k mixed records 72 us with 445 tiles, 46 with
     444), and room for many short strings */
  const uint64_t each = ((in.len + 15) / ((uint64_t)in.sms * IT_BLOCKS) + 32) & ~31ull;
  uint32_t per_word = 9; /* window bytes per word for strings */
  if (each < tile) { tile = each < 4096 ? 4096 : each; per_word = 2; }
  if (in.tile_opt) tile = in.tile_opt < ST_MIN_TILE_BYTES ? ST_MIN_TILE_BYTES : (in.tile_opt > 32768 ? 32768u : in.tile_opt);
  /* as many resident blocks as leave three quarters of that tile; strings give up room first */
  const uint64_t least = tile - tile / 4;
  for (uint32_t blocks = IT_BLOCKS;;) {
    ItemShape t;
    t.tile_bytes = (uint32_t)(tile & ~31ull);
    if (t.tile_bytes < ST_MIN_TILE_BYTES) t.tile_bytes = ST_MIN_TILE_BYTES;
    t.win_bytes = t.tile_bytes + slack < IT_MAX_WIN ? t.tile_bytes + slack : IT_MAX_WIN & ~15u;
    const double recs = (double)t.tile_bytes / avg * 1.3 + 24;
    t.row_cap = recs > IT_MAX_LINES ? IT_MAX_LINES : (uint32_t)recs;
    for (uint32_t w = per_word; w <= 9; ++w) {
      t.str_words = t.win_bytes / w;
      const uint32_t known = (uint32_t)((uint64_t)t.win_bytes * in.strs_per_kb / 819u) + 16u; /* a quarter more, for rows of elements */
      if (in.strs_per_kb && known > t.str_words) t.str_words = known < 4u * IT_MAX_STRS ? known : 4u * IT_MAX_STRS;
      if (item_layout(t.win_bytes, t.str_words, t.row_cap, in.stride).total <= item_room(blocks)) return t;
    }
    /* (the smallest tile fits two blocks whatever the records are, the largest fits one: tests/test_item_emulation.py) */
    if (t.tile_bytes <= ST_MIN_TILE_BYTES || blocks == 1) return t;
    if (in.tile_opt) --blocks;
    else if (tile - 512 >= least || blocks == 2) tile -= 512;
    else { tile = least + least / 3; --blocks; }
  }
}

}  // namespace pj
#endif
