/*
 * pj_item_tables.h — compile-time tables of the item-parallel parse kernel (pj_item.cuh), derived from the model tables
 * of pj_schema.h: where a record's values stand in its row of shared memory, the hash table of property names and
 * what a property name means in which object.
 *
 * Rows. Every line of a tile has one row of 32-bit words. Words 0-3 are the row's own (flags, first failure, first byte and
 * closing brace, list of strings); then follow property 0 (`id`, the one property the models share by name,
 * kind and position), the enums, the other properties and those of the embedded object. While a record is tokenised a
 * word holds a reference to the value's text (ItemRef); int64 takes two words, a date-time four, because the decoded
 * value replaces the reference.
 *
 * An element of a list of objects is three words: the two of its integer and one for its string and flags (ItElem).
 */
#ifndef PJ_ITEM_TABLES_H
#define PJ_ITEM_TABLES_H

#include "pj_schema.h"

#if defined(__CUDACC__)
#define PJ_CX constexpr __host__ __device__
#else
#define PJ_CX constexpr
#endif

namespace pj {

/* what kind of object a string lies in */
enum { IS_ROOT = 0, IS_CHILD = 1, IS_LIST = 2, IS_ELEM = 3 };
/* what follows the colon of a key: a string, a number or literal, `{"`, `["`, `[{"`, `{}`, `[]` */
enum { IV_NONE = 0, IV_STR = 1, IV_SCALAR = 2, IV_OBJ = 3, IV_LIST = 4, IV_ELEM = 5, IV_EOBJ = 6, IV_ELIST = 7 };
/* words of a record's row; where a model has lists two more stand behind its fields: the list of objects (like IW_LIST: first
 * string or row | length << 16) and the bytes of both lists' strings (list of strings | list of objects << 16) */
enum { IW_FLAGS = 0, IW_ERR = 1, IW_POS = 2, IW_LIST = 3, IW_FIELDS = 4 };
/* IW_FLAGS: bits 0-11 keys met, 12-23 values present, 24-26 models the record cannot be (mixed streams), 27: the text of a
 * string was decoded in place (positions in the window are not the input's any more), 28: the line is a record, 29: the walk
 * did not recognise it, 30: the list of objects has rows of its own (else it is read off its strings), 31: the record failed
 * (IW_LIST then is the failure's offset). From the verdicts on bit 29 says that the record is a valid one of a kind only the exact
 * parser knows: it stands apart, and its row holds, from IW_FIELDS on, what it adds to each of its model's counters. */
static constexpr uint32_t IF_PRESENT = 12, IF_NOTMODEL = 24, IF_MOVED = 1u << 27, IF_RECORD = 1u << 28, IF_ODD = 1u << 29, IF_APART = IF_ODD, IF_ROWS = 1u << 30, IF_BAD = 1u << 31;
static constexpr uint32_t IB_CHILD = 8;  /* first bit of the embedded object's properties */
static constexpr uint32_t IB_SHARED = 10; /* a property of several models at different places of theirs (mixed streams) */
/* IW_ERR: window offset << 8 | kind of the first failure in reading order; kind 0xFF: the exact parser has to say */
static constexpr uint32_t IE_NONE = 0xFFFFFFFFu, IE_REFUSED = 0xFFu;

PJ_CX uint32_t it_kind_words(uint32_t kind) {
  return kind == K_I64 ? 2u : (kind == K_DATETIME ? 4u : ((kind == K_OBJ || kind == K_LIST_STR || kind == K_LIST_OBJ) ? 0u : 1u));
}
/* index of the property of this kind, -1: none (the models have at most one of each container kind) */
template <int OBJ>
PJ_CX int it_find(uint32_t kind) {
  int at = -1;
  for (int i = 0; i < CObj<OBJ>::N; ++i) if (CObj<OBJ>::f[i].kind == kind) at = i;
  return at;
}
template <int OBJ>
PJ_CX int it_count(uint32_t kind) {
  int n = 0;
  for (int i = 0; i < CObj<OBJ>::N; ++i) n += CObj<OBJ>::f[i].kind == kind;
  return n;
}
/* row word of property i of root OBJ; i == N: the first word behind the root's own */
template <int OBJ>
PJ_CX uint32_t it_root_word(int i) {
  uint32_t at = IW_FIELDS;
  for (int pass = 0; pass < 3; ++pass)
    for (int k = 0; k < CObj<OBJ>::N; ++k) {
      const uint32_t kind = CObj<OBJ>::f[k].kind;
      if ((k == 0 ? 0 : (kind == K_ENUM ? 1 : 2)) != pass) continue;
      if (k == i) return at;
      at += it_kind_words(kind);
    }
  return at;
}
template <int OBJ>
PJ_CX uint32_t it_flat_word(int i) { /* the same inside a flat object, from 0 */
  uint32_t at = 0;
  for (int k = 0; k < CObj<OBJ>::N && k < i; ++k) at += it_kind_words(CObj<OBJ>::f[k].kind);
  return at;
}
template <int OBJ>
struct ItModel {
  static constexpr int oi = it_find<OBJ>(K_OBJ), li = it_find<OBJ>(K_LIST_STR), ei = it_find<OBJ>(K_LIST_OBJ), di = it_find<OBJ>(K_DATETIME);
  static_assert(it_count<OBJ>(K_OBJ) <= 1 && it_count<OBJ>(K_LIST_STR) <= 1 && it_count<OBJ>(K_LIST_OBJ) <= 1, "one container of each kind");
  static_assert(CObj<OBJ>::N <= (int)IB_CHILD, "flag bits");
  static constexpr int child = oi >= 0 ? (int)CObj<OBJ>::f[oi < 0 ? 0 : oi].child : -1, elem = ei >= 0 ? (int)CObj<OBJ>::f[ei < 0 ? 0 : ei].child : -1;
  static constexpr uint32_t child_word = it_root_word<OBJ>(CObj<OBJ>::N);
};
template <int OBJ, int CH>
PJ_CX uint32_t it_row_words() {
  if constexpr (CH >= 0) return ItModel<OBJ>::child_word + it_flat_word<CH>(CObj<CH>::N);
  else return ItModel<OBJ>::child_word;
}
template <int OBJ> struct ItWords { static constexpr uint32_t n = it_row_words<OBJ, ItModel<OBJ>::child>(); };
PJ_CX uint32_t it_max(uint32_t a, uint32_t b) { return a > b ? a : b; }
/* words per row of a schema; odd, so that a warp that walks 32 rows meets 32 banks */
template <int SCHEMA>
struct ItStride {
  static constexpr uint32_t raw = SCHEMA == PJ_SCHEMA_PET ? ItWords<OBJ_PET>::n + 2u
                                  : (SCHEMA == PJ_SCHEMA_ORDER ? ItWords<OBJ_ORDER>::n
                                     : (SCHEMA == PJ_SCHEMA_USER ? ItWords<OBJ_USER>::n : it_max(ItWords<OBJ_PET>::n + 2u, it_max(ItWords<OBJ_ORDER>::n, ItWords<OBJ_USER>::n))));
  static constexpr uint32_t n = raw | 1u;
};

/* A property name in an object. 0: not a property (its value is skipped). */
struct ItField {
  static PJ_CX uint32_t make(uint32_t word, uint32_t bit, uint32_t kind, uint32_t models, uint32_t len) {
    uint32_t allowed = 0;
    if (kind == K_I64 || kind == K_I32 || kind == K_BOOL) allowed = 1u << IV_SCALAR;
    else if (kind == K_STR || kind == K_ENUM || kind == K_DATETIME) allowed = 1u << IV_STR;
    else if (kind == K_OBJ) allowed = (1u << IV_OBJ) | (1u << IV_EOBJ);
    else if (kind == K_LIST_STR) allowed = (1u << IV_LIST) | (1u << IV_ELIST);
    else allowed = (1u << IV_ELEM) | (1u << IV_ELIST);
    return word | (bit << 6) | (kind << 10) | (allowed << 14) | (models << 22) | (len << 25) | (1u << 31);
  }
  static PJ_CX uint32_t word(uint32_t f) { return f & 63u; }
  static PJ_CX uint32_t bit(uint32_t f) { return (f >> 6) & 15u; }
  static PJ_CX uint32_t kind(uint32_t f) { return (f >> 10) & 15u; }
  static PJ_CX uint32_t allowed(uint32_t f) { return (f >> 14) & 255u; }
  static PJ_CX uint32_t models(uint32_t f) { return (f >> 22) & 7u; }
  static PJ_CX uint32_t len(uint32_t f) { return (f >> 25) & 15u; } /* bytes of the name */
};

/* Names hash by their first two bytes and their length; the multiplier is searched at compile time so that no two of
 * the names share a slot. An entry is the name (text and byte masks, four words each; its length is in ItField: what follows a key
 * that was decoded in place is not its quote). */
static constexpr uint32_t IT_SLOTS = 32;
struct ItTables {
  uint32_t key[IT_SLOTS][8];
  uint32_t field[3][IT_SLOTS]; /* [root, embedded object, list element] */
  uint32_t mul;
};
PJ_CX uint32_t it_hash(uint32_t c01, uint32_t len, uint32_t mul) { return ((c01 + len * 0x3D51u) * mul) >> 27; }
struct ItName { uint64_t lo, hi; uint32_t len; };
struct ItNames { ItName n[40]; uint32_t count; };
PJ_CX void it_add_name(ItNames& s, const CF& f) {
  for (uint32_t k = 0; k < s.count; ++k) if (s.n[k].lo == f.lo && s.n[k].hi == f.hi && s.n[k].len == f.len) return;
  s.n[s.count].lo = f.lo; s.n[s.count].hi = f.hi; s.n[s.count].len = f.len;
  s.count++;
}
template <int OBJ>
PJ_CX void it_add_names(ItNames& s) {
  for (int i = 0; i < CObj<OBJ>::N; ++i) it_add_name(s, CObj<OBJ>::f[i]);
}
PJ_CX ItNames it_all_names() {
  ItNames s{};
  it_add_names<OBJ_PET>(s); it_add_names<OBJ_CATEGORY>(s); it_add_names<OBJ_TAG>(s); it_add_names<OBJ_ORDER>(s); it_add_names<OBJ_USER>(s);
  return s;
}
PJ_CX uint32_t it_find_mul() {
  const ItNames s = it_all_names();
  for (uint32_t t = 0; t < 4000; ++t) {
    const uint32_t mul = 0x9E3779B1u + t * 0x2545F492u;
    uint32_t used = 0;
    bool ok = true;
    for (uint32_t k = 0; k < s.count && ok; ++k) {
      const uint32_t b = 1u << it_hash((uint32_t)(s.n[k].lo & 0xFFFFu), s.n[k].len, mul);
      ok = !(used & b);
      used |= b;
    }
    if (ok) return mul;
  }
  return 0;
}
static constexpr uint32_t IT_MUL = it_find_mul();
static_assert(IT_MUL != 0, "a hash multiplier without collisions");
PJ_CX uint32_t it_name_byte(uint64_t lo, uint64_t hi, uint32_t k) { return (uint32_t)((k < 8 ? lo >> (8 * k) : hi >> (8 * (k - 8))) & 0xFF); }
PJ_CX uint32_t it_slot_of(const CF& f) { return it_hash((uint32_t)(f.lo & 0xFFFFu), f.len, IT_MUL); }
template <int OBJ>
PJ_CX void it_fill_root(ItTables& t, uint32_t model) {
  for (int i = 0; i < CObj<OBJ>::N; ++i) {
    const CF f = CObj<OBJ>::f[i];
    uint32_t& e = t.field[0][it_slot_of(f)];
    uint32_t bit = (uint32_t)i;
    if (e && ItField::bit(e) != bit) bit = IB_SHARED;
    e = ItField::make(it_root_word<OBJ>(i), bit, f.kind, model | (e ? ItField::models(e) : 0u), f.len);
  }
}
template <int OBJ, int CH>
PJ_CX void it_fill_flat(ItTables& t, int which, uint32_t word0, uint32_t bit0) {
  if constexpr (CH >= 0) {
    for (int i = 0; i < CObj<CH>::N; ++i) {
      const CF f = CObj<CH>::f[i];
      t.field[which][it_slot_of(f)] = ItField::make(word0 + (which == 1 ? it_flat_word<CH>(i) : (uint32_t)i), bit0 + (uint32_t)i, f.kind, 7u, f.len);
    }
  }
}
template <int OBJ>
PJ_CX void it_fill_model(ItTables& t, uint32_t model) {
  it_fill_root<OBJ>(t, model);
  it_fill_flat<OBJ, ItModel<OBJ>::child>(t, 1, ItModel<OBJ>::child_word, IB_CHILD);
  it_fill_flat<OBJ, ItModel<OBJ>::elem>(t, 2, 0u, 0u);
}
PJ_CX ItTables it_tables(int schema) {
  ItTables t{};
  const ItNames s = it_all_names();
  for (uint32_t k = 0; k < s.count; ++k) {
    const uint32_t slot = it_hash((uint32_t)(s.n[k].lo & 0xFFFFu), s.n[k].len, IT_MUL);
    for (uint32_t b = 0; b < s.n[k].len; ++b) {
      t.key[slot][b >> 2] |= it_name_byte(s.n[k].lo, s.n[k].hi, b) << (8 * (b & 3));
      t.key[slot][4 + (b >> 2)] |= 0xFFu << (8 * (b & 3));
    }
  }
  if (schema == PJ_SCHEMA_PET || schema == PJ_SCHEMA_MIXED) it_fill_model<OBJ_PET>(t, 1u);
  if (schema == PJ_SCHEMA_ORDER || schema == PJ_SCHEMA_MIXED) it_fill_model<OBJ_ORDER>(t, 2u);
  if (schema == PJ_SCHEMA_USER || schema == PJ_SCHEMA_MIXED) it_fill_model<OBJ_USER>(t, 4u);
  t.mul = IT_MUL;
  return t;
}
/* ---- gaps --------------------------------------------------------------------------------------------------------
 * What stands between two strings of a record, or behind its last one, without blanks and with '0' for a number or a literal,
 * is one of 26 texts of at most eight bytes in every valid record. Each tells what the string before it is (a key and the kind
 * of its value, or a value), in which object that string must lie and which one the next lies in. */
struct ItGap {
  /* bits 0-2 IV_*, 3-6 object the gap needs (15: any), 7-8 object it leads to, 9: it tells the object at all, 10: the record
     ends, 11: an element of a list of objects begins, 12: the string before is a key, 13: valid */
  static PJ_CX uint32_t make(uint32_t vk, uint32_t need, uint32_t out, bool telling, bool ends, bool elem, bool key) {
    return vk | (need << 3) | (out << 7) | ((telling ? 1u : 0u) << 9) | ((ends ? 1u : 0u) << 10) | ((elem ? 1u : 0u) << 11) | ((key ? 1u : 0u) << 12) | (1u << 13);
  }
  static constexpr uint32_t TELLS = 1u << 9, ENDS = 1u << 10, ELEM = 1u << 11, KEY = 1u << 12;
  static PJ_CX uint32_t vk(uint32_t d) { return d & 7u; }
  static PJ_CX uint32_t need(uint32_t d) { return (d >> 3) & 15u; }
  static PJ_CX uint32_t out(uint32_t d) { return (d >> 7) & 3u; }
};
static constexpr uint32_t IG_SLOTS = 32;
struct ItGapEntry { uint32_t lo, hi, desc, len; };
struct ItGapTable { ItGapEntry e[IG_SLOTS]; bool ok; };
/* multipliers without a collision among the 26 texts, found by search */
PJ_CX uint32_t it_gap_hash(uint32_t lo, uint32_t hi) { return (lo * 0x3ED35535u + hi * 0x43D40BE5u) >> 27; }
PJ_CX void it_gap_add(ItGapTable& t, const char* head, const char* tail, uint32_t desc) {
  uint32_t w[2] = {0, 0};
  uint32_t n = 0;
  for (int part = 0; part < 2; ++part)
    for (const char* p = part ? tail : head; *p; ++p, ++n) w[n >> 2] |= (uint32_t)(uint8_t)*p << (8 * (n & 3));
  ItGapEntry& e = t.e[it_gap_hash(w[0], w[1])];
  t.ok = t.ok && e.desc == 0 && n <= 8;
  e.lo = w[0]; e.hi = w[1]; e.desc = desc; e.len = n;
}
PJ_CX ItGapTable it_gap_table() {
  ItGapTable t{};
  t.ok = true;
  it_gap_add(t, ":", "", ItGap::make(IV_STR, 15, 0, false, false, false, true));
  it_gap_add(t, ":{", "", ItGap::make(IV_OBJ, IS_ROOT, IS_CHILD, true, false, false, true));
  it_gap_add(t, ":[", "", ItGap::make(IV_LIST, IS_ROOT, IS_LIST, true, false, false, true));
  it_gap_add(t, ":[{", "", ItGap::make(IV_ELEM, IS_ROOT, IS_ELEM, true, false, true, true));
  for (uint32_t h = 0; h < 4; ++h) {
    const char* const heads[4] = {"", ":0", ":[]", ":{}"};
    const uint32_t vk = h == 0 ? IV_NONE : (h == 1 ? IV_SCALAR : (h == 2 ? IV_ELIST : IV_EOBJ));
    it_gap_add(t, heads[h], ",", ItGap::make(vk, 15, 0, false, false, false, h != 0));
    it_gap_add(t, heads[h], "}", ItGap::make(vk, IS_ROOT, IS_ROOT, true, true, false, h != 0));
    if (h > 1) continue; /* empty containers stand in the root only */
    it_gap_add(t, heads[h], "},", ItGap::make(vk, IS_CHILD, IS_ROOT, true, false, false, h != 0));
    it_gap_add(t, heads[h], "],", ItGap::make(vk, IS_LIST, IS_ROOT, true, false, false, h != 0));
    it_gap_add(t, heads[h], "}],", ItGap::make(vk, IS_ELEM, IS_ROOT, true, false, false, h != 0));
    it_gap_add(t, heads[h], "},{", ItGap::make(vk, IS_ELEM, IS_ELEM, true, false, true, h != 0));
    it_gap_add(t, heads[h], "}}", ItGap::make(vk, IS_CHILD, IS_ROOT, true, true, false, h != 0));
    it_gap_add(t, heads[h], "]}", ItGap::make(vk, IS_LIST, IS_ROOT, true, true, false, h != 0));
    it_gap_add(t, heads[h], "}]}", ItGap::make(vk, IS_ELEM, IS_ROOT, true, true, false, h != 0));
  }
  return t;
}
static_assert(it_gap_table().ok, "gap texts hash without collisions");

static_assert(it_root_word<OBJ_PET>(0) == it_root_word<OBJ_ORDER>(0) && it_root_word<OBJ_PET>(0) == it_root_word<OBJ_USER>(0), "id at one place");
static_assert(it_root_word<OBJ_PET>(5) == it_root_word<OBJ_ORDER>(4), "status at one place");

}  // namespace pj
#endif
