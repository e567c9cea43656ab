// Onesweep-style LSD radix sort of (key, row) pairs with 8-bit digits, used by
// `sort` (multi-key, stable) and by `hash_partition` (stable bucket order).
#pragma once

#include "table_ops.cuh"

namespace ldf {

// Rows per onesweep tile (threads x items per thread).
constexpr int kRadixThreads = 256;
constexpr int kRadixItems   = 12;
constexpr int kRadixTile    = kRadixThreads * kRadixItems;
// Resident onesweep CTAs per SM the register budget is sized for.
constexpr int kRadixMinBlocks = 4;

// How a pass obtains the digit of a row.
enum class DigitSrc : int {
  CARRIED = 0,  // byte `shift/8` of the carried key word (written beforehand: radix_sort_words)
  COLUMN  = 1,  // load the key column at the row, transform, then byte
  CLASS   = 2,  // 0/1/2 class of the row: value / NaN / null, ordered by nulls_at_end
  BUCKET  = 3,  // hash of the key columns % nparts (then byte)
  FUSED   = 4   // byte of the fused word of several keys (FusedKey)
};

// Value transform of one sort key column into an order-preserving unsigned
// word (ascending), inverted for descending; null and NaN rows give 0 (their
// order comes from the CLASS pass).
struct SortKeyDesc {
  DCol col;
  int descending;
  int nulls_at_end;
  int key_bytes;  // bytes of the transformed word (1..8)
};

// Order-preserving word of a sort key from the value's raw bits (zero for a
// null or a NaN: those rows are placed by the CLASS pass).
__device__ __forceinline__ uint64_t sort_word_of(const SortKeyDesc& k, uint64_t raw, bool valid)
{
  if (!valid) return 0;
  uint64_t o;
  switch (k.col.type) {
    case LDF_INT8: o = (raw & 0xffu) ^ 0x80u; break;
    case LDF_INT16: o = (raw & 0xffffu) ^ 0x8000u; break;
    case LDF_INT32: o = (raw & 0xffffffffu) ^ 0x80000000u; break;
    case LDF_INT64:
    case LDF_TIMESTAMP_US: o = raw ^ (1ull << 63); break;
    case LDF_FLOAT32: {
      uint32_t b = static_cast<uint32_t>(raw);
      if ((b & 0x7f800000u) == 0x7f800000u && (b & 0x007fffffu)) return 0;  // NaN: CLASS pass
      if ((b & 0x7fffffffu) == 0) b = 0;                                    // -0.0 == 0.0
      o = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
      o &= 0xffffffffull;
      break;
    }
    case LDF_FLOAT64: {
      uint64_t b = raw;
      if ((b & 0x7ff0000000000000ull) == 0x7ff0000000000000ull && (b & 0x000fffffffffffffull)) return 0;
      if ((b & 0x7fffffffffffffffull) == 0) b = 0;
      o = (b & (1ull << 63)) ? ~b : (b | (1ull << 63));
      break;
    }
    default: o = raw; break;  // unsigned, bool, string ranks (uint32)
  }
  if (k.descending) {
    const uint64_t mask = k.key_bytes >= 8 ? ~0ull : ((1ull << (8 * k.key_bytes)) - 1);
    o                   = ~o & mask;
  }
  return o;
}

__device__ __forceinline__ uint64_t sort_word(const SortKeyDesc& k, int64_t row)
{
  return sort_word_of(k, dbits(k.col, row), dvalid(k.col, row));
}

// 0 = value, 1 = NaN, 2 = null when nulls_at_end; reversed otherwise
// (Arrow places NaN next to the values and nulls outermost, either direction).
__device__ __forceinline__ uint32_t class_digit(const SortKeyDesc& k, int64_t row)
{
  const DCol& c = k.col;
  uint32_t cls  = 0;
  if (!dvalid(c, row)) cls = 2;
  else if (c.type == LDF_FLOAT64) {
    uint64_t b = static_cast<const uint64_t*>(c.data)[row];
    if ((b & 0x7ff0000000000000ull) == 0x7ff0000000000000ull && (b & 0x000fffffffffffffull)) cls = 1;
  } else if (c.type == LDF_FLOAT32) {
    uint32_t b = static_cast<const uint32_t*>(c.data)[row];
    if ((b & 0x7f800000u) == 0x7f800000u && (b & 0x007fffffu)) cls = 1;
  }
  return k.nulls_at_end ? cls : 2 - cls;
}

struct RadixPass {
  DigitSrc src;
  int shift;      // bit offset of the digit in the key word (FUSED: in C)
  int fused_low;  // FUSED: the pass of the fused word's low byte
  SortKeyDesc key;
  KeyCols hash_keys;  // BUCKET
  uint32_t nparts;    // BUCKET
};

// Several sort keys packed into one word, least significant key first: W =
// sum_k code_k << off_k, at most kFusedMaxBits bits in all.  code_k is
// word_k - min_k, word_k the key's order-preserving word (inverted when
// descending) and min_k its minimum over the rows; a key with nulls or NaNs
// takes two codes more, before or behind its values (fused_code).  With `drop`
// (0, or 8 and more) the low `drop` bits are left out and W >> drop sorted.
// A word of at most 64 bits is written by one pass over the key columns, which
// counts all its digits too (radix_sort_words).  Of a wider one the pass of
// the low byte loads every key at the row and carries C = W >> 8; the later
// passes take byte shift / 8 of C.  One word for all the keys means that no
// pass gathers a key column through the permutation.
constexpr int kFuseMax      = 4;
constexpr int kFusedMaxBits = 72;
struct FusedKey {
  int n;
  SortKeyDesc key[kFuseMax];
  uint64_t min[kFuseMax];
  uint64_t span[kFuseMax];  // largest word - min
  int off[kFuseMax];
  int has_class[kFuseMax];
  int drop;
};

// Minimum and maximum of the order-preserving words of `keys` over n rows,
// nulls and NaNs aside (~0 and 0 when there are no others), one read of each
// column.
void sort_word_ranges(const OpContext& ctx, const SortKeyDesc* keys, int nkeys, int64_t n, uint64_t* mn,
                      uint64_t* mx);

// Fewest rows for which bits are dropped: below, the sample and its read-back
// cost what they save.
constexpr int64_t kDropMinRows = int64_t(1) << 21;

// Dropped bits (0: none) with which sorting on the rest of the fused word of
// `bits` bits, and then ordering the few rows that tie on it, takes fewest
// passes: from the ties among a sample of the rows.  whole_rows: for
// radix_sort_pairs, which orders many ties cheaply.
int choose_drop(const OpContext& ctx, const FusedKey& f, int bits, int64_t n, bool whole_rows = false);

// Orders the rows of every run of equal `words` (the sorted W >> f.drop, 4 or
// 8 bytes each) in `perm` by the dropped bits, equal rows in the order they
// have.  False when a run is longer than kTieRunMax (perm is then no longer
// useful).
constexpr int kTieRunMax = 4096;
bool order_ties(const OpContext& ctx, const FusedKey& f, const void* words, int word_bytes, int64_t n, int32_t* perm);

// Upfront digit histograms of every candidate pass: hist[p * 256 + d].
void radix_histograms(const OpContext& ctx, const std::vector<RadixPass>& passes, int64_t n,
                      uint32_t* d_hist, const FusedKey* fused = nullptr);

// Columns the last radix pass moves into sorted order itself: dst[j][pos] =
// src[j][row] (and the null masks), written as the pass's coalesced runs
// while the tile's source rows are still in cache.  Widths 1, 2, 4, 8, and 16
// (the ranges of a string column; its characters stay where they are).
// A payload may also carry one 16-byte record per row (`packed`, 16-byte
// aligned) holding up to kPassPayload non-nullable fixed-width values: part k
// is pwidth[k] bytes at byte offset poff[k] (a multiple of its width) and goes
// to pdst[k].  One random load per row then serves all of them.
constexpr int kPassPayload = 4;
struct RadixPayload {
  int n;
  DCol src[kPassPayload];
  void* dst[kPassPayload];
  uint8_t* dst_valid[kPassPayload];
  const ulonglong2* packed;
  int nparts;
  int pwidth[kPassPayload];
  int poff[kPassPayload];
  void* pdst[kPassPayload];
};

inline bool payload_empty(const RadixPayload& p) { return p.n == 0 && p.nparts == 0; }

// Stable sort of rows by a list of passes, least significant first; `perm` (n
// entries) receives the row order.  A pass whose digit is the same in every row
// is skipped.
// `inv` (optional, n entries): inv[row] = the row's position in the sorted
// order, written by the last pass.  `payload` (optional): columns the last
// pass writes in sorted order.  `fused`: the FusedKey of FUSED passes.
// `counted` (optional): the digit counts of all passes ([pass][256]), when the
// caller has them; otherwise one read of the keys counts them.
void radix_sort_rows(const OpContext& ctx, const std::vector<RadixPass>& passes, int64_t n,
                     int32_t* perm, const std::vector<uint32_t>* counted = nullptr, int32_t* inv = nullptr,
                     const RadixPayload* payload = nullptr, const FusedKey* fused = nullptr);

// The same on the fused word W >> f.drop of at most 64 bits (W has `bits`).
// `words` (optional, instead of a payload): the sorted words, *word_bytes each
// (4 when they have at most 32 bits, else 8).
void radix_sort_words(const OpContext& ctx, const FusedKey& f, int bits, int64_t n, int32_t* perm,
                      const RadixPayload* payload, Buffer<uint8_t>* words = nullptr, int* word_bytes = nullptr);

// Sort of a whole table (outputs allocated) whose rows fit in the passes
// themselves (radix_pairs_fit): one integer key, at most 8 bytes of up to
// kPassPayload other fixed-width columns, no nulls.  The passes carry the whole word and those
// columns instead of row ids, so nothing is gathered afterwards, and the key
// column is the word turned back.  100M rows of an int64 key and an int32
// column: 4.0 ms (three passes of 0.79, the last step 1.0), against 7.2 ms with row
// ids and one random 16-byte read a row.
// From kDropMinRows rows, as for the bits dropped: the passes of smaller
// tables stay in L2 with row ids too.
bool radix_pairs_fit(const FusedKey& f, int64_t n, const ldf_column* table, int ncols, int key);
void radix_sort_pairs(const OpContext& ctx, FusedKey f, int bits, int64_t n, const ldf_column* table, int ncols, int key,
                      ldf_column* out);

// The payload's columns gathered through `perm` (payload.dst[position] =
// src[perm[position]]).
void move_by_perm(const OpContext& ctx, const RadixPayload& payload, const int32_t* perm, int64_t n);

// ---- small inputs (rank_sort.cu) -----------------------------------------
// The whole sort of a table of at most kRankSortRows rows in one or two
// launches: a row's position is the number of rows that sort before it.
// `kd`: the keys, least significant first.  False (nothing done) when the
// table is larger or the keys do not fit.
constexpr int64_t kRankSortRows = 16384;
bool rank_sort(const OpContext& ctx, const ldf_column* table, int ncols, const std::vector<SortKeyDesc>& kd, int64_t n,
               int64_t first, int64_t rows, ldf_column* out);

// rank[d] = bytewise rank of the string of row repr[d] among the D distinct
// strings of rows repr[0..D), for D of at most kRankStrings; longest: bytes of
// the longest of them.
constexpr int64_t kRankStrings = 8192;
void rank_distinct_strings(const OpContext& ctx, const DCol& col, const int32_t* repr, int64_t D, int64_t longest,
                           uint32_t* rank);

}  // namespace ldf
