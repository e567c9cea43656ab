// Onesweep LSD radix sort (Adinets & Merrill, "Onesweep", 2022) of row ids by
// 8-bit digits, stable.  One upfront kernel builds the digit histograms of all
// passes from the unpermuted columns (histograms do not depend on order); each
// pass is then ONE kernel: tile load -> warp-level stable ranking (peer lanes
// from one ballot per digit bit) -> per-digit decoupled look-back across
// tiles -> tile staged in shared memory in digit order -> coalesced runs
// written out.  Passes whose digit is constant over all rows are skipped from
// the histograms.
#include "radix.cuh"

#include <algorithm>

namespace ldf {
namespace {

constexpr int RT    = kRadixThreads;
constexpr int RW    = RT / 32;

// Rows per thread of a onesweep tile, and the resident CTAs per SM its
// registers are sized for.  A pass on carried words gains from large tiles
// (fewer look-backs and barriers per row): when first measured, one carried pass
// over 100M rows took 0.94 / 0.84 / 0.82 ms with 12 / 16 / 20 rows of 4-byte
// words (0.65 ms now, with 4-byte status words and full tiles loaded without
// bounds), and 8-byte words were fastest with 16 (20 spill).  Passes that load their word from the
// columns hold more per row and stay at 12.
template <bool GATHER, typename KT, typename VT>
__host__ __device__ constexpr int radix_items()
{
  return GATHER || sizeof(VT) == 8 ? kRadixItems : sizeof(KT) == 4 ? 20 : 16;
}
template <bool GATHER>
__host__ __device__ constexpr int radix_min_blocks()
{
  return GATHER ? kRadixMinBlocks : 3;
}

__device__ __forceinline__ uint64_t bucket_word(const RadixPass& p, int64_t row)
{
  return key_bits<KeyMode::GEN>(p.hash_keys, row) % p.nparts;
}

__device__ __forceinline__ uint64_t pass_word(const RadixPass& p, int64_t row)
{
  if (p.src == DigitSrc::BUCKET) return bucket_word(p, row);
  return sort_word(p.key, row);
}

// Adds a fused-word component v placed at bit `off` of W to C = W >> 8 and
// to W's low byte (components do not overlap, so OR adds them).  Since W has
// at most 72 bits, v << (off - 8) fits C.
__device__ __forceinline__ void fused_add(uint64_t v, int off, uint64_t& c, uint32_t& low)
{
  if (v == 0) return;  // also every component of no bits, whose `off` may reach 72
  if (off >= 8) {
    c |= v << (off - 8);
  } else {
    c |= v >> (8 - off);
    low |= static_cast<uint32_t>(v << off) & 0xffu;
  }
}

__device__ __forceinline__ bool is_nan_raw(int type, uint64_t raw)
{
  if (type == LDF_FLOAT64)
    return (raw & 0x7ff0000000000000ull) == 0x7ff0000000000000ull && (raw & 0x000fffffffffffffull) != 0;
  if (type == LDF_FLOAT32) return (raw & 0x7f800000u) == 0x7f800000u && (raw & 0x007fffffu) != 0;
  return false;
}

// code_k of a row from its raw value: values in order, NaNs next to them and
// nulls outermost, both behind (nulls_at_end) or before the values.
__device__ __forceinline__ uint64_t fused_code(const FusedKey& f, int k, uint64_t raw, bool valid)
{
  const SortKeyDesc& d = f.key[k];
  if (!f.has_class[k]) return sort_word_of(d, raw, true) - f.min[k];
  if (!valid) return d.nulls_at_end ? f.span[k] + 2 : 0;
  if (is_nan_raw(d.col.type, raw)) return d.nulls_at_end ? f.span[k] + 1 : 1;
  return sort_word_of(d, raw, true) - f.min[k] + (d.nulls_at_end ? 0 : 2);
}

// C = W >> 8 of the fused word W of a row (FusedKey); *low = W's low byte.
__device__ __forceinline__ uint64_t fused_word(const FusedKey& f, int64_t row, uint32_t& low)
{
  uint64_t c = 0;
  low        = 0;
#pragma unroll
  for (int k = 0; k < kFuseMax; ++k)
    if (k < f.n) fused_add(fused_code(f, k, dbits(f.key[k].col, row), dvalid(f.key[k].col, row)), f.off[k], c, low);
  return c;
}

constexpr int kHistPassesPerLaunch = 16;
struct HistArgs {
  int npasses;
  uint32_t reuse;  // bit q: pass q reads the same key word as pass q - 1
  RadixPass p[kHistPassesPerLaunch];
  FusedKey fused;
  int64_t n;
  uint32_t* hist;  // [npasses][256]
};

// Raw bits of kHR rows of a column of width W, all loads in flight together.
constexpr int kHR = 4;
template <int W>
__device__ __forceinline__ void load_raw_rows(const DCol& c, const int64_t (&r)[kHR], int64_t n, uint64_t (&raw)[kHR],
                                              bool (&ok)[kHR])
{
#pragma unroll
  for (int j = 0; j < kHR; ++j) {
    raw[j] = 0;
    ok[j]  = false;
    if (r[j] >= n) continue;
    if (W == 1) raw[j] = __ldg(static_cast<const uint8_t*>(c.data) + r[j]);
    else if (W == 2) raw[j] = __ldg(static_cast<const uint16_t*>(c.data) + r[j]);
    else if (W == 4) raw[j] = __ldg(static_cast<const uint32_t*>(c.data) + r[j]);
    else raw[j] = __ldg(static_cast<const unsigned long long*>(c.data) + r[j]);
    ok[j] = c.valid == nullptr || __ldg(c.valid + r[j]) != 0;
  }
}

// All digit histograms of up to kHistPassesPerLaunch passes in one read of the
// columns: kHR rows per thread, each key word loaded once for all the passes
// over it (their loads in flight together), shared-memory counts.
template <bool FUSED>
__global__ void __launch_bounds__(RT) histogram_kernel(HistArgs a)
{
  __shared__ uint32_t sh[kHistPassesPerLaunch * 256];
  for (int i = threadIdx.x; i < a.npasses * 256; i += RT) sh[i] = 0;
  __syncthreads();
  const int64_t per_iter = static_cast<int64_t>(RT) * kHR;
  for (int64_t base = blockIdx.x * per_iter; base < a.n; base += static_cast<int64_t>(gridDim.x) * per_iter) {
    int64_t r[kHR];
#pragma unroll
    for (int j = 0; j < kHR; ++j) r[j] = base + j * RT + threadIdx.x;
    uint64_t w[kHR];
    uint32_t low[kHR];
#pragma unroll
    for (int j = 0; j < kHR; ++j) w[j] = 0, low[j] = 0;
    for (int q = 0; q < a.npasses; ++q) {
      const RadixPass& p = a.p[q];
      uint32_t d[kHR];
      if (p.src == DigitSrc::CLASS) {
#pragma unroll
        for (int j = 0; j < kHR; ++j) d[j] = r[j] < a.n ? class_digit(p.key, r[j]) : 256u;
      } else {
        if (!((a.reuse >> q) & 1u)) {
          if (p.src == DigitSrc::BUCKET) {
#pragma unroll
            for (int j = 0; j < kHR; ++j) w[j] = r[j] < a.n ? bucket_word(p, r[j]) : 0;
          } else if (FUSED && p.src == DigitSrc::FUSED) {
#pragma unroll
            for (int j = 0; j < kHR; ++j) w[j] = r[j] < a.n ? fused_word(a.fused, r[j], low[j]) : 0;
          } else {
            uint64_t raw[kHR];
            bool ok[kHR];
            switch (p.key.col.width) {
              case 1: load_raw_rows<1>(p.key.col, r, a.n, raw, ok); break;
              case 2: load_raw_rows<2>(p.key.col, r, a.n, raw, ok); break;
              case 4: load_raw_rows<4>(p.key.col, r, a.n, raw, ok); break;
              default: load_raw_rows<8>(p.key.col, r, a.n, raw, ok); break;
            }
#pragma unroll
            for (int j = 0; j < kHR; ++j) w[j] = sort_word_of(p.key, raw[j], ok[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < kHR; ++j)
          d[j] = r[j] < a.n ? ((FUSED && p.fused_low) ? low[j] : static_cast<uint32_t>(w[j] >> p.shift) & 0xffu)
                            : 256u;
      }
#pragma unroll
      for (int j = 0; j < kHR; ++j)
        if (d[j] < 256) atomicAdd(&sh[q * 256 + d[j]], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < a.npasses * 256; i += RT)
    if (sh[i]) atomicAdd(&a.hist[i], sh[i]);
}

struct PassArgs {
  RadixPass p;
  int64_t n;
  const void* keys_in;  // carried words, KT each
  void* keys_out;
  const void* vals_in;  // VT each: row ids (null: identity), or the rows' other values (radix_sort_pairs)
  void* vals_out;
  const uint64_t* digit_base;  // [256]
  uint32_t* status;            // [tiles * 256] (tile_status)
  unsigned long long* counter;
  int32_t* inv_out;  // != null: inv_out[row] = the row's output position
  RadixPayload pay;  // columns moved by this pass (payload_empty: none)
  FusedKey fused;    // FUSED passes
  int* err;
  // > 0: each tile stages in L2, by bulk prefetches, the rows of the tile
  // this many tiles ahead (about one wave of resident CTAs; tiles are taken
  // in order): the values (pf_vals) and carried words of a pass on the carried
  // word, and the key columns of a first pass over rows in input order
  // (pf_columns).
  int64_t pf_ahead;
  int pf_vals;
  int pf_columns;
};

// L2 prefetch of rows [lo, hi) of a fixed-width column and its validity.
__device__ __forceinline__ void prefetch_column(const DCol& c, int64_t lo, int64_t hi)
{
  if (c.type == LDF_STRING || c.data == nullptr) return;
  l2_prefetch_bulk(c.data, lo * c.width, hi * c.width);
  if (c.valid) l2_prefetch_bulk(c.valid, lo, hi);
}

// Rows of a thread whose payload loads are issued together in a pass that
// moves columns.
constexpr int kMoveBatch = 3;

// First 8-byte word of a row's string range; rows from 2^30 on pass 32 bits.
__host__ __device__ __forceinline__ int64_t range_word(int32_t row) { return 2 * static_cast<int64_t>(row); }

// dst[pos[k]] = src[row[k]] for 16-byte string ranges (8-byte aligned at the
// source: two 8-byte loads; the scratch destination is 16-byte aligned), every
// load issued before the first store.  pos < 0: no row.
__device__ __forceinline__ void move_ranges(const void* src, void* dst, const int32_t (&pos)[kMoveBatch],
                                            const int32_t (&row)[kMoveBatch])
{
  const unsigned long long* sp = static_cast<const unsigned long long*>(src);
  ulonglong2 v[kMoveBatch];
#pragma unroll
  for (int k = 0; k < kMoveBatch; ++k)
    if (pos[k] >= 0) {
      const unsigned long long* r = sp + range_word(row[k]);
      v[k]                        = make_ulonglong2(__ldg(r), __ldg(r + 1));
    }
#pragma unroll
  for (int k = 0; k < kMoveBatch; ++k)
    if (pos[k] >= 0) static_cast<ulonglong2*>(dst)[pos[k]] = v[k];
}

__device__ __forceinline__ unsigned long long ld_fixed(const DCol& c, int32_t row)
{
  switch (c.width) {
    case 1: return __ldg(static_cast<const uint8_t*>(c.data) + row);
    case 2: return __ldg(static_cast<const uint16_t*>(c.data) + row);
    case 4: return __ldg(static_cast<const uint32_t*>(c.data) + row);
    default: return __ldg(static_cast<const unsigned long long*>(c.data) + row);
  }
}

__device__ __forceinline__ void st_fixed(void* dst, int width, int64_t pos, unsigned long long v)
{
  switch (width) {
    case 1: static_cast<uint8_t*>(dst)[pos] = static_cast<uint8_t>(v); break;
    case 2: static_cast<uint16_t*>(dst)[pos] = static_cast<uint16_t>(v); break;
    case 4: static_cast<uint32_t*>(dst)[pos] = static_cast<uint32_t>(v); break;
    default: static_cast<unsigned long long*>(dst)[pos] = v; break;
  }
}

// Part of a packed payload record at byte offset `off` (the store truncates it
// to the part's width).
__device__ __forceinline__ unsigned long long record_part(const ulonglong2& r, int off)
{
  return (off < 8 ? r.x : r.y) >> ((off & 7) * 8);
}

// dst[pos] = src[row] for every payload column (one row: the identity copy).
__device__ __forceinline__ void move_payload(const RadixPayload& p, int64_t pos, int64_t row)
{
  if (p.nparts) {
    const ulonglong2 r = __ldg(p.packed + row);
    for (int k = 0; k < p.nparts; ++k) st_fixed(p.pdst[k], p.pwidth[k], pos, record_part(r, p.poff[k]));
  }
  for (int c = 0; c < p.n; ++c) {
    const DCol& sc = p.src[c];
    if (sc.width <= 8) {
      st_fixed(p.dst[c], sc.width, pos, ld_fixed(sc, static_cast<int32_t>(row)));
    } else {  // 16: string ranges (8-byte aligned at the source; the scratch is 16-byte aligned)
      const unsigned long long* r = static_cast<const unsigned long long*>(sc.data) + 2 * row;
      static_cast<ulonglong2*>(p.dst[c])[pos] = make_ulonglong2(__ldg(r), __ldg(r + 1));
    }
    if (p.dst_valid[c]) p.dst_valid[c][pos] = dvalid(sc, row) ? 1 : 0;
  }
}

// Every payload column's values (and masks) of kMoveBatch rows: the packed
// records first (one load per row for all their parts), then the other
// fixed-width columns with all their loads issued before the first store, so
// that their random rows are in flight together, then string ranges.
__device__ __forceinline__ void move_payload_rows(const RadixPayload& p, const int32_t (&pos)[kMoveBatch],
                                                  const int32_t (&row)[kMoveBatch])
{
  if (p.nparts) {
    ulonglong2 rv[kMoveBatch];
#pragma unroll
    for (int k = 0; k < kMoveBatch; ++k)
      if (pos[k] >= 0) rv[k] = __ldg(p.packed + row[k]);
#pragma unroll
    for (int k = 0; k < kMoveBatch; ++k)
      if (pos[k] >= 0)
        for (int q = 0; q < p.nparts; ++q) st_fixed(p.pdst[q], p.pwidth[q], pos[k], record_part(rv[k], p.poff[q]));
  }
  unsigned long long v[kPassPayload][kMoveBatch];
#pragma unroll
  for (int c = 0; c < kPassPayload; ++c)
    if (c < p.n && p.src[c].width <= 8) {
#pragma unroll
      for (int k = 0; k < kMoveBatch; ++k) v[c][k] = pos[k] >= 0 ? ld_fixed(p.src[c], row[k]) : 0;
    }
#pragma unroll
  for (int c = 0; c < kPassPayload; ++c)
    if (c < p.n && p.src[c].width <= 8) {
#pragma unroll
      for (int k = 0; k < kMoveBatch; ++k)
        if (pos[k] >= 0) st_fixed(p.dst[c], p.src[c].width, pos[k], v[c][k]);
    }
  for (int c = 0; c < p.n; ++c) {
    const DCol& sc = p.src[c];
    if (sc.width > 8) move_ranges(sc.data, p.dst[c], pos, row);
    if (p.dst_valid[c]) {
      uint8_t m[kMoveBatch];
#pragma unroll
      for (int k = 0; k < kMoveBatch; ++k) m[k] = pos[k] >= 0 && dvalid(sc, row[k]) ? 1 : 0;
#pragma unroll
      for (int k = 0; k < kMoveBatch; ++k)
        if (pos[k] >= 0) p.dst_valid[c][pos[k]] = m[k];
    }
  }
}

// Predecessor tiles whose status words one look-back round trip loads.
constexpr int kLookback = 4;

// Status word of one digit of a tile: 0 not ready; a tile's own count + 1 (top
// bit clear); the count of the tile and all before it, with the top bit set
// (fewer than 2^31 rows).
constexpr uint32_t kTilePrefix = 0x80000000u;
__device__ __forceinline__ uint32_t ld_status(const uint32_t* p)
{
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Each word stands for itself (no other data is read on the strength of it).
__device__ __forceinline__ void st_status(uint32_t* p, uint32_t v)
{
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Shared state of one onesweep tile.
struct OsShared {
  uint32_t whist[RW][256];  // per-warp digit counts, then tile-local positions
  int32_t delta[256];        // output position of staged row j of digit d: delta[d] + j
  uint32_t scan[RW + 1];
  int64_t tile[2];
};

// Lanes of the warp whose digit equals this lane's: one ballot per digit bit,
// each lane keeping the lanes that agree with it on that bit.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d)
{
  uint32_t peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const uint32_t bit = (d >> b) & 1u;
    const uint32_t set = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? set : ~set;
  }
  return peers;
}

// Everything of one pass over one tile after its rows are in registers:
// key[i] / val[i] / dr[i] (digit) of item i of this thread, item order (warp,
// i, lane).  Items past the last row, at the end of the last tile, count as
// rows of digit 255: they land behind the tile's rows and are not written.
// Stable warp-level ranking, the tile's digit counts published at once,
// tile-local scan, rows staged in digit order into s_keys / s_vals / s_dig
// (tile-local positions need no look-back), per-digit decoupled look-back, then
// coalesced runs written out.  sh.whist must be zero on entry.  Ends with every
// thread past its reads of the staging arrays.
//
// The bound of a pass on carried words is its instructions (about 140 per row
// and warp, half the issue slots; DRAM 25 %), most of them the ranking.
template <bool WRITE_KEYS, bool MOVE, typename KT, typename VT, int RI>
__device__ __forceinline__ void rank_and_scatter(const PassArgs& a, int64_t tile, KT (&key)[RI],
                                                 VT (&val)[RI], uint32_t (&dr)[RI], OsShared& sh,
                                                 KT* s_keys, VT* s_vals, uint8_t* s_dig)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lt_mask = (1u << lane) - 1u;
  // stable warp-level ranking, items in (i, lane) order
  uint32_t* whist = sh.whist[warp];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const uint32_t d     = dr[i];
    const uint32_t peers = digit_peers(d);
    const uint32_t rank  = __popc(peers & lt_mask);
    const uint32_t base  = whist[d];
    __syncwarp();
    if (rank == 0) whist[d] = base + __popc(peers);
    __syncwarp();
    dr[i] = d | ((base + rank) << 8);
  }
  __syncthreads();
  // per-digit warp prefixes and tile counts (thread t owns digit t); the
  // counts are published before anything else, so that the tiles after this one
  // can finish their look-back while it stages its rows
  const int t = threadIdx.x;
  uint32_t run = 0, count[RW];
#pragma unroll
  for (int w = 0; w < RW; ++w) {
    count[w] = sh.whist[w][t];
    run += count[w];
  }
  uint32_t* st = a.status;
  if (tile == 0) st_status(&st[t], kTilePrefix | run);
  else st_status(&st[tile * 256 + t], run + 1);
  uint32_t tile_total;
  const uint32_t start = block_exclusive_scan<uint32_t, RT>(run, sh.scan, &tile_total);
  {
    uint32_t at = start;
#pragma unroll
    for (int w = 0; w < RW; ++w) {
      sh.whist[w][t] = at;  // tile-local position of the warp's first row of the digit
      at += count[w];
    }
  }
  __syncthreads();
  // stage the tile in digit order
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const uint32_t d  = dr[i] & 0xffu;
    const uint32_t lp = whist[d] + (dr[i] >> 8);
    if (WRITE_KEYS) s_keys[lp] = key[i];
    s_vals[lp] = val[i];
    s_dig[lp]  = static_cast<uint8_t>(d);
  }
  // per-digit decoupled look-back, kLookback predecessors' status words
  // loaded together per round trip
  {
    uint32_t excl = 0;
    if (tile > 0) {
      int64_t j      = tile - 1;  // next predecessor to fold in
      uint32_t spins = 0;
      while (j >= 0) {
        uint32_t sv[kLookback];
#pragma unroll
        for (int w = 0; w < kLookback; ++w) sv[w] = j - w >= 0 ? ld_status(&st[(j - w) * 256 + t]) : kTilePrefix;
        int used  = 0;
        bool done = false, stall = false;
#pragma unroll
        for (int w = 0; w < kLookback; ++w) {
          if (done || stall) continue;
          if (sv[w] == 0) {
            stall = true;
            continue;
          }
          done = (sv[w] & kTilePrefix) != 0;
          excl += done ? sv[w] & ~kTilePrefix : sv[w] - 1;
          ++used;
        }
        if (done) break;
        j -= used;
        if (stall) {
          if (++spins > kSpinLimit) {
            atomicExch(a.err, LDF_ERR_TIMEOUT);
            break;
          }
          __nanosleep(32);
        }
      }
      st_status(&st[tile * 256 + t], kTilePrefix | (excl + run));
    }
    // positions fit 32 bits (fewer than 2^31 rows)
    sh.delta[t] = static_cast<int32_t>(a.digit_base[t] + excl) - static_cast<int32_t>(start);
  }
  __syncthreads();
  constexpr int RTILE = RT * RI;
  const int64_t tbase = tile * RTILE;
  const int cnt       = static_cast<int>(a.n - tbase < RTILE ? a.n - tbase : RTILE);
  if constexpr (!MOVE) {
#pragma unroll 4
    for (int j = threadIdx.x; j < cnt; j += RT) {
      const int32_t pos = sh.delta[s_dig[j]] + j;
      if (WRITE_KEYS) static_cast<KT*>(a.keys_out)[pos] = s_keys[j];
      static_cast<VT*>(a.vals_out)[pos] = s_vals[j];
      if (a.inv_out) a.inv_out[s_vals[j]] = static_cast<int32_t>(pos);
    }
  } else {
    // a pass that moves columns: kMoveBatch rows of a thread at a time, so the
    // payload's loads (random rows after the first pass) overlap.  Positions
    // and rows fit 32 bits (fewer than 2^31 rows).
    for (int j0 = threadIdx.x; j0 < cnt; j0 += RT * kMoveBatch) {
      int32_t pos[kMoveBatch], row[kMoveBatch];
#pragma unroll
      for (int k = 0; k < kMoveBatch; ++k) {
        const int j = j0 + k * RT;
        pos[k]      = -1;
        row[k]      = 0;
        if (j < cnt) {
          pos[k]           = sh.delta[s_dig[j]] + j;
          row[k]           = static_cast<int32_t>(s_vals[j]);
          static_cast<int32_t*>(a.vals_out)[pos[k]] = row[k];
          if (a.inv_out) a.inv_out[row[k]] = pos[k];
        }
      }
      move_payload_rows(a.pay, pos, row);
    }
  }
}

// Rows of a tile straight from global memory (GATHER: the word is loaded from
// the columns at the row, the first pass of a word; otherwise the carried key).
// In a pass on the carried word, all row ids and then all words are loaded
// before any digit is taken, so that the thread's loads are in flight together.
template <bool GATHER, bool FUSEDG, typename KT, typename VT, int RI>
__device__ __forceinline__ void load_tile_rows(const PassArgs& a, int64_t tile, KT (&key)[RI],
                                               VT (&val)[RI], uint32_t (&dr)[RI])
{
  const VT* vals_in = static_cast<const VT*>(a.vals_in);
  constexpr int RTILE = RT * RI;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t wbase = tile * RTILE + warp * (32 * RI) + lane;
  if (!GATHER && a.p.src != DigitSrc::CLASS && (tile + 1) * RTILE <= a.n) {  // a full tile: no bounds
    const KT* k = static_cast<const KT*>(a.keys_in) + wbase;
    if (vals_in) {
      const VT* v = vals_in + wbase;
#pragma unroll
      for (int i = 0; i < RI; ++i) val[i] = __ldg(v + i * 32);
    } else {
#pragma unroll
      for (int i = 0; i < RI; ++i) val[i] = static_cast<VT>(wbase) + i * 32;
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) key[i] = __ldg(k + i * 32);
#pragma unroll
    for (int i = 0; i < RI; ++i) dr[i] = static_cast<uint32_t>(key[i] >> a.p.shift) & 0xffu;
    return;
  }
  if (!GATHER && a.p.src != DigitSrc::CLASS) {
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int64_t idx = wbase + i * 32;
      val[i] = idx < a.n ? (vals_in ? __ldg(vals_in + idx) : static_cast<VT>(idx)) : 0;
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int64_t idx = wbase + i * 32;
      key[i] = idx < a.n ? __ldg(static_cast<const KT*>(a.keys_in) + idx) : KT(0);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i)
      dr[i] = wbase + i * 32 < a.n ? static_cast<uint32_t>(key[i] >> a.p.shift) & 0xffu : 255u;
    return;
  }
  if (FUSEDG) {
    // the fused word from its key columns, one column at a time with the
    // items' loads in flight together; dr[i] gathers W's low byte
    uint64_t c[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int64_t idx = wbase + i * 32;
      val[i] = idx < a.n ? (vals_in ? __ldg(vals_in + idx) : static_cast<VT>(idx)) : -1;
      c[i]   = 0;
      dr[i]  = 0;
    }
    for (int k = 0; k < a.fused.n; ++k) {
      const SortKeyDesc& kk = a.fused.key[k];
      uint64_t raw[RI];
      uint32_t ok = 0;
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        raw[i] = 0;
        if (val[i] < 0) continue;
        switch (kk.col.width) {
          case 1: raw[i] = __ldg(static_cast<const uint8_t*>(kk.col.data) + val[i]); break;
          case 2: raw[i] = __ldg(static_cast<const uint16_t*>(kk.col.data) + val[i]); break;
          case 4: raw[i] = __ldg(static_cast<const uint32_t*>(kk.col.data) + val[i]); break;
          default: raw[i] = __ldg(static_cast<const unsigned long long*>(kk.col.data) + val[i]); break;
        }
        if (dvalid(kk.col, val[i])) ok |= 1u << i;
      }
#pragma unroll
      for (int i = 0; i < RI; ++i)
        if (val[i] >= 0) fused_add(fused_code(a.fused, k, raw[i], (ok >> i) & 1u), a.fused.off[k], c[i], dr[i]);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      key[i] = static_cast<KT>(c[i]);
      if (val[i] < 0) {
        val[i] = 0;
        dr[i]  = 255;
      } else if (!a.p.fused_low) {
        dr[i] = static_cast<uint32_t>(c[i] >> a.p.shift) & 0xffu;
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int64_t idx = wbase + i * 32;
    key[i]            = 0;
    val[i]            = 0;
    dr[i]             = 255;
    if (idx < a.n) {
      const int64_t row = vals_in ? vals_in[idx] : idx;
      val[i]            = static_cast<VT>(row);
      if (a.p.src == DigitSrc::CLASS) {
        dr[i] = class_digit(a.p.key, row);
      } else {
        key[i] = static_cast<KT>(GATHER ? pass_word(a.p, row) : static_cast<const KT*>(a.keys_in)[idx]);
        dr[i]  = static_cast<uint32_t>(key[i] >> a.p.shift) & 0xffu;
      }
    }
  }
}

// Whether a onesweep tile prefetches the rows of the tile one wave of resident
// CTAs ahead into L2 (LDF_B200_L2_PREFETCH=0 turns it off).
bool prefetch_ahead()
{
  static const bool on = [] {
    const char* e = std::getenv("LDF_B200_L2_PREFETCH");
    return e == nullptr || std::atoi(e) != 0;
  }();
  return on;
}
// Whether a first pass over rows in input order prefetches its key columns
// (LDF_B200_L2_PREFETCH_FIRST=0 turns it off).
int prefetch_first_pass()
{
  static const bool off = [] {
    const char* e = std::getenv("LDF_B200_L2_PREFETCH_FIRST");
    return e != nullptr && std::atoi(e) == 0;
  }();
  return off ? 0 : 1;
}

// Whether p points into device memory (not pinned host or managed memory, as
// a zero-copy legate store would be): the first pass prefetches only columns
// held there.
bool on_device(const void* p)
{
  if (p == nullptr) return true;
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice;
}
bool column_on_device(const DCol& c) { return on_device(c.data) && on_device(c.valid); }

// Whether pass k prefetches the rows' values: later passes read scratch, the
// first one `vals`, which may be a column of the caller (null: row ids).
template <typename F>
int prefetch_values(size_t pass, const void* vals, F device)
{
  return pass > 0 || (vals != nullptr && prefetch_first_pass() != 0 && device(vals)) ? 1 : 0;
}

// The key columns the first pass of `p` reads in row order are all in
// device memory.
bool pass_columns_on_device(const RadixPass& p, const FusedKey* fused)
{
  if (p.src == DigitSrc::FUSED) {
    if (fused == nullptr) return false;
    for (int k = 0; k < fused->n; ++k)
      if (!column_on_device(fused->key[k].col)) return false;
    return true;
  }
  if (p.src == DigitSrc::BUCKET) {
    for (int k = 0; k < p.hash_keys.n; ++k)
      if (!column_on_device(p.hash_keys.c[k])) return false;
    return true;
  }
  return column_on_device(p.key.col);
}

// One tile per CTA.  WRITE_KEYS: later passes of the same word follow (or the
// sorted words are wanted), so carry the word along.  MOVE: the pass also
// moves a.pay's columns (the last pass only, which carries no word).  KT: the
// carried word, 4 bytes when that holds it: 8 instead of 12 bytes a row read
// and written in every pass.
template <bool GATHER, bool WRITE_KEYS, bool MOVE, bool FUSEDG, typename KT, typename VT>
__global__ void __launch_bounds__(RT, radix_min_blocks<GATHER>()) onesweep_kernel(PassArgs a)
{
  constexpr int RI    = radix_items<GATHER, KT, VT>();
  constexpr int RTILE = RT * RI;
  __shared__ OsShared sh;
  // staged tile (dynamic): [keys KT x RTILE when carried][values VT x RTILE][digits u8 x RTILE]
  extern __shared__ __align__(16) unsigned char s_stage[];
  KT* s_keys      = reinterpret_cast<KT*>(s_stage);
  VT* s_vals      = reinterpret_cast<VT*>(s_stage + (WRITE_KEYS ? RTILE * sizeof(KT) : 0));
  uint8_t* s_dig  = reinterpret_cast<uint8_t*>(s_vals + RTILE);

  const int64_t tile = next_tile_id(a.counter, &sh.tile[0]);
  for (int i = threadIdx.x; i < RW * 256; i += RT) (&sh.whist[0][0])[i] = 0;
  __syncthreads();
  KT key[RI];
  VT val[RI];
  uint32_t dr[RI];
  if (a.pf_ahead > 0 && threadIdx.x == 0 && (tile + a.pf_ahead) * RTILE < a.n) {
    const int64_t lo = (tile + a.pf_ahead) * RTILE;
    const int64_t hi = min(lo + static_cast<int64_t>(RTILE), a.n);
    if (!GATHER) {
      constexpr int64_t vb = sizeof(VT);
      if (a.pf_vals && a.vals_in) l2_prefetch_bulk(a.vals_in, lo * vb, hi * vb);
      if (a.p.src != DigitSrc::CLASS)
        l2_prefetch_bulk(a.keys_in, lo * static_cast<int64_t>(sizeof(KT)), hi * static_cast<int64_t>(sizeof(KT)));
    } else if (a.pf_columns && a.vals_in == nullptr) {  // rows in input order: the key columns are read in order
      if (FUSEDG) {
        for (int k = 0; k < a.fused.n; ++k) prefetch_column(a.fused.key[k].col, lo, hi);
      } else if (a.p.src == DigitSrc::BUCKET) {
        for (int k = 0; k < a.p.hash_keys.n; ++k) prefetch_column(a.p.hash_keys.c[k], lo, hi);
      } else {
        prefetch_column(a.p.key.col, lo, hi);
      }
    }
  }
  load_tile_rows<GATHER, FUSEDG, KT, VT, RI>(a, tile, key, val, dr);
  rank_and_scatter<WRITE_KEYS, MOVE, KT, VT, RI>(a, tile, key, val, dr, sh, s_keys, s_vals, s_dig);
}

// Runs the pass over a.n rows; clears the status words and the tile counter
// behind them first.
template <bool GATHER, bool WRITE_KEYS, bool MOVE = false, bool FUSEDG = false, typename KT = uint64_t,
          typename VT = int32_t>
void launch_onesweep(cudaStream_t s, PassArgs& a)
{
  static_assert(!(MOVE && WRITE_KEYS), "the pass that moves columns is the last one");
  constexpr int64_t tile_rows = RT * radix_items<GATHER, KT, VT>();
  constexpr size_t smem = (WRITE_KEYS ? tile_rows * sizeof(KT) : 0) + tile_rows * (sizeof(VT) + 1);
  const int64_t tiles   = ceil_div(a.n, tile_rows);
  auto kernel           = onesweep_kernel<GATHER, WRITE_KEYS, MOVE, FUSEDG, KT, VT>;
  a.counter             = reinterpret_cast<unsigned long long*>(a.status + tiles * 256);
  a.pf_ahead            = prefetch_ahead() ? int64_t(num_sms()) * radix_min_blocks<GATHER>() : 0;
  LDF_CUDA(cudaMemsetAsync(a.status, 0, (tiles * 256 + 2) * sizeof(uint32_t), s));
  LDF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  // profile names: a pass that loads its word from the columns, one that
  // moves the payload columns, the others
  const char* name = MOVE ? "onesweep_move" : (GATHER ? "onesweep_gather" : "onesweep");
  launch(name, kernel, static_cast<unsigned>(tiles), RT, smem, s, a);
}

// Status words of a pass, of the smallest tiles (the counter's included).
int64_t status_words(int64_t n) { return ceil_div(n, int64_t(kRadixTile)) * 256 + 2; }

// Identity order: the payload columns copied as they are.
__global__ void copy_payload_kernel(RadixPayload p, int64_t n)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    move_payload(p, i, i);
}

__global__ void iota_kernel(int32_t* p, int64_t n)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = static_cast<int32_t>(i);
}

unsigned hblocks(int64_t n)
{
  int64_t b   = ceil_div(n, RT);
  int64_t cap = static_cast<int64_t>(num_sms()) * 4;
  return static_cast<unsigned>(b < 1 ? 1 : (b > cap ? cap : b));
}

// Histogram grid: one block per RT * kHR rows, at most five resident per SM.
unsigned hist_blocks(int64_t n)
{
  int64_t b   = ceil_div(n, static_cast<int64_t>(RT) * kHR);
  int64_t cap = static_cast<int64_t>(num_sms()) * 5;
  return static_cast<unsigned>(b < 1 ? 1 : (b > cap ? cap : b));
}

// Two passes belong to the same carried word when they read the same column
// transform (or bucket) and differ only in shift.
bool same_word(const RadixPass& a, const RadixPass& b)
{
  if (a.src != b.src || a.src == DigitSrc::CLASS) return false;
  if (a.src == DigitSrc::BUCKET || a.src == DigitSrc::FUSED || a.src == DigitSrc::CARRIED) return true;
  return a.key.col.data == b.key.col.data && a.key.descending == b.key.descending;
}

struct WordRangeArgs {
  int n;
  SortKeyDesc key[kFuseMax];
};

// mm[2k] = min, mm[2k + 1] = max of key k's words (init ~0 and 0).  Eight
// rows per thread, one key column at a time, loads in flight together.
constexpr int kRangeRows = 8;
__global__ void __launch_bounds__(256) word_range_kernel(WordRangeArgs a, int64_t n, unsigned long long* mm)
{
  unsigned long long lo[kFuseMax], hi[kFuseMax];
#pragma unroll
  for (int k = 0; k < kFuseMax; ++k) lo[k] = ~0ull, hi[k] = 0;
  const int64_t per_iter = static_cast<int64_t>(blockDim.x) * kRangeRows;
  for (int64_t base = blockIdx.x * per_iter; base < n; base += static_cast<int64_t>(gridDim.x) * per_iter) {
#pragma unroll
    for (int k = 0; k < kFuseMax; ++k) {
      if (k >= a.n) continue;
      const DCol& c = a.key[k].col;
      uint64_t raw[kRangeRows];
      uint32_t ok = 0;
#pragma unroll
      for (int j = 0; j < kRangeRows; ++j) {
        const int64_t r = base + j * blockDim.x + threadIdx.x;
        raw[j]          = 0;
        if (r >= n) continue;
        switch (c.width) {
          case 1: raw[j] = __ldg(static_cast<const uint8_t*>(c.data) + r); break;
          case 2: raw[j] = __ldg(static_cast<const uint16_t*>(c.data) + r); break;
          case 4: raw[j] = __ldg(static_cast<const uint32_t*>(c.data) + r); break;
          default: raw[j] = __ldg(static_cast<const unsigned long long*>(c.data) + r); break;
        }
        if (dvalid(c, r)) ok |= 1u << j;
      }
#pragma unroll
      for (int j = 0; j < kRangeRows; ++j) {
        if (base + j * blockDim.x + threadIdx.x >= n) continue;
        if (!((ok >> j) & 1u) || is_nan_raw(c.type, raw[j])) continue;
        const unsigned long long w = sort_word_of(a.key[k], raw[j], true);
        lo[k]                      = w < lo[k] ? w : lo[k];
        hi[k]                      = w > hi[k] ? w : hi[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kFuseMax; ++k) {
    if (k >= a.n) continue;
    for (int d = 16; d > 0; d >>= 1) {
      const unsigned long long l = __shfl_xor_sync(0xffffffffu, lo[k], d);
      const unsigned long long h = __shfl_xor_sync(0xffffffffu, hi[k], d);
      lo[k]                      = l < lo[k] ? l : lo[k];
      hi[k]                      = h > hi[k] ? h : hi[k];
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(mm + 2 * k, lo[k]);
      atomicMax(mm + 2 * k + 1, hi[k]);
    }
  }
}

}  // namespace

void sort_word_ranges(const OpContext& ctx, const SortKeyDesc* keys, int nkeys, int64_t n, uint64_t* mn,
                      uint64_t* mx)
{
  LDF_REQUIRE(nkeys >= 1 && nkeys <= kFuseMax, "sort_word_ranges: too many keys");
  cudaStream_t s = ctx.stream();
  Buffer<unsigned long long> mm(ctx.alloc(), 2 * kFuseMax);
  std::vector<unsigned long long> h(2 * kFuseMax);
  for (int k = 0; k < kFuseMax; ++k) h[2 * k] = ~0ull, h[2 * k + 1] = 0;
  LDF_CUDA(cudaMemcpyAsync(mm.get(), h.data(), h.size() * 8, cudaMemcpyHostToDevice, s));
  WordRangeArgs a{};
  a.n = nkeys;
  for (int k = 0; k < nkeys; ++k) a.key[k] = keys[k];
  if (n > 0)
    launch("word_range", word_range_kernel,
           static_cast<unsigned>(std::min<int64_t>(ceil_div(n, int64_t(256) * kRangeRows), 8 * num_sms())), 256, 0, s, a,
           n, mm.get());
  ctx.fetch(h.data(), mm.get(), h.size() * 8);
  ctx.finish();
  for (int k = 0; k < nkeys; ++k) {
    mn[k] = h[2 * k];
    mx[k] = h[2 * k + 1];
  }
}

void radix_histograms(const OpContext& ctx, const std::vector<RadixPass>& passes, int64_t n,
                      uint32_t* d_hist, const FusedKey* fused)
{
  cudaStream_t s = ctx.stream();
  LDF_CUDA(cudaMemsetAsync(d_hist, 0, passes.size() * 256 * sizeof(uint32_t), s));
  for (size_t b = 0; b < passes.size(); b += kHistPassesPerLaunch) {
    HistArgs h{};
    h.npasses = static_cast<int>(std::min<size_t>(kHistPassesPerLaunch, passes.size() - b));
    for (int q = 0; q < h.npasses; ++q) {
      h.p[q] = passes[b + q];
      if (q > 0 && same_word(passes[b + q - 1], passes[b + q])) h.reuse |= 1u << q;
    }
    if (fused) h.fused = *fused;
    h.n    = n;
    h.hist = d_hist + b * 256;
    if (n > 0 && fused) launch("histogram", histogram_kernel<true>, hist_blocks(n), RT, 0, s, h);
    else if (n > 0) launch("histogram", histogram_kernel<false>, hist_blocks(n), RT, 0, s, h);
    LDF_CHECK_LAUNCH();
  }
}

namespace {

// Writes the word W >> drop (KT) of every row and counts all its digits: one
// read of the key columns, kWordRows rows a thread with a column's loads in
// flight together.
constexpr int kWordRows = 4;
struct WordArgs {
  FusedKey f;
  int64_t n;
  int npasses;
  void* words;
  uint32_t* hist;  // [npasses][256]
};
template <typename KT>
__global__ void __launch_bounds__(RT) fused_words_kernel(WordArgs a)
{
  __shared__ uint32_t sh[sizeof(KT) * 256];
  for (int i = threadIdx.x; i < a.npasses * 256; i += RT) sh[i] = 0;
  __syncthreads();
  const int64_t per_iter = static_cast<int64_t>(RT) * kWordRows;
  for (int64_t base = blockIdx.x * per_iter; base < a.n; base += static_cast<int64_t>(gridDim.x) * per_iter) {
    uint64_t c[kWordRows];
    uint32_t low[kWordRows];
#pragma unroll
    for (int j = 0; j < kWordRows; ++j) c[j] = 0, low[j] = 0;
    for (int k = 0; k < a.f.n; ++k) {
      const DCol& col = a.f.key[k].col;
      uint64_t raw[kWordRows];
      bool ok[kWordRows];
#pragma unroll
      for (int j = 0; j < kWordRows; ++j) {
        const int64_t r = base + j * RT + threadIdx.x;
        raw[j]          = r < a.n ? dbits_stream(col, r) : 0;
        ok[j]           = r < a.n && dvalid_stream(col, r);
      }
#pragma unroll
      for (int j = 0; j < kWordRows; ++j)
        if (base + j * RT + threadIdx.x < a.n) fused_add(fused_code(a.f, k, raw[j], ok[j]), a.f.off[k], c[j], low[j]);
    }
#pragma unroll
    for (int j = 0; j < kWordRows; ++j) {
      const int64_t r = base + j * RT + threadIdx.x;
      if (r >= a.n) continue;
      const KT w = static_cast<KT>(a.f.drop ? c[j] >> (a.f.drop - 8) : c[j] << 8 | low[j]);
      static_cast<KT*>(a.words)[r] = w;
      for (int q = 0; q < a.npasses; ++q) atomicAdd(&sh[q * 256 + (static_cast<uint32_t>(w >> (8 * q)) & 0xffu)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < a.npasses * 256; i += RT)
    if (sh[i]) atomicAdd(&a.hist[i], sh[i]);
}

// The passes `run` (none of a constant digit) of `passes`, in order; hist: all
// passes' digit counts.  first_words: the word that the first pass carries
// (null: it is loaded from the columns), kb bytes.  first_vals: the rows' values
// of vb bytes (null: their ids), which go to `perm` in the end.
void run_passes(const OpContext& ctx, const std::vector<RadixPass>& passes, const std::vector<int>& run,
                const std::vector<uint32_t>& hist, int64_t n, void* perm, int32_t* inv, const RadixPayload* payload,
                const FusedKey* fused, Buffer<uint8_t>* first_words, size_t kb, Buffer<uint8_t>* words,
                const void* first_vals = nullptr, size_t vb = 4)
{
  const Allocator& al = ctx.alloc();
  cudaStream_t s      = ctx.stream();
  std::vector<uint64_t> bases(run.size() * 256);
  for (size_t k = 0; k < run.size(); ++k) {
    uint64_t acc = 0;
    for (int d = 0; d < 256; ++d) {
      bases[k * 256 + d] = acc;
      acc += hist[run[k] * 256 + d];
    }
  }
  Buffer<uint64_t> d_bases(al, bases.size());
  LDF_CUDA(cudaMemcpyAsync(d_bases.get(), bases.data(), bases.size() * 8, cudaMemcpyHostToDevice, s));

  Buffer<uint32_t> status(al, status_words(n));
  Buffer<uint8_t> keys[2] = {Buffer<uint8_t>(al, n * kb), first_words ? std::move(*first_words) : Buffer<uint8_t>(al, n * kb)};
  Buffer<uint8_t> vals_tmp(al, n * vb);
  // ping-pong so that the last pass writes into `perm`
  void* vbuf[2];
  const bool odd = run.size() % 2 == 1;
  vbuf[0]        = odd ? perm : vals_tmp.get();
  vbuf[1]        = odd ? vals_tmp.get() : perm;
  const void* vin = first_vals;
  const void* kin    = first_words ? keys[1].get() : nullptr;
  for (size_t k = 0; k < run.size(); ++k) {
    const RadixPass& p    = passes[run[k]];
    const bool last       = k + 1 == run.size();
    const bool gather     = p.src != DigitSrc::CARRIED && (k == 0 || !same_word(passes[run[k - 1]], p));
    const bool write_keys = p.src != DigitSrc::CLASS && (last ? words != nullptr : same_word(p, passes[run[k + 1]]));
    PassArgs a{};
    a.p          = p;
    a.n          = n;
    a.keys_in    = kin;
    a.keys_out   = keys[k % 2].get();
    a.vals_in    = vin;
    a.vals_out   = vbuf[k % 2];
    a.digit_base = d_bases.get() + k * 256;
    a.status     = status.get();
    a.inv_out    = last ? inv : nullptr;
    if (last && payload) a.pay = *payload;
    if (fused) a.fused = *fused;
    a.err        = ctx.err();
    a.pf_vals    = prefetch_values(k, first_vals, on_device);
    a.pf_columns = gather && k == 0 && prefetch_first_pass() && pass_columns_on_device(p, fused) ? 1 : 0;
    const bool move = !payload_empty(a.pay);
    if (vb == 8) {
      launch_onesweep<false, true, false, false, uint64_t, int64_t>(s, a);
    } else if (kb == 4) {
      if (move) launch_onesweep<false, false, true, false, uint32_t>(s, a);
      else if (write_keys) launch_onesweep<false, true, false, false, uint32_t>(s, a);
      else launch_onesweep<false, false, false, false, uint32_t>(s, a);
    } else if (gather && p.src == DigitSrc::FUSED) {  // the fused word's first pass
      if (move) launch_onesweep<true, false, true, true>(s, a);
      else if (write_keys) launch_onesweep<true, true, false, true>(s, a);
      else launch_onesweep<true, false, false, true>(s, a);
    } else if (move && gather) launch_onesweep<true, false, true>(s, a);
    else if (move) launch_onesweep<false, false, true>(s, a);
    else if (gather && write_keys) launch_onesweep<true, true>(s, a);
    else if (gather) launch_onesweep<true, false>(s, a);
    else if (write_keys) launch_onesweep<false, true>(s, a);
    else launch_onesweep<false, false>(s, a);
    vin = vbuf[k % 2];
    kin = keys[k % 2].get();
    if (words && last) *words = std::move(keys[k % 2]);
  }
}

// Passes whose digit is not the same in every row.
std::vector<int> varying_passes(const std::vector<uint32_t>& hist, size_t P, int64_t n)
{
  std::vector<int> run;
  for (size_t q = 0; q < P; ++q) {
    bool constant = false;
    for (int d = 0; d < 256; ++d)
      if (hist[q * 256 + d] == static_cast<uint32_t>(n)) constant = true;
    if (!constant && n > 0) run.push_back(static_cast<int>(q));
  }
  return run;
}

// The identity order.
void identity_order(const OpContext& ctx, int64_t n, int32_t* perm, int32_t* inv, const RadixPayload* payload)
{
  cudaStream_t s = ctx.stream();
  if (n > 0) launch("iota", iota_kernel, hblocks(n), RT, 0, s, perm, n);
  if (n > 0 && inv) launch("iota", iota_kernel, hblocks(n), RT, 0, s, inv, n);
  if (n > 0 && payload && !payload_empty(*payload))
    launch("copy_payload", copy_payload_kernel, hblocks(n), RT, 0, s, *payload, n);
}

}  // namespace

void radix_sort_rows(const OpContext& ctx, const std::vector<RadixPass>& passes, int64_t n,
                     int32_t* perm, const std::vector<uint32_t>* counted, int32_t* inv, const RadixPayload* payload,
                     const FusedKey* fused)
{
  const size_t P = passes.size();
  std::vector<uint32_t> hist(P * 256, 0);
  if (counted) {
    hist = *counted;
  } else if (P > 0 && n > 0) {
    Buffer<uint32_t> d_hist(ctx.alloc(), P * 256);
    radix_histograms(ctx, passes, n, d_hist.get(), fused);
    ctx.fetch(hist.data(), d_hist.get(), P * 256 * sizeof(uint32_t));
    ctx.finish();
  }
  // skip constant-digit passes; the first executed pass of a word gathers it,
  // later passes of the same word read it carried
  const std::vector<int> run = varying_passes(hist, P, n);
  if (run.empty()) identity_order(ctx, n, perm, inv, payload);
  else run_passes(ctx, passes, run, hist, n, perm, inv, payload, fused, nullptr, 8, nullptr);
}

void radix_sort_words(const OpContext& ctx, const FusedKey& f, int bits, int64_t n, int32_t* perm,
                      const RadixPayload* payload, Buffer<uint8_t>* words, int* word_bytes)
{
  cudaStream_t s = ctx.stream();
  const int P    = (bits - f.drop + 7) / 8;
  const int kb   = P <= 4 ? 4 : 8;
  if (word_bytes) *word_bytes = kb;
  std::vector<uint32_t> hist(static_cast<size_t>(P) * 256, 0);
  Buffer<uint8_t> first;
  if (P > 0 && n > 0) {
    first = Buffer<uint8_t>(ctx.alloc(), static_cast<size_t>(n) * kb);
    Buffer<uint32_t> d_hist(ctx.alloc(), hist.size());
    LDF_CUDA(cudaMemsetAsync(d_hist.get(), 0, hist.size() * sizeof(uint32_t), s));
    WordArgs a{};
    a.f       = f;
    a.n       = n;
    a.npasses = P;
    a.words   = first.get();
    a.hist    = d_hist.get();
    const unsigned g =
      static_cast<unsigned>(std::min<int64_t>(ceil_div(n, int64_t(RT) * kWordRows), 8 * num_sms()));
    launch("fused_words", kb == 4 ? fused_words_kernel<uint32_t> : fused_words_kernel<uint64_t>, g, RT, 0, s, a);
    ctx.fetch(hist.data(), d_hist.get(), hist.size() * sizeof(uint32_t));
    ctx.finish();
  }
  std::vector<RadixPass> passes(P);
  for (int q = 0; q < P; ++q) {
    passes[q].src   = DigitSrc::CARRIED;
    passes[q].shift = 8 * q;
  }
  const std::vector<int> run = varying_passes(hist, P, n);
  if (run.empty()) {
    identity_order(ctx, n, perm, nullptr, payload);
    if (words) *words = std::move(first);  // equal words are in order
  } else {
    run_passes(ctx, passes, run, hist, n, perm, nullptr, payload, &f, &first, kb, words);
  }
}

// ---- sorting on the leading bits -----------------------------------------------
namespace {

constexpr int kSampleTies     = 1 << 17;        // sampled rows
constexpr int kDropCands      = 7;              // passes 2 .. 8

struct TieSampleArgs {
  FusedKey f;
  int64_t n;
  int bits;  // of the largest row number
  int ncand;
  int drop[kDropCands];
  unsigned long long* slots;  // [ncand][2 * kSampleTies]
  unsigned int* same;         // [ncand][2 * kSampleTies], or null: sampled rows of the slot's word after the first
  unsigned int* ties;         // [ncand]
  unsigned int* most;         // [ncand]
};

// Sampled row i of n: the rows in a scrambled order, each once (a permutation of
// the numbers of `bits` bits, applied again while it leaves the table).  Equal
// keys in neighbouring rows, as in event logs, are then met as often as in any
// other order; every 763rd row met each of 200,000 groups of 500 neighbours at
// most once, and the sort took 24.9 ms instead of 6.6.
__host__ __device__ __forceinline__ uint32_t sample_row(uint32_t i, uint32_t n, int bits)
{
  const uint32_t mask = (bits >= 32 ? 0u : 1u << bits) - 1u;
  uint32_t x          = i;
  do {
    for (int round = 0; round < 3; ++round) {
      x = (x * 0x9e3779b1u + 0x85ebca6bu) & mask;
      x ^= x >> ((bits + 1) / 2);
    }
  } while (x >= n);
  return x;
}

// ties[c] += sampled rows whose W >> drop[c] another sampled row has.  With
// `same`, pairs of such rows, and most[c] the most rows that share one (both
// no longer exact past kSameMax rows, which no rule accepts).
constexpr unsigned int kSameMax = 256;
__global__ void tie_sample_kernel(TieSampleArgs a)
{
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t r = sample_row(static_cast<uint32_t>(i), static_cast<uint32_t>(a.n), a.bits);
  uint32_t low;
  const uint64_t w = r < a.n ? fused_word(a.f, r, low) : 0;
  for (int c = 0; c < a.ncand; ++c) {
    unsigned int tie = 0;
    if (r < a.n) {
      const unsigned long long key = w >> (a.drop[c] - 8);
      unsigned long long* s        = a.slots + static_cast<int64_t>(c) * 2 * kSampleTies;
      uint32_t at                  = static_cast<uint32_t>(fastrange(mix64(key), 2 * kSampleTies));
      for (int probe = 0; key != ~0ull; ++probe) {
        unsigned long long v = *static_cast<volatile unsigned long long*>(s + at);
        if (v == ~0ull) v = atomicCAS(s + at, ~0ull, key);
        if (v == ~0ull) break;
        if (v == key) {
          tie = 1;
          if (a.same) {
            unsigned int* q = a.same + static_cast<int64_t>(c) * 2 * kSampleTies + at;
            tie             = *static_cast<volatile unsigned int*>(q) >= kSameMax ? kSameMax : atomicAdd(q, 1u) + 1;
          }
          break;
        }
        at = at + 1 == 2 * kSampleTies ? 0 : at + 1;
      }
    }
    const unsigned int sum = __reduce_add_sync(0xffffffffu, tie);
    const unsigned int top = __reduce_max_sync(0xffffffffu, tie);
    if (sum && (threadIdx.x & 31) == 0) {
      atomicAdd(a.ties + c, sum);
      if (a.same) atomicMax(a.most + c, top + 1);
    }
  }
}

// The bits of a row's W below f.drop.
__device__ __forceinline__ uint64_t dropped_bits(const FusedKey& f, int64_t row)
{
  uint32_t low;
  const uint64_t c = fused_word(f, row, low);
  const int d      = f.drop - 8;  // of C; f.drop <= 64
  return (d ? (c & (~0ull >> (64 - d))) << 8 : 0ull) | low;
}

constexpr int kTieThread = 12;  // longest run a thread orders by itself
struct TieRun {
  int32_t start, len;
};

// A thread per run of equal words: short runs are ordered in place by
// insertion, longer ones listed (count[0]; count[1]: a run over kTieRunMax).
template <typename KT>
__global__ void __launch_bounds__(256) order_ties_kernel(FusedKey f, const KT* w, int64_t n, int32_t* perm, TieRun* runs,
                                                         unsigned int* count)
{
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i + 1 < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const KT x = __ldg(w + i);
    if (x != __ldg(w + i + 1) || (i > 0 && __ldg(w + i - 1) == x)) continue;
    int len = 2;
    while (i + len < n && len <= kTieRunMax && __ldg(w + i + len) == x) ++len;
    if (len > kTieThread) {
      if (len > kTieRunMax) atomicExch(count + 1, 1u);
      else runs[atomicAdd(count, 1u)] = TieRun{static_cast<int32_t>(i), len};
      continue;
    }
    int32_t row[kTieThread];
    uint64_t low[kTieThread];
    for (int k = 0; k < len; ++k) {
      const int32_t r  = perm[i + k];
      const uint64_t l = dropped_bits(f, r);
      int at           = k;
      for (; at > 0 && low[at - 1] > l; --at) {
        low[at] = low[at - 1];
        row[at] = row[at - 1];
      }
      low[at] = l;
      row[at] = r;
    }
    for (int k = 0; k < len; ++k) perm[i + k] = row[k];
  }
}

// A block per listed run: each row's place counted among the run's rows.
__global__ void __launch_bounds__(256) order_runs_kernel(FusedKey f, const TieRun* runs, int32_t* perm)
{
  __shared__ uint64_t low[kTieRunMax];
  const TieRun t = runs[blockIdx.x];
  int32_t row[kTieRunMax / 256];
#pragma unroll
  for (int q = 0; q < kTieRunMax / 256; ++q) {
    const int k = q * 256 + threadIdx.x;
    row[q]      = 0;
    if (k < t.len) {
      row[q] = perm[t.start + k];
      low[k] = dropped_bits(f, row[q]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kTieRunMax / 256; ++q) {
    const int k = q * 256 + threadIdx.x;
    if (k >= t.len) continue;
    const uint64_t x = low[k];
    int at           = 0;
    for (int j = 0; j < t.len; ++j) at += low[j] < x || (low[j] == x && j < k) ? 1 : 0;
    perm[t.start + at] = row[q];
  }
}

// Random reads of one 16-byte record a row: as many in flight per thread as
// the registers hold.
constexpr int kPermRows = 8;
__global__ void __launch_bounds__(256) move_records_kernel(RadixPayload pay, const int32_t* perm, int64_t n)
{
  const int64_t per = static_cast<int64_t>(blockDim.x) * kPermRows;
  for (int64_t base = blockIdx.x * per + threadIdx.x; base < n; base += static_cast<int64_t>(gridDim.x) * per) {
    int32_t row[kPermRows];
    ulonglong2 v[kPermRows];
#pragma unroll
    for (int k = 0; k < kPermRows; ++k) row[k] = base + k * blockDim.x < n ? __ldcs(perm + base + k * blockDim.x) : -1;
#pragma unroll
    for (int k = 0; k < kPermRows; ++k) v[k] = row[k] >= 0 ? __ldg(pay.packed + row[k]) : make_ulonglong2(0, 0);
#pragma unroll
    for (int q = 0; q < kPassPayload; ++q) {
      if (q >= pay.nparts) break;
#pragma unroll
      for (int k = 0; k < kPermRows; ++k)
        if (row[k] >= 0) st_fixed(pay.pdst[q], pay.pwidth[q], base + k * blockDim.x, record_part(v[k], pay.poff[q]));
    }
  }
}

// ---- rows that travel whole ---------------------------------------------------
// One integer key as its whole word W = (raw ^ flip) - min, and at most 8
// bytes of other columns V (radix_sort_pairs).

// Writes W of every row and counts the digits that the passes sort on, from
// bit `drop` up: one read and one write (100M int64 keys: 281 us, 5.7 TB/s;
// fused_words' general codes took 508 us for the same bytes).
constexpr int kPairRows = 4;
template <typename T, typename KT>
__global__ void __launch_bounds__(RT) pair_words_kernel(const T* raw, T flip, T min, int64_t n, int drop, int npasses,
                                                        KT* words, uint32_t* hist)
{
  __shared__ uint32_t sh[8 * 256];
  for (int i = threadIdx.x; i < npasses * 256; i += RT) sh[i] = 0;
  __syncthreads();
  const int64_t per_iter = static_cast<int64_t>(RT) * kPairRows;
  for (int64_t base = blockIdx.x * per_iter + threadIdx.x; base < n; base += static_cast<int64_t>(gridDim.x) * per_iter) {
    T x[kPairRows];
#pragma unroll
    for (int j = 0; j < kPairRows; ++j) x[j] = base + j * RT < n ? __ldcs(raw + base + j * RT) : T(0);
#pragma unroll
    for (int j = 0; j < kPairRows; ++j) {
      if (base + j * RT >= n) break;
      const KT w             = static_cast<KT>(static_cast<T>((x[j] ^ flip) - min));
      words[base + j * RT] = w;
      uint64_t d             = static_cast<uint64_t>(w) >> drop;
      for (int q = 0; q < npasses; ++q, d >>= 8) atomicAdd(&sh[q * 256 + (static_cast<uint32_t>(d) & 0xffu)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < npasses * 256; i += RT)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

struct PairCols {
  uint64_t flip, min;  // the key: raw = (W + min) ^ flip
  int width;
  void* key;
  int n;  // columns packed into V (0: V is one column)
  int part_width[kPassPayload];
  int off[kPassPayload];  // byte offset in V, a multiple of the width
  const void* src[kPassPayload];
  void* dst[kPassPayload];
};

template <typename KT, typename VT>
__device__ __forceinline__ void store_pair(const PairCols& c, int64_t pos, KT w, VT v, VT* vout)
{
  st_fixed(c.key, c.width, pos, (static_cast<uint64_t>(w) + c.min) ^ c.flip);
  if (vout) vout[pos] = v;
  for (int q = 0; q < c.n; ++q) st_fixed(c.dst[q], c.part_width[q], pos, static_cast<uint64_t>(v) >> (8 * c.off[q]));
}

template <typename VT>
__global__ void __launch_bounds__(256) pack_pairs_kernel(PairCols c, int64_t n, VT* v)
{
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    uint64_t x = 0;
    for (int q = 0; q < c.n; ++q) {
      DCol d{};
      d.data  = c.src[q];
      d.width = c.part_width[q];
      x |= dbits_stream(d, i) << (8 * c.off[q]);
    }
    v[i] = static_cast<VT>(x);
  }
}

// Rows sorted on W >> drop to their final places and out of W.  A row's place
// among the rows that agree with it in W >> drop is counted: with up to
// kPairRun of them (6 on average when a 100M-row sort drops all but 24 bits)
// each row compares itself with its neighbours in shared memory; longer runs
// are listed for order_pair_runs (count[0]; count[1]: one over kTieRunMax).
// Bound by those compares: 1.0 ms at 100M rows, for 2.4 GB of traffic; a
// bitmap of the runs' first rows and one loop over a run took 1.17 ms.
// vout: where V goes as it is (null: nowhere).  drop 0: nothing is left to order.
constexpr int kPairRun  = 32;
constexpr int kPairTile = 8;  // rows per thread
template <typename KT, typename VT>
__global__ void __launch_bounds__(256) finish_pairs_kernel(PairCols c, const KT* w, const VT* vin, VT* vout, int64_t n,
                                                           int drop, TieRun* runs, unsigned int* count)
{
  constexpr int T = 256 * kPairTile;
  __shared__ KT s[T + 2 * kPairRun];
  const int64_t base = blockIdx.x * static_cast<int64_t>(T);
  VT v[kPairTile];
#pragma unroll
  for (int j = 0; j < kPairTile; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    v[j]            = i < n && vin ? __ldcs(vin + i) : VT(0);
  }
  for (int j = threadIdx.x; j < T + 2 * kPairRun; j += 256) {
    const int64_t i = base - kPairRun + j;
    if (i >= 0 && i < n) s[j] = __ldg(w + i);
  }
  __syncthreads();
  const KT below = drop ? (KT(1) << drop) - 1 : KT(0);
#pragma unroll
  for (int j = 0; j < kPairTile; ++j) {
    const int64_t i = base + j * 256 + threadIdx.x;
    if (i >= n) break;
    const KT* at = s + kPairRun + j * 256 + threadIdx.x;
    const KT x   = *at;
    int64_t pos  = i;
    if (drop) {
      const int left  = i < kPairRun ? static_cast<int>(i) : kPairRun;
      const int right = n - 1 - i < kPairRun ? static_cast<int>(n - 1 - i) : kPairRun;
      int l = 0, r = 0, before = 0;
      for (; l < left && at[-1 - l] >= (x & ~below); ++l) before += at[-1 - l] <= x ? 1 : 0;
      for (; r < right && at[1 + r] <= (x | below); ++r) before += at[1 + r] < x ? 1 : 0;
      if (l + r >= kPairRun) {
        if (l > 0) continue;
        int len = r + 1;  // the run's first row
        while (i + len < n && len <= kTieRunMax && __ldg(w + i + len) <= (x | below)) ++len;
        if (len > kTieRunMax) atomicExch(count + 1, 1u);
        else runs[atomicAdd(count, 1u)] = TieRun{static_cast<int32_t>(i), len};
        continue;
      }
      pos = i - l + before;
    }
    store_pair(c, pos, x, v[j], vout);
  }
}

template <typename KT, typename VT>
__global__ void __launch_bounds__(256) order_pair_runs_kernel(PairCols c, const KT* w, const VT* vin, VT* vout,
                                                              const TieRun* runs)
{
  __shared__ KT key[kTieRunMax];
  const TieRun t = runs[blockIdx.x];
  for (int k = threadIdx.x; k < t.len; k += 256) key[k] = w[t.start + k];
  __syncthreads();
  for (int k = threadIdx.x; k < t.len; k += 256) {
    const KT x = key[k];
    int at     = 0;
    for (int j = 0; j < t.len; ++j) at += key[j] < x || (key[j] == x && j < k) ? 1 : 0;
    store_pair(c, t.start + at, x, vin[t.start + k], vout);
  }
}

__global__ void __launch_bounds__(256) move_by_perm_kernel(RadixPayload pay, const int32_t* perm, int64_t n)
{
  const int64_t per = static_cast<int64_t>(blockDim.x) * kMoveBatch;
  for (int64_t base = blockIdx.x * per; base < n; base += static_cast<int64_t>(gridDim.x) * per) {
    int32_t pos[kMoveBatch], row[kMoveBatch];
#pragma unroll
    for (int k = 0; k < kMoveBatch; ++k) {
      const int64_t i = base + k * blockDim.x + threadIdx.x;
      pos[k]          = i < n ? static_cast<int32_t>(i) : -1;
      row[k]          = i < n ? __ldg(perm + i) : 0;
    }
    move_payload_rows(pay, pos, row);
  }
}

}  // namespace

namespace {
// sort_word_of of an integer key: its raw bits ^ int_flip.
uint64_t int_flip(const SortKeyDesc& k)
{
  const uint64_t all = k.key_bytes >= 8 ? ~0ull : (1ull << (8 * k.key_bytes)) - 1;
  return (is_signed_int(k.col.type) ? all ^ (all >> 1) : 0) ^ (k.descending ? all : 0);
}

template <typename T, typename KT>
void pair_words(const OpContext& ctx, const FusedKey& f, const PairCols& c, int64_t n, int npasses, void* words,
                uint32_t* hist)
{
  launch("pair_words", pair_words_kernel<T, KT>,
         static_cast<unsigned>(std::min<int64_t>(ceil_div(n, int64_t(RT) * kPairRows), 8 * num_sms())), RT, 0, ctx.stream(),
         static_cast<const T*>(f.key[0].col.data), static_cast<T>(c.flip), static_cast<T>(c.min), n, f.drop, npasses,
         static_cast<KT*>(words), hist);
}

// vals: V of every row; vout: its column in sorted order (null: packed).
template <typename KT, typename VT>
bool sort_pairs(const OpContext& ctx, const FusedKey& f, int bits, int64_t n, const PairCols& cols, const VT* vals, VT* vout)
{
  cudaStream_t s = ctx.stream();
  const int P    = std::max(1, (bits - f.drop + 7) / 8);
  std::vector<uint32_t> hist(static_cast<size_t>(P) * 256, 0);
  Buffer<uint8_t> words(ctx.alloc(), static_cast<size_t>(n) * sizeof(KT));
  {
    Buffer<uint32_t> d_hist(ctx.alloc(), hist.size());
    LDF_CUDA(cudaMemsetAsync(d_hist.get(), 0, hist.size() * sizeof(uint32_t), s));
    switch (cols.width) {
      case 1: pair_words<uint8_t, KT>(ctx, f, cols, n, P, words.get(), d_hist.get()); break;
      case 2: pair_words<uint16_t, KT>(ctx, f, cols, n, P, words.get(), d_hist.get()); break;
      case 4: pair_words<uint32_t, KT>(ctx, f, cols, n, P, words.get(), d_hist.get()); break;
      default: pair_words<uint64_t, KT>(ctx, f, cols, n, P, words.get(), d_hist.get()); break;
    }
    ctx.fetch(hist.data(), d_hist.get(), hist.size() * sizeof(uint32_t));
    ctx.finish();
  }
  std::vector<RadixPass> passes(P);
  for (int q = 0; q < P; ++q) {
    passes[q].src   = DigitSrc::CARRIED;
    passes[q].shift = f.drop + 8 * q;
  }
  std::vector<int> run = varying_passes(hist, P, n);
  if (run.empty()) run.push_back(P - 1);  // some pass has to write the rows
  const bool direct = f.drop == 0 && vout != nullptr;  // the last pass's order is final
  Buffer<VT> sorted;
  if (!direct) sorted = Buffer<VT>(ctx.alloc(), static_cast<size_t>(n));
  run_passes(ctx, passes, run, hist, n, direct ? vout : sorted.get(), nullptr, nullptr, &f, &words, sizeof(KT), &words,
             vals, sizeof(VT));
  const KT* w  = reinterpret_cast<const KT*>(words.get());
  const VT* v  = sorted.get();
  VT* vo       = direct ? nullptr : vout;
  Buffer<TieRun> runs(ctx.alloc(), f.drop ? static_cast<size_t>(n / kPairRun + 1) : 1);
  Buffer<unsigned int> count(ctx.alloc(), 2);
  LDF_CUDA(cudaMemsetAsync(count.get(), 0, 2 * sizeof(unsigned int), s));
  launch("finish_pairs", finish_pairs_kernel<KT, VT>, static_cast<unsigned>(ceil_div(n, 256 * kPairTile)), 256, 0, s, cols,
         w, v, vo, n, f.drop, runs.get(), count.get());
  if (f.drop == 0) return true;
  unsigned int h[2];
  ctx.fetch(h, count.get(), sizeof(h));
  ctx.finish();
  if (h[1]) return false;
  if (h[0])
    launch("order_pair_runs", order_pair_runs_kernel<KT, VT>, h[0], 256, 0, s, cols, w, v, vo,
           static_cast<const TieRun*>(runs.get()));
  return true;
}

template <typename VT>
void sort_pairs_of(const OpContext& ctx, FusedKey f, int bits, int64_t n, PairCols c)
{
  const VT* vals = static_cast<const VT*>(c.src[0]);
  VT* vout       = static_cast<VT*>(c.dst[0]);
  Buffer<VT> packed;
  if (c.n > 1 || c.part_width[0] != static_cast<int>(sizeof(VT))) {
    packed = Buffer<VT>(ctx.alloc(), static_cast<size_t>(n));
    launch("pack_pairs", pack_pairs_kernel<VT>,
           static_cast<unsigned>(std::min<int64_t>(ceil_div(n, 256), 16 * num_sms())), 256, 0, ctx.stream(), c, n, packed.get());
    vals = packed.get();
    vout = nullptr;
  } else {
    c.n = 0;
  }
  auto sort = [&] {
    if constexpr (sizeof(VT) == 4)
      if (bits <= 32) return sort_pairs<uint32_t, VT>(ctx, f, bits, n, c, vals, vout);
    return sort_pairs<uint64_t, VT>(ctx, f, bits, n, c, vals, vout);
  };
  if (sort()) return;
  f.drop = 0;  // too many rows tie: the whole word
  sort();
}
}  // namespace

bool radix_pairs_fit(const FusedKey& f, int64_t n, const ldf_column* table, int ncols, int key)
{
  if (n < kDropMinRows || f.n != 1 || f.has_class[0] || table[key].type == LDF_STRING) return false;
  int bytes = 0;
  for (int j = 0; j < ncols; ++j) {
    if (j == key) continue;
    if (table[j].type == LDF_STRING || table[j].valid != nullptr) return false;
    bytes += type_width(table[j].type);
  }
  return bytes > 0 && bytes <= 8 && ncols - 1 <= kPassPayload;
}

void radix_sort_pairs(const OpContext& ctx, FusedKey f, int bits, int64_t n, const ldf_column* table, int ncols, int key,
                      ldf_column* out)
{
  PairCols c{};
  int order[kPassPayload], bytes = 0;
  for (int j = 0; j < ncols; ++j) {
    if (j == key) continue;
    order[c.n++] = j;
    bytes += type_width(table[j].type);
  }
  std::stable_sort(order, order + c.n, [&](int x, int y) { return type_width(table[x].type) > type_width(table[y].type); });
  for (int q = 0, off = 0; q < c.n; ++q) {
    c.part_width[q] = type_width(table[order[q]].type);
    c.off[q]        = off;
    c.src[q]        = table[order[q]].data;
    c.dst[q]        = out[order[q]].data;
    off += c.part_width[q];
  }
  c.flip  = int_flip(f.key[0]);
  c.min   = f.min[0];
  c.width = f.key[0].col.width;
  c.key   = out[key].data;
  f.drop  = choose_drop(ctx, f, bits, n, true);
  if (bytes <= 4) sort_pairs_of<int32_t>(ctx, f, bits, n, c);
  else sort_pairs_of<int64_t>(ctx, f, bits, n, c);
}

int choose_drop(const OpContext& ctx, const FusedKey& f, int bits, int64_t n, bool whole_rows)
{
  if (n < kDropMinRows) return 0;
  TieSampleArgs a{};
  a.f    = f;
  a.n    = n;
  a.bits = 1;
  while ((n - 1) >> a.bits != 0) ++a.bits;
  const double rate = static_cast<double>(n) / kSampleTies;  // rows for each that is sampled
  // two passes fewer than the whole word takes, at least (whole rows: one, as
  // they are written once more after the passes anyhow), and a prefix that
  // could tell n rows apart
  const int full = (bits + 7) / 8;
  for (int k = 2; k <= full - (whole_rows ? 1 : 2) && k <= 8; ++k)
    if (bits - 8 * k >= 8 && (int64_t(1) << std::min(8 * k, 62)) >= n / 16) a.drop[a.ncand++] = bits - 8 * k;
  if (a.ncand == 0) return 0;
  cudaStream_t s = ctx.stream();
  Buffer<unsigned long long> slots(ctx.alloc(), static_cast<size_t>(a.ncand) * 2 * kSampleTies);
  Buffer<unsigned int> ties(ctx.alloc(), 2 * kDropCands), same;
  LDF_CUDA(cudaMemsetAsync(slots.get(), 0xff, slots.bytes(), s));
  LDF_CUDA(cudaMemsetAsync(ties.get(), 0, 2 * kDropCands * sizeof(unsigned int), s));
  if (whole_rows) {
    same = Buffer<unsigned int>(ctx.alloc(), static_cast<size_t>(a.ncand) * 2 * kSampleTies);
    LDF_CUDA(cudaMemsetAsync(same.get(), 0, same.bytes(), s));
  }
  a.slots = slots.get();
  a.same  = same.get();
  a.ties  = ties.get();
  a.most  = ties.get() + kDropCands;
  launch("tie_sample", tie_sample_kernel, static_cast<unsigned>(kSampleTies / 256), 256, 0, s, a);
  unsigned int h[2 * kDropCands];
  ctx.fetch(h, ties.get(), sizeof(h));
  ctx.finish();
  if (whole_rows) {
    // p sampled pairs of rows that tie stand for p rate^2.  A row's comparison
    // with one that ties with it takes 0.15 of a pass per row (100M rows in
    // groups of 10 to 50 equal neighbours: 0.11 to 0.15 ms for each further
    // row, a pass 0.79).  A group of kTieRunMax rows shows 2^12 / rate of them.
    const double rows = std::min<double>(std::max(4.0, kTieRunMax / 2 / rate), kSameMax);
    const double each = 2.0 * rate * rate / static_cast<double>(n);
    double best = full;
    int drop    = 0;
    for (int c = 0; c < a.ncand; ++c) {
      const double cost = (bits - a.drop[c]) / 8 + 0.15 * each * h[c];
      if (h[kDropCands + c] > rows || cost >= best) continue;
      best = cost;
      drop = a.drop[c];
    }
    return drop;
  }
  // t tying rows in the sample stand for about t rate^2 tying pairs of rows;
  // ties of a 64th of the rows or so cost less than a pass does.  A single
  // group of rows behind up to 8 sampled ties has some 4 rate rows, which
  // order_ties still takes at 100M rows.
  const double most = std::min(8.0, std::max(2.0, static_cast<double>(n) / 64 / (rate * rate)));
  for (int c = 0; c < a.ncand; ++c)
    if (h[c] <= most) return a.drop[c];
  return 0;
}

bool order_ties(const OpContext& ctx, const FusedKey& f, const void* words, int word_bytes, int64_t n, int32_t* perm)
{
  cudaStream_t s = ctx.stream();
  Buffer<TieRun> runs(ctx.alloc(), static_cast<size_t>(n / kTieThread + 1));
  Buffer<unsigned int> count(ctx.alloc(), 2);
  LDF_CUDA(cudaMemsetAsync(count.get(), 0, 2 * sizeof(unsigned int), s));
  const unsigned g = static_cast<unsigned>(std::min<int64_t>(ceil_div(n, 256), 16 * num_sms()));
  if (word_bytes == 4)
    launch("order_ties", order_ties_kernel<uint32_t>, g, 256, 0, s, f, static_cast<const uint32_t*>(words), n, perm,
           runs.get(), count.get());
  else
    launch("order_ties", order_ties_kernel<unsigned long long>, g, 256, 0, s, f,
           static_cast<const unsigned long long*>(words), n, perm, runs.get(), count.get());
  unsigned int h[2];
  ctx.fetch(h, count.get(), sizeof(h));
  ctx.finish();
  if (h[1]) return false;
  if (h[0])
    launch("order_runs", order_runs_kernel, h[0], 256, 0, s, f, static_cast<const TieRun*>(runs.get()), perm);
  return true;
}

void move_by_perm(const OpContext& ctx, const RadixPayload& payload, const int32_t* perm, int64_t n)
{
  if (n == 0 || payload_empty(payload)) return;
  RadixPayload rest = payload;
  if (payload.nparts) {
    launch("move_records", move_records_kernel,
           static_cast<unsigned>(std::min<int64_t>(ceil_div(n, int64_t(256) * kPermRows), 16 * num_sms())), 256, 0,
           ctx.stream(), payload, perm, n);
    rest.nparts = 0;
  }
  if (!payload_empty(rest))
    launch("move_by_perm", move_by_perm_kernel,
           static_cast<unsigned>(std::min<int64_t>(ceil_div(n, int64_t(256) * kMoveBatch), 16 * num_sms())), 256, 0,
           ctx.stream(), rest, perm, n);
}

}  // namespace ldf

// ---- raw-pointer helpers for the no-allocation hash partition ---------------
namespace ldf {

void radix_histogram_raw(cudaStream_t s, const RadixPass& p, int64_t n, uint32_t* d_hist)
{
  LDF_CUDA(cudaMemsetAsync(d_hist, 0, 256 * sizeof(uint32_t), s));
  if (n <= 0) return;
  HistArgs h{};
  h.npasses = 1;
  h.p[0]    = p;
  h.n       = n;
  h.hist    = d_hist;
  launch("histogram", histogram_kernel<false>, hist_blocks(n), RT, 0, s, h);
}

int64_t radix_status_words(int64_t n) { return ceil_div(status_words(n), int64_t(2)); }

void onesweep_gather_pass_raw(cudaStream_t s, const RadixPass& p, int64_t n, int32_t* rows_out,
                              const uint64_t* d_bases, uint64_t* status, int* err)
{
  if (n <= 0) return;
  PassArgs a{};
  a.p          = p;
  a.n          = n;
  a.keys_in    = nullptr;
  a.keys_out   = nullptr;
  a.vals_in    = nullptr;
  a.vals_out   = rows_out;
  a.digit_base = d_bases;
  a.status     = reinterpret_cast<uint32_t*>(status);
  a.err        = err;
  launch_onesweep<true, false>(s, a);
}

}  // namespace ldf
