// Sorts of small inputs by counting: the position of a row is the number of
// rows that sort before it, so one kernel compares every row with every other
// and writes each row straight to its place.  A radix sort of a few thousand
// rows is all launches and waits (histogram, a read-back, one kernel per key
// byte, each with a look-back chain); the n^2 compares of this one are cheap
// next to that up to kRankSortRows.
#include <algorithm>

#include "radix.cuh"

namespace ldf {
namespace {

// Rows up to which every block transforms the key columns itself; above, one
// kernel writes the words first (n / 32 blocks would each repeat the work).
constexpr int64_t kRankInline = 2048;
constexpr int kRankKeys       = 8;
constexpr int kRankCols       = 16;
constexpr int kRankThreads    = 256;
constexpr int kRankWarps      = kRankThreads / 32;
constexpr int kRankTile       = 1024;  // rows compared with per shared-memory tile

struct RankSortArgs {
  int nkeys;
  SortKeyDesc key[kRankKeys];  // most significant first
  int has_class[kRankKeys];    // nulls or NaNs: two bits of class before the word
  int64_t n;
  int64_t first, rows;    // positions [first, first + rows) are written
  const uint64_t* words;  // [K][n], or null: transform the columns here
  int ncols;
  DCol src[kRankCols];
  void* dst[kRankCols];
  uint8_t* dst_valid[kRankCols];
  int32_t* perm;  // != null: perm[position - first] = row
};

// Append the `bits` low bits of v to a bit string of K words (most
// significant first) that is `pos` bits long.
template <int K>
__device__ __forceinline__ void append_bits(uint64_t (&w)[K], int& pos, uint64_t v, int bits)
{
  const int q = pos >> 6, room = 64 - (pos & 63);
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (k == q) w[k] |= bits <= room ? v << (room - bits) : v >> (bits - room);
    if (k == q + 1 && bits > room) w[k] |= v << (64 - (bits - room));
  }
  pos += bits;
}

// All keys of a row as one bit string that compares like the rows do.
template <int K>
__device__ __forceinline__ void row_words(const RankSortArgs& a, int64_t r, uint64_t (&w)[K])
{
#pragma unroll
  for (int k = 0; k < K; ++k) w[k] = 0;
  int pos = 0;
  for (int j = 0; j < a.nkeys; ++j) {
    const SortKeyDesc& k = a.key[j];
    if (a.has_class[j]) append_bits<K>(w, pos, class_digit(k, r), 2);
    append_bits<K>(w, pos, sort_word(k, r), 8 * k.key_bytes);
  }
}

template <int K>
__global__ void __launch_bounds__(256) rank_words_kernel(RankSortArgs a, uint64_t* words)
{
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= a.n) return;
  uint64_t w[K];
  row_words<K>(a, r, w);
#pragma unroll
  for (int k = 0; k < K; ++k) words[k * a.n + r] = w[k];
}

// x < y, words most significant first; the first words mostly decide.
template <int K>
__device__ __forceinline__ bool words_less(const uint64_t (&x)[K], const uint64_t (&y)[K])
{
  if (K == 1 || x[0] != y[0]) return x[0] < y[0];
  bool lt = x[K - 1] < y[K - 1];
#pragma unroll
  for (int k = K - 2; k > 0; --k) lt = x[k] < y[k] || (x[k] == y[k] && lt);
  return lt;
}

// A block ranks 32 rows, one per lane; its warps share out the rows compared
// with, which pass through shared memory a tile at a time (every lane reads
// the same word: a broadcast).  Equal rows keep their order: rows before the
// block's own count when they are not greater, rows after it when they are
// less.  The bound is the compares and, below some 2,000 rows, launch and
// load latency.  Whole calls, three columns, radix passes -> this: one int64
// key 223 -> 59 us at 100 rows, 228 -> 142 us at 16,384; two nullable int64
// keys (three words) 291 -> 66 and 347 -> 237 us.
template <int K>
__global__ void __launch_bounds__(kRankThreads) rank_sort_kernel(RankSortArgs a)
{
  __shared__ uint64_t tile[K][kRankTile];
  __shared__ uint32_t part[kRankWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * 32;
  const int64_t i  = i0 + lane;
  uint64_t w[K];
#pragma unroll
  for (int k = 0; k < K; ++k) w[k] = 0;
  if (i < a.n) {
    if (a.words) {
#pragma unroll
      for (int k = 0; k < K; ++k) w[k] = __ldg(a.words + k * a.n + i);
    } else {
      row_words<K>(a, i, w);
    }
  }
  uint32_t cnt = 0;
  for (int64_t t0 = 0; t0 < a.n; t0 += kRankTile) {
    const int m = static_cast<int>(a.n - t0 < kRankTile ? a.n - t0 : kRankTile);
    __syncthreads();
    for (int j = threadIdx.x; j < m; j += kRankThreads) {
      uint64_t x[K];
      if (a.words) {
#pragma unroll
        for (int k = 0; k < K; ++k) x[k] = __ldg(a.words + k * a.n + t0 + j);
      } else {
        row_words<K>(a, t0 + j, x);
      }
#pragma unroll
      for (int k = 0; k < K; ++k) tile[k][j] = x[k];
    }
    __syncthreads();
    const int per = (m + kRankWarps - 1) / kRankWarps;
    const int lo = warp * per, hi = min(m, lo + per);
    auto at = [&](int j, uint64_t(&x)[K]) {
#pragma unroll
      for (int k = 0; k < K; ++k) x[k] = tile[k][j];
    };
    uint64_t x[K];
    if (t0 + hi <= i0) {
#pragma unroll 4
      for (int j = lo; j < hi; ++j) {
        at(j, x);
        cnt += words_less<K>(w, x) ? 0u : 1u;
      }
    } else if (t0 + lo >= i0 + 32) {
#pragma unroll 4
      for (int j = lo; j < hi; ++j) {
        at(j, x);
        cnt += words_less<K>(x, w) ? 1u : 0u;
      }
    } else {
      for (int j = lo; j < hi; ++j) {
        at(j, x);
        cnt += (words_less<K>(x, w) || (t0 + j < i && !words_less<K>(w, x))) ? 1u : 0u;
      }
    }
  }
  part[warp][lane] = cnt;
  __syncthreads();
  uint32_t rank = 0;
#pragma unroll
  for (int q = 0; q < kRankWarps; ++q) rank += part[q][lane];
  const int64_t pos = static_cast<int64_t>(rank) - a.first;
  if (i >= a.n || pos < 0 || pos >= a.rows) return;
  for (int c = warp; c < a.ncols; c += kRankWarps) {
    const DCol& s = a.src[c];
    copy_fixed(a.dst[c], pos, s.data, i, s.width);
    if (a.dst_valid[c]) a.dst_valid[c][pos] = dvalid(s, i) ? 1 : 0;
  }
  if (a.perm && warp == a.ncols % kRankWarps) a.perm[pos] = static_cast<int32_t>(i);
}

template <int K>
void launch_rank_sort(const OpContext& ctx, RankSortArgs& a)
{
  cudaStream_t s = ctx.stream();
  Buffer<uint64_t> words;
  if (a.n > kRankInline) {
    words = Buffer<uint64_t>(ctx.alloc(), K * a.n);
    launch("rank_words", rank_words_kernel<K>, static_cast<unsigned>(ceil_div(a.n, 256)), 256, 0, s, a, words.get());
    a.words = words.get();
  }
  launch("rank_sort", rank_sort_kernel<K>, static_cast<unsigned>(ceil_div(a.n, 32)), kRankThreads, 0, s, a);
}

// ---- ranks of a few thousand distinct strings -------------------------------
// Ranked on their first 32 bytes, as rank_sort_kernel ranks rows; while strings
// of equal bytes so far both go on, in rounds on the rank so far and the next 24.
constexpr int kHeadWords = 4;
constexpr int kHeadTile  = 256;
constexpr int kHeadBytes = 8 * kHeadWords;
constexpr int kNextBytes = kHeadBytes - 8;

// heads: bytes [from, from + 32) of every string, big-endian and zero-padded;
// from != 0: its rank so far, then bytes [from, from + 24).
__global__ void __launch_bounds__(256) string_heads_kernel(DCol col, const int32_t* repr, int64_t D, int64_t from,
                                                           const uint32_t* rank, uint64_t* heads, uint32_t* lens)
{
  const int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (d >= D) return;
  const int64_t r   = repr[d];
  const int64_t len = dstr_len(col, r);
  const uint8_t* p  = dstr_ptr(col, r) + (len > from ? from : 0);
  const int64_t n   = len > from ? (len - from < kHeadBytes ? len - from : kHeadBytes) : 0;
  uint64_t w[kHeadWords];
  if (!str_words(col, p, n, w)) {
#pragma unroll
    for (int k = 0; k < kHeadWords; ++k) {
      w[k] = 0;
      for (int b = 0; b < 8; ++b)
        if (8 * k + b < n) w[k] |= static_cast<uint64_t>(p[8 * k + b]) << (8 * b);
    }
  }
  const int shift = from != 0 ? 1 : 0;
#pragma unroll
  for (int k = 0; k < kHeadWords; ++k) {
    if (k + shift >= kHeadWords) continue;
    const uint32_t lo = static_cast<uint32_t>(w[k]), hi = static_cast<uint32_t>(w[k] >> 32);
    heads[(k + shift) * D + d] =
      (static_cast<uint64_t>(__byte_perm(lo, 0, 0x0123)) << 32) | __byte_perm(hi, 0, 0x0123);
  }
  if (shift) heads[d] = rank[d];
  lens[d] = static_cast<uint32_t>(len < 0xffffffffll ? len : 0xffffffffll);
}

// rank[d] = strings that sort before string d; covered: the bytes that the
// heads stand for.  Of two strings of equal heads the one that ends within them
// is a prefix of the other; two that both go on tie (*ties = 1), and share
// their rank.  Sorting 8,000 distinct ids of 8 to 24 characters: 509 -> 251 us a
// call against radix passes over 8-byte chunks with their read-backs (100 rows
// of 50 ids: 465 -> 158 us).
__global__ void __launch_bounds__(kRankThreads) rank_strings_kernel(int64_t D, const uint64_t* heads,
                                                                    const uint32_t* lens, int64_t covered,
                                                                    uint32_t* rank, int* ties)
{
  __shared__ uint64_t tile[kHeadWords][kHeadTile];
  __shared__ uint32_t tile_len[kHeadTile];
  __shared__ uint32_t part[kRankWarps][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * 32 + lane;
  uint64_t w[kHeadWords];
#pragma unroll
  for (int k = 0; k < kHeadWords; ++k) w[k] = i < D ? __ldg(heads + k * D + i) : 0;
  const uint32_t len = i < D ? __ldg(lens + i) : 0;
  uint32_t cnt       = 0;
  int tie            = 0;
  for (int64_t t0 = 0; t0 < D; t0 += kHeadTile) {
    const int m = static_cast<int>(D - t0 < kHeadTile ? D - t0 : kHeadTile);
    __syncthreads();
    if (static_cast<int>(threadIdx.x) < m) {
#pragma unroll
      for (int k = 0; k < kHeadWords; ++k) tile[k][threadIdx.x] = __ldg(heads + k * D + t0 + threadIdx.x);
      tile_len[threadIdx.x] = __ldg(lens + t0 + threadIdx.x);
    }
    __syncthreads();
    const int per = (m + kRankWarps - 1) / kRankWarps;
    const int lo = warp * per, hi = min(m, lo + per);
    for (int j = lo; j < hi; ++j) {
      const uint64_t x0 = tile[0][j];
      bool lt           = x0 < w[0];
      if (x0 == w[0]) {
        uint64_t x[kHeadWords];
#pragma unroll
        for (int k = 0; k < kHeadWords; ++k) x[k] = tile[k][j];
        lt = words_less<kHeadWords>(x, w);
        if (!lt && x[1] == w[1] && x[2] == w[2] && x[3] == w[3] && t0 + j != i) {
          const uint32_t l = tile_len[j];
          if (l <= covered || len <= covered) lt = l < len;
          else tie = 1;
        }
      }
      cnt += lt ? 1u : 0u;
    }
  }
  part[warp][lane] = cnt;
  if (__syncthreads_or(tie != 0 && i < D) && threadIdx.x == 0) *ties = 1;
  if (warp != 0 || i >= D) return;
  uint32_t r = 0;
#pragma unroll
  for (int q = 0; q < kRankWarps; ++q) r += part[q][lane];
  rank[i] = r;
}

}  // namespace

void rank_distinct_strings(const OpContext& ctx, const DCol& col, const int32_t* repr, int64_t D, int64_t longest,
                           uint32_t* rank)
{
  LDF_REQUIRE(D >= 1 && D <= kRankStrings, "rank_distinct_strings: too many strings");
  cudaStream_t s = ctx.stream();
  Buffer<uint64_t> heads(ctx.alloc(), kHeadWords * D);
  Buffer<uint32_t> lens(ctx.alloc(), D);
  Buffer<int> ties(ctx.alloc(), 1);
  auto round = [&](int64_t from, int64_t covered) {
    LDF_CUDA(cudaMemsetAsync(ties.get(), 0, sizeof(int), s));
    launch("string_heads", string_heads_kernel, static_cast<unsigned>(ceil_div(D, 256)), 256, 0, s, col, repr, D, from,
           static_cast<const uint32_t*>(rank), heads.get(), lens.get());
    launch("rank_strings", rank_strings_kernel, static_cast<unsigned>(ceil_div(D, 32)), kRankThreads, 0, s, D,
           static_cast<const uint64_t*>(heads.get()), static_cast<const uint32_t*>(lens.get()), covered, rank,
           ties.get());
  };
  int64_t covered = kHeadBytes;
  round(0, covered);
  while (longest > covered) {
    int tied = 0;
    ctx.fetch(&tied, ties.get(), sizeof(int));
    ctx.finish();
    if (tied == 0) break;
    round(covered, covered + kNextBytes);
    covered += kNextBytes;
  }
}

bool rank_sort(const OpContext& ctx, const ldf_column* table, int ncols, const std::vector<SortKeyDesc>& kd, int64_t n,
               int64_t first, int64_t rows, ldf_column* out)
{
  if (n < 1 || n > kRankSortRows || kd.size() > kRankKeys) return false;
  RankSortArgs a{};
  int bits = 0;
  for (size_t j = 0; j < kd.size(); ++j) {
    const SortKeyDesc& k     = kd[kd.size() - 1 - j];
    a.key[a.nkeys]           = k;
    a.has_class[a.nkeys]     = k.col.valid != nullptr || is_float(k.col.type) ? 1 : 0;
    bits += 8 * k.key_bytes + 2 * a.has_class[a.nkeys];
    ++a.nkeys;
  }
  if (bits > 3 * 64) return false;
  const Allocator& al = ctx.alloc();
  a.n     = n;
  a.first = first;
  a.rows  = rows;
  std::vector<int> later;  // columns gathered through the permutation
  for (int j = 0; j < ncols; ++j) {
    out[j] = alloc_out_column(al, table[j].type, rows, table[j].valid != nullptr);
    if (table[j].type == LDF_STRING || a.ncols == kRankCols) {
      later.push_back(j);
      continue;
    }
    a.src[a.ncols]       = make_dcol(table[j]);
    a.dst[a.ncols]       = out[j].data;
    a.dst_valid[a.ncols] = out[j].valid;
    ++a.ncols;
  }
  Buffer<int32_t> perm;
  if (!later.empty()) {
    perm   = Buffer<int32_t>(al, std::max<int64_t>(rows, 1));
    a.perm = perm.get();
  }
  switch ((bits + 63) / 64) {
    case 1: launch_rank_sort<1>(ctx, a); break;
    case 2: launch_rank_sort<2>(ctx, a); break;
    default: launch_rank_sort<3>(ctx, a); break;
  }
  std::vector<DCol> fsrc;
  std::vector<ldf_column*> fdst;
  for (int j : later) {
    if (table[j].type == LDF_STRING) {
      gather_strings(ctx, make_dcol(table[j]), perm.get(), rows, out[j]);
    } else {
      fsrc.push_back(make_dcol(table[j]));
      fdst.push_back(&out[j]);
    }
  }
  gather_fixed_columns(ctx, fsrc.data(), perm.get(), rows, fdst.data(), static_cast<int>(fsrc.size()));
  return true;
}

}  // namespace ldf
