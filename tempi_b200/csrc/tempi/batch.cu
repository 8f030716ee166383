// Batched pack/unpack: every region of a step in one launch.
//
// The reference packs one object per MPI_Pack call, each with its own launch
// and stream synchronisation (src/pack.cpp:56, packer_2d.cu:101-109), so the
// 26 halo regions of a 3-D grid cost 26 launches and 26 synchronisations.
// Here the regions become a table in device memory; one grid-stride kernel
// walks it.
//
// Work is cut into warp chunks: one warp copies one chunk in `passes`
// passes of 32 x L words, where L is the words in flight per lane and
// `passes` (1, 2 or 4) is chosen per region class.  Warps take chunks
// warp_id, warp_id + total warps, ... with no CTA-wide barrier between
// chunks; each finds its chunk's region by ballot rounds over the table's
// first-chunk column, kept in shared memory.  Each region keeps its own
// geometry and proven vector width, so a 16-B row face and a 2-KiB row face
// run at their own width inside the same launch.
//
// Two sets of kernels do this.  Batches whose regions all have at most two
// strided dimensions (every region of a grid) run the compact ones
// (k_batch_small, k_batch_copy_small and their _param forms): 64-byte
// entries, words reached by stepping their digits instead of dividing, one
// code path for every width at 64 registers, and launches that overlap the
// kernel before them (wait_for_previous).  What bounds them is the rate of
// scattered lines of the x faces (about 41 G lines/s by a one-load gather) and,
// for small halos, the launch.  Measured on B200, launches back to back over
// rotating buffers, pack / unpack / exchange in us: 8 mixed grids (208
// regions, 16.8 MB, whose lines take 9.8) 24.0 / 17.6 / 28.8 by the other
// set, 10.5 / 10.9 / 14.4 by these; the 256^3 halo 8.0 / 7.8 / 8.5 and 4.3 /
// 3.9 / 5.9; 320 x 300 x 310 doubles radius 3 12.4 / 12.5 / 17.5 and 7.0 /
// 6.5 / 8.8.  A 256^3 pack alone on the GPU: 19.5 and 14.4 us a call.  The
// other kernels (k_batch, k_batch_copy) divide every word's index over any
// number of dimensions, at 80 registers.
//
// The passes of each region class (width x words per row) and the launch
// shape of a batch (threads per CTA, CTAs per SM) come from defaults or from
// tempi_batch_tune, a measured autotuner whose choices are kept per batch
// signature for later batches of the same classes (and in
// TEMPI_CACHE_DIR/tempi_b200_batch_tune.txt).
//
// A batch can capture one launch into a CUDA graph and replay it; because
// the pointers live in the table, replays see new buffer contents without
// re-capture.
//
// A copy batch (tempi_batch_create_copy) fuses pack, transfer and unpack:
// each entry pairs a source layout with a destination layout of the same
// byte count, and word w of the entry is read at the source geometry's
// offset of w and written at the destination geometry's offset of w.  Both
// geometries are built at the same proven width, so one word index walks
// both.

#include "internal.hpp"
#include "runtime.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

namespace tempi {

namespace {

constexpr int kSmemTableBytes = 32768; // tables up to this size are staged
constexpr int kClasses = 40;           // 5 widths x 8 row-length buckets
constexpr int kPassChoices[3] = {1, 2, 4};

// Words each lane keeps in flight in one pass.  The compact kernels take 4 of
// any width: 64 registers, so 32 warps an SM, whose lanes' 4 requests are more
// than DRAM takes for short rows, and whose chunks are small enough to spread
// over all warps.  The kernels for any number of dimensions take 64 bytes for
// 8- and 16-byte words (registers allow no more), 8 words for narrower ones.
constexpr int kSmallWords = 4;
template <int W> constexpr int lane_words() { return W == 16 ? 4 : 8; }
__host__ __device__ constexpr uint32_t lane_words_of(uint32_t w, bool small) {
  return small ? uint32_t(kSmallWords) : w == 16 ? 4u : 8u;
}

struct BatchRegion {
  char *strided; // origin + start
  char *packed;
  Geometry g;
  uint32_t chunk_begin; // first warp chunk of this region
  uint32_t passes;      // passes of a warp over one chunk: 1, 2 or 4
};

struct CopyPair {
  const char *src; // src origin + start
  char *dst;       // dst origin + start
  Geometry gs, gd; // same width and word count
  uint32_t chunk_begin;
  uint32_t passes;
};

// the geometry that sets a record's words and class
const Geometry &geometry_of(const BatchRegion &r) { return r.g; }
const Geometry &geometry_of(const CopyPair &r) { return r.gs; }

// One strided side of a compact record: at most two strided dimensions (the
// regions of a grid never have more once contiguous ones are merged), word
// divisors, and what a step of 32 words adds to the digits of a word.
struct Side {
  char *base;           // origin + start
  int64_t s0, s1;       // strides of the two dimensions (0: unused)
  uint32_t wpr, wm;     // words per row and their FastDiv multiplier
  uint32_t c0, cm;      // count of dimension 0 and its FastDiv multiplier
  uint8_t ws, cs;       // the FastDiv shifts
  uint8_t dcol, ddig, dq; // 32 words = dq x c0 + ddig rows and dcol words
  uint8_t lwidth;       // log2 of the word's bytes
  uint8_t passes;       // passes of a warp over one chunk: 1, 2 or 4
  uint8_t spare;
};

// What the kernels read for a region or pair of at most two strided
// dimensions: 64 and 112 bytes instead of 168 and 288, so a halo's 26 regions
// take 2 KB of kernel parameters.  A warp loads the first 64 bytes of its
// entry at once (four 16-byte loads, one round trip), a pair's destination
// side behind its data loads.
struct alignas(16) SmallRegion {
  Side s;
  char *packed;
  uint32_t total_words;
  uint32_t chunk_begin;
};

struct alignas(16) SmallPair {
  Side s; // its passes and lwidth hold for both sides
  uint64_t spare;
  uint32_t total_words;
  uint32_t chunk_begin;
  Side d;
};
static_assert(sizeof(Side) == 48 && sizeof(SmallRegion) == 64 &&
                  sizeof(SmallPair) == 112 && offsetof(SmallPair, d) == 64 &&
                  offsetof(SmallPair, total_words) ==
                      offsetof(SmallRegion, total_words) &&
                  offsetof(SmallPair, chunk_begin) ==
                      offsetof(SmallRegion, chunk_begin),
              "entries start with 64 bytes of one layout");

Side make_side(const char *base, const Geometry &g, uint32_t passes) {
  Side s{};
  s.base = const_cast<char *>(base);
  s.s0 = g.strides[0];
  s.s1 = g.strides[1];
  s.wpr = g.wpr;
  s.wm = g.wdiv.m;
  s.ws = uint8_t(g.wdiv.s);
  s.c0 = std::max(1u, g.cdiv[0].d);
  s.cm = g.cdiv[0].m;
  s.cs = uint8_t(g.cdiv[0].s);
  const uint32_t drow = 32 / s.wpr;
  s.dcol = uint8_t(32 - drow * s.wpr);
  s.dq = uint8_t(drow / s.c0);
  s.ddig = uint8_t(drow % s.c0);
  s.lwidth = uint8_t(31 - __builtin_clz(g.width));
  s.passes = uint8_t(passes);
  return s;
}
bool is_small(const BatchRegion &r) { return r.g.nd <= 2; }
bool is_small(const CopyPair &r) { return r.gs.nd <= 2 && r.gd.nd <= 2; }
SmallRegion make_small(const BatchRegion &r) {
  return {make_side(r.strided, r.g, r.passes), r.packed, r.g.total_words,
          r.chunk_begin};
}
SmallPair make_small(const CopyPair &r) {
  return {make_side(r.src, r.gs, r.passes), 0, r.gs.total_words, r.chunk_begin,
          make_side(r.dst, r.gd, r.passes)};
}

template <int W> struct BWord;
template <> struct BWord<1> { using T = uint8_t; };
template <> struct BWord<2> { using T = uint16_t; };
template <> struct BWord<4> { using T = uint32_t; };
template <> struct BWord<8> { using T = uint2; };
template <> struct BWord<16> { using T = uint4; };

__device__ __forceinline__ uint32_t bdiv(uint32_t n, const FastDiv &f) {
  return f.m ? (__umulhi(n, f.m) >> f.s) : n;
}

// strided-side offset of row `row`: its digits over the counts, fastest
// first (a runtime loop, so that the unrolled word loops around it keep few
// registers live)
__device__ __forceinline__ int64_t brow_offset(uint32_t row, const Geometry &g) {
  const int nd = int(g.nd);
  if (nd == 0)
    return 0;
  int64_t off = 0;
#pragma unroll 1
  for (int k = 0; k + 1 < nd; ++k) {
    const uint32_t q = bdiv(row, g.cdiv[k]);
    off += int64_t(row - q * g.cdiv[k].d) * g.strides[k];
    row = q;
  }
  return off + int64_t(row) * g.strides[nd - 1];
}

// byte offset of word w on the strided side of g
template <int W>
__device__ __forceinline__ int64_t word_offset(uint32_t w, const Geometry &g) {
  const uint32_t row = bdiv(w, g.wdiv);
  return brow_offset(row, g) + int64_t(w - row * g.wpr) * W;
}

// One warp chunk of a pack or unpack region: words w0 + lane + 32 u.  Each
// load issues as soon as its address is known and only the loaded words
// stay live until the stores, so U loads are in flight per lane without
// holding U offsets in registers.
template <int W, int U>
__device__ __forceinline__ void pack_chunk(const BatchRegion &r, uint32_t w0,
                                           uint32_t lane, bool unpack) {
  using T = typename BWord<W>::T;
  const uint32_t total = r.g.total_words;
  char *strided = r.strided;
  T *packed = reinterpret_cast<T *>(r.packed);
  T v[U];
  if (!unpack) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t w = w0 + lane + 32 * u;
      if (w < total)
        v[u] = __ldg(reinterpret_cast<const T *>(strided + word_offset<W>(w, r.g)));
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (w0 + lane + 32 * u < total)
        packed[w0 + lane + 32 * u] = v[u];
  } else {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (w0 + lane + 32 * u < total)
        v[u] = __ldg(packed + (w0 + lane + 32 * u));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t w = w0 + lane + 32 * u;
      if (w < total)
        *reinterpret_cast<T *>(strided + word_offset<W>(w, r.g)) = v[u];
    }
  }
}

// one warp chunk of a copy pair: the loads at the source geometry first,
// then the stores at the destination geometry
template <int W, int U>
__device__ __forceinline__ void copy_chunk(const CopyPair &r, uint32_t w0,
                                           uint32_t lane) {
  using T = typename BWord<W>::T;
  const uint32_t total = r.gs.total_words;
  T v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t w = w0 + lane + 32 * u;
    if (w < total)
      v[u] = __ldg(reinterpret_cast<const T *>(r.src + word_offset<W>(w, r.gs)));
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint32_t w = w0 + lane + 32 * u;
    if (w < total)
      *reinterpret_cast<T *>(r.dst + word_offset<W>(w, r.gd)) = v[u];
  }
}

// a warp chunk is `passes` passes of 32 x lane_words<W>() words
template <int W>
__device__ __forceinline__ void pack_chunk_p(const BatchRegion &r, uint32_t c,
                                             uint32_t lane, bool unpack) {
  constexpr uint32_t kPass = 32u * lane_words<W>();
  const uint32_t passes = r.passes;
  uint32_t w0 = (c - r.chunk_begin) * passes * kPass;
  for (uint32_t p = 0; p < passes && w0 < r.g.total_words; ++p, w0 += kPass)
    pack_chunk<W, lane_words<W>()>(r, w0, lane, unpack);
}

template <int W>
__device__ __forceinline__ void copy_chunk_p(const CopyPair &r, uint32_t c,
                                             uint32_t lane) {
  constexpr uint32_t kPass = 32u * lane_words<W>();
  const uint32_t passes = r.passes;
  uint32_t w0 = (c - r.chunk_begin) * passes * kPass;
  for (uint32_t p = 0; p < passes && w0 < r.gs.total_words; ++p, w0 += kPass)
    copy_chunk<W, lane_words<W>()>(r, w0, lane);
}

// Index of the last entry whose first chunk is <= chunk, found by one warp:
// each round the lanes sample 32 evenly spaced entries of the remaining
// stretch and a ballot narrows it 32-fold, so n entries take ceil(log32 n)
// rounds (one for a 26-region halo, two for up to 1024 regions).  `begin(i)`
// is entry i's first chunk.
template <typename Begin>
__device__ __forceinline__ int find_region(Begin begin, int n, uint32_t chunk,
                                           uint32_t lane) {
  int base = 0, len = n;
  while (true) {
    const int step = (len + 31) / 32;
    const int off = int(lane) * step;
    const bool le = off < len && begin(base + off) <= chunk;
    const unsigned m = __ballot_sync(0xffffffffu, le);
    const int seg = 31 - __clz(m); // the stretch's first entry always qualifies
    base += seg * step;
    if (step == 1)
      return base;
    len = min(step, len - seg * step);
  }
}

// The table in shared memory when `staged` (the caller sized the dynamic
// shared memory for it), else in global memory.
template <typename Rec, int THREADS>
__device__ __forceinline__ const Rec *stage_table(const Rec *__restrict__ g,
                                                  int n, int staged,
                                                  uint32_t *s_table) {
  if (!staged)
    return g;
  const uint32_t *from = reinterpret_cast<const uint32_t *>(g);
  const int words = n * int(sizeof(Rec) / 4);
  for (int i = threadIdx.x; i < words; i += THREADS)
    s_table[i] = from[i];
  __syncthreads();
  return reinterpret_cast<const Rec *>(s_table);
}

// every warp chunk of the table `tab`, warps taking chunks warp_id,
// warp_id + total warps, ...
template <int THREADS>
__device__ __forceinline__ void batch_chunks(const BatchRegion *tab,
                                             int nregions,
                                             uint32_t total_chunks,
                                             int unpack) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * (THREADS / 32);
  for (uint32_t c = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);
       c < total_chunks; c += nwarps) {
    const BatchRegion &r = tab[find_region([&](int i) { return tab[i].chunk_begin; },
                                           nregions, c, lane)];
    switch (r.g.width) {
    case 16: pack_chunk_p<16>(r, c, lane, unpack); break;
    case 8: pack_chunk_p<8>(r, c, lane, unpack); break;
    case 4: pack_chunk_p<4>(r, c, lane, unpack); break;
    case 2: pack_chunk_p<2>(r, c, lane, unpack); break;
    default: pack_chunk_p<1>(r, c, lane, unpack); break;
    }
  }
}

// at least 768 threads per SM: registers are capped at 85 per thread
template <int THREADS>
__global__ void __launch_bounds__(THREADS, (768 + THREADS - 1) / THREADS)
    k_batch(const BatchRegion *__restrict__ regions, int nregions,
            uint32_t total_chunks, int unpack, int staged) {
  extern __shared__ __align__(16) uint32_t s_table[];
  const BatchRegion *tab =
      stage_table<BatchRegion, THREADS>(regions, nregions, staged, s_table);
  batch_chunks<THREADS>(tab, nregions, total_chunks, unpack);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, (768 + THREADS - 1) / THREADS)
    k_batch_copy(const CopyPair *__restrict__ pairs, int npairs,
                 uint32_t total_chunks, int staged) {
  extern __shared__ __align__(16) uint32_t s_table[];
  const CopyPair *tab =
      stage_table<CopyPair, THREADS>(pairs, npairs, staged, s_table);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * (THREADS / 32);
  for (uint32_t c = blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);
       c < total_chunks; c += nwarps) {
    const CopyPair &r = tab[find_region([&](int i) { return tab[i].chunk_begin; },
                                        npairs, c, lane)];
    switch (r.gs.width) {
    case 16: copy_chunk_p<16>(r, c, lane); break;
    case 8: copy_chunk_p<8>(r, c, lane); break;
    case 4: copy_chunk_p<4>(r, c, lane); break;
    case 2: copy_chunk_p<2>(r, c, lane); break;
    default: copy_chunk_p<1>(r, c, lane); break;
    }
  }
}

// ---- records of at most two strided dimensions -----------------------------

// Strided-side offsets of the words w, w + 32, w + 64, ... of a Side, for one
// lane: a word is (column, digit of dimension 0, digit of dimension 1), and a
// step of 32 words adds fixed amounts to the digits with at most one carry
// each, so a step is two compares and three 64-bit adds, where dividing every
// word anew took about 40 instructions and twice the registers.
struct Walk {
  int64_t off;
  uint32_t col, dig;         // column in words, digit of dimension 0
  uint32_t wpr, c0;          // their limits
  uint32_t dcol, ddig;       // added to them by a step
  int64_t step, wrap, carry; // added to off: by a step, when the column
                             // passes the row's end, when the digit passes c0

  __device__ __forceinline__ Walk(uint32_t w, const Side &g) {
    const int64_t s0 = g.s0, s1 = g.s1;
    const uint32_t lw = g.lwidth;
    wpr = g.wpr;
    c0 = g.c0;
    dcol = g.dcol;
    ddig = g.ddig;
    const uint32_t row = g.wm ? __umulhi(w, g.wm) >> g.ws : w;
    const uint32_t q = g.cm ? __umulhi(row, g.cm) >> g.cs : row;
    col = w - row * wpr;
    dig = row - q * c0;
    off = int64_t(q) * s1 + int64_t(dig) * s0 + int64_t(col << lw);
    step = int64_t(g.dq) * s1 + int64_t(ddig) * s0 + int64_t(dcol << lw);
    wrap = s0 - (int64_t(wpr) << lw);
    carry = s1 - int64_t(c0) * s0;
  }
  __device__ __forceinline__ void next() {
    off += step;
    col += dcol;
    dig += ddig;
    if (col >= wpr) {
      col -= wpr;
      ++dig;
      off += wrap;
    }
    if (dig >= c0) {
      dig -= c0;
      off += carry;
    }
  }
};

// The words of a lane's pass, whatever their width: U loads in flight, then U
// stores.  The width is switched on around the loads and again around the
// stores, and the offsets are computed outside: the code of a pass exists
// once, not once a width (five copies of it, whose common arithmetic the
// compiler hoists out of them, spill at 64 registers).  `at(u)` is the address
// of word u, `left` the words from word 0 to the region's end (32 apart).
// Loads bypass the L1: a kernel may have started before the previous one wrote
// what it reads.
template <int U, typename At>
__device__ __forceinline__ void load_words(uint4 (&v)[U], uint32_t lwidth,
                                           int left, At at) {
#define TEMPI_EACH(...)                                                        \
  _Pragma("unroll") for (int u = 0; u < U; ++u) if (32 * u < left) {           \
    const char *p = at(u);                                                     \
    __VA_ARGS__                                                                \
  }                                                                            \
  break;
  switch (lwidth) {
  case 4: TEMPI_EACH(v[u] = __ldcg(reinterpret_cast<const uint4 *>(p));)
  case 3: TEMPI_EACH(const uint2 t = __ldcg(reinterpret_cast<const uint2 *>(p));
                     v[u].x = t.x; v[u].y = t.y;)
  case 2: TEMPI_EACH(v[u].x = __ldcg(reinterpret_cast<const uint32_t *>(p));)
  case 1: TEMPI_EACH(v[u].x = __ldcg(reinterpret_cast<const uint16_t *>(p));)
  default: TEMPI_EACH(v[u].x = __ldcg(reinterpret_cast<const uint8_t *>(p));)
  }
}
template <int U, typename At>
__device__ __forceinline__ void store_words(const uint4 (&v)[U],
                                            uint32_t lwidth, int left, At at) {
  switch (lwidth) {
  case 4: TEMPI_EACH(*reinterpret_cast<uint4 *>(const_cast<char *>(p)) = v[u];)
  case 3: TEMPI_EACH(*reinterpret_cast<uint2 *>(const_cast<char *>(p)) =
                         make_uint2(v[u].x, v[u].y);)
  case 2: TEMPI_EACH(*reinterpret_cast<uint32_t *>(const_cast<char *>(p)) = v[u].x;)
  case 1: TEMPI_EACH(*reinterpret_cast<uint16_t *>(const_cast<char *>(p)) =
                         uint16_t(v[u].x);)
  default: TEMPI_EACH(*const_cast<char *>(p) = char(v[u].x);)
  }
#undef TEMPI_EACH
}

// the offsets of the pass's words on a strided side
template <int U> struct Offsets {
  int64_t off[U];
  __device__ __forceinline__ Offsets(uint32_t w, const Side &s) {
    Walk at(w, s);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      off[u] = at.off;
      if (u + 1 < U)
        at.next();
    }
  }
};

// N 16-byte loads of a table entry, all in flight together
template <int N, typename To>
__device__ __forceinline__ To load_entry(const void *from) {
  static_assert(sizeof(To) == 16 * N, "whole 16-byte words");
  union Both {
    uint4 q[N];
    To to;
    __device__ Both() {}
  } u;
#pragma unroll
  for (int i = 0; i < N; ++i)
    u.q[i] = static_cast<const uint4 *>(from)[i];
  return u.to;
}

// one pass of a warp over words w, w + 32, ... of a region
template <bool UNPACK>
__device__ __forceinline__ void move_words(const SmallRegion &r,
                                           const SmallRegion *, uint32_t w,
                                           int left) {
  constexpr int U = kSmallWords;
  const uint32_t lw = r.s.lwidth;
  char *strided = r.s.base, *packed = r.packed + (uint64_t(w) << lw);
  uint4 v[U];
  auto in_packed = [&](int u) { return packed + (32u * u << lw); };
  if (!UNPACK) {
    const Offsets<U> o(w, r.s);
    load_words<U>(v, lw, left, [&](int u) { return strided + o.off[u]; });
    store_words<U>(v, lw, left, in_packed);
  } else {
    load_words<U>(v, lw, left, in_packed);
    const Offsets<U> o(w, r.s);
    store_words<U>(v, lw, left, [&](int u) { return strided + o.off[u]; });
  }
}

// and of a copy pair, `r` its first 64 bytes: the destination side is read and
// its offsets are computed behind the data loads
template <bool UNPACK>
__device__ __forceinline__ void move_words(const SmallRegion &r,
                                           const SmallPair *entry, uint32_t w,
                                           int left) {
  constexpr int U = kSmallWords;
  const uint32_t lw = r.s.lwidth;
  uint4 v[U];
  {
    const char *src = r.s.base;
    const Offsets<U> o(w, r.s);
    load_words<U>(v, lw, left, [&](int u) { return src + o.off[u]; });
  }
  const Side d = load_entry<3, Side>(&entry->d);
  char *dst = d.base;
  const Offsets<U> o(w, d);
  store_words<U>(v, lw, left, [&](int u) { return dst + o.off[u]; });
}

// Programmatic dependent launch.  A batch kernel lets the next kernel of its
// stream be set up as soon as all its own CTAs run, and itself waits for the
// kernels before it to have finished, with their writes visible, before it
// touches a buffer: launch latency and the reading of the table overlap the
// kernel before.  Both are no-ops where a neighbour was launched without the
// attribute.  Measured back to back on B200, per launch: a 64^3 grid (bound by
// the launch) 6.2 us without, 2.6 us with, 2.2 us with the first chunk's entry
// looked up before the wait too; the 256^3 halo 7.3, 4.5 and 4.3 us; 8 mixed
// grids 13.5, 11.2 and 10.5 us.
__device__ __forceinline__ void let_next_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Every warp chunk of the table `tab`, warps taking chunks warp_id,
// warp_id + total warps, ...  The searches read the first-chunk column from
// `s_begin` (shared memory, filled here once per CTA) when `staged`, else
// from the table; the entries themselves are read in place, each field once
// per pass with one address for all lanes.
template <bool UNPACK, typename Rec>
__device__ __forceinline__ void small_chunks(const Rec *tab, int n,
                                             uint32_t total_chunks, int staged,
                                             uint32_t *s_begin) {
  let_next_launch();
  if (staged) {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      s_begin[i] = tab[i].chunk_begin;
    __syncthreads();
  }
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int at = 0;
  SmallRegion r; // the entry of chunk c
  auto look_up = [&] {
    at = staged ? find_region([&](int i) { return s_begin[i]; }, n, c, lane)
                : find_region([&](int i) { return tab[i].chunk_begin; }, n, c, lane);
    r = load_entry<4, SmallRegion>(tab + at);
  };
  // the first chunk's entry is at hand when the kernels before have finished
  if (c < total_chunks)
    look_up();
  wait_for_previous();
#pragma unroll 1
  while (c < total_chunks) {
    const uint32_t passes = r.s.passes;
    constexpr uint32_t per = 32 * kSmallWords;
    uint32_t w = (c - r.chunk_begin) * passes * per + lane;
#pragma unroll 1
    for (uint32_t p = 0; p < passes; ++p, w += per) {
      const int left = int(r.total_words - w);
      if (left <= 0)
        break;
      move_words<UNPACK>(r, tab + at, w, left);
    }
    c += nwarps;
    if (c < total_chunks)
      look_up();
  }
}

constexpr int kSmallThreadsPerSm = 1024;
template <int THREADS, bool UNPACK>
__global__ void
__launch_bounds__(THREADS, kSmallThreadsPerSm / THREADS)
    k_batch_small(const SmallRegion *__restrict__ regions, int nregions,
                  uint32_t total_chunks, int staged) {
  extern __shared__ __align__(16) uint32_t s_begin[];
  small_chunks<UNPACK>(regions, nregions, total_chunks, staged, s_begin);
}

template <int THREADS>
__global__ void
__launch_bounds__(THREADS, kSmallThreadsPerSm / THREADS)
    k_batch_copy_small(const SmallPair *__restrict__ pairs, int npairs,
                       uint32_t total_chunks, int staged) {
  extern __shared__ __align__(16) uint32_t s_begin[];
  small_chunks<false>(pairs, npairs, total_chunks, staged, s_begin);
}

// read every 16-B word of a buffer larger than the L2 (the autotuner's
// flush between timed launches), leaving clean lines behind
__global__ void k_tune_flush(const uint4 *__restrict__ buf, size_t n,
                             unsigned *__restrict__ sink) {
  unsigned acc = 0;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n;
       i += size_t(gridDim.x) * blockDim.x) {
    const uint4 v = __ldcg(buf + i);
    acc ^= v.x ^ v.y ^ v.z ^ v.w;
  }
  if (acc == 0x9e3779b9u)
    *sink = acc;
}

// ---- region classes and launch shapes --------------------------------------

int ilog2(uint32_t x) { return x ? 31 - __builtin_clz(x) : 0; }

// class of a geometry: its width and the log2 of its words per row (7 for
// 128 words or more)
int region_class(const Geometry &g) {
  return 8 * ilog2(g.width) + std::min(7, ilog2(g.wpr));
}

// passes per chunk of a class before any tuning
uint32_t default_passes(int cls) {
  (void)cls;
  return 1;
}

struct Shape {
  int threads = 256;
  int ctas_per_sm = 0; // 0: as many as fit
};

// the batch kernels: what they do (rows) at 128, 256 and 512 threads; the
// first three take compact records, the others any number of dimensions
enum { kSmallPack, kSmallUnpack, kSmallCopy, kAnyPack, kAnyCopy };
const void *batch_kernel(int kind, int threads) {
  static const void *fns[5][3] = {
      {(const void *)k_batch_small<128, false>,
       (const void *)k_batch_small<256, false>,
       (const void *)k_batch_small<512, false>},
      {(const void *)k_batch_small<128, true>,
       (const void *)k_batch_small<256, true>,
       (const void *)k_batch_small<512, true>},
      {(const void *)k_batch_copy_small<128>,
       (const void *)k_batch_copy_small<256>,
       (const void *)k_batch_copy_small<512>},
      {(const void *)k_batch<128>, (const void *)k_batch<256>,
       (const void *)k_batch<512>},
      {(const void *)k_batch_copy<128>, (const void *)k_batch_copy<256>,
       (const void *)k_batch_copy<512>}};
  return fns[kind][threads == 128 ? 0 : threads == 512 ? 2 : 1];
}

// how many CTAs of a batch kernel fit one SM (cached per kernel and size)
int max_ctas(int kind, int threads, int smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, int, int>, int> cache;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> l(mu);
  auto key = std::make_tuple(kind, threads, smem, dev);
  auto it = cache.find(key);
  if (it != cache.end())
    return it->second;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          &n, batch_kernel(kind, threads), threads, smem) != cudaSuccess ||
      n < 1) {
    cudaGetLastError();
    n = 1;
  }
  cache[key] = n;
  return n;
}

uint64_t chunks_of(const Geometry &g, uint32_t passes, bool small) {
  const uint64_t per = 32ull * lane_words_of(g.width, small) * passes;
  return (g.total_words + per - 1) / per;
}

// Whether a batch takes the compact kernels: every entry fits a compact
// record, and its chunks, up to twice as many as the other kernels cut, can
// be counted in 32 bits even at one pass each (so that no tuning of the
// passes changes the answer).
template <typename Rec> bool all_small(const Rec *recs, size_t n) {
  uint64_t chunks = 0;
  for (size_t i = 0; i < n; ++i) {
    chunks += chunks_of(geometry_of(recs[i]), 1, true);
    if (!is_small(recs[i]) || chunks > UINT32_MAX)
      return false;
  }
  return true;
}
template <typename Rec> bool all_small(const std::vector<Rec> &recs) {
  return all_small(recs.data(), recs.size());
}

// warp chunks of every record, in order; the total (or more than
// UINT32_MAX when the batch is too large)
template <typename Rec> uint64_t assign_chunks(std::vector<Rec> &recs) {
  const bool small = all_small(recs);
  uint64_t chunks = 0;
  for (Rec &r : recs) {
    const Geometry &g = geometry_of(r);
    r.chunk_begin = uint32_t(std::min<uint64_t>(chunks, UINT32_MAX));
    chunks += chunks_of(g, r.passes, small);
  }
  return chunks;
}

} // namespace

template <typename Rec> static int kind_of(bool small, int unpack) {
  if (std::is_same<Rec, CopyPair>::value)
    return small ? kSmallCopy : kAnyCopy;
  return !small ? kAnyPack : unpack ? kSmallUnpack : kSmallPack;
}

// A launch into a capture becomes a node without the programmatic attribute:
// its edges are then the ordinary ones, whatever node comes before it.
static bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return cs != cudaStreamCaptureStatusNone;
}

// a launch configuration with programmatic dependent launch
struct Overlapped {
  cudaLaunchAttribute attr{};
  cudaLaunchConfig_t config{};
  Overlapped(uint32_t grid, int threads, int smem, cudaStream_t s) {
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    config.gridDim = dim3(grid);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = size_t(smem);
    config.stream = s;
    config.attrs = &attr;
    config.numAttrs = 1;
  }
  Overlapped(const Overlapped &) = delete;
};

// Launch the pack kernel (or, for pairs, the copy kernel) over a table in
// device memory on `s`: compact entries when `small`.  `overlap`: the table
// was complete before the kernels ahead on `s` were issued, so the launch may
// overlap them.
template <typename Rec>
static int launch_table(const void *table, int n, bool small,
                        uint32_t total_chunks, int unpack, Shape shape,
                        cudaStream_t s, bool overlap) {
  constexpr bool kCopy = std::is_same<Rec, CopyPair>::value;
  if (n <= 0 || total_chunks == 0)
    return TEMPI_OK;
  const int smem_need = n * int(small ? sizeof(uint32_t) : sizeof(Rec));
  int staged = smem_need <= kSmemTableBytes ? 1 : 0;
  const int smem = staged ? smem_need : 0;
  const int threads = shape.threads == 128 || shape.threads == 512
                          ? shape.threads
                          : 256;
  const int kind = kind_of<Rec>(small, unpack);
  const int fit = max_ctas(kind, threads, smem);
  const int per_sm = shape.ctas_per_sm > 0 ? std::min(shape.ctas_per_sm, fit)
                                           : fit;
  const uint32_t warps_per_cta = uint32_t(threads / 32);
  const uint32_t want = (total_chunks + warps_per_cta - 1) / warps_per_cta;
  const uint32_t grid = std::max<uint32_t>(
      1, std::min<uint32_t>(want, uint32_t(num_sms()) * uint32_t(per_sm)));
  void *general[] = {&table, &n, &total_chunks, &unpack, &staged};
  void *others[] = {&table, &n, &total_chunks, &staged};
  Overlapped launch(grid, threads, smem, s);
  launch.config.numAttrs = small && overlap && !capturing(s) ? 1 : 0;
  cudaLaunchKernelExC(&launch.config, batch_kernel(kind, threads),
                      kind == kAnyPack ? general : others);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return cuda_error(e, kCopy ? "copy batch launch" : "batch launch");
  counters().kernel_launches++;
  set_last_kernel(kCopy ? "batch_copy" : unpack ? "batch_unpack" : "batch_pack");
  return TEMPI_OK;
}

// ---- tuned choices, kept per batch signature -------------------------------

namespace {

struct Tuned {
  Shape shape;
  uint8_t passes[kClasses] = {}; // 0: the class's default
};

std::mutex g_tune_mu;
std::map<uint64_t, Tuned> g_tuned;
bool g_tune_loaded = false;

std::string tune_path() {
  return env().cache_dir + "/tempi_b200_batch_tune.txt";
}

void load_tuned_locked() {
  if (g_tune_loaded)
    return;
  g_tune_loaded = true;
  FILE *f = std::fopen(tune_path().c_str(), "r");
  if (!f)
    return;
  unsigned long long sig;
  int th, cps;
  while (std::fscanf(f, "%llx %d %d", &sig, &th, &cps) == 3) {
    Tuned t;
    t.shape.threads = th;
    t.shape.ctas_per_sm = cps;
    bool ok = true;
    for (int c = 0; c < kClasses && ok; ++c) {
      unsigned u;
      ok = std::fscanf(f, "%u", &u) == 1;
      t.passes[c] = uint8_t(u == 1 || u == 2 || u == 4 ? u : 0);
    }
    if (!ok)
      break;
    g_tuned[sig] = t;
  }
  std::fclose(f);
}

// Signature of a batch: the kernels that run it, what kind of launch it is, and
// the multiset of its records' (class, log2 words).  Choices hold for the
// kernels that were timed: a pass of the compact ones is 4 words a lane, of the
// others up to 8, and a different number of CTAs fits an SM.
// kTunedKernels changes when either set's pass or occupancy does, so that a
// tune file written before is left unused.
constexpr uint32_t kTunedKernels = 2;
template <typename Rec> uint64_t signature(const Rec *recs, size_t n, int unpack) {
  std::vector<uint32_t> keys;
  keys.reserve(n);
  for (size_t i = 0; i < n; ++i) {
    const Geometry &g = geometry_of(recs[i]);
    keys.push_back(uint32_t(region_class(g)) << 8 | uint32_t(ilog2(g.total_words)));
  }
  std::sort(keys.begin(), keys.end());
  uint64_t h = 1469598103934665603ull; // FNV-1a
  auto mix = [&](uint32_t v) {
    for (int i = 0; i < 4; ++i) {
      h ^= (v >> (8 * i)) & 0xff;
      h *= 1099511628211ull;
    }
  };
  mix(kTunedKernels);
  mix(all_small(recs, n));
  mix(std::is_same<Rec, CopyPair>::value ? 2u : uint32_t(unpack));
  for (uint32_t k : keys)
    mix(k);
  return h;
}

bool anything_tuned() {
  std::lock_guard<std::mutex> l(g_tune_mu);
  load_tuned_locked();
  return !g_tuned.empty();
}

// the choices tuned for this signature, if any
template <typename Rec>
bool find_tuned(const Rec *recs, size_t n, int unpack, Tuned *out) {
  std::lock_guard<std::mutex> l(g_tune_mu);
  load_tuned_locked();
  auto it = g_tuned.find(signature(recs, n, unpack));
  if (it == g_tuned.end())
    return false;
  *out = it->second;
  return true;
}

// the passes of every record from `t` (or the defaults) and the chunk count
template <typename Rec>
uint64_t apply_passes(std::vector<Rec> &recs, const Tuned *t) {
  for (Rec &r : recs) {
    const int c = region_class(geometry_of(r));
    r.passes = t && t->passes[c] ? t->passes[c] : default_passes(c);
  }
  return assign_chunks(recs);
}

} // namespace

struct BatchImpl {
  std::vector<BatchRegion> host;
  std::vector<CopyPair> host_pairs; // a copy batch
  void *dev = nullptr; // the table: compact entries when `small`
  bool small = false;
  uint32_t total_chunks = 0;
  int unpack = 0;
  Shape shape;
  Tuned tuned;       // this batch's choices
  bool has_tuned = false;
  uint64_t sig = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

} // namespace tempi

struct tempi_batch {
  tempi::BatchImpl impl;
};

using namespace tempi;

// choices for a new batch: the tuned ones of its signature if any; sets the
// records' passes and chunks, returns the chunk total
template <typename Rec>
static uint64_t plan_batch(BatchImpl &bi, std::vector<Rec> &recs) {
  bi.sig = signature(recs.data(), recs.size(), bi.unpack);
  {
    std::lock_guard<std::mutex> l(g_tune_mu);
    load_tuned_locked();
    auto it = g_tuned.find(bi.sig);
    if (it != g_tuned.end()) {
      bi.tuned = it->second;
      bi.has_tuned = true;
      bi.shape = it->second.shape;
    }
  }
  return apply_passes(recs, bi.has_tuned ? &bi.tuned : nullptr);
}

template <typename Rec>
static std::vector<decltype(make_small(std::declval<Rec>()))>
small_table(const std::vector<Rec> &recs) {
  std::vector<decltype(make_small(std::declval<Rec>()))> t;
  t.reserve(recs.size());
  for (const Rec &r : recs)
    t.push_back(make_small(r));
  return t;
}

template <typename Rec>
static int upload(const std::vector<Rec> &recs, void **dev) {
  if (recs.empty())
    return TEMPI_OK;
  const size_t bytes = recs.size() * sizeof(Rec);
  cudaError_t e = cudaSuccess;
  if (!*dev)
    e = cudaMalloc(dev, bytes);
  if (e == cudaSuccess)
    e = copy_complete(*dev, recs.data(), bytes);
  if (e != cudaSuccess)
    return cuda_error(e, "batch table upload");
  return TEMPI_OK;
}

// the batch's table, as its kernels read it, into device memory
static int upload_table(BatchImpl &bi) {
  if (!bi.host_pairs.empty()) {
    bi.small = all_small(bi.host_pairs);
    return bi.small ? upload(small_table(bi.host_pairs), &bi.dev)
                    : upload(bi.host_pairs, &bi.dev);
  }
  bi.small = all_small(bi.host);
  return bi.small ? upload(small_table(bi.host), &bi.dev)
                  : upload(bi.host, &bi.dev);
}

extern "C" int tempi_batch_create(const tempi_region *regions, int32_t n,
                                  int32_t unpack, tempi_batch **out) {
  if (!out || n < 0 || (n > 0 && !regions))
    return set_error(TEMPI_ERR_ARG, "bad batch arguments");
  *out = nullptr;
  auto *b = new tempi_batch();
  b->impl.unpack = unpack ? 1 : 0;
  for (int32_t i = 0; i < n; ++i) {
    const tempi_region &r = regions[i];
    BatchRegion br{};
    char *strided = (char *)r.origin + r.desc.start;
    bool empty = false;
    int err = make_geometry(&r.desc, r.incount, uintptr_t(strided),
                            uintptr_t(r.packed), 0, &br.g, &empty);
    if (err) {
      delete b;
      return err;
    }
    if (empty)
      continue;
    br.strided = strided;
    br.packed = (char *)r.packed;
    b->impl.host.push_back(br);
  }
  const uint64_t chunks = plan_batch(b->impl, b->impl.host);
  if (chunks > UINT32_MAX) {
    delete b;
    return set_error(TEMPI_ERR_ARG, "batch too large");
  }
  b->impl.total_chunks = uint32_t(chunks);
  int err = upload_table(b->impl);
  if (err) {
    cudaFree(b->impl.dev);
    delete b;
    return err;
  }
  *out = b;
  return TEMPI_OK;
}

template <int P, typename Rec = BatchRegion> struct StaticPiece {
  Rec r[P];
};

// A batch of up to kParamRegions regions in one launch with its table in the
// kernel's parameters (2 KB of compact entries, or 5.4 KB for more than two
// strided dimensions), for calls that bring their regions with them: the
// allocation-free entry point (neither a fill kernel nor the fixed array is
// involved) and the interposed MPI_Neighbor_alltoallw (no upload).
constexpr int kParamRegions = 32;

template <int P>
__global__ void __launch_bounds__(256, 3)
    k_batch_param(const __grid_constant__ StaticPiece<P> piece, int nregions,
                  uint32_t total_chunks, int unpack) {
  // read in place: a warp's region search reads one field of up to 32
  // entries, its copy loop one entry that every lane shares
  batch_chunks<256>(piece.r, nregions, total_chunks, unpack);
}

// The parameter block as ordinary memory: read through the constant cache,
// the entries that an SM's warps share miss one after another (a 256^3
// exchange alone on the GPU 19.3 us a call that way, 18.2 this way).
template <typename Rec>
__device__ __forceinline__ const Rec *in_memory(const Rec *param) {
  asm volatile("" : "+l"(param));
  return param;
}

template <int P, bool UNPACK>
__global__ void __launch_bounds__(256, kSmallThreadsPerSm / 256)
    k_batch_param_small(const __grid_constant__ StaticPiece<P, SmallRegion> piece,
                        int nregions, uint32_t total_chunks) {
  __shared__ uint32_t s_begin[P];
  small_chunks<UNPACK>(in_memory(piece.r), nregions, total_chunks, 1, s_begin);
}

template <int P>
__global__ void __launch_bounds__(256, kSmallThreadsPerSm / 256)
    k_batch_copy_param(const __grid_constant__ StaticPiece<P, SmallPair> piece,
                       int npairs, uint32_t total_chunks) {
  __shared__ uint32_t s_begin[P];
  small_chunks<false>(in_memory(piece.r), npairs, total_chunks, 1, s_begin);
}

// whether a tuned shape is one that the kernels with a parameter table have
static bool param_shape(const Shape &s) {
  return s.threads == 0 || s.threads == 256;
}

// k_batch_param(_small) over the `n` <= kParamRegions entries of `table`
// (host memory), `per_sm` CTAs per SM (0: as many as fit)
template <typename Rec>
static int launch_param(const Rec *table, int n, uint32_t total_chunks,
                        int unpack, int per_sm, cudaStream_t s) {
  constexpr bool kSmall = !std::is_same<Rec, BatchRegion>::value;
  StaticPiece<kParamRegions, Rec> piece;
  std::memcpy(piece.r, table, size_t(n) * sizeof(Rec));
  const int fit = kSmall ? kSmallThreadsPerSm / 256 : 3; // by the launch bounds
  per_sm = per_sm > 0 ? std::min(per_sm, fit) : fit;
  const uint32_t grid = std::max<uint32_t>(
      1, std::min<uint32_t>((total_chunks + 7) / 8,
                            uint32_t(num_sms()) * uint32_t(per_sm)));
  Overlapped launch(grid, 256, 0, s);
  launch.config.numAttrs = capturing(s) ? 0 : 1;
  if constexpr (!kSmall)
    k_batch_param<kParamRegions><<<grid, 256, 0, s>>>(piece, n, total_chunks,
                                                       unpack);
  else if constexpr (std::is_same<Rec, SmallPair>::value)
    cudaLaunchKernelEx(&launch.config, k_batch_copy_param<kParamRegions>, piece,
                       n, total_chunks);
  else
    cudaLaunchKernelEx(&launch.config,
                       unpack ? k_batch_param_small<kParamRegions, true>
                              : k_batch_param_small<kParamRegions, false>,
                       piece, n, total_chunks);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return cuda_error(e, "batch launch");
  counters().kernel_launches++;
  return TEMPI_OK;
}

// `direct`: a launch of its own (tempi_batch_launch), which may overlap the
// kernel before it; graph captures and the tuner's timings are plain.  The
// table stays in device memory for all of them: with the same entries in the
// kernel's parameters a 256^3 pack alone on the GPU took 17.2 us a call
// against 14.4 (a parameter block is new memory at every launch, the table is
// in the L2).
static int batch_launch(tempi_batch *b, cudaStream_t s, bool direct) {
  BatchImpl &bi = b->impl;
  if (!bi.host_pairs.empty())
    return launch_table<CopyPair>(bi.dev, int(bi.host_pairs.size()), bi.small,
                                  bi.total_chunks, 0, bi.shape, s, direct);
  return launch_table<BatchRegion>(bi.dev, int(bi.host.size()), bi.small,
                                   bi.total_chunks, bi.unpack, bi.shape, s,
                                   direct);
}

// Copy pairs for `regions`, each at the default passes of its class; empty
// regions are dropped.  Returns the chunk count through *chunks_out.
static int build_pairs(const tempi_copy_region *regions, int32_t n,
                       std::vector<CopyPair> *pairs, uint64_t *chunks_out) {
  pairs->clear();
  for (int32_t i = 0; i < n; ++i) {
    const tempi_copy_region &r = regions[i];
    if (r.src_count < 0 || r.dst_count < 0 ||
        r.src_desc.size * r.src_count != r.dst_desc.size * r.dst_count) {
      return set_error(TEMPI_ERR_ARG,
                       "copy region %d: source and destination sizes differ",
                       int(i));
    }
    const char *src = (const char *)r.src_origin + r.src_desc.start;
    char *dst = (char *)r.dst_origin + r.dst_desc.start;
    CopyPair cp{};
    bool es = false, ed = false;
    // the widest width both layouts prove, then both geometries at it
    int err = make_geometry(&r.src_desc, r.src_count, uintptr_t(src), 0, 0,
                            &cp.gs, &es);
    if (!err)
      err = make_geometry(&r.dst_desc, r.dst_count, uintptr_t(dst), 0, 0,
                          &cp.gd, &ed);
    if (!err && !es && !ed) {
      const int w = int(std::min(cp.gs.width, cp.gd.width));
      if (int(cp.gs.width) != w)
        err = make_geometry(&r.src_desc, r.src_count, uintptr_t(src), 0, w,
                            &cp.gs, &es);
      if (int(cp.gd.width) != w)
        err = make_geometry(&r.dst_desc, r.dst_count, uintptr_t(dst), 0, w,
                            &cp.gd, &ed);
    }
    if (err)
      return err;
    if (es || ed)
      continue; // nothing to copy
    if (cp.gs.width != cp.gd.width || cp.gs.total_words != cp.gd.total_words)
      return set_error(TEMPI_ERR_ARG, "copy region %d: layouts disagree",
                       int(i));
    cp.src = src;
    cp.dst = dst;
    pairs->push_back(cp);
  }
  *chunks_out = apply_passes(*pairs, nullptr);
  if (*chunks_out > UINT32_MAX)
    return set_error(TEMPI_ERR_ARG, "batch too large");
  return TEMPI_OK;
}

extern "C" int tempi_batch_create_copy(const tempi_copy_region *regions,
                                       int32_t n, tempi_batch **out) {
  if (!out || n < 0 || (n > 0 && !regions))
    return set_error(TEMPI_ERR_ARG, "bad copy batch arguments");
  *out = nullptr;
  auto *b = new tempi_batch();
  uint64_t chunks = 0;
  int err = build_pairs(regions, n, &b->impl.host_pairs, &chunks);
  if (!err) {
    chunks = plan_batch(b->impl, b->impl.host_pairs);
    if (chunks > UINT32_MAX)
      err = set_error(TEMPI_ERR_ARG, "batch too large");
  }
  if (!err) {
    b->impl.total_chunks = uint32_t(chunks);
    err = upload_table(b->impl);
  }
  if (err) {
    cudaFree(b->impl.dev);
    delete b;
    return err;
  }
  *out = b;
  return TEMPI_OK;
}

namespace tempi {

// the pair of an edge of single objects
static CopyPair unit_pair(const CopyEdge &e, uint32_t chunk_begin) {
  const TypeRecord &a = *e.src_type, &b = *e.dst_type;
  const char *src = e.src_origin + a.desc.start;
  char *dst = e.dst_origin + b.desc.start;
  const uint32_t bits = uint32_t(reinterpret_cast<uintptr_t>(src) |
                                 reinterpret_cast<uintptr_t>(dst)) |
                        a.unit[4].width | b.unit[4].width;
  const int k = __builtin_ctz(bits); // the width both sides prove: 2^k <= 16
  return {src, dst, a.unit[k], b.unit[k], chunk_begin, 0};
}

// The entries of single objects at the choices tuned for their signature, if
// any; false when those need another kernel.  (Kept out of the loop that forms
// the entries: processes that tuned nothing do not pay for it.)
__attribute__((noinline)) static bool take_tuned(const CopyEdge *edges, int n,
                                                 SmallPair *entries,
                                                 uint64_t *chunks, Tuned *tuned) {
  std::vector<CopyPair> pairs;
  for (int i = 0; i < n; ++i)
    if (edges[i].src_count)
      pairs.push_back(unit_pair(edges[i], 0));
  if (!find_tuned(pairs.data(), pairs.size(), 0, tuned))
    return true;
  if (!param_shape(tuned->shape))
    return false;
  *chunks = apply_passes(pairs, tuned);
  for (size_t i = 0; i < pairs.size(); ++i)
    entries[i] = make_small(pairs[i]);
  return true;
}

// The exchange of up to kParamRegions single objects whose two sides have at
// most two strided dimensions (a halo's 26 regions), whatever number of edges
// exchange nothing: entries straight from the
// geometries settled when the types were committed, no division of lengths and
// no descriptors copied (a 256^3 exchange: 4.1 us less host time a call, with
// the types looked up under one lock).  An exchange whose own signature was
// tuned takes its passes and shape; what else was tuned changes nothing.
// False when some edge is not of this kind, or the tuned shape needs another
// kernel.
static bool run_single_objects(const CopyEdge *edges, int n, cudaStream_t s,
                               int *err) {
  SmallPair entries[kParamRegions];
  int used = 0;
  uint64_t chunks = 0;
  for (int i = 0; i < n; ++i) {
    const CopyEdge &e = edges[i];
    if (e.src_count == 0 && e.dst_count == 0)
      continue;
    if (used == kParamRegions)
      return false;
    const TypeRecord &a = *e.src_type, &b = *e.dst_type;
    if (e.src_count != 1 || e.dst_count != 1 || !a.has_unit || !b.has_unit ||
        a.unit[4].nd > 2 || b.unit[4].nd > 2)
      return false;
    CopyPair p = unit_pair(e, uint32_t(chunks));
    p.passes = default_passes(region_class(p.gs));
    entries[used++] = make_small(p);
    chunks += chunks_of(p.gs, p.passes, true);
  }
  Tuned tuned;
  if (anything_tuned() && !take_tuned(edges, n, entries, &chunks, &tuned))
    return false;
  if (chunks > UINT32_MAX)
    return false;
  *err = used ? launch_param(entries, used, uint32_t(chunks), 0,
                             tuned.shape.ctas_per_sm, s)
              : TEMPI_OK;
  if (!*err && used)
    set_last_kernel("batch_copy");
  counters().neighbor_unit++;
  return true;
}

// One copy batch on `s`.  Up to kParamRegions pairs of at most two strided
// dimensions (a halo's 26) travel in the kernel's parameters: nothing is
// uploaded, whatever regions the previous call had.  Larger tables go to a
// grow-only device buffer: no allocation once it is large enough, and no copy
// while it holds the same entries byte for byte (a loop that exchanges the same
// regions every step uploads them once: 33 edges 15.7 us a call, 18.4 with the
// copy; 200 edges 32.7 and 35.5; 26 edges of three strided dimensions 17.3 and
// 20.0).  Every call is on `s`, TEMPI's one stream, so a new table is copied
// behind the launches that read the old one.
int copy_batch_run(const CopyEdge *edges, int n, cudaStream_t s) {
  static std::mutex mu;
  static void *table = nullptr;
  // room for 64 full entries or 164 compact ones, so that exchanges of a few
  // more edges each do not free and allocate every time
  constexpr size_t kLeastTable = 64 * sizeof(CopyPair);
  static size_t capacity = 0; // bytes
  static std::vector<char> on_device; // the entries in the table
  static std::vector<CopyPair> pairs;
  std::lock_guard<std::mutex> l(mu);
  int err;
  if (run_single_objects(edges, n, s, &err))
    return err;
  std::vector<tempi_copy_region> regions(static_cast<size_t>(n));
  for (int i = 0; i < n; ++i) {
    const CopyEdge &e = edges[i];
    regions[i] = {e.src_origin, e.dst_origin, e.src_type->desc,
                  e.dst_type->desc, e.src_count, e.dst_count};
  }
  uint64_t chunks = 0;
  err = build_pairs(regions.data(), n, &pairs, &chunks);
  if (err || pairs.empty())
    return err;
  // a batch of a tuned signature takes the tuned choices
  Tuned tuned;
  if (anything_tuned() && find_tuned(pairs.data(), pairs.size(), 0, &tuned))
    chunks = apply_passes(pairs, &tuned);
  const Shape shape = tuned.shape;
  const int count = int(pairs.size());
  const bool small = all_small(pairs);
  if (small && count <= kParamRegions && param_shape(shape)) {
    SmallPair entries[kParamRegions];
    for (int i = 0; i < count; ++i)
      entries[i] = make_small(pairs[i]);
    err = launch_param(entries, count, uint32_t(chunks), 0, shape.ctas_per_sm, s);
    if (!err)
      set_last_kernel("batch_copy");
    return err;
  }
  std::vector<SmallPair> entries;
  if (small)
    entries = small_table(pairs);
  const void *from = small ? static_cast<const void *>(entries.data())
                           : static_cast<const void *>(pairs.data());
  const size_t bytes = pairs.size() * (small ? sizeof(SmallPair) : sizeof(CopyPair));
  if (bytes > capacity) {
    cudaFree(table);
    table = nullptr;
    capacity = 0;
    on_device.clear();
    const size_t want = std::max(bytes, kLeastTable);
    cudaError_t e = cudaMalloc(&table, want);
    if (e != cudaSuccess)
      return cuda_error(e, "copy table allocation");
    capacity = want;
    counters().neighbor_tables++;
  }
  const char *b = static_cast<const char *>(from);
  if (on_device.size() != bytes || std::memcmp(on_device.data(), b, bytes) != 0) {
    on_device.clear();
    cudaError_t e = cudaMemcpyAsync(table, from, bytes, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess)
      return cuda_error(e, "copy table upload");
    on_device.assign(b, b + bytes);
    counters().neighbor_uploads++;
  }
  return launch_table<CopyPair>(table, count, small, uint32_t(chunks), 0, shape, s,
                                false);
}

} // namespace tempi

extern "C" int tempi_batch_launch(tempi_batch *b, void *stream) {
  if (!b)
    return set_error(TEMPI_ERR_ARG, "null batch");
  return batch_launch(b, static_cast<cudaStream_t>(stream), true);
}

static void drop_graph(BatchImpl &bi) {
  if (bi.exec) {
    cudaGraphExecDestroy(bi.exec);
    cudaGraphDestroy(bi.graph);
    bi.exec = nullptr;
    bi.graph = nullptr;
  }
}

extern "C" int tempi_batch_capture(tempi_batch *b, void *stream) {
  if (!b)
    return set_error(TEMPI_ERR_ARG, "null batch");
  BatchImpl &bi = b->impl;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  drop_graph(bi);
  cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess)
    return cuda_error(e, "begin capture");
  int err = batch_launch(b, s, false);
  e = cudaStreamEndCapture(s, &bi.graph);
  if (err)
    return err;
  if (e != cudaSuccess)
    return cuda_error(e, "end capture");
  e = cudaGraphInstantiate(&bi.exec, bi.graph, 0);
  if (e != cudaSuccess)
    return cuda_error(e, "graph instantiate");
  return TEMPI_OK;
}

extern "C" int tempi_batch_replay(tempi_batch *b, void *stream) {
  if (!b || !b->impl.exec)
    return set_error(TEMPI_ERR_ARG, "batch has no captured graph");
  cudaError_t e = cudaGraphLaunch(b->impl.exec, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess)
    return cuda_error(e, "graph launch");
  if (!b->impl.host.empty() || !b->impl.host_pairs.empty())
    counters().kernel_launches++;
  return TEMPI_OK;
}

// ---- the autotuner ----------------------------------------------------------

namespace {

// median device time (ms) of `reps` launches of the batch as configured,
// the L2 flushed before each
float time_batch(tempi_batch *b, cudaStream_t s, const uint4 *flush,
                 size_t flush_words, unsigned *sink, cudaEvent_t e0,
                 cudaEvent_t e1, int reps, int *err) {
  std::vector<float> ts;
  for (int r = 0; r < reps && !*err; ++r) {
    k_tune_flush<<<num_sms() * 8, 256, 0, s>>>(flush, flush_words, sink);
    cudaEventRecord(e0, s);
    *err = batch_launch(b, s, false);
    cudaEventRecord(e1, s);
    if (cudaEventSynchronize(e1) != cudaSuccess) {
      *err = cuda_error(cudaGetLastError(), "tuning launch");
      break;
    }
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    ts.push_back(ms);
  }
  if (ts.empty())
    return 1e30f;
  std::sort(ts.begin(), ts.end());
  return ts[ts.size() / 2];
}

// re-plan the records with `t`, upload the table
int replan(tempi_batch *b, const Tuned &t) {
  BatchImpl &bi = b->impl;
  bi.shape = t.shape;
  uint64_t chunks;
  int err;
  if (!bi.host_pairs.empty()) {
    chunks = apply_passes(bi.host_pairs, &t);
  } else {
    chunks = apply_passes(bi.host, &t);
  }
  err = upload_table(bi);
  if (chunks > UINT32_MAX)
    return set_error(TEMPI_ERR_ARG, "batch too large");
  bi.total_chunks = uint32_t(chunks);
  return err;
}

template <typename Rec> std::vector<int> classes_of(const std::vector<Rec> &recs) {
  std::vector<int> out;
  for (const Rec &r : recs)
    out.push_back(region_class(geometry_of(r)));
  std::sort(out.begin(), out.end());
  out.erase(std::unique(out.begin(), out.end()), out.end());
  return out;
}

} // namespace

extern "C" int tempi_batch_tune(tempi_batch *b, void *stream, int32_t reps) {
  if (!b)
    return set_error(TEMPI_ERR_ARG, "null batch");
  BatchImpl &bi = b->impl;
  if (bi.host.empty() && bi.host_pairs.empty())
    return TEMPI_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  reps = std::max(1, std::min(50, int(reps)));
  // Launches of this batch may be in flight on any stream; they read the table
  // that every plan below rewrites.
  if (cudaDeviceSynchronize() != cudaSuccess)
    return cuda_error(cudaGetLastError(), "tuning: launches before it");
  drop_graph(bi);
  int dev = 0, l2 = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev) != cudaSuccess)
    l2 = 128 << 20;
  const size_t flush_bytes = (size_t(l2) * 2 + 15) & ~size_t(15);
  void *flush = nullptr;
  unsigned *sink = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t ce = cudaMalloc(&flush, flush_bytes + 16);
  if (ce == cudaSuccess)
    ce = cudaMemsetAsync(flush, 0, flush_bytes + 16, s);
  if (ce == cudaSuccess)
    ce = cudaEventCreate(&e0);
  if (ce == cudaSuccess)
    ce = cudaEventCreate(&e1);
  int err = ce == cudaSuccess ? TEMPI_OK : cuda_error(ce, "tuning set-up");
  sink = reinterpret_cast<unsigned *>(static_cast<char *>(flush) + flush_bytes);
  const uint4 *fl = static_cast<const uint4 *>(flush);
  const size_t fw = flush_bytes / 16;
  Tuned best = bi.has_tuned ? bi.tuned : Tuned{};
  const std::vector<int> cls = !bi.host_pairs.empty() ? classes_of(bi.host_pairs)
                                                      : classes_of(bi.host);
  float t_best = 1e30f;
  if (!err) {
    err = replan(b, best);
    if (!err) {
      time_batch(b, s, fl, fw, sink, e0, e1, 2, &err); // warm
      t_best = time_batch(b, s, fl, fw, sink, e0, e1, reps, &err);
    }
  }
  // each class's passes in turn, the others held
  for (int c : cls) {
    for (int p : kPassChoices) {
      if (err)
        break;
      Tuned t = best;
      t.passes[c] = uint8_t(p);
      if ((best.passes[c] ? best.passes[c] : default_passes(c)) == uint32_t(p))
        continue;
      err = replan(b, t);
      const float tt = err ? 1e30f : time_batch(b, s, fl, fw, sink, e0, e1, reps, &err);
      if (tt < t_best) {
        t_best = tt;
        best = t;
      }
    }
  }
  // then the launch shape
  for (int th : {128, 256, 512}) {
    for (int cps : {1, 2, 3, 4, 6, 8, 12, 16}) {
      if (err)
        break;
      Tuned t = best;
      t.shape.threads = th;
      t.shape.ctas_per_sm = cps;
      if (cps > max_ctas(!bi.host_pairs.empty() ? kind_of<CopyPair>(bi.small, 0)
                                            : kind_of<BatchRegion>(bi.small, bi.unpack),
                         th, 0) ||
          (th == best.shape.threads && cps == best.shape.ctas_per_sm))
        continue;
      err = replan(b, t);
      const float tt = err ? 1e30f : time_batch(b, s, fl, fw, sink, e0, e1, reps, &err);
      if (tt < t_best) {
        t_best = tt;
        best = t;
      }
    }
  }
  if (!err)
    err = replan(b, best);
  if (e0)
    cudaEventDestroy(e0);
  if (e1)
    cudaEventDestroy(e1);
  cudaStreamSynchronize(s);
  cudaFree(flush);
  if (err)
    return err;
  for (int c = 0; c < kClasses; ++c) // record resolved choices
    if (!best.passes[c])
      best.passes[c] = uint8_t(default_passes(c));
  bi.tuned = best;
  bi.has_tuned = true;
  std::lock_guard<std::mutex> l(g_tune_mu);
  load_tuned_locked();
  g_tuned[bi.sig] = best;
  if (FILE *f = std::fopen(tune_path().c_str(), "a")) {
    std::fprintf(f, "%llx %d %d", (unsigned long long)bi.sig, best.shape.threads,
                 best.shape.ctas_per_sm);
    for (int c = 0; c < kClasses; ++c)
      std::fprintf(f, " %u", unsigned(best.passes[c]));
    std::fprintf(f, "\n");
    std::fclose(f);
  }
  return TEMPI_OK;
}

extern "C" int tempi_batch_config(const tempi_batch *b, int32_t *threads,
                                  int32_t *ctas_per_sm, int32_t *classes,
                                  int32_t *passes, int32_t max_classes) {
  if (!b)
    return -set_error(TEMPI_ERR_ARG, "null batch");
  const BatchImpl &bi = b->impl;
  if (threads)
    *threads = bi.shape.threads;
  if (ctas_per_sm)
    *ctas_per_sm = bi.shape.ctas_per_sm;
  std::vector<std::pair<int, int>> cu;
  auto add = [&](const Geometry &g, uint32_t u) { // u: passes
    const int c = region_class(g);
    for (auto &p : cu)
      if (p.first == c)
        return;
    cu.push_back({c, int(u)});
  };
  for (const BatchRegion &r : bi.host)
    add(r.g, r.passes);
  for (const CopyPair &r : bi.host_pairs)
    add(r.gs, r.passes);
  std::sort(cu.begin(), cu.end());
  int k = 0;
  for (auto &p : cu) {
    if (k >= max_classes)
      break;
    if (classes)
      classes[k] = p.first;
    if (passes)
      passes[k] = p.second;
    ++k;
  }
  return k;
}

// ---- batched pack without allocation ------------------------------------
//
// tempi_batch_create puts the region table in memory it obtains with
// cudaMalloc.  Some callers cannot allocate device memory where they pack:
// a halo-exchange step inside a latency-critical loop (cudaMalloc can
// synchronise the whole device), or an application whose memory pool
// already owns the GPU's memory, so any further cudaMalloc fails.  For them
// tempi_batch_run_static keeps the table in the fixed array below instead.
//
// The array is a file-scope device variable: every GPU that loads this
// library holds it (kStaticBatchRegions = 1024 entries of 168 B: 168 KiB) until the
// process exits.  Host code cannot use the name `g_static_regions` as a
// device address (it denotes a host-side stand-in), so the first call on
// each device, with that device current, asks the runtime for the array's
// device address once (cudaGetSymbolAddress) and every call passes that
// address to the kernel.  Because of that set-up, the first call on a
// device should come before any stream capture.  The cached address is not
// refreshed if the application resets the device (cudaDeviceReset).
//
// A table of up to kParamRegions entries is passed BY VALUE as the batch
// kernel's own parameter (k_batch_param_small, or k_batch_param where a region
// has more than two strided dimensions): one launch, the array untouched.
// A larger table reaches the array without a host-to-device copy: the host
// builds it in pieces of up to kFillPiece entries and passes each piece BY
// VALUE as the parameter of a small kernel (k_static_fill) that writes it
// into the array, on the caller's stream ahead of the batch kernel.  Kernel
// parameters are copied when the launch is issued, so the host's piece can
// be reused at once, and the host never waits for earlier work on the
// stream (a copy from pageable host memory would).  All calls share the one
// array and it keeps the last call's table; each call rewrites every entry
// it uses, so nothing needs clearing, but calls whose launches can overlap
// on the GPU (different streams, no ordering) race on the table.
constexpr int kStaticBatchRegions = 1024;
constexpr int kMaxDevices = 64;
constexpr int kFillPiece = 128; // 21.5 KB of parameters (the limit is 32,764 B)

static_assert(sizeof(BatchRegion) == 168 && sizeof(BatchRegion) % 4 == 0,
              "table entry size is documented");
static __device__ __align__(256) BatchRegion g_static_regions[kStaticBatchRegions];
static_assert(sizeof(StaticPiece<kFillPiece>) + 8 <= 32764,
              "a piece fits the kernel parameter space");

// entries [first, first + count) of the array from the piece, a 32-bit
// word per thread; the host guarantees first + count <= kStaticBatchRegions
// and count <= P
template <int P, typename Rec>
__global__ void __launch_bounds__(256)
    k_static_fill(const __grid_constant__ StaticPiece<P, Rec> piece, int first,
                  int count) {
  constexpr int kWords = sizeof(Rec) / 4;
  const uint32_t *from = reinterpret_cast<const uint32_t *>(piece.r);
  uint32_t *to = reinterpret_cast<uint32_t *>(g_static_regions) + first * kWords;
  for (int w = threadIdx.x; w < count * kWords; w += blockDim.x)
    to[w] = from[w];
}

static std::mutex g_static_mu;
static BatchRegion *g_static_ptr[kMaxDevices] = {};

static int static_table(BatchRegion **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess)
    return cuda_error(e, "cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices)
    return set_error(TEMPI_ERR_ARG, "device %d out of range", dev);
  std::lock_guard<std::mutex> l(g_static_mu);
  if (!g_static_ptr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_regions);
    if (e != cudaSuccess)
      return cuda_error(e, "cudaGetSymbolAddress of the static region table");
    g_static_ptr[dev] = static_cast<BatchRegion *>(p);
  }
  *out = g_static_ptr[dev];
  return TEMPI_OK;
}

// launch k_static_fill for entries [first, first + count) of `piece`
template <typename Rec>
static int static_fill(const StaticPiece<kFillPiece, Rec> &piece, int first,
                       int count, cudaStream_t s) {
  if (count <= 32) { // a small table: a quarter of the parameter block
    StaticPiece<32, Rec> few;
    std::memcpy(few.r, piece.r, size_t(count) * sizeof(Rec));
    k_static_fill<32, Rec><<<1, 256, 0, s>>>(few, first, count);
  } else {
    k_static_fill<kFillPiece, Rec><<<1, 256, 0, s>>>(piece, first, count);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
    return cuda_error(e, "static region table fill");
  counters().kernel_launches++;
  return TEMPI_OK;
}

// the same from full entries, compacted first when `small`
static int static_fill(const StaticPiece<kFillPiece> &piece, int first,
                       int count, bool small, cudaStream_t s) {
  if (!small)
    return static_fill<BatchRegion>(piece, first, count, s);
  StaticPiece<kFillPiece, SmallRegion> compact;
  for (int i = 0; i < count; ++i)
    compact.r[i] = make_small(piece.r[i]);
  return static_fill<SmallRegion>(compact, first, count, s);
}

extern "C" int tempi_batch_run_static(const tempi_region *regions, int32_t n,
                                      int32_t unpack, void *stream) {
  if (n < 0 || (n > 0 && !regions))
    return set_error(TEMPI_ERR_ARG, "bad batch arguments");
  if (n > kStaticBatchRegions)
    return set_error(TEMPI_ERR_ARG,
                     "tempi_batch_run_static takes at most %d regions, got %d",
                     kStaticBatchRegions, n);
  BatchRegion *table = nullptr;
  int err = static_table(&table);
  if (err)
    return err;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // every region is checked before anything is launched, so a bad region
  // leaves the array and the stream untouched
  StaticPiece<kFillPiece> piece;
  int used = 0, filled = 0;
  uint64_t chunks = 0;
  uint64_t compact = 0;
  bool small = true; // every entry, once pass 0 is over
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1 && used <= kParamRegions) { // pass 0 left them all in piece
      if (used == 0)
        return TEMPI_OK;
      if (small) {
        SmallRegion few[kParamRegions];
        chunks = 0;
        for (int i = 0; i < used; ++i) {
          piece.r[i].chunk_begin = uint32_t(chunks);
          chunks += chunks_of(piece.r[i].g, piece.r[i].passes, true);
          few[i] = make_small(piece.r[i]);
        }
        err = launch_param(few, used, uint32_t(chunks), unpack ? 1 : 0, 0, s);
      } else {
        err = launch_param(piece.r, used, uint32_t(chunks), unpack ? 1 : 0, 0, s);
      }
      if (!err)
        set_last_kernel(unpack ? "batch_unpack_static" : "batch_pack_static");
      return err;
    }
    used = filled = 0;
    chunks = 0;
    for (int32_t i = 0; i < n; ++i) {
      const tempi_region &r = regions[i];
      BatchRegion &br = piece.r[filled];
      br = BatchRegion{};
      char *strided = (char *)r.origin + r.desc.start;
      bool empty = false;
      err = make_geometry(&r.desc, r.incount, uintptr_t(strided),
                          uintptr_t(r.packed), 0, &br.g, &empty);
      if (err)
        return err;
      if (empty)
        continue;
      br.strided = strided;
      br.packed = (char *)r.packed;
      br.passes = default_passes(region_class(br.g));
      small = small && is_small(br); // settled by pass 0
      br.chunk_begin = uint32_t(chunks);
      chunks += chunks_of(br.g, br.passes, pass == 1 && small);
      if (chunks > UINT32_MAX)
        return set_error(TEMPI_ERR_ARG, "batch too large");
      if (pass == 0) {
        compact += chunks_of(br.g, br.passes, true);
        small = small && compact <= UINT32_MAX;
      }
      if (++filled == kFillPiece) {
        if (pass == 1 && (err = static_fill(piece, used, filled, small, s)))
          return err;
        used += filled;
        filled = 0;
      }
    }
    if (filled) { // a partial last piece (empty regions are never stored)
      if (pass == 1 && (err = static_fill(piece, used, filled, small, s)))
        return err;
      used += filled;
      filled = 0;
    }
  }
  if (used == 0)
    return TEMPI_OK;
  err = launch_table<BatchRegion>(table, used, small, uint32_t(chunks), unpack ? 1 : 0,
                                  Shape{}, s, false);
  if (err)
    return err;
  set_last_kernel(unpack ? "batch_unpack_static" : "batch_pack_static");
  return TEMPI_OK;
}

extern "C" int tempi_batch_destroy(tempi_batch *b) {
  if (!b)
    return TEMPI_OK;
  if (b->impl.exec)
    cudaGraphExecDestroy(b->impl.exec);
  if (b->impl.graph)
    cudaGraphDestroy(b->impl.graph);
  cudaFree(b->impl.dev);
  delete b;
  return TEMPI_OK;
}
