// uc_sort.cu — the lines of a finished job in byte order (sorted output).
//
// Every line begins with a distinct k-mer, so its first k chars order it, and
// most lines are that k-mer plus a few chars.  A line is therefore sorted as
// a record that holds all of it in 2-bit codes (one or two key words and a
// tail word), and the sorted text is spelled from the records:
//   (k_tile_warp   closed lines of warp tiles come as records already)
//   k_line_recs    text -> records, and a count per bin of leading key bits
//   k_line_plan    bins -> tiles of about TILE_WINDOW records
//   k_line_group   records -> their tiles (by groups of tiles first)
//   k_line_tiles   one block per tile: order in shared memory, the tile's
//                  place in the output by look-back, lines spelled and stored
// Nothing returns to the host in between, unless a bin holds many tiles' worth
// of lines (low-complexity k-mers: thousands of lines with the same first
// chars).  Such bins are sorted by the whole grid first (k_over_count,
// k_over_pass).  The text is read once and written once.  Lines with more than
// TAIL_MAX chars after the k-mer keep their chars in a copy and are copied.
//
// 256 Mbp, k = 31 (107M lines, 3.6 GB, a fifth of them reaching the sort as
// text) on a B200: 0.42 + 2.2 + 3.0 ms (records, groups, tiles), where a radix
// sort of (key, line index) pairs with a gather of the lines (seven passes over
// pairs or lines) took 28 ms.
#include <algorithm>
#include <cstring>
#include <utility>

#include "uc_kernels.cuh"
#include "uc_lookback.cuh"
#include "uc_pipeline.h"

namespace uc {

namespace {

constexpr unsigned long long HUGE_LINE = 1ull << 16; // bytes from which a line is copied by the whole grid

constexpr uint32_t LR_CHUNK = 16384;  // text bytes whose line starts one block pass takes
constexpr uint32_t LR_PRE = 16;       // bytes before them (the line break before the first start)
constexpr uint32_t LR_HALO = 112;     // bytes after them: k + TAIL_MAX + 1 <= 92, read in words
constexpr uint32_t LR_PIECES = (LR_PRE + LR_CHUNK + LR_HALO) / 16;

constexpr uint32_t TILE_THREADS = 256;
constexpr uint32_t TILE_SUB = 2048;  // sub-bins of a tile
// records a tile sorts in shared memory: four blocks per SM (three with two
// key words) fit
template <int RW>
__host__ __device__ constexpr uint32_t tile_cap() {
  return RW == 2 ? 2048u : 1536u;
}
// records per tile, give or take a bin (not a power of two: the tiles fill at one
// pace, and with windows of 1024 their write frontiers lay 16 KB apart, in few
// of L2's slices and sets)
constexpr uint32_t WIN = 1000;
constexpr uint32_t PLAN_ITEMS = 16;  // bins per thread of the plan
// Cursors lie 32 bytes apart: atomics on words of one L2 line queue up (about
// 2 ns each).
constexpr uint32_t CUR_STRIDE = 8;

struct LongLine {
  unsigned long long at;   // offset in the text
  unsigned long long kept; // of the copy of its chars
  unsigned long long len;  // bytes, line break included
  unsigned long long to;   // of a huge line: offset in the sorted text
};

struct SortCtr {
  uint32_t nrec, nhuge, ntiles, pad;
  unsigned long long longs;  // long lines (low half), 16-byte units of their copies (high half)
  uint32_t plan_ticket, tile_ticket, fail;
  uint32_t nover;  // oversized bins
};

// An oversized bin's records are sorted beforehand and cut into tiles of their
// own, marked in the tile's first bin.
constexpr uint32_t TILE_RUN = 0x80000000u;
// A bin is oversized from OVER_WINS windows on.  It then spans OVER_WINS tile
// numbers at least, of which all but the last are its own: at most 1.5 windows
// per tile, which fit.  Below that a tile of more than its capacity (6 windows at
// most) is sorted by its block.  At most OVER_MAX bins are oversized (the limit
// grows with the number of lines).
constexpr uint32_t OVER_WINS = 5, OVER_MAX = 4096;
struct OverBin {
  uint32_t beg, n;   // records
  uint32_t tile, nt; // tiles of its own
};
static_assert(WIN + WIN / 2 + 1 <= tile_cap<2>() && WIN + WIN / 2 + 1 <= tile_cap<3>(), "its tiles fit");

__device__ __forceinline__ unsigned long long line_bytes_of(uint64_t tail, int k, const LongLine* longs) {
  return (tail & TAIL_LONG) ? longs[uint32_t(tail)].len : uint64_t(k) + 1u + ((tail >> TAIL_LEN_SHIFT) & 31u);
}

// Text -> records.  A block reads a chunk of text with 16-byte loads and keeps
// its 2-bit codes and a bit per line break in shared memory (the text itself
// is not staged: a line's key and tail are then a few funnel shifts of code
// words), lists the chunk's line starts from the bits (two words per thread,
// one block scan), and makes one line's record per thread.
// The records come in no particular order: a block reserves the places of its
// lines with one atomic.  256 Mbp, k = 31: 0.42 ms for the lines that are not
// records already; 1.9 ms when it took all of them (5.3 GB), bound by issue (60%)
// and barriers, where converting each line from staged text took 2.3.
template <int RW>
__global__ void __launch_bounds__(256, 5) k_line_recs(const char* __restrict__ out, uint64_t n, int k, int bits,
                                                   RecArr<RW> rec, uint32_t* __restrict__ counts,
                                                   LongLine* __restrict__ longs, uint32_t* __restrict__ huge,
                                                   SortCtr* sc) {
  __shared__ uint32_t code[LR_PIECES];  // 16 chars each
  __shared__ __align__(16) uint32_t nlw[LR_PIECES / 2 + 1];
  __shared__ uint32_t scan[33];
  __shared__ uint32_t s_base, s_open;
  __shared__ unsigned long long s_end;
  extern __shared__ uint16_t starts[];  // LR_CHUNK / (k + 1) + 2
  uint16_t* nl16 = reinterpret_cast<uint16_t*>(nlw);
  const uint32_t tid = threadIdx.x;
  // positions are relative to the 16-byte boundary at or below out
  const char* A = reinterpret_cast<const char*>(reinterpret_cast<uintptr_t>(out) & ~uintptr_t(15));
  const uint64_t off0 = uint64_t(out - A), end = off0 + n;
  const uint64_t nchunks = (end + LR_CHUNK - 1) / LR_CHUNK;
  const uint64_t m0 = (2 * k >= 64) ? ~0ull : ((1ull << (2 * k)) - 1ull);
  for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
    const uint64_t c0 = c * LR_CHUNK;
    // (all loads of the chunk in flight together; a chunk inside the text
    // needs no checks)
    const bool inside = c0 >= off0 + LR_PRE && c0 + LR_CHUNK + LR_HALO <= end;
    constexpr uint32_t PP = (LR_PIECES + 255) / 256;
    uint4 v[PP];
#pragma unroll
    for (uint32_t q = 0; q < PP; ++q) {
      const uint32_t p = q * 256 + tid;
      const int64_t x = int64_t(c0) - int64_t(LR_PRE) + 16 * int64_t(p);
      v[q] = make_uint4(0x41414141u, 0x41414141u, 0x41414141u, 0x41414141u);
      if (p < LR_PIECES && (inside || (x >= int64_t(off0) && x + 16 <= int64_t(end))))
        v[q] = __ldcs(reinterpret_cast<const uint4*>(A + x));
    }
#pragma unroll
    for (uint32_t q = 0; q < PP; ++q) {
      const uint32_t p = q * 256 + tid;
      if (p >= LR_PIECES) break;
      const int64_t x = int64_t(c0) - int64_t(LR_PRE) + 16 * int64_t(p);
      if (!inside && (x < int64_t(off0) || x + 16 > int64_t(end)) && x + 16 > int64_t(off0) && x < int64_t(end)) {
        uint32_t w[4] = {0x41414141u, 0x41414141u, 0x41414141u, 0x41414141u};  // a piece at an end of the text
#pragma unroll
        for (int b = 0; b < 16; ++b)
          if (x + b >= int64_t(off0) && x + b < int64_t(end))
            w[b >> 2] ^= (uint32_t(static_cast<unsigned char>(A[x + b])) ^ 0x41u) << (8 * (b & 3));
        v[q] = make_uint4(w[0], w[1], w[2], w[3]);
      }
      code[p] = codes16(v[q]);
      nl16[p] = uint16_t(breaks16(v[q]));
    }
    if (tid == 0) {
      s_open = 0;
      nlw[LR_PIECES / 2] = 0;
    }
    __syncthreads();
    // a line starts after each line break, and at the text's first byte
    uint32_t sb[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t w = 2 * tid + q;
      uint32_t b = __funnelshift_r(nlw[w], nlw[w + 1], LR_PRE - 1);
      const uint64_t x0 = c0 + 32ull * w;
      if (x0 == 0) b |= 1u << off0;
      if (x0 + 32 > end) b &= (x0 >= end) ? 0u : (0xFFFFFFFFu >> (32u - uint32_t(end - x0)));
      sb[q] = b;
    }
    uint32_t nl;
    uint32_t at = block_excl_scan(uint32_t(__popc(sb[0]) + __popc(sb[1])), scan, &nl);
    const uint32_t cap = LR_CHUNK / (uint32_t(k) + 1u) + 2u;
    if (nl > cap) {  // a line shorter than k: not this library's output
      if (tid == 0) atomicOr(&sc->fail, 2u);
      nl = 0;
    }
    if (nl) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        for (uint32_t b = sb[q]; b; b &= b - 1) starts[at++] = uint16_t(64 * tid + 32 * q + (__ffs(b) - 1));
    }
    if (tid == 0) s_base = nl ? atomicAdd(&sc->nrec, nl) : 0u;
    __syncthreads();
    // len: chars of the line; returns its bin
    auto emit = [&](uint32_t j, uint32_t s, unsigned long long len) -> uint32_t {
      const bool is_long = len > uint64_t(k + TAIL_MAX);
      const uint32_t t = is_long ? 0u : uint32_t(len) - uint32_t(k);
      // the line's code stream from its first char (words past the halo are
      // not reached: k + TAIL_MAX chars at most count)
      const uint32_t wi = (LR_PRE + s) >> 4, sh = 2u * ((LR_PRE + s) & 15u);
      constexpr int NC = RW == 2 ? 4 : 6;
      uint32_t c[NC + 1], x[NC];
#pragma unroll
      for (int q = 0; q <= NC; ++q) c[q] = code[wi + q];
#pragma unroll
      for (int q = 0; q < NC; ++q) x[q] = __funnelshift_r(c[q], c[q + 1], sh);
      const uint64_t s0 = x[0] | (uint64_t(x[1]) << 32), s1 = x[2] | (uint64_t(x[3]) << 32);
      uint64_t tl;
      Rec<RW> r;
      if constexpr (RW == 2) {
        r.hi = rev2(s0 & m0);
        r.lo = 0;
        tl = (s0 >> (2 * k)) | (s1 << (64 - 2 * k));
      } else {
        const uint64_t s2 = x[NC - 2] | (uint64_t(x[NC - 1]) << 32);
        const int u = 2 * k - 64;
        r.hi = rev2(s0);
        r.lo = rev2(s1 & ((1ull << u) - 1ull));
        tl = u ? ((s1 >> u) | (s2 << (64 - u))) : s1;
      }
      if (is_long) {
        const unsigned long long v = atomicAdd(&sc->longs, (((len + 16) >> 4) << 32) | 1ull);
        const uint32_t i = uint32_t(v);
        longs[i] = LongLine{c0 + s - off0, (v >> 32) << 4, len + 1, 0ull};
        if (len + 1 >= HUGE_LINE) huge[atomicAdd(&sc->nhuge, 1u)] = i;
        r.tail = TAIL_LONG | i;
      } else {
        r.tail = (uint64_t(t) << TAIL_LEN_SHIFT) | (tl & ((1ull << (2 * t)) - 1ull));
      }
      st_rec<RW>(rec, s_base + j, r);
      return uint32_t(r.hi >> (64 - bits));
    };
    for (uint32_t j0 = 0; j0 < nl; j0 += 256) {  // (whole warps together)
      const uint32_t j = j0 + tid, s = j < nl ? starts[j] : 0u;
      uint32_t len = 0, bin = NONE;
      if (j >= nl) {
        // no line
      } else if (j + 1 < nl) {
        len = uint32_t(starts[j + 1]) - s - 1u;
      } else {
        // the chunk's last line: its break in the bits, or past the halo
        const uint32_t i0 = LR_PRE + s + uint32_t(k);
        uint32_t w = i0 >> 5, m = nlw[w] & (0xFFFFFFFFu << (i0 & 31u));
        while (!m && ++w < LR_PIECES / 2) m = nlw[w];
        len = m ? 32u * w + uint32_t(__ffs(m) - 1) - LR_PRE - s : 0u;
        if (!m) s_open = j + 1u;
      }
      if (len >= uint32_t(k)) bin = emit(j, s, len);
      else if (j < nl && (len || j + 1 < nl)) atomicOr(&sc->fail, 2u);
      count_bin(counts, bin);
    }
    __syncthreads();
    if (s_open) {
      // the last line goes on past the halo: the whole block looks for its break
      const uint32_t j = s_open - 1u, s = starts[j];
      if (tid == 0) s_end = end;
      __syncthreads();
      for (uint64_t x0 = c0 + LR_CHUNK + LR_HALO; x0 < end; x0 += 8u * 16u * 256u) {
        unsigned long long found = end;
#pragma unroll
        for (int q = 7; q >= 0; --q) {
          const uint64_t x = x0 + 16u * (uint32_t(q) * 256u + tid);
          if (x + 16 <= end) {
            const uint4 v = __ldcs(reinterpret_cast<const uint4*>(A + x));
            const uint32_t m = breaks16(v);
            if (m) found = x + uint32_t(__ffs(m) - 1);
          } else {
            for (uint64_t y = end; y > x;) {
              --y;
              if (A[y] == '\n') found = y;
            }
          }
        }
        if (found < end) atomicMin(&s_end, found);
        __syncthreads();
        const bool stop = s_end < end;
        __syncthreads();
        if (stop) break;
      }
      if (tid == 0) atomicAdd(counts + emit(j, s, s_end - (c0 + s)), 1u);
    }
    __syncthreads();  // code, nlw, starts are reused
  }
}

// Bins -> tiles.  Tile t takes the bins whose first record's rank lies in
// [t * win, (t + 1) * win), so a tile holds at most one window and the rest of
// its last bin.  One pass: prefix sums by look-back, each bin's tile in place
// of its count, each tile's first record and first bin, and the cursors of
// the tiles and of the groups of 2^gsh tiles.
//
// A bin of more than `big` records is listed, and gets the tile numbers that
// lie inside it alone: its records go to the first of them as one run, which
// k_over_items cuts into tiles of equal size.
__global__ void __launch_bounds__(256) k_line_plan(uint32_t* __restrict__ counts, uint32_t m, uint32_t win,
                                                   uint32_t big, OverBin* __restrict__ over,
                                                   uint2* __restrict__ tile, uint32_t* __restrict__ cur,
                                                   uint32_t* __restrict__ gcur, uint32_t gsh, unsigned long long* st,
                                                   SortCtr* sc) {
  __shared__ uint32_t scan[33];
  __shared__ uint32_t s_t, s_base;
  if (threadIdx.x == 0) s_t = atomicAdd(&sc->plan_ticket, 1u);
  __syncthreads();
  const uint32_t b = s_t;
  const uint32_t i0 = (b * 256u + threadIdx.x) * PLAN_ITEMS;
  uint32_t c[PLAN_ITEMS];
  uint32_t sum = 0;
  uint4* src = reinterpret_cast<uint4*>(counts + i0);
#pragma unroll
  for (uint32_t q = 0; q < PLAN_ITEMS / 4; ++q) {
    const uint4 v = i0 < m ? src[q] : make_uint4(0u, 0u, 0u, 0u);
    c[4 * q] = v.x;
    c[4 * q + 1] = v.y;
    c[4 * q + 2] = v.z;
    c[4 * q + 3] = v.w;
    sum += v.x + v.y + v.z + v.w;
  }
  uint32_t tot;
  const uint32_t pre = block_excl_scan(sum, scan, &tot);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) lb_publish(st, b, LB_SUM, tot);
    __syncwarp();
    const uint32_t e = uint32_t(lb_exclusive(st, b, tot, &sc->fail));
    if (threadIdx.x == 0) s_base = e;
  }
  __syncthreads();
  uint32_t p = s_base + pre;
  if (i0 >= m) return;
  if (i0 == 0) {
    tile[0] = make_uint2(0u, 0u);
    cur[0] = gcur[0] = 0;
  }
  uint32_t tp = p / win;
  uint32_t most = 0;
#pragma unroll
  for (uint32_t q = 0; q < PLAN_ITEMS; ++q) most = max(most, c[q]);
  if (most <= big) {
#pragma unroll
    for (uint32_t q = 0; q < PLAN_ITEMS; ++q) {
      const uint32_t nx = p + c[q], tn = nx / win;
      c[q] = tp;
      for (uint32_t t = tp + 1; t <= tn; ++t) {
        tile[t] = make_uint2(nx, i0 + q + 1);
        cur[t * CUR_STRIDE] = nx;
        if (!(t & ((1u << gsh) - 1u))) gcur[(t >> gsh) * CUR_STRIDE] = nx;
      }
      p = nx;
      tp = tn;
    }
#pragma unroll
    for (uint32_t q = 0; q < PLAN_ITEMS / 4; ++q)
      src[q] = make_uint4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
  } else {
    const uint32_t gm = (1u << gsh) - 1u;
#pragma unroll 1
    for (uint32_t q = 0; q < PLAN_ITEMS; ++q) {
      const uint32_t n = counts[i0 + q], nx = p + n, tn = nx / win;
      counts[i0 + q] = tp + (n > big ? 1u : 0u);
      if (n > big) {
        const uint32_t t0 = tp + 1u;
        over[atomicAdd(&sc->nover, 1u)] = OverBin{p, n, t0, tn - t0};
        tile[t0] = make_uint2(p, (i0 + q) | TILE_RUN);
        cur[t0 * CUR_STRIDE] = p;
        if (!(t0 & gm)) gcur[(t0 >> gsh) * CUR_STRIDE] = p;
        if (gsh)
          for (uint32_t t = (t0 | gm) + 1u; t < tn; t += gm + 1u) gcur[(t >> gsh) * CUR_STRIDE] = nx;
        tp = tn - 1u;
      }
      for (uint32_t t = tp + 1; t <= tn; ++t) {
        tile[t] = make_uint2(nx, i0 + q + 1);
        cur[t * CUR_STRIDE] = nx;
        if (!(t & gm)) gcur[(t >> gsh) * CUR_STRIDE] = nx;
      }
      p = nx;
      tp = tn;
    }
  }
  if (i0 + PLAN_ITEMS >= m) {
    tile[tp + 1] = make_uint2(p, m);
    sc->ntiles = tp + 1;
  }
}

// Records -> groups of 2^sh tiles (sh = 0: their tiles), in any order inside a
// group.  A block takes a chunk of records, counts them per group in shared
// memory, reserves one run per group present (cursors at cur) and writes the
// runs out.  Groups are counted from the chunk's lowest one; a record past
// the counted ones reserves its own place (a chunk that spans many groups:
// few records among bins that overflow their tiles).
//
// Records scattered one by one, each with its own atomic, ran at 32 to 45 G
// records/s whatever the occupancy (3.3 ms at 256 Mbp); as runs, two levels
// take 2.2 ms.  With at most GRP_BINS tiles one level does.
constexpr uint32_t GRP_THREADS = 512, GRP_BINS = 1024;
template <int RW>
__host__ __device__ constexpr uint32_t grp_chunk() {
  return RW == 2 ? 4096u : 2048u;
}
template <int RW>
__host__ __device__ constexpr size_t grp_smem() {
  return size_t(grp_chunk<RW>()) * (8 * RW + 2) + GRP_BINS * 8 + 16;
}
template <int RW>
__global__ void __launch_bounds__(GRP_THREADS, 2) k_line_group(RecArr<RW> in, RecArr<RW> to,
                                                               const uint32_t* __restrict__ tmap, int bits, uint32_t sh,
                                                               uint32_t* __restrict__ cur, const SortCtr* sc) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr uint32_t CH = grp_chunk<RW>(), PER = CH / GRP_THREADS, BPT = GRP_BINS / GRP_THREADS;
  static_assert(BPT == 2 && CH <= 4096, "a record's bin (10 bits) and its place in it share a word");
  ulonglong2* sa = reinterpret_cast<ulonglong2*>(sm);
  unsigned long long* stl = reinterpret_cast<unsigned long long*>(sa + CH);  // RW == 3
  uint32_t* lofs = reinterpret_cast<uint32_t*>(sm + size_t(CH) * 8 * RW);    // [GRP_BINS] counts, then offsets
  uint32_t* gofs = lofs + GRP_BINS;                                          // [GRP_BINS] global place of slot 0
  uint16_t* sbin = reinterpret_cast<uint16_t*>(gofs + GRP_BINS);             // [CH]
  __shared__ uint32_t scan[33], s_min;
  const uint32_t tid = threadIdx.x;
  if (sc->fail) return;
  const uint32_t n = sc->nrec;
  for (uint64_t c0 = uint64_t(blockIdx.x) * CH; c0 < n; c0 += uint64_t(gridDim.x) * CH) {
    const uint32_t cn = uint32_t(min(uint64_t(n) - c0, uint64_t(CH)));
    Rec<RW> r[PER];
    uint32_t g[PER], low = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q)
      if (q * GRP_THREADS + tid < cn) r[q] = ld_rec<RW>(in, c0 + q * GRP_THREADS + tid);
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
      g[q] = 0xFFFFFFFFu;
      if (q * GRP_THREADS + tid < cn) g[q] = tmap[r[q].hi >> (64 - bits)] >> sh;
      low = min(low, g[q]);
    }
    if (tid == 0) s_min = 0xFFFFFFFFu;
    lofs[2 * tid] = lofs[2 * tid + 1] = 0;
    __syncthreads();
    low = __reduce_min_sync(0xFFFFFFFFu, low);
    if ((tid & 31u) == 0) atomicMin(&s_min, low);
    __syncthreads();
    low = s_min;
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
      if (q * GRP_THREADS + tid >= cn) continue;
      const uint32_t b = g[q] - low;
      if (b < GRP_BINS) {
        g[q] = (atomicAdd(lofs + b, 1u) << 10) | b;
      } else {
        const uint32_t pos = atomicAdd(cur + g[q] * CUR_STRIDE, 1u);
        if (pos < n) st_rec<RW>(to, pos, r[q]);
        g[q] = 0xFFFFFFFFu;
      }
    }
    __syncthreads();
    uint32_t placed;
    {
      const uint32_t h0 = lofs[2 * tid], h1 = lofs[2 * tid + 1];
      const uint32_t pre = block_excl_scan(h0 + h1, scan, &placed);
      uint32_t* cc = cur + (low + 2 * tid) * CUR_STRIDE;
      lofs[2 * tid] = pre;
      lofs[2 * tid + 1] = pre + h0;
      if (h0) gofs[2 * tid] = atomicAdd(cc, h0) - pre;
      if (h1) gofs[2 * tid + 1] = atomicAdd(cc + CUR_STRIDE, h1) - (pre + h0);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
      if (q * GRP_THREADS + tid >= cn || g[q] == 0xFFFFFFFFu) continue;
      const uint32_t b = g[q] & (GRP_BINS - 1u), sl = lofs[b] + (g[q] >> 10);
      if constexpr (RW == 2) {
        sa[sl] = make_ulonglong2(r[q].hi, r[q].tail);
      } else {
        sa[sl] = make_ulonglong2(r[q].hi, r[q].lo);
        stl[sl] = r[q].tail;
      }
      sbin[sl] = uint16_t(b);
    }
    __syncthreads();
    for (uint32_t sl = tid; sl < placed; sl += GRP_THREADS) {
      const uint32_t pos = gofs[sbin[sl]] + sl;
      if (pos >= n) continue;  // (counts that disagree: nothing out of bounds)
      to.a[pos] = sa[sl];
      if constexpr (RW == 3) to.t[pos] = stl[sl];
    }
    __syncthreads();  // the shared arrays are reused
  }
}

// The chars of the long lines are kept: the sorted text overwrites them.
__global__ void __launch_bounds__(256) k_line_keep(const char* __restrict__ out, char* __restrict__ keep,
                                                   const LongLine* __restrict__ longs,
                                                   const uint32_t* __restrict__ huge, const SortCtr* sc) {
  const uint32_t nlong = uint32_t(sc->longs), nhuge = sc->nhuge;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = warp; i < nlong; i += nwarps) {
    const LongLine L = longs[i];
    if (L.len < HUGE_LINE) copy_bytes(keep + L.kept, out + L.at, L.len, threadIdx.x & 31u, 32u);
  }
  for (uint32_t h = 0; h < nhuge; ++h) {
    const LongLine L = longs[huge[h]];
    for (unsigned long long x = blockIdx.x * HUGE_LINE; x < L.len; x += gridDim.x * HUGE_LINE)
      copy_bytes(keep + L.kept + x, out + L.at + x, min(HUGE_LINE, L.len - x), threadIdx.x, blockDim.x);
  }
}

// The line (k-mer, tail, break) at shared-memory position pos of buf.
template <int RW>
__device__ __forceinline__ void spell_line(uint32_t* buf, uint32_t pos, const Rec<RW>& r, int k) {
  const uint32_t t = uint32_t(r.tail >> TAIL_LEN_SHIFT) & 31u;
  const uint64_t codes = r.tail & ((1ull << TAIL_LEN_SHIFT) - 1ull);
  constexpr int NC = RW == 2 ? 4 : 6;
  uint64_t w[3];
  w[0] = rev2(r.hi);
  w[1] = w[2] = 0;
  if constexpr (RW == 2) {
    w[0] |= codes << (2 * k);
    w[1] = codes >> (64 - 2 * k);
  } else {
    const int u = 2 * k - 64;
    w[1] = rev2(r.lo) | (codes << u);
    w[2] = u ? codes >> (64 - u) : 0ull;
  }
  uint32_t x[NC];
#pragma unroll
  for (int q = 0; q < NC; ++q) x[q] = uint32_t(w[q >> 1] >> (32 * (q & 1)));
  spell_text<NC>(buf, pos, x, uint32_t(k) + t, 1u);
}

// Stores the lines of ranks [r0, r1) of one warp, the first at byte `at` of
// the sorted text, 32 lines at a time.  get(r) gives the record of rank r.
template <int RW, class Get>
__device__ __forceinline__ void store_lines(char* out, uint64_t at, uint32_t r0, uint32_t r1, int k, uint32_t* buf,
                                            LongLine* longs, const char* keep, Get get) {
  const uint32_t lane = threadIdx.x & 31u;
  WarpText T;
  T.begin(out + at);
  for (uint32_t base = r0; base < r1; base += 32) {
    const bool live = base + lane < r1;
    Rec<RW> r{0ull, 0ull, 0ull};
    if (live) r = get(base + lane);
    const bool is_long = live && (r.tail & TAIL_LONG);
    const unsigned long long len = live ? line_bytes_of(r.tail, k, longs) : 0ull;
    if (__any_sync(0xFFFFFFFFu, is_long)) {
      T.end(buf);
      unsigned long long inc = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= uint32_t(o)) inc += v;
      }
      const unsigned long long total = __shfl_sync(0xFFFFFFFFu, inc, 31);
      if (live && !is_long) {
        // into the lane's own part of the buffer, then byte by byte
        char* p = T.dst + (inc - len);
        uint32_t* mine = buf + lane * ((uint32_t(k) + TAIL_MAX + 4u) >> 2);
        spell_line<RW>(mine, 0u, r, k);
        for (uint32_t q = 0; q < uint32_t(len); ++q) p[q] = reinterpret_cast<char*>(mine)[q];
      }
      uint32_t todo = __ballot_sync(0xFFFFFFFFu, is_long);
      while (todo) {
        const int q = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint32_t i = uint32_t(__shfl_sync(0xFFFFFFFFu, r.tail, q));
        const unsigned long long n = __shfl_sync(0xFFFFFFFFu, len, q);
        const unsigned long long o = __shfl_sync(0xFFFFFFFFu, inc - len, q);
        char* p = T.dst + o;
        const unsigned long long src = longs[i].kept;
        if (n < HUGE_LINE) copy_bytes(p, keep + src, n, lane, 32u);
        else if (lane == 0) longs[i].to = uint64_t(p - out);  // copied by k_huge_lines
      }
      __syncwarp();
      T.begin(T.dst + total);
      continue;
    }
    uint32_t inc = uint32_t(len);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= uint32_t(o)) inc += v;
    }
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    if (live) spell_line<RW>(buf, T.fill + inc - uint32_t(len), r, k);
    __syncwarp();
    T.flush(buf, total);
  }
  T.end(buf);
}

// ---- oversized bins: their records, one run per bin, in order by radix passes
// over the whole grid, 8 bits of the key each, least significant first, between the
// two record arrays (k_line_group has left the runs in the first).  A pass is
// one kernel: blocks take chunks in order from a ticket, rank their records per
// digit, and find the digits' places from the run's counts of them and a look-back over
// the chunks before theirs.  The time does not depend on how the keys are spread.
// 2M to 3M lines, k = 31, of which n share 12 chars, whole call: 0.56, 0.83, 1.18, 2.29 ms
// for n = 10k, 100k, 300k, 1M; with one block for each such bin 0.76, 3.4, 9.3, 30
// (the call without ordering: 0.35, 0.55, 0.84, 1.78).  A pass is 18 us at 300k
// records (the round trips of one chunk: few blocks have work).
constexpr uint32_t OV_THREADS = 256, OV_PER = 8, OV_CHUNK = OV_THREADS * OV_PER;
constexpr uint32_t OV_PASSES = 16;
constexpr int OV_PASS_SHIFT = 40;  // look-back words: the tag, the pass, the value (40 bits)

struct OverBins {
  const OverBin* bin;      // [n]
  uint32_t* item_start;    // [n + 1] first chunk of each
  // cleared before the first pass:
  uint32_t* ticket;        // [OV_PASSES]
  uint32_t* hist;          // [passes][n][256] digit counts
  unsigned long long* st;  // [chunks][256] look-back words
  uint32_t n;
};
// The key's bytes that order a run, least significant first: byte position in
// Rec::hi, or 64 and up in Rec::lo.
struct Digits {
  uint32_t n;
  uint32_t sh[OV_PASSES];
};
template <int RW>
__device__ __forceinline__ uint32_t digit_of(const Rec<RW>& r, uint32_t sh) {
  if constexpr (RW == 3) return uint32_t((sh & 64u ? r.lo : r.hi) >> (sh & 63u)) & 255u;
  else return uint32_t(r.hi >> sh) & 255u;
}

// First chunk of each run, and the runs' tiles.
__global__ void __launch_bounds__(1024) k_over_items(OverBins o, uint2* __restrict__ tile) {
  __shared__ uint32_t scan[33];
  constexpr uint32_t PER = OVER_MAX / 1024;
  if (blockIdx.x == 0) {
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
      const uint32_t i = threadIdx.x * PER + q;
      c[q] = i < o.n ? (o.bin[i].n + OV_CHUNK - 1) / OV_CHUNK : 0u;
      sum += c[q];
    }
    uint32_t tot, at = block_excl_scan(sum, scan, &tot);
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
      const uint32_t i = threadIdx.x * PER + q;
      if (i < o.n) o.item_start[i] = at;
      at += c[q];
    }
    if (threadIdx.x == 0) o.item_start[o.n] = tot;
  }
  for (uint32_t i = blockIdx.x; i < o.n; i += gridDim.x) {
    const OverBin B = o.bin[i];
    const uint32_t each = B.n / B.nt, more = B.n % B.nt;
    for (uint32_t j = threadIdx.x + 1u; j < B.nt; j += blockDim.x)  // (the first is written)
      tile[B.tile + j] = make_uint2(B.beg + j * each + min(j, more), TILE_RUN);
  }
}

// The run of chunk t (one warp calls): the last one that starts at or before it.
__device__ __forceinline__ uint32_t over_bin_of(const OverBins& o, uint32_t t) {
  uint32_t lo = 0, n = o.n;  // among [lo, lo + n)
  while (n > 1) {
    const uint32_t step = (n + 31u) / 32u, i = step * (threadIdx.x & 31u);
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, i < n && o.item_start[lo + i] <= t);
    const uint32_t j = step * (31u - uint32_t(__clz(m)));  // (lane 0 always agrees)
    lo += j;
    n = min(step, n - j);
  }
  return lo;
}

// All passes' digit counts of each run.
template <int RW>
__global__ void __launch_bounds__(OV_THREADS) k_over_count(RecArr<RW> in, OverBins o, Digits dg) {
  __shared__ uint32_t cnt[OV_PASSES / (4 - RW)][256], s_bin;  // (8 passes with one key word)
  const uint32_t tid = threadIdx.x, nitems = o.item_start[o.n];
  for (uint32_t t = blockIdx.x; t < nitems; t += gridDim.x) {
    if (tid < 32) {
      const uint32_t b = over_bin_of(o, t);
      if (tid == 0) s_bin = b;
    }
    for (uint32_t p = 0; p < dg.n; ++p) cnt[p][tid] = 0;
    __syncthreads();
    const uint32_t b = s_bin, c0 = (t - o.item_start[b]) * OV_CHUNK;
    const OverBin B = o.bin[b];
    const uint32_t cn = min(OV_CHUNK, B.n - c0);
    for (uint32_t i = tid; i < cn; i += OV_THREADS) {
      const Rec<RW> r = ld_rec<RW>(in, uint64_t(B.beg) + c0 + i);
      for (uint32_t p = 0; p < dg.n; ++p) atomicAdd(&cnt[p][digit_of<RW>(r, dg.sh[p])], 1u);
    }
    __syncthreads();
    for (uint32_t p = 0; p < dg.n; ++p)
      if (cnt[p][tid]) atomicAdd(o.hist + (uint64_t(p) * o.n + b) * 256u + tid, cnt[p][tid]);
    __syncthreads();
  }
}

template <int RW>
__global__ void __launch_bounds__(OV_THREADS) k_over_pass(RecArr<RW> in, RecArr<RW> to, OverBins o, uint32_t pass,
                                                          uint32_t sh, SortCtr* sc) {
  constexpr uint32_t W = OV_THREADS / 32;
  __shared__ uint32_t wcnt[W][256], place[256], scan[33], s_t, s_bin;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  const uint32_t nitems = o.item_start[o.n];
  const unsigned long long mark = static_cast<unsigned long long>(pass) << OV_PASS_SHIFT;
  for (;;) {
    if (tid < 32) {
      uint32_t t = 0;
      if (tid == 0) t = atomicAdd(o.ticket + pass, 1u);
      t = __shfl_sync(0xFFFFFFFFu, t, 0);
      const uint32_t b = over_bin_of(o, min(t, nitems - 1u));
      if (tid == 0) {
        s_t = t;
        s_bin = b;
      }
    }
#pragma unroll
    for (uint32_t w = 0; w < W; ++w) wcnt[w][tid] = 0;
    __syncthreads();
    const uint32_t t = s_t, b = s_bin;
    if (t >= nitems) break;
    const OverBin B = o.bin[b];
    const uint32_t chunk = t - o.item_start[b], c0 = chunk * OV_CHUNK, cn = min(OV_CHUNK, B.n - c0);
    // the warp's records, 32 at a time in order, each ranked among the warp's of
    // its digit
    Rec<RW> r[OV_PER];
    uint32_t rk[OV_PER];
    const uint32_t i0 = wid * (OV_CHUNK / W) + lane;
#pragma unroll
    for (uint32_t q = 0; q < OV_PER; ++q)
      if (i0 + 32 * q < cn) r[q] = ld_rec<RW>(in, uint64_t(B.beg) + c0 + i0 + 32 * q);
    const uint32_t count = o.hist[(uint64_t(pass) * o.n + b) * 256u + tid];
#pragma unroll
    for (uint32_t q = 0; q < OV_PER; ++q) {
      const bool live = i0 + 32 * q < cn;
      const uint32_t d = live ? digit_of<RW>(r[q], sh) : 256u;
      const uint32_t same = __match_any_sync(0xFFFFFFFFu, d), below = same & ((1u << lane) - 1u);
      const uint32_t before = live ? wcnt[wid][d] : 0u;
      __syncwarp();
      if (live && below == 0) wcnt[wid][d] = before + uint32_t(__popc(same));
      __syncwarp();
      rk[q] = (before + uint32_t(__popc(below))) | (d << 16);
    }
    __syncthreads();
    // thread d: digit d's records of the warps before each, and of the chunk
    uint32_t mine = 0;
#pragma unroll
    for (uint32_t w = 0; w < W; ++w) {
      const uint32_t c = wcnt[w][tid];
      wcnt[w][tid] = mine;
      mine += c;
    }
    unsigned long long* const word = o.st + uint64_t(t) * 256u + tid;
    atomicExch(word, (chunk ? LB_SUM : LB_PREFIX) | mark | mine);
    uint32_t tot, first = block_excl_scan(count, scan, &tot);
    if (chunk) {  // the chunks of the run before this one
      uint32_t before = 0;
      for (uint32_t j = 1; j <= chunk; ++j) {
        unsigned long long v = 0;
        bool there = false;
        for (uint32_t p = 0; p < LB_POLLS && !there; ++p) {
          v = *reinterpret_cast<volatile unsigned long long*>(word - uint64_t(j) * 256u);
          there = v > LB_VALUE && ((v & LB_VALUE) >> OV_PASS_SHIFT) == pass;
          if ((p & 1023u) == 1023u && *reinterpret_cast<volatile uint32_t*>(&sc->fail)) break;
        }
        if (!there) {
          atomicOr(&sc->fail, 1u);
          break;
        }
        before += uint32_t(v);
        if (v & LB_PREFIX) break;
      }
      atomicExch(word, LB_PREFIX | mark | (before + mine));
      first += before;
    }
    place[tid] = first;
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < OV_PER; ++q) {
      if (i0 + 32 * q >= cn) continue;
      const uint32_t d = rk[q] >> 16, pos = place[d] + wcnt[wid][d] + (rk[q] & 0xFFFFu);
      if (pos < B.n) st_rec<RW>(to, uint64_t(B.beg) + pos, r[q]);  // (a failed wait: nothing out of bounds)
    }
    __syncthreads();  // the shared arrays are reused
  }
}

// Stable order of n records of one tile too large for shared memory, by one
// block: 8 bits of the key per pass, least significant first, between two
// buffers.  Returns 1 where the result lies in y.  (A bin of more than a
// tile's records, up to OVER_WINS windows of them.)
template <int RW>
__device__ int order_in_memory(RecArr<RW> x, RecArr<RW> y, uint64_t beg, uint32_t n, int k, uint32_t* hist,
                               uint32_t* wcnt) {
  constexpr uint32_t W = TILE_THREADS / 32;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  __shared__ uint32_t sc[33];
  int in_y = 0;
  for (int pass = 0; pass < (RW == 3 ? 16 : 8); ++pass) {
    const bool low = RW == 3 && pass < 8;
    const int sh = 8 * (pass & 7);
    // bytes below the k-mer's last char hold nothing
    if (low ? (sh + 8 <= 128 - 2 * k) : (sh + 8 <= 64 - 2 * k)) continue;
    const RecArr<RW> a = in_y ? y : x, b = in_y ? x : y;
    auto digit = [&](const Rec<RW>& r) { return uint32_t((low ? r.lo : r.hi) >> sh) & 255u; };
    hist[tid] = 0;  // (TILE_THREADS = 256 digits)
    __syncthreads();
    for (uint32_t i = tid; i < n; i += TILE_THREADS) atomicAdd(hist + digit(ld_rec<RW>(a, beg + i)), 1u);
    __syncthreads();
    uint32_t tot;
    const uint32_t pre = block_excl_scan(hist[tid], sc, &tot);
    hist[tid] = pre;
    for (uint32_t i0 = 0; i0 < n; i0 += TILE_THREADS) {
      for (uint32_t q = tid; q < W * 256u; q += TILE_THREADS) wcnt[q] = 0;
      __syncthreads();
      const bool live = i0 + tid < n;
      Rec<RW> r{0ull, 0ull, 0ull};
      if (live) r = ld_rec<RW>(a, beg + i0 + tid);
      const uint32_t d = live ? digit(r) : 256u;
      const uint32_t same = __match_any_sync(0xFFFFFFFFu, d);
      const uint32_t rank = __popc(same & ((1u << lane) - 1u));
      if (live && rank == 0) wcnt[wid * 256u + d] = __popc(same);
      __syncthreads();
      uint32_t run = hist[tid];
      for (uint32_t w = 0; w < W; ++w) {
        const uint32_t c = wcnt[w * 256u + tid];
        wcnt[w * 256u + tid] = run;
        run += c;
      }
      hist[tid] = run;
      __syncthreads();
      if (live) st_rec<RW>(b, beg + wcnt[wid * 256u + d] + rank, r);
      __syncthreads();
    }
    in_y ^= 1;
  }
  return in_y;
}

template <int RW>
__host__ __device__ constexpr uint32_t tile_buf_words(int k) {
  // a warp's buffer: 15 bytes kept, 32 lines, word stores
  return (16u + 32u * ((uint32_t(k) + TAIL_MAX + 4u) & ~3u) + 16u) / 4u;
}
// Shared memory of a tile: the records; the sub-bins and the first index
// list, whose place the warps' buffers take; the final index list.
template <int RW>
__host__ __device__ constexpr size_t tile_area_words(int k) {
  const size_t a = TILE_SUB + 2 + tile_cap<RW>() / 2;
  const size_t b = size_t(TILE_THREADS / 32) * tile_buf_words<RW>(k);
  const size_t c = (TILE_THREADS / 32 + 1) * 256;  // order_in_memory
  return ((a > b ? (a > c ? a : c) : (b > c ? b : c)) + 3) & ~size_t(3);
}
template <int RW>
__host__ __device__ constexpr size_t tile_smem(int k) {
  return size_t(tile_cap<RW>()) * (8 * RW + 2) + tile_area_words<RW>(k) * 4;
}

// One block per tile.  The records' keys are spread over TILE_SUB sub-bins of
// the tile's key range (about one record each), counted and placed with
// shared-memory atomics, and each record's final rank is its sub-bin's start
// plus the smaller records in the sub-bin.  The tile's first byte comes from
// the look-back over the tiles' byte counts.  Then each warp stores a run of
// ranks (store_lines).  256 Mbp, k = 31: 3.0 ms for 5.3 GB, bound by shared memory
// (67% of L1 throughput) and issue (63%; about 650 instructions per line, spelling
// the most of them); 3.5 ms with three blocks per SM instead of four.
template <int RW>
__global__ void __launch_bounds__(TILE_THREADS, RW == 2 ? 4 : 3) k_line_tiles(RecArr<RW> rec, RecArr<RW> spare,
                                                             const uint2* __restrict__ tile, int bits, char* out, int k,
                                                             LongLine* longs, const char* keep,
                                                             unsigned long long* st, SortCtr* sc, int runs) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr uint32_t TILE_CAP = tile_cap<RW>();
  uint64_t* khi = reinterpret_cast<uint64_t*>(sm);
  uint64_t* klo = khi + TILE_CAP;                      // RW == 3
  uint64_t* tl = khi + size_t(TILE_CAP) * (RW - 1);
  uint32_t* area = reinterpret_cast<uint32_t*>(khi + size_t(TILE_CAP) * RW);
  uint32_t* sub = area;                                // [TILE_SUB + 1]
  uint16_t* ord = reinterpret_cast<uint16_t*>(area + TILE_SUB + 2);
  uint16_t* fin = reinterpret_cast<uint16_t*>(area + tile_area_words<RW>(k));
  __shared__ uint32_t scan[33], s_t;
  __shared__ unsigned long long s_sum[TILE_THREADS / 32], s_at, s_w[TILE_THREADS / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5;
  constexpr uint32_t W = TILE_THREADS / 32, PER = TILE_CAP / TILE_THREADS;
  if (sc->fail) return;  // (of the kernels before; uniform)
  // oversized bins have to be sorted first (runs: they are, 1 in rec, 2 in spare)
  if (!runs && sc->nover) return;
  const uint32_t ntiles = sc->ntiles;
  for (;;) {
    if (tid == 0) s_t = atomicAdd(&sc->tile_ticket, 1u);
    __syncthreads();
    const uint32_t t = s_t;
    if (t >= ntiles) break;
    const uint2 T0 = tile[t], T1 = tile[t + 1];
    const uint32_t beg = T0.x, n = T1.x - beg;
    const bool run = (T0.y & TILE_RUN) != 0;  // in order already (and fits)
    const bool fits = run || n <= TILE_CAP;
    // the tile's key range, spread over the sub-bins
    const uint64_t kmin = T0.y ? uint64_t(T0.y) << (64 - bits) : 0ull;
    const uint32_t nbins = (T1.y & ~TILE_RUN) - (T0.y & ~TILE_RUN);
    const int sh = max(0, 53 - bits + (nbins > 1u ? 32 - __clz(nbins - 1u) : 0));
    unsigned long long bytes = 0;
    uint32_t rk[PER];
    for (uint32_t j = tid; j < TILE_SUB; j += TILE_THREADS) sub[j] = 0;
    __syncthreads();
    if (run) {
      const RecArr<RW> src = runs == 2 ? spare : rec;
      for (uint32_t i = tid; i < n; i += TILE_THREADS) {
        const Rec<RW> r = ld_rec<RW>(src, uint64_t(beg) + i);
        khi[i] = r.hi;
        if constexpr (RW == 3) klo[i] = r.lo;
        tl[i] = r.tail;
        bytes += line_bytes_of(r.tail, k, longs);
        fin[i] = uint16_t(i);
      }
    } else if (fits) {
#pragma unroll
      for (uint32_t q = 0; q < PER; ++q) {
        if (q * TILE_THREADS >= n) break;
        const uint32_t i = q * TILE_THREADS + tid;
        if (i < n) {
          const Rec<RW> r = ld_rec<RW>(rec, uint64_t(beg) + i);
          khi[i] = r.hi;
          if constexpr (RW == 3) klo[i] = r.lo;
          tl[i] = r.tail;
          bytes += line_bytes_of(r.tail, k, longs);
          // the sub-bin and the record's place in it
          const uint32_t b = min(uint32_t((r.hi - kmin) >> sh), TILE_SUB - 1u);
          rk[q] = (atomicAdd(sub + b, 1u) << 11) | b;
        }
      }
    } else {
      for (uint32_t i = tid; i < n; i += TILE_THREADS)
        bytes += line_bytes_of(ld_rec<RW>(rec, uint64_t(beg) + i).tail, k, longs);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) bytes += __shfl_xor_sync(0xFFFFFFFFu, bytes, o);
    if (lane == 0) s_sum[wid] = bytes;
    __syncthreads();
    bytes = 0;
#pragma unroll
    for (uint32_t w = 0; w < W; ++w) bytes += s_sum[w];
    if (tid == 0) lb_publish(st, t, LB_SUM, bytes);
    int in_spare = 0;
    if (run) {
    } else if (fits) {
      {
        constexpr uint32_t C = TILE_SUB / TILE_THREADS;
        uint32_t c[C], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < C; ++q) {
          c[q] = sub[tid * C + q];
          sum += c[q];
        }
        uint32_t tot;
        uint32_t pre = block_excl_scan(sum, scan, &tot);
#pragma unroll
        for (uint32_t q = 0; q < C; ++q) {
          sub[tid * C + q] = pre;
          pre += c[q];
        }
        if (tid == 0) sub[TILE_SUB] = n;
      }
      __syncthreads();
#pragma unroll
      for (uint32_t q = 0; q < PER; ++q) {
        if (q * TILE_THREADS >= n) break;
        const uint32_t i = q * TILE_THREADS + tid;
        if (i < n) ord[sub[rk[q] & (TILE_SUB - 1u)] + (rk[q] >> 11)] = uint16_t(i);
      }
      __syncthreads();
      for (uint32_t j = tid; j < n; j += TILE_THREADS) {
        const uint32_t i = ord[j];
        const uint64_t h = khi[i];
        const uint32_t b = min(uint32_t((h - kmin) >> sh), TILE_SUB - 1u);
        const uint32_t lo = sub[b], hi = sub[b + 1];
        uint32_t rank = lo;
        for (uint32_t m = lo; m < hi; ++m) {
          const uint32_t o = ord[m];
          const uint64_t x = khi[o];
          bool less = x < h;
          if (x == h) {
            if constexpr (RW == 3) less = klo[o] < klo[i] || (klo[o] == klo[i] && o < i);
            else less = o < i;
          }
          rank += less ? 1u : 0u;
        }
        fin[rank] = uint16_t(i);
      }
    } else {
      in_spare = order_in_memory<RW>(rec, spare, beg, n, k, area, area + 256);
    }
    __syncthreads();
    const RecArr<RW> sorted = in_spare ? spare : rec;
    auto get = [&](uint32_t r) {
      if (!fits) return ld_rec<RW>(sorted, uint64_t(beg) + r);
      const uint32_t i = fin[r];
      Rec<RW> x;
      x.hi = khi[i];
      if constexpr (RW == 3) x.lo = klo[i];
      else x.lo = 0;
      x.tail = tl[i];
      return x;
    };
    // each warp's run of ranks and its bytes, and the tile's first byte
    const uint32_t per = ((n + W - 1) / W + 31u) & ~31u;
    const uint32_t r0 = min(n, wid * per), r1 = min(n, r0 + per);
    unsigned long long wb = 0;
    for (uint32_t r = r0 + lane; r < r1; r += 32)
      wb += line_bytes_of(fits ? tl[fin[r]] : get(r).tail, k, longs);
#pragma unroll
    for (int o = 16; o; o >>= 1) wb += __shfl_xor_sync(0xFFFFFFFFu, wb, o);
    if (lane == 0) s_w[wid] = wb;
    if (wid == 0) {
      const unsigned long long e = lb_exclusive(st, t, bytes, &sc->fail);
      if (lane == 0) s_at = e;
    }
    __syncthreads();
    unsigned long long at = s_at;
    for (uint32_t w = 0; w < wid; ++w) at += s_w[w];
    // (a failed wait leaves the text as it is)
    if (r0 < r1 && !*reinterpret_cast<volatile uint32_t*>(&sc->fail))
      store_lines<RW>(out, at, r0, r1, k, area + wid * tile_buf_words<RW>(k), longs, keep, get);
    __syncthreads();  // the tile's shared memory is reused
  }
}

// Lines of HUGE_LINE bytes or more, each by the whole grid: from the kept
// copy to the place k_line_tiles noted.
__global__ void __launch_bounds__(256) k_huge_lines(char* out, const char* keep, const LongLine* longs,
                                                    const uint32_t* huge, const SortCtr* sc) {
  const uint32_t nhuge = sc->nhuge;
  for (uint32_t h = 0; h < nhuge; ++h) {
    const LongLine L = longs[huge[h]];
    for (unsigned long long x = blockIdx.x * HUGE_LINE; x < L.len; x += gridDim.x * HUGE_LINE)
      copy_bytes(out + L.to + x, keep + L.kept + x, min(HUGE_LINE, L.len - x), threadIdx.x, blockDim.x);
  }
}

// The oversized bins' records in order: in a (runs = 1) or b (2) after it.
template <int RW>
int sort_over(Env& e, RecArr<RW> a, RecArr<RW> b, OverBins ov, const SortCtr& h, int k, int bits, uint2* tile,
              SortCtr* sc, int& runs) {
  ov.n = h.nover;
  const uint64_t nchunk = h.nrec / OV_CHUNK + h.nover;  // at most
  // the bytes that hold chars, but for those within the bins' own bits
  Digits dg{};
  for (int sh = 0; RW == 3 && sh < 64; sh += 8)
    if (sh + 8 > 128 - 2 * k) dg.sh[dg.n++] = uint32_t(64 + sh);
  for (int sh = 0; sh < 64 - bits; sh += 8)
    if (sh + 8 > 64 - 2 * k) dg.sh[dg.n++] = uint32_t(sh);
  runs = 1;
  int occ = 0;
  if (const int ro = occupancy(e, occ, k_over_pass<RW>, int(OV_THREADS), 0)) return ro;
  const unsigned g = unsigned(std::min<uint64_t>(nchunk, uint64_t(e.sm_count) * uint64_t(std::max(1, occ))));
  e.launches += 2 + dg.n;
  k_over_items<<<std::min(ov.n, unsigned(e.sm_count)), 1024, 0, e.stream>>>(ov, tile);
  // tickets, counts and look-back words lie in one piece
  ov.st = reinterpret_cast<unsigned long long*>(ov.hist + uint64_t(dg.n) * ov.n * 256);
  UC_CK(cudaMemsetAsync(ov.ticket, 0, size_t(reinterpret_cast<char*>(ov.st + nchunk * 256) -
                                             reinterpret_cast<char*>(ov.ticket)), e.stream));
  k_over_count<RW><<<g, OV_THREADS, 0, e.stream>>>(a, ov, dg);
  for (uint32_t i = 0; i < dg.n; ++i) {
    k_over_pass<RW><<<g, OV_THREADS, 0, e.stream>>>(a, b, ov, i, dg.sh[i], sc);
    std::swap(a, b);
    runs = 3 - runs;
  }
  UC_CK(cudaGetLastError());
  return UC_OK;
}

// The launch sequence for one key width: the lines of out[0, bytes) and
// those of pre.
template <int RW>
int sort_lines_rw(Env& e, char* out, uint64_t bytes, int k, const LineRecs& pre) {
  const uint64_t lmax = bytes / uint64_t(k + 1) + pre.n;  // lines at most
  const int bits = pre.bits;
  if (lmax > pre.cap) return e.fail(UC_EINTERNAL, "more lines than k-mers");
  const uint32_t m = 1u << bits;
  // shorter windows while there are fewer than two tiles per SM
  uint32_t win = WIN;
  while (win > 250 && lmax / win < 2ull * e.sm_count) win /= 2;
  const uint64_t ntmax = lmax / win + 2;
  const uint64_t nplan = (uint64_t(m) + 256 * PLAN_ITEMS - 1) / (256 * PLAN_ITEMS);
  // (fewer than OVER_MAX bins hold more than lmax / OVER_MAX lines each)
  const uint32_t big = uint32_t(std::max<uint64_t>(OVER_WINS * win, lmax / OVER_MAX));
  const uint64_t nover = lmax / big + 1, nchunk = lmax / OV_CHUNK + nover + 1;  // at most
  // a long line holds TAIL_MAX + 2 k-mers or more, and k bytes and one per k-mer
  const uint64_t nlongs = std::min(bytes / uint64_t(k + TAIL_MAX + 2), pre.kmers / (TAIL_MAX + 2)) + 1;
  const uint64_t kept = std::min(bytes, pre.kmers + nlongs * uint64_t(k)) + nlongs * 16;
  const uint64_t nhuges = bytes / HUGE_LINE + 1;
  // more tiles than k_line_group counts at once: groups of 2^gsh first
  uint32_t gsh = 0;
  if (ntmax > GRP_BINS)
    for (gsh = 5; (ntmax >> gsh) > GRP_BINS / 2; ) ++gsh;
  // cleared: the counters and the look-back words
  const size_t zero = 256 + (nplan + ntmax) * 8;
  const size_t ovb = OV_PASSES * 4 + (nover * OV_PASSES / (4 - RW) * 4 + nchunk * 8) * 256;
  // The job's arrays are used up but for the records and their counts, and the
  // scratch takes what lies around those in both arenas: sorted output fits where
  // the job does.  (The second records and tails take one of the scatter's regions;
  // the front arena's 16 or 24 bytes per k-mer hold the rest, 4 bytes per k-mer of
  // kept chars at most, 1.1 of their index, and 5 per line.)
  struct Room {
    uintptr_t at, end;
  };
  auto addr = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
  const uintptr_t mid = addr(pre.a) + pre.cap * 16;  // the tails (two key words)
  const uintptr_t last = RW == 3 ? mid + lmax * 8 : addr(pre.a) + lmax * 16;
  Room room[4] = {{addr(e.ar[1].base), addr(pre.a)},
                  {addr(pre.a) + lmax * 16, RW == 3 ? mid : 0},
                  {last, addr(e.ar[1].base) + e.ar[1].cap},
                  {addr(pre.counts) + (size_t(4) << bits), addr(e.ar[0].base) + e.ar[0].cap}};
  bool fits = true;
  auto take = [&](size_t b) -> char* {
    for (Room& r : room) {
      const uintptr_t at = (r.at + 255) & ~uintptr_t(255);
      if (at + b > r.end) continue;
      r.at = at + b;
      return reinterpret_cast<char*>(at);
    }
    fits = false;
    return nullptr;
  };
  char* recs = take(lmax * 16);
  char* tails = RW == 3 ? take(lmax * 8) : nullptr;
  char* keep = take(kept);
  char* z = take(zero);
  uint2* tile = reinterpret_cast<uint2*>(take((ntmax + 1) * 8));
  uint32_t* cur = reinterpret_cast<uint32_t*>(take((ntmax + GRP_BINS) * CUR_STRIDE * 4));
  uint32_t* gcur = reinterpret_cast<uint32_t*>(take(((ntmax >> gsh) + 1 + GRP_BINS) * CUR_STRIDE * 4));
  LongLine* longs = reinterpret_cast<LongLine*>(take(nlongs * sizeof(LongLine)));
  uint32_t* huge = reinterpret_cast<uint32_t*>(take(nhuges * 4));
  OverBin* over = reinterpret_cast<OverBin*>(take(nover * sizeof(OverBin)));
  OverBins ov{};
  ov.bin = over;
  ov.item_start = reinterpret_cast<uint32_t*>(take((nover + 1) * 4));
  ov.ticket = reinterpret_cast<uint32_t*>(take(ovb));
  ov.hist = ov.ticket + OV_PASSES;
  if (!fits) return e.fail(UC_EBUDGET, "scratch for sorted output");
  const RecArr<RW> ra{reinterpret_cast<ulonglong2*>(pre.a), reinterpret_cast<unsigned long long*>(mid)};
  const RecArr<RW> rb{reinterpret_cast<ulonglong2*>(recs), reinterpret_cast<unsigned long long*>(tails)};
  SortCtr* sc = reinterpret_cast<SortCtr*>(z);
  unsigned long long* st_plan = reinterpret_cast<unsigned long long*>(z + 256);
  unsigned long long* st_tile = st_plan + nplan;
  uint32_t* counts = pre.counts;
  UC_CK(cudaMemsetAsync(z, 0, zero, e.stream));
  if (pre.n) UC_CK(cudaMemcpyAsync(&sc->nrec, &e.ctr->rec_slots, 4, cudaMemcpyDeviceToDevice, e.stream));
  auto grid = [&](uint64_t want, int occ) {
    return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(want, uint64_t(e.sm_count) * uint64_t(std::max(1, occ)))));
  };
  const uint64_t nchunks = (bytes + 15 + LR_CHUNK - 1) / LR_CHUNK;
  const size_t sm_recs = (LR_CHUNK / (uint32_t(k) + 1u) + 2u) * 2u;
  const size_t sm_tile = tile_smem<RW>(k);
  int occ = 0;
  if (const int ro = occupancy(e, occ, k_line_recs<RW>, 256, sm_recs)) return ro;
  ++e.launches;
  if (bytes) ++e.launches;
  if (bytes) k_line_recs<RW><<<grid(nchunks, occ), 256, sm_recs, e.stream>>>(out, bytes, k, bits, ra, counts, longs, huge, sc);
  k_line_plan<<<unsigned(nplan), 256, 0, e.stream>>>(counts, m, win, big, over, tile, cur, gcur, gsh, st_plan, sc);
  if (nlongs > 1) {
    ++e.launches;
    k_line_keep<<<grid((nlongs + 7) / 8, 4), 256, 0, e.stream>>>(out, keep, longs, huge, sc);
  }
  int r = allow_max_smem(e, k_line_group<RW>);
  if (r) return r;
  RecArr<RW> from = ra, to = rb;
  for (uint32_t level = gsh ? 0u : 1u; level < 2; ++level) {
    ++e.launches;
    k_line_group<RW><<<grid((lmax + grp_chunk<RW>() - 1) / grp_chunk<RW>(), 2), GRP_THREADS, grp_smem<RW>(),
                       e.stream>>>(from, to, counts, bits, level ? 0u : gsh, level ? cur : gcur, sc);
    std::swap(from, to);
  }
  r = allow_max_smem(e, k_line_tiles<RW>);
  if (r) return r;
  if (const int ro = occupancy(e, occ, k_line_tiles<RW>, int(TILE_THREADS), sm_tile)) return ro;
  if (occ < 1) return e.fail(UC_EINTERNAL, "line tile kernel does not fit an SM");
  static_assert(sizeof(SortCtr) <= Env::HOST_IO, "the counters fit the pinned area");
  SortCtr& h = *reinterpret_cast<SortCtr*>(e.h_io());
  auto tiles = [&](int runs) -> int {
    ++e.launches;
    k_line_tiles<RW><<<grid(ntmax, occ), TILE_THREADS, sm_tile, e.stream>>>(from, to, tile, bits, out, k, longs, keep,
                                                                           st_tile, sc, runs);
    UC_CK(cudaGetLastError());
    UC_CK(cudaMemcpyAsync(&h, sc, sizeof h, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    return UC_OK;
  };
  r = tiles(0);
  if (r) return r;
  if (h.nover && !h.fail) {
    int runs = 1;
    r = sort_over<RW>(e, from, to, ov, h, k, bits, tile, sc, runs);
    if (!r) r = tiles(runs);
    if (r) return r;
  }
  if (h.fail & 1u) return e.fail(UC_ETIMEOUT, "a bounded device wait ran out (sorted output)");
  if (h.fail) return e.fail(UC_EINTERNAL, "a line of the output is shorter than k");
  if (h.nhuge) {
    ++e.launches;
    k_huge_lines<<<unsigned(e.sm_count) * 4u, 256, 0, e.stream>>>(out, keep, longs, huge, sc);
    UC_CK(cudaGetLastError());
    UC_CK(cudaStreamSynchronize(e.stream));
  }
  return UC_OK;
}

}  // namespace

int line_bin_bits(uint64_t lines, int k) {
  // about 32 records per bin at most: a tile then is a window and a fraction
  // of one, and a bin can be 32 times as dense before its tile outgrows
  // shared memory.  Counts of 23 bits stay in L2 (32 MiB).
  int bits = 4;
  while (bits < std::min(23, 2 * k) && (lines >> bits) > 32) ++bits;
  return bits;
}

int sort_lines(Env& e, char* out, uint64_t bytes, int k, const LineRecs& pre) {
  if (bytes == 0 && pre.n == 0) return UC_OK;
  const int r = k <= 31 ? sort_lines_rw<2>(e, out, bytes, k, pre) : sort_lines_rw<3>(e, out, bytes, k, pre);
  e.reset();
  return r;
}

}  // namespace uc
