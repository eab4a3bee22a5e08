// uc_kernels.cuh — kernel declarations and launch helpers shared by the
// pipeline (uc_pipeline.cu) and the C ABI (uc_capi.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "uc_common.cuh"

namespace uc {

// Device-side counters of one pipeline run (one allocation, zeroed per run).
// Atomics on words of one 128-byte line queue up in L2 (about 2 ns each), so
// the counters that every tile adds to have lines of their own: with all of
// them in one line, 1.24M warp tiles with four atomics each took 9.7 ms.
struct Counters {
  alignas(128) unsigned long long seg_char_cursor;
  // lines the tiles left as records (low half) and head-pool ids taken (high
  // half), in sorted output
  alignas(128) unsigned long long rec_slots;
  alignas(128) uint32_t wtile_next;
  alignas(128) unsigned long long rec_bytes;  // the records' lines
  unsigned long long cycles;
  unsigned long long copies;         // total of the bucket counts
  uint32_t cross_count;
  uint32_t ntiles;
  uint32_t tile_next;
  uint32_t nbig;
  uint32_t err;
  uint32_t work_mid, work_sub;       // work counters of scatter levels 2 and 3
  uint32_t nwarp, nblock;            // tiles per tier
  uint32_t walked, left;             // line walk: segments on lines written, lines left
};

// After the counters, cleared with them: the look-back words of the tile plan
// and of the bucket offsets, each behind its ticket (uc_lookback.cuh).
constexpr size_t PLAN_LB_WORDS = 512, SCAN_LB_WORDS = 8192 + 1;
constexpr size_t COUNTERS_BYTES = sizeof(Counters) + (PLAN_LB_WORDS + SCAN_LB_WORDS) * 8;

// A line as a record (sorted output): its k-mer big-endian (first char in the
// top bits of hi, chars 32.. in lo), so that numeric order is byte order, and a
// tail word: the chars after the k-mer as codes (first one lowest) under their
// count, or, with TAIL_LONG, the index of a line kept as text.  Two words (hi,
// tail) for k <= 31, three otherwise; the first two lie together.
constexpr int TAIL_MAX = 28;
constexpr uint64_t TAIL_LONG = 1ull << 63;
constexpr int TAIL_LEN_SHIFT = 58;
template <int RW>
struct Rec {
  uint64_t hi, lo, tail;
};
template <int RW>
struct RecArr {
  ulonglong2* a;
  unsigned long long* t;  // tails (RW == 3)
};
template <int RW>
__device__ __forceinline__ Rec<RW> ld_rec(const RecArr<RW>& r, uint64_t i) {
  const ulonglong2 v = r.a[i];
  if constexpr (RW == 2) return Rec<RW>{v.x, 0ull, v.y};
  else return Rec<RW>{v.x, v.y, r.t[i]};
}
template <int RW>
__device__ __forceinline__ void st_rec(const RecArr<RW>& r, uint64_t i, const Rec<RW>& x) {
  if constexpr (RW == 2) {
    r.a[i] = make_ulonglong2(x.hi, x.tail);
  } else {
    r.a[i] = make_ulonglong2(x.hi, x.lo);
    r.t[i] = x.tail;
  }
}

// One more record in each lane's bin (NONE: no record; whole warps call).  Lines
// that share their first chars come by the thousand, and atomics on one word take
// 0.27 ns per lane (1M lines in one bin: k_line_recs 270 us), so where two
// neighbours agree the warp's records of one bin are added together.  (Always
// looking for them cost k_tile_warp 88 of 6400 us at 256 Mbp.)
__device__ __forceinline__ void count_bin(uint32_t* counts, uint32_t bin) {
  uint32_t n = bin != NONE ? 1u : 0u;
  if (__any_sync(0xFFFFFFFFu, bin == __shfl_xor_sync(0xFFFFFFFFu, bin, 1) && n)) {
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, bin);
    n = n && (same & ((1u << (threadIdx.x & 31u)) - 1u)) == 0 ? uint32_t(__popc(same)) : 0u;
  }
  if (n) atomicAdd(counts + bin, n);
}

// Lines the tiles left as records: the records (rec_bytes bytes of lines) and a
// count per bin of the key's leading bits.  The records lie in the back arena, the
// counts at the start of the front arena (in the keys, which the scatter has
// read); nothing else of either arena is in use by then.
struct LineRecs {
  char* a = nullptr;
  uint64_t cap = 0;  // records that fit at a
  uint64_t kmers = 0;
  uint32_t* counts = nullptr;
  int bits = 0;
  uint32_t n = 0;
  uint64_t bytes = 0;
};

// One open segment of the fused path (written by the tile that finds it): the
// offset of its chars in the segment-char area (low 40 bits) and its job
// (high 24 bits), its copy count, and the cross index through which its line
// continues (NONE where the line ends).  A segment that starts a line keeps
// k - 1 + len chars there; the others keep the len - 1 chars they add (their
// first k-mer ends the segment before).  Segment ids: a segment that starts
// at the S-only copy of cross k-mer x has id x; a segment that starts a line
// (at a P-role copy) takes an id from its job's head pool, after all cross
// indices.
struct __align__(16) SegRec {
  unsigned long long off_job;
  uint32_t len;
  uint32_t next;
};
constexpr int SEG_OFF_BITS = 40;
constexpr unsigned long long SEG_OFF_MASK = (1ull << SEG_OFF_BITS) - 1ull;

// One job of a batch (a single call is a batch of one).  Its k-mers occupy
// keys[koff, koff + n); its buckets are (job << job_bits) | local; its lines
// go to out[obase, obase + ocap); the segments that start its stitched
// lines take head-pool ids [seg_base, seg_base + seg_cap) (after the cross
// indices).
struct JobTab {
  const uint8_t* text;
  unsigned long long tbytes, body, end, n, koff, lb0;  // lb0: first block of lines (k_pack)
  unsigned long long obase, ocap;
  uint32_t seg_base, seg_cap;
  uint32_t fixed;  // every line is k chars + '\n'
  uint32_t err;    // header/layout problems found on the device
};

struct TileParams {
  const uint64_t* pkeys;        // copies (NW words each, role bits in the last word)
  const uint32_t* plink;        // cross index (fused) or k-mer id (edges)
  const unsigned long long* tile_begin;  // [ntiles + 1] copy offsets
  Counters* ctr;
  const uint32_t* big_list;     // big-tile launch: tile ids
  const uint32_t* wlist;        // warp-tier tile ids
  const uint32_t* blist;        // block-tier tile ids
  uint32_t wcap, wts, wbytes;   // warp tiles: capacity, hash slots, shared bytes per warp
  const JobTab* jobs;
  const uint32_t* tile_job;     // job of each tile
  unsigned long long* jout;     // per-job closed-line cursor (bytes)
  uint32_t* jseg;               // per-job head-pool cursor
  char* big_scratch;
  const unsigned long long* big_off;
  int k;
  uint32_t cap;                 // shared-memory tile capacity (copies)
  uint32_t tslots;              // shared-memory hash slots (power of two >= 2*cap)
  uint32_t lf, wlf;             // hash slots per 100 copies of a block / warp tile (150..800)
  int mode;                     // 0 = edges by id, 1 = fused emission
  uint32_t* succ;
  uint32_t* pred;
  char* out;
  unsigned long long out_cap;
  char* segchars;
  unsigned long long segchars_cap;
  uint32_t seg_cap;
  SegRec* seg;                  // open segments by id
  uint32_t xcount;              // cross k-mers (the head pool starts there)
  // sorted output: closed lines of warp tiles leave as records (rec_a null:
  // all lines as text)
  ulonglong2* rec_a;
  unsigned long long* rec_t;
  uint32_t* rec_counts;
  int rec_bits;
};

// Shared memory of one tile: keys plus four 16-bit arrays per copy (sized
// in fours), and 16-bit hash slots.
__host__ __device__ inline size_t tile_bytes(int nw, uint32_t cap, uint32_t tslots) {
  return size_t(cap) * 8u * nw + size_t((cap + 3u) & ~3u) * 8u + size_t(tslots) * 2u;
}

// Smallest power of two >= x, for x <= 2^31 (callers bound x first); larger
// x returns 2^31 after at most 31 doublings.
__host__ __device__ inline uint32_t pow2_at_least(uint64_t x) {
  uint32_t p = 1;
  for (int i = 0; i < 31 && p < x; ++i) p <<= 1;
  return p;
}

// Carved table of a tile of c copies: the hash slots, and at least 2c
// entries because the table doubles as rank scratch after hashing.
__host__ __device__ inline uint32_t big_slots(uint64_t c, uint32_t lf) {
  const uint64_t want = c * lf / 100;
  return pow2_at_least(want > 2 * c ? want : 2 * c);
}

}  // namespace uc
