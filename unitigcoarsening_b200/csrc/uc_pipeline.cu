// uc_pipeline.cu — CUDA kernels of the unitig compactor and the host code
// that sequences them.
//
// Data flow of the fused path (all device resident; a batch of jobs shares
// every launch):
//   text --k_pack (fused minimizers)--> keys[n], (b1,b2)[n], bucket counts
//   --k_bucket_offsets, k_scatter_coarse/mid/sub--> copies in bucket order
//   --k_tile_plan--> tiles of whole buckets --k_tile_warp / k_tile /
//   k_tile_big (persistent; a warp, a CTA, or global scratch per tile)-->
//   finished lines + open segments (one record per segment id: its chars,
//   length and continuation)
//   --stitch (k_walk_emit: each line from its head; list ranking,
//   k_chain_len, k_seg_copy for what the walk leaves)--> cross-tile lines.
// The phase-by-phase entry points (pack, minimizers, find_edges, contract,
// emit) run the same kernels separately.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/uc.h"
#include "uc_kernels.cuh"
#include "uc_lookback.cuh"
#include "uc_pipeline.h"

#include <cuda_pipeline.h>

namespace uc {

// ===================================================================== scan

// Exclusive prefix sums of the bucket (or count group) counts, and their
// total, in one look-back pass: 4096 counts per block.
constexpr uint32_t SCAN_TILE = 4096;
__global__ void __launch_bounds__(256) k_bucket_offsets(const uint32_t* __restrict__ in, uint64_t n,
                                                        unsigned long long* __restrict__ out, unsigned long long* lb,
                                                        uint32_t* err, unsigned long long* total) {
  __shared__ unsigned long long scan[33], s_base;
  __shared__ uint32_t s_b;
  if (threadIdx.x == 0) s_b = atomicAdd(reinterpret_cast<uint32_t*>(lb), 1u);
  __syncthreads();
  const uint32_t b = s_b;
  const uint64_t i0 = uint64_t(b) * SCAN_TILE + 16u * threadIdx.x;
  uint32_t c[16];
  unsigned long long sum = 0;
#pragma unroll
  for (int v = 0; v < 4; ++v) {  // (the counts start 256-byte aligned)
    uint4 x = make_uint4(0u, 0u, 0u, 0u);
    if (i0 + 4 * v + 4 <= n) {
      x = reinterpret_cast<const uint4*>(in + i0)[v];
    } else {
      if (i0 + 4 * v < n) x.x = in[i0 + 4 * v];
      if (i0 + 4 * v + 1 < n) x.y = in[i0 + 4 * v + 1];
      if (i0 + 4 * v + 2 < n) x.z = in[i0 + 4 * v + 2];
    }
    c[4 * v] = x.x;
    c[4 * v + 1] = x.y;
    c[4 * v + 2] = x.z;
    c[4 * v + 3] = x.w;
    sum += uint64_t(x.x) + x.y + x.z + x.w;
  }
  unsigned long long tot;
  const unsigned long long pre = block_excl_scan(sum, scan, &tot);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) lb_publish(lb + 1, b, LB_SUM, tot);
    __syncwarp();
    const unsigned long long e = lb_exclusive(lb + 1, b, tot, err, ERR_TIMEOUT);
    if (threadIdx.x == 0) s_base = e;
  }
  __syncthreads();
  unsigned long long p = s_base + pre;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    if (i0 + q < n) out[i0 + q] = p;
    p += c[q];
  }
  if (b == gridDim.x - 1 && threadIdx.x == 0) out[n] = *total = s_base + tot;
}

// ===================================================================== pack

__device__ __forceinline__ uint32_t base_code(uint32_t c) {
  // char_map of compact_kmers (driver.cpp:228-232): A=0 C=1 G=2 T=3, else 0
  return (c == 'C') ? 1u : (c == 'G') ? 2u : (c == 'T') ? 3u : 0u;
}

// A block packs 512 consecutive lines per pass.  Their text comes in by
// asynchronous copies while the pass before is packed; each 16 bytes become
// one word of 2-bit codes in shared memory, and a thread's line is then a few
// funnel shifts of code words.
//
// Lines of k chars and a break (k >= 15): a 16-byte piece holds at most one
// line break, at a place that follows from its offset, so it is checked by
// spelling its codes again and comparing, with the break expected at its
// place.  A pass where every piece agrees needs no other check.
//
// Any other pass (another layout, the count line's and the last piece, a
// byte that is not ACGT) keeps, per piece, a bit per line break and a bit per
// byte that is neither ACGT nor a break, and checks each line's bits; a byte
// that is not ACGT packs as A (the zeroed char_map of compact_kmers,
// driver.cpp:228-232), so its code is cleared.
//
// With FUSE the prefix/suffix minimizer buckets of every key are computed and
// counted in the same pass (lmin_buckets.h:299-318).
//
// Bound by the ALU pipe (half rate: 76% at 30 Mbp, k = 31).  256 Mbp, k = 31:
// 3.6 ms (8.2 GB of text); 6.3 ms when each thread converted its own line
// from staged text, 3.8 ms with bits per byte for every piece.
constexpr int PACK_LINES = 512;
constexpr int PACK_SPAN = 36864;  // text bytes staged per pass at most (wider lines: byte by byte)

// 16-byte pieces a pass stages: those of its lines at fixed width, or
// PACK_SPAN where the lines' starts are given.  Even, as two share a mask word.
static uint32_t pack_pieces(bool fixed, int k) {
  const uint32_t bytes = fixed ? uint32_t(PACK_LINES) * uint32_t(k + 1) + 16u : uint32_t(PACK_SPAN);
  return ((std::min<uint32_t>(bytes, PACK_SPAN) + 31u) / 32u) * 2u;
}
// raw text, codes, two masks (a line's last words reach past the pieces)
static size_t pack_smem(uint32_t pieces) { return size_t(pieces) * 16 + (size_t(pieces) + 8) * 8; }

// Bit i to bit 2i.
__device__ __forceinline__ uint64_t even_bits(uint32_t x) {
  uint64_t y = x;
  y = (y | (y << 16)) & 0x0000FFFF0000FFFFull;
  y = (y | (y << 8)) & 0x00FF00FF00FF00FFull;
  y = (y | (y << 4)) & 0x0F0F0F0F0F0F0F0Full;
  y = (y | (y << 2)) & 0x3333333333333333ull;
  return (y | (y << 1)) & 0x5555555555555555ull;
}

// The piece v of 16 text bytes: codes (of bytes that are ACGT), possible line
// breaks (nl: a break where the code is 1, which is checked per line) and
// other bytes (bad), a bit per byte.  Bits 1 and 2 of a letter are free, the
// others follow from them (T has bit 2 without bit 1, bit 4 and no bit 0); a
// byte with bit 3 set has to agree with 0x0A in the others.
__device__ __forceinline__ uint32_t text_piece(const uint4& v, uint32_t& nl, uint32_t& bad) {
  const uint32_t x[4] = {v.x, v.y, v.z, v.w};
  uint32_t f[4], d[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    f[q] = (x[q] >> 3) & 0x01010101u;
    const uint32_t t = (x[q] >> 2) & ~(x[q] >> 1) & 0x01010101u;
    const uint32_t want = 0x41414141u + t * 0x0Fu - f[q] * 0x39u;  // (no byte borrows: 0x41 or 0x50, less 0x39)
    d[q] = (x[q] & 0xF9F9F9F9u) ^ want;
  }
  nl = __byte_perm(f[0] * 0x01020408u + f[1] * 0x10204080u, f[2] * 0x01020408u + f[3] * 0x10204080u, 0x4473) & 0xFFFFu;
  bad = 0;
  if (d[0] | d[1] | d[2] | d[3]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t z = (((d[q] & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | d[q]) & 0x80808080u;  // bytes that differ
      bad |= (((z >> 7) * 0x01020408u) >> 24) << (4 * q);
    }
    nl &= ~bad;
  }
  return codes16(v);
}

__device__ __forceinline__ uint32_t job_of_block(const JobTab* __restrict__ jobs, uint32_t njobs, uint64_t g) {
  uint32_t lo = 0, hi = njobs;  // last job with lb0 <= g
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (jobs[mid].lb0 <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Bucket counts while packing.  The resident path counts copies per group
// of 2^cshift buckets in 32-bit words, at most 2^20 of them (4 MiB, so the
// count reductions stay in L2 at 2^25 buckets); level 3 of the scatter counts
// the buckets of each group itself.  The streamed path (cshift = CNT16)
// counts every bucket in a 16-bit half of a 32-bit word (64 MiB at 2^25
// buckets); a half that wraps shows up as a low total, and the counts are
// then taken again at 32 bits (k_count_buckets).  k_widen16 turns them into
// 32-bit counts.
constexpr uint32_t CNT16 = 32;
constexpr uint32_t COUNT_GROUPS_BITS = 20;
__device__ __forceinline__ void count16(uint32_t* c16, uint32_t b) {
  // a reduction (no value returned, so no wait): a count that wraps its 16
  // bits carries into its neighbour or out of the word, which shows up on
  // the host as a total below the copies the pack counted (k-mers plus cross
  // k-mers), and the counts are then taken again at 32 bits
  atomicAdd(c16 + (b >> 1), 1u << ((b & 1u) * 16u));
}
__global__ void k_widen16(const uint32_t* __restrict__ c16, uint64_t M, uint32_t* __restrict__ counts) {
  for (uint64_t b = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; b < M; b += uint64_t(gridDim.x) * blockDim.x)
    counts[b] = (c16[b >> 1] >> ((b & 1u) * 16u)) & 0xFFFFu;
}

__global__ void k_count_buckets(const uint32_t* __restrict__ b1, const uint32_t* __restrict__ b2, uint64_t n,
                                uint32_t* __restrict__ counts) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t a = b1[i], b = b2[i];
    atomicAdd(counts + a, 1u);
    if (a != b) atomicAdd(counts + b, 1u);
  }
}

// What regular_piece expects of a piece whose line break is byte p (none for
// p >= 16).
struct Break16 {
  uint32_t e[4];  // per word, the break's difference from the letter its bits read as
  uint32_t lo, at;  // the break's two bits as read, and their place
};
__device__ __forceinline__ Break16 break_at(uint32_t p) {
  Break16 x;
  const uint32_t d = uint32_t('C' ^ '\n') << (8 * (p & 3u));
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) x.e[q] = (p >> 2) == q ? d : 0u;
  x.lo = p < 16u ? 1u << (2 * (p & 15u)) : 0u;
  x.at = 3u * x.lo;
  return x;
}
// The codes of the 16 text bytes v where they are letters, but for a line
// break where x says; bad becomes nonzero where they are not.  (The letters
// that bits 1 and 2 of each byte read as are compared with the bytes; the
// break reads as C, and no other byte that does differs from C as it does.)
__device__ __forceinline__ uint32_t regular_piece(const uint4& v, const Break16& x, uint32_t& bad) {
  const uint32_t r = letter_bits16(v);
  uint32_t w[4];
  spread16(0x47544341u, r, w);  // A C T G
  bad |= (w[0] ^ v.x ^ x.e[0]) | (w[1] ^ v.y ^ x.e[1]);
  bad |= (w[2] ^ v.z ^ x.e[2]) | (w[3] ^ v.w ^ x.e[3]);
  bad |= (r ^ x.lo) & x.at;
  return codes_of_bits(r);
}

// Prefix and suffix minimizer buckets of a packed key in the fused path.  An
// l-mer's id is its 2l bits of the key as they lie (first char lowest), so
// each costs a funnel shift by a constant, a multiply-add and a min, with no
// reversal of the key: chars right of the l-mer are in the id's upper bits and
// drop out of the product (lmins, with (id * m + a) << (32 - 2l) as there).
// The priority order is free (find_edges and uc_minimizers use lmins' order).
template <int NW, int KC>
__device__ __forceinline__ void key_buckets(const Key<NW>& key, int k, int l, uint64_t seed, uint32_t bits, uint32_t& b1,
                                            uint32_t& b2) {
  const uint32_t ps = 32u - 2u * uint32_t(l);
  const uint32_t m = lmer_mult(seed) << ps, a = static_cast<uint32_t>(seed >> 32) << ps;
  uint32_t x[2 * NW + 1];
#pragma unroll
  for (int q = 0; q < 2 * NW; ++q) x[q] = uint32_t(key.w[q >> 1] >> (32 * (q & 1)));
  x[2 * NW] = 0;
  const int last = k - l;  // l-mers 0 .. last
  uint32_t mid = 0xFFFFFFFFu;
  auto pri = [&](int p) { return __funnelshift_r(x[p >> 4], x[(p >> 4) + 1], 2 * (p & 15)) * m + a; };
#pragma unroll
  for (int p = 1; p < 32 * NW - 2; p += 2) {  // 1 .. last - 1 (l <= 16: KC - 17 of them at least)
    if ((KC == 0 || p >= KC - 16) && p >= last) break;
    const uint32_t u = pri(p), v = pri(p + 1);
    mid = __vimin3_u32(mid, u, ((KC == 0 || p + 1 >= KC - 16) && p + 1 >= last) ? u : v);
  }
  const int s = 2 * last;
  uint32_t e;
  if constexpr (NW == 1) e = uint32_t(key.w[0] >> s);
  else e = s >= 64 ? uint32_t(key.w[NW - 1] >> (s - 64)) : uint32_t((key.w[0] >> s) | (s ? key.w[NW - 1] << (64 - s) : 0ull));
  b1 = bucket_of(min(mid, x[0] * m + a) >> ps, bits);
  b2 = bucket_of(min(mid, e * m + a) >> ps, bits);
}

// MULTI: the block's job comes from the job table (batches); otherwise the
// one job is a kernel parameter, read from the constant bank.
// KC: k fixed at compile time (0: taken from the argument).
template <int NW, bool FUSE, bool MULTI, int KC = 0>
__global__ void __launch_bounds__(256, NW == 1 && KC ? 6 : 5) k_pack(const JobTab* __restrict__ jobs, const JobTab one, uint32_t njobs,
                                              uint64_t nblocks,
                                              const unsigned long long* __restrict__ starts, int k_arg,
                                              uint64_t* __restrict__ keys, uint32_t* err, int l, uint64_t seed,
                                              uint32_t jb, uint32_t* __restrict__ b1, uint32_t* __restrict__ b2,
                                              uint32_t* __restrict__ counts, uint32_t cshift,
                                              uint32_t* __restrict__ jcross, uint32_t pcap) {
  extern __shared__ __align__(16) unsigned char sm_pack[];
  uint4* raw = reinterpret_cast<uint4*>(sm_pack);                        // [pcap] text of the next pass
  uint32_t* code = reinterpret_cast<uint32_t*>(raw + pcap);              // [pcap + 8]
  uint32_t* nlw = code + pcap + 8;                                       // [(pcap + 8) / 2]
  uint32_t* badw = nlw + (pcap + 8) / 2;                                 // [(pcap + 8) / 2]
  uint16_t* nl16 = reinterpret_cast<uint16_t*>(nlw);
  uint16_t* bad16 = reinterpret_cast<uint16_t*>(badw);
  __shared__ uint32_t s_cross;
  const int k = KC ? KC : k_arg;
  uint32_t bad = 0, mycross = 0;
  const uint32_t stride = uint32_t(k) + 1;
  const uint64_t kmask_hi = (1ull << (2 * k - 64 * (NW - 1))) - 1ull;  // (at most 62 bits)
  // a bit per char of a line, and the place of the break after it (k <= 31 or 63)
  using Mask = typename std::conditional<NW == 1, uint32_t, uint64_t>::type;
  const Mask term = Mask(1) << k, chars = term - 1;
  // one pass: its lines and their text
  struct Pass {
    const uint8_t* text;
    uint64_t end, b0, s0, span, koff;
    uint32_t j, cnt, first, nterm;
  };
  // The pass's text on its way into raw (each thread its own pieces, which it
  // converts itself: no barrier between the copy and the conversion).
  auto fetch = [&](uint64_t g) {
    Pass P;
    P.j = MULTI ? job_of_block(jobs, njobs, g) : 0u;
    P.text = MULTI ? jobs[P.j].text : one.text;
    const uint64_t tbytes = MULTI ? jobs[P.j].tbytes : one.tbytes;
    const uint64_t body = MULTI ? jobs[P.j].body : one.body;
    P.end = MULTI ? jobs[P.j].end : one.end;
    const uint64_t n = MULTI ? jobs[P.j].n : one.n;
    P.koff = MULTI ? jobs[P.j].koff : one.koff;
    P.b0 = (g - (MULTI ? jobs[P.j].lb0 : one.lb0)) * PACK_LINES;
    const uintptr_t tb = reinterpret_cast<uintptr_t>(P.text);
    P.cnt = uint32_t((n - P.b0) < PACK_LINES ? (n - P.b0) : PACK_LINES);
    P.s0 = starts ? uint64_t(starts[P.b0]) : body + P.b0 * stride;
    const bool more = P.b0 + P.cnt < n;
    const uint64_t s1 = more ? (starts ? uint64_t(starts[P.b0 + P.cnt]) : body + (P.b0 + P.cnt) * stride) : P.end;
    P.first = uint32_t((tb + P.s0) & 15u);  // first line's start in the staged span
    P.span = s1 - P.s0 + P.first;
    P.nterm = starts ? 0u : (more ? P.cnt : P.cnt - 1u);  // lines whose break is checked
    if (P.span <= uint64_t(pcap) * 16) {
      const uintptr_t A0 = tb + P.s0 - P.first;
      const uint32_t nch = uint32_t(P.span + 15) / 16;
      const bool inside = A0 >= tb && A0 + 16u * nch <= tb + tbytes;
      uint32_t c = threadIdx.x;
      if (inside) {
        const uint4* src = reinterpret_cast<const uint4*>(A0);
        for (; c + 768 < nch; c += 1024) {
#pragma unroll
          for (int q = 0; q < 4; ++q) __pipeline_memcpy_async(raw + c + 256 * q, src + c + 256 * q, 16);
        }
      }
      for (; c < nch; c += 256) {
        const uintptr_t a = A0 + 16u * c;
        if (inside || (a >= tb && a + 16 <= tb + tbytes)) {
          __pipeline_memcpy_async(raw + c, reinterpret_cast<const void*>(a), 16);
        } else {
          for (int b = 0; b < 16; ++b) {
            const uintptr_t x = a + b;
            reinterpret_cast<uint8_t*>(raw + c)[b] =
                (x >= tb && x < tb + tbytes) ? *reinterpret_cast<const uint8_t*>(x) : uint8_t('\n');
          }
        }
      }
    }
    __pipeline_commit();
    return P;
  };
  if (blockIdx.x >= nblocks) return;
  Pass next = fetch(blockIdx.x);
  for (uint64_t g = blockIdx.x; g < nblocks; g += gridDim.x) {
    const Pass P = next;
    const uint64_t end = P.end, b0 = P.b0, s0 = P.s0;
    const uint8_t* text = P.text;
    const uint32_t cnt = P.cnt, j = P.j;
    const bool staged = P.span <= uint64_t(pcap) * 16;
    uint64_t* kout = keys + (P.koff + b0) * NW;
    uint32_t* o1 = FUSE ? b1 + P.koff + b0 : nullptr;
    uint32_t* o2 = FUSE ? b2 + P.koff + b0 : nullptr;
    if (MULTI && threadIdx.x == 0) s_cross = 0;
    __pipeline_wait_prior(0);
    const uint32_t nch = uint32_t(P.span + 15) / 16;
    bool regular = staged && !starts && stride >= 16;
    if (regular) {
      uint32_t odd = 0, c = threadIdx.x;
      // the piece's offset from a line's start, in [0, stride)
      uint32_t r = (16u * threadIdx.x + stride - P.first % stride) % stride;
      Break16 x = break_at(uint32_t(k) - r);
      auto step = [&] {
        if constexpr (KC == 0 || 4096 % (KC + 1) != 0) {
          r += 4096u % stride;
          r -= r >= stride ? stride : 0u;
          x = break_at(uint32_t(k) - r);
        }
      };
      for (; c + 768 < nch; c += 1024) {
        uint4 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = raw[c + 256 * q];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          code[c + 256 * q] = regular_piece(v[q], x, odd);
          step();
        }
      }
      for (; c < nch; c += 256) {
        code[c] = regular_piece(raw[c], x, odd);
        step();
      }
      regular = !__syncthreads_or(odd != 0);
    }
    if (!regular) {
      if (staged) {
        for (uint32_t c = threadIdx.x; c < nch; c += 256) {
          uint32_t nl, bd;
          code[c] = text_piece(raw[c], nl, bd);
          nl16[c] = uint16_t(nl);
          bad16[c] = uint16_t(bd);
        }
      }
      __syncthreads();
    }
    if (g + gridDim.x < nblocks) next = fetch(g + gridDim.x);
    for (uint32_t t = threadIdx.x; t < cnt; t += 256) {
      Key<NW> key;
      bool lbad = false;
      const bool check_term = t < P.nterm;
      if (regular) {
        const uint32_t off = P.first + t * stride, wi = off >> 4, sh = 2u * (off & 15u);
        uint32_t c[2 * NW + 1];
#pragma unroll
        for (int w = 0; w <= 2 * NW; ++w) c[w] = code[wi + w];
#pragma unroll
        for (int w = 0; w < NW; ++w)
          key.w[w] = __funnelshift_r(c[2 * w], c[2 * w + 1], sh) |
                     (uint64_t(__funnelshift_r(c[2 * w + 1], c[2 * w + 2], sh)) << 32);
        key.w[NW - 1] &= kmask_hi;
      } else if (staged) {
        // (a line past the staged ones is an error: it reads the first line's place)
        uint32_t off = P.first + (starts ? uint32_t(uint64_t(starts[b0 + t]) - s0) : t * stride);
        lbad = off + uint32_t(k) > uint32_t(P.span);
        if (lbad) off = 0;
        const uint32_t wi = off >> 4, sh = 2u * (off & 15u), mi = off >> 5, ms = off & 31u;
        uint32_t c[2 * NW + 1];
#pragma unroll
        for (int w = 0; w <= 2 * NW; ++w) c[w] = code[wi + w];
#pragma unroll
        for (int w = 0; w < NW; ++w)
          key.w[w] = __funnelshift_r(c[2 * w], c[2 * w + 1], sh) |
                     (uint64_t(__funnelshift_r(c[2 * w + 1], c[2 * w + 2], sh)) << 32);
        // possible line breaks and other bytes among the k chars, and the
        // break after them
        Mask nm = __funnelshift_r(nlw[mi], nlw[mi + 1], ms), bm = __funnelshift_r(badw[mi], badw[mi + 1], ms);
        if constexpr (NW == 2) {
          nm |= uint64_t(__funnelshift_r(nlw[mi + 1], nlw[mi + 2], ms)) << 32;
          bm |= uint64_t(__funnelshift_r(badw[mi + 1], badw[mi + 2], ms)) << 32;
        }
        const uint32_t after = uint32_t((NW == 1 || k < 32) ? key.w[0] >> (2 * k) : key.w[NW - 1] >> (2 * k - 64)) & 3u;
        lbad |= check_term && (!(nm & term) || after != 1u);
        key.w[NW - 1] &= kmask_hi;
        if ((nm | bm) & chars) {
#pragma unroll
          for (int w = 0; w < NW; ++w) {
            const uint64_t nl = even_bits(uint32_t((nm & chars) >> (w ? 32 : 0)));
            const uint64_t any = even_bits(uint32_t(((nm | bm) & chars) >> (w ? 32 : 0)));
            if (nl & key.w[w] & ~(key.w[w] >> 1)) lbad = true;  // a line break
            key.w[w] &= ~(3ull * any);
          }
        }
      } else {
#pragma unroll
        for (int w = 0; w < NW; ++w) key.w[w] = 0;
        const uint64_t s = starts ? uint64_t(starts[b0 + t]) : s0 + uint64_t(t) * stride;
        for (int c = 0; c <= k; ++c) {
          const uint64_t pos = s + c;
          const uint32_t ch = (pos < end) ? uint32_t(__ldg(text + pos)) : uint32_t('\n');
          if (c < k) {
            lbad |= (ch == '\n') || (pos >= end);
            const uint64_t cd = base_code(ch);
            if (c < 32) key.w[0] |= cd << (2 * c);
            else key.w[NW - 1] |= cd << (2 * (c - 32));
          } else if (check_term && ch != '\n') {
            lbad = true;
          }
        }
      }
      if (lbad) bad = 1;
      // keys and bucket ids stream out with evict-first stores, so that the
      // text and them do not push the bucket counts out of L2
      if constexpr (NW == 1) __stcs(reinterpret_cast<unsigned long long*>(kout) + t,
                                    static_cast<unsigned long long>(key.w[0]));
      else st_key<NW>(kout, t, key);
      if constexpr (FUSE) {
        uint32_t a, b;
        key_buckets<NW, KC>(key, k, l, seed, jb, a, b);
        if (MULTI) {
          a |= j << jb;
          b |= j << jb;
        }
        __stcs(o1 + t, a);
        __stcs(o2 + t, b);
        if (counts) {  // (the streamed path's second pass only needs the buckets)
          if (cshift == CNT16) {
            count16(counts, a);
            if (a != b) count16(counts, b);
          } else {
            // one 32-bit count per group of 2^cshift buckets (a reduction)
            atomicAdd(counts + (a >> cshift), 1u);
            if (a != b) atomicAdd(counts + (b >> cshift), 1u);
          }
          mycross += (a != b) ? 1u : 0u;
        }
      }
    }
    if (FUSE && MULTI) {  // (one job: counted over all passes)
      mycross = __reduce_add_sync(0xFFFFFFFFu, mycross);
      if ((threadIdx.x & 31) == 0 && mycross) atomicAdd(&s_cross, mycross);
      mycross = 0;
    }
    __syncthreads();
    if (FUSE && MULTI && threadIdx.x == 0 && s_cross && jcross) atomicAdd(jcross + j, s_cross);
  }
  if (FUSE && !MULTI) {
    mycross = __reduce_add_sync(0xFFFFFFFFu, mycross);
    if ((threadIdx.x & 31) == 0 && mycross && jcross) atomicAdd(jcross, mycross);
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(err, starts ? ERR_LINE : ERR_LAYOUT);
}

// Header and end of every job's text (batches of more than one job): the
// count line, the first k-mer line, the end of the last line, and whether
// every line is k chars + '\n'.  One thread per job.
__global__ void k_headers(JobTab* __restrict__ jobs, uint32_t njobs, int k) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= njobs) return;
  JobTab J = jobs[j];
  const uint8_t* t = J.text;
  const uint64_t bytes = J.tbytes;
  uint64_t p = 0;
  while (p < bytes && (t[p] == ' ' || t[p] == '\t' || t[p] == '\r')) ++p;
  uint32_t e = 0;
  uint64_t v = 0;
  if (p >= bytes || t[p] < '0' || t[p] > '9') e = 1;
  while (!e && p < bytes && t[p] >= '0' && t[p] <= '9') {
    v = v * 10 + uint64_t(t[p] - '0');
    if (v > 0x7FFFFFFEull) e = 1;
    ++p;
  }
  while (p < bytes && t[p] != '\n') ++p;
  const uint64_t body = (p < bytes) ? p + 1 : bytes;
  uint64_t end = bytes;
  while (end > body && (t[end - 1] == '\n' || t[end - 1] == '\r')) --end;
  J.n = e ? 0 : v;
  J.body = body;
  J.end = end;
  J.err = e;
  const uint64_t stride = uint64_t(k) + 1;
  J.fixed = (!e && ((J.n == 0 && end == body) || (J.n > 0 && end - body == J.n * stride - 1))) ? 1u : 0u;
  jobs[j] = J;
}

// Line starts for the general layout: starts[0] = body, and one past each
// line break in [body, end), at most nlines of them; *total gets the breaks.
// One pass: a block reads a chunk with 16-byte loads into a bit per line break
// in shared memory, a thread takes two words of bits, and the chunk's first
// line comes from the look-back over the chunks' counts.  (130 MB of k = 21
// text with a count column: 56 us; a byte-wise count and a byte-wise
// write pass took 1280.)
constexpr uint32_t INDEX_CHUNK = 16384;
__global__ void __launch_bounds__(256) k_line_index(const uint8_t* __restrict__ text, uint64_t body, uint64_t end,
                                                    uint64_t nlines, unsigned long long* __restrict__ starts,
                                                    unsigned long long* st, uint32_t* ticket, uint32_t* fail,
                                                    unsigned long long* total) {
  __shared__ __align__(16) uint32_t nlw[INDEX_CHUNK / 32];
  __shared__ uint32_t scan[33], s_c;
  __shared__ unsigned long long s_base;
  uint16_t* nl16 = reinterpret_cast<uint16_t*>(nlw);
  if (threadIdx.x == 0) s_c = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t chunk = s_c;
  // positions are relative to the 16-byte boundary at or below the text
  const uint8_t* A = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(text) & ~uintptr_t(15));
  const uint64_t off = uint64_t(text - A), lo = off + body, hi = off + end;
  const uint64_t c0 = (lo & ~uint64_t(15)) + uint64_t(chunk) * INDEX_CHUNK;
  uint4 v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint64_t x = c0 + 16u * (256u * q + threadIdx.x);
    v[q] = make_uint4(0u, 0u, 0u, 0u);
    if (x >= lo && x + 16 <= hi) v[q] = *reinterpret_cast<const uint4*>(A + x);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t p = 256u * q + threadIdx.x;
    const uint64_t x = c0 + 16u * p;
    uint32_t m = 0;
    if (x >= lo && x + 16 <= hi) {
      const uint32_t w[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t z = w[i] ^ 0x0A0A0A0Au;
        const uint32_t eq = ~(((z & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | z) & 0x80808080u;  // 0x80 per line break
        m |= (((eq >> 7) * 0x01020408u) >> 24) << (4 * i);
      }
    } else if (x + 16 > lo && x < hi) {  // a piece at an end of the lines
      for (int i = 0; i < 16; ++i)
        if (x + i >= lo && x + i < hi && A[x + i] == '\n') m |= 1u << i;
    }
    nl16[p] = uint16_t(m);
  }
  __syncthreads();
  const uint32_t b0 = nlw[2 * threadIdx.x], b1 = nlw[2 * threadIdx.x + 1];
  uint32_t tot;
  const uint32_t pre = block_excl_scan(uint32_t(__popc(b0) + __popc(b1)), scan, &tot);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) lb_publish(st, chunk, LB_SUM, tot);
    __syncwarp();
    const unsigned long long e = lb_exclusive(st, chunk, tot, fail);
    if (threadIdx.x == 0) s_base = e;
  }
  __syncthreads();
  uint64_t r = s_base + pre;
  const uint64_t x0 = c0 + 64u * threadIdx.x - off + 1;  // one past bit 0, from the text's first byte
#pragma unroll
  for (int q = 0; q < 2; ++q)
    for (uint32_t b = q ? b1 : b0; b; b &= b - 1)
      if (++r < nlines) starts[r] = x0 + 32 * q + uint32_t(__ffs(b) - 1);
  if (chunk == 0 && threadIdx.x == 0) starts[0] = body;
  if (chunk == gridDim.x - 1 && threadIdx.x == 0) *total = s_base + tot;
}

// ============================================================== minimizers

template <int NW>
__global__ void k_lmin(const uint64_t* __restrict__ keys, uint64_t n, int k, int l, uint64_t seed,
                       const uint32_t* __restrict__ table, uint32_t* __restrict__ l1,
                       uint32_t* __restrict__ l2) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t a, b;
    lmins<NW>(ld_key<NW>(keys, i), k, l, seed, table, a, b);
    l1[i] = a;
    l2[i] = b;
  }
}

// Minimizers -> prefix bucket b1 and suffix bucket b2, counted per bucket
// (find_l_minimizer "calc lmins" + "count lmins", lmin_buckets.h:299-318).
template <int NW>
__global__ void __launch_bounds__(256) k_lmin_count(const uint64_t* __restrict__ keys, uint64_t n,
                                                    int k, int l, uint64_t seed, uint32_t bbits,
                                                    uint32_t* __restrict__ b1, uint32_t* __restrict__ b2,
                                                    uint32_t* __restrict__ counts) {
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += uint64_t(gridDim.x) * blockDim.x) {
    uint32_t a, b;
    lmins<NW>(ld_key<NW>(keys, i), k, l, seed, nullptr, a, b);
    a = bucket_of(a, bbits);
    b = bucket_of(b, bbits);
    b1[i] = a;
    b2[i] = b;
    atomicAdd(counts + a, 1u);
    if (a != b) atomicAdd(counts + b, 1u);
  }
}

// ============================================================ tile planning

// One tile's tier by its size: warp tiles and block tiles up to wcap and cap
// copies, larger ones with the global scratch they need.
struct Tiers {
  uint32_t wcap, cap, lf;
  int nw;
  uint32_t *wlist, *blist, *big_list;
  unsigned long long* big_size;
};
__device__ __forceinline__ void list_larger_tile(const Tiers& T, Counters* ctr, uint32_t t, uint64_t c) {
  // (a tile's line bytes must fit 32-bit offsets: c * 64 < 2^32)
  if (c > (1ull << 26)) {
    atomicOr(&ctr->err, ERR_INTERNAL);
  } else if (c <= T.cap) {
    T.blist[atomicAdd(&ctr->nblock, 1u)] = t;
  } else {
    const uint32_t i = atomicAdd(&ctr->nbig, 1u);
    T.big_list[i] = t;
    const uint64_t ts = big_slots(c, T.lf);
    T.big_size[i] = (c * 8ull * T.nw + ((c + 3ull) & ~3ull) * 16ull + ts * 4ull + 255ull) & ~255ull;
  }
}

// Tiles pack consecutive whole buckets, next fit: each thread walks a run of
// `runlen` buckets (a multiple of 16) and starts a new tile at the run's
// first bucket, at a job's first bucket, and wherever the next bucket would
// take the tile past `cap` copies.  A tile of several buckets therefore
// holds at most `cap` copies; a bucket larger than `cap` sits alone.  Counts
// move 16 at a time (the array starts 256-byte aligned).  A first walk counts
// the run's tiles and warp tiles, a look-back numbers them, a second walk
// writes them and, with lists, sorts them into tiers: one kernel for what took
// six (flags, three for a scan, writing, classification).
__global__ void __launch_bounds__(256) k_tile_plan(const uint32_t* __restrict__ counts,
                                                   const unsigned long long* __restrict__ off, uint32_t m,
                                                   uint32_t cap, uint32_t jb, uint32_t runlen,
                                                   unsigned long long* __restrict__ tile_begin,
                                                   uint32_t* __restrict__ tile_job, Tiers T, int lists,
                                                   unsigned long long* lb, Counters* ctr) {
  __shared__ unsigned long long scan[33], s_base;
  __shared__ uint32_t s_b;
  if (threadIdx.x == 0) s_b = atomicAdd(reinterpret_cast<uint32_t*>(lb), 1u);
  __syncthreads();
  const uint32_t r = s_b * 256u + threadIdx.x, nruns = (m + runlen - 1) / runlen;
  const uint32_t b0 = r < nruns ? r * runlen : m, b1 = min(m, b0 + min(runlen, m - b0));
  // open(bucket): a tile starts there; close(copies): the tile before it ends
  auto walk = [&](auto open, auto close) {
    uint32_t run = 0;
    for (uint32_t c0 = b0; c0 < b1; c0 += 16) {
      uint32_t c[16];
      if (c0 + 16 <= b1) {
        const uint4* src = reinterpret_cast<const uint4*>(counts + c0);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 x = src[v];
          c[4 * v] = x.x;
          c[4 * v + 1] = x.y;
          c[4 * v + 2] = x.z;
          c[4 * v + 3] = x.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < 16; ++q) c[q] = (c0 + q < b1) ? counts[c0 + q] : 0u;
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const uint32_t b = c0 + uint32_t(q);
        if (b >= b1) break;
        if (b == b0 || ((b >> jb) != ((b - 1) >> jb)) || run + c[q] > cap) {
          if (b > b0) close(run);
          open(b);
          run = c[q];
        } else {
          run += c[q];
        }
      }
    }
    if (b1 > b0) close(run);
  };
  uint32_t nt = 0, nwt = 0;
  walk([&](uint32_t) { ++nt; }, [&](uint32_t c) { nwt += (c && c <= T.wcap) ? 1u : 0u; });
  // (62 bits travel: tiles and warp tiles are both below 2^31)
  unsigned long long tot;
  const unsigned long long pre = block_excl_scan((static_cast<unsigned long long>(nwt) << 31) | nt, scan, &tot);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) lb_publish(lb + 1, s_b, LB_SUM, tot);
    __syncwarp();
    const unsigned long long e = lb_exclusive(lb + 1, s_b, tot, &ctr->err, ERR_TIMEOUT);
    if (threadIdx.x == 0) s_base = e;
  }
  __syncthreads();
  if (b0 >= b1) return;
  uint32_t t = uint32_t((s_base + pre) & 0x7FFFFFFFull), w = uint32_t((s_base + pre) >> 31);
  unsigned long long o = off[b0];
  walk(
      [&](uint32_t b) {
        tile_begin[t] = o;
        tile_job[t] = b >> jb;
      },
      [&](uint32_t c) {
        if (lists && c) {
          if (c <= T.wcap) T.wlist[w++] = t;
          else list_larger_tile(T, ctr, t, c);
        }
        o += c;
        ++t;
      });
  if (b1 == m) {
    tile_begin[t] = o;
    ctr->ntiles = t;
    if (lists) ctr->nwarp = w;
  }
}

// The tiles [t0, t1) into tiers (the streamed path's groups; the resident
// path's tiers come with the plan).
__global__ void k_classify(const unsigned long long* __restrict__ tile_begin, Counters* ctr, Tiers T, uint32_t t0,
                           uint32_t t1) {
  const uint32_t nt = min(ctr->ntiles, t1);
  for (uint32_t t = t0 + blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
    const uint64_t c = tile_begin[t + 1] - tile_begin[t];
    if (c == 0) continue;
    if (c <= T.wcap) T.wlist[atomicAdd(&ctr->nwarp, 1u)] = t;
    else list_larger_tile(T, ctr, t, c);
  }
}

// ================================================================= scatter

// Every k-mer goes to its prefix bucket (role P) and, when its suffix
// minimizer lands in another bucket, a second copy goes to that bucket (role
// S) ("partition by lmins" + "write kmers", lmin_buckets.h:357-407).  The two
// copies of a cross k-mer share one cross index; in edges mode every copy
// carries the k-mer's id instead.
//
// Three levels keep the write frontier inside L2 and the global atomics few.
// Level 1 groups each block's copies by coarse partition (high bucket bits,
// at most 256 partitions) in shared memory and writes them out as contiguous
// runs, one reservation per block and partition.  A coarse partition
// occupies exactly the final positions of its buckets, so level 1 writes
// (key, link, bucket) records into the same index range of a staging
// region.  Level 2 groups each partition's records the same way by
// sub-partition (2^sb buckets), into the same index ranges of a second
// region; all blocks take chunks in partition order.  Level 3 gives each
// sub-partition to one block, which places the records inside its range with
// shared-memory cursors per bucket.
// k-mers per level-1 block pass (at most twice as many copies): large chunks
// spread the per-chunk reservations and barriers over more copies; 3072
// 64-bit keys (100 KB of staging, 2 CTAs per SM) beat 2048 (3 CTAs per SM)
// by 6% at 1 Gbp, and 128-bit keys keep 2048 (98 KB)
template <int NW>
__host__ __device__ constexpr int sc_chunk() {
  return NW == 1 ? 3072 : 2048;
}
static_assert(2 * sc_chunk<1>() < 65536 && 2 * sc_chunk<2>() < 65536, "chunk copy counts share a 32-bit scan");

// Staged records (key, link, bucket), packed: one 16-byte record with a one-word
// key; with a two-word key, link and bucket as one word behind the keys.
// Levels 1 and 2 are bound by the runs that they write more than by their
// bytes (13 to 16 records each, starting and ending inside a sector in every
// array), and packed there are a third or half as many.  260M k-mers, k = 31,
// 289M copies: levels 1, 2, 3 took 2.82, 2.17, 2.12 ms with arrays of their own
// for key, link and bucket, and 2.40, 1.96, 2.00 now; k = 63, 66M copies:
// 0.90, 0.85, 0.58 and 0.84, 0.72, 0.55.  (Level 2's staging in shared memory
// keeps three arrays for one-word keys: 16-byte records there cost it 0.3 ms.)
template <int NW, bool PACKED>
struct Stage {
  uint64_t* k = nullptr;
  uint32_t *l = nullptr, *b = nullptr;  // (packed: l is the second array of a two-word key's)
  // over n records at base, 256-byte aligned (scatter_stage_bytes)
  __host__ __device__ static Stage over(void* base, uint64_t n) {
    Stage s;
    s.k = static_cast<uint64_t*>(base);
    s.l = reinterpret_cast<uint32_t*>(s.k + NW * n);
    s.b = s.l + n;
    return s;
  }
  __device__ __forceinline__ void get(uint64_t i, Key<NW>& key, uint32_t& link, uint32_t& bkt) const {
    if constexpr (PACKED) {
      unsigned long long w;
      if constexpr (NW == 1) {  // (two loads: one of 16 bytes was 0.15 ms slower in level 2)
        key.w[0] = k[2 * i];
        w = k[2 * i + 1];
      } else {
        key = ld_key<NW>(k, i);
        w = reinterpret_cast<const unsigned long long*>(l)[i];
      }
      link = uint32_t(w);
      bkt = uint32_t(w >> 32);
    } else {
      bkt = b[i];
      key = ld_key<NW>(k, i);
      link = l[i];
    }
  }
  __device__ __forceinline__ void put(uint64_t i, const Key<NW>& key, uint32_t link, uint32_t bkt) const {
    if constexpr (PACKED) {
      const unsigned long long w = (static_cast<unsigned long long>(bkt) << 32) | link;
      if constexpr (NW == 1) {
        reinterpret_cast<ulonglong2*>(k)[i] = make_ulonglong2(key.w[0], w);
      } else {
        st_key<NW>(k, i, key);
        reinterpret_cast<unsigned long long*>(l)[i] = w;
      }
    } else {
      st_key<NW>(k, i, key);
      l[i] = link;
      b[i] = bkt;
    }
  }
  __device__ __forceinline__ uint32_t bucket(uint64_t i) const {
    static_assert(PACKED, "read from global memory only");
    if constexpr (NW == 1) return uint32_t(k[2 * i + 1] >> 32);
    else return uint32_t(reinterpret_cast<const unsigned long long*>(l)[i] >> 32);
  }
};

__global__ void k_coarse_init(const unsigned long long* __restrict__ boff, uint32_t fb, uint32_t mc,
                              unsigned long long* __restrict__ ccur) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < mc; j += gridDim.x * blockDim.x)
    ccur[j] = boff[uint64_t(j) << fb];
}

constexpr int COARSE_THREADS = 512;

template <int NW>
__global__ void __launch_bounds__(COARSE_THREADS, 2) k_scatter_coarse(const uint64_t* __restrict__ keys,
                                                        const uint32_t* __restrict__ b1,
                                                        const uint32_t* __restrict__ b2, uint64_t n,
                                                        uint32_t fb, uint32_t mc,
                                                        unsigned long long* __restrict__ ccur,
                                                        Stage<NW, true> to, int ids_mode, Counters* ctr) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  constexpr int SC_CHUNK = sc_chunk<NW>();
  const auto own = Stage<NW, true>::over(sm_raw, 2 * SC_CHUNK);
  unsigned long long* gbase = reinterpret_cast<unsigned long long*>(sm_raw + 2 * SC_CHUNK * (8 * NW + 8));  // [mc]
  uint32_t* hist = reinterpret_cast<uint32_t*>(gbase + mc);                     // [mc]
  uint32_t* lofs = hist + mc;                                                   // [mc + 1]
  __shared__ uint32_t sc[33];
  // A chunk's loads are all issued at once, for the first chunk here and for
  // every later one before its predecessor is written out, so that they are
  // in flight meanwhile; the values stay in registers.  A copy's rank within its
  // partition is what the count returns: no second atomic to place it.
  constexpr int PT = SC_CHUNK / COARSE_THREADS;
  Key<NW> kk[PT];
  uint32_t aa[PT], bb[PT];
  auto load = [&](uint64_t at) {
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const uint64_t i = at + uint32_t(q) * COARSE_THREADS + threadIdx.x;
      const uint64_t j = i < n ? i : 0;  // (a load behind a branch is waited for at once)
      kk[q] = ld_key<NW>(keys, j);
      aa[q] = b1[j];
      bb[q] = b2[j];
    }
  };
  const uint64_t stride = uint64_t(gridDim.x) * SC_CHUNK;
  uint64_t c0 = uint64_t(blockIdx.x) * SC_CHUNK;
  load(c0);
  for (; c0 < n; c0 += stride) {
    const uint32_t cn = uint32_t((n - c0) < uint64_t(SC_CHUNK) ? (n - c0) : uint64_t(SC_CHUNK));
    for (uint32_t j = threadIdx.x; j < mc; j += blockDim.x) hist[j] = 0;
    __syncthreads();
    // count copies per coarse partition; bit q of cmask marks a cross k-mer
    uint32_t cmask = 0;
    uint32_t rr[PT];  // ranks: of the first copy in the low half, of the second in the high half
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const uint32_t t = uint32_t(q) * COARSE_THREADS + threadIdx.x;
      rr[q] = 0;
      if (t < cn) {
        rr[q] = atomicAdd(hist + (aa[q] >> fb), 1u);
        if (aa[q] != bb[q]) {
          rr[q] |= atomicAdd(hist + (bb[q] >> fb), 1u) << 16;
          cmask |= 1u << q;
        }
      }
    }
    __syncthreads();
    // local offsets (scan over the partitions), this thread's first cross
    // index within the chunk, and global reservations.  One scan carries both
    // sums: the copy count in the low half (<= 2 * chunk < 2^16) and the
    // cross count in the high half (<= chunk).  The chunk's cross indices are reserved with a
    // single atomic: a counter shared by every block of the grid serialises
    // in L2, so one reservation per warp and k-mer slot would bound the kernel.
    uint32_t xpre;
    {
      const uint32_t per = (mc + blockDim.x - 1) / blockDim.x;
      const uint32_t j0 = min(mc, threadIdx.x * per), j1 = min(mc, j0 + per);
      uint32_t acc = 0;
      for (uint32_t j = j0; j < j1; ++j) acc += hist[j];
      uint32_t tot;
      const uint32_t both = block_excl_scan(acc | (uint32_t(__popc(cmask)) << 16), sc, &tot);
      uint32_t pre = both & 0xFFFFu;
      xpre = both >> 16;
      for (uint32_t j = j0; j < j1; ++j) {
        const uint32_t h = hist[j];
        lofs[j] = pre;
        // (less the run's place in the staging area: staged position + gbase)
        gbase[j] = (h ? atomicAdd(ccur + j, (unsigned long long)h) : 0ull) - pre;
        pre += h;
      }
      if (threadIdx.x == 0) {
        lofs[mc] = tot & 0xFFFFu;
        const uint32_t xt = tot >> 16;
        sc[32] = (!ids_mode && xt) ? atomicAdd(&ctr->cross_count, xt) : 0u;
      }
    }
    __syncthreads();
    xpre += sc[32];
    // place every copy in its partition's run of the staging area
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const uint32_t t = uint32_t(q) * COARSE_THREADS + threadIdx.x;
      const bool live = t < cn;
      uint32_t a = 0, b = 0;
      Key<NW> key;
#pragma unroll
      for (int w = 0; w < NW; ++w) key.w[w] = 0;
      if (live) {
        key = kk[q];
        a = aa[q];
        b = bb[q];
      }
      const bool cross = (cmask >> q) & 1u;
      const uint32_t x = (!ids_mode && cross) ? xpre + __popc(cmask & ((1u << q) - 1u)) : NONE;
      if (live) {
        const uint32_t link = ids_mode ? uint32_t(c0 + t) : x;
        Key<NW> kp = key;
        kp.w[NW - 1] |= ROLE_P | (cross ? 0ull : ROLE_S);
        const uint32_t sp = lofs[a >> fb] + (rr[q] & 0xFFFFu);
        own.put(sp, kp, link, a);
        if (cross) {
          Key<NW> ks = key;
          ks.w[NW - 1] |= ROLE_S;
          const uint32_t sq = lofs[b >> fb] + (rr[q] >> 16);
          own.put(sq, ks, link, b);
        }
      }
    }
    __syncthreads();
    // write the runs out: consecutive slots of a partition are consecutive
    // global positions
    const uint32_t total = lofs[mc];
    load(c0 + stride);
    for (uint32_t sl = threadIdx.x; sl < total; sl += blockDim.x) {
      Key<NW> key;
      uint32_t link, bk;
      own.get(sl, key, link, bk);
      to.put(gbase[bk >> fb] + sl, key, link, bk);
    }
    __syncthreads();
  }
}

// Level 2: within each coarse partition the staged records are grouped again
// by sub-partition (2^sb consecutive buckets, a few thousand copies), the way
// level 1 groups by partition: a block takes a chunk of one partition's
// staged records, counts them per sub-partition in shared memory, reserves
// one run per sub-partition (one global atomic per run, a few records each
// instead of one per record) and writes its records out as contiguous runs.
// Chunks never span partitions (their list comes from k_mid_items), so the
// counts index one partition's sub-partitions.  All blocks take chunks in
// partition order and reserve at the same cursors, so the runs of the
// chunks in flight stay next to each other: the write frontier is one
// partition's cursors and stays inside L2.  (Reserving for ranges of
// several chunks per block instead gives every block its own frontier:
// 1024 partly written runs per block, more than L2 holds at 1 Gbp.)
constexpr int MID_CHUNK = 4096;    // staged records per level-2 chunk
constexpr int MID_MAX_BINS = 1024; // sub-partitions per coarse partition
static_assert(MID_CHUNK <= 4096 && MID_MAX_BINS <= 4096, "a record's rank and bucket share a word");
constexpr int SUB_MAX_BITS = 9;    // buckets per sub-partition: at most 2^9
constexpr int MID_THREADS = 512;

// Chunk list of level 2: item_start[p] = first chunk of coarse partition p
// (partition p holds the staged records [boff[p << fb], boff[(p+1) << fb])).
__global__ void k_mid_items(const unsigned long long* __restrict__ boff, uint32_t fb, uint32_t mc,
                            uint32_t* __restrict__ item_start) {
  __shared__ uint32_t sc[33];
  const uint32_t p = threadIdx.x;
  uint32_t items = 0;
  if (p < mc) {
    const unsigned long long lo = boff[uint64_t(p) << fb], hi = boff[uint64_t(p + 1) << fb];
    items = uint32_t((hi - lo + MID_CHUNK - 1) / MID_CHUNK);
  }
  uint32_t tot;
  const uint32_t pre = block_excl_scan(items, sc, &tot);
  if (p < mc) item_start[p] = pre;
  if (p == 0) item_start[mc] = tot;
}

template <int NW>
__global__ void __launch_bounds__(MID_THREADS, NW == 1 ? 2 : 1) k_scatter_mid(
    Stage<NW, true> from, const unsigned long long* __restrict__ goff, uint32_t cg, const uint32_t* __restrict__ item_start, uint32_t fb,
    uint32_t sb, uint32_t mc, unsigned long long* __restrict__ scur, Stage<NW, true> to, Counters* ctr) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  const auto own = Stage<NW, NW == 2>::over(sm_raw, MID_CHUNK);
  unsigned long long* gbase = reinterpret_cast<unsigned long long*>(sm_raw + MID_CHUNK * (8 * NW + 8));  // [nb]
  const uint32_t nb = 1u << (fb - sb);
  uint32_t* hist = reinterpret_cast<uint32_t*>(gbase + nb);                          // [nb]
  uint32_t* lofs = hist + nb;                                                        // [nb + 1]
  uint32_t* istart = lofs + nb + 1;                                                  // [mc + 1]
  __shared__ uint32_t sc[33];
  // the next chunk, looked up by thread 0 while the block works on this one:
  // its first record, records and partition (no records: none left)
  __shared__ unsigned long long s_c0;
  __shared__ uint32_t s_cn, s_p;
  for (uint32_t j = threadIdx.x; j <= mc; j += blockDim.x) istart[j] = item_start[j];
  __syncthreads();
  const uint32_t nitems = istart[mc];
  constexpr int PT = MID_CHUNK / MID_THREADS;
  // the bins this thread scans and reserves
  const uint32_t per = (nb + blockDim.x - 1) / blockDim.x;
  const uint32_t j0 = min(nb, threadIdx.x * per), j1 = min(nb, j0 + per);
  // (goff: offsets of count groups of 2^cg buckets; partition p starts at
  // group p << (fb - cg))
  auto item = [&](uint32_t t, unsigned long long& at, unsigned long long& end, uint32_t& part) {
    at = end = 0;
    part = 0;
    if (t >= nitems) return;
    uint32_t lo = 0, hi = mc;  // the partition p with istart[p] <= t < istart[p + 1]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (istart[mid] <= t) lo = mid;
      else hi = mid;
    }
    part = lo;
    at = goff[uint64_t(lo) << (fb - cg)] + uint64_t(t - istart[lo]) * MID_CHUNK;
    end = goff[uint64_t(lo + 1) << (fb - cg)];
  };
  auto put = [&](unsigned long long at, unsigned long long end, uint32_t part) {
    s_c0 = at;
    s_cn = uint32_t(min(end - at, (unsigned long long)MID_CHUNK));
    s_p = part;
  };
  // a chunk's records, all loads issued at once, the first chunk's here and
  // every later one's before its predecessor is written out
  uint32_t bb[PT], ll[PT];
  Key<NW> kk[PT];
  unsigned long long c0;
  uint32_t cn, p;
  auto load = [&] {
    c0 = s_c0;
    cn = s_cn;
    p = s_p;
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const uint32_t i = uint32_t(q) * MID_THREADS + threadIdx.x;
      if (i < cn) from.get(c0 + i, kk[q], ll[q], bb[q]);
    }
  };
  uint32_t ticket = 0;  // thread 0: the chunk after the one in s_c0
  if (threadIdx.x == 0) {
    unsigned long long at, end;
    uint32_t part;
    const uint32_t t = atomicAdd(&ctr->work_mid, 1u);
    ticket = atomicAdd(&ctr->work_mid, 1u);
    item(t, at, end, part);
    put(at, end, part);
  }
  __syncthreads();
  load();
  while (cn) {
    const uint32_t sub0 = p << (fb - sb);  // first sub-partition of partition p
    for (uint32_t j = threadIdx.x; j < nb; j += blockDim.x) hist[j] = 0;
    __syncthreads();
    unsigned long long nat = 0, nend = 0;
    uint32_t npart = 0;
    if (threadIdx.x == 0) {
      item(ticket, nat, nend, npart);
      ticket = atomicAdd(&ctr->work_mid, 1u);
    }
    // The counts per sub-partition; a record keeps its rank there (12 bits)
    // above its bucket within the partition (fb <= 19 bits).  A record outside
    // partition p would be a broken staging order: flag it and leave it out
    // rather than index past the counts.
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const uint32_t i = uint32_t(q) * MID_THREADS + threadIdx.x;
      if (i < cn) {
        const uint32_t lb = bb[q] - (p << fb), bin = lb >> sb;
        if (bin < nb) {
          bb[q] = lb | (atomicAdd(hist + bin, 1u) << 20);
        } else {
          bb[q] = NONE;
          atomicOr(&ctr->err, ERR_INTERNAL);
        }
      }
    }
    __syncthreads();
    // local offsets and one reservation per non-empty sub-partition
    {
      uint32_t acc = 0;
      for (uint32_t j = j0; j < j1; ++j) acc += hist[j];
      uint32_t tot;
      uint32_t pre = block_excl_scan(acc, sc, &tot);
      for (uint32_t j = j0; j < j1; ++j) {
        const uint32_t h = hist[j];
        lofs[j] = pre;
        gbase[j] = (h ? atomicAdd(scur + sub0 + j, (unsigned long long)h) : 0ull) - pre;
        pre += h;
      }
      if (threadIdx.x == 0) {
        lofs[nb] = tot;
        put(nat, nend, npart);
      }
    }
    __syncthreads();
    // place every record in its sub-partition's run of the staging area
#pragma unroll
    for (int q = 0; q < PT; ++q) {
      const uint32_t i = uint32_t(q) * MID_THREADS + threadIdx.x;
      if (i < cn && bb[q] != NONE) {
        const uint32_t lb = bb[q] & 0xFFFFFu;
        const uint32_t sl = lofs[lb >> sb] + (bb[q] >> 20);
        own.put(sl, kk[q], ll[q], lb);
      }
    }
    __syncthreads();
    const uint32_t placed = lofs[nb], b0 = p << fb;
    load();
    for (uint32_t sl = threadIdx.x; sl < placed; sl += blockDim.x) {
      Key<NW> key;
      uint32_t link, lb;
      own.get(sl, key, link, lb);
      to.put(gbase[lb >> sb] + sl, key, link, b0 + lb);
    }
    __syncthreads();
  }
}

// Level 3: one block owns a sub-partition (2^sb buckets, whole count
// groups of the pack).  With count groups (cout given) it counts its
// records per bucket in shared memory, takes the buckets' offsets from a
// block scan and writes every bucket's count (and offset, to bout) for the
// tile plan; otherwise goff holds every bucket's offset.  It then places
// each record at its bucket's offset plus a rank from a shared-memory
// cursor: no global atomics.  A sub-partition of at most
// `cap` records is assembled in shared memory and written out as one
// contiguous range; a larger one (a large repeat bucket) is placed straight
// into global memory.  Blocks take sub-partitions from a counter.
template <int NW>
__global__ void __launch_bounds__(512, 2) k_scatter_sub(Stage<NW, true> from,
                                                     const unsigned long long* __restrict__ goff, uint32_t gsh,
                                                     uint32_t sb, uint32_t nsub, uint32_t cap,
                                                     uint64_t* __restrict__ pkeys, uint32_t* __restrict__ plink,
                                                     uint32_t* __restrict__ cout, unsigned long long* __restrict__ bout,
                                                     Counters* ctr) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  uint64_t* skey = reinterpret_cast<uint64_t*>(sm_raw);        // [cap * NW]
  uint32_t* slink = reinterpret_cast<uint32_t*>(skey + size_t(cap) * NW);  // [cap]
  __shared__ unsigned long long s_off[1 << SUB_MAX_BITS];
  __shared__ uint32_t s_cur[1 << SUB_MAX_BITS];
  // buckets' records among the first batch (when there are more records)
  __shared__ uint32_t s_first[1 << SUB_MAX_BITS];
  // the next sub-partition and its records, looked up by thread 0 while the
  // block works on this one
  __shared__ uint32_t s_sp;
  __shared__ unsigned long long s_lo, s_hi;
  __shared__ uint32_t sc[33];
  const uint32_t nbk = 1u << sb;  // <= 2^SUB_MAX_BITS <= blockDim.x
  // records per thread and pass: their loads are in flight together (two
  // CTAs per SM fit the registers)
  constexpr int PER = NW == 1 ? 8 : 5;
  const uint32_t batch = blockDim.x * PER;
  // known: goff holds every bucket's offset (no count groups)
  const bool known = cout == nullptr;
  // The first batch of a sub-partition: loaded before the one before it is
  // written out, in registers from there to its placement.  Counting it gives
  // each record its rank in its bucket (kept above the bucket), so
  // that only records past it take a second atomic to be placed.
  uint32_t bk[PER];
  Key<NW> kk[PER];
  uint32_t ln[PER];
  uint32_t sp;
  unsigned long long lo, hi;
  auto load = [&](unsigned long long i0) {
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const unsigned long long i = i0 + uint64_t(q) * blockDim.x + threadIdx.x;
      if (i < hi) from.get(i, kk[q], ln[q], bk[q]);
    }
  };
  auto next = [&] {
    sp = s_sp;
    lo = s_lo;
    hi = s_hi;
    load(lo);
  };
  uint32_t ticket = 0;  // thread 0: the sub-partition after s_sp
  auto look = [&](uint32_t t, unsigned long long& a, unsigned long long& b) {
    a = b = 0;
    if (t < nsub) {
      a = goff[uint64_t(t) << gsh];
      b = goff[uint64_t(t + 1) << gsh];
    }
  };
  if (threadIdx.x == 0) {
    unsigned long long a, b;
    const uint32_t t = atomicAdd(&ctr->work_sub, 1u);
    ticket = atomicAdd(&ctr->work_sub, 1u);
    look(t, a, b);
    s_sp = t;
    s_lo = a;
    s_hi = b;
  }
  __syncthreads();
  next();
  while (sp < nsub) {
    const uint64_t b0 = uint64_t(sp) << sb;
    for (uint32_t j = threadIdx.x; j < nbk; j += blockDim.x) {
      if (known) s_off[j] = goff[b0 + j];
      s_cur[j] = 0;
    }
    __syncthreads();
    unsigned long long nlo = 0, nhi = 0;
    uint32_t nsp = 0;
    if (threadIdx.x == 0) {
      nsp = ticket;
      look(nsp, nlo, nhi);
      ticket = atomicAdd(&ctr->work_sub, 1u);
    }
    const bool staged = hi - lo <= cap, more = hi - lo > batch;
    auto put = [&](int q, uint64_t pos) {
      if (staged) {
        st_key<NW>(skey, pos - lo, kk[q]);
        slink[pos - lo] = ln[q];
      } else {
        st_key<NW>(pkeys, pos, kk[q]);
        plink[pos] = ln[q];
      }
    };
    // places the records in registers by the buckets' cursors
    auto place = [&](unsigned long long i0) {
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const unsigned long long i = i0 + uint64_t(q) * blockDim.x + threadIdx.x;
        if (i < hi) {
          const uint32_t lb = bk[q] - uint32_t(b0);
          if (lb >= nbk) {  // not this sub-partition's: a broken order upstream
            atomicOr(&ctr->err, ERR_INTERNAL);
            continue;
          }
          put(q, s_off[lb] + atomicAdd(s_cur + lb, 1u));
        }
      }
    };
    if (known) {
      place(lo);
    } else {
      // the sub-partition's counts per bucket
#pragma unroll
      for (int q = 0; q < PER; ++q) {
        const unsigned long long i = lo + uint64_t(q) * blockDim.x + threadIdx.x;
        const uint32_t lb = bk[q] - uint32_t(b0);
        bk[q] = 0xFFFFFFFFu;
        if (i < hi) {
          if (lb < nbk) bk[q] = lb | (atomicAdd(s_cur + lb, 1u) << SUB_MAX_BITS);
          else atomicOr(&ctr->err, ERR_INTERNAL);
        }
      }
      __syncthreads();
      if (more) {
        for (uint32_t j = threadIdx.x; j < nbk; j += blockDim.x) s_first[j] = s_cur[j];
        __syncthreads();
        for (unsigned long long i0 = lo + batch; i0 < hi; i0 += batch) {
          uint32_t bq[PER];
#pragma unroll
          for (int q = 0; q < PER; ++q) {
            const unsigned long long i = i0 + uint64_t(q) * blockDim.x + threadIdx.x;
            bq[q] = (i < hi) ? from.bucket(i) : 0xFFFFFFFFu;
          }
#pragma unroll
          for (int q = 0; q < PER; ++q) {
            const uint32_t lb = bq[q] - uint32_t(b0);
            if (lb < nbk) atomicAdd(s_cur + lb, 1u);
          }
        }
        __syncthreads();
      }
      {
        const uint32_t cnt = threadIdx.x < nbk ? s_cur[threadIdx.x] : 0u;
        uint32_t tot;
        const uint32_t ex = block_excl_scan(cnt, sc, &tot);
        if (threadIdx.x < nbk) {
          s_off[threadIdx.x] = lo + ex;
          if (more) s_cur[threadIdx.x] = s_first[threadIdx.x];
          cout[b0 + threadIdx.x] = cnt;
          if (bout) bout[b0 + threadIdx.x] = lo + ex;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (bk[q] != 0xFFFFFFFFu) put(q, s_off[bk[q] & ((1u << SUB_MAX_BITS) - 1u)] + (bk[q] >> SUB_MAX_BITS));
    }
    if (more) {
      for (unsigned long long i0 = lo + batch; i0 < hi; i0 += batch) {
        load(i0);
        place(i0);
      }
    }
    if (threadIdx.x == 0) {
      s_sp = nsp;
      s_lo = nlo;
      s_hi = nhi;
    }
    __syncthreads();
    const unsigned long long at = lo;
    const uint32_t cnt = staged ? uint32_t(hi - lo) : 0u;
    next();
    for (uint32_t t = threadIdx.x; t < cnt; t += blockDim.x) {
      st_key<NW>(pkeys, at + t, ld_key<NW>(skey, t));
      plink[at + t] = slink[t];
    }
    __syncthreads();  // the staging area, s_off / s_cur are reused
  }
}

// ==================================================================== tiles

// List-ranking entries: (pointer, distance) in one 64-bit word.
__device__ __forceinline__ unsigned long long pk(uint32_t p, uint32_t o) {
  return (static_cast<unsigned long long>(o) << 32) | p;
}
__device__ __forceinline__ uint32_t pk_p(unsigned long long v) { return uint32_t(v); }
__device__ __forceinline__ uint32_t pk_o(unsigned long long v) { return uint32_t(v >> 32); }
// A head's own entry carries HEAD_BIT in its pointer, so "reached a head" is
// a property of the target entry, not a self-pointer (which a pointer running
// around a cycle can also produce).  Entry counts stay below 2^31.
constexpr uint32_t HEAD_BIT = 0x80000000u;
__device__ __forceinline__ uint32_t ptr_of(unsigned long long v) { return pk_p(v) & ~HEAD_BIT; }
__device__ __forceinline__ bool is_head_entry(unsigned long long v) { return (pk_p(v) & HEAD_BIT) != 0; }


// In-tile indices: 16-bit for shared-memory tiles (capacity <= 32766), 32-bit
// for oversized tiles worked in global scratch.  The top bit of A marks a
// shared prefix ("nullified", assembler.h:138-144) during the edge passes and
// a cycle copy during the cycle cut.
template <typename IT>
struct Ix;
template <>
struct Ix<uint16_t> {
  static constexpr uint32_t NONE = 0xFFFFu, DUP = 0x8000u, CNONE = 0x7FFFu;
};
template <>
struct Ix<uint32_t> {
  static constexpr uint32_t NONE = 0xFFFFFFFFu, DUP = 0x80000000u, CNONE = 0x7FFFFFFFu;
};

// 32-bit atomics on the word holding a 16-bit element; counters stay below
// 2^15 so no carry reaches the neighbouring element.
__device__ __forceinline__ uint32_t* word_of(uint16_t* p, uint32_t& sh) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  sh = uint32_t(a & 2u) * 8u;
  return reinterpret_cast<uint32_t*>(a & ~uintptr_t(3));
}
__device__ __forceinline__ void at_or(uint16_t* p, uint32_t v) {
  uint32_t sh;
  uint32_t* w = word_of(p, sh);
  atomicOr(w, v << sh);
}
__device__ __forceinline__ void at_or(uint32_t* p, uint32_t v) { atomicOr(p, v); }
__device__ __forceinline__ void at_inc(uint16_t* p) {
  uint32_t sh;
  uint32_t* w = word_of(p, sh);
  atomicAdd(w, 1u << sh);
}
__device__ __forceinline__ void at_inc(uint32_t* p) { atomicAdd(p, 1u); }
__device__ __forceinline__ uint32_t at_cas(uint16_t* p, uint32_t cmp, uint32_t val) {
  return atomicCAS(reinterpret_cast<unsigned short*>(p), static_cast<unsigned short>(cmp),
                   static_cast<unsigned short>(val));
}
__device__ __forceinline__ uint32_t at_cas(uint32_t* p, uint32_t cmp, uint32_t val) { return atomicCAS(p, cmp, val); }

template <int NW, typename IT>
struct TileMem {
  uint64_t* key;  // [cap * NW], role bits in the last word
  IT* A;          // suffix-lookup candidate | DUP  -> local successor
  IT* B;          // in-count                       -> scratch
  IT* P;          // who                            -> local predecessor -> segment id
  IT* Q;          // rank pointer / scratch
  IT* T;          // hash slots [ts >= 2*cap]       -> ranks / scratch
  uint32_t ts;
};

template <int NW, typename IT>
__device__ __forceinline__ TileMem<NW, IT> carve(char* base, uint32_t cap, uint32_t ts) {
  TileMem<NW, IT> m;
  const uint32_t cap4 = (cap + 3u) & ~3u;  // the index arrays in fours (vector initialisation)
  m.key = reinterpret_cast<uint64_t*>(base);
  m.A = reinterpret_cast<IT*>(m.key + size_t(cap) * NW);
  m.B = m.A + cap4;
  m.P = m.B + cap4;
  m.Q = m.P + cap4;
  m.T = m.Q + cap4;
  m.ts = ts;
  return m;
}

template <int NW, typename IT>
__device__ __forceinline__ Key<NW> skey(const TileMem<NW, IT>& m, uint32_t i) {
  Key<NW> k;
#pragma unroll
  for (int w = 0; w < NW; ++w) k.w[w] = m.key[size_t(i) * NW + w];
  return k;
}

struct U3 {
  unsigned long long a, b, c;
};
__device__ __forceinline__ U3 u3_add(U3 x, U3 y) { return U3{x.a + y.a, x.b + y.b, x.c + y.c}; }
__device__ __forceinline__ U3 u3_shfl_up(U3 v, int o) {
  return U3{__shfl_up_sync(0xFFFFFFFFu, v.a, o), __shfl_up_sync(0xFFFFFFFFu, v.b, o),
            __shfl_up_sync(0xFFFFFFFFu, v.c, o)};
}
// Exclusive block scan of three counters at once.
__device__ __forceinline__ U3 block_excl_scan3(U3 v, U3* sc, U3* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  U3 inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const U3 t = u3_shfl_up(inc, o);
    if (lane >= o) inc = u3_add(inc, t);
  }
  if (lane == 31) sc[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    U3 s = (lane < nw) ? sc[lane] : U3{0, 0, 0};
    U3 si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const U3 t = u3_shfl_up(si, o);
      if (lane >= o) si = u3_add(si, t);
    }
    if (lane < nw) sc[lane] = U3{si.a - s.a, si.b - s.b, si.c - s.c};
    if (lane == nw - 1) sc[32] = si;
  }
  __syncthreads();
  const U3 base = sc[wid];
  *total = sc[32];
  const U3 r{base.a + inc.a - v.a, base.b + inc.b - v.b, base.c + inc.c - v.c};
  __syncthreads();
  return r;
}

// Reserve a tile's closed-line bytes, open-segment chars and segment ids.
__device__ __forceinline__ int reserve_space(const TileParams& p, uint32_t job, const U3& tot,
                                             unsigned long long* b) {
  const JobTab& J = p.jobs[job];
  b[0] = tot.a ? atomicAdd(p.jout + job, tot.a) : 0ull;
  b[1] = tot.b ? atomicAdd(&p.ctr->seg_char_cursor, tot.b) : 0ull;
  b[2] = !tot.c ? 0u
         : p.rec_a ? atomicAdd(&p.ctr->rec_slots, tot.c << 32) >> 32
                   : (unsigned long long)atomicAdd(p.jseg + job, uint32_t(tot.c));
  if (b[0] + tot.a > J.ocap || b[1] + tot.b > p.segchars_cap || b[2] + tot.c > J.seg_cap) {
    atomicOr(&p.ctr->err, ERR_CAPACITY);
    return 0;
  }
  b[0] += J.obase;
  b[2] += J.seg_base;
  return 1;
}

// Thread-group policies: a tile is worked by a whole block or by one warp.
struct BlockGroup {
  static __device__ __forceinline__ uint32_t rank() { return threadIdx.x; }
  static __device__ __forceinline__ uint32_t size() { return blockDim.x; }
  static __device__ __forceinline__ void sync() { __syncthreads(); }
  static __device__ __forceinline__ int sync_or(int v) { return __syncthreads_or(v); }
  static __device__ __forceinline__ U3 scan3(U3 v, U3* total) {
    __shared__ U3 sc[33];
    return block_excl_scan3(v, sc, total);
  }
  // The leader reserves output space for the tile; false if a bound was hit.
  static __device__ __forceinline__ bool reserve(const TileParams& p, uint32_t job, const U3& tot,
                                                 unsigned long long* base) {
    __shared__ unsigned long long s_base[3];
    __shared__ int s_ok;
    if (threadIdx.x == 0) s_ok = reserve_space(p, job, tot, s_base);
    __syncthreads();
    base[0] = s_base[0];
    base[1] = s_base[1];
    base[2] = s_base[2];
    const int ok = s_ok;
    __syncthreads();
    return ok;
  }
};

struct WarpGroup {
  static __device__ __forceinline__ uint32_t rank() { return threadIdx.x & 31u; }
  static __device__ __forceinline__ uint32_t size() { return 32u; }
  static __device__ __forceinline__ void sync() { __syncwarp(); }
  static __device__ __forceinline__ bool reserve(const TileParams& p, uint32_t job, const U3& tot,
                                                 unsigned long long* base) {
    unsigned long long b[3] = {0, 0, 0};
    int ok = 1;
    if ((threadIdx.x & 31) == 0) ok = reserve_space(p, job, tot, b);
    base[0] = __shfl_sync(0xFFFFFFFFu, b[0], 0);
    base[1] = __shfl_sync(0xFFFFFFFFu, b[1], 0);
    base[2] = __shfl_sync(0xFFFFFFFFu, b[2], 0);
    return __shfl_sync(0xFFFFFFFFu, ok, 0);
  }
};

// Pointer-jumping rounds over (px, rx) with second buffers (py, ry); the
// result lands in (ptr, rnk).  Starts point at themselves with rank 0.
template <typename G, typename IT>
__device__ void jump_rounds(uint32_t c, IT* px, IT* rx, IT* py, IT* ry, IT*& ptr, IT*& rnk) {
  uint32_t rounds = 1;
  for (uint32_t lim = 1; lim < c; lim <<= 1) ++rounds;
  for (uint32_t r = 0; r < rounds; ++r) {
    int changed = 0;
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      const uint32_t p = px[i];
      const uint32_t np = px[p];
      py[i] = IT(np);
      ry[i] = IT(uint32_t(rx[i]) + uint32_t(rx[p]));
      changed |= (np != p);
    }
    IT* t = px; px = py; py = t;
    t = rx; rx = ry; ry = t;
    if (!G::sync_or(changed)) break;
  }
  ptr = px;
  rnk = rx;
}

// Segments and lines of a warp tile whose kept edges are known (A: local
// successor or NONE, P: local predecessor or NONE).  In-tile paths are short
// (the consecutive k-mers that share one minimizer, and half of the edges of
// canonical k-mers drop), so a lane takes a segment's end and walks back to
// its start, gathering the chars the later copies add as 2-bit codes; the
// text of 32 segments at a time is spelled into shared memory from those codes
// and leaves as 16-byte stores.  Against ranking the copies by pointer jumping
// and storing each copy's char by itself: 64 Mbp, k = 63, the kernel takes
// 2.36 instead of 3.01 ms; at k = 31 it was as long either way, with half as many
// stores.  (Now, with longer tables and closed lines as records: 1.77 ms, and 6.4
// at 256 Mbp, k = 31.)  Segments with more than TAIL_MAX later chars store them
// byte by byte.
template <int NW, int KC>
__device__ __forceinline__ void emit_warp_tile(const TileParams& p, const TileMem<NW, uint16_t>& m, uint64_t beg,
                                               uint32_t c, uint32_t job, unsigned long long& rec_bytes) {
  constexpr uint32_t NONE_I = Ix<uint16_t>::NONE;
  const int k = KC ? KC : p.k;
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  // segment ends, in B (the in-counts are used up)
  uint32_t nend = 0;
  for (uint32_t base = 0; base < c; base += 32) {
    const uint32_t i = base + lane;
    const bool e = i < c && m.A[i] == NONE_I;
    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, e);
    if (e) m.B[nend + __popc(mask & below)] = uint16_t(i);
    nend += uint32_t(__popc(mask));
  }
  __syncwarp();
  // sizes; the closed segments' ends to the front of A, the open ones' to its
  // back (the successors are used up: cycles are found from P)
  uint32_t nclosed, nopen, heads, cbytes, obytes;
  bool longer;  // a closed line with more later chars than a record holds
  for (bool cut = false;; cut = true) {
    nclosed = nopen = 0;
    uint32_t h = 0, cb = 0, ob = 0, covered = 0, lmax = 0;
    for (uint32_t base = 0; base < nend; base += 32) {
      const bool live = base + lane < nend;
      uint32_t i = 0, s = 0, len = 0;
      bool starts_p = false, closed = false;
      if (live) {
        i = s = m.B[base + lane];
        len = 1;
        for (uint32_t q = m.P[s]; q != NONE_I && len < c; q = m.P[s]) {
          s = q;
          ++len;
        }
        starts_p = (roles(skey(m, s)) & ROLE_P) != 0;
        closed = starts_p && (roles(skey(m, i)) & ROLE_S);
        covered += len;
        if (closed) {
          cb += uint32_t(k) + len;
          lmax = max(lmax, len);
        } else {
          ob += starts_p ? uint32_t(k) - 1u + len : len - 1u;
          h += starts_p ? 1u : 0u;
        }
      }
      const uint32_t cm = __ballot_sync(0xFFFFFFFFu, closed), om = __ballot_sync(0xFFFFFFFFu, live && !closed);
      if (closed) m.A[nclosed + __popc(cm & below)] = uint16_t(i);
      else if (live) m.A[c - 1u - nopen - __popc(om & below)] = uint16_t(i);
      nclosed += uint32_t(__popc(cm));
      nopen += uint32_t(__popc(om));
    }
    covered = __reduce_add_sync(0xFFFFFFFFu, covered);
    heads = __reduce_add_sync(0xFFFFFFFFu, h);
    cbytes = __reduce_add_sync(0xFFFFFFFFu, cb);
    obytes = __reduce_add_sync(0xFFFFFFFFu, ob);
    longer = __any_sync(0xFFFFFFFFu, lmax > uint32_t(TAIL_MAX) + 1u);
    if (covered == c || cut) break;
    // local cycles hold the copies no end reaches (rare): one lane cuts each
    // before its smallest key, which then starts a segment
    for (uint32_t i = lane; i < c; i += 32) m.Q[i] = 0;
    __syncwarp();
    for (uint32_t j = lane; j < nend; j += 32)
      for (uint32_t s = m.B[j], n = 0; s != NONE_I && n < c; s = m.P[s], ++n) m.Q[s] = 1;
    __syncwarp();
    if (lane == 0) {
      for (uint32_t i = 0; i < c; ++i) {
        if (m.Q[i]) continue;
        uint32_t best = i;
        m.Q[i] = 1;
        for (uint32_t s = m.P[i], n = 0; s != i && s != NONE_I && n < c; s = m.P[s], ++n) {
          m.Q[s] = 1;
          if (key_lt(skey(m, s), skey(m, best))) best = s;
        }
        m.B[nend++] = m.P[best];
        m.P[best] = uint16_t(NONE_I);
      }
    }
    nend = __shfl_sync(0xFFFFFFFFu, nend, 0);
    __syncwarp();
  }
  // sorted output: the closed lines leave as records (unless one is too long)
  const bool recs = p.rec_a != nullptr && !longer;
  unsigned long long at[3] = {0, 0, 0};
  if (recs) {
    unsigned long long v = 0;
    uint32_t ok = 1;
    if (lane == 0) {
      if (nclosed | heads) v = atomicAdd(&p.ctr->rec_slots, (static_cast<unsigned long long>(heads) << 32) | nclosed);
      if (obytes) at[1] = atomicAdd(&p.ctr->seg_char_cursor, (unsigned long long)obytes);
      if (at[1] + obytes > p.segchars_cap || (v >> 32) + heads > p.jobs[job].seg_cap) {
        atomicOr(&p.ctr->err, ERR_CAPACITY);
        ok = 0;
      }
    }
    v = __shfl_sync(0xFFFFFFFFu, v, 0);
    at[1] = __shfl_sync(0xFFFFFFFFu, at[1], 0);
    if (!__shfl_sync(0xFFFFFFFFu, ok, 0)) return;
    at[2] = (v >> 32) + p.jobs[job].seg_base;
    rec_bytes += cbytes;
    const uint32_t slot = uint32_t(v);
    __syncwarp();
    const RecArr<NW + 1> out{p.rec_a, p.rec_t};
    for (uint32_t base = 0; base < nclosed; base += 32) {
      const uint32_t j = base + lane;
      uint32_t bin = NONE;
      if (j < nclosed) {
        uint32_t s = m.A[j], len = 1;
        uint64_t tail = 0;
        for (uint32_t q = m.P[s]; q != NONE_I && len < c; q = m.P[s]) {
          tail = (tail << 2) | key_char(skey(m, s), k - 1);
          s = q;
          ++len;
        }
        const Key<NW> x = strip(skey(m, s));
        Rec<NW + 1> r;
        if constexpr (NW == 1) {
          r.hi = rev2(x.w[0]);
          r.lo = 0;
        } else {
          r.hi = rev2(x.w[0]);
          r.lo = rev2(x.w[1]);
        }
        r.tail = (uint64_t(len - 1u) << TAIL_LEN_SHIFT) | tail;
        st_rec<NW + 1>(out, uint64_t(slot) + j, r);
        bin = uint32_t(r.hi >> (64 - p.rec_bits));
      }
      count_bin(p.rec_counts, bin);
    }
  } else {
    if (!WarpGroup::reserve(p, job, U3{cbytes, obytes, heads}, at)) return;
    __syncwarp();
  }
  // text buffer: the arrays Q and T, less the piece that WarpText::flush may
  // read past the text (room for one line is left in the smallest tile: 32
  // copies have 192 bytes there)
  const uintptr_t q0 = reinterpret_cast<uintptr_t>(m.Q);
  uint32_t* buf = reinterpret_cast<uint32_t*>((q0 + 15) & ~uintptr_t(15));
  const uint32_t room =
      (uint32_t(reinterpret_cast<uintptr_t>(m.T + m.ts) - reinterpret_cast<uintptr_t>(buf)) & ~15u) - 16u;
  uint32_t head0 = p.xcount + uint32_t(at[2]);  // id of the next segment that starts a line
  constexpr int NC = NW == 1 ? 4 : 6;
#pragma unroll 1
  for (uint32_t open = recs ? 1u : 0u; open < 2; ++open) {
    const uint32_t nseg = open ? nopen : nclosed;
    WarpText T;
    T.begin(open ? p.segchars + at[1] : p.out + at[0]);
    for (uint32_t base = 0; base < nseg;) {
      const bool live = base + lane < nseg;
      uint32_t i = 0, s = 0, len = 0;
      uint64_t tail = 0;
      Key<NW> ks;
#pragma unroll
      for (int w = 0; w < NW; ++w) ks.w[w] = 0;
      bool starts_p = false;
      uint32_t xs = NONE, xe = NONE;
      if (live) {
        i = s = open ? m.A[c - 1u - base - lane] : m.A[base + lane];
        len = 1;
        for (uint32_t q = m.P[s]; q != NONE_I && len < c; q = m.P[s]) {
          tail = (tail << 2) | key_char(skey(m, s), k - 1);
          s = q;
          ++len;
        }
        ks = skey(m, s);
        starts_p = (roles(ks) & ROLE_P) != 0;
        if (open) {
          // this segment's id (S-only start), the next one's (P-only end)
          if (!starts_p) xs = p.plink[beg + s];
          if (!(roles(skey(m, i)) & ROLE_S)) xe = p.plink[beg + i];
        }
      }
      // chars: the first k-mer in full, unless it ends the segment before
      const uint32_t nch = live ? (starts_p ? uint32_t(k) - 1u + len : len - 1u) : 0u;
      const uint32_t nb = live ? nch + (open ? 0u : 1u) : 0u;
      uint32_t inc = nb;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= uint32_t(o)) inc += v;
      }
      const bool direct = __any_sync(0xFFFFFFFFu, len > uint32_t(TAIL_MAX) + 1u);
      // the lanes whose text fits the buffer (all of them when it is not used)
      const bool take = live && (direct || T.fill + inc <= room);
      const uint32_t taken = __ballot_sync(0xFFFFFFFFu, take);
      const uint32_t cnt = uint32_t(__popc(taken));  // a prefix of the lanes
      const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, int(cnt) - 1);
      char* const first = T.dst + (inc - nb);
      if (!direct) {
        if (take) {
          uint64_t w[3];
          const uint64_t codes = len > 1u ? tail : 0ull;
          w[0] = w[1] = w[2] = 0;
          const Key<NW> x = strip(ks);
          if (!starts_p) {
            w[0] = codes;
          } else if constexpr (NW == 1) {
            w[0] = x.w[0] | (codes << (2 * k));
            w[1] = codes >> (64 - 2 * k);
          } else {
            const int u = 2 * k - 64;
            w[0] = x.w[0];
            w[1] = x.w[1] | (codes << u);
            w[2] = u ? codes >> (64 - u) : 0ull;
          }
          uint32_t xx[NC];
#pragma unroll
          for (int q = 0; q < NC; ++q) xx[q] = uint32_t(w[q >> 1] >> (32 * (q & 1)));
          spell_text<NC>(buf, T.fill + inc - nb, xx, nch, open ? 0u : 1u);
        }
        __syncwarp();
        T.flush(buf, total);
      } else {
        T.end(buf);
        if (live) {
          if (starts_p) spell_key<NW>(first, ks, k);
          char* d = first + nch;  // the chars of the later copies, last first
          if (!open) *d = '\n';
          uint32_t t = i;
          for (uint32_t r = 1; r < len; ++r) {
            *--d = acgt(key_char(skey(m, t), k - 1));
            t = m.P[t];
          }
        }
        __syncwarp();
        T.begin(T.dst + total);
      }
      if (open) {
        const uint32_t hm = __ballot_sync(0xFFFFFFFFu, take && starts_p);
        if (take) {
          // the segment's record under its id; it continues in segment xe
          SegRec rec;
          rec.off_job = uint64_t(first - p.segchars) | (static_cast<unsigned long long>(job) << SEG_OFF_BITS);
          rec.len = len;
          rec.next = xe;
          p.seg[starts_p ? head0 + __popc(hm & below) : xs] = rec;
        }
        head0 += uint32_t(__popc(hm));
      }
      base += cnt;
    }
    T.end(buf);
  }
}

// KC: k fixed at compile time (0: p.k), so that the masks, shifts and
// spelling loops of the common shapes are constants.
template <int NW, typename IT, typename G, int KC = 0>
__device__ void process_tile(const TileParams& p, const TileMem<NW, IT>& m, uint64_t beg, uint32_t c,
                             uint32_t job, unsigned long long& rec_bytes) {
  constexpr uint32_t NONE_I = Ix<IT>::NONE, DUP_I = Ix<IT>::DUP, CNONE_I = Ix<IT>::CNONE;
  constexpr uint32_t OPEN_S = NONE_I - 1u;  // an open segment that starts at an S-only copy
  constexpr bool WARP = std::is_same<G, WarpGroup>::value;
  const int k = KC ? KC : p.k;
  const PrefMask pm = pref_mask(k);
  // this tile's hash slots: the power of two above c * lf / 100, at most the
  // carved table (32-bit arithmetic for shared-memory tiles, c <= 8192)
  uint32_t ts;
  {
    const uint32_t lf = WARP ? p.wlf : p.lf;
    const uint32_t want = (sizeof(IT) == 2) ? (c * lf) / 100u : uint32_t((uint64_t(c) * lf) / 100u);
    const uint32_t x = want > c ? want : c + 1u;
    ts = 1u << (32 - __clz(x - 1u));
    ts = ts < m.ts ? ts : m.ts;
  }
  const uint32_t tmask = ts - 1;
  // ---- stage the tile's keys (async copies), initialise the work arrays
  if constexpr (sizeof(IT) == 2) {
    // shared-memory tile: asynchronous copies overlap the initialisation
    for (uint32_t i = G::rank(); i < c; i += G::size())
      __pipeline_memcpy_async(m.key + size_t(i) * NW, p.pkeys + (beg + i) * NW, 8 * NW);
    __pipeline_commit();
  } else {
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      const Key<NW> x = ld_key<NW>(p.pkeys, beg + i);
#pragma unroll
      for (int w = 0; w < NW; ++w) m.key[size_t(i) * NW + w] = x.w[w];
    }
  }
  if constexpr (sizeof(IT) == 2) {
    // four 16-bit entries per store (carve sizes the arrays in fours)
    uint64_t* A4 = reinterpret_cast<uint64_t*>(m.A);
    uint64_t* B4 = reinterpret_cast<uint64_t*>(m.B);
    uint64_t* P4 = reinterpret_cast<uint64_t*>(m.P);
    for (uint32_t i = G::rank(); i < (c + 3u) >> 2; i += G::size()) {
      A4[i] = 0x7FFF7FFF7FFF7FFFull;  // CNONE
      B4[i] = 0ull;
      P4[i] = ~0ull;                  // NONE
    }
    if (ts >= 4) {
      uint64_t* T4 = reinterpret_cast<uint64_t*>(m.T);
      for (uint32_t i = G::rank(); i < (ts >> 2); i += G::size()) T4[i] = ~0ull;
    } else {
      for (uint32_t i = G::rank(); i < ts; i += G::size()) m.T[i] = IT(NONE_I);
    }
  } else {
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      m.A[i] = IT(CNONE_I);
      m.B[i] = 0;
      m.P[i] = IT(NONE_I);
    }
    for (uint32_t i = G::rank(); i < ts; i += G::size()) m.T[i] = IT(NONE_I);
  }
  if constexpr (sizeof(IT) == 2) __pipeline_wait_prior(0);
  G::sync();
  // ---- prefix table of the P copies (generate_hashmap, assembler.h:120-150):
  // one slot per distinct (k-1)-prefix; a prefix held by two copies marks the
  // slot's copy DUP ("nullified")
  if constexpr (WARP) {
    // one warp works the table, so a free slot is taken by a plain store and
    // a look at who won it (16-bit compare-and-swaps are several times as long)
    for (uint32_t base = 0; base < c; base += 32) {
      const uint32_t i = base + G::rank();
      bool open = i < c;
      Key<NW> pf;
      uint32_t h = 0;
      if (open) {
        const Key<NW> x = skey(m, i);
        open = (roles(x) & ROLE_P) != 0;
        pf = prefix_of(x, pm);
        h = key_hash(pf) & tmask;
      }
      while (__any_sync(0xFFFFFFFFu, open)) {
        if (open && m.T[h] == NONE_I) m.T[h] = IT(i);
        __syncwarp();
        if (open) {
          const uint32_t cur = m.T[h];
          if (cur == i) {
            open = false;
          } else if (key_eq(prefix_of(skey(m, cur), pm), pf)) {
            m.A[cur] = IT(CNONE_I | DUP_I);
            open = false;
          } else {
            h = (h + 1) & tmask;
          }
        }
        __syncwarp();
      }
    }
  } else {
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    const Key<NW> x = skey(m, i);
    if (!(roles(x) & ROLE_P)) continue;
    const Key<NW> pf = prefix_of(x, pm);
    uint32_t h = key_hash(pf) & tmask;
    for (uint32_t probe = 0; probe <= tmask; ++probe) {
      const uint32_t cur = at_cas(m.T + h, NONE_I, i);
      if (cur == NONE_I) break;
      if (key_eq(prefix_of(skey(m, cur), pm), pf)) {
        at_or(m.A + cur, DUP_I);
        break;
      }
      h = (h + 1) & tmask;
    }
  }
  }
  G::sync();
  // ---- suffix lookups of the S copies (find_vtx_from_edge, assembler.h:89-111)
  // and in-degree counts ("count edges", assembler.h:180-188)
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    const Key<NW> x = skey(m, i);
    if (!(roles(x) & ROLE_S)) continue;
    const Key<NW> sf = suffix_of(x, pm);
    uint32_t h = key_hash(sf) & tmask;
    uint32_t cand = CNONE_I;
    for (uint32_t probe = 0; probe <= tmask; ++probe) {
      const uint32_t cur = m.T[h];
      if (cur == NONE_I) break;
      if (key_eq(prefix_of(skey(m, cur), pm), sf)) {
        if (!(uint32_t(m.A[cur]) & DUP_I)) cand = cur;
        break;
      }
      h = (h + 1) & tmask;
    }
    if (cand != CNONE_I) {
      at_inc(m.B + cand);
      m.P[cand] = IT(i);
    }
    m.A[i] = IT((uint32_t(m.A[i]) & DUP_I) | cand);
  }
  G::sync();
  // ---- kept edges: u->v iff v is u's unique successor and u is v's only
  // predecessor ("write edges", assembler.h:189-197); rank init alongside
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    const uint32_t cand = uint32_t(m.A[i]) & CNONE_I;
    const uint32_t s = (cand != CNONE_I && m.B[cand] == 1u) ? cand : NONE_I;
    const uint32_t q = (m.B[i] == 1u) ? uint32_t(m.P[i]) : NONE_I;
    m.A[i] = IT(s);
    m.P[i] = IT(q);
    if constexpr (!WARP) {
      m.Q[i] = IT(q == NONE_I ? i : q);
      m.T[i] = IT(q == NONE_I ? 0u : 1u);
    }
  }
  G::sync();
  if (p.mode == 0) {
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      const uint64_t r = roles(skey(m, i));
      const uint32_t id = p.plink[beg + i];
      // (both arrays hold NONE: only links are stored)
      if ((r & ROLE_S) && m.A[i] != NONE_I) p.succ[id] = p.plink[beg + m.A[i]];
      if ((r & ROLE_P) && m.P[i] != NONE_I) p.pred[id] = p.plink[beg + m.P[i]];
    }
    return;
  }
  if constexpr (WARP) {
    emit_warp_tile<NW, KC>(p, m, beg, c, job, rec_bytes);
    return;
  } else {
  // ---- local segments: list ranking by pointer jumping
  IT *ptr, *rnk;
  jump_rounds<G, IT>(c, m.Q, m.T, m.B, m.T + c, ptr, rnk);
  // ---- local cycles (every copy has a local predecessor): cut each at its
  // smallest key, then rank again
  int cyc = 0;
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    // a path copy points at its start (no predecessor); a cycle copy at
    // another cycle copy.  Cycle copies have a successor, so A = index | DUP.
    if (m.P[ptr[i]] != NONE_I) {
      m.A[i] = IT(uint32_t(m.A[i]) | DUP_I);
      cyc = 1;
    }
  }
  if (G::sync_or(cyc)) {
    IT *lx = m.T, *jx = m.T + c, *ly = m.B, *jy = m.Q;
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      lx[i] = IT(i);
      jx[i] = IT(m.P[i] == NONE_I ? i : uint32_t(m.P[i]));
    }
    G::sync();
    uint32_t rounds = 1;
    for (uint32_t lim = 1; lim < c; lim <<= 1) ++rounds;
    for (uint32_t r = 0; r < rounds; ++r) {
      for (uint32_t i = G::rank(); i < c; i += G::size()) {
        const uint32_t j = jx[i];
        const uint32_t a = lx[i], b = lx[j];
        ly[i] = IT(key_lt(skey(m, b), skey(m, a)) ? b : a);
        jy[i] = jx[j];
      }
      G::sync();
      IT* t = lx; lx = ly; ly = t;
      t = jx; jx = jy; jy = t;
    }
    // after ceil(log2 c)+1 rounds a cycle copy's label covers its whole cycle:
    // exactly one copy per cycle (the smallest key) is its own label; the edge
    // into it is cut, path copies are untouched
    auto on_cycle = [](uint32_t a) { return a != NONE_I && (a & DUP_I); };
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      if (on_cycle(m.A[i]) && lx[i] == i) {
        const uint32_t q = m.P[i];
        m.A[q] = IT(NONE_I);
        m.P[i] = IT(NONE_I);
      }
    }
    G::sync();
    for (uint32_t i = G::rank(); i < c; i += G::size()) {
      const uint32_t a = m.A[i];
      if (on_cycle(a)) m.A[i] = IT(a & ~DUP_I);
      const uint32_t q = m.P[i];
      m.Q[i] = IT(q == NONE_I ? i : q);
      m.T[i] = IT(q == NONE_I ? 0u : 1u);
    }
    G::sync();
    jump_rounds<G, IT>(c, m.Q, m.T, m.B, m.T + c, ptr, rnk);
  }
  // every copy now reaches a segment start.  Free arrays: the pair not
  // holding (ptr, rnk) keeps each start's byte offset (lo/hi halves), P its
  // local segment id.
  IT* lo_a = (ptr == m.Q) ? m.B : m.Q;
  IT* hi_a = (rnk == m.T) ? m.T + c : m.T;
  // ---- emission: closed segments (start has role P, end has role S) are
  // whole unitigs; the others are stitched across tiles.  Open segments that
  // start at a P-role copy start a stitched line: they take head-pool ids;
  // the others start at an S-only copy and take its cross index.
  // Each thread's lines are contiguous in the tile's output, in the order the
  // thread visits them (the order of lines is free).
  U3 mine{0, 0, 0};
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    if (m.A[i] != NONE_I) continue;  // not a segment's end
    const uint32_t s = ptr[i];
    const uint32_t len = uint32_t(rnk[i]) + 1;
    const bool starts_p = (roles(skey(m, s)) & ROLE_P) != 0;
    const bool closed = starts_p && (roles(skey(m, i)) & ROLE_S);
    if (closed) mine.a += uint64_t(k) + len;
    else { mine.b += starts_p ? uint64_t(k) - 1 + len : uint64_t(len) - 1; mine.c += starts_p ? 1 : 0; }
  }
  U3 tot;
  U3 pre = G::scan3(mine, &tot);
  unsigned long long s_base[3];
  if (!G::reserve(p, job, tot, s_base)) return;
  const unsigned long long cbase = s_base[0], obase = s_base[1], sbase = s_base[2];
  // per segment (the lane that sized it): its offset (kept at its start for
  // the per-copy pass), its first k-mer in full (a segment that starts at an
  // S-only copy keeps only the chars it adds to its line: that k-mer ends
  // the segment before), then its line break or, for an open segment, its
  // record.  The cross indices the record needs are loaded first, so that
  // they arrive while the rest is worked out.
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    if (m.A[i] != NONE_I) continue;  // not a segment's end
    const uint32_t s = ptr[i];
    const Key<NW> ks = skey(m, s);
    const uint64_t re = roles(skey(m, i));
    const bool starts_p = (roles(ks) & ROLE_P) != 0;
    const bool p_only = (re & ROLE_S) == 0;
    const bool closed = starts_p && !p_only;
    const uint32_t xs = starts_p ? NONE : p.plink[beg + s];  // this segment's id (S-only start)
    const uint32_t xe = p_only ? p.plink[beg + i] : NONE;   // the next segment's id
    const uint32_t r = rnk[i];
    const uint32_t len = r + 1;
    uint64_t loc;
    uint32_t sid;
    if (closed) {
      loc = pre.a;
      sid = NONE_I;
      pre.a += uint64_t(k) + len;
    } else {
      loc = pre.b;
      sid = starts_p ? uint32_t(pre.c) : OPEN_S;
      pre.b += starts_p ? uint64_t(k) - 1 + len : uint64_t(len) - 1;
      if (starts_p) pre.c += 1;
    }
    m.P[s] = IT(sid);
    if constexpr (sizeof(IT) == 2) {
      lo_a[s] = IT(loc & 0xFFFFu);
      hi_a[s] = IT(loc >> 16);
    } else {
      lo_a[s] = IT(loc);
    }
    char* dst = closed ? (p.out + cbase + loc) : (p.segchars + obase + loc);
    if (sid != OPEN_S) spell_key<NW>(dst, ks, k);
    if (closed) {
      dst[k + r] = '\n';
    } else {
      // the segment's record under its id; a segment that ends at the P-only
      // copy of cross k-mer xe continues in segment xe
      const uint32_t g = starts_p ? p.xcount + uint32_t(sbase) + sid : xs;
      SegRec rec;
      rec.off_job = (obase + loc) | (static_cast<unsigned long long>(job) << SEG_OFF_BITS);
      rec.len = len;
      rec.next = xe;
      p.seg[g] = rec;
    }
  }
  G::sync();
  // every later copy of a segment adds its last char
  for (uint32_t i = G::rank(); i < c; i += G::size()) {
    const uint32_t r = rnk[i];
    if (r == 0) continue;
    const uint32_t s = ptr[i];
    uint64_t loc = lo_a[s];
    if constexpr (sizeof(IT) == 2) loc |= uint64_t(hi_a[s]) << 16;
    const uint32_t sid = m.P[s];
    char* dst = (sid == NONE_I) ? (p.out + cbase + loc) : (p.segchars + obase + loc);
    dst[(sid == OPEN_S ? 0u : uint32_t(k)) + r - 1] = acgt(key_char(skey(m, i), k - 1));
  }
  }  // (block tiles)
}

// Persistent tile kernels.  Warp tiles (<= warp capacity copies): every warp
// of a CTA owns a slice of shared memory and takes the next warp tile from a
// global counter, with warp-level synchronisation only.  Block tiles (up to
// the tile capacity): the whole CTA works one tile.  Larger tiles go to
// k_tile_big.
template <int NW, int KC>
__global__ void __launch_bounds__(256, NW == 1 ? 4 : 3) k_tile_warp(TileParams p) {
  extern __shared__ __align__(16) char smem[];
  const uint32_t wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const TileMem<NW, uint16_t> m = carve<NW, uint16_t>(smem + size_t(wid) * p.wbytes, p.wcap, p.wts);
  if (p.ctr->err & ERR_TIMEOUT) return;  // the plan did not finish
  const uint32_t nt = p.ctr->nwarp, nw = gridDim.x * (blockDim.x >> 5);
  unsigned long long rec_bytes = 0;
  uint32_t j = blockIdx.x * (blockDim.x >> 5) + wid;  // the first tile needs no counter
  while (j < nt) {
    uint32_t jn = 0;  // the next tile's index is in flight while this tile is worked
    if (lane == 0) jn = nw + atomicAdd(&p.ctr->wtile_next, 1u);
    const uint32_t t = p.wlist[j];
    const uint64_t beg = p.tile_begin[t];
    const uint32_t c = uint32_t(p.tile_begin[t + 1] - beg);
    process_tile<NW, uint16_t, WarpGroup, KC>(p, m, beg, c, p.tile_job[t], rec_bytes);
    __syncwarp();
    j = __shfl_sync(0xFFFFFFFFu, jn, 0);
  }
  if (lane == 0 && rec_bytes) atomicAdd(&p.ctr->rec_bytes, rec_bytes);
}

template <int NW, int KC>
__global__ void __launch_bounds__(512) k_tile(TileParams p) {
  extern __shared__ __align__(16) char smem[];
  __shared__ uint32_t s_t;
  const TileMem<NW, uint16_t> m = carve<NW, uint16_t>(smem, p.cap, p.tslots);
  if (p.ctr->err & ERR_TIMEOUT) return;  // the plan did not finish
  const uint32_t nt = p.ctr->nblock;
  for (;;) {
    if (threadIdx.x == 0) s_t = atomicAdd(&p.ctr->tile_next, 1u);
    __syncthreads();
    const uint32_t j = s_t;
    __syncthreads();
    if (j >= nt) break;
    const uint32_t t = p.blist[j];
    const uint64_t beg = p.tile_begin[t];
    const uint32_t c = uint32_t(p.tile_begin[t + 1] - beg);
    unsigned long long none = 0;
    process_tile<NW, uint16_t, BlockGroup, KC>(p, m, beg, c, p.tile_job[t], none);
    __syncthreads();
  }
}

// One CTA per oversized tile, working in global scratch.
template <int NW>
__global__ void __launch_bounds__(1024) k_tile_big(TileParams p) {
  const uint32_t t = p.big_list[blockIdx.x];
  const uint64_t beg = p.tile_begin[t];
  const uint64_t c = p.tile_begin[t + 1] - beg;
  const uint32_t ts = big_slots(c, p.lf);
  const TileMem<NW, uint32_t> m = carve<NW, uint32_t>(p.big_scratch + p.big_off[blockIdx.x], uint32_t(c), ts);
  unsigned long long none = 0;
  process_tile<NW, uint32_t, BlockGroup>(p, m, beg, uint32_t(c), p.tile_job[t], none);
}

// ================================================================= stitch
//
// Open segments continue through cross k-mers: the segment that ends at the
// P-only copy of cross k-mer x is followed by segment x (the one that starts
// at x's S-only copy); both hold x, so every later segment of a line drops
// its first k chars (write_unitigs4, compact.h:59-112), and the tiles keep
// only the chars it adds.  The tiles write each segment's record under its
// id.  The common case is one kernel (k_walk_emit): a thread per line head
// walks its line twice, once for its length, then, after one output
// reservation per job and warp, to copy the segments' chars into one
// contiguous line.  Lines longer than WALK_CAP segments and cycles (no
// head) go through list ranking (pointer jumping from the first state
// rebuilt from the records, or HEC), line lengths at the heads
// (k_chain_len), one reservation per line (k_line_reserve) and a copy per
// segment (k_seg_copy).

// The chars a segment adds to its line: all k - 1 + len for a line's first
// segment (a head-pool id), len - 1 for the others.
__device__ __forceinline__ uint32_t seg_w(uint32_t s, uint32_t len, uint32_t nx, int k) {
  return s < nx ? len - 1u : uint32_t(k) - 1u + len;
}

// First of c consecutive slots for each thread of a block that appends to a
// shared list: one atomic per block.  A list counter that every block of the
// grid bumps serialises in L2, so per-warp appends would bound a pass that
// appends most of its elements.  Every thread of the block must call it;
// sc holds 33 values.
__device__ __forceinline__ uint32_t block_append(uint32_t* count, uint32_t c, uint32_t* sc) {
  uint32_t tot;
  const uint32_t pre = block_excl_scan(c, sc, &tot);  // ends with a barrier after every read of sc
  if (threadIdx.x == 0) sc[32] = tot ? atomicAdd(count, tot) : 0u;
  __syncthreads();
  const uint32_t b = sc[32] + pre;
  __syncthreads();  // sc is reused by the next call
  return b;
}

// X[v] = (start pointer, weight distance); heads point at themselves.
__global__ void __launch_bounds__(256) k_rank_init(const uint32_t* __restrict__ prev, const uint32_t* __restrict__ w,
                            uint64_t n, unsigned long long* __restrict__ X,
                            uint32_t* __restrict__ act, uint32_t* act_count) {
  __shared__ uint32_t sc[33];
  const uint64_t N = n;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  // whole blocks iterate together (block_append needs every thread)
  for (uint64_t s0 = uint64_t(blockIdx.x) * blockDim.x; s0 < N; s0 += stride) {
    const uint64_t s = s0 + threadIdx.x;
    bool tail = false;
    if (s < N) {
      const uint32_t pv = prev[s];
      if (pv == NONE) {
        X[s] = pk(uint32_t(s) | HEAD_BIT, 0);
      } else {
        X[s] = pk(pv, w ? w[pv] : 1u);
        tail = true;
      }
    }
    const uint32_t slot = block_append(act_count, tail ? 1u : 0u, sc);
    if (tail) act[slot] = uint32_t(s);
  }
}

// One round of asynchronous pointer jumping over the active list (act ==
// nullptr: the first round, over the ids [0, *act_count)).  Entries are
// (pointer, distance) pairs in one 64-bit word, so a concurrent reader
// always sees a consistent pair; the list keeps the entries whose pointer
// does not yet reach a head.  Any mix of first-state entries (predecessor,
// its chars) and final ones (head, chars before) is a valid state.
__global__ void __launch_bounds__(256) k_rank_round(unsigned long long* __restrict__ X, const uint32_t* __restrict__ act,
                             const uint32_t* act_count, uint32_t* __restrict__ act_out,
                             uint32_t* act_out_count) {
  __shared__ uint32_t sc[33];
  const uint32_t na = *act_count;
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  // whole blocks iterate together (block_append needs every thread)
  for (uint64_t j0 = uint64_t(blockIdx.x) * blockDim.x; j0 < na; j0 += stride) {
    const uint64_t j = j0 + threadIdx.x;
    bool keep = false;
    uint32_t s = 0;
    if (j < na) {
      s = act ? act[j] : uint32_t(j);
      const unsigned long long v = reinterpret_cast<volatile unsigned long long*>(X)[s];
      const unsigned long long u = reinterpret_cast<volatile unsigned long long*>(X)[ptr_of(v)];
      if (!is_head_entry(u)) {  // not yet pointing at a head
        const unsigned long long nv = pk(ptr_of(u), pk_o(v) + pk_o(u));
        reinterpret_cast<volatile unsigned long long*>(X)[s] = nv;
        const unsigned long long z = reinterpret_cast<volatile unsigned long long*>(X)[ptr_of(nv)];
        keep = !is_head_entry(z);
      }
    }
    const uint32_t slot = block_append(act_out_count, keep ? 1u : 0u, sc);
    if (keep) act_out[slot] = s;
  }
}

// ---- the line walk
constexpr uint32_t WALK_CAP = 1024;                // segments a line walk follows
constexpr int WALK_REG = 4;                         // later segments a walk keeps in registers
constexpr unsigned long long LINE_WALKED = ~0ull;  // line base of a line k_walk_emit wrote
constexpr uint32_t JOB_NONE = 0xFFFFFFFFu;

// Reserves want bytes of job's output for each lane of a warp (every lane
// calls; a lane with want 0 or job JOB_NONE takes nothing) with one atomic
// per job present in the warp.  The lanes of one job must be consecutive,
// apart from lanes that take nothing (head-pool ids lie in job order).
// Returns the lane's offset in its job's output.
__device__ __forceinline__ unsigned long long warp_reserve(unsigned long long* jout, uint32_t job,
                                                           unsigned long long want) {
  const uint32_t lane = threadIdx.x & 31u;
  unsigned long long inc = want;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xFFFFFFFFu, inc, d);
    if (lane >= uint32_t(d)) inc += v;
  }
  const uint32_t grp = __match_any_sync(0xFFFFFFFFu, job);
  const uint32_t first = uint32_t(__ffs(grp)) - 1u, last = 31u - uint32_t(__clz(grp));
  const unsigned long long before = __shfl_sync(0xFFFFFFFFu, inc - want, first);
  const unsigned long long total = __shfl_sync(0xFFFFFFFFu, inc, last) - before;
  unsigned long long base = 0;
  if (lane == first && job != JOB_NONE && total) base = atomicAdd(jout + job, total);
  base = __shfl_sync(0xFFFFFFFFu, base, first);
  return base + (inc - want - before);
}

// One thread writes one line: whole aligned 4-byte words as they fill, and
// byte by byte the bytes of its first and last words (which it shares with
// the neighbouring lines, or which lie outside the output buffer: the
// buffer may start at any byte).  Positions are addresses.
struct LineOut {
  uintptr_t p;   // next byte of the line
  uintptr_t p0;  // its first byte
  uint32_t acc;  // the bytes of the word at p & ~3 below p
};

// 4 bytes at any alignment from two aligned words (the segment chars'
// allocation ends with slack, so the second word is inside it)
__device__ __forceinline__ uint32_t load4u(const char* src) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(src);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
  const uint32_t sh = 8u * uint32_t(a & 3u);
  return sh ? __funnelshift_r(w[0], w[1], sh) : w[0];
}

// Appends bytes [0, n) of v (n <= 4 - (p & 3)) and stores the word they fill.
__device__ __forceinline__ void line_bytes(LineOut& L, uint32_t v, uint32_t n) {
  const uint32_t fill = uint32_t(L.p & 3u);
  const uintptr_t wpos = L.p - fill;
  L.acc |= (n == 4 ? v : (v & ((1u << (8 * n)) - 1u))) << (8 * fill);
  L.p += n;
  if (fill + n == 4) {
    if (wpos >= L.p0) {
      *reinterpret_cast<uint32_t*>(wpos) = L.acc;
    } else {
      for (uint32_t b = uint32_t(L.p0 - wpos); b < 4; ++b) reinterpret_cast<char*>(wpos)[b] = char(L.acc >> (8 * b));
    }
    L.acc = 0;
  }
}

// Appends n bytes from src: up to the destination's next word boundary,
// then whole words from an aligned source stream (one new load per word),
// then the rest.
__device__ __forceinline__ void line_put(LineOut& L, const char* src, uint32_t n) {
  const uint32_t head = min(n, (4u - uint32_t(L.p & 3u)) & 3u);
  if (head) {
    line_bytes(L, load4u(src), head);
    src += head;
    n -= head;
  }
  if (n >= 4) {
    // the destination is word aligned here and the words lie inside the line
    const uintptr_t a = reinterpret_cast<uintptr_t>(src);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
    const uint32_t sh = 8u * uint32_t(a & 3u);
    uint32_t* d = reinterpret_cast<uint32_t*>(L.p);
    const uint32_t nw = n >> 2;
    uint32_t cur = w[0];
    for (uint32_t i = 0; i < nw; ++i) {
      const uint32_t nxt = sh ? w[i + 1] : 0u;
      d[i] = sh ? __funnelshift_r(cur, nxt, sh) : w[i];
      cur = nxt;
    }
    L.p += 4u * nw;
    src += 4u * nw;
    n &= 3u;
  }
  if (n) line_bytes(L, load4u(src), n);
}

// Appends n <= 4 bytes held in v (its low bytes first).
__device__ __forceinline__ void line_put4(LineOut& L, uint32_t v, uint32_t n) {
  const uint32_t take = min(n, 4u - uint32_t(L.p & 3u));
  if (take) line_bytes(L, v, take);
  if (n > take) line_bytes(L, v >> (8 * take), n - take);
}

// The line break, then the bytes of the last word not yet stored.
__device__ __forceinline__ void line_end(LineOut& L) {
  line_bytes(L, uint32_t('\n'), 1);
  const uint32_t fill = uint32_t(L.p & 3u);
  if (fill) {
    const uintptr_t wpos = L.p - fill;
    for (uint32_t b = (wpos >= L.p0 ? 0u : uint32_t(L.p0 - wpos)); b < fill; ++b)
      reinterpret_cast<char*>(wpos)[b] = char(L.acc >> (8 * b));
  }
}

// Every stitched line from its head, one thread per head-pool id: the walk
// follows the line's records for its length (up to WALK_CAP segments after
// the head; the first WALK_REG records stay in registers), the warp
// reserves its lines' bytes, and the walk copies each segment's chars into
// the line (records past the kept ones read again, now mostly in L2).  A line that goes on past WALK_CAP segments is left to the ranking
// path: its head goes to longl.  walked counts the segments of the lines
// written (those with ids below nx), left the lines left.  cap <=
// WALK_CAP (smaller only to test the ranking path).
__global__ void __launch_bounds__(256) k_walk_emit(uint32_t H, const SegRec* __restrict__ seg, uint32_t nx, int k,
                                                   const JobTab* __restrict__ jobs, unsigned long long* __restrict__ jout,
                                                   const char* __restrict__ segchars, char* __restrict__ out,
                                                   uint32_t cap, uint32_t* __restrict__ longl, uint32_t lcap,
                                                   int guard, Counters* ctr) {
  // guard: enqueued before it was known that the tiles are complete
  __shared__ uint32_t skip;
  if (threadIdx.x == 0) skip = guard ? ctr->nbig | ctr->err : 0u;
  __syncthreads();
  if (skip) return;
  __shared__ uint32_t sc[33];
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  uint32_t walked = 0;
  // whole warps iterate together (warp_reserve needs every lane)
  for (uint64_t h0 = uint64_t(blockIdx.x) * blockDim.x; h0 < H; h0 += stride) {
    const uint64_t h = h0 + threadIdx.x;
    SegRec r{0ull, 0u, NONE};
    if (h < H) r = seg[nx + h];
    const bool live = r.len != 0;
    unsigned long long len = live ? uint64_t(k) - 1u + r.len : 0ull;
    uint32_t s = live ? r.next : NONE, hops = 0;
    // the first WALK_REG later segments stay in registers for the copy
    SegRec c[WALK_REG];
#pragma unroll
    for (int q = 0; q < WALK_REG; ++q) {
      c[q] = SegRec{0ull, 1u, NONE};
      if (s < nx && hops < cap) {
        c[q] = seg[s];
        len += c[q].len - 1u;
        s = c[q].next;
        ++hops;
      }
    }
    while (s < nx && hops < cap) {
      const SegRec q = seg[s];
      len += q.len - 1u;
      s = q.next;
      ++hops;
    }
    const bool done = live && s == NONE;
    const uint32_t job = done ? uint32_t(r.off_job >> SEG_OFF_BITS) : JOB_NONE;
    const unsigned long long o = warp_reserve(jout, job, done ? len + 1u : 0ull);
    if (live && !done) {
      const uint32_t i = atomicAdd(&ctr->left, 1u);
      if (i < lcap) longl[i] = uint32_t(h);
      else atomicOr(&ctr->err, ERR_INTERNAL);  // a left line holds more than cap cross ids
    }
    if (done) {
      walked += hops;
      const JobTab& J = jobs[job];
      if (o + len + 1u > J.ocap) {
        atomicOr(&ctr->err, ERR_CAPACITY);
      } else {
        // the kept segments' first words load together (most later
        // segments add no more than 4 chars)
        uint32_t fw[WALK_REG];
#pragma unroll
        for (int q = 0; q < WALK_REG; ++q)
          fw[q] = (uint32_t(q) < hops && c[q].len > 1u) ? load4u(segchars + (c[q].off_job & SEG_OFF_MASK)) : 0u;
        const uintptr_t a = reinterpret_cast<uintptr_t>(out + J.obase + o);
        LineOut L{a, a, 0u};
        line_put(L, segchars + (r.off_job & SEG_OFF_MASK), uint32_t(k) - 1u + r.len);
#pragma unroll
        for (int q = 0; q < WALK_REG; ++q) {
          if (uint32_t(q) < hops) {
            const uint32_t n = c[q].len - 1u;
            if (n <= 4u) line_put4(L, fw[q], n);
            else line_put(L, segchars + (c[q].off_job & SEG_OFF_MASK), n);
          }
        }
        uint32_t t = c[WALK_REG - 1].next;
        for (uint32_t q = WALK_REG; q < hops; ++q) {
          const SegRec g = seg[t];
          line_put(L, segchars + (g.off_job & SEG_OFF_MASK), g.len - 1u);
          t = g.next;
        }
        line_end(L);
      }
    }
  }
  uint32_t tot;
  block_excl_scan(walked, sc, &tot);
  if (threadIdx.x == 0 && tot) atomicAdd(&ctr->walked, tot);
}

// The ranking's first state from the segment records (when the walk left
// lines or cycles, and for HEC): a line's first segment is a head; segment
// x (x < nx) points at its predecessor, with the chars the predecessor adds.
__global__ void __launch_bounds__(256) k_seg_xinit(uint32_t S, const SegRec* __restrict__ seg, uint32_t nx, int k,
                                                   unsigned long long* __restrict__ X) {
  for (uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < S; s += uint64_t(gridDim.x) * blockDim.x) {
    const SegRec r = seg[s];
    if (!r.len) continue;
    if (s >= nx) X[s] = pk(uint32_t(s) | HEAD_BIT, 0);
    if (r.next < nx) X[r.next] = pk(uint32_t(s), seg_w(uint32_t(s), r.len, nx, k));
  }
}

__global__ void k_set_u32(uint32_t* p, uint32_t v) { *p = v; }

// Line length of each chain, stored at its head (every live chain has one
// tail, which writes it; the array is zeroed before).  A line's tail starts
// at an S-only copy (a line's first segment always continues).
__global__ void k_chain_len(uint32_t S, const SegRec* __restrict__ seg, const unsigned long long* __restrict__ X,
                            const uint8_t* __restrict__ oncycle, uint32_t nx, int k, uint32_t* __restrict__ linelen,
                            Counters* ctr) {
  constexpr int PER = 4;  // slots per thread and pass: their loads are in flight together
  const uint64_t span = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t s0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; s0 < S; s0 += span * PER) {
    SegRec r[PER];
    uint8_t cyc[PER];
    unsigned long long v[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const uint64_t s = s0 + uint64_t(q) * span;
      const bool in = s < S;
      r[q] = in ? seg[s] : SegRec{0ull, 0u, 0u};
      cyc[q] = in ? oncycle[s] : uint8_t(1);
      v[q] = in ? X[s] : 0ull;
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      if (!r[q].len || r[q].next != NONE || cyc[q]) continue;
      const uint32_t h = ptr_of(v[q]);
      const uint32_t s = uint32_t(s0 + uint64_t(q) * span);
      if (h < nx || h >= S) {
        atomicOr(&ctr->err, ERR_INTERNAL);
        continue;
      }
      linelen[h - nx] = pk_o(v[q]) + seg_w(s, r[q].len, nx, k) + 1u;
    }
  }
}

// Each line's base in the output, reserved after the job's lines so far:
// over the heads in list (the lines the walk left), or over all head-pool
// ids (list == nullptr, after HEC ranking: one reservation per job and
// warp).  A head without a length keeps LINE_WALKED, so no segment copies
// into it.
__global__ void __launch_bounds__(256) k_line_reserve(uint32_t n, const uint32_t* __restrict__ list,
                                                      const SegRec* __restrict__ heads,
                                                      const JobTab* __restrict__ jobs,
                                                      unsigned long long* __restrict__ jout,
                                                      const uint32_t* __restrict__ hlen,
                                                      unsigned long long* __restrict__ lbase, Counters* ctr) {
  const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
  // whole warps iterate together (warp_reserve needs every lane)
  for (uint64_t i0 = uint64_t(blockIdx.x) * blockDim.x; i0 < n; i0 += stride) {
    const uint64_t i = i0 + threadIdx.x;
    uint32_t h = 0, job = JOB_NONE, want = 0;
    if (i < n) {
      h = list ? list[i] : uint32_t(i);
      const SegRec r = heads[h];
      want = r.len ? hlen[h] : 0u;
      if (want) job = uint32_t(r.off_job >> SEG_OFF_BITS);
    }
    // a list's heads come in any job order: one atomic each
    const unsigned long long o = list ? (want ? atomicAdd(jout + job, (unsigned long long)want) : 0ull)
                                      : warp_reserve(jout, job, want);
    if (want) {
      const JobTab& J = jobs[job];
      if (o + want > J.ocap) atomicOr(&ctr->err, ERR_CAPACITY);
      else lbase[h] = J.obase + o;
    }
  }
}

// Copy each segment's chars into its line.  A warp takes 4 x 32 consecutive
// segments: each lane resolves four segments' source, destination and
// length (their records and ranking entries, then their heads' line bases;
// all four gathers in flight together), then groups of 8 lanes copy the
// segments word by word.
__global__ void __launch_bounds__(256) k_seg_copy(
    uint32_t S, const SegRec* __restrict__ seg, const unsigned long long* __restrict__ X,
    const uint8_t* __restrict__ oncycle, uint32_t nx, const unsigned long long* __restrict__ lbase,
    const char* __restrict__ segchars, char* __restrict__ out, int k) {
  constexpr int PER = 4;
  const int lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  for (uint64_t base = uint64_t(warp) * 32u * PER; base < S; base += uint64_t(nwarps) * 32u * PER) {
    uint64_t dst[PER], src[PER];
    uint32_t nb[PER], last[PER], hd[PER];
    unsigned long long off[PER];
    bool live[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const uint64_t s = base + uint64_t(q) * 32u + uint32_t(lane);
      live[q] = s < S;
      dst[q] = src[q] = 0;
      nb[q] = last[q] = 0;
      hd[q] = 0;
      off[q] = 0;
      if (live[q]) {
        const SegRec r = seg[s];
        const uint8_t cyc = oncycle[s];
        const unsigned long long v = X[s];
        // (a pointer short of a head is flagged by k_chain_len)
        live[q] = r.len != 0 && !cyc && ptr_of(v) >= nx && ptr_of(v) < S;
        if (live[q]) {
          hd[q] = ptr_of(v) - nx;
          off[q] = pk_o(v);
          src[q] = r.off_job & SEG_OFF_MASK;
          nb[q] = seg_w(uint32_t(s), r.len, nx, k);
          last[q] = r.next == NONE;
        }
      }
    }
    // (segments of lines the walk wrote copy nothing)
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      if (!live[q]) continue;
      const unsigned long long lb = lbase[hd[q]];
      if (lb == LINE_WALKED) {
        nb[q] = 0;
        last[q] = 0;
      } else {
        dst[q] = lb + off[q];
      }
    }
    // groups of 8 lanes: group g copies, one after another, the segments
    // resolved by its own 8 lanes.  Each lane of the group stores aligned
    // 4-byte words of the destination, funnel-shifted from the two aligned
    // source words that hold them; the up to 3 bytes before the first
    // aligned word and after the last one go byte by byte.  Source words
    // are read only where they hold a byte of the segment, so they stay in
    // the segment chars' allocation.
    const uint32_t gl = uint32_t(lane) & 7u;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
#pragma unroll 1
      for (int i = 0; i < 8; ++i) {
        const uint64_t d = __shfl_sync(0xFFFFFFFFu, dst[q], i, 8);
        const uint64_t c = __shfl_sync(0xFFFFFFFFu, src[q], i, 8);
        const uint32_t m = __shfl_sync(0xFFFFFFFFu, nb[q], i, 8);
        const uint32_t e = __shfl_sync(0xFFFFFFFFu, last[q], i, 8);
        // bytes before the first aligned word of the destination (the output
        // buffer itself may start at any byte)
        const uint32_t hb = min((4u - uint32_t(reinterpret_cast<uintptr_t>(out + d) & 3u)) & 3u, m);
        const uint32_t nbody = (m - hb) >> 2;
        const uint32_t tb = (m - hb) & 3u;
        const char* sp = segchars + c + hb;
        char* dp = out + d + hb;
        const uint32_t sh = 8u * uint32_t(reinterpret_cast<uintptr_t>(sp) & 3u);
        const uint32_t* sw = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(sp) & ~uintptr_t(3));
        for (uint32_t wi = gl; wi < nbody; wi += 8) {
          const uint32_t w0 = sw[wi];
          const uint32_t v = sh ? __funnelshift_r(w0, sw[wi + 1], sh) : w0;
          reinterpret_cast<uint32_t*>(dp)[wi] = v;
        }
        if (gl < hb) out[d + gl] = segchars[c + gl];
        if (gl >= 4 && gl - 4 < tb) dp[4 * nbody + (gl - 4)] = sp[4 * nbody + (gl - 4)];
        if (gl == 7 && e) out[d + m] = '\n';
      }
    }
  }
}

__global__ void k_mark_cycle(const uint32_t* __restrict__ act, const uint32_t* act_count,
                             uint8_t* __restrict__ oncycle) {
  const uint32_t na = *act_count;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < na; j += gridDim.x * blockDim.x)
    oncycle[act[j]] = 1;
}

// Cycles of segments (rare; they hold only segments that start at S-only
// copies): one thread spells each cycle starting at its smallest k-mer.  The
// cycle's distinct k-mers are the last chars of each segment after its first
// k-mer, read circularly.
template <int NW>
__global__ void k_seg_cycles(Counters* ctr, uint32_t S, const uint32_t* __restrict__ act, uint32_t na,
                             uint8_t* __restrict__ oncycle, const SegRec* __restrict__ seg,
                             const JobTab* __restrict__ jobs, unsigned long long* __restrict__ jout,
                             const char* __restrict__ segchars, char* __restrict__ out, int k) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  for (uint32_t j = 0; j < na; ++j) {
    const uint32_t s0 = act[j];
    if (oncycle[s0] != 1) continue;
    // total distinct k-mers N and the circular char accessor
    uint64_t N = 0;
    uint32_t s = s0, steps = 0;
    do {
      N += seg[s].len - 1u;
      oncycle[s] = 2;
      s = seg[s].next;
    } while (s != s0 && s < S && ++steps <= S);
    if (s != s0 || N == 0) {
      atomicOr(&ctr->err, ERR_INTERNAL);
      continue;
    }
    // char q of the circular string: segment chars after the first k
    // (q < N and the cycle was walked above, so the loop ends within it)
    auto at = [&](uint64_t q) -> char {
      uint32_t t = s0;
      for (uint32_t guard = 0; guard <= S; ++guard) {
        const SegRec r = seg[t];
        const uint64_t m = r.len - 1u;
        if (q < m) return segchars[(r.off_job & SEG_OFF_MASK) + q];
        q -= m;
        t = r.next;
      }
      return 'A';
    };
    // the k-mer ending at circular position q; find the smallest
    auto kmer_at = [&](uint64_t q) {
      Key<NW> x;
#pragma unroll
      for (int w = 0; w < NW; ++w) x.w[w] = 0;
      for (int c = 0; c < k; ++c) {
        const char ch = at((q + N * 64 - (k - 1) + c) % N);
        const uint64_t code = (ch == 'C') ? 1 : (ch == 'G') ? 2 : (ch == 'T') ? 3 : 0;
        if (c < 32) x.w[0] |= code << (2 * c);
        else if (NW == 2) x.w[NW - 1] |= code << (2 * (c - 32));
      }
      return x;
    };
    uint64_t best = 0;
    Key<NW> bk = kmer_at(0);
    for (uint64_t q = 1; q < N; ++q) {
      const Key<NW> x = kmer_at(q);
      if (key_lt(x, bk)) { bk = x; best = q; }
    }
    const uint64_t len = uint64_t(k) + N;  // k + (N - 1) chars + '\n'
    const uint32_t job = uint32_t(seg[s0].off_job >> SEG_OFF_BITS);
    const unsigned long long o = atomicAdd(jout + job, len);
    if (o + len > jobs[job].ocap) {
      atomicOr(&ctr->err, ERR_CAPACITY);
      return;
    }
    char* dst = out + jobs[job].obase + o;
    for (uint64_t t = 0; t + 1 < len; ++t) dst[t] = at((best + N * 64 - (k - 1) + t) % N);
    dst[len - 1] = '\n';
    atomicAdd(&ctr->cycles, 1ull);
  }
}

// ===================================================== HEC contraction
//
// Heavy-edge coarsening over a set of paths (and rare cycles), restating the
// reference's round loop (coarsen_de_bruijn_full_cycle, coarseners.h:437-485):
// every node with a predecessor wants to merge with it, a head wants its
// successor, an isolated node is a finished chain (coarsen_HEC,
// heuristics.h:224-245); two compare-and-swaps pair a node with its choice or
// let it join the choice's aggregate (parallel_map_construct,
// heuristics.h:106-203, with bounded retries and a singleton fallback instead
// of unbounded spins); aggregates become the next level's nodes
// (coarsen_de_bruijn_graph, coarseners.h:68-92).  Members are ordered by
// walking from the aggregate's first member (instead of the O(m^2) sort of
// transpose_and_sort, coarseners.h:182-235) and their offsets are composed
// top-down (instead of copying member lists, compact_graph.h:55-112).
// Levels live in one node pool; level r occupies [lb[r], lb[r] + ln[r]).
// All rounds run in one cooperative kernel (k_hec_all) whose blocks meet at a
// barrier between the steps and stop at the first empty level: paths of
// canonical k-mers are short, so a few of the rounds a list could need are
// enough.  (2M k-mers, k = 63: 0.40 ms for the call; six launches per round for
// the 50 rounds of the bound took 1.78, most of them on empty levels.)
constexpr uint32_t HV_UNSET = 0xFFFFFFFFu, HV_LOCK = 0xFFFFFFFEu, HV_FIN = 0xFFFFFFFDu, HV_CYC = 0xFFFFFFFCu;

struct HecPool {
  uint32_t *prv, *nxt, *wt, *hn, *vc, *agg, *loc, *first0;
  uint32_t* lb;  // [R+1] level base
  uint32_t* ln;  // [R+1] level size, then the blocks' meeting place (two words)
  uint32_t cap;
  Counters* ctr;
};

__global__ void k_hec_level0(HecPool h, const uint32_t* __restrict__ prev, const uint32_t* __restrict__ next,
                             const uint32_t* __restrict__ w, uint64_t n) {
  const uint64_t N = n;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    h.lb[0] = 0;
    h.ln[0] = uint32_t(N);
  }
  for (uint64_t u = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; u < N; u += uint64_t(gridDim.x) * blockDim.x) {
    h.prv[u] = prev[u];
    h.nxt[u] = next[u];
    h.wt[u] = w ? w[u] : 1u;
    h.first0[u] = uint32_t(u);
  }
}

// Level 0 from the fused path's segments: next from the records, prev from
// the ranking's first state built from them (k_seg_xinit; ids [0, nx) only:
// a line's first segment has none), weights from the lengths.  Unused head-pool ids have
// length 0 and stay isolated.
__global__ void k_hec_level0_seg(HecPool h, const SegRec* __restrict__ seg, const unsigned long long* __restrict__ X0,
                                 uint64_t S, uint32_t nx, int k) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    h.lb[0] = 0;
    h.ln[0] = uint32_t(S);
  }
  for (uint64_t u = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; u < S; u += uint64_t(gridDim.x) * blockDim.x) {
    const SegRec r = seg[u];
    uint32_t pv = NONE, nx_ = NONE, w = 0;
    if (r.len) {
      pv = (u < nx) ? ptr_of(X0[u]) : NONE;
      nx_ = r.next;
      w = seg_w(uint32_t(u), r.len, nx, k);
    }
    h.prv[u] = pv;
    h.nxt[u] = nx_;
    h.wt[u] = w;
    h.first0[u] = uint32_t(u);
  }
}

// Values other blocks wrote in an earlier step are read past L1.
__device__ __forceinline__ uint32_t hec_ld(const uint32_t* p) { return __ldcg(p); }

// choice (hn) per node; isolated nodes are finished chains; a node whose
// predecessor is itself is a one-node cycle
__device__ __forceinline__ void hec_prep(const HecPool& h, uint32_t u, uint32_t pv, uint32_t nx) {
  const uint32_t c = (pv != NONE) ? pv : nx;
  const bool cyc = pv == u;
  h.hn[u] = cyc ? NONE : c;
  h.vc[u] = cyc ? HV_CYC : (c == NONE) ? HV_FIN : HV_UNSET;
}

// One pass of the two-CAS pairing.  A label is the pool index of the
// aggregate's root.  Pass 1 gives up after 10 tries when u > v (the
// reference's deadlock break, heuristics.h:142-146); pass 2 retries the rest
// a bounded number of times and then leaves u a singleton aggregate.
__device__ __forceinline__ void hec_match(const HecPool& h, uint32_t u, uint32_t v, int pass) {
  bool done = false;
  const int limit = (pass == 1) ? 64 : 256;
  for (int it = 0; it < limit && !done; ++it) {
    if (atomicCAS(h.vc + u, HV_UNSET, HV_LOCK) == HV_UNSET) {
      if (atomicCAS(h.vc + v, HV_UNSET, HV_LOCK) == HV_UNSET) {
        atomicExch(h.vc + v, u);
        atomicExch(h.vc + u, u);
        done = true;
      } else {
        const uint32_t lv = atomicAdd(h.vc + v, 0u);
        if (lv < HV_CYC) {  // v already labelled: join its aggregate
          atomicExch(h.vc + u, lv);
          done = true;
        } else {
          atomicExch(h.vc + u, HV_UNSET);  // release and retry
        }
      }
    } else {
      done = true;  // u is labelled (or being labelled) by a neighbour
    }
    if (pass == 1 && it > 10 && u > v) break;
  }
  if (pass == 2 && !done) atomicCAS(h.vc + u, HV_UNSET, u);  // singleton
}

// The first member of each aggregate (predecessor outside it) walks its
// members along next: local offsets, total weight, coarse neighbours, and the
// coarse node's choice.  (ap: the aggregate of u's predecessor)
__device__ __forceinline__ void hec_order(const HecPool& h, uint32_t u, uint32_t A, uint32_t ap, uint32_t N) {
  uint32_t off = 0, m = u, nx = NONE;
  for (uint32_t guard = 0; guard < N; ++guard) {
    h.loc[m] = off;
    off += hec_ld(h.wt + m);
    nx = hec_ld(h.nxt + m);
    if (nx == NONE || hec_ld(h.agg + nx) != A) break;
    m = nx;
  }
  const uint32_t an = (nx == NONE) ? NONE : hec_ld(h.agg + nx);
  h.wt[A] = off;
  h.first0[A] = hec_ld(h.first0 + u);
  h.nxt[A] = an;
  h.prv[A] = ap;
  hec_prep(h, A, ap, an);
}

// Top-down: (head, offset) of every node from its aggregate's, stored in
// (hn, loc).  A finished node is a whole chain headed by its first member; a
// cycle node marks its members with head NONE.
__device__ __forceinline__ void hec_down(const HecPool& h, uint32_t u) {
  const uint32_t c = hec_ld(h.vc + u);
  uint32_t hd = NONE, of = 0;
  if (c == HV_FIN) {
    hd = hec_ld(h.first0 + u);
  } else if (c != HV_CYC) {
    const uint32_t A = hec_ld(h.agg + u);
    hd = (A == NONE || A >= h.cap) ? NONE : hec_ld(h.hn + A);
    of = (hd == NONE) ? 0 : hec_ld(h.loc + A) + hec_ld(h.loc + u);
  }
  h.hn[u] = hd;
  h.loc[u] = of;
}

// All blocks of a cooperative grid meet here (gen counts the meetings): the
// last one to arrive (bar[0]) lets the others go (bar[1]).  A wait that runs
// out, or meets another block's, sets the error flag and returns false; the
// kernel then ends.
__device__ __forceinline__ bool grid_meet(uint32_t* bar, uint32_t& gen, uint32_t* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ++gen;
    int ok = 1;
    __threadfence();
    if (atomicAdd(bar, 1u) + 1u == gen * gridDim.x) {
      atomicExch(bar + 1, gen);
    } else {
      uint32_t p = 0;
      while (*reinterpret_cast<volatile uint32_t*>(bar + 1) < gen) {
        __nanosleep(20);
        if (++p >= (1u << 22) || ((p & 1023u) == 0 && (*reinterpret_cast<volatile uint32_t*>(err) & ERR_INTERNAL))) {
          atomicOr(err, ERR_INTERNAL | ERR_TIMEOUT);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// One round over level r (base b, N nodes; level 0 and coarse nodes have
// their choices): threads t0, t0 + span, ... of all blocks or of one, meet()
// between the steps.  Sets the next level's base, size and choices.
template <class Meet>
__device__ __forceinline__ bool hec_round(const HecPool& h, uint32_t r, uint32_t& b, uint32_t& N, uint32_t t0,
                                          uint32_t span, Meet meet) {
  __shared__ uint32_t sc[33];
  uint32_t* const err = &h.ctr->err;
  for (int pass = 1; pass <= 2; ++pass) {
    for (uint32_t j0 = t0; j0 < N; j0 += 4 * span) {
      uint32_t v[4];
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) v[q] = j0 + q * span < N ? hec_ld(h.hn + b + j0 + q * span) : NONE;
      if (pass == 2) {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
          if (v[q] != NONE && hec_ld(h.vc + b + j0 + q * span) != HV_UNSET) v[q] = NONE;
      }
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        if (v[q] != NONE) hec_match(h, b + j0 + q * span, v[q], pass);
    }
    if (!meet()) return false;
  }
  // roots (label == self) take the next level's pool slots; the root's hn
  // holds its new index.  A coarse node no first member reaches (hec_order)
  // is a whole cycle collapsed into one.
  // (whole blocks iterate together: one append per block and pass)
  for (uint32_t j0 = t0 - threadIdx.x; j0 < N; j0 += 4 * span) {
    uint32_t root = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t j = j0 + threadIdx.x + q * span;
      if (j < N && hec_ld(h.vc + b + j) == b + j) root |= 1u << q;
    }
    uint32_t a = b + N + block_append(h.ln + r + 1, uint32_t(__popc(root)), sc);
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      if (!((root >> q) & 1u)) continue;
      if (a >= h.cap) {
        atomicOr(err, ERR_CAPACITY);
      } else {
        h.hn[b + j0 + threadIdx.x + q * span] = a;
        h.prv[a] = NONE;
        h.nxt[a] = NONE;
        h.wt[a] = 0;
        h.first0[a] = NONE;
        h.hn[a] = NONE;
        h.vc[a] = HV_CYC;
      }
      ++a;
    }
  }
  if (!meet()) return false;
  for (uint32_t j0 = t0; j0 < N; j0 += 4 * span) {
    uint32_t c[4], a[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) c[q] = j0 + q * span < N ? hec_ld(h.vc + b + j0 + q * span) : NONE;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) a[q] = c[q] < HV_CYC ? hec_ld(h.hn + c[q]) : NONE;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q)
      if (j0 + q * span < N) h.agg[b + j0 + q * span] = a[q];
  }
  if (!meet()) return false;
  for (uint32_t j0 = t0; j0 < N; j0 += 4 * span) {
    // which nodes are first members, then their walks
    uint32_t A[4], pv[4], ap[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t u = b + j0 + q * span;
      A[q] = j0 + q * span < N ? hec_ld(h.agg + u) : NONE;
      pv[q] = j0 + q * span < N ? hec_ld(h.prv + u) : NONE;
    }
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) ap[q] = (A[q] != NONE && pv[q] != NONE) ? hec_ld(h.agg + pv[q]) : NONE;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q)
      if (A[q] != NONE && A[q] < h.cap && ap[q] != A[q]) hec_order(h, b + j0 + q * span, A[q], ap[q], N);
  }
  if (t0 == 0) h.lb[r + 1] = b + N;
  if (!meet()) return false;
  b += N;
  N = min(hec_ld(h.ln + r + 1), h.cap - min(h.cap, b));
  return true;
}

// The rounds (level 0 is set), at most R of them, then the way down and the
// level-0 results in the (pointer | HEAD_BIT, offset) form of the ranking.
// Levels of at most HEC_SOLO nodes are worked by one block, up and down, while
// the others wait at one meeting.  Lists still open after R rounds set
// ERR_TIMEOUT.
constexpr uint32_t HEC_THREADS = 1024, HEC_SOLO = 4096;
__global__ void __launch_bounds__(HEC_THREADS, 2) k_hec_all(HecPool h, uint32_t R, unsigned long long* __restrict__ X,
                                                         uint8_t* __restrict__ oncycle) {
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, span = gridDim.x * blockDim.x;
  uint32_t* const bar = h.ln + R + 1;
  uint32_t* const err = &h.ctr->err;
  uint32_t gen = 0, r = 0, b = 0, N = hec_ld(h.ln);
  const uint32_t N0 = N;
  auto all = [&] { return grid_meet(bar, gen, err); };
  auto own = [] {
    __syncthreads();
    return true;
  };
  for (uint32_t u = t0; u < N; u += span) hec_prep(h, u, hec_ld(h.prv + u), hec_ld(h.nxt + u));
  if (!all()) return;
  for (; r < R && N > HEC_SOLO; ++r)
    if (!hec_round(h, r, b, N, t0, span, all)) return;
  const uint32_t rs = r;
  if (N) {
    if (blockIdx.x == 0) {
      for (; r < R && N; ++r) hec_round(h, r, b, N, threadIdx.x, HEC_THREADS, own);
      if (N) {
        if (threadIdx.x == 0) atomicOr(err, ERR_TIMEOUT);
      } else {
        while (r-- > rs) {
          b = r ? hec_ld(h.lb + r) : 0u;
          N = hec_ld(h.ln + r);
          for (uint32_t j = threadIdx.x; j < N; j += HEC_THREADS) hec_down(h, b + j);
          __syncthreads();
        }
      }
    }
    if (!all()) return;
    if (hec_ld(err) & ERR_TIMEOUT) return;  // the rounds ran out
  }
  for (r = rs; r-- > 0;) {
    b = r ? hec_ld(h.lb + r) : 0u;
    N = hec_ld(h.ln + r);
    for (uint32_t j = t0; j < N; j += span) hec_down(h, b + j);
    if (!all()) return;
  }
  for (uint32_t s = t0; s < N0; s += span) {
    const uint32_t hd = hec_ld(h.hn + s);
    if (hd == NONE) {
      X[s] = pk(s, 0);
      if (oncycle) oncycle[s] = 1;
    } else {
      X[s] = pk(hd == s ? (hd | HEAD_BIT) : hd, hec_ld(h.loc + s));
    }
  }
}

__global__ void k_cycle_list(const uint8_t* __restrict__ oncycle, uint64_t n,
                             uint32_t* __restrict__ act, uint32_t* __restrict__ cnt) {
  const uint64_t N = n;
  for (uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; s < N; s += uint64_t(gridDim.x) * blockDim.x)
    if (oncycle[s]) act[atomicAdd(cnt, 1u)] = uint32_t(s);
}

// ======================================================= phase-API helpers

// Contraction by ranking from the predecessors: every vertex first walks up to
// RANK_STEPS of them, and one that meets a head on the way is done.  K-mers of a
// canonical set keep each neighbour with probability about a half, so lines
// are short and few vertices are left (1 in 2^RANK_STEPS), whose pointer and
// distance go to X and whose ids go to the list that k_rank_rest works off.
// The walk is a chain of dependent 4-byte gathers from the predecessors,
// which L2 holds (65 MB at 16M k-mers), so a thread walks four vertices at a
// time; pointer jumping from the first state wrote and gathered (pointer,
// distance) pairs, twice the bytes and past L2.  16.3M k-mers: 134 us, and 29 for
// the rest, where the first state, the rounds and the split of the pairs took
// 92, 323 and 50.
// A warp whose vertices are nearly all left halfway stops there (long lines).
// head[v] == NONE: not ranked yet.
constexpr uint32_t RANK_STEPS = 8;
__global__ void __launch_bounds__(256) k_rank_walk(const uint32_t* __restrict__ pred, uint64_t n,
                                                   uint32_t* __restrict__ head, uint32_t* __restrict__ rank,
                                                   unsigned long long* __restrict__ X, uint32_t* __restrict__ act,
                                                   uint32_t* act_count) {
  __shared__ uint32_t sc[33];
  // whole blocks iterate together (block_append needs every thread)
  for (uint64_t s0 = uint64_t(blockIdx.x) * 1024u; s0 < n; s0 += uint64_t(gridDim.x) * 1024u) {
    uint32_t p[4], h[4], d[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint64_t v = s0 + q * 256u + threadIdx.x;
      h[q] = uint32_t(v);
      d[q] = 0;
      p[q] = v < n ? pred[v] : NONE;
    }
    auto walk = [&](uint32_t steps) {
#pragma unroll 1
      for (uint32_t i = 0; i < steps; ++i) {
        if ((p[0] & p[1] & p[2] & p[3]) == NONE) break;
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
          if (p[q] != NONE) {
            h[q] = p[q];
            ++d[q];
            p[q] = pred[h[q]];
          }
        }
      }
    };
    walk(RANK_STEPS / 2);
    // (long lines: the rounds get there sooner)
    uint32_t left = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) left += uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, p[q] != NONE)));
    if (left <= 112) walk(RANK_STEPS - RANK_STEPS / 2);
    uint32_t open = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint64_t v = s0 + q * 256u + threadIdx.x;
      if (v >= n) continue;
      if (p[q] == NONE) {
        head[v] = h[q];
        rank[v] = d[q];
      } else {
        head[v] = NONE;
        X[v] = pk(h[q], d[q]);
        ++open;
      }
    }
    // (most blocks have some open vertex, all of them few)
    uint32_t slot = block_append(act_count, open, sc);
    if (open) {
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q)
        if (p[q] != NONE) act[slot++] = uint32_t(s0 + q * 256u + threadIdx.x);
    }
  }
}

// The vertices left by k_rank_walk: rounds of pointer jumping over ever
// shorter lists, in one cooperative kernel whose blocks meet after each round
// and that ends at the first empty list (a launch per round ran all
// 2 + log2(n) of them, 2.4 us each when empty).  A vertex whose pointer is
// ranked takes its head; one whose pointer is not jumps to where that one
// points.  rank is stored before head, so whoever sees the head sees the rank.
// Lists open after the last round hold cycles (and what leads into one): count
// in cnt[rounds].  More than `most` vertices left by the walk: nothing is done.
__global__ void __launch_bounds__(1024, 2) k_rank_rest(unsigned long long* X, uint32_t* head, uint32_t* rank,
                                                       uint32_t* list0, uint32_t* list1, uint32_t* cnt,
                                                       uint32_t rounds, uint32_t most, uint32_t* bar, uint32_t* err) {
  __shared__ uint32_t sc[33];
  uint32_t gen = 0;
  volatile unsigned long long* const vX = X;
  volatile uint32_t *const vh = head, *const vr = rank;
  for (uint32_t r = 0; r < rounds; ++r) {
    const uint32_t na = *reinterpret_cast<volatile uint32_t*>(cnt + r);
    if (na == 0 || na > most) return;
    volatile uint32_t* const in = (r & 1) ? list1 : list0;
    uint32_t* const out = (r & 1) ? list0 : list1;
    // whole blocks iterate together (block_append needs every thread)
    for (uint64_t j0 = uint64_t(blockIdx.x) * blockDim.x; j0 < na; j0 += uint64_t(gridDim.x) * blockDim.x) {
      const uint64_t j = j0 + threadIdx.x;
      bool keep = false;
      uint32_t s = 0;
      if (j < na) {
        s = in[j];
        const unsigned long long v = vX[s];
        const uint32_t p = pk_p(v), hp = vh[p];
        if (hp != NONE) {
          __threadfence();
          vr[s] = vr[p] + pk_o(v);
          __threadfence();
          vh[s] = hp;
        } else {
          const unsigned long long u = vX[p];
          vX[s] = pk(pk_p(u), pk_o(v) + pk_o(u));
          keep = true;
        }
      }
      const uint32_t slot = block_append(cnt + r + 1, keep ? 1u : 0u, sc);
      if (keep) out[slot] = s;
    }
    if (!grid_meet(bar, gen, err)) return;
  }
  const uint32_t na = *reinterpret_cast<volatile uint32_t*>(cnt + rounds);
  volatile uint32_t* const in = (rounds & 1) ? list1 : list0;
  for (uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < na; j += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t s = in[j];
    const unsigned long long v = vX[s];
    rank[s] = pk_o(v);
    head[s] = pk_p(v);
  }
}

// Long lines (the k-mers of one strand): most vertices are left after the walk, and a
// round of k_rank_rest gathers head and entry of each pointer.  With more than
// three quarters of them left (lines of 32 and more) every vertex gets its entry, in
// k_rank_round's form, and the rounds run as launches of that, two gathers of
// entries each that make up for two to three rounds of doubling, over all ids first.
// The host sees the count at the wait it has anyway; below RANK_DENSE vertices
// that wait and the launches are longer than what they save (100k: 200 us against 155).
// 8M k-mers, shuffled, lines of 20, 50, 1000 and 1M k-mers, the whole call: 434, 623, 912,
// 1821 us; with k_rank_rest alone 433, 667, 1277, 2190; with rounds from the first state
// alone 492, 593, 924, 1968.
constexpr uint64_t RANK_DENSE = 1ull << 19;
__global__ void k_rank_fill(const uint32_t* __restrict__ head, const uint32_t* __restrict__ rank, uint64_t n,
                            unsigned long long* __restrict__ X, uint32_t* count) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *count = uint32_t(n);  // the first round takes them all, in order
  for (uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v < n; v += uint64_t(gridDim.x) * blockDim.x)
    if (head[v] != NONE) X[v] = pk(head[v] == uint32_t(v) ? head[v] | HEAD_BIT : head[v], rank[v]);
}

__global__ void k_head_rank(const unsigned long long* __restrict__ X, uint64_t n,
                            uint32_t* __restrict__ head, uint32_t* __restrict__ rank) {
  for (uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v < n;
       v += uint64_t(gridDim.x) * blockDim.x) {
    const unsigned long long x = X[v];
    head[v] = ptr_of(x);
    rank[v] = pk_o(x);
  }
}

// Cycle vertices of the global graph (rare): one thread ranks each cycle from
// its smallest key.
template <int NW>
__global__ void k_vertex_cycles(const uint32_t* __restrict__ act, uint32_t na,
                                const uint32_t* __restrict__ succ, const uint64_t* __restrict__ keys,
                                uint64_t n_all, uint32_t* __restrict__ head, uint32_t* __restrict__ rank,
                                uint8_t* __restrict__ seen, unsigned long long* ncyc) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  for (uint32_t j = 0; j < na; ++j) {
    const uint32_t v0 = act[j];
    if (seen[v0]) continue;
    uint32_t best = v0;
    Key<NW> bk = ld_key<NW>(keys, v0);
    uint64_t steps = 0;
    uint32_t x = succ[v0];
    for (; x != v0 && x != NONE && steps < n_all; x = succ[x], ++steps) {
      const Key<NW> xk = ld_key<NW>(keys, x);
      if (key_lt(xk, bk)) { bk = xk; best = x; }
    }
    if (x != v0) continue;  // not a cycle: left as ranked
    uint32_t r = 0;
    x = best;
    steps = 0;
    do {
      head[x] = best;
      rank[x] = r++;
      seen[x] = 1;
      x = succ[x];
    } while (x != best && x != NONE && ++steps < n_all);
    ++*ncyc;
  }
}

// Later members per head, four vertices per thread in flight.  The heads (half
// of a canonical set's k-mers) leave themselves out.  16.3M k-mers: 70 -> 64 us
// (k_count_heads, four in flight likewise: 36 -> 24).
__global__ void __launch_bounds__(256) k_count_members(const uint32_t* __restrict__ head, uint64_t n,
                                                       uint32_t* __restrict__ cnt) {
  const uint64_t span = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t v0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v0 < n; v0 += 4 * span) {
    uint32_t h[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) h[q] = v0 + q * span < n ? head[v0 + q * span] : uint32_t(v0 + q * span);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (h[q] != uint32_t(v0 + q * span)) atomicAdd(cnt + h[q], 1u);
  }
}

// Unitig lines from (head, rank), ordered by head id (write_intra_bucket_
// outputs, compact.h:187-208).  A line is its head's k-mer and the last char
// of each later member.  The later members counted per head (k_count_members) give,
// by one look-back pass, each line's first position among all members
// (k_emit_scan); each later member stores its char at its position, one byte
// into an n-byte array that L2 holds (k_emit_chars); then blocks take heads in
// id order and store their lines as one stream, spelled in shared memory
// (k_emit_lines).  17M k-mers, k = 31: 540 us in all; every member storing its
// char straight into the output (290 MB, a random byte each) took 950 of 1600.
constexpr uint32_t EMIT_TILE = 1024;  // vertices per block of k_emit_scan and k_emit_lines

// heads among [0, n)
__global__ void __launch_bounds__(256) k_count_heads(const uint32_t* __restrict__ head, uint64_t n,
                                                     unsigned long long* total) {
  uint32_t acc = 0;
  const uint64_t span = uint64_t(gridDim.x) * blockDim.x;
  for (uint64_t v0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v0 < n; v0 += 4 * span) {
    uint32_t h[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) h[q] = v0 + q * span < n ? head[v0 + q * span] : ~uint32_t(v0 + q * span);
#pragma unroll
    for (int q = 0; q < 4; ++q) acc += h[q] == uint32_t(v0 + q * span);
  }
  acc = __reduce_add_sync(0xFFFFFFFFu, acc);
  if ((threadIdx.x & 31u) == 0 && acc) atomicAdd(total, (unsigned long long)acc);
}

// Four consecutive words at p[v], v a multiple of four; those from n on are
// `out`.  One load where p is aligned for it (a caller's array may not be).
__device__ __forceinline__ uint4 ld4(const uint32_t* __restrict__ p, uint64_t v, uint64_t n, uint32_t out) {
  if (v + 4 <= n && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) return *reinterpret_cast<const uint4*>(p + v);
  return make_uint4(v < n ? p[v] : out, v + 1 < n ? p[v + 1] : out, v + 2 < n ? p[v + 2] : out,
                    v + 3 < n ? p[v + 3] : out);
}

// voff[v]: members of the heads before v.  base[b]: lines (high half) and
// members (low half) before block b's vertices; base[blocks] the totals.
// Loads of four words and stores likewise: 87 -> 70 us at 16.3M k-mers.
// Lines and members share a look-back word, 31 bits each; WIDE (from EMIT_WIDE
// vertices on): members in st, lines in the words behind it.
constexpr uint64_t EMIT_WIDE = 0x7FFFFFFFull;
template <bool WIDE>
__global__ void __launch_bounds__(256) k_emit_scan(const uint32_t* __restrict__ head, const uint32_t* __restrict__ cnt,
                                                   uint64_t n, uint32_t* __restrict__ voff,
                                                   unsigned long long* __restrict__ base, unsigned long long* st,
                                                   uint32_t* ctl) {
  __shared__ unsigned long long scan[33], s_base, s_lines;
  __shared__ uint32_t s_b, lscan[33];
  if (threadIdx.x == 0) s_b = atomicAdd(ctl, 1u);
  __syncthreads();
  const uint32_t b = s_b;
  const uint64_t v0 = uint64_t(b) * EMIT_TILE + 4u * threadIdx.x;
  // (past the last vertex: no vertex's own id)
  const uint4 h = ld4(head, v0, n, ~uint32_t(v0)), m = ld4(cnt, v0, n, 0u);
  const uint32_t hd[4] = {h.x, h.y, h.z, h.w}, mem[4] = {m.x, m.y, m.z, m.w};
  uint32_t c[4], lines = 0;
  unsigned long long sum = 0;
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    c[q] = hd[q] == uint32_t(v0 + q) ? mem[q] + 1u : 0u;
    if (WIDE) {
      sum += c[q];
      lines += c[q] ? 1u : 0u;
    } else {
      sum += c[q] ? (1ull << 31) + c[q] : 0ull;  // (62 bits travel: both below 2^31)
    }
  }
  unsigned long long tot;
  uint32_t ltot = 0;
  const unsigned long long pre = block_excl_scan(sum, scan, &tot);
  if (WIDE) block_excl_scan(lines, lscan, &ltot);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) {
      lb_publish(st, b, LB_SUM, tot);
      if (WIDE) lb_publish(st + gridDim.x, b, LB_SUM, ltot);
    }
    __syncwarp();
    const unsigned long long e = lb_exclusive(st, b, tot, ctl + 1);
    const unsigned long long l = WIDE ? lb_exclusive(st + gridDim.x, b, ltot, ctl + 1) : 0ull;
    if (threadIdx.x == 0) {
      s_base = e;
      s_lines = l;
    }
  }
  __syncthreads();
  const uint32_t p = WIDE ? uint32_t(s_base + pre) : uint32_t((s_base + pre) & 0x7FFFFFFFull);
  const uint4 o = make_uint4(p, p + c[0], p + c[0] + c[1], p + c[0] + c[1] + c[2]);
  if (v0 + 4 <= n) {
    *reinterpret_cast<uint4*>(voff + v0) = o;  // (scratch: aligned)
  } else {
    if (v0 < n) voff[v0] = o.x;
    if (v0 + 1 < n) voff[v0 + 1] = o.y;
    if (v0 + 2 < n) voff[v0 + 2] = o.z;
  }
  auto split = [](unsigned long long x, unsigned long long l) {
    return WIDE ? (l << 32) | (x & 0xFFFFFFFFull) : ((x >> 31) << 32) | (x & 0x7FFFFFFFull);
  };
  if (threadIdx.x == 0) {
    base[b] = split(s_base, s_lines);
    if (b == gridDim.x - 1) base[b + 1] = split(s_base + tot, s_lines + ltot);
  }
}

// Each later member's last char at its position, four members per thread and
// pass in flight.
template <int NW>
__global__ void __launch_bounds__(256) k_emit_chars(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ head,
                                                    const uint32_t* __restrict__ rank,
                                                    const uint32_t* __restrict__ voff, uint64_t n, int k,
                                                    char* __restrict__ chars) {
  constexpr int PER = 4;
  const uint64_t span = uint64_t(gridDim.x) * blockDim.x;
  // the word that holds char k - 1
  const uint32_t w = (NW == 2 && k > 32) ? 1u : 0u, sh = 2u * uint32_t(k - 1 - 32 * int(w));
  for (uint64_t v0 = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v0 < n; v0 += span * PER) {
    uint32_t r[PER], h[PER];
    uint64_t x[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const uint64_t v = v0 + q * span;
      r[q] = v < n ? rank[v] : 0u;
      h[q] = v < n ? head[v] : 0u;
      x[q] = v < n ? keys[v * NW + w] : 0u;
    }
    uint32_t at[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) at[q] = r[q] ? voff[h[q]] + r[q] : 0u;
#pragma unroll
    for (int q = 0; q < PER; ++q)
      if (r[q] && at[q] < n) chars[at[q]] = acgt(uint32_t(x[q] >> sh) & 3u);
  }
}

// The lines of a tile's heads, in id order.  Lines of EMIT_HUGE members or
// more leave their chars to k_emit_huge.
constexpr uint32_t EMIT_HUGE = 1u << 16;
template <int NW>
__global__ void __launch_bounds__(256) k_emit_lines(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ head,
                                                    const uint32_t* __restrict__ cnt,
                                                    const uint32_t* __restrict__ voff, const char* __restrict__ chars,
                                                    const unsigned long long* __restrict__ base, uint64_t n, int k,
                                                    char* __restrict__ out, uint32_t* ctl, uint32_t* __restrict__ huge) {
  constexpr int NC = NW == 1 ? 4 : 6;
  constexpr uint32_t BUF = (16 + 32 * (32 * NW + TAIL_MAX + 4) + 16) / 4;  // a warp's text: 32 lines
  __shared__ __align__(16) uint32_t buf_all[8][BUF];
  __shared__ uint16_t list[EMIT_TILE];
  __shared__ uint32_t scan[33];
  const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5;
  uint32_t* buf = buf_all[wid];
  const uint64_t t0 = uint64_t(blockIdx.x) * EMIT_TILE, v0 = t0 + 4u * threadIdx.x;
  const uint4 h = ld4(head, v0, n, ~uint32_t(v0));
  const uint32_t mask = (h.x == uint32_t(v0) ? 1u : 0u) | (h.y == uint32_t(v0 + 1) ? 2u : 0u) |
                        (h.z == uint32_t(v0 + 2) ? 4u : 0u) | (h.w == uint32_t(v0 + 3) ? 8u : 0u);
  uint32_t nl;
  uint32_t at = block_excl_scan(uint32_t(__popc(mask)), scan, &nl);
  for (uint32_t m = mask; m; m &= m - 1) list[at++] = uint16_t(4 * threadIdx.x + uint32_t(__ffs(m)) - 1u);
  __syncthreads();
  const unsigned long long line0 = base[blockIdx.x] >> 32;
  const uint32_t per = ((nl + 7) / 8 + 31u) & ~31u;
  const uint32_t r0 = min(nl, wid * per), r1 = min(nl, r0 + per);
  if (r0 >= r1) return;
  WarpText T;
  T.begin(out + (line0 + r0) * uint64_t(k) + voff[t0 + list[r0]]);
  for (uint32_t i0 = r0; i0 < r1; i0 += 32) {
    const bool live = i0 + lane < r1;
    uint64_t v = 0;
    uint32_t c = 0, p = 0;
    Key<NW> x;
#pragma unroll
    for (int w = 0; w < NW; ++w) x.w[w] = 0;
    if (live) {
      v = t0 + list[i0 + lane];
      c = cnt[v] + 1u;
      p = voff[v];
      x = ld_key<NW>(keys, v);
    }
    const unsigned long long nb = live ? uint64_t(k) + c : 0ull;
    unsigned long long inc = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= uint32_t(o)) inc += u;
    }
    const unsigned long long total = __shfl_sync(0xFFFFFFFFu, inc, 31);
    if (!__any_sync(0xFFFFFFFFu, c > uint32_t(TAIL_MAX) + 1u)) {
      if (live) {
        uint64_t codes = 0;
        for (uint32_t r = 1; r < c; ++r) {
          const uint32_t b = uint32_t(chars[p + r]);
          codes |= uint64_t(codes_of_bits((b >> 1) & 3u)) << (2 * (r - 1));
        }
        uint64_t w[3] = {x.w[0], 0, 0};
        if constexpr (NW == 1) {
          w[0] |= codes << (2 * k);
          w[1] = codes >> (64 - 2 * k);
        } else {
          const int u = 2 * k - 64;
          w[1] = x.w[1] | (codes << u);
          w[2] = u ? codes >> (64 - u) : 0ull;
        }
        uint32_t xx[NC];
#pragma unroll
        for (int q = 0; q < NC; ++q) xx[q] = uint32_t(w[q >> 1] >> (32 * (q & 1)));
        spell_text<NC>(buf, T.fill + uint32_t(inc - nb), xx, uint32_t(k) - 1u + c, 1u);
      }
      __syncwarp();
      T.flush(buf, uint32_t(total));
    } else {
      // a longer line among the 32: k-mers by their lanes, later chars by the
      // warp, line after line
      T.end(buf);
      char* const dst = T.dst + (inc - nb);
      if (live) {
        spell_key<NW>(dst, x, k);
        dst[uint64_t(k) - 1 + c] = '\n';
        if (c >= EMIT_HUGE) huge[atomicAdd(ctl + 2, 1u)] = uint32_t(v);
      }
      for (uint32_t q = 0; q < 32; ++q) {
        const uint32_t m = __shfl_sync(0xFFFFFFFFu, c, int(q)), f = __shfl_sync(0xFFFFFFFFu, p, int(q));
        char* const d = reinterpret_cast<char*>(
            __shfl_sync(0xFFFFFFFFu, (unsigned long long)reinterpret_cast<uintptr_t>(dst), int(q)));
        if (m > 1 && m < EMIT_HUGE) copy_bytes(d + k, chars + f + 1, m - 1, lane, 32u);
      }
      __syncwarp();
      T.begin(T.dst + total);
    }
  }
  T.end(buf);
}

// The later chars of the lines of EMIT_HUGE members or more, each line by the
// whole grid.
__global__ void __launch_bounds__(256) k_emit_huge(const uint32_t* __restrict__ head, const uint32_t* __restrict__ cnt,
                                                   const uint32_t* __restrict__ voff, const char* __restrict__ chars,
                                                   const unsigned long long* __restrict__ base, int k,
                                                   char* __restrict__ out, const uint32_t* __restrict__ huge,
                                                   uint32_t nhuge) {
  __shared__ uint32_t scan[33];
  for (uint32_t i = 0; i < nhuge; ++i) {
    const uint32_t v = huge[i], c = cnt[v] + 1u, p = voff[v];
    // the line's index: its tile's first and the heads before it there
    const uint64_t t0 = uint64_t(v) / EMIT_TILE * EMIT_TILE;
    uint32_t before = 0;
    for (uint64_t u = t0 + threadIdx.x; u < v; u += blockDim.x) before += head[u] == uint32_t(u);
    uint32_t tot;
    block_excl_scan(before, scan, &tot);
    char* const dst = out + ((base[v / EMIT_TILE] >> 32) + tot) * uint64_t(k) + p + k;
    for (uint64_t x = uint64_t(blockIdx.x) * EMIT_HUGE; x < c - 1u; x += uint64_t(gridDim.x) * EMIT_HUGE)
      copy_bytes(dst + x, chars + p + 1 + x, min((unsigned long long)EMIT_HUGE, c - 1ull - x), threadIdx.x, blockDim.x);
  }
}

// =========================================================== host pipeline

static int grid_for(const Env& e, uint64_t work, int block) {
  const uint64_t want = (work + block - 1) / block;
  const uint64_t cap = uint64_t(e.sm_count) * 16;
  return int(std::max<uint64_t>(1, std::min(want, cap)));
}

int Env::fail(int code, const std::string& msg) {
  err = msg;
  return code;
}

cudaError_t Env::dev_malloc(void** p, size_t bytes) {
  fault_hit = faults.fail_alloc_after && --faults.fail_alloc_after == 0;
  if (fault_hit) {
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaMalloc(p, bytes);
}

void* Env::take(int w, size_t bytes) {
  Arena& a = ar[w];
  const size_t o = (a.used + 255) & ~size_t(255);
  if (o + bytes > a.cap) return nullptr;
  a.used = o + bytes;
  return a.base + o;
}

int Env::reserve(int w, size_t bytes) {
  Arena& a = ar[w];
  bytes += size_t(16) << 20;
  if (bytes <= a.cap) return UC_OK;
  if (pool)
    return fail(UC_EBUDGET, "job needs " + std::to_string(bytes >> 20) + " MiB in arena " + std::to_string(w) +
                                ", its pool slice holds " + std::to_string(a.cap >> 20) + " MiB");
  if (a.used) return fail(UC_EINTERNAL, "arena grown while in use");
  const size_t other = ar[1 - w].cap;
  if (bytes + other > budget)
    return fail(UC_EBUDGET, "job needs " + std::to_string((bytes + other) >> 20) + " MiB of scratch, budget " +
                                std::to_string(budget >> 20) + " MiB");
  if (a.base) {
    cudaStreamSynchronize(stream);
    cudaFree(a.base);
    a.base = nullptr;
    a.cap = 0;
  }
  if (dev_malloc(reinterpret_cast<void**>(&a.base), bytes) != cudaSuccess) {
    cudaGetLastError();
    a.base = nullptr;
    return fail(UC_ENOMEM, "cudaMalloc of " + std::to_string(bytes >> 20) + " MiB failed");
  }
  a.cap = bytes;
  return UC_OK;
}

int Env::big_scratch(size_t bytes, char*& p, const char* what) {
  if (bytes > big_cap) {
    if (big_buf) {
      cudaStreamSynchronize(stream);
      cudaFree(big_buf);
    }
    big_buf = nullptr;
    big_cap = 0;
    if (bytes > budget) return fail(UC_EBUDGET, what);
    if (dev_malloc(reinterpret_cast<void**>(&big_buf), bytes) != cudaSuccess) {
      cudaGetLastError();
      big_buf = nullptr;
      return fail(UC_ENOMEM, what);
    }
    big_cap = bytes;
  }
  p = big_buf;
  return UC_OK;
}

int Env::check_err(const Counters* h) {
  const uint32_t f = h->err;
  if (!f) return UC_OK;
  if (f & ERR_LINE) return fail(UC_EINPUT, "a k-mer line is shorter than k");
  if (f & ERR_COUNT) return fail(UC_EINPUT, "header count differs from the number of lines");
  if (f & ERR_TIMEOUT) return fail(UC_ETIMEOUT, "a bounded device wait ran out");
  if (f & ERR_CAPACITY) return fail(UC_EINTERNAL, "an output bound was exceeded");
  return fail(UC_EINTERNAL, "internal invariant failed (flags " + std::to_string(f) + ")");
}

int Env::read_ctr() {
  Env& e = *this;
  UC_CK(cudaMemcpyAsync(h_ctr, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, stream));
  UC_CK(cudaStreamSynchronize(stream));
  return UC_OK;
}

// Parse the count line: reads the first bytes back to the host.
int parse_header(Env& e, const char* d_text, size_t bytes, uint64_t& n, uint64_t& body) {
  std::vector<char> h;
  size_t want = std::min<size_t>(bytes, 256);
  for (;;) {
    h.resize(want);
    if (want) UC_CK(cudaMemcpyAsync(h.data(), d_text, want, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    size_t p = 0;
    while (p < want && (h[p] == ' ' || h[p] == '\t' || h[p] == '\r')) ++p;
    if (p >= want || h[p] < '0' || h[p] > '9') {
      if (want < bytes && p >= want) {
        want = std::min(bytes, want * 4);
        continue;
      }
      return e.fail(UC_EINPUT, "missing k-mer count header");
    }
    uint64_t v = 0;
    while (p < want && h[p] >= '0' && h[p] <= '9') {
      v = v * 10 + uint64_t(h[p] - '0');
      if (v > 0xFFFFFFFEull) return e.fail(UC_EINPUT, "k-mer count too large");
      ++p;
    }
    while (p < want && h[p] != '\n') ++p;
    if (p >= want && want < bytes) {
      want = std::min(bytes, want * 4);
      continue;
    }
    n = v;
    body = (p < want) ? p + 1 : want;
    return UC_OK;
  }
}

// End of the k-mer lines: trailing '\n' / '\r' bytes are not a line.
static int text_end(Env& e, const char* d_text, size_t bytes, uint64_t body, uint64_t& end) {
  end = bytes;
  char tail[256];
  while (end > body) {
    const size_t take = std::min<uint64_t>(256, end - body);
    UC_CK(cudaMemcpyAsync(tail, d_text + end - take, take, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    size_t j = take;
    while (j > 0 && (tail[j - 1] == '\n' || tail[j - 1] == '\r')) --j;
    end -= (take - j);
    if (j > 0) break;
  }
  return UC_OK;
}

static size_t line_index_bytes(size_t bytes, uint64_t n) {
  return (bytes / INDEX_CHUNK + 4) * 8 + (n + 1) * 8 + 4 * 256;
}

struct FuseArgs {
  int l = 0;
  uint64_t seed = 0;
  uint32_t jb = 0;
  uint32_t *b1 = nullptr, *b2 = nullptr, *jcross = nullptr;
  uint32_t* counts = nullptr;  // group counts (cshift), or 16-bit counts two per word (CNT16)
  uint32_t cshift = CNT16;
  uint64_t cbytes = 0;         // bytes of counts to clear before a second pack
  uint64_t M = 0;
};

// One wave of resident CTAs: blocks stride over equal-sized line blocks, so a
// partial second wave would double the time.
template <int NW, bool FUSE, bool MULTI, int KC>
static void launch_pack_as(Env& e, const JobTab* jobs, const JobTab& J, uint32_t njobs, uint64_t nblocks,
                           const unsigned long long* starts, int k, uint64_t* keys, const FuseArgs& fz) {
  const uint32_t pcap = pack_pieces(starts == nullptr, k);
  const size_t sm = pack_smem(pcap);
  if (sm > 48 * 1024) allow_max_smem(e, k_pack<NW, FUSE, MULTI, KC>);
  int occ = 0;
  occupancy(e, occ, k_pack<NW, FUSE, MULTI, KC>, 256, sm);
  const int grid = int(std::max<uint64_t>(1, std::min<uint64_t>(nblocks, uint64_t(e.sm_count) * std::max(1, occ))));
  ++e.launches;
  k_pack<NW, FUSE, MULTI, KC><<<grid, 256, sm, e.stream>>>(jobs, J, njobs, nblocks, starts, k, keys, &e.ctr->err, fz.l,
                                                           fz.seed, fz.jb, fz.b1, fz.b2, fz.counts, fz.cshift,
                                                           fz.jcross, pcap);
}

// one: the job of a single-job launch (host copy), or NULL for a batch
// whose jobs the kernel finds in the table.
template <int NW>
static void launch_pack(Env& e, const JobTab* jobs, const JobTab* one, uint32_t njobs, uint64_t nblocks,
                        const unsigned long long* starts, int k, uint64_t* keys, const FuseArgs* fz) {
  constexpr int KC = NW == 1 ? 31 : 63;
  const JobTab J = one ? *one : JobTab{};
  if (!fz) {
    if (k == KC) launch_pack_as<NW, false, false, KC>(e, jobs, J, njobs, nblocks, starts, k, keys, FuseArgs{});
    else launch_pack_as<NW, false, false, 0>(e, jobs, J, njobs, nblocks, starts, k, keys, FuseArgs{});
  } else if (one) {
    if (k == KC) launch_pack_as<NW, true, false, KC>(e, jobs, J, njobs, nblocks, starts, k, keys, *fz);
    else launch_pack_as<NW, true, false, 0>(e, jobs, J, njobs, nblocks, starts, k, keys, *fz);
  } else {
    if (k == KC) launch_pack_as<NW, true, true, KC>(e, jobs, J, njobs, nblocks, starts, k, keys, *fz);
    else launch_pack_as<NW, true, true, 0>(e, jobs, J, njobs, nblocks, starts, k, keys, *fz);
  }
}

// Grow-only device buffers for the job table and the per-job counters.
static int job_buffers(Env& e, uint32_t njobs) {
  const size_t want = size_t(njobs) * (sizeof(JobTab) + 4 * 8) + 1024;
  if (want <= e.jcap) return UC_OK;
  if (e.jbuf) {
    cudaStreamSynchronize(e.stream);
    cudaFree(e.jbuf);
  }
  e.jbuf = nullptr;
  e.jcap = 0;
  if (e.dev_malloc(reinterpret_cast<void**>(&e.jbuf), want) != cudaSuccess) {
    cudaGetLastError();
    e.jbuf = nullptr;
    return e.fail(UC_ENOMEM, "job table");
  }
  e.jcap = want;
  return UC_OK;
}
struct JobDev {
  JobTab* tab;
  uint32_t* jcross;
  uint32_t* jseg;
  unsigned long long* jout;
  unsigned long long* jclosed;
};
static JobDev job_dev(Env& e, uint32_t njobs) {
  JobDev d;
  d.tab = reinterpret_cast<JobTab*>(e.jbuf);
  char* q = e.jbuf + ((size_t(njobs) * sizeof(JobTab) + 255) & ~size_t(255));
  // (jout and jseg, which every tile adds to, in L2 lines of their own)
  auto line = [](void* p) { return reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(p) + 127) & ~uintptr_t(127)); };
  d.jout = reinterpret_cast<unsigned long long*>(q);
  d.jseg = reinterpret_cast<uint32_t*>(line(d.jout + njobs));
  d.jclosed = reinterpret_cast<unsigned long long*>(line(d.jseg + njobs));
  d.jcross = reinterpret_cast<uint32_t*>(d.jclosed + njobs);
  return d;
}

// Text -> keys for one job (and, with fz, buckets + counts).  Fixed-width
// lines are packed directly; any other layout indexes the line starts first
// (back arena, which must be empty).
// defer: fixed-width lines are only enqueued; the caller reads the counters
// and, on ERR_LAYOUT, clears them and calls again with J.fixed = 0.
static int pack_single(Env& e, const char* d_text, size_t bytes, int k, uint64_t* d_keys, const FuseArgs* fz,
                       JobTab& J, JobTab* jdev, bool defer = false) {
  const uint8_t* text = reinterpret_cast<const uint8_t*>(d_text);
  const uint64_t n = J.n, body = J.body, end = J.end;
  if (!defer) UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));  // (cleared with the counters)
  if (n == 0) {
    if (end > body) return e.fail(UC_EINPUT, "header count differs from the number of lines");
    return UC_OK;
  }
  const int nw = (k <= 31) ? 1 : 2;
  const uint64_t nblocks = (n + PACK_LINES - 1) / PACK_LINES;
  bool fixed = J.fixed != 0;
  int st;
  if (fixed) {
    if (nw == 1) launch_pack<1>(e, jdev, &J, 1, nblocks, nullptr, k, d_keys, fz);
    else launch_pack<2>(e, jdev, &J, 1, nblocks, nullptr, k, d_keys, fz);
    UC_CK(cudaGetLastError());
    if (defer) return UC_OK;
    st = e.read_ctr();
    if (st) return st;
    if (e.h_ctr->err & ERR_LAYOUT) {
      fixed = false;
      UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
      if (fz) {
        UC_CK(cudaMemsetAsync(fz->counts, 0, fz->cbytes, e.stream));
        UC_CK(cudaMemsetAsync(fz->jcross, 0, 4, e.stream));
      }
    } else if (e.h_ctr->err) {
      return e.check_err(e.h_ctr);
    }
  }
  if (!fixed) {
    const uint64_t nchunks = (end - body + 15) / INDEX_CHUNK + 1;
    st = e.reserve(1, line_index_bytes(bytes, n));
    if (st) return st;
    // the look-back words, then the count of breaks, the ticket and the wait's flag
    unsigned long long* lbw = static_cast<unsigned long long*>(e.take(1, (nchunks + 2) * 8));
    unsigned long long* starts = static_cast<unsigned long long*>(e.take(1, (n + 1) * 8));
    if (!lbw || !starts) return e.fail(UC_EBUDGET, "scratch for the line index");
    UC_CK(cudaMemsetAsync(lbw, 0, (nchunks + 2) * 8, e.stream));
    uint32_t* flags = reinterpret_cast<uint32_t*>(lbw + nchunks + 1);
    ++e.launches;
    k_line_index<<<unsigned(nchunks), 256, 0, e.stream>>>(text, body, end, n, starts, lbw, flags, flags + 1,
                                                          lbw + nchunks);
    UC_CK(cudaGetLastError());
    unsigned long long got[2] = {0, 0};
    UC_CK(cudaMemcpyAsync(got, lbw + nchunks, 16, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    if (got[1] >> 32) return e.fail(UC_ETIMEOUT, "a bounded device wait ran out (line index)");
    const unsigned long long lines_m1 = got[0];
    if (lines_m1 + 1 != n) return e.fail(UC_EINPUT, "header count differs from the number of lines");
    if (nw == 1) launch_pack<1>(e, jdev, &J, 1, nblocks, starts, k, d_keys, fz);
    else launch_pack<2>(e, jdev, &J, 1, nblocks, starts, k, d_keys, fz);
    UC_CK(cudaGetLastError());
    st = e.read_ctr();
    e.ar[1].used = 0;
    if (st) return st;
    if (e.h_ctr->err) return e.check_err(e.h_ctr);
  }
  return UC_OK;
}

// Host view of one job's text: count line, body offset, end, layout.  The
// first and the last bytes come back in one wait; a longer count line or tail
// is read by parse_header and text_end.
static int host_job(Env& e, const char* d_text, size_t bytes, int k, JobTab& J) {
  uint64_t n = 0, body = 0, end = 0;
  constexpr size_t W = 256;
  const size_t w = std::min<size_t>(bytes, W);
  char *head = e.h_io(), *tail = e.h_io() + W;
  if (w) {
    UC_CK(cudaMemcpyAsync(head, d_text, w, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaMemcpyAsync(tail, d_text + bytes - w, w, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
  }
  size_t p = 0;
  while (p < w && (head[p] == ' ' || head[p] == '\t' || head[p] == '\r')) ++p;
  bool known = p < w && head[p] >= '0' && head[p] <= '9';
  for (; known && p < w && head[p] >= '0' && head[p] <= '9'; ++p) {
    n = n * 10 + uint64_t(head[p] - '0');
    if (n > 0xFFFFFFFEull) known = false;
  }
  while (p < w && head[p] != '\n') ++p;
  known = known && (p < w || w == bytes);
  if (known) {
    body = (p < w) ? p + 1 : w;
  } else {
    const int st = parse_header(e, d_text, bytes, n, body);
    if (st) return st;
  }
  end = bytes;
  const size_t at = bytes - w;  // of the tail
  while (end > body && end > at && (tail[end - at - 1] == '\n' || tail[end - at - 1] == '\r')) --end;
  if (end > body && end == at) {  // nothing but line breaks there
    const int st = text_end(e, d_text, bytes, body, end);
    if (st) return st;
  }
  J = JobTab{};
  J.text = reinterpret_cast<const uint8_t*>(d_text);
  J.tbytes = bytes;
  J.n = n;
  J.body = body;
  J.end = end;
  const uint64_t stride = uint64_t(k) + 1;
  J.fixed = ((n == 0 && end == body) || (n > 0 && end - body == n * stride - 1)) ? 1u : 0u;
  return UC_OK;
}

int pack(Env& e, const char* d_text, size_t bytes, int k, uint64_t* d_keys, uint64_t& n_out) {
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  e.reset();
  JobTab J;
  int r = host_job(e, d_text, bytes, k, J);
  if (r) return r;
  n_out = J.n;
  r = job_buffers(e, 1);
  if (r) return r;
  JobDev jd = job_dev(e, 1);
  r = pack_single(e, d_text, bytes, k, d_keys, nullptr, J, jd.tab);
  e.reset();
  return r;
}

int minimizers(Env& e, const uint64_t* d_keys, uint64_t n, int k, int l, uint64_t seed,
               const uint32_t* d_table, uint32_t* l1, uint32_t* l2) {
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  if (l < 1 || l > 16 || l > k - 1) return e.fail(UC_EINPUT, "l must be in [1, min(16, k-1)]");
  if (n == 0) return UC_OK;
  const int grid = grid_for(e, n, 256);
  ++e.launches;
  if (k <= 31) k_lmin<1><<<grid, 256, 0, e.stream>>>(d_keys, n, k, l, seed, d_table, l1, l2);
  else k_lmin<2><<<grid, 256, 0, e.stream>>>(d_keys, n, k, l, seed, d_table, l1, l2);
  UC_CK(cudaGetLastError());
  return UC_OK;
}

// Bucket plan.  A job's buckets are (job << jb) | local: the largest job
// sizes jb, and njobs << jb buckets in all (rounded up to a power of two,
// bits = log2 of that).
struct Plan {
  uint32_t bits, jb, cap, pack, tslots, wcap, wts, wbytes, lf, wlf;
  uint32_t cg;  // the pack's count groups: 2^cg buckets each
  int l_used;
  uint64_t M;
};

// Count groups of 2^bits buckets: at most 2^COUNT_GROUPS_BITS of them,
// from 2^24 buckets on (below that one 32-bit count per bucket, at most
// 32 MiB, stays in L2 and level 3 needs no counting pass).
static uint32_t count_group_bits(uint32_t bits) {
  return bits >= 24 ? bits - COUNT_GROUPS_BITS : 0u;
}
static uint64_t count_groups(uint64_t M) { return std::min<uint64_t>(M, 1ull << COUNT_GROUPS_BITS); }

static uint32_t ceil_log2(uint64_t x) {
  uint32_t b = 0;
  while ((1ull << b) < x) ++b;
  return b;
}

// lean: for a job that does not fit otherwise; l-mers as short as the buckets allow,
// which make fewer cross k-mers (and larger tiles).
static Plan plan_buckets(const Env& e, uint64_t nmax, uint32_t njobs, int k, int l, bool lean = false) {
  Plan P{};
  const int nw = (k <= 31) ? 1 : 2;
  uint32_t cap = e.tune.tile_capacity ? e.tune.tile_capacity : 4096;
  while (cap > 256 && tile_bytes(nw, cap, pow2_at_least(2ull * cap)) > size_t(e.smem_optin)) cap -= 256;
  // warp tiles: <= wcap copies, one warp each (1 disables the tier)
  uint32_t wcap = e.tune.warp_capacity ? e.tune.warp_capacity : 256;
  if (wcap > cap) wcap = cap;
  const bool warp_tier = wcap >= 32;
  const uint32_t pack_cap = warp_tier ? wcap : cap;  // tiles are packed for this capacity
  const uint32_t jbits_max = 25 - std::min<uint32_t>(25, ceil_log2(njobs));
  const uint64_t copies = nmax + nmax / 8 + 1;
  uint32_t jb = 0;
  if (e.tune.bucket_bits) {
    jb = e.tune.bucket_bits;
  } else {
    // about bucket_fill buckets per tile: small enough that tiles pack well,
    // large enough that each bucket gathers several l-mers
    // (256 Mbp, k = 31: 4 per tile of 256 copies takes the bucket phase from
    // 7.85 to 7.5 ms against 8, with 2% more tiles; 200 Mbp stays below the
    // count groups that way)
    const uint32_t fill = e.tune.bucket_fill ? e.tune.bucket_fill : 4;
    while ((copies >> jb) > std::max<uint32_t>(1, pack_cap / fill) && jb < 25) ++jb;
  }
  jb = std::min(jb, jbits_max);
  // enough l-mers that each bucket gathers several of them, and that the most
  // taken l-mer (the lowest priority: every k-mer that holds it) brings at
  // most about 20 k-mers in a uniform genome, some hundreds at 30% GC, so that
  // few buckets outgrow a warp tile.  Longer ones only add cross k-mers.
  // Tile kernels at the l of the first rule and of both: 13M k-mers, k = 47,
  // 30% GC, l = 11 and 14: 0.83 and 0.61 ms; 66M, k = 63, l = 12 and 14: 3.66
  // and 3.32; 257M, k = 31, l = 13 and 14: 9.27 and 8.86 (15: the whole job is
  // as long as at 13).
  int lmin = int((jb + 2 + 1) / 2);
  while (!lean && lmin < std::min(16, k - 1) && 20.0 * std::ldexp(1.0, 2 * lmin) < double(nmax) * double(k - lmin)) ++lmin;
  int lu = std::max(l, lmin);
  lu = std::min(lu, std::min(16, k - 1));
  // hash slots per 100 copies: 300 for warp tiles (a table of 1024 slots at 218
  // copies; a warp's probes end with its longest one: 257M k-mers, k = 31, 8.7
  // ms at 200 and 7.5 at 300), 200 for block tiles (two of them per SM)
  const uint32_t lf = e.tune.load_factor_pct ? e.tune.load_factor_pct : 200;
  const uint32_t wlf = e.tune.load_factor_pct ? e.tune.load_factor_pct : 300;
  uint32_t ts = big_slots(cap, lf);
  while (ts > pow2_at_least(2ull * cap) && tile_bytes(nw, cap, ts) > size_t(e.smem_optin)) ts >>= 1;
  P.jb = jb;
  P.bits = ceil_log2(uint64_t(njobs) << jb);
  P.cap = cap;
  P.pack = pack_cap;
  P.tslots = ts;
  P.wcap = warp_tier ? wcap : 0;
  uint32_t wts = warp_tier ? big_slots(wcap, wlf) : 0;
  // eight warp tiles share a CTA's shared memory
  while (warp_tier && wts > pow2_at_least(2ull * wcap) && 8 * tile_bytes(nw, wcap, wts) > size_t(e.smem_optin))
    wts >>= 1;
  P.wts = wts;
  P.lf = lf;
  P.wlf = wlf;
  P.wbytes = warp_tier ? uint32_t((tile_bytes(nw, wcap, P.wts) + 15) & ~size_t(15)) : 0;
  P.l_used = lu;
  P.M = 1ull << P.bits;
  P.cg = count_group_bits(P.bits);
  return P;
}

struct Front {
  uint64_t* keys;
  uint32_t *b1, *b2, *counts, *c16, *gcount;
  unsigned long long *boff, *cursor, *fcur, *tile_begin, *goff;
  uint32_t *big_list, *wlist, *blist, *tile_job;
  unsigned long long* big_size;
};

static size_t front_bytes(uint64_t n, int nw, uint64_t M, bool own_keys) {
  size_t need = 0;
  auto add = [&](size_t b) { need += (b + 255) & ~size_t(255); };
  if (own_keys) add(n * 8 * nw);
  add(n * 4); add(n * 4); add(M * 4); add((M + 1) * 8); add(M * 8); add(M * 8); add((M + 2) * 8);
  add(M * 4); add(M * 8);
  add(M * 4); add(M * 4); add(M * 4);
  add((M + 1) / 2 * 4);
  add(count_groups(M) * 4); add((count_groups(M) + 1) * 8);
  return need;
}

static int take_front(Env& e, uint64_t n, int nw, uint64_t M, bool own_keys, Front& f) {
  f.keys = own_keys ? static_cast<uint64_t*>(e.take(0, n * 8 * nw)) : nullptr;
  f.b1 = static_cast<uint32_t*>(e.take(0, n * 4));
  f.b2 = static_cast<uint32_t*>(e.take(0, n * 4));
  f.counts = static_cast<uint32_t*>(e.take(0, M * 4));
  f.boff = static_cast<unsigned long long*>(e.take(0, (M + 1) * 8));
  f.cursor = static_cast<unsigned long long*>(e.take(0, M * 8));
  f.fcur = static_cast<unsigned long long*>(e.take(0, M * 8));
  f.tile_begin = static_cast<unsigned long long*>(e.take(0, (M + 2) * 8));
  f.big_list = static_cast<uint32_t*>(e.take(0, M * 4));
  f.big_size = static_cast<unsigned long long*>(e.take(0, M * 8));
  f.wlist = static_cast<uint32_t*>(e.take(0, M * 4));
  f.blist = static_cast<uint32_t*>(e.take(0, M * 4));
  f.tile_job = static_cast<uint32_t*>(e.take(0, M * 4));
  f.c16 = static_cast<uint32_t*>(e.take(0, (M + 1) / 2 * 4));
  f.gcount = static_cast<uint32_t*>(e.take(0, count_groups(M) * 4));
  f.goff = static_cast<unsigned long long*>(e.take(0, (count_groups(M) + 1) * 8));
  if (!f.goff) return e.fail(UC_EBUDGET, "front arena overflow");
  return UC_OK;
}

// Clears the counters and the look-back words behind them.
static int clear_counters(Env& e) {
  UC_CK(cudaMemsetAsync(e.ctr, 0, COUNTERS_BYTES, e.stream));
  return UC_OK;
}
static unsigned long long* plan_lb(const Env& e) { return reinterpret_cast<unsigned long long*>(e.ctr + 1); }
static unsigned long long* scan_lb(const Env& e) { return plan_lb(e) + PLAN_LB_WORDS; }

// counts -> offsets (M entries: buckets or count groups) and their total in
// the counters.
static int launch_bucket_offsets(Env& e, const uint32_t* counts, uint64_t M, unsigned long long* offs) {
  const uint64_t nb = (M + SCAN_TILE - 1) / SCAN_TILE;
  if (nb + 1 > SCAN_LB_WORDS) return e.fail(UC_EINTERNAL, "bucket count beyond the look-back words");
  ++e.launches;
  k_bucket_offsets<<<unsigned(nb), 256, 0, e.stream>>>(counts, M, offs, scan_lb(e), &e.ctr->err, &e.ctr->copies);
  UC_CK(cudaGetLastError());
  return UC_OK;
}
// The same, and the total (host sync).  Clears the scan's look-back words
// first: a run may take offsets more than once.
static int bucket_offsets(Env& e, const uint32_t* counts, uint64_t M, unsigned long long* offs, uint64_t& copies) {
  UC_CK(cudaMemsetAsync(scan_lb(e), 0, SCAN_LB_WORDS * 8, e.stream));
  int r = launch_bucket_offsets(e, counts, M, offs);
  if (r) return r;
  r = e.read_ctr();
  if (r) return r;
  copies = e.h_ctr->copies;
  return (e.h_ctr->err & ERR_TIMEOUT) ? e.check_err(e.h_ctr) : UC_OK;
}
static int bucket_offsets(Env& e, const Front& f, uint64_t M, uint64_t& copies) {
  return bucket_offsets(e, f.counts, M, f.boff, copies);
}

// Level split of the scatter: 2^mcb coarse partitions of 2^fb buckets.
static void scatter_split(uint32_t bbits, uint32_t& mcb, uint32_t& fb) {
  mcb = std::min<uint32_t>(bbits, 8);
  fb = bbits - mcb;
}

static size_t scatter_stage_bytes(uint64_t copies, int nw) { return copies * (8ull * nw + 8ull); }

static Tiers tiers_of(const Front& f, const Plan& P, int nw) {
  return Tiers{P.wcap, P.cap, P.lf, nw, f.wlist, f.blist, f.big_list, f.big_size};
}
// Tiles from the bucket counts: next-fit runs of whole buckets.  lists: sorted
// into their tiers too.
static int plan_tiles(Env& e, const Front& f, const Plan& P, int nw, bool lists) {
  const uint64_t M = P.M;
  ++e.launches;
  // about 256 threads per SM; each run ends a tile, so runs stay long where
  // there are enough buckets
  const uint64_t want = (M + uint64_t(e.sm_count) * 256 - 1) / (uint64_t(e.sm_count) * 256);
  const uint32_t runlen = uint32_t(std::min<uint64_t>(512, std::max<uint64_t>(16, (want + 15) & ~uint64_t(15))));
  const uint64_t nb = ((M + runlen - 1) / runlen + 255) / 256;
  if (nb + 1 > PLAN_LB_WORDS) return e.fail(UC_EINTERNAL, "bucket count beyond the look-back words");
  k_tile_plan<<<unsigned(nb), 256, 0, e.stream>>>(f.counts, f.boff, uint32_t(M), P.pack, P.jb, runlen, f.tile_begin,
                                                   f.tile_job, tiers_of(f, P, nw), lists ? 1 : 0, plan_lb(e), e.ctr);
  UC_CK(cudaGetLastError());
  return UC_OK;
}

// The three placement levels of the bucketed copies.  Level 1
// (k_scatter_coarse) writes region r1; then either level 2 (k_scatter_mid)
// writes r2 and level 3 (k_scatter_sub) writes back into r1, or, where a
// coarse partition is already small, level 3 writes r2 straight away.  Both
// regions hold scatter_stage_bytes(copies, nw); the final copies (pkeys,
// plink) are arrays at the start of the region level 3 wrote.  Level 1
// may run over the k-mers in several launches (the streamed path's chunks):
// its cursors and the cross-index counter carry over.
struct Scatter {
  uint32_t mcb = 0, fb = 0, mc = 0, sb = 0, nsub = 0, cap3 = 0;
  // offsets of the pack's count groups (2^cg buckets each); level 3 writes
  // every bucket's count and offset to cout / bout (null: they are known)
  const unsigned long long* goff = nullptr;
  uint32_t cg = 0;
  uint32_t* cout = nullptr;
  unsigned long long* bout = nullptr;
  bool mid = false;
  int nw = 1;
  uint64_t copies = 0;
  char *r1 = nullptr, *r2 = nullptr;
};

// cg > 0: the copies are counted per group of 2^cg buckets (offsets in
// f.goff) and level 3 writes f.counts and f.boff; cg = 0 with
// group_offsets false: f.boff holds every bucket's offset already.
static int scatter_begin(Env& e, const Front& f, const Plan& P, int nw, char* r1, char* r2, uint64_t copies,
                         Scatter& sc, uint32_t cg = 0, bool group_offsets = false) {
  const uint64_t M = P.M;
  sc.nw = nw;
  sc.copies = copies;
  sc.cg = cg;
  sc.goff = group_offsets ? f.goff : f.boff;
  sc.cout = group_offsets ? f.counts : nullptr;
  sc.bout = group_offsets ? f.boff : nullptr;
  sc.r1 = r1;
  sc.r2 = r2;
  scatter_split(P.bits, sc.mcb, sc.fb);
  sc.mc = 1u << sc.mcb;
  // level-3 staging holds cap3 records (two CTAs per SM); sub-partitions of
  // about half that many copies, at most 2^SUB_MAX_BITS buckets and at most
  // MID_MAX_BINS of them per coarse partition
  sc.cap3 = (nw == 1) ? 8192u : 4096u;
  const double avg = double(copies) / double(M);
  int sbi = avg > 0 ? int(std::lround(std::log2(0.5 * sc.cap3 / avg))) : SUB_MAX_BITS;
  sbi = std::min(sbi, SUB_MAX_BITS);
  sbi = std::min(sbi, int(sc.fb));
  sbi = std::max(sbi, int(sc.fb) - int(std::log2(double(MID_MAX_BINS))));
  sbi = std::max(sbi, int(cg));  // a sub-partition is whole count groups
  sbi = std::max(sbi, 0);
  if (sbi > SUB_MAX_BITS || sbi > int(sc.fb))
    return e.fail(UC_EINTERNAL, "bucket count beyond the three scatter levels");
  sc.sb = uint32_t(sbi);
  sc.mid = sc.sb < sc.fb;
  sc.nsub = uint32_t(M >> sc.sb);
  int r0 = allow_max_smem(e, k_scatter_coarse<1>);
  if (!r0) r0 = allow_max_smem(e, k_scatter_coarse<2>);
  if (!r0) r0 = allow_max_smem(e, k_scatter_mid<1>);
  if (!r0) r0 = allow_max_smem(e, k_scatter_mid<2>);
  if (r0) return r0;
  e.launches += 1;
  k_coarse_init<<<grid_for(e, sc.mc, 256), 256, 0, e.stream>>>(sc.goff, sc.fb - sc.cg, sc.mc, f.cursor);
  UC_CK(cudaGetLastError());
  return UC_OK;
}

static int scatter_l1(Env& e, const Front& f, const Scatter& sc, const uint64_t* keys, const uint32_t* b1,
                      const uint32_t* b2, uint64_t n, int ids_mode) {
  if (n == 0) return UC_OK;
  const int nw = sc.nw;
  const uint64_t chunk = (nw == 1) ? sc_chunk<1>() : sc_chunk<2>();
  const size_t sm1 = size_t(2 * chunk) * (8 * nw + 8) + size_t(sc.mc) * 16 + 16;
  // one wave of resident CTAs (the chunks are strided statically)
  int o1 = 0;
  if (const int ro = nw == 1 ? occupancy(e, o1, k_scatter_coarse<1>, COARSE_THREADS, sm1)
                             : occupancy(e, o1, k_scatter_coarse<2>, COARSE_THREADS, sm1))
    return ro;
  if (o1 < 1) return e.fail(UC_EINTERNAL, "scatter kernel does not fit an SM");
  const int g1 = int(std::max<uint64_t>(1, std::min<uint64_t>((n + chunk - 1) / chunk,
                                                              uint64_t(e.sm_count) * uint64_t(o1))));
  e.launches += 1;
  if (nw == 1)
    k_scatter_coarse<1><<<g1, COARSE_THREADS, sm1, e.stream>>>(keys, b1, b2, n, sc.fb, sc.mc, f.cursor,
                                                               Stage<1, true>::over(sc.r1, sc.copies), ids_mode, e.ctr);
  else
    k_scatter_coarse<2><<<g1, COARSE_THREADS, sm1, e.stream>>>(keys, b1, b2, n, sc.fb, sc.mc, f.cursor,
                                                               Stage<2, true>::over(sc.r1, sc.copies), ids_mode, e.ctr);
  UC_CK(cudaGetLastError());
  return UC_OK;
}

template <int NW>
static int launch_sub(Env& e, const Scatter& sc, char* from, uint64_t* pkeys, uint32_t* plink) {
  const size_t smem = size_t(sc.cap3) * (8 * NW + 4);
  int r = allow_max_smem(e, k_scatter_sub<NW>);
  if (r) return r;
  int occ = 0;
  r = occupancy(e, occ, k_scatter_sub<NW>, 512, smem);
  if (r) return r;
  if (occ < 1) return e.fail(UC_EINTERNAL, "scatter kernel does not fit an SM");
  const int g = int(std::min<uint64_t>(sc.nsub, uint64_t(e.sm_count) * uint64_t(occ)));
  k_scatter_sub<NW><<<g, 512, smem, e.stream>>>(Stage<NW, true>::over(from, sc.copies), sc.goff, sc.sb - sc.cg, sc.sb,
                                                sc.nsub, sc.cap3, pkeys, plink, sc.cout, sc.bout, e.ctr);
  return UC_OK;
}

static int scatter_finish(Env& e, const Front& f, const Scatter& sc, uint64_t*& pkeys, uint32_t*& plink) {
  const int nw = sc.nw;
  // the staged records level 3 reads, and the final copies in the other region
  char* const from = sc.mid ? sc.r2 : sc.r1;
  char* const to = sc.mid ? sc.r1 : sc.r2;
  pkeys = reinterpret_cast<uint64_t*>(to);
  plink = reinterpret_cast<uint32_t*>(to + sc.copies * 8ull * nw);
  if (sc.copies == 0) {
    if (sc.bout) {  // no copies: every bucket empty
      const uint64_t M = uint64_t(sc.nsub) << sc.sb;
      UC_CK(cudaMemsetAsync(sc.cout, 0, M * 4, e.stream));
      UC_CK(cudaMemsetAsync(sc.bout, 0, (M + 1) * 8, e.stream));
    }
    return UC_OK;
  }
  if (sc.mid) {
    const uint32_t nb = 1u << (sc.fb - sc.sb);
    uint32_t* item_start = reinterpret_cast<uint32_t*>(f.cursor + sc.mc);
    const size_t sm2 = size_t(MID_CHUNK) * (8 * nw + 8) + size_t(nb) * 16 + 4 + size_t(sc.mc + 1) * 4;
    int o2 = 0;
    if (const int ro = nw == 1 ? occupancy(e, o2, k_scatter_mid<1>, MID_THREADS, sm2)
                               : occupancy(e, o2, k_scatter_mid<2>, MID_THREADS, sm2))
      return ro;
    if (o2 < 1) return e.fail(UC_EINTERNAL, "scatter kernel does not fit an SM");
    e.launches += 3;
    k_mid_items<<<1, 256, 0, e.stream>>>(sc.goff, sc.fb - sc.cg, sc.mc, item_start);
    k_coarse_init<<<grid_for(e, sc.nsub, 256), 256, 0, e.stream>>>(sc.goff, sc.sb - sc.cg, sc.nsub, f.fcur);
    if (nw == 1)
      k_scatter_mid<1><<<e.sm_count * o2, MID_THREADS, sm2, e.stream>>>(
          Stage<1, true>::over(sc.r1, sc.copies), sc.goff, sc.cg, item_start, sc.fb, sc.sb, sc.mc, f.fcur,
          Stage<1, true>::over(sc.r2, sc.copies), e.ctr);
    else
      k_scatter_mid<2><<<e.sm_count * o2, MID_THREADS, sm2, e.stream>>>(
          Stage<2, true>::over(sc.r1, sc.copies), sc.goff, sc.cg, item_start, sc.fb, sc.sb, sc.mc, f.fcur,
          Stage<2, true>::over(sc.r2, sc.copies), e.ctr);
  }
  e.launches += 1;
  const int r = nw == 1 ? launch_sub<1>(e, sc, from, pkeys, plink) : launch_sub<2>(e, sc, from, pkeys, plink);
  if (r) return r;
  UC_CK(cudaGetLastError());
  if (sc.bout) {
    // the total after the last bucket, for the tile plan
    UC_CK(cudaMemcpyAsync(sc.bout + (uint64_t(sc.nsub) << sc.sb), sc.goff + (uint64_t(sc.nsub) << (sc.sb - sc.cg)),
                          8, cudaMemcpyDeviceToDevice, e.stream));
  }
  return UC_OK;
}

// Sort the tiles [t0, t1) (clipped to the tile count) into their tiers.
static int classify_tiles(Env& e, const Front& f, const Plan& P, int nw, uint32_t t0 = 0,
                          uint32_t t1 = 0xFFFFFFFFu) {
  ++e.launches;
  k_classify<<<grid_for(e, P.M, 256), 256, 0, e.stream>>>(f.tile_begin, e.ctr, tiers_of(f, P, nw), t0, t1);
  UC_CK(cudaGetLastError());
  return UC_OK;
}

// The bucketed copies of all k-mers in one pass, then the tiles (from the
// bucket counts, which level 3 writes when the pack counted groups).
static int plan_and_scatter(Env& e, const Front& f, const Plan& P, uint64_t n, int nw, int ids_mode,
                            char* r1, char* r2, uint64_t copies, uint64_t*& pkeys, uint32_t*& plink,
                            bool group_offsets = false) {
  Scatter sc;
  int r = scatter_begin(e, f, P, nw, r1, r2, copies, sc, group_offsets ? P.cg : 0u, group_offsets);
  if (r) return r;
  r = scatter_l1(e, f, sc, f.keys, f.b1, f.b2, n, ids_mode);
  if (r) return r;
  r = scatter_finish(e, f, sc, pkeys, plink);
  if (r) return r;
  return plan_tiles(e, f, P, nw, true);
}

template <int NW, int KC>
static int run_tiles(Env& e, TileParams& tp, const Front& f, uint32_t threads) {
  tp.wlist = f.wlist;
  tp.blist = f.blist;
  const size_t wsm = size_t(tp.wbytes) * 8;
  int wocc = 0;
  if (tp.wcap) {
    const int r0 = allow_max_smem(e, k_tile_warp<NW, KC>);
    if (r0) return r0;
    if (const int ro = occupancy(e, wocc, k_tile_warp<NW, KC>, 256, wsm)) return ro;
    if (wocc < 1) return e.fail(UC_EINTERNAL, "warp tile kernel does not fit an SM");
  }
  if (e.timed) cudaEventRecord(e.ev[8], e.stream);
  if (tp.wcap) {
    ++e.launches;
    k_tile_warp<NW, KC><<<e.sm_count * wocc, 256, wsm, e.stream>>>(tp);
    UC_CK(cudaGetLastError());
  }
  if (e.timed) cudaEventRecord(e.ev[9], e.stream);
  const size_t smem = tile_bytes(NW, tp.cap, tp.tslots);
  const int r1 = allow_max_smem(e, k_tile<NW, KC>);
  if (r1) return r1;
  int occ = 0;
  if (const int ro = occupancy(e, occ, k_tile<NW, KC>, int(threads), smem)) return ro;
  if (occ < 1) return e.fail(UC_EINTERNAL, "tile kernel does not fit an SM");
  ++e.launches;
  k_tile<NW, KC><<<e.sm_count * occ, threads, smem, e.stream>>>(tp);
  UC_CK(cudaGetLastError());
  if (e.timed) cudaEventRecord(e.ev[5], e.stream);
  e.tiles_timed = e.timed;
  return UC_OK;
}

// The oversized tiles, one CTA each in global scratch: nbig of them, known
// once the tile kernels' counters are read.  Waits for them.
static int run_big_tiles(Env& e, TileParams& tp, const Front& f, int nw, uint32_t nbig) {
  std::vector<unsigned long long> sz(nbig), off(nbig);
  UC_CK(cudaMemcpyAsync(sz.data(), f.big_size, nbig * 8, cudaMemcpyDeviceToHost, e.stream));
  UC_CK(cudaStreamSynchronize(e.stream));
  unsigned long long tot = 0;
  for (uint32_t i = 0; i < nbig; ++i) {
    off[i] = tot;
    tot += sz[i];
  }
  const size_t want = size_t(tot) + size_t(nbig) * 8 + 4096;
  char* big = nullptr;
  if (e.pool) {
    big = static_cast<char*>(e.take(1, want));
    if (!big) return e.fail(UC_EBUDGET, "scratch for oversized buckets exceeds the pool slice");
  } else {
    const int r = e.big_scratch(want, big, "scratch for oversized buckets");
    if (r) return r;
  }
  unsigned long long* d_off = reinterpret_cast<unsigned long long*>(big);
  char* scratch = big + ((size_t(nbig) * 8 + 255) & ~size_t(255));
  UC_CK(cudaMemcpyAsync(d_off, off.data(), nbig * 8, cudaMemcpyHostToDevice, e.stream));
  tp.big_list = f.big_list;
  tp.big_scratch = scratch;
  tp.big_off = d_off;
  ++e.launches;
  if (nw == 1) k_tile_big<1><<<nbig, 1024, 0, e.stream>>>(tp);
  else k_tile_big<2><<<nbig, 1024, 0, e.stream>>>(tp);
  UC_CK(cudaGetLastError());
  UC_CK(cudaStreamSynchronize(e.stream));
  return UC_OK;
}

// The tile kernels for tp.k: compile-time k = 31 (64-bit keys) and 63
// (128-bit keys), the generic form otherwise.
static int launch_tiles(Env& e, TileParams& tp, const Front& f, uint32_t threads, int nw) {
  if (nw == 1) return tp.k == 31 ? run_tiles<1, 31>(e, tp, f, threads) : run_tiles<1, 0>(e, tp, f, threads);
  return tp.k == 63 ? run_tiles<2, 63>(e, tp, f, threads) : run_tiles<2, 0>(e, tp, f, threads);
}
// Every tier, the oversized tiles included (waits once for the counters).
static int run_tiles_k(Env& e, TileParams& tp, const Front& f, uint32_t threads, int nw) {
  int r = launch_tiles(e, tp, f, threads, nw);
  if (!r) r = e.read_ctr();
  if (r) return r;
  if (e.h_ctr->err) return e.check_err(e.h_ctr);
  return e.h_ctr->nbig ? run_big_tiles(e, tp, f, nw, e.h_ctr->nbig) : UC_OK;
}

int find_edges(Env& e, const uint64_t* d_keys, uint64_t n, int k, int l, uint64_t seed, uint32_t* succ,
               uint32_t* pred) {
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  if (l < 1 || l > 16 || l > k - 1) return e.fail(UC_EINPUT, "l must be in [1, min(16, k-1)]");
  if (n >= 0x7FFFFFFFull) return e.fail(UC_EINPUT, "too many k-mers for 31-bit ids");
  if (n == 0) return UC_OK;
  e.reset();
  const int nw = (k <= 31) ? 1 : 2;
  const Plan P = plan_buckets(e, n, 1, k, l);
  int r = e.reserve(0, front_bytes(n, nw, P.M, false));
  if (r) return r;
  Front f{};
  r = take_front(e, n, nw, P.M, false, f);
  if (r) return r;
  f.keys = const_cast<uint64_t*>(d_keys);
  r = clear_counters(e);
  if (r) return r;
  UC_CK(cudaMemsetAsync(f.counts, 0, P.M * 4, e.stream));
  ++e.launches;
  if (nw == 1) k_lmin_count<1><<<grid_for(e, n, 256), 256, 0, e.stream>>>(d_keys, n, k, P.l_used, seed, P.jb, f.b1, f.b2, f.counts);
  else k_lmin_count<2><<<grid_for(e, n, 256), 256, 0, e.stream>>>(d_keys, n, k, P.l_used, seed, P.jb, f.b1, f.b2, f.counts);
  r = launch_bucket_offsets(e, f.counts, P.M, f.boff);
  if (!r) r = e.read_ctr();
  if (r) return r;
  if (e.h_ctr->err) return e.check_err(e.h_ctr);
  const uint64_t copies = e.h_ctr->copies;
  r = e.reserve(1, 2 * scatter_stage_bytes(copies, nw) + 4096);
  if (r) return r;
  char* region1 = static_cast<char*>(e.take(1, scatter_stage_bytes(copies, nw)));
  char* region2 = static_cast<char*>(e.take(1, scatter_stage_bytes(copies, nw)));
  if (!region2) return e.fail(UC_EBUDGET, "back arena overflow");
  uint64_t* pkeys = nullptr;
  uint32_t* plink = nullptr;
  r = plan_and_scatter(e, f, P, n, nw, 1, region1, region2, copies, pkeys, plink);
  if (r) return r;
  TileParams tp{};
  tp.pkeys = pkeys;
  tp.plink = plink;
  tp.tile_begin = f.tile_begin;
  tp.tile_job = f.tile_job;
  tp.ctr = e.ctr;
  tp.k = k;
  tp.cap = P.cap;
  tp.tslots = P.tslots;
  tp.lf = P.lf;
  tp.wlf = P.wlf;
  tp.wcap = P.wcap;
  tp.wts = P.wts;
  tp.wbytes = P.wbytes;
  tp.mode = 0;
  tp.succ = succ;
  tp.pred = pred;
  // The tiles' stores go to random ids, four bytes to a sector of 32, so the
  // values that need none (about half of them: a neighbour of a canonical
  // k-mer is as likely as not to be stored the other way round) are written as
  // a stream beforehand.  16.3M k-mers: tile kernel 815 -> 507 us, for 24 of
  // streaming.
  UC_CK(cudaMemsetAsync(succ, 0xFF, n * 4, e.stream));
  UC_CK(cudaMemsetAsync(pred, 0xFF, n * 4, e.stream));
  e.timed = false;
  r = run_tiles_k(e, tp, f, 512, nw);
  if (r) return r;
  // (oversized tiles may have set the error flag after the counters were read)
  if (e.h_ctr->nbig) r = e.read_ctr();
  e.reset();
  if (r) return r;
  return e.check_err(e.h_ctr);
}

// Enqueue `body` through a CUDA graph: capture it, update the cached
// executable of this slot when the shape key matches (cudaGraphExecUpdate),
// instantiate otherwise, and launch.  The body must only enqueue work.
template <class F>
static int run_graph(Env& e, int slot, uint64_t key, F&& body) {
  if (!e.use_graphs) {
    body();
    return UC_OK;
  }
  const uint32_t before = e.launches;
  // the legacy default stream cannot be captured: capture on an internal
  // stream joined to the caller's stream by events
  const cudaStream_t user = e.stream;
  const bool swap = (user == nullptr || user == cudaStreamLegacy || user == cudaStreamPerThread);
  if (swap) {
    if (!e.gstream) UC_CK(cudaStreamCreateWithFlags(&e.gstream, cudaStreamNonBlocking));
    UC_CK(cudaEventRecord(e.ev[6], user));
    UC_CK(cudaStreamWaitEvent(e.gstream, e.ev[6], 0));
    e.stream = e.gstream;
  }
  struct Restore {
    Env& e;
    cudaStream_t user;
    bool swap;
    ~Restore() {
      if (swap) {
        cudaEventRecord(e.ev[7], e.stream);
        cudaStreamWaitEvent(user, e.ev[7], 0);
        e.stream = user;
      }
    }
  } restore{e, user, swap};
  UC_CK(cudaStreamBeginCapture(e.stream, cudaStreamCaptureModeThreadLocal));
  body();
  cudaGraph_t g = nullptr;
  UC_CK(cudaStreamEndCapture(e.stream, &g));
  bool ok = false;
  if (e.gexec[slot] && e.gkey[slot] == key) {
    cudaGraphExecUpdateResultInfo info;
    ok = cudaGraphExecUpdate(e.gexec[slot], g, &info) == cudaSuccess;
    if (!ok) cudaGetLastError();
  }
  if (!ok) {
    if (e.gexec[slot]) cudaGraphExecDestroy(e.gexec[slot]);
    e.gexec[slot] = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&e.gexec[slot], g, 0);
    if (ie != cudaSuccess) {
      cudaGraphDestroy(g);
      return e.fail(UC_ECUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(ie));
    }
    e.gkey[slot] = key;
  }
  cudaGraphDestroy(g);
  UC_CK(cudaGraphLaunch(e.gexec[slot], e.stream));
  e.graph_nodes += e.launches - before;
  return UC_OK;
}

static uint32_t rank_rounds(uint64_t nmax) {
  uint32_t r = 2;
  for (uint64_t t = 1; t < nmax; t <<= 1) ++r;
  return r;
}

// prefilled: X already holds a state (written by the tiles and the line
// walk) and the first round runs over the ids [0, cnt[0]), cnt[0] set on the
// device before.
static int rank_lists(Env& e, const uint32_t* prev, const uint32_t* w, uint64_t nmax,
                      unsigned long long* X, uint32_t* act0, uint32_t* act1, uint32_t* cnt, uint32_t& rounds,
                      uint32_t*& act_final, uint32_t*& cnt_final, bool prefilled = false) {
  rounds = rank_rounds(nmax);
  const int grid = grid_for(e, nmax ? nmax : 1, 256);
  if (prefilled) {
    UC_CK(cudaMemsetAsync(cnt + 1, 0, rounds * 4, e.stream));
  } else {
    UC_CK(cudaMemsetAsync(cnt, 0, (rounds + 1) * 4, e.stream));
    ++e.launches;
    k_rank_init<<<grid, 256, 0, e.stream>>>(prev, w, nmax, X, act0, cnt);
  }
  uint32_t* lists[2] = {act0, act1};
  for (uint32_t r = 0; r < rounds; ++r) {
    ++e.launches;
    const uint32_t* in = (r == 0 && prefilled) ? nullptr : lists[r & 1];
    k_rank_round<<<grid, 256, 0, e.stream>>>(X, in, cnt + r, lists[(r + 1) & 1], cnt + r + 1);
  }
  UC_CK(cudaGetLastError());
  act_final = lists[rounds & 1];
  cnt_final = cnt + rounds;
  return UC_OK;
}

static size_t hec_bytes(uint64_t nmax, uint32_t R) {
  const uint64_t cap = 2 * nmax + 64;
  return 8 * ((cap * 4 + 255) & ~uint64_t(255)) + 2 * 256 + 2 * (R + 1) * 4 + 1024;
}

static int hec_take(Env& e, uint64_t nmax, uint32_t R, HecPool& h) {
  const uint64_t cap = 2 * nmax + 64;
  uint32_t** arr[8] = {&h.prv, &h.nxt, &h.wt, &h.hn, &h.vc, &h.agg, &h.loc, &h.first0};
  for (auto a : arr) *a = static_cast<uint32_t*>(e.take(1, cap * 4));
  h.lb = static_cast<uint32_t*>(e.take(1, (R + 1) * 4));
  h.ln = static_cast<uint32_t*>(e.take(1, (R + 3) * 4));
  h.cap = uint32_t(std::min<uint64_t>(cap, 0xFFFFFFF0ull));
  h.ctr = e.ctr;
  if (!h.ln) return e.fail(UC_EBUDGET, "arena overflow (HEC pool)");
  return UC_OK;
}

static uint32_t hec_rounds(uint64_t nmax) {
  uint32_t r = 8;
  for (uint64_t t = 1; t < nmax; t <<= 1) r += 2;
  return r;
}
// The rounds a run enqueues: the bound above, or the injected cap.
static uint32_t hec_rounds(const Env& e, uint64_t nmax) {
  const uint32_t r = hec_rounds(nmax);
  return (e.faults.hec_round_cap && e.faults.hec_round_cap < r) ? e.faults.hec_round_cap : r;
}

// HEC contraction of the lists (prev, next, w) into X (pointer | HEAD_BIT,
// offset) and cycle flags, enqueued on the stream (one kernel for all rounds).
// With seg, level 0 comes from the fused path's segment records and the
// ranking's first state in X (built from them by k_seg_xinit; nx cross
// indices) instead of (prev, next, w).
static int hec_contract(Env& e, HecPool& h, uint32_t R, const uint32_t* prev, const uint32_t* next,
                         const uint32_t* w, uint64_t nmax, unsigned long long* X,
                         uint8_t* oncycle, const SegRec* seg = nullptr, uint32_t nx = 0, int k = 0) {
  const int grid = grid_for(e, nmax ? nmax : 1, 256);
  UC_CK(cudaMemsetAsync(h.ln, 0, (R + 3) * 4, e.stream));
  e.launches += 2;
  if (seg) k_hec_level0_seg<<<grid, 256, 0, e.stream>>>(h, seg, X, nmax, nx, k);
  else k_hec_level0<<<grid, 256, 0, e.stream>>>(h, prev, next, w, nmax);
  // every block resident (they meet)
  int occ = 0;
  if (const int ro = occupancy(e, occ, k_hec_all, int(HEC_THREADS), 0)) return ro;
  const uint64_t want = (nmax + HEC_THREADS - 1) / HEC_THREADS;
  const unsigned g = unsigned(std::max<uint64_t>(1, std::min<uint64_t>(want, uint64_t(e.sm_count) * std::max(1, occ))));
  void* args[] = {&h, &R, &X, &oncycle};
  UC_CK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_hec_all), dim3(g), dim3(HEC_THREADS), args, 0,
                                    e.stream));
  return UC_OK;
}

static int contract_hec(Env& e, const uint64_t* d_keys, const uint32_t* succ, const uint32_t* pred, uint64_t n,
                        int k, uint32_t* head, uint32_t* rank, uint64_t& ncyc, bool& fell_back) {
  fell_back = false;
  e.reset();
  const uint32_t R = hec_rounds(e, n);
  int r = e.reserve(1, hec_bytes(n, R) + n * (8 + 4 + 1) + 8 + 4096);
  if (r) return r;
  HecPool h{};
  r = hec_take(e, n, R, h);
  if (r) return r;
  unsigned long long* X = static_cast<unsigned long long*>(e.take(1, n * 8));
  uint32_t* act = static_cast<uint32_t*>(e.take(1, n * 4));
  uint8_t* flag = static_cast<uint8_t*>(e.take(1, n));
  uint32_t* cnt = static_cast<uint32_t*>(e.take(1, 4));
  unsigned long long* dcyc = static_cast<unsigned long long*>(e.take(1, 8));
  if (!dcyc) return e.fail(UC_EBUDGET, "arena overflow");
  UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
  UC_CK(cudaMemsetAsync(flag, 0, n, e.stream));
  r = hec_contract(e, h, R, pred, succ, nullptr, n, X, flag);
  if (r) return r;
  e.launches += 2;
  k_head_rank<<<grid_for(e, n, 256), 256, 0, e.stream>>>(X, n, head, rank);
  UC_CK(cudaMemsetAsync(cnt, 0, 4, e.stream));
  k_cycle_list<<<grid_for(e, n, 256), 256, 0, e.stream>>>(flag, n, act, cnt);
  uint32_t hleft = 0;
  UC_CK(cudaMemcpyAsync(&hleft, cnt, 4, cudaMemcpyDeviceToHost, e.stream));
  r = e.read_ctr();
  if (r) return r;
  if (e.h_ctr->err) {
    if (e.faults.hec_strict) {
      r = e.check_err(e.h_ctr);
      UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
      e.reset();
      return r;
    }
    fell_back = true;
    UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
    e.reset();
    return UC_OK;
  }
  ncyc = 0;
  if (hleft) {
    UC_CK(cudaMemsetAsync(flag, 0, n, e.stream));
    UC_CK(cudaMemsetAsync(dcyc, 0, 8, e.stream));
    ++e.launches;
    if (k <= 31) k_vertex_cycles<1><<<1, 1, 0, e.stream>>>(act, hleft, succ, d_keys, n, head, rank, flag, dcyc);
    else k_vertex_cycles<2><<<1, 1, 0, e.stream>>>(act, hleft, succ, d_keys, n, head, rank, flag, dcyc);
    unsigned long long hc = 0;
    UC_CK(cudaMemcpyAsync(&hc, dcyc, 8, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    ncyc = hc;
  }
  e.reset();
  return UC_OK;
}

int contract(Env& e, const uint64_t* d_keys, const uint32_t* succ, const uint32_t* pred, uint64_t n, int k,
             int method, uint32_t* head, uint32_t* rank, uint64_t& ncyc) {
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  if (n >= 0x7FFFFFFFull) return e.fail(UC_EINPUT, "too many k-mers for 31-bit ids");
  ncyc = 0;
  if (n == 0) return UC_OK;
  if (method == UC_CONTRACT_HEC) {
    bool fell_back = false;
    const int r = contract_hec(e, d_keys, succ, pred, n, k, head, rank, ncyc, fell_back);
    if (r || !fell_back) return r;
    // HEC did not finish inside its pool or rounds: pointer jumping instead
  }
  e.reset();
  int r = e.reserve(1, n * (8 + 4 + 4 + 1) + 64 * 8 + 4096);
  if (r) return r;
  unsigned long long* X = static_cast<unsigned long long*>(e.take(1, n * 8));
  uint32_t* a0 = static_cast<uint32_t*>(e.take(1, n * 4));
  uint32_t* a1 = static_cast<uint32_t*>(e.take(1, n * 4));
  uint8_t* seen = static_cast<uint8_t*>(e.take(1, n));
  uint32_t* cnt = static_cast<uint32_t*>(e.take(1, 64 * 4));
  unsigned long long* dcyc = static_cast<unsigned long long*>(e.take(1, 8));
  if (!dcyc) return e.fail(UC_EBUDGET, "arena overflow");
  uint32_t rounds = rank_rounds(n);
  UC_CK(cudaMemsetAsync(cnt, 0, 64 * 4, e.stream));  // list counts (34 at most); the meetings at 48
  UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
  e.launches += 2;
  // results over the predecessors: walk a copy (the list that fills later)
  auto over = [&](const uint32_t* o) { return o < pred + n && pred < o + n; };
  const uint32_t* from = pred;
  if (over(head) || over(rank)) {
    UC_CK(cudaMemcpyAsync(a1, pred, n * 4, cudaMemcpyDeviceToDevice, e.stream));
    from = a1;
  }
  k_rank_walk<<<grid_for(e, (n + 3) / 4, 256), 256, 0, e.stream>>>(from, n, head, rank, X, a0, cnt);
  UC_CK(cudaGetLastError());
  int occ = 0;
  if (const int ro = occupancy(e, occ, k_rank_rest, 1024, 0)) return ro;
  const uint64_t want = (n + 1023) / 1024;
  const unsigned g = unsigned(std::max<uint64_t>(1, std::min<uint64_t>(want, uint64_t(e.sm_count) * std::max(1, occ))));
  uint32_t *bar = cnt + 48, *errp = &e.ctr->err;
  uint32_t most = n < RANK_DENSE ? uint32_t(n) : uint32_t(n - n / 4);
  void* args[] = {&X, &head, &rank, &a0, &a1, &cnt, &rounds, &most, &bar, &errp};
  UC_CK(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_rank_rest), dim3(g), dim3(1024), args, 0, e.stream));
  uint32_t* const hl = reinterpret_cast<uint32_t*>(e.h_io());  // the lists' sizes
  UC_CK(cudaMemcpyAsync(hl, cnt, (rounds + 1) * 4, cudaMemcpyDeviceToHost, e.stream));
  r = e.read_ctr();
  if (r) return r;
  if (hl[0] > most && !e.h_ctr->err) {
    const int grid = grid_for(e, n, 256);
    e.launches += 2 + rounds;
    k_rank_fill<<<grid, 256, 0, e.stream>>>(head, rank, n, X, cnt);
    for (uint32_t i = 0; i < rounds; ++i)
      k_rank_round<<<grid, 256, 0, e.stream>>>(X, i == 0 ? nullptr : (i & 1) ? a1 : a0, cnt + i, (i & 1) ? a0 : a1, cnt + i + 1);
    k_head_rank<<<grid, 256, 0, e.stream>>>(X, n, head, rank);
    UC_CK(cudaGetLastError());
    UC_CK(cudaMemcpyAsync(hl, cnt, (rounds + 1) * 4, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
  }
  if (e.h_ctr->err) {
    r = e.check_err(e.h_ctr);
    UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
    e.reset();
    return r;
  }
  const uint32_t hleft = hl[rounds];
  const uint32_t* act = (rounds & 1) ? a1 : a0;
  if (hleft) {
    UC_CK(cudaMemsetAsync(seen, 0, n, e.stream));
    UC_CK(cudaMemsetAsync(dcyc, 0, 8, e.stream));
    ++e.launches;
    if (k <= 31) k_vertex_cycles<1><<<1, 1, 0, e.stream>>>(act, hleft, succ, d_keys, n, head, rank, seen, dcyc);
    else k_vertex_cycles<2><<<1, 1, 0, e.stream>>>(act, hleft, succ, d_keys, n, head, rank, seen, dcyc);
    unsigned long long hc = 0;
    UC_CK(cudaMemcpyAsync(&hc, dcyc, 8, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    ncyc = hc;
  }
  e.reset();
  return UC_OK;
}

// emit() and emit_in() over scratch of emit_scratch_bytes(n) bytes.  With out
// null only the size: every member but a line's first adds one char.
static int emit_over(cudaStream_t s, int sm_count, const uint64_t* keys, const uint32_t* head, const uint32_t* rank,
                     uint64_t n, int k, char* out, uint64_t cap, uint64_t& out_bytes, char* scratch, uint32_t& launches,
                     std::string& err) {
  auto al = [](uint64_t b) { return (b + 255) & ~uint64_t(255); };
  const uint64_t tiles = (n + EMIT_TILE - 1) / EMIT_TILE;
  auto ck = [&](cudaError_t c, const char* what) -> int {
    if (c == cudaSuccess) return UC_OK;
    err = std::string(what) + ": " + cudaGetErrorString(c);
    return int(UC_ECUDA);
  };
  auto take = [&](uint64_t b) {
    char* p = scratch;
    scratch += al(b);
    return p;
  };
  // cleared: the control words (ticket, wait flag, long lines, heads), the
  // look-back words, the member counts
  const bool wide = n >= EMIT_WIDE;
  const uint64_t zero = 256 + tiles * (wide ? 16 : 8);
  char* z = take(zero);
  uint32_t* ctl = reinterpret_cast<uint32_t*>(z);
  unsigned long long* heads = reinterpret_cast<unsigned long long*>(z + 16);
  unsigned long long* st = reinterpret_cast<unsigned long long*>(z + 256);
  unsigned long long* base = reinterpret_cast<unsigned long long*>(take((tiles + 1) * 8));
  uint32_t* cnt = reinterpret_cast<uint32_t*>(take(n * 4));
  uint32_t* voff = reinterpret_cast<uint32_t*>(take(n * 4));
  uint32_t* huge = reinterpret_cast<uint32_t*>(take((n / EMIT_HUGE + 1) * 4));
  char* chars = take(n + 16);
  const uint64_t want = (n + 255) / 256, gcap = uint64_t(sm_count) * 16;
  const int grid = int(std::max<uint64_t>(1, std::min(want, gcap)));
  int r = ck(cudaMemsetAsync(z, 0, zero, s), "cudaMemsetAsync");
  if (r) return r;
  unsigned long long got = 0;
  if (!out) {
    ++launches;
    k_count_heads<<<grid, 256, 0, s>>>(head, n, heads);
    if ((r = ck(cudaGetLastError(), "launch"))) return r;
    if ((r = ck(cudaMemcpyAsync(&got, heads, 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync"))) return r;
    if ((r = ck(cudaStreamSynchronize(s), "cudaStreamSynchronize"))) return r;
    out_bytes = got * uint64_t(k) + n;
    return UC_OK;
  }
  if ((r = ck(cudaMemsetAsync(cnt, 0, n * 4, s), "cudaMemsetAsync"))) return r;
  launches += 2;
  k_count_members<<<grid, 256, 0, s>>>(head, n, cnt);
  if (wide) k_emit_scan<true><<<unsigned(tiles), 256, 0, s>>>(head, cnt, n, voff, base, st, ctl);
  else k_emit_scan<false><<<unsigned(tiles), 256, 0, s>>>(head, cnt, n, voff, base, st, ctl);
  if ((r = ck(cudaGetLastError(), "launch"))) return r;
  if ((r = ck(cudaMemcpyAsync(&got, base + tiles, 8, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync"))) return r;
  uint32_t c[3] = {0, 0, 0};
  if ((r = ck(cudaMemcpyAsync(c, ctl, 12, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync"))) return r;
  if ((r = ck(cudaStreamSynchronize(s), "cudaStreamSynchronize"))) return r;
  if (c[1]) {
    err = "a bounded device wait ran out";
    return UC_ETIMEOUT;
  }
  out_bytes = (got >> 32) * uint64_t(k) + (got & 0xFFFFFFFFull);
  if (out_bytes > cap) {
    err = "output buffer too small";
    return UC_EINPUT;
  }
  launches += 2;
  if (k <= 31) {
    k_emit_chars<1><<<grid, 256, 0, s>>>(keys, head, rank, voff, n, k, chars);
    k_emit_lines<1><<<unsigned(tiles), 256, 0, s>>>(keys, head, cnt, voff, chars, base, n, k, out, ctl, huge);
  } else {
    k_emit_chars<2><<<grid, 256, 0, s>>>(keys, head, rank, voff, n, k, chars);
    k_emit_lines<2><<<unsigned(tiles), 256, 0, s>>>(keys, head, cnt, voff, chars, base, n, k, out, ctl, huge);
  }
  if ((r = ck(cudaGetLastError(), "launch"))) return r;
  if ((r = ck(cudaMemcpyAsync(c, ctl, 12, cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync"))) return r;
  if ((r = ck(cudaStreamSynchronize(s), "cudaStreamSynchronize"))) return r;
  if (c[2]) {
    ++launches;
    k_emit_huge<<<unsigned(sm_count) * 4u, 256, 0, s>>>(head, cnt, voff, chars, base, k, out, huge, c[2]);
    if ((r = ck(cudaGetLastError(), "launch"))) return r;
    if ((r = ck(cudaStreamSynchronize(s), "cudaStreamSynchronize"))) return r;
  }
  return UC_OK;
}

uint64_t emit_scratch_bytes(uint64_t n) {
  auto al = [](uint64_t b) { return (b + 255) & ~uint64_t(255); };
  const uint64_t tiles = (n + EMIT_TILE - 1) / EMIT_TILE;
  return al(256 + tiles * (n >= EMIT_WIDE ? 16 : 8)) + al((tiles + 1) * 8) + 2 * al(n * 4) + al((n / EMIT_HUGE + 1) * 4) + al(n + 16);
}

int emit(Env& e, const uint64_t* d_keys, const uint32_t* succ, const uint32_t* head, const uint32_t* rank,
         uint64_t n, int k, char* out, uint64_t cap, uint64_t& out_bytes) {
  (void)succ;
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  out_bytes = 0;
  if (n == 0) return UC_OK;
  if (n > 0xFFFFFFFFull) return e.fail(UC_EINPUT, "too many k-mers for 32-bit ids");
  e.reset();
  int r = e.reserve(1, emit_scratch_bytes(n) + 4096);
  if (r) return r;
  char* scratch = static_cast<char*>(e.take(1, emit_scratch_bytes(n)));
  if (!scratch) return e.fail(UC_EBUDGET, "arena overflow");
  std::string err;
  r = emit_over(e.stream, e.sm_count, d_keys, head, rank, n, k, out, cap, out_bytes, scratch, e.launches, err);
  e.reset();
  return r ? e.fail(r, err) : UC_OK;
}

int emit_preload(std::string& err) {
  const void* fns[] = {
      reinterpret_cast<const void*>(k_count_members),
      reinterpret_cast<const void*>(k_count_heads),
      reinterpret_cast<const void*>(k_emit_scan<false>),
      reinterpret_cast<const void*>(k_emit_chars<1>),
      reinterpret_cast<const void*>(k_emit_chars<2>),
      reinterpret_cast<const void*>(k_emit_lines<1>),
      reinterpret_cast<const void*>(k_emit_lines<2>),
      reinterpret_cast<const void*>(k_emit_huge)};
  for (const void* f : fns) {
    cudaFuncAttributes a;
    const cudaError_t c = cudaFuncGetAttributes(&a, f);
    if (c != cudaSuccess) {
      cudaGetLastError();
      err = std::string("cudaFuncGetAttributes: ") + cudaGetErrorString(c);
      return UC_ECUDA;
    }
  }
  return UC_OK;
}

int emit_in(cudaStream_t s, int sm_count, const uint64_t* d_keys, const uint32_t* head, const uint32_t* rank,
            uint64_t n, int k, char* out, uint64_t cap, uint64_t& out_bytes, void* scratch, std::string& err) {
  out_bytes = 0;
  if (k < 2 || k > 63) {
    err = "k must be in [2, 63]";
    return UC_EINPUT;
  }
  if (n == 0) return UC_OK;
  uint32_t launches = 0;
  return emit_over(s, sm_count, d_keys, head, rank, n, k, out, cap, out_bytes, static_cast<char*>(scratch), launches,
                   err);
}

uint64_t output_bound(size_t text_bytes, int k) {
  (void)k;
  return uint64_t(text_bytes) + 64;
}

// Segment arrays of the fused path's stitch (in the back arena).
struct StitchBufs {
  SegRec* seg;
  unsigned long long* Xr;
  char* segc;
  uint32_t *act0, *act1;
  uint8_t* oncyc;
  uint32_t* hlen;
  unsigned long long* lbase;
  uint32_t* longl;  // heads of the lines the walk leaves (lcap entries)
  uint32_t lcap;
  uint32_t* rcnt;
  HecPool hp;
};

// Heads the walk can leave: each left line holds more than the walk's cap
// of cross ids.
static uint32_t walk_cap(const Env& e) {
  return (e.faults.walk_cap && e.faults.walk_cap < WALK_CAP) ? e.faults.walk_cap : WALK_CAP;
}
static uint64_t long_cap(const Env& e, uint64_t X) { return X / walk_cap(e) + 64; }

// The stitch's line walk alone, enqueued (its counters, walked and left, are zero before).
static int launch_walk(Env& e, const StitchBufs& b, uint64_t X, uint64_t Hp, int k, const JobDev& jd, char* out,
                       bool guard) {
  ++e.launches;
  k_walk_emit<<<grid_for(e, Hp, 256), 256, 0, e.stream>>>(uint32_t(Hp), b.seg, uint32_t(X), k, jd.tab, jd.jout, b.segc,
                                                          out, walk_cap(e), b.longl, b.lcap, guard ? 1 : 0, e.ctr);
  UC_CK(cudaGetLastError());
  return UC_OK;
}
// The cross-tile stitch over X cross-indexed segments and Hp head-pool ids,
// into out after each job's closed lines (jd.jout: each job's byte count,
// closed lines before, all lines after): the line walk, then, for the
// lines it leaves and for cycles, ranking (pointer jumping, or HEC with
// pointer jumping when its rounds run out), line lengths at the heads, one
// reservation per line, the segment copies, and the rare segment cycles.
// walked: the walk is done and its counters are in h_ctr.
static int run_stitch(Env& e, const StitchBufs& b, uint64_t X, uint64_t Hp, int k, int nw, bool want_hec,
                      uint32_t RH, const JobDev& jd, char* out, uint32_t& rounds, bool walked = false) {
  rounds = 0;
  const uint32_t S = uint32_t(X + Hp), nx = uint32_t(X), H = uint32_t(Hp);
  SegRec* seg = b.seg;
  unsigned long long* Xr = b.Xr;
  char* segc = b.segc;
  uint32_t *act0 = b.act0, *act1 = b.act1, *hlen = b.hlen, *rcnt = b.rcnt;
  uint8_t* oncyc = b.oncyc;
  unsigned long long* lbase = b.lbase;
  HecPool hp = b.hp;
  int r = UC_OK;
  const int gs = grid_for(e, S, 256);
  uint32_t *act = nullptr, *left = nullptr;
  uint32_t nlong = 0;
  if (!want_hec) {
    // the line walk writes every line its head reaches within WALK_CAP
    // segments; the rest is ranked from the first state, built below
    if (!walked) {
      UC_CK(cudaMemsetAsync(&e.ctr->walked, 0, 8, e.stream));  // walked, left
      r = launch_walk(e, b, X, Hp, k, jd, out, false);
      if (!r) r = e.read_ctr();
      if (r) return r;
      if (e.h_ctr->err) return e.check_err(e.h_ctr);
    }
    if (e.h_ctr->walked == nx && e.h_ctr->left == 0) return UC_OK;
    nlong = std::min(e.h_ctr->left, b.lcap);
    ++e.launches;
    k_set_u32<<<1, 1, 0, e.stream>>>(rcnt, nx);
  }
  // the first state (HEC's level 0 takes the predecessors from it)
  ++e.launches;
  k_seg_xinit<<<gs, 256, 0, e.stream>>>(S, seg, nx, k, Xr);
  bool hec = want_hec;
  if (hec) {
    UC_CK(cudaMemsetAsync(oncyc, 0, S, e.stream));
    r = hec_contract(e, hp, RH, nullptr, nullptr, nullptr, S, Xr, oncyc, seg, nx, k);
    if (r) return r;
    UC_CK(cudaMemsetAsync(rcnt, 0, 4, e.stream));
    ++e.launches;
    k_cycle_list<<<gs, 256, 0, e.stream>>>(oncyc, S, act0, rcnt);
    act = act0;
    left = rcnt;
    rounds = RH;
    r = e.read_ctr();
    if (r) return r;
    if (e.h_ctr->err) {  // did not finish in its pool/rounds: pointer jumping
      if (e.faults.hec_strict) return e.check_err(e.h_ctr);
      UC_CK(cudaMemsetAsync(&e.ctr->err, 0, 4, e.stream));
      hec = false;
    }
  }
  if (!hec) {
    // pointer-jumping rounds, captured as one graph: after the walk from the
    // state rebuilt above (over the ids [0, X)); after a HEC attempt from
    // the level-0 links the HEC pool kept
    uint32_t rr = 2;
    for (uint64_t t = 1; t < S; t <<= 1) ++rr;
    int rl = UC_OK;
    const bool prefilled = !want_hec;
    r = run_graph(e, 0, (uint64_t(rr) << 33) | (uint64_t(prefilled) << 32) | uint32_t(gs), [&] {
      rl = prefilled ? rank_lists(e, nullptr, nullptr, S, Xr, act0, act1, rcnt, rounds, act, left, true)
                     : rank_lists(e, hp.prv, hp.wt, S, Xr, act0, act1, rcnt, rounds, act, left);
      cudaMemsetAsync(oncyc, 0, S, e.stream);
      ++e.launches;
      k_mark_cycle<<<gs, 256, 0, e.stream>>>(act, left, oncyc);
    });
    if (r) return r;
    if (rl) return rl;
  }
  // line length at each head, one reservation per line not yet written,
  // then every segment's chars (the segments of written lines skip)
  UC_CK(cudaMemsetAsync(hlen, 0, size_t(H) * 4, e.stream));
  UC_CK(cudaMemsetAsync(lbase, 0xFF, size_t(H) * 8, e.stream));
  e.launches += 2;
  k_chain_len<<<gs, 256, 0, e.stream>>>(S, seg, Xr, oncyc, nx, k, hlen, e.ctr);
  if (want_hec) {
    ++e.launches;
    k_line_reserve<<<grid_for(e, H, 256), 256, 0, e.stream>>>(H, nullptr, seg + nx, jd.tab, jd.jout, hlen, lbase,
                                                              e.ctr);
  } else if (nlong) {
    ++e.launches;
    k_line_reserve<<<grid_for(e, nlong, 256), 256, 0, e.stream>>>(nlong, b.longl, seg + nx, jd.tab, jd.jout, hlen,
                                                                  lbase, e.ctr);
  }
  k_seg_copy<<<grid_for(e, S, 256), 256, 0, e.stream>>>(S, seg, Xr, oncyc, nx, lbase, segc, out, k);
  uint32_t hleft = 0;
  UC_CK(cudaMemcpyAsync(&hleft, left, 4, cudaMemcpyDeviceToHost, e.stream));
  UC_CK(cudaStreamSynchronize(e.stream));
  if (hleft) {
    ++e.launches;
    if (nw == 1)
      k_seg_cycles<1><<<1, 1, 0, e.stream>>>(e.ctr, S, act, hleft, oncyc, seg, jd.tab, jd.jout, segc, out, k);
    else
      k_seg_cycles<2><<<1, 1, 0, e.stream>>>(e.ctr, S, act, hleft, oncyc, seg, jd.tab, jd.jout, segc, out, k);
  }
  UC_CK(cudaGetLastError());
  return UC_OK;
}

// Back arena bytes of the fused path: the bucketed copies and their staging,
// the segment pool (Sp segments for X cross k-mers) and the stitch arrays.
static size_t back_bytes(const Env& e, uint64_t copies, uint64_t X, uint64_t Sp, int nw, int k, bool want_hec) {
  const uint64_t segchars = Sp * uint64_t(k) + copies + 64;
  const uint32_t R = 64;
  size_t back = 0;
  auto add = [&](size_t b) { back += (b + 255) & ~size_t(255); };
  const uint64_t Hp = Sp - X;                                             // head pools
  add(scatter_stage_bytes(copies, nw)); add(scatter_stage_bytes(copies, nw));  // the scatter's two regions
  add(Sp * sizeof(SegRec)); add(Sp * 8);                                  // segment records, ranking
  add(segchars);
  add(Sp * 4); add(Sp * 4); add(Sp);                                      // act0, act1, oncyc
  add(Hp * 4); add(Hp * 8); add(long_cap(e, X) * 4);                         // line lengths, bases, left lines
  add(R * 4);
  if (want_hec) add(hec_bytes(Sp, hec_rounds(Sp)));
  return back;
}

void batch_footprint(const Env& e, uint32_t njobs, const size_t* bytes, int k, int l, size_t& front,
                     size_t& back) {
  const int nw = (k <= 31) ? 1 : 2;
  uint64_t N = 0, nmax = 0, tb = 0;
  for (uint32_t j = 0; j < njobs; ++j) {
    const uint64_t n = (uint64_t(bytes[j]) + 1) / uint64_t(k + 1) + 1;
    N += n;
    nmax = std::max(nmax, n);
    tb = std::max<uint64_t>(tb, bytes[j]);
  }
  const Plan P = plan_buckets(e, nmax, njobs, k, l);
  const size_t slack = size_t(16) << 20;
  front = front_bytes(N, nw, P.M, true) + slack + 4096;
  const uint64_t X = N, copies = N + X, Sp = 2 * X + njobs;
  back = std::max(back_bytes(e, copies, X, Sp, nw, k, e.tune.contract_method == UC_CONTRACT_HEC),
                  line_index_bytes(tb, nmax)) + slack + 4096;
}

// The fused path.  Device memory: the front arena holds per-k-mer arrays
// (keys, bucket ids) and per-bucket arrays; the back arena, sized once the
// cross k-mers X are counted, holds the n+X bucketed copies and the segment
// arrays (at most 2X open segments: each holds an S-only start or a P-only
// end, one of each per cross k-mer).
// The fused path over a batch of jobs (one job is a batch of one).  Device
// memory: the front arena holds per-k-mer arrays (keys, bucket ids) and
// per-bucket arrays; the back arena, sized once the cross k-mers are counted,
// holds the bucketed copies and the segment pools (a job with X cross k-mers
// has at most 2X open segments: each holds an S-only start or a P-only end).
//
// recs (a batch of one job whose lines are sorted next): the warp tiles' closed
// lines are left as records in the scatter's spare region; out_len counts the
// text lines alone.
static int compact_jobs(Env& e, uint32_t njobs, const char* const* texts, const size_t* bytes, int k, int l, char* out,
                        uint64_t out_cap, uint64_t* out_off, uint64_t* out_len, uc_stats* st, LineRecs* recs,
                        bool lean = false) {
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  if (l < 1 || l > 16 || l > k - 1) return e.fail(UC_EINPUT, "l must be in [1, min(16, k-1)]");
  if (njobs == 0) return UC_OK;
  const int nw = (k <= 31) ? 1 : 2;
  e.reset();
  e.launches = 0;
  e.graph_nodes = 0;
  e.timed = st != nullptr;
  e.tiles_timed = false;
  auto mark = [&](int i) {
    if (e.timed) cudaEventRecord(e.ev[i], e.stream);
  };
  int r = job_buffers(e, njobs);
  if (r) return r;
  JobDev jd = job_dev(e, njobs);
  std::vector<JobTab> J(njobs);
  if (njobs == 1) {
    r = host_job(e, texts[0], bytes[0], k, J[0]);
    if (r) return r;
  } else {
    for (uint32_t j = 0; j < njobs; ++j) {
      J[j] = JobTab{};
      J[j].text = reinterpret_cast<const uint8_t*>(texts[j]);
      J[j].tbytes = bytes[j];
    }
    UC_CK(cudaMemcpyAsync(jd.tab, J.data(), njobs * sizeof(JobTab), cudaMemcpyHostToDevice, e.stream));
    ++e.launches;
    k_headers<<<(njobs + 127) / 128, 128, 0, e.stream>>>(jd.tab, njobs, k);
    UC_CK(cudaMemcpyAsync(J.data(), jd.tab, njobs * sizeof(JobTab), cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    for (uint32_t j = 0; j < njobs; ++j) {
      if (J[j].err) return e.fail(UC_EINPUT, "job " + std::to_string(j) + ": missing or too large k-mer count");
      if (!J[j].fixed)
        return e.fail(UC_EINPUT, "job " + std::to_string(j) +
                                     ": batched jobs need k chars + '\\n' per line and a matching count");
    }
  }
  uint64_t N = 0, lb = 0, ob = 0, nmax = 0;
  for (uint32_t j = 0; j < njobs; ++j) {
    J[j].koff = N;
    J[j].lb0 = lb;
    J[j].obase = ob;
    J[j].ocap = output_bound(bytes[j], k);
    N += J[j].n;
    lb += (J[j].n + PACK_LINES - 1) / PACK_LINES;
    ob += (J[j].ocap + 15) & ~uint64_t(15);
    nmax = std::max<uint64_t>(nmax, J[j].n);
  }
  if (N >= 0x7FFFFFFFull) return e.fail(UC_EINPUT, "too many k-mers for 31-bit ids");
  if (ob > out_cap + 15) return e.fail(UC_EINPUT, "output buffer smaller than uc_output_bound");
  const Plan P = plan_buckets(e, nmax, njobs, k, l, lean);
  r = e.reserve(0, front_bytes(N, nw, P.M, true));
  if (r) return r;
  Front f{};
  r = take_front(e, N, nw, P.M, true, f);
  if (r) return r;
  // the pack's counts: per group of 2^cg buckets, or (cg = 0) per bucket
  const uint64_t G = P.M >> P.cg;
  uint32_t* gcount = P.cg ? f.gcount : f.counts;
  unsigned long long* goff = P.cg ? f.goff : f.boff;
  r = clear_counters(e);
  if (r) return r;
  UC_CK(cudaMemsetAsync(gcount, 0, G * 4, e.stream));
  // the per-job counters (jout, jseg, jclosed, jcross) in one piece
  const size_t jbytes = size_t(reinterpret_cast<char*>(jd.jcross + njobs) - reinterpret_cast<char*>(jd.jout));
  UC_CK(cudaMemsetAsync(jd.jout, 0, jbytes, e.stream));
  // their copy on the host: pinned where it fits
  std::vector<char> jhost(jbytes <= Env::HOST_IO - 1024 ? 0 : jbytes);
  char* const jh = jhost.empty() ? e.h_io() + 1024 : jhost.data();
  auto on_host = [&](const void* p) { return jh + (static_cast<const char*>(p) - reinterpret_cast<char*>(jd.jout)); };
  // counters and per-job counters to the host (waits)
  auto read_back = [&]() -> int {
    UC_CK(cudaMemcpyAsync(jh, jd.jout, jbytes, cudaMemcpyDeviceToHost, e.stream));
    return e.read_ctr();
  };
  if (njobs > 1)
    UC_CK(cudaMemcpyAsync(jd.tab, J.data(), njobs * sizeof(JobTab), cudaMemcpyHostToDevice, e.stream));
  mark(0);
  FuseArgs fz;
  fz.l = P.l_used;
  fz.seed = e.seed;
  fz.jb = P.jb;
  fz.b1 = f.b1;
  fz.b2 = f.b2;
  fz.counts = gcount;
  fz.cshift = P.cg;
  fz.cbytes = G * 4;
  fz.jcross = jd.jcross;
  fz.M = P.M;
  if (njobs == 1) {
    r = pack_single(e, texts[0], bytes[0], k, f.keys, &fz, J[0], jd.tab, J[0].fixed != 0);
    if (r) return r;
  } else if (N > 0) {
    if (nw == 1) launch_pack<1>(e, jd.tab, nullptr, njobs, lb, nullptr, k, f.keys, &fz);
    else launch_pack<2>(e, jd.tab, nullptr, njobs, lb, nullptr, k, f.keys, &fz);
    UC_CK(cudaGetLastError());
  }
  if (e.timed || e.after_pack) cudaEventRecord(e.ev[1], e.stream);
  r = launch_bucket_offsets(e, gcount, G, goff);
  if (!r) r = read_back();
  if (r) return r;
  if (njobs == 1 && J[0].fixed && (e.h_ctr->err & ERR_LAYOUT)) {
    // not k chars and a break per line after all: again, from the line starts
    J[0].fixed = 0;
    r = clear_counters(e);
    if (r) return r;
    UC_CK(cudaMemsetAsync(gcount, 0, G * 4, e.stream));
    UC_CK(cudaMemsetAsync(jd.jout, 0, jbytes, e.stream));
    r = pack_single(e, texts[0], bytes[0], k, f.keys, &fz, J[0], jd.tab);
    if (r) return r;
    if (e.timed || e.after_pack) cudaEventRecord(e.ev[1], e.stream);
    r = launch_bucket_offsets(e, gcount, G, goff);
    if (!r) r = read_back();
    if (r) return r;
  }
  const uint64_t copies = e.h_ctr->copies;
  const uint32_t* xc = reinterpret_cast<const uint32_t*>(on_host(jd.jcross));
  uint64_t xsum = 0;
  for (uint32_t j = 0; j < njobs; ++j) xsum += xc[j];
  if (copies != N + xsum && !e.h_ctr->err) return e.fail(UC_EINTERNAL, "bucket counts disagree with the copies");
  if (e.h_ctr->err) {
    if (e.h_ctr->err & ERR_LAYOUT) return e.fail(UC_EINPUT, "a k-mer line is shorter than k");
    return e.check_err(e.h_ctr);
  }
  const uint64_t X = copies - N;
  // segment ids: [0, X) the segments that start at a cross k-mer's S-only
  // copy; then each job's head pool (a line's first open segment ends at a
  // P-only copy, so a job has at most one per cross k-mer)
  uint64_t Hp = 0;
  for (uint32_t j = 0; j < njobs; ++j) {
    J[j].seg_base = uint32_t(Hp);
    J[j].seg_cap = xc[j] + 1;
    Hp += J[j].seg_cap;
  }
  const uint64_t Sp = X + Hp;
  if (Sp >= 0x7FFFFFF0ull) return e.fail(UC_EINPUT, "too many cross-tile segments");
  if (njobs >= (1u << (64 - SEG_OFF_BITS))) return e.fail(UC_EINPUT, "too many jobs in one batch");
  if (njobs == 1) {
    // (pinned: the copy does not wait)
    static_assert(sizeof(JobTab) <= 512, "the job fits the pinned area");
    JobTab* hj = reinterpret_cast<JobTab*>(e.h_io() + 512);
    *hj = J[0];
    UC_CK(cudaMemcpyAsync(jd.tab, hj, sizeof(JobTab), cudaMemcpyHostToDevice, e.stream));
  } else {
    UC_CK(cudaMemcpyAsync(jd.tab, J.data(), njobs * sizeof(JobTab), cudaMemcpyHostToDevice, e.stream));
  }
  const uint64_t segchars = Sp * uint64_t(k) + copies + 64;
  if (segchars > SEG_OFF_MASK) return e.fail(UC_EINPUT, "segment chars beyond the 40-bit offsets");
  const uint32_t R = 64;
  const bool want_hec = e.tune.contract_method == UC_CONTRACT_HEC;
  const uint32_t RH = hec_rounds(e, Sp);
  const size_t back = back_bytes(e, copies, X, Sp, nw, k, want_hec);
  // (half of the k-mers start a line at most in canonical input)
  const int rbits = recs ? line_bin_bits(N / 2, k) : 0;
  r = e.reserve(1, back);
  if (!lean && e.too_large(r) && plan_buckets(e, nmax, njobs, k, l, true).l_used < P.l_used)
    return compact_jobs(e, njobs, texts, bytes, k, l, out, out_cap, out_off, out_len, st, recs, true);
  if (r) return r;
  if (e.after_pack) e.after_pack();
  auto T64 = [&](uint64_t c) { return static_cast<unsigned long long*>(e.take(1, c * 8)); };
  auto T32 = [&](uint64_t c) { return static_cast<uint32_t*>(e.take(1, c * 4)); };
  char* region1 = static_cast<char*>(e.take(1, scatter_stage_bytes(copies, nw)));
  char* region2 = static_cast<char*>(e.take(1, scatter_stage_bytes(copies, nw)));
  SegRec* seg = static_cast<SegRec*>(e.take(1, Sp * sizeof(SegRec)));
  unsigned long long* Xr = T64(Sp);
  char* segc = static_cast<char*>(e.take(1, segchars));
  uint32_t* act0 = T32(Sp);
  uint32_t* act1 = T32(Sp);
  uint8_t* oncyc = static_cast<uint8_t*>(e.take(1, Sp));
  uint32_t* hlen = T32(Hp);
  unsigned long long* lbase = T64(Hp);
  uint32_t* longl = T32(long_cap(e, X));
  uint32_t* rcnt = T32(R);
  if (!rcnt) return e.fail(UC_EBUDGET, "back arena overflow");
  HecPool hp{};
  if (want_hec) {
    r = hec_take(e, Sp, RH, hp);
    if (r) return r;
  }
  // unused head-pool ids keep length 0 (every id below X gets a record)
  UC_CK(cudaMemsetAsync(seg + X, 0, Hp * sizeof(SegRec), e.stream));
  uint64_t* pkeys = nullptr;
  uint32_t* plink = nullptr;
  r = plan_and_scatter(e, f, P, N, nw, 0, region1, region2, copies, pkeys, plink, P.cg > 0);
  if (r) return r;
  mark(2);

  TileParams tp{};
  tp.pkeys = pkeys;
  tp.plink = plink;
  tp.tile_begin = f.tile_begin;
  tp.tile_job = f.tile_job;
  tp.ctr = e.ctr;
  tp.k = k;
  tp.cap = P.cap;
  tp.tslots = P.tslots;
  tp.lf = P.lf;
  tp.wlf = P.wlf;
  tp.wcap = P.wcap;
  tp.wts = P.wts;
  tp.wbytes = P.wbytes;
  tp.mode = 1;
  tp.out = out;
  tp.segchars = segc;
  tp.segchars_cap = segchars - 64;  // the line walk reads up to 7 bytes past a segment's chars
  tp.seg = seg;
  tp.xcount = uint32_t(X);
  tp.jobs = jd.tab;
  tp.jout = jd.jout;
  tp.jseg = jd.jseg;
  if (recs) {
    // the scatter's region that does not hold the copies
    recs->a = reinterpret_cast<char*>(pkeys) == region1 ? region2 : region1;
    recs->cap = copies;
    recs->kmers = N;
    // (no more of them than a sixteenth of the lines, or 16)
    recs->counts = reinterpret_cast<uint32_t*>(f.keys);
    recs->bits = rbits;
    UC_CK(cudaMemsetAsync(recs->counts, 0, size_t(4) << rbits, e.stream));
    tp.rec_a = reinterpret_cast<ulonglong2*>(recs->a);
    tp.rec_t = reinterpret_cast<unsigned long long*>(tp.rec_a + copies);
    tp.rec_counts = recs->counts;
    tp.rec_bits = rbits;
  }
  const uint32_t threads = e.tune.tile_threads ? e.tune.tile_threads : 512;
  // The tiles, and behind them, before the host knows that none is oversized,
  // the line walk (which does nothing when one is): one wait for both.
  uint32_t rounds = 0;
  StitchBufs sbuf{seg, Xr, segc, act0, act1, oncyc, hlen, lbase, longl, uint32_t(long_cap(e, X)), rcnt, hp};
  auto closed_now = [&]() -> int {
    if (st) UC_CK(cudaMemcpyAsync(jd.jclosed, jd.jout, njobs * 8, cudaMemcpyDeviceToDevice, e.stream));
    mark(3);
    return UC_OK;
  };
  bool stitched = false;
  r = launch_tiles(e, tp, f, threads, nw);
  if (!r) r = closed_now();
  if (!r && !want_hec) r = launch_walk(e, sbuf, X, Hp, k, jd, out, true);
  mark(4);
  if (!r) r = read_back();
  if (r) return r;
  if (e.h_ctr->err) return e.check_err(e.h_ctr);
  const uint32_t nbig = e.h_ctr->nbig;
  if (nbig) {
    r = run_big_tiles(e, tp, f, nw, nbig);
    if (!r) r = closed_now();
    if (r) return r;
  } else {
    stitched = !want_hec && e.h_ctr->walked == X && e.h_ctr->left == 0;
  }
  if (!stitched) {
    r = run_stitch(e, sbuf, X, Hp, k, nw, want_hec, RH, jd, out, rounds, !nbig && !want_hec);
    mark(4);
    if (!r) r = read_back();
    if (r) return r;
    if (e.h_ctr->err) return e.check_err(e.h_ctr);
  }
  const unsigned long long* jo = reinterpret_cast<const unsigned long long*>(on_host(jd.jout));
  const unsigned long long* jc = reinterpret_cast<const unsigned long long*>(on_host(jd.jclosed));
  uint64_t total = 0;
  if (recs) {
    recs->n = uint32_t(e.h_ctr->rec_slots);
    recs->bytes = total = e.h_ctr->rec_bytes;
    if (jo[0] + total > J[0].ocap) return e.fail(UC_EINTERNAL, "output bound exceeded");
  }
  for (uint32_t j = 0; j < njobs; ++j) {
    if (jo[j] > J[j].ocap) return e.fail(UC_EINTERNAL, "output bound exceeded");
    if (out_off) out_off[j] = J[j].obase;
    if (out_len) out_len[j] = jo[j];
    total += jo[j];
  }
  if (st) {
    st->n_kmers = N;
    st->n_copies = copies;
    st->n_cross = X;
    st->n_tiles = e.h_ctr->ntiles;
    st->n_big_tiles = e.h_ctr->nbig;
    st->n_segments = Sp;
    st->n_cycles = e.h_ctr->cycles;
    st->closed_bytes = recs ? recs->bytes : 0;
    for (uint32_t j = 0; j < njobs; ++j) st->closed_bytes += jc[j];
    st->seg_chars = e.h_ctr->seg_char_cursor;
    st->out_bytes = total;
    st->stitch_rounds = rounds;
    st->l_used = uint32_t(P.l_used);
    st->bucket_bits = P.bits;
    st->tile_capacity = P.cap;
    st->launches = e.launches;
    st->graph_nodes = e.graph_nodes;
    float a = 0, b = 0, c = 0, d = 0;
    cudaEventElapsedTime(&a, e.ev[0], e.ev[1]);
    cudaEventElapsedTime(&b, e.ev[1], e.ev[2]);
    cudaEventElapsedTime(&c, e.ev[2], e.ev[3]);
    cudaEventElapsedTime(&d, e.ev[3], e.ev[4]);
    st->ms_pack = a;
    st->ms_bucket = b;
    st->ms_tiles = c;
    st->ms_stitch = d;
    st->ms_total = a + b + c + d;
    if (e.tiles_timed) {
      cudaEventElapsedTime(&st->ms_tile_warp, e.ev[8], e.ev[9]);
      cudaEventElapsedTime(&st->ms_tile_block, e.ev[9], e.ev[5]);
    }
  }
  e.reset();
  return UC_OK;
}

int compact_batch(Env& e, uint32_t njobs, const char* const* texts, const size_t* bytes, int k, int l, char* out,
                  uint64_t out_cap, uint64_t* out_off, uint64_t* out_len, uc_stats* st) {
  return compact_jobs(e, njobs, texts, bytes, k, l, out, out_cap, out_off, out_len, st, nullptr);
}

// The streamed form of the fused path, for a job from host memory whose text
// and lines do not fit in device memory beside the working arrays.  The text
// goes to the device in chunks of whole lines, twice: the first pass counts
// the buckets (the 16-bit counts, taken again at 32 bits in a third pass if
// one wrapped), the second builds the bucketed copies (level 1 of the
// scatter per chunk, its cursors carried over; levels 2 and 3 once).  The
// tiles then run in groups of whole tiles; each group's closed lines go back
// to host memory before the next group, while the open segments stay on the
// device for the stitch, whose lines follow.  The device holds one chunk's
// text, keys and buckets, the copies' two scatter regions, the segment
// arrays and the output of one tile group; k-mer indices are 64-bit
// throughout (the reference's LARGE/HUGE widths, defs.h:30-42), cross
// indices and segment ids 31-bit.  Lines must be k chars + '\n' (the layout
// the chunks are cut on).  Unsorted output only.
int compact_streamed(Env& e, const char* h_text, size_t bytes, int k, int l, char* h_out, uint64_t cap,
                     uint64_t& out_bytes, uc_stats* st, uint64_t chunk_lines, uint64_t group_copies, bool lean) {
  out_bytes = 0;
  if (k < 2 || k > 63) return e.fail(UC_EINPUT, "k must be in [2, 63]");
  if (l < 1 || l > 16 || l > k - 1) return e.fail(UC_EINPUT, "l must be in [1, min(16, k-1)]");
  if (e.sorted) return e.fail(UC_EINPUT, "the streamed path writes unsorted output");
  const int nw = (k <= 31) ? 1 : 2;
  const uint64_t stride = uint64_t(k) + 1;
  // count line (driver.cpp:296-304) and the fixed line layout
  size_t p = 0;
  while (p < bytes && (h_text[p] == ' ' || h_text[p] == '\t' || h_text[p] == '\r')) ++p;
  if (p >= bytes || h_text[p] < '0' || h_text[p] > '9') return e.fail(UC_EINPUT, "missing k-mer count header");
  uint64_t n = 0;
  while (p < bytes && h_text[p] >= '0' && h_text[p] <= '9') {
    n = n * 10 + uint64_t(h_text[p] - '0');
    if (n > (1ull << 40)) return e.fail(UC_EINPUT, "k-mer count too large");
    ++p;
  }
  while (p < bytes && h_text[p] != '\n') ++p;
  const uint64_t body = (p < bytes) ? p + 1 : bytes;
  uint64_t end = bytes;
  while (end > body && (h_text[end - 1] == '\n' || h_text[end - 1] == '\r')) --end;
  if (!((n == 0 && end == body) || (n > 0 && end - body == n * stride - 1)))
    return e.fail(UC_EINPUT, "the streamed path needs k chars + '\\n' per line and a matching count");
  e.reset();
  e.launches = 0;
  e.graph_nodes = 0;
  e.timed = true;
  if (n == 0) return UC_OK;
  if (!chunk_lines) chunk_lines = 64ull << 20;
  if (!group_copies) group_copies = 256ull << 20;
  chunk_lines = std::min(chunk_lines, n);
  const Plan P = plan_buckets(e, n, 1, k, l, lean);
  const size_t chunk_text = size_t(chunk_lines * stride + 64);
  int r = e.reserve(0, front_bytes(chunk_lines, nw, P.M, true) + chunk_text + 4096);
  if (r) return r;
  Front f{};
  r = take_front(e, chunk_lines, nw, P.M, true, f);
  if (r) return r;
  char* d_chunk = static_cast<char*>(e.take(0, chunk_text));
  if (!d_chunk) return e.fail(UC_EBUDGET, "front arena overflow");
  r = job_buffers(e, 1);
  if (r) return r;
  JobDev jd = job_dev(e, 1);
  r = clear_counters(e);
  if (r) return r;
  UC_CK(cudaMemsetAsync(f.c16, 0, (P.M + 1) / 2 * 4, e.stream));
  UC_CK(cudaMemsetAsync(jd.jcross, 0, 4, e.stream));
  FuseArgs fz;
  fz.l = P.l_used;
  fz.seed = e.seed;
  fz.jb = P.jb;
  fz.b1 = f.b1;
  fz.b2 = f.b2;
  fz.M = P.M;
  // one chunk of lines to the device and packed (fz.counts / fz.jcross null:
  // buckets only)
  auto pack_chunk = [&](uint64_t c0, uint64_t cl, uint32_t* counts, uint32_t* jcross) -> int {
    const uint64_t src = body + c0 * stride;
    const uint64_t len = std::min<uint64_t>(cl * stride, uint64_t(bytes) - src);
    UC_CK(cudaMemcpyAsync(d_chunk, h_text + src, len, cudaMemcpyHostToDevice, e.stream));
    JobTab J{};
    J.text = reinterpret_cast<const uint8_t*>(d_chunk);
    J.tbytes = len;
    J.body = 0;
    J.end = cl * stride - 1;
    J.n = cl;
    J.fixed = 1;
    FuseArgs z = fz;
    z.counts = counts;
    z.jcross = jcross;
    const uint64_t nblocks = (cl + PACK_LINES - 1) / PACK_LINES;
    if (nw == 1) launch_pack<1>(e, jd.tab, &J, 1, nblocks, nullptr, k, f.keys, &z);
    else launch_pack<2>(e, jd.tab, &J, 1, nblocks, nullptr, k, f.keys, &z);
    UC_CK(cudaGetLastError());
    return UC_OK;
  };
  cudaEventRecord(e.ev[0], e.stream);
  for (uint64_t c0 = 0; c0 < n; c0 += chunk_lines) {
    r = pack_chunk(c0, std::min(chunk_lines, n - c0), f.c16, jd.jcross);
    if (r) return r;
  }
  r = e.read_ctr();
  if (r) return r;
  if (e.h_ctr->err) {
    if (e.h_ctr->err & ERR_LAYOUT) return e.fail(UC_EINPUT, "a k-mer line is shorter than k");
    return e.check_err(e.h_ctr);
  }
  cudaEventRecord(e.ev[1], e.stream);
  ++e.launches;
  k_widen16<<<grid_for(e, P.M, 256), 256, 0, e.stream>>>(f.c16, P.M, f.counts);
  uint64_t copies = 0;
  r = bucket_offsets(e, f, P.M, copies);
  if (r) return r;
  uint32_t xc = 0;
  UC_CK(cudaMemcpyAsync(&xc, jd.jcross, 4, cudaMemcpyDeviceToHost, e.stream));
  UC_CK(cudaStreamSynchronize(e.stream));
  if (copies != n + xc) {
    // a bucket holds 65536 copies or more: count again at 32 bits
    UC_CK(cudaMemsetAsync(f.counts, 0, P.M * 4, e.stream));
    for (uint64_t c0 = 0; c0 < n; c0 += chunk_lines) {
      const uint64_t cl = std::min(chunk_lines, n - c0);
      r = pack_chunk(c0, cl, nullptr, nullptr);
      if (r) return r;
      ++e.launches;
      k_count_buckets<<<grid_for(e, cl, 256), 256, 0, e.stream>>>(f.b1, f.b2, cl, f.counts);
    }
    r = bucket_offsets(e, f, P.M, copies);
    if (r) return r;
  }
  const uint64_t X = copies - n;
  const uint64_t Hp = X + 1;
  const uint64_t Sp = X + Hp;
  if (Sp >= 0x7FFFFFF0ull) return e.fail(UC_EINPUT, "too many cross-tile segments");
  const uint64_t segchars = Sp * uint64_t(k) + copies + 64;
  if (segchars > SEG_OFF_MASK) return e.fail(UC_EINPUT, "segment chars beyond the 40-bit offsets");
  // the tiles, grouped: whole tiles up to group_copies copies (a larger tile
  // alone); a group's closed lines fit its copies' lines
  r = plan_tiles(e, f, P, nw, false);
  if (r) return r;
  r = e.read_ctr();
  if (r) return r;
  const uint32_t ntiles = e.h_ctr->ntiles;
  std::vector<unsigned long long> tb(size_t(ntiles) + 1);
  UC_CK(cudaMemcpyAsync(tb.data(), f.tile_begin, (size_t(ntiles) + 1) * 8, cudaMemcpyDeviceToHost, e.stream));
  UC_CK(cudaStreamSynchronize(e.stream));
  std::vector<uint32_t> groups{0};
  uint64_t gmax = 0;
  for (uint32_t t = 0; t < ntiles;) {
    const uint32_t g0 = t;
    do {
      ++t;
    } while (t < ntiles && tb[t + 1] - tb[g0] <= group_copies);
    groups.push_back(t);
    gmax = std::max<uint64_t>(gmax, tb[t] - tb[g0]);
  }
  const uint64_t gout = gmax * stride + 64;
  const uint64_t sout = segchars + Sp + 64;  // stitched lines: segment chars and a break each at most
  const uint32_t R = 64;
  const bool want_hec = e.tune.contract_method == UC_CONTRACT_HEC;
  const uint32_t RH = hec_rounds(e, Sp);
  r = e.reserve(1, back_bytes(e, copies, X, Sp, nw, k, want_hec) + gout + sout + 4096);
  if (!lean && e.too_large(r) && plan_buckets(e, n, 1, k, l, true).l_used < P.l_used)
    return compact_streamed(e, h_text, bytes, k, l, h_out, cap, out_bytes, st, chunk_lines, group_copies, true);
  if (r) return r;
  auto T64 = [&](uint64_t c) { return static_cast<unsigned long long*>(e.take(1, c * 8)); };
  auto T32 = [&](uint64_t c) { return static_cast<uint32_t*>(e.take(1, c * 4)); };
  char* region1 = static_cast<char*>(e.take(1, scatter_stage_bytes(copies, nw)));
  char* region2 = static_cast<char*>(e.take(1, scatter_stage_bytes(copies, nw)));
  SegRec* seg = static_cast<SegRec*>(e.take(1, Sp * sizeof(SegRec)));
  unsigned long long* Xr = T64(Sp);
  char* segc = static_cast<char*>(e.take(1, segchars));
  uint32_t* act0 = T32(Sp);
  uint32_t* act1 = T32(Sp);
  uint8_t* oncyc = static_cast<uint8_t*>(e.take(1, Sp));
  uint32_t* hlen = T32(Hp);
  unsigned long long* lbase = T64(Hp);
  uint32_t* longl = T32(long_cap(e, X));
  uint32_t* rcnt = T32(R);
  char* d_gout = static_cast<char*>(e.take(1, gout));
  char* d_sout = static_cast<char*>(e.take(1, sout));
  if (!d_sout) return e.fail(UC_EBUDGET, "back arena overflow");
  HecPool hp{};
  if (want_hec) {
    r = hec_take(e, Sp, RH, hp);
    if (r) return r;
  }
  UC_CK(cudaMemsetAsync(seg + X, 0, Hp * sizeof(SegRec), e.stream));
  UC_CK(cudaMemsetAsync(jd.jseg, 0, 4, e.stream));
  // the bucketed copies: level 1 chunk by chunk, then levels 2 and 3
  Scatter sc;
  r = scatter_begin(e, f, P, nw, region1, region2, copies, sc);
  if (r) return r;
  for (uint64_t c0 = 0; c0 < n; c0 += chunk_lines) {
    const uint64_t cl = std::min(chunk_lines, n - c0);
    r = pack_chunk(c0, cl, nullptr, nullptr);
    if (r) return r;
    r = scatter_l1(e, f, sc, f.keys, f.b1, f.b2, cl, 0);
    if (r) return r;
  }
  uint64_t* pkeys = nullptr;
  uint32_t* plink = nullptr;
  r = scatter_finish(e, f, sc, pkeys, plink);
  if (r) return r;
  cudaEventRecord(e.ev[2], e.stream);
  // one job whose region is a tile group's output buffer
  JobTab J{};
  J.n = n;
  J.obase = 0;
  J.ocap = gout;
  J.seg_base = 0;
  J.seg_cap = uint32_t(Hp);
  UC_CK(cudaMemcpyAsync(jd.tab, &J, sizeof(JobTab), cudaMemcpyHostToDevice, e.stream));
  TileParams tp{};
  tp.pkeys = pkeys;
  tp.plink = plink;
  tp.tile_begin = f.tile_begin;
  tp.tile_job = f.tile_job;
  tp.ctr = e.ctr;
  tp.k = k;
  tp.cap = P.cap;
  tp.tslots = P.tslots;
  tp.lf = P.lf;
  tp.wlf = P.wlf;
  tp.wcap = P.wcap;
  tp.wts = P.wts;
  tp.wbytes = P.wbytes;
  tp.mode = 1;
  tp.out = d_gout;
  tp.segchars = segc;
  tp.segchars_cap = segchars - 64;  // the line walk reads up to 7 bytes past a segment's chars
  tp.seg = seg;
  tp.xcount = uint32_t(X);
  tp.jobs = jd.tab;
  tp.jout = jd.jout;
  tp.jseg = jd.jseg;
  const uint32_t threads = e.tune.tile_threads ? e.tune.tile_threads : 512;
  uint64_t closed = 0;
  float ms_tiles = 0;
  for (size_t g = 0; g + 1 < groups.size(); ++g) {
    // per group: the tier lists and their counters, the group's line cursor
    UC_CK(cudaMemsetAsync(&e.ctr->tile_next, 0, 4, e.stream));
    UC_CK(cudaMemsetAsync(&e.ctr->nbig, 0, 4, e.stream));
    UC_CK(cudaMemsetAsync(&e.ctr->nwarp, 0, 8, e.stream));  // nwarp, nblock
    UC_CK(cudaMemsetAsync(&e.ctr->wtile_next, 0, 4, e.stream));
    UC_CK(cudaMemsetAsync(jd.jout, 0, 8, e.stream));
    r = classify_tiles(e, f, P, nw, groups[g], groups[g + 1]);
    if (r) return r;
    r = run_tiles_k(e, tp, f, threads, nw);
    if (r) return r;
    float a = 0;
    cudaEventElapsedTime(&a, e.ev[8], e.ev[5]);
    ms_tiles += a;
    unsigned long long gb = 0;
    UC_CK(cudaMemcpyAsync(&gb, jd.jout, 8, cudaMemcpyDeviceToHost, e.stream));
    r = e.read_ctr();
    if (r) return r;
    if (e.h_ctr->err) return e.check_err(e.h_ctr);
    if (closed + gb > cap) return e.fail(UC_EINPUT, "output buffer smaller than uc_output_bound");
    UC_CK(cudaMemcpyAsync(h_out + closed, d_gout, gb, cudaMemcpyDeviceToHost, e.stream));
    UC_CK(cudaStreamSynchronize(e.stream));
    closed += gb;
  }
  cudaEventRecord(e.ev[3], e.stream);
  // the stitch into its own buffer (no closed lines before it there)
  J.ocap = sout;
  UC_CK(cudaMemcpyAsync(jd.tab, &J, sizeof(JobTab), cudaMemcpyHostToDevice, e.stream));
  UC_CK(cudaMemsetAsync(jd.jclosed, 0, 8, e.stream));
  UC_CK(cudaMemsetAsync(jd.jout, 0, 8, e.stream));
  uint32_t rounds = 0;
  StitchBufs sbuf{seg, Xr, segc, act0, act1, oncyc, hlen, lbase, longl, uint32_t(long_cap(e, X)), rcnt, hp};
  r = run_stitch(e, sbuf, X, Hp, k, nw, want_hec, RH, jd, d_sout, rounds);
  if (r) return r;
  cudaEventRecord(e.ev[4], e.stream);
  unsigned long long sb = 0;
  UC_CK(cudaMemcpyAsync(&sb, jd.jout, 8, cudaMemcpyDeviceToHost, e.stream));
  r = e.read_ctr();
  if (r) return r;
  if (e.h_ctr->err) return e.check_err(e.h_ctr);
  if (sb > sout) return e.fail(UC_EINTERNAL, "output bound exceeded");
  if (closed + sb > cap) return e.fail(UC_EINPUT, "output buffer smaller than uc_output_bound");
  UC_CK(cudaMemcpyAsync(h_out + closed, d_sout, sb, cudaMemcpyDeviceToHost, e.stream));
  UC_CK(cudaStreamSynchronize(e.stream));
  out_bytes = closed + sb;
  if (st) {
    st->n_kmers = n;
    st->n_copies = copies;
    st->n_cross = X;
    st->n_tiles = ntiles;
    st->n_segments = Sp;
    st->n_cycles = e.h_ctr->cycles;
    st->closed_bytes = closed;
    st->seg_chars = e.h_ctr->seg_char_cursor;
    st->out_bytes = out_bytes;
    st->stitch_rounds = rounds;
    st->l_used = uint32_t(P.l_used);
    st->bucket_bits = P.bits;
    st->tile_capacity = P.cap;
    st->launches = e.launches;
    st->graph_nodes = e.graph_nodes;
    float a = 0, b = 0, d = 0;
    cudaEventElapsedTime(&a, e.ev[0], e.ev[1]);
    cudaEventElapsedTime(&b, e.ev[1], e.ev[2]);
    cudaEventElapsedTime(&d, e.ev[3], e.ev[4]);
    st->ms_pack = a;
    st->ms_bucket = b;
    st->ms_tiles = ms_tiles;
    st->ms_stitch = d;
    st->ms_total = a + b + ms_tiles + d;
  }
  e.reset();
  return UC_OK;
}

int compact_device(Env& e, const char* d_text, size_t bytes, int k, int l, char* out, uint64_t cap,
                   uint64_t& out_bytes, uc_stats* st) {
  uint64_t off = 0, len = 0;
  LineRecs recs;
  int r = compact_jobs(e, 1, &d_text, &bytes, k, l, out, cap, &off, &len, st, e.sorted ? &recs : nullptr);
  out_bytes = len + recs.bytes;
  if (r == UC_OK && e.sorted) r = sort_lines(e, out, len, k, recs);
  return r;
}

}  // namespace uc
