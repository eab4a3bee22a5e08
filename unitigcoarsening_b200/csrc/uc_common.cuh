// uc_common.cuh — key layout, minimizer priority and small device helpers
// shared by the unitig-compaction kernels.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace uc {

constexpr uint32_t NONE = 0xFFFFFFFFu;
// Role bits live in the two top bits of a key's last 64-bit word; a key uses
// at most 62 bits of that word (k <= 31 in one word, k <= 63 in two).
constexpr uint64_t ROLE_P = 1ull << 63;  // copy sits in its prefix-minimizer bucket
constexpr uint64_t ROLE_S = 1ull << 62;  // copy sits in its suffix-minimizer bucket
constexpr uint64_t ROLE_MASK = ROLE_P | ROLE_S;

// device error word bits
enum : uint32_t {
  ERR_LINE = 1u,      // a k-mer line shorter than k
  ERR_COUNT = 2u,     // header count differs from the line count
  ERR_TIMEOUT = 4u,   // a bounded device wait gave up
  ERR_CAPACITY = 8u,  // an output or scratch bound was exceeded
  ERR_LAYOUT = 16u,   // fixed-width line layout did not hold (fast path)
  ERR_INTERNAL = 32u,
};

template <int NW>
struct Key {
  uint64_t w[NW];
};

template <int NW>
__device__ __forceinline__ Key<NW> ld_key(const uint64_t* p, size_t i) {
  Key<NW> k;
  if constexpr (NW == 1) {
    k.w[0] = p[i];
  } else {
    const ulonglong2 v = reinterpret_cast<const ulonglong2*>(p)[i];
    k.w[0] = v.x;
    k.w[1] = v.y;
  }
  return k;
}

template <int NW>
__device__ __forceinline__ void st_key(uint64_t* p, size_t i, const Key<NW>& k) {
  if constexpr (NW == 1) {
    p[i] = k.w[0];
  } else {
    reinterpret_cast<ulonglong2*>(p)[i] = make_ulonglong2(k.w[0], k.w[1]);
  }
}

template <int NW>
__device__ __forceinline__ uint64_t roles(const Key<NW>& k) {
  return k.w[NW - 1] & ROLE_MASK;
}

template <int NW>
__device__ __forceinline__ Key<NW> strip(Key<NW> k) {
  k.w[NW - 1] &= ~ROLE_MASK;
  return k;
}

// Mask keeping the low 2*(k-1) bits: the (k-1)-prefix.
struct PrefMask {
  uint64_t m0, m1;
};
__host__ __device__ inline PrefMask pref_mask(int k) {
  const int bits = 2 * (k - 1);
  PrefMask m;
  if (bits >= 64) {
    m.m0 = ~0ull;
    m.m1 = (bits == 64) ? 0ull : ((1ull << (bits - 64)) - 1ull);
  } else {
    m.m0 = (1ull << bits) - 1ull;
    m.m1 = 0ull;
  }
  return m;
}

template <int NW>
__device__ __forceinline__ Key<NW> prefix_of(const Key<NW>& x, const PrefMask& m) {
  Key<NW> r;
  r.w[0] = x.w[0] & m.m0;
  if constexpr (NW == 2) r.w[1] = x.w[1] & m.m1;
  return r;
}

// chars 1..k-1 moved down to position 0 (role bits fall outside the mask)
template <int NW>
__device__ __forceinline__ Key<NW> suffix_of(const Key<NW>& x, const PrefMask& m) {
  Key<NW> r;
  if constexpr (NW == 1) {
    r.w[0] = (x.w[0] >> 2) & m.m0;
  } else {
    r.w[0] = ((x.w[0] >> 2) | (x.w[1] << 62)) & m.m0;
    r.w[1] = (x.w[1] >> 2) & m.m1;
  }
  return r;
}

template <int NW>
__device__ __forceinline__ bool key_eq(const Key<NW>& a, const Key<NW>& b) {
  bool e = a.w[0] == b.w[0];
  if constexpr (NW == 2) e = e && (a.w[1] == b.w[1]);
  return e;
}

// numeric order of the packed value (last word most significant), roles ignored
template <int NW>
__device__ __forceinline__ bool key_lt(const Key<NW>& a, const Key<NW>& b) {
  if constexpr (NW == 1) {
    return (a.w[0] & ~ROLE_MASK) < (b.w[0] & ~ROLE_MASK);
  } else {
    const uint64_t ah = a.w[1] & ~ROLE_MASK, bh = b.w[1] & ~ROLE_MASK;
    return ah < bh || (ah == bh && a.w[0] < b.w[0]);
  }
}

// Slot hash of a (k-1)-mer for the tile tables (at most 2^15 slots): the
// high half of a multiplicative (Fibonacci) hash, which every key bit reaches.
template <int NW>
__device__ __forceinline__ uint32_t key_hash(const Key<NW>& p) {
  uint64_t h = p.w[0] * 0x9E3779B97F4A7C15ull;
  if constexpr (NW == 2) h += p.w[1] * 0xC2B2AE3D27D4EB4Full;
  return static_cast<uint32_t>(h >> 32);
}

// 2-bit code of char x of a packed key
template <int NW>
__device__ __forceinline__ uint32_t key_char(const Key<NW>& x, int i) {
  if constexpr (NW == 1) {
    return static_cast<uint32_t>(x.w[0] >> (2 * i)) & 3u;
  } else {
    return static_cast<uint32_t>((i < 32 ? x.w[0] >> (2 * i) : x.w[1] >> (2 * (i - 32)))) & 3u;
  }
}

__device__ __forceinline__ char acgt(uint32_t c) {
  return static_cast<char>(0x54474341u >> (8 * c));  // "ACGT"
}

// Seeded bijection of [0, 4^l): the l-mer priority.  The reference draws a
// random permutation of the 4^l l-mers (generate_permutation,
// driver.cpp:356-402); any permutation gives the same unitigs.  Multiplying
// by an odd number and adding are each invertible modulo 4^l; both come from
// the seed.
__host__ __device__ __forceinline__ uint32_t lmer_mult(uint64_t seed) {
  return (0x9E3779B1u ^ (static_cast<uint32_t>(seed) << 1)) | 1u;
}
__host__ __device__ __forceinline__ uint32_t lmer_priority(uint32_t x, int l, uint64_t seed) {
  const uint32_t b = 2u * static_cast<uint32_t>(l);
  const uint32_t mask = (b >= 32u) ? 0xFFFFFFFFu : ((1u << b) - 1u);
  return (x * lmer_mult(seed) + static_cast<uint32_t>(seed >> 32)) & mask;
}

// Bucket of a minimizer priority.  Any function of the minimizer keeps every
// (k-1)-overlap inside one bucket; this one spreads the small-valued
// minimizers (a minimum is biased low) evenly over 2^bits buckets.
__host__ __device__ __forceinline__ uint32_t bucket_of(uint32_t pr, uint32_t bits) {
  uint32_t h = pr * 0x9E3779B1u;
  h ^= h >> 16;
  h *= 0x85EBCA6Bu;
  h ^= h >> 13;
  h *= 0xC2B2AE35u;
  h ^= h >> 16;
  return bits ? (h >> (32u - bits)) : 0u;
}

// ASCII of the 4 codes in the low 8 bits of c (first char in the low byte):
// spread the 2-bit codes into nibbles, then select bytes of "ACGT".
__device__ __forceinline__ uint32_t ascii4(uint32_t c) {
  uint32_t x = (c | (c << 4)) & 0x0F0Fu;
  x = (x | (x << 2)) & 0x3333u;
  return __byte_perm(0x54474341u, 0u, x);
}

// Bits 1 and 2 of 16 letters, first letter lowest: A 0, C 1, T 2, G 3 (a line
// break reads as 1).  Each 4 letters' pairs are gathered into a byte by one
// multiply (the partial products below bit 24 do not meet, so nothing carries).
__device__ __forceinline__ uint32_t letter_bits16(const uint4& v) {
  auto g = [](uint32_t x) { return (x & 0x06060606u) * 0x00820820u; };  // in byte 3
  return __byte_perm(__byte_perm(g(v.x), g(v.y), 0x0073), __byte_perm(g(v.z), g(v.w), 0x0073), 0x5410);
}
// Those bits -> codes (A 0, C 1, G 2, T 3).
__device__ __forceinline__ uint32_t codes_of_bits(uint32_t r) { return r ^ ((r >> 1) & 0x55555555u); }
// 16 bytes of letters and line breaks -> 16 codes, first byte lowest.
__device__ __forceinline__ uint32_t codes16(const uint4& v) { return codes_of_bits(letter_bits16(v)); }
// Of 16 bytes of ACGT and line breaks, a bit per line break (bit 6 is clear
// in '\n' and set in the letters), the first byte's lowest.  Two words share
// one byte of a product; the partial products do not meet.
__device__ __forceinline__ uint32_t breaks16(const uint4& v) {
  const uint32_t a = (~v.x >> 6) & 0x01010101u, b = (~v.y >> 6) & 0x01010101u;
  const uint32_t c = (~v.z >> 6) & 0x01010101u, d = (~v.w >> 6) & 0x01010101u;
  return __byte_perm(a * 0x01020408u + b * 0x10204080u, c * 0x01020408u + d * 0x10204080u, 0x4473) & 0xFFFFu;
}
// 16 two-bit values (first lowest) -> their letters by a table of four: the
// letters of the even and of the odd chars, then their bytes interleaved.
__device__ __forceinline__ void spread16(uint32_t table, uint32_t c, uint32_t w[4]) {
  const uint32_t e = c & 0x33333333u, o = (c >> 2) & 0x33333333u;
  const uint32_t e0 = __byte_perm(table, 0u, e), e1 = __byte_perm(table, 0u, e >> 16);
  const uint32_t o0 = __byte_perm(table, 0u, o), o1 = __byte_perm(table, 0u, o >> 16);
  w[0] = __byte_perm(e0, o0, 0x5140);
  w[1] = __byte_perm(e0, o0, 0x7362);
  w[2] = __byte_perm(e1, o1, 0x5140);
  w[3] = __byte_perm(e1, o1, 0x7362);
}
__device__ __forceinline__ void letters16(uint32_t codes, uint32_t w[4]) { spread16(0x54474341u, codes, w); }

// n bytes from src to dst (any alignment) by `size` threads: 16-byte stores
// of the destination, each from five source words.  Reads up to 3 bytes on
// either side of the source bytes' words.
__device__ __forceinline__ void copy_bytes(char* dst, const char* src, unsigned long long n, uint32_t rank,
                                           uint32_t size) {
  const uint32_t head = uint32_t(min((unsigned long long)((16u - uint32_t(reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u), n));
  if (rank < head) dst[rank] = src[rank];
  dst += head;
  src += head;
  n -= head;
  const uint32_t sh = 8u * uint32_t(reinterpret_cast<uintptr_t>(src) & 3u);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(src) & ~uintptr_t(3));
  const unsigned long long np = n >> 4;
  for (unsigned long long p = rank; p < np; p += size) {
    const uint32_t a = w[4 * p], b = w[4 * p + 1], c = w[4 * p + 2], d = w[4 * p + 3];
    const uint32_t e = sh ? w[4 * p + 4] : 0u;
    reinterpret_cast<uint4*>(dst)[p] = make_uint4(__funnelshift_r(a, b, sh), __funnelshift_r(b, c, sh),
                                                  __funnelshift_r(c, d, sh), __funnelshift_r(d, e, sh));
  }
  const uint32_t rest = uint32_t(n & 15u);
  for (uint32_t q = rank; q < rest; q += size) dst[16 * np + q] = src[16 * np + q];
}

// Text of n chars (codes x, first char lowest) and, with brk = 1, a line break
// at byte pos of a shared-memory buffer: whole words where the text owns them,
// halves and bytes at its two ends (shared with its neighbours).
template <int NC>
__device__ __forceinline__ void spell_text(uint32_t* buf, uint32_t pos, const uint32_t x[NC], uint32_t n, uint32_t brk) {
  const uint32_t a = pos & 3u;
  // the code stream, moved up by the chars before the text in its first word
  uint32_t c[NC];
  c[0] = x[0] << (2 * a);
#pragma unroll
  for (int q = 1; q < NC; ++q) c[q] = __funnelshift_l(x[q - 1], x[q], 2 * a);
  const uint32_t last = a + n;                      // one past the last char, from the first word's start
  const uint32_t nw = last >> 2, rem = last & 3u;   // its word, and the chars before it there
  uint32_t* d = buf + (pos >> 2);
  uint32_t first = 0, tail = 0;
#pragma unroll
  for (int g = 0; g < NC; ++g) {
    if (4u * g > nw) break;
    uint32_t w[4];
    letters16(c[g], w);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = 4u * g + q;
      if (j == nw) tail = w[q];
      if (j < nw && (j > 0 || a == 0)) d[j] = w[q];
    }
    if (g == 0) first = w[0];
  }
  if (brk) tail = (tail & ((1u << (8 * rem)) - 1u)) | (uint32_t('\n') << (8 * rem));
  const uint32_t nb = rem + brk;  // bytes of the last word
  char* e = reinterpret_cast<char*>(d + nw);
  if (nw == 0 && a) {  // inside one word
    for (uint32_t q = a; q < nb; ++q) e[q] = char(tail >> (8 * q));
    return;
  }
  if (nb == 4) {
    d[nw] = tail;
  } else {
    if (nb & 2u) *reinterpret_cast<uint16_t*>(e) = uint16_t(tail);
    if (nb & 1u) e[nb & 2u] = char(tail >> (8 * (nb & 2u)));
  }
  if (a) {
    char* f = reinterpret_cast<char*>(d);
    if (a & 1u) f[a] = char(first >> (8 * a));
    if (a < 3) *reinterpret_cast<uint16_t*>(f + 2) = uint16_t(first >> 16);
  }
}

// A stream of text to global memory by one warp: texts are spelled one after
// another into the warp's shared-memory buffer and leave as 16-byte stores.
// The bytes after the last whole piece stay in the buffer for the next
// texts; the first and the last piece, shared with other streams, go byte by
// byte.
struct WarpText {
  char* dst;      // next byte of the stream
  uint32_t fill;  // bytes of buf before it, from the 16-byte boundary below dst
  uint32_t head;  // of which another stream's
  __device__ __forceinline__ void begin(char* at) {
    dst = at;
    fill = head = uint32_t(reinterpret_cast<uintptr_t>(at) & 15u);
  }
  // total bytes were spelled into buf from byte fill on (every lane calls,
  // after a __syncwarp).  Reads buf up to 16 bytes past them.
  __device__ __forceinline__ void flush(uint32_t* buf, uint32_t total) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t full = (fill + total) >> 4;
    char* w = dst - fill;
    for (uint32_t p = lane; p < full; p += 32) {
      if (p == 0 && head) {
        for (uint32_t q = head; q < 16; ++q) w[q] = reinterpret_cast<const char*>(buf)[q];
      } else {
        reinterpret_cast<uint4*>(w)[p] = reinterpret_cast<const uint4*>(buf)[p];
      }
    }
    __syncwarp();
    if (full) {
      if (lane < 4) buf[lane] = buf[4 * full + lane];
      head = 0;
    }
    __syncwarp();
    fill = (fill + total) & 15u;
    dst += total;
  }
  __device__ __forceinline__ void end(const uint32_t* buf) const {
    const uint32_t lane = threadIdx.x & 31u;
    if (lane >= head && lane < fill) (dst - fill)[lane] = reinterpret_cast<const char*>(buf)[lane];
    __syncwarp();
  }
};

// codes of chars ch..ch+3 of a packed key in the low 8 bits (chars past the
// key read as 0)
template <int NW>
__device__ __forceinline__ uint32_t codes4(const Key<NW>& x, int ch) {
  if constexpr (NW == 1) {
    return uint32_t(x.w[0] >> (2 * ch)) & 0xFFu;
  } else {
    const uint64_t v = (ch < 32) ? ((x.w[0] >> (2 * ch)) | (ch > 0 ? (x.w[1] << (64 - 2 * ch)) : 0ull))
                                 : (x.w[1] >> (2 * (ch - 32)));
    return uint32_t(v) & 0xFFu;
  }
}

// Write the k chars of a packed key at dst (any alignment): byte stores up
// to the first aligned word, then the key moved down by those chars (one
// shift) and aligned 32-bit stores from constant shifts, then byte stores
// for the rest.
template <int NW>
__device__ __forceinline__ void spell_key(char* dst, const Key<NW>& x, int k) {
  const int ch0 = min(k, int((4u - uint32_t(reinterpret_cast<uintptr_t>(dst) & 3u)) & 3u));
  Key<NW> y = x;
  if (ch0) {
    const uint32_t a = ascii4(codes4(x, 0));
    for (int i = 0; i < ch0; ++i) dst[i] = char(a >> (8 * i));
    if constexpr (NW == 1) {
      y.w[0] = x.w[0] >> (2 * ch0);
    } else {
      y.w[0] = (x.w[0] >> (2 * ch0)) | (x.w[1] << (64 - 2 * ch0));
      y.w[1] = x.w[1] >> (2 * ch0);
    }
  }
  const int rest = k - ch0;
  const int nw4 = rest >> 2;
  uint32_t* d = reinterpret_cast<uint32_t*>(dst + ch0);
#pragma unroll
  for (int w = 0; w < 8 * NW; ++w)
    if (w < nw4) d[w] = ascii4(codes4(y, 4 * w));
  if (rest & 3) {
    const uint32_t a = ascii4(codes4(y, 4 * nw4));
    for (int i = 0; i < (rest & 3); ++i) dst[ch0 + 4 * nw4 + i] = char(a >> (8 * i));
  }
}

// reverse the order of the 2-bit groups of a 64-bit word
__device__ __forceinline__ uint64_t rev2(uint64_t x) {
  x = __brevll(x);
  return ((x >> 1) & 0x5555555555555555ull) | ((x & 0x5555555555555555ull) << 1);
}

// Prefix (l1) and suffix (l2) minimizer priorities of one k-mer
// (get_double_lmin, lmin_buckets.h:67-94): l-mer ids are big-endian (first
// char in the top bits); l1 covers the l-mers inside chars [0, k-1), l2 the
// ones inside chars [1, k).  Requires 1 <= l <= min(16, k-1).
//
// Without a table the priority is computed in the top 2l bits of a 32-bit
// word: (id * m + a) << (32 - 2l) equals id * (m << (32 - 2l)) + (a << ...)
// modulo 2^32, and chars left of the l-mer in the id's upper bits drop out of
// that product, so each l-mer costs one shift, one multiply-add and one min.
template <int NW>
__device__ __forceinline__ void lmins(const Key<NW>& key, int k, int l, uint64_t seed,
                                      const uint32_t* __restrict__ table, uint32_t& l1,
                                      uint32_t& l2) {
  uint64_t hi, lo;
  if constexpr (NW == 1) {
    hi = rev2(key.w[0] & ~ROLE_MASK);
    lo = 0;
  } else {
    hi = rev2(key.w[0]);
    lo = rev2(key.w[1] & ~ROLE_MASK);
  }
  const int w = k - l + 1;  // l-mers in the k-mer (>= 2)
  if (table == nullptr) {
    const uint32_t ps = 32u - 2u * uint32_t(l);
    const uint32_t m = lmer_mult(seed) << ps, a = static_cast<uint32_t>(seed >> 32) << ps;
    uint32_t first, mid = 0xFFFFFFFFu, last;
    if constexpr (NW == 1) {
      // l-mer p sits in bits [64 - 2p - 2l, 64 - 2p) of hi
      int s = 64 - 2 * l;
      first = static_cast<uint32_t>(hi >> s) * m + a;
#pragma unroll
      for (int p = 1; p < w - 1; ++p) {
        s -= 2;
        mid = min(mid, static_cast<uint32_t>(hi >> s) * m + a);
      }
      last = static_cast<uint32_t>(hi >> (s - 2)) * m + a;
    } else {
      const int s = 64 - 2 * l;
      first = static_cast<uint32_t>(hi >> s) * m + a;
#pragma unroll
      for (int p = 1; p < w - 1; ++p) {
        hi = (hi << 2) | (lo >> 62);
        lo <<= 2;
        mid = min(mid, static_cast<uint32_t>(hi >> s) * m + a);
      }
      hi = (hi << 2) | (lo >> 62);
      last = static_cast<uint32_t>(hi >> s) * m + a;
    }
    l1 = min(first, mid) >> ps;
    l2 = min(mid, last) >> ps;
    return;
  }
  const int sh = 64 - 2 * l;
  auto pri = [&](uint32_t id) { return __ldg(table + id); };
  const uint32_t first = pri(static_cast<uint32_t>(hi >> sh));
  uint32_t mid = NONE;
  for (int p = 1; p < w - 1; ++p) {
    hi = (hi << 2) | (lo >> 62);
    lo <<= 2;
    mid = min(mid, pri(static_cast<uint32_t>(hi >> sh)));
  }
  hi = (hi << 2) | (lo >> 62);
  const uint32_t last = pri(static_cast<uint32_t>(hi >> sh));
  l1 = min(first, mid);
  l2 = min(mid, last);
}

// ---- warp / block helpers ---------------------------------------------

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T t = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// Exclusive block scan; every thread of the block must call it.  scratch
// holds at least 33 values.  Returns the exclusive prefix, total in *total.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* scratch, T* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  T inc = warp_incl_scan(v);
  if (lane == 31) scratch[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    T s = (lane < nw) ? scratch[lane] : T(0);
    T si = warp_incl_scan(s);
    if (lane < nw) scratch[lane] = si - s;
    if (lane == nw - 1) scratch[32] = si;
  }
  __syncthreads();
  T r = scratch[wid] + inc - v;
  *total = scratch[32];
  __syncthreads();
  return r;
}

}  // namespace uc
