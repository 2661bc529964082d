// Warp-cooperative walks of the payload's record chains: FoR sub-blocks, ALP
// sub-blocks and ALP-RD exceptions.  Each record's size depends on its own
// header, so the next record's start is known only once the header is read,
// and a walk by one thread pays a memory latency per record (75 ns to 0.6 us:
// 237 us for the 1,000 exceptions of a 32,768-value frame, 60 us for a
// 128-sub-block chain).  Consecutive records mostly have the same size, so the
// warp reads the headers where the next 32 (128 exceptions) would start if
// they did, keeps the leading ones that really have that size, and goes on
// from the first that differs with its size as the next guess.  Every record
// is accepted only at a start that the records before it prove, in order, so
// the result and the first error are the sequential walk's; the cost is one
// memory latency per run of equal sizes (at most 32 or 128 records).
#pragma once
#include "qb_common.cuh"

namespace qb {

// Leading true lanes of a warp vote.
__device__ __forceinline__ uint32_t leading_ones(uint32_t m) { return m == 0xFFFFFFFFu ? 32u : __ffs(~m) - 1; }

// FoR sub-block chain (reference codecs/for_bitpack.rs:108-157) over
// p[pos .. bound): varint(n) then sub-blocks [width u8][min u64][128*width B],
// their header offsets in offs (offs[nsub] = the end).  All lanes call it with
// the same arguments and get the same error.
__device__ inline uint32_t warp_for_walk(const uint8_t* p, uint64_t bound, uint64_t pos, uint64_t n_values,
                                         uint32_t* offs) {
  const uint32_t l = threadIdx.x & 31;
  uint64_t n64;
  uint32_t e = rd_varint(p, bound, &pos, &n64);
  if (e) return e;
  if (n64 != n_values) return E_CORRUPT;
  const uint32_t nsub = (uint32_t)((n_values + kSub - 1) / kSub);
  if (nsub) {
    if (pos >= bound) return E_TRUNCATED;
    uint32_t w = p[pos];
    if (w > 64) return E_CORRUPT;
    for (uint32_t k = 0; k < nsub;) {
      const uint64_t size = 9 + 128ull * w, q = pos + l * size;
      uint32_t b = 256;
      if (k + l < nsub && q < bound) b = p[q];
      const bool ok = b == w && bound - q >= size;
      const uint32_t c = leading_ones(__ballot_sync(0xffffffffu, ok));
      if (l < c) offs[k + l] = (uint32_t)q;
      pos += c * size;
      k += c;
      if (c == 32 || k >= nsub) continue;
      // the sub-block at pos, whose header lane c read: its own size, or its error
      if (pos >= bound) return E_TRUNCATED;
      w = __shfl_sync(0xffffffffu, b, c);
      if (w > 64) return E_CORRUPT;
      if (bound - pos - 1 < 8) return E_TRUNCATED;
      if (bound - pos - 9 < 128ull * w) return E_TRUNCATED;
    }
  }
  if (l == 0) offs[nsub] = (uint32_t)pos;
  return E_OK;
}

// One ALP sub-block at p[q] (reference codecs/alp.rs:168-248) holding `count`
// values: its width and exception count, or the sequential decoder's error.
__device__ inline uint32_t alp_sub_check(const uint8_t* p, uint64_t plen, uint64_t q, uint64_t count, uint32_t* w,
                                         uint32_t* exc) {
  if (q >= plen) return E_TRUNCATED;
  uint32_t ee = p[q];
  if (q + 1 >= plen) return E_TRUNCATED;
  uint32_t ff = p[q + 1];
  if (ee > 18 || ff > ee) return E_CORRUPT;
  if (plen < q + 4) return E_TRUNCATED;
  *exc = ld_u16(p + q + 2);
  if (plen < q + 12 || q + 12 >= plen) return E_TRUNCATED;
  *w = p[q + 12];
  if (*w > 32) return E_CORRUPT;
  uint64_t x = q + 13;
  if (plen - x < 128ull * *w) return E_TRUNCATED;
  x += 128ull * *w;
  for (uint32_t k = 0; k < *exc; k++, x += 10) {
    if (plen < x + 10) return E_TRUNCATED;
    if (ld_u16(p + x) >= count) return E_CORRUPT;
  }
  return E_OK;
}

// ALP sub-block chain of an n-value frame, offsets as warp_for_walk.
__device__ inline uint32_t warp_alp_walk(const uint8_t* p, uint64_t plen, uint64_t n, uint32_t* offs) {
  const uint32_t l = threadIdx.x & 31;
  uint64_t pos = 0, n64;
  uint32_t e = rd_varint(p, plen, &pos, &n64);
  if (e) return e;
  if (n64 != n) return E_CORRUPT;
  const uint32_t nsub = (uint32_t)((n + kSub - 1) / kSub);
  uint32_t gw = 0, gx = 0;
  for (uint32_t k = 0; k < nsub;) {
    const uint64_t size = 13 + 128ull * gw + 10ull * gx, q = pos + l * size;
    uint32_t w = 0, x = 0, er = E_OK;
    const bool in = k + l < nsub;
    if (in) er = alp_sub_check(p, plen, q, qmin(kSub, n - (uint64_t)(k + l) * kSub), &w, &x);
    const uint32_t c = leading_ones(__ballot_sync(0xffffffffu, in && !er && w == gw && x == gx));
    if (l < c) offs[k + l] = (uint32_t)q;
    pos += c * size;
    k += c;
    if (c == 32 || k >= nsub) continue;
    er = __shfl_sync(0xffffffffu, er, c);  // of the sub-block at pos
    if (er) return er;
    gw = __shfl_sync(0xffffffffu, w, c);
    gx = __shfl_sync(0xffffffffu, x, c);
  }
  return E_OK;
}

// ALP-RD exception list (reference codecs/alp_rd.rs:230-245): nexc records of
// a varint position and 8 bytes from *pos.  rec(active, x, q, v) is called by
// the whole warp for groups of up to 32 consecutive records, the active lanes
// first: record x starts at q and has position v (0 without VALUES, for a
// caller that only looks for the end); it returns false for a position out of
// range (E_CORRUPT).  On success *pos is the list's end.
template <bool VALUES, class R>
__device__ inline uint32_t warp_exc_walk(const uint8_t* p, uint64_t plen, uint64_t* pos, uint64_t nexc, R rec) {
  constexpr uint32_t kPer = 4;
  const uint32_t l = threadIdx.x & 31;
  uint64_t o = *pos;
  uint32_t len = 0;  // varint bytes of the records guessed at
  for (uint64_t x = 0; x < nexc;) {
    uint32_t got = 0;
    if (len) {
      const uint32_t size = len + 8;
      uint32_t ok[kPer];
      uint64_t v[kPer];
#pragma unroll
      for (uint32_t j = 0; j < kPer; j++) {
        const uint32_t i = j * 32 + l;
        const uint64_t q = o + (uint64_t)i * size;
        ok[j] = x + i < nexc && q + size <= plen;
        uint64_t w = ok[j] ? ld_u64(p + q) : 0ull;
        v[j] = 0;
        if (len <= 8) {
          const uint64_t high = w & 0x8080808080808080ull & (~0ull >> (64 - 8 * len));
          ok[j] = ok[j] && high == (0x0080808080808080ull & (len == 1 ? 0ull : (~0ull >> (64 - 8 * (len - 1)))));
#pragma unroll
          for (uint32_t b = 0; VALUES && b < 8; b++)
            if (b < len) v[j] |= ((w >> (8 * b)) & 0x7Full) << (7 * b);
        } else if (ok[j]) {
          uint64_t t = q;
          ok[j] = rd_varint(p, plen, &t, &v[j]) == E_OK && t - q == len;
        }
      }
      bool bad = false;
      for (uint32_t j = 0; j < kPer; j++) {
        const uint32_t c = leading_ones(__ballot_sync(0xffffffffu, ok[j]));
        if (!rec(l < c, x + j * 32 + l, o + (uint64_t)(j * 32 + l) * size, v[j]) && l < c) bad = true;
        got += c;
        if (c < 32) break;
      }
      if (__any_sync(0xffffffffu, bad)) return E_CORRUPT;
      x += got;
      o += (uint64_t)got * size;
      if (got == 32 * kPer || x >= nexc) continue;
    }
    // the record at o: its varint length, or its error
    uint64_t t = o, v;
    uint32_t e = rd_varint(p, plen, &t, &v);
    if (e) return e;
    if (plen - t < 8) return E_TRUNCATED;
    len = (uint32_t)(t - o);
  }
  *pos = o;
  return E_OK;
}

}  // namespace qb
