// Block planner, per-block codec competition and winner emission
// (reference src/encoder.rs:154-469,644-759 and the encode functions of the
// in-path codecs).  The competition is one CTA per block and never materialises a
// candidate payload: every candidate's exact byte length is computed in closed
// form from warp-reduced statistics (sub-block widths, exception counts,
// distinct/run counts, ALP (e,f) search, ALP-RD cut search), the argmin of
// `len + penalty` is taken in the reference's candidate order with a strict
// `<`, and only the winner is written, by one or two CTAs per window (k_emit).
#include <cooperative_groups.h>

#include "qb_common.cuh"
#include "qb_layout.h"
#include "qb_kernels.h"

namespace qb {

constexpr int kEncThreads = 512;
constexpr int kEncWarps = kEncThreads / 32;
constexpr int kSubsMax = kMaxBlock / kSub;  // 128
constexpr uint32_t kHashCap = 2048;         // smem hash slots (dict / ALP-RD left parts)
constexpr uint32_t kHashLimit = 1536;       // distinct keys before falling back to scratch
constexpr uint32_t kLbBits = 1u << 17;      // dict cardinality lower-bound bitset
constexpr uint32_t kNoLb = 0xFFFFFFFFu;

// 17-bit bucket of the dictionary cardinality lower-bound bitset.
__device__ __forceinline__ uint32_t dict_lb_bucket(uint64_t x) {
  return ((uint32_t)x * 0x9E3779B1u + (uint32_t)(x >> 32) * 0x85EBCA77u) >> (32 - 17);
}
constexpr uint64_t kEmpty64 = ~0ull;
constexpr uint32_t kEmpty32 = 0xFFFFFFFFu;

__device__ unsigned long long g_wins[64];  // reference src/diag.rs:8-23

// Candidate decode weights (reference encoder.rs:79-89).
__host__ __device__ inline uint64_t decode_weight(int m) {
  switch (m) {
    case M_RAW: case M_CONST: case M_STRIDE: return 0;
    case M_XORZ: case M_FOR_BITPACK: case M_DELTA_BITPACK: case M_RLE: return 1;
    case M_ALP: case M_ALP_RD: case M_DICT: return 2;
    case M_PRED: return 3;
    case M_BYTE_TRANSPOSE: case M_FLOAT_MULT: return 6;
    case M_PRED_RC: case M_PRED2: return 10;
    default: return 7;
  }
}
__host__ __device__ inline uint64_t level_lambda(int level) {  // reference lib.rs:126-138
  return level == 0 ? 16 : level == 1 ? 4 : level == 2 ? 2 : 0;
}

// ---------------------------------------------------------------------------
// Small device utilities
// ---------------------------------------------------------------------------
__device__ inline void put_u8(uint8_t* d, uint32_t v) { *d = (uint8_t)v; }
__device__ inline void put_u16(uint8_t* d, uint32_t v) { d[0] = (uint8_t)v; d[1] = (uint8_t)(v >> 8); }
__device__ inline void put_u32(uint8_t* d, uint32_t v) {
#pragma unroll
  for (int i = 0; i < 4; i++) d[i] = (uint8_t)(v >> (8 * i));
}
__device__ inline void put_u64(uint8_t* d, uint64_t v) {
#pragma unroll
  for (int i = 0; i < 8; i++) d[i] = (uint8_t)(v >> (8 * i));
}
__device__ inline uint32_t put_varint(uint8_t* d, uint64_t v) {
  uint32_t n = 0;
  for (;;) {
    uint8_t b = (uint8_t)(v & 0x7f);
    v >>= 7;
    if (v) { d[n++] = b | 0x80; } else { d[n++] = b; return n; }
  }
}
__device__ inline uint64_t u64min(uint64_t a, uint64_t b) { return a < b ? a : b; }
__device__ inline uint64_t u64max(uint64_t a, uint64_t b) { return a > b ? a : b; }
__device__ inline uint32_t warp_or(uint32_t v) {
  for (int o = 16; o; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ inline uint64_t warp_or64(uint64_t v) {
  for (int o = 16; o; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ inline int64_t warp_min_i64(int64_t v) { return (int64_t)(warp_min_u64((uint64_t)v ^ kSignBit) ^ kSignBit); }
__device__ inline int64_t warp_max_i64(int64_t v) { return (int64_t)(warp_max_u64((uint64_t)v ^ kSignBit) ^ kSignBit); }
__device__ inline uint32_t pow2_at_least(uint32_t x) {
  uint32_t p = 1;
  while (p < x) p <<= 1;
  return p;
}
__device__ inline void atomic_min_u64(unsigned long long* a, uint64_t v) { atomicMin(a, (unsigned long long)v); }
__device__ inline void atomic_max_u64(unsigned long long* a, uint64_t v) { atomicMax(a, (unsigned long long)v); }

// In-place ascending bitonic sort of P (power of two) keys; all threads.
__device__ void block_bitonic_sort(uint64_t* a, uint32_t P) {
  for (uint32_t k = 2; k <= P; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
        uint32_t ixj = i ^ j;
        if (ixj > i) {
          uint64_t x = a[i], y = a[ixj];
          bool up = (i & k) == 0;
          if ((x > y) == up) { a[i] = y; a[ixj] = x; }
        }
      }
      __syncthreads();
    }
  }
}

// (e, f) of the c-th pair in the reference's search order (alp.rs:61-62).
__device__ inline void alp_combo(uint32_t c, int* e, int* f) {
  int ee = 0;
  while ((uint32_t)((ee + 1) * (ee + 2) / 2) <= c) ee++;
  *e = ee;
  *f = (int)(c - (uint32_t)(ee * (ee + 1) / 2));
}

__device__ inline int64_t fm_k(uint64_t x, int s) {
  return __double2ll_rz(round_half_away(__dmul_rn(as_f64(x), kFmScales[s])));
}

// ---------------------------------------------------------------------------
// Shared memory of the competition and emission kernels
// ---------------------------------------------------------------------------
struct RdArea {
  uint32_t smp[2][4096];  // the sample's top 24 bits (two buffers of the sort)
  uint8_t cp[4096];       // leading bits (of 24) a sorted key shares with the one before
  uint32_t hkey[kHashCap];
  uint32_t hcnt[kHashCap];
};
struct DictArea {
  uint64_t hkey[kHashCap];
  uint32_t hval[kHashCap];
  uint64_t sorted[kHashCap];
};
union BigArea {
  RdArea rd;
  DictArea dict;
};
constexpr uint32_t kRansChunk = 4096;  // bytes staged per step of the rANS encoder
struct RansArea {
  uint32_t hist[256];
  uint2 fc[256];                    // (frequency, cumulative frequency) per symbol
  uint4 enc[256];                   // the coding step's constants per symbol (rans_enc)
  alignas(16) uint8_t buf[2][kRansChunk];  // double-buffered input bytes
  uint32_t hdr, emitted;
  uint32_t bound;  // a lower bound on the coded bytes (rans_plan)
};

// What the competition leaves for the emission besides the mode: per sub-block
// the ALP-RD (or RLE) layout, per block its dictionary of left parts and the DICT
// dictionary's size (kept in the block's scratch when it is small), so that
// the emission makes no pass over the block before it packs, and several CTAs
// can share a block.
struct RdRec {
  uint64_t rmin;    // smallest right part (RLE: smallest length of the run chunk)
  uint32_t eb;      // exception bytes
  uint16_t ne;      // exceptions
  uint8_t cw, rw;   // code and right widths (RLE: rw, the chunk's)
  uint8_t cmin, pad[7];
};
static_assert(sizeof(RdRec) == 24, "RdRec layout");
struct BlkRec {
  uint64_t dict8[8];
  uint64_t vlen;    // DICT value bytes
  uint32_t dl, card, vtag, pad;  // card: DICT's values (0 = not kept), RLE's runs
};
static_assert(sizeof(BlkRec) == 88, "BlkRec layout");

struct EncSmem {
  uint8_t w_a[kSubsMax];   // FoR widths (also ALP widths in emit)
  uint8_t w_b[kSubsMax];   // delta / rights widths
  uint8_t w_c[kSubsMax];   // ALP / codes widths
  uint8_t w_d[kSubsMax];   // FLOAT_MULT widths
  uint8_t alp_ef[kSubsMax][2];
  uint16_t alp_exc[kSubsMax];
  uint32_t neq_k[kSubsMax];
  uint32_t subsz[kSubsMax + 1];
  uint64_t submin[kSubsMax];
  uint64_t item_min[kSubsMax], item_max[kSubsMax];
  unsigned long long xor_bytes, umin, umax, e_vmin, e_vmax, e_dmax, acc64;
  uint32_t neq, stride_bad, fm_mask, alp_fail, flag, ovf, card, has_max, max_rank, cnt32, dl;
  uint32_t distinct_bits[512];
  uint64_t alp_smp[kEncWarps][32];
  double rd_pv[24];
  uint32_t rd_top[24][8];  // per cut: the sample's largest left-part groups (size << 12 | first sorted key)
  uint32_t rd_cand[8], rd_cnt[8], rd_ncand;
  uint8_t rd_mask[kSubsMax];  // per sub-block: which of rd_cand occur
  uint32_t rd_ne[kSubsMax], rd_eb[kSubsMax];  // per sub-block: ALP-RD exceptions and their bytes
  uint64_t dict8[8];
  uint64_t red[kEncWarps];
  uint32_t red32[kEncWarps];
  uint64_t sc[8];
  uint32_t exp_lo, exp_hi;
  alignas(16) BigArea big;
  RansArea ra;
};

// ---------------------------------------------------------------------------
// Warp-level FoR statistics of one sub-block: width of (max - min).
// ---------------------------------------------------------------------------
template <class V>
__device__ inline void warp_minmax(uint32_t cnt, bool sgn, V val, uint64_t* mn_out, uint32_t* w_out) {
  int lane = threadIdx.x & 31;
  uint64_t umn = kEmpty64, umx = 0;
  int64_t smn = INT64_MAX, smx = INT64_MIN;
  for (uint32_t i0 = lane; i0 < cnt; i0 += 32 * 8) {
   uint64_t xs[8];
#pragma unroll
   for (int q = 0; q < 8; q++) {
     uint32_t iq = i0 + 32 * q;
     xs[q] = iq < cnt ? val(iq) : 0ull;
   }
#pragma unroll
   for (int q = 0; q < 8; q++) {
    if (i0 + 32 * q >= cnt) break;
    uint64_t x = xs[q];
    umn = u64min(umn, x);
    umx = u64max(umx, x);
    int64_t s = (int64_t)x;
    smn = s < smn ? s : smn;
    smx = s > smx ? s : smx;
   }
  }
  if (sgn) {
    smn = warp_min_i64(smn);
    smx = warp_max_i64(smx);
    *mn_out = (uint64_t)smn;
    *w_out = bit_width64((uint64_t)smx - (uint64_t)smn);
  } else {
    umn = warp_min(umn);
    umx = warp_max(umx);
    *mn_out = umn;
    *w_out = bit_width64(umx - umn);
  }
}

// The low `k` bytes of v at d (k <= 4).
__device__ __forceinline__ void put_low(uint8_t* d, uint32_t v, uint32_t k) {
  for (uint32_t i = 0; i < k; i++) d[i] = (uint8_t)(v >> (8 * i));
}

// Pack one FoR sub-block (header + FastLanes words) at dst; residual of
// index i = val(i) - mn for i < cnt, 0 for the padding (reference
// for_bitpack.rs:47-96, bitpack.rs:48-133).  Consecutive lanes' words are
// consecutive in memory, at any byte address: a lane writes the aligned word
// that ends its own and starts with the top of its neighbour's (lane 0: of the
// last lane's word a row earlier), so a row of 32 words is one aligned store
// and only the stream's first and last bytes are written singly (a byte per
// store took 55 us for 16,777,216 timestamps' frames, a third of the copy rate).
// Above 32 bits, 16 lanes hold 64-bit words; the two half warps take rows 0-31
// and 32-63, whose bits meet at the middle of a word when the width is odd:
// the second half's first word waits for the first half's end.
template <class V>
__device__ inline void warp_for_pack(uint8_t* dst, uint32_t cnt, uint64_t mn, uint32_t w, V val) {
  int lane = threadIdx.x & 31;
  if (lane < 8) dst[1 + lane] = (uint8_t)(mn >> (8 * lane));
  if (lane == 8) put_u8(dst, w);
  if (w == 0) return;
  uint8_t* words = dst + 9;
  const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(words) & 3), sh = 8 * mis;
  uint32_t* al = reinterpret_cast<uint32_t*>(words - mis);  // al[j]: the aligned word that ends word j of the stream
  if (w <= 32) {
    uint64_t acc = 0;
    uint32_t nb = 0, carry = 0, first = 0;
    uint32_t* o = al + lane;
    for (uint32_t r0 = 0; r0 < 32; r0 += 8) {
     uint32_t rs[8];
#pragma unroll
     for (int q = 0; q < 8; q++) {
       uint32_t iq = (r0 + q) * 32 + lane;
       rs[q] = iq < cnt ? (uint32_t)(val(iq) - mn) : 0u;
     }
#pragma unroll
     for (int q = 0; q < 8; q++) {
      uint32_t res = rs[q];
      if (w < 32) res &= (1u << w) - 1u;
      acc |= (uint64_t)res << nb;
      nb += w;
      if (nb >= 32) {
        const uint32_t x = (uint32_t)acc, rot = __shfl_sync(0xffffffffu, x, (lane + 31) & 31);
        const uint32_t out = __funnelshift_l(lane ? rot : carry, x, sh);
        if (o != al || !mis) *o = out;  // the very first word is shared with what precedes the stream
        else first = x;
        carry = rot;
        o += 32;
        acc >>= 32;
        nb -= 32;
      }
     }
    }
    if (lane == 0 && mis) {
      put_low(words, first, 4 - mis);
      put_low(reinterpret_cast<uint8_t*>(o), carry >> (32 - sh), mis);
    }
  } else {
    const uint32_t h = (uint32_t)lane >> 4, fl = lane & 15;
    const uint32_t half = h * 32 * w;  // the half's first bit
    uint64_t acc = 0, first = 0;
    uint32_t nb = half & 63, wi = half >> 6, carry = 0;
    bool wait = h != 0;
    auto put = [&](uint32_t k, uint64_t x, uint32_t prev) {  // word k of the lane; prev: the 32 bits before it
      const uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32), j = 2 * (k * 16 + fl);
      if (mis && j == 0) put_low(words, lo, 4 - mis);
      else al[j] = __funnelshift_l(prev, lo, sh);
      al[j + 1] = __funnelshift_l(lo, hi, sh);
    };
    for (uint32_t r0 = 0; r0 < 32; r0 += 8) {
     uint64_t rs[8];
#pragma unroll
     for (int q = 0; q < 8; q++) {
       uint32_t iq = (h * 32 + r0 + q) * 16 + fl;
       rs[q] = iq < cnt ? (val(iq) - mn) : 0ull;
     }
#pragma unroll
     for (int q = 0; q < 8; q++) {
      uint64_t res = rs[q];
      if (w < 64) res &= (1ull << w) - 1ull;
      acc |= res << nb;
      nb += w;
      const uint32_t rot = __shfl_sync(0xffffffffu, (uint32_t)(acc >> 32), (fl + 15) & 15, 16);
      if (nb >= 64) {  // the same for the lanes of a half
        if (wait) first = acc;
        else put(wi, acc, fl ? rot : carry);
        wait = false;
        carry = rot;
        wi++;
        nb -= 64;
        acc = nb ? res >> (w - nb) : 0ull;
      }
     }
    }
    // the second half's first word: its low bits (an odd width) and what
    // precedes lane 0's are the first half's last
    const uint32_t low = __shfl_sync(0xffffffffu, (uint32_t)acc, fl), before = __shfl_sync(0xffffffffu, carry, 0);
    if (w & 1) first |= low;
    const uint32_t rot = __shfl_sync(0xffffffffu, (uint32_t)(first >> 32), (fl + 15) & 15, 16);
    if (h) put(w >> 1, first, fl ? rot : before);
    if (lane == 16 && mis) put_low(reinterpret_cast<uint8_t*>(al + 32u * w), carry >> (32 - sh), mis);
  }
}

// S.subsz[0 .. nsub) (sizes) turned into offsets from `base`, the end in
// S.subsz[nsub].  All threads call it; the sizes are written before.
__device__ inline void block_offsets(EncSmem& S, uint32_t nsub, uint32_t base) {
  __syncthreads();
  if (threadIdx.x < 32) {
    uint32_t c[kSubsMax / 32], s = 0;
#pragma unroll
    for (int j = 0; j < kSubsMax / 32; j++) {
      uint32_t k = threadIdx.x * (kSubsMax / 32) + j;
      c[j] = k < nsub ? S.subsz[k] : 0u;
      s += c[j];
    }
    uint32_t inc = warp_incl_scan(s), off = base + inc - s;
#pragma unroll
    for (int j = 0; j < kSubsMax / 32; j++) {
      uint32_t k = threadIdx.x * (kSubsMax / 32) + j;
      if (k < nsub) S.subsz[k] = off;
      off += c[j];
    }
    if (threadIdx.x == 31) S.subsz[nsub] = base + inc;
  }
  __syncthreads();
}

// Second half of the FoR stream writer: with S.w_a[k] / S.submin[k] set for
// every sub-block, lays out varint(M) + sub-blocks and (dst non-null) packs
// sub-blocks k0 .. k1 of val(0..M), the varint with the first.  Returns the
// byte length (all threads).
template <class V>
__device__ uint64_t block_for_write(EncSmem& S, uint8_t* dst, uint32_t M, V val, uint32_t k0 = 0,
                                    uint32_t k1 = kSubsMax) {
  int warp = threadIdx.x >> 5;
  uint32_t nsub = (M + kSub - 1) / kSub;
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.subsz[k] = 9 + 128u * S.w_a[k];
  block_offsets(S, nsub, varint_len(M));
  if (threadIdx.x == 0 && dst && k0 == 0) put_varint(dst, M);
  uint64_t total = S.subsz[nsub];
  if (dst) {
    for (uint32_t k = k0 + warp; k < min(nsub, k1); k += kEncWarps) {
      uint32_t cnt = min((uint32_t)kSub, M - k * kSub);
      warp_for_pack(dst + S.subsz[k], cnt, S.submin[k], S.w_a[k], [&](uint32_t i) { return val(k * kSub + i); });
    }
  }
  __syncthreads();
  return total;
}

// Whole-CTA FoR stream writer: varint(M) + sub-blocks of val(0..M).  When
// dst is null only the size is computed.  Returns the byte length (all threads).
template <class V>
__device__ uint64_t block_for(EncSmem& S, uint8_t* dst, uint32_t M, bool sgn, V val) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t nsub = (M + kSub - 1) / kSub;
  for (uint32_t k = warp; k < nsub; k += kEncWarps) {
    uint32_t cnt = min((uint32_t)kSub, M - k * kSub);
    uint64_t mn;
    uint32_t w;
    warp_minmax(cnt, sgn, [&](uint32_t i) { return val(k * kSub + i); }, &mn, &w);
    if (lane == 0) {
      S.w_a[k] = (uint8_t)w;
      S.submin[k] = mn;
    }
  }
  __syncthreads();
  return block_for_write(S, dst, M, val);
}

// alp_roundtrips_r with the four powers of ten of its (e, f) given:
// pe = 10^e, pf = 10^-f (encode), qf = 10^f, qe = 10^-e (decode).
__device__ __forceinline__ bool alp_rt_pow(uint64_t bits, double pe, double pf, double qf, double qe, double* r) {
  double tmp = __dmul_rn(__dmul_rn(as_f64(bits), pe), pf);
  const double kUpper = 9.223372036854776e18, kMagic = 6755399441055744.0;
  if (!is_finite_f64(tmp) || tmp >= kUpper || tmp <= -kUpper) return false;
  double rr = __dadd_rn(__dadd_rn(tmp, kMagic), -kMagic);
  *r = rr;
  return f64_bits(__dmul_rn(__dmul_rn(rr, qf), qe)) == bits;
}

// ALP for one sub-block (reference alp.rs:49-166): find_ef on the 32-value
// sample, then the full encode statistics.  Warp-cooperative; returns false
// when the sub-block (hence the block) bails.
struct AlpSub {
  int e, f;
  uint32_t w, exc;
  int64_t mn, filler;
};
__device__ bool alp_subblock_ef(const uint64_t* sv, uint32_t cnt, int e, int f, const double* pexp,
                                const double* pfrac, AlpSub* out);
__device__ bool alp_subblock(const uint64_t* sv, uint32_t cnt, uint64_t* smp, const double* pexp, const double* pfrac,
                             AlpSub* out) {
  int lane = threadIdx.x & 31;
  uint32_t st = max(cnt / 32u, 1u);
  uint32_t sl = min(32u, (cnt + st - 1) / st);
  smp[lane] = (uint32_t)lane < sl ? sv[lane * st] : 0ull;
  __syncwarp();
  uint64_t best_cost = kEmpty64;
  uint32_t best_c = 0xFFFF, best_exc = 0;
  const double kInf = __longlong_as_double(0x7FF0000000000000ll);
  for (uint32_t c = lane; c < 190; c += 32) {
    int e, f;
    alp_combo(c, &e, &f);
    const double pe = pexp[e], pf = pfrac[f], qf = pexp[f], qe = pfrac[e];
    uint32_t ex = 0;
    double lo = kInf, hi = -kInf;  // digits as the integral doubles they are cast from
    for (uint32_t s = 0; s < sl; s++) {
      double r;
      if (alp_rt_pow(smp[s], pe, pf, qf, qe, &r)) {
        lo = r < lo ? r : lo;
        hi = r > hi ? r : hi;
      } else {
        ex++;
      }
    }
    int64_t lo_i = ex == sl ? 0 : f64_as_i64(lo), hi_i = ex == sl ? 0 : f64_as_i64(hi);
    uint32_t width = (ex == sl) ? 64u : (hi_i <= lo_i ? 0u : bit_width64((uint64_t)hi_i - (uint64_t)lo_i));
    uint64_t cost = (uint64_t)width * sl + (uint64_t)ex * 80;
    if (cost < best_cost) {
      best_cost = cost;
      best_c = c;
      best_exc = ex;
    }
  }
  for (int o = 16; o; o >>= 1) {
    uint64_t oc = __shfl_xor_sync(0xffffffffu, best_cost, o);
    uint32_t occ = __shfl_xor_sync(0xffffffffu, best_c, o);
    uint32_t oe = __shfl_xor_sync(0xffffffffu, best_exc, o);
    if (oc < best_cost || (oc == best_cost && occ < best_c)) {
      best_cost = oc;
      best_c = occ;
      best_exc = oe;
    }
  }
  __syncwarp();
  if (best_exc * 2 > sl) return false;
  int e, f;
  alp_combo(best_c, &e, &f);
  return alp_subblock_ef(sv, cnt, e, f, pexp, pfrac, out);
}

// The encode pass of one sub-block for a chosen (e, f) (alp.rs:109-166):
// exceptions, digit range, the filler digit.  Warp-cooperative; false when
// the digits need more than 32 bits.
__device__ bool alp_subblock_ef(const uint64_t* sv, uint32_t cnt, int e, int f, const double* pexp,
                                const double* pfrac, AlpSub* out) {
  int lane = threadIdx.x & 31;
  const double kInf = __longlong_as_double(0x7FF0000000000000ll);
  const double pe = pexp[e], pf = pfrac[f], qf = pexp[f], qe = pfrac[e];
  uint32_t exc = 0, first_li = 0xFFFFFFFFu;
  double rmn = kInf, rmx = -kInf, first_r = 0.0;
  for (uint32_t j = 0; j < 32; j++) {
    uint32_t li = j * 32 + lane;
    bool ok = li < cnt;
    double r = 0.0;
    bool rt = ok && alp_rt_pow(sv[li], pe, pf, qf, qe, &r);
    if (rt) {
      rmn = r < rmn ? r : rmn;
      rmx = r > rmx ? r : rmx;
      if (li < first_li) {
        first_li = li;
        first_r = r;
      }
    }
    exc += __popc(__ballot_sync(0xffffffffu, ok && !rt));
  }
  int64_t first_d = f64_as_i64(first_r);
  int64_t dmn = rmn == kInf ? INT64_MAX : f64_as_i64(rmn), dmx = rmx == -kInf ? INT64_MIN : f64_as_i64(rmx);
  dmn = warp_min_i64(dmn);
  dmx = warp_max_i64(dmx);
  for (int o = 16; o; o >>= 1) {
    uint32_t ol = __shfl_xor_sync(0xffffffffu, first_li, o);
    int64_t od = __shfl_xor_sync(0xffffffffu, first_d, o);
    if (ol < first_li) {
      first_li = ol;
      first_d = od;
    }
  }
  int64_t filler = first_li == 0xFFFFFFFFu ? 0 : first_d;
  if (first_li == 0xFFFFFFFFu) dmn = dmx = 0;
  uint32_t w = bit_width64((uint64_t)dmx - (uint64_t)dmn);
  if (w > 32) return false;
  out->e = e;
  out->f = f;
  out->w = w;
  out->exc = exc;
  out->mn = dmn;
  out->filler = filler;
  return true;
}

// ---------------------------------------------------------------------------
// ALP-RD: cut search on the sample (reference alp_rd.rs:80-107).  Uses the
// sorted sample: for a cut, the equal-left groups are runs of the sorted
// sample, and only the sum of the 8 largest group counts matters.
// ---------------------------------------------------------------------------
__device__ inline void top8_insert(uint32_t (&t)[8], uint32_t c) {
  if (c <= t[7]) return;
  t[7] = c;
#pragma unroll
  for (int i = 7; i > 0; i--) {
    if (t[i] > t[i - 1]) {
      uint32_t x = t[i];
      t[i] = t[i - 1];
      t[i - 1] = x;
    }
  }
}
__device__ inline uint32_t rd_code_bits(uint32_t dl) {
  if (dl <= 1) return 1;
  uint32_t b = bit_width64((uint64_t)(dl - 1));
  return b ? b : 1;
}

// Ascending bitonic sort of 512 * K u32 keys, K per thread: a warp holds
// 32 * K consecutive positions (row r, lane l at 32r + l), so only the
// exchanges between warps (10 of the 66 steps at 2,048 keys) pass through
// shared memory and take a barrier.  `buf` holds two buffers; the sorted keys
// end in the returned one, readable after the barrier inside.
template <int K>
__device__ uint32_t* block_sort_u32(uint32_t (&a)[K], uint32_t (*buf)[4096]) {
  constexpr uint32_t P = kEncThreads * K, W = 32 * K;
  const uint32_t l = threadIdx.x & 31, base = (threadIdx.x >> 5) * W;
  int cur = 0;
  for (uint32_t k = 2; k <= P; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      if (j >= W) {
#pragma unroll
        for (int r = 0; r < K; r++) buf[cur][base + 32 * r + l] = a[r];
        __syncthreads();
        const bool keep_min = ((base & j) == 0) == ((base & k) == 0);
#pragma unroll
        for (int r = 0; r < K; r++) {
          uint32_t o = buf[cur][(base ^ j) + 32 * r + l];
          a[r] = keep_min ? min(a[r], o) : max(a[r], o);
        }
        cur ^= 1;  // the next exchange writes the other buffer: one barrier each
      } else if (j >= 32) {
#pragma unroll
        for (int d = 1; d < K; d <<= 1) {
          if (j != 32u * d) continue;
#pragma unroll
          for (int r = 0; r < K; r++) {
            if (r & d) continue;
            const bool up = ((base + 32 * r) & k) == 0;
            uint32_t x = a[r], y = a[r | d];
            a[r] = up ? min(x, y) : max(x, y);
            a[r | d] = up ? max(x, y) : min(x, y);
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < K; r++) {
          uint32_t o = __shfl_xor_sync(0xffffffffu, a[r], j);
          const bool keep_min = ((l & j) == 0) == (((base + 32 * r + l) & k) == 0);
          a[r] = keep_min ? min(a[r], o) : max(a[r], o);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < K; r++) buf[cur][base + 32 * r + l] = a[r];
  __syncthreads();
  return buf[cur];
}

// Returns the chosen left bit width, or 0 when ALP-RD does not apply.  The
// sample is block[0], block[step], ... (step = max(n/2048, 1)); when `pre` is
// given it holds those values at pre[i * pre_stride].  A cut keeps at most 24
// left bits, so the keys are the sample's top 24 bits; sorted, a cut's groups
// are the runs between positions that share fewer leading bits with their
// predecessor than the cut keeps.  One warp per cut gathers those positions as
// 32-bit words, a lane's words together cover consecutive positions, and each
// lane ranks the groups that end in its own.  S.rd_cand gets the largest
// groups of the chosen cut.  (With 64-bit keys sorted through shared memory
// and a vote per 32 positions it took 56 us of the 144 us that a 32,768-price
// block's competition took.)
template <int K>
__device__ uint32_t* rd_sort_sample(EncSmem& S, const uint64_t* v, uint32_t sn, uint32_t step, const uint64_t* pre,
                                    uint32_t pre_stride) {
  uint32_t a[K];
  const uint32_t base = (threadIdx.x >> 5) * 32 * K + (threadIdx.x & 31);
#pragma unroll
  for (int r = 0; r < K; r++) {
    uint32_t i = base + 32 * r;
    a[r] = i < sn ? (uint32_t)((pre ? pre[(uint64_t)i * pre_stride] : v[(uint64_t)i * step]) >> 40) : 0xFFFFFFFFu;
  }
  return block_sort_u32<K>(a, S.big.rd.smp);
}
__device__ uint32_t rd_choose_cut(EncSmem& S, const uint64_t* v, uint32_t n, const uint64_t* pre, uint32_t pre_stride) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t step = max(n / 2048u, 1u);
  uint32_t sn = (n + step - 1) / step;  // at most 4095
  static_assert(kEncThreads * 8 == 4096, "a sample of 4,095 values, eight a thread");
  __syncthreads();  // the area is free
  const uint32_t* key = sn <= kEncThreads * 4 ? rd_sort_sample<4>(S, v, sn, step, pre, pre_stride)
                                              : rd_sort_sample<8>(S, v, sn, step, pre, pre_stride);
  for (uint32_t i = threadIdx.x; i < sn; i += blockDim.x) {
    uint32_t d = i ? key[i] ^ key[i - 1] : 0x800000u;
    S.big.rd.cp[i] = (uint8_t)(d ? __clz(d) - 8 : 24);
  }
  __syncthreads();
  const uint32_t rows = (sn + 31) / 32, q = (rows + 31) / 32;  // a lane takes q consecutive rows (at most 4)
  for (uint32_t lbw = warp + 1; lbw <= 24; lbw += kEncWarps) {
    uint32_t rbw = 64 - lbw;
    uint32_t w[4] = {0, 0, 0, 0};
    for (uint32_t o = 0; o * q < rows; o++) {
#pragma unroll
      for (uint32_t u = 0; u < 4; u++) {
        uint32_t i = (o * q + u) * 32 + lane;
        uint32_t m = u < q ? __ballot_sync(0xffffffffu, i < sn && S.big.rd.cp[i] < lbw) : 0u;
        if ((uint32_t)lane == o) w[u] = m;
      }
    }
    uint32_t G = 0, last = 0;  // last: 1 + the lane's last group start
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      G += __popc(w[u]);
      if (w[u]) last = (lane * q + u) * 32 + 32 - __clz(w[u]);
    }
    G = __reduce_add_sync(0xffffffffu, G);
    uint32_t before = last;  // the largest over the lanes up to this one, then those before it
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t x = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before = max(before, x);
    }
    const uint32_t end = __shfl_sync(0xffffffffu, before, 31);
    uint32_t start = __shfl_up_sync(0xffffffffu, before, 1);
    if (lane == 0) start = 0;
    uint32_t t[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // size << 12 | first key, descending
    // Groups of two and more, each at the start that follows it (a start whose
    // predecessor is none): the many of one key that a deep cut leaves cost
    // nothing, and only their number matters.
    uint32_t tail = start && start == lane * q * 32 ? 1u : 0u;  // the position before the lane's words starts a group
#pragma unroll
    for (uint32_t u = 0; u < 4; u++) {
      if (u >= q) break;
      const uint32_t b0 = (lane * q + u) * 32;
      uint32_t m = w[u] & ~(w[u] << 1 | tail);
      tail = w[u] >> 31;
      while (m) {
        const uint32_t j = __ffs(m) - 1;
        m &= m - 1;
        const uint32_t prev = w[u] & ((1u << j) - 1u);
        const uint32_t st = prev ? b0 + 32 - __clz(prev) : start;  // 1 + the group's first key
        if (st) top8_insert(t, (b0 + j - (st - 1)) << 12 | (st - 1));
      }
      if (w[u]) start = b0 + 32 - __clz(w[u]);
    }
    if (lane == 0 && sn - (end - 1) >= 2) top8_insert(t, (sn - (end - 1)) << 12 | (end - 1));
    uint32_t cov = 0, have = 0;
    for (int r = 0; r < 8; r++) {
      uint32_t mx = __reduce_max_sync(0xffffffffu, t[0]);
      if (lane == 0) S.rd_top[lbw - 1][r] = mx;
      if (t[0] == mx && mx) {  // one lane: the packed groups differ
#pragma unroll
        for (int i = 0; i < 7; i++) t[i] = t[i + 1];
        t[7] = 0;
      }
      cov += mx >> 12;
      have += mx ? 1u : 0u;
    }
    if (have < 8) cov += min(8u - have, G - have);  // groups of one key
    uint32_t dl = min(G, 8u);
    uint64_t num = (uint64_t)sn * (uint64_t)(rbw + rd_code_bits(dl)) + ((uint64_t)sn - cov) * 96ull;
    if (lane == 0) S.rd_pv[lbw - 1] = __ddiv_rn(__ull2double_rn(num), __ull2double_rn((uint64_t)sn));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t best = 0;
    double bb = __longlong_as_double(0x7FF0000000000000ll);  // +inf
    for (uint32_t lbw = 1; lbw <= 24; lbw++) {
      if (S.rd_pv[lbw - 1] < bb) {
        bb = S.rd_pv[lbw - 1];
        best = lbw;
      }
    }
    if (best == 0 || bb >= 63.0) best = 0;
    S.sc[0] = best;
    uint32_t nc = 0;
    for (; best && nc < 8 && S.rd_top[best - 1][nc]; nc++)
      S.rd_cand[nc] = key[S.rd_top[best - 1][nc] & 4095u] >> (24 - best);
    S.rd_ncand = nc;
  }
  __syncthreads();
  uint32_t best = (uint32_t)S.sc[0];
  __syncthreads();
  return best;
}

// One value's left part counted in a table of cap slots (a power of two):
// false when it holds no free slot for it.  `fresh` counts the keys.
__device__ __forceinline__ void rd_count(uint32_t* hk, uint32_t* hc, uint32_t cap, uint32_t lg, uint32_t key,
                                         uint32_t add, uint32_t* fresh) {
  uint32_t h = (uint32_t)(((uint64_t)key * 0x9E3779B97F4A7C15ull) >> (64 - lg));
  for (uint32_t probe = 0; probe < cap; probe++) {
    uint32_t cur = hk[h];
    if (cur == kEmpty32) {
      uint32_t old = atomicCAS(&hk[h], kEmpty32, key);
      if (old == kEmpty32) {
        if (fresh) atomicAdd(fresh, 1u);
        cur = key;
      } else {
        cur = old;
      }
    }
    if (cur == key) {
      atomicAdd(&hc[h], add);
      return;
    }
    h = (h + 1) & (cap - 1);
  }
}

// The block's eight most frequent left parts and everything that the payload
// needs to know of them: the chosen cut's largest sample groups (S.rd_cand)
// are counted by comparison; the other left parts (a few in a hundred where
// ALP-RD is any good) are listed in shared memory and counted in a table
// afterwards.  If none of those is as frequent as the rarest candidate, the
// candidates are the dictionary; otherwise the table names the right ones and
// the pass runs once more with them.  On true S.dict8 holds the dictionary by
// (count desc, key asc) (alp_rd.rs:47-68), and per sub-block S.w_a the codes'
// width and S.w_c their smallest code, S.rd_ne the exceptions and S.rd_eb
// their bytes.  False (more keys than the shared table holds): the general
// pass decides (rd_top8).  (A vote for equal left parts and an
// atomic per 32 values, eight searches of the table and a second pass took
// 75 us for 32,768 values.)
constexpr uint32_t kRdList = 2 * 4096 / kEncWarps;  // listed left parts a warp (over the sample's sort buffers)
__device__ bool rd_dict_pass(EncSmem& S, const uint64_t* v, uint32_t n, uint32_t lbw) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t rbw = 64 - lbw, nsub = (n + kSub - 1) / kSub, below = (1u << lane) - 1u;
  uint32_t* hk = S.big.rd.hkey;
  uint32_t* hc = S.big.rd.hcnt;
  uint32_t* list = &S.big.rd.smp[0][0] + warp * kRdList;
  bool full = false;  // the table has no room for more keys
  auto count_list = [&](uint32_t m) {
    __syncwarp();
    for (uint32_t i = lane; i < m && !full; i += 32) {
      full = *(volatile uint32_t*)&S.card >= kHashLimit;
      if (!full) rd_count(hk, hc, kHashCap, 11, list[i], 1, &S.card);
    }
    __syncwarp();
  };
  for (int round = 0;; round++) {
    const uint32_t nc = S.rd_ncand;
    for (uint32_t i = threadIdx.x; i < kHashCap; i += blockDim.x) {
      hk[i] = kEmpty32;
      hc[i] = 0;
    }
    if (threadIdx.x < 8) S.rd_cnt[threadIdx.x] = 0;
    if (threadIdx.x == 0) S.card = 0;  // keys in the table
    uint32_t listed = 0;
    uint32_t cand[8], cnt[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      cand[j] = (uint32_t)j < nc ? S.rd_cand[j] : kEmpty32;  // left parts are below 2^24
      cnt[j] = 0;
    }
    __syncthreads();
    for (uint32_t k = warp; k < nsub; k += kEncWarps) {
      const uint32_t base = k * kSub, m = min((uint32_t)kSub, n - base);
      uint32_t seen = 0, ne = 0, eb = 0;
      for (uint32_t i0 = 0; i0 < m; i0 += 32 * 8) {
        uint64_t xs[8];
#pragma unroll
        for (int u = 0; u < 8; u++) xs[u] = i0 + 32 * u + lane < m ? v[base + i0 + 32 * u + lane] : 0ull;
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t i = i0 + 32 * u + lane;
          const bool in = i < m;
          const uint32_t left = in ? (uint32_t)(xs[u] >> rbw) : 0xFFFFFFFEu;
          uint32_t hit = 0;
#pragma unroll
          for (int j = 0; j < 8; j++)
            if (left == cand[j]) {
              cnt[j]++;
              hit = 1u << j;
            }
          seen |= hit;
          const bool other = in && !hit;
          const uint32_t om = __ballot_sync(0xffffffffu, other);
          if (!om) continue;
          if (other) {
            list[listed + __popc(om & below)] = left;
            ne++;
            eb += 9 + (base + i >= (1u << 7) ? 1u : 0u) + (base + i >= (1u << 14) ? 1u : 0u);  // i < 2^17
          }
          listed += __popc(om);
          if (listed > kRdList - 32) {
            count_list(listed);
            listed = 0;
          }
        }
      }
      seen = __reduce_or_sync(0xffffffffu, seen);
      ne = __reduce_add_sync(0xffffffffu, ne);
      eb = __reduce_add_sync(0xffffffffu, eb);
      if (lane == 0) {
        S.rd_mask[k] = (uint8_t)seen;
        S.rd_ne[k] = ne;
        S.rd_eb[k] = eb;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint32_t c = __reduce_add_sync(0xffffffffu, cnt[j]);
      if (lane == 0 && c) atomicAdd(&S.rd_cnt[j], c);
    }
    count_list(listed);
    if (__syncthreads_or(full)) return false;
    // is another left part at least as frequent as the rarest candidate?
    uint32_t rarest = nc == 8 ? 0xFFFFFFFFu : 0u;
    for (uint32_t j = 0; j < nc && nc == 8; j++) rarest = min(rarest, S.rd_cnt[j]);
    uint32_t other = 0;
    for (uint32_t i = threadIdx.x; i < kHashCap; i += blockDim.x) other = max(other, hc[i]);
    if (!__syncthreads_or(other && other >= rarest)) break;
    if (round) return false;  // not reached: the exact eight were counted
    // the exact eight among the candidates and the table's keys
    if (threadIdx.x < nc) rd_count(hk, hc, kHashCap, 11, S.rd_cand[threadIdx.x], S.rd_cnt[threadIdx.x], nullptr);
    __syncthreads();
    uint64_t top[4];  // the thread's four slots: (count, key) packed, larger first in the dictionary
#pragma unroll
    for (int u = 0; u < 4; u++) {
      uint32_t i = threadIdx.x + kEncThreads * u;
      top[u] = hc[i] ? (uint64_t)hc[i] << 32 | (0xFFFFFFFFu - hk[i]) : 0ull;
    }
    static_assert(kHashCap == 4 * kEncThreads, "four table slots a thread");
    uint32_t found = 0;
    for (int r = 0; r < 8; r++) {
      uint64_t mx = top[0];
#pragma unroll
      for (int u = 1; u < 4; u++) mx = u64max(mx, top[u]);
      mx = warp_max(mx);
      if (lane == 0) S.red[warp] = mx;
      __syncthreads();
      mx = 0;
      for (int w = 0; w < kEncWarps; w++) mx = u64max(mx, S.red[w]);
      __syncthreads();
      if (!mx) break;
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (top[u] == mx) top[u] = 0;
      if (threadIdx.x == 0) S.rd_cand[r] = 0xFFFFFFFFu - (uint32_t)mx;
      found++;
    }
    if (threadIdx.x == 0) S.rd_ncand = found;
    __syncthreads();
  }
  const uint32_t nc = S.rd_ncand;
  if (threadIdx.x < nc) {  // ranks by (count desc, key asc)
    const uint32_t j = threadIdx.x;
    const uint64_t mine = (uint64_t)S.rd_cnt[j] << 32 | (0xFFFFFFFFu - S.rd_cand[j]);
    uint32_t rank = 0;
    for (uint32_t i = 0; i < nc; i++)
      rank += ((uint64_t)S.rd_cnt[i] << 32 | (0xFFFFFFFFu - S.rd_cand[i])) > mine ? 1u : 0u;
    S.dict8[rank] = S.rd_cand[j];
    S.red32[j] = rank;
  }
  if (threadIdx.x == 0) S.dl = nc;
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) {
    uint32_t lo = 8, hi = 0;
    for (uint32_t j = 0; j < nc; j++)
      if (S.rd_mask[k] >> j & 1u) {
        lo = min(lo, S.red32[j]);
        hi = max(hi, S.red32[j]);
      }
    if (S.rd_ne[k]) lo = 0;  // an exception's code is 0
    S.w_a[k] = (uint8_t)bit_width64((uint64_t)(hi - min(lo, hi)));
    S.w_c[k] = (uint8_t)min(lo, hi);
  }
  __syncthreads();
  return true;
}

// Full-block top-8 left parts by (count desc, key asc) (reference
// alp_rd.rs:47-68).  Counts go to a smem hash; when the block has more
// distinct left parts than the smem table holds, a scratch table is used.
__device__ void rd_top8(EncSmem& S, const uint64_t* v, uint32_t n, uint32_t lbw, uint8_t* scratch) {
  uint32_t rbw = 64 - lbw;
  uint32_t* hk = S.big.rd.hkey;
  uint32_t* hc = S.big.rd.hcnt;
  for (uint32_t i = threadIdx.x; i < kHashCap; i += blockDim.x) {
    hk[i] = kEmpty32;
    hc[i] = 0;
  }
  if (threadIdx.x == 0) {
    S.ovf = 0;
    S.cnt32 = 0;
  }
  __syncthreads();
  // Counts are warp-aggregated: the lanes holding equal left parts (few
  // distinct ones is the common case) add once, by their lowest lane.
  int lane0 = threadIdx.x & 31;
  for (uint32_t base = threadIdx.x & ~31u; base < n; base += blockDim.x) {
    if (__any_sync(0xffffffffu, *(volatile uint32_t*)&S.ovf != 0)) break;
    uint32_t i = base + lane0;
    uint32_t key = i < n ? (uint32_t)(v[i] >> rbw) : kEmpty32;  // left parts are < 2^24
    uint32_t peers = __match_any_sync(0xffffffffu, key);
    if (key == kEmpty32 || lane0 != __ffs(peers) - 1) continue;
    uint32_t add = __popc(peers);
    uint32_t h = (uint32_t)(((uint64_t)key * 0x9E3779B97F4A7C15ull) >> 53);  // 11 bits
    for (uint32_t probe = 0; probe < kHashCap; probe++) {
      uint32_t cur = hk[h];
      if (cur == kEmpty32) {
        uint32_t old = atomicCAS(&hk[h], kEmpty32, key);
        if (old == kEmpty32) {
          if (atomicAdd(&S.cnt32, 1u) >= kHashLimit) S.ovf = 1;
          cur = key;
        } else {
          cur = old;
        }
      }
      if (cur == key) {
        atomicAdd(&hc[h], add);
        break;
      }
      h = (h + 1) & (kHashCap - 1);
    }
  }
  __syncthreads();
  uint32_t* tk = hk;
  uint32_t* tc = hc;
  uint32_t cap = kHashCap;
  if (S.ovf) {  // scratch table: capacity >= 2n, (key, count) pairs
    cap = pow2_at_least(2 * n);
    tk = reinterpret_cast<uint32_t*>(scratch);
    tc = tk + cap;
    uint32_t lg = 31 - __clz(cap);
    for (uint32_t i = threadIdx.x; i < cap; i += blockDim.x) {
      tk[i] = kEmpty32;
      tc[i] = 0;
    }
    __syncthreads();
    for (uint32_t base = threadIdx.x & ~31u; base < n; base += blockDim.x) {
      uint32_t i = base + lane0;
      uint32_t key = i < n ? (uint32_t)(v[i] >> rbw) : kEmpty32;
      uint32_t peers = __match_any_sync(0xffffffffu, key);
      if (key == kEmpty32 || lane0 != __ffs(peers) - 1) continue;
      uint32_t add = __popc(peers);
      uint32_t h = (uint32_t)(((uint64_t)key * 0x9E3779B97F4A7C15ull) >> (64 - lg));
      for (uint32_t probe = 0; probe < cap; probe++) {
        uint32_t cur = tk[h];
        if (cur == kEmpty32) {
          uint32_t old = atomicCAS(&tk[h], kEmpty32, key);
          cur = old == kEmpty32 ? key : old;
        }
        if (cur == key) {
          atomicAdd(&tc[h], add);
          break;
        }
        h = (h + 1) & (cap - 1);
      }
    }
    __syncthreads();
  }
  // 8 rounds of block argmax over (count desc, key asc).
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) S.dl = 0;
  for (int r = 0; r < 8; r++) {
    uint64_t best = 0;  // (count << 32) | (0xFFFFFFFF - key); 0 = none
    uint32_t bslot = 0;
    for (uint32_t i = threadIdx.x; i < cap; i += blockDim.x) {
      uint32_t c = tc[i];
      if (c) {
        uint64_t kk = ((uint64_t)c << 32) | (uint64_t)(0xFFFFFFFFu - tk[i]);
        if (kk > best) {
          best = kk;
          bslot = i;
        }
      }
    }
    for (int o = 16; o; o >>= 1) {
      uint64_t ob = __shfl_xor_sync(0xffffffffu, best, o);
      uint32_t os = __shfl_xor_sync(0xffffffffu, bslot, o);
      if (ob > best) {
        best = ob;
        bslot = os;
      }
    }
    if (lane == 0) {
      S.red[warp] = best;
      S.red32[warp] = bslot;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t b = 0;
      uint32_t s = 0;
      for (int w = 0; w < kEncWarps; w++)
        if (S.red[w] > b) {
          b = S.red[w];
          s = S.red32[w];
        }
      if (b) {
        S.dict8[S.dl++] = tk[s];
        tc[s] = 0;
      }
    }
    __syncthreads();
  }
}

// Code (0..dl-1) of a left part, or -1 for an exception.
__device__ inline int rd_code(const EncSmem& S, uint64_t left) {
  int c = -1;
  for (uint32_t j = 0; j < S.dl; j++)
    if (S.dict8[j] == left && c < 0) c = (int)j;
  return c;
}

// ---------------------------------------------------------------------------
// DICT preparation (reference dict.rs:87-123): distinct values, the sorted
// dictionary and a value -> rank lookup.  Fast path: smem hash.  Fallback:
// scratch hash + scratch bitonic sort + binary-search ranks.  Sets S.card and
// S.flag (1 = dictionary bails: cardinality > n/2+1).
// ---------------------------------------------------------------------------
// Stable LSD radix sort (8-bit digits) of m u64 keys in a, using b as the
// second buffer; digits on which every key agrees are skipped.  Returns the
// buffer that holds the sorted keys.  All threads of a kEncThreads CTA; the
// per-warp digit counters live in the dictionary smem area.
__device__ uint64_t* block_radix_sort(EncSmem& S, uint64_t* a, uint64_t* b, uint32_t m) {
  static_assert(kEncThreads >= 256 && kEncWarps * 256 * 4 <= sizeof(S.big.dict.sorted),
                "one thread per digit in the offset scan; per-warp digit counters fit the dictionary area");
  // per-warp digit counters [kEncWarps][256] over the sorted-keys array of
  // the dictionary area (not in use here)
  uint32_t* hist = reinterpret_cast<uint32_t*>(S.big.dict.sorted);
  int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint64_t k0 = m ? a[0] : 0ull, diff = 0;
  for (uint32_t i0 = t; i0 < m; i0 += blockDim.x * 8) {
    uint64_t ks[8];
#pragma unroll
    for (int q = 0; q < 8; q++) ks[q] = i0 + q * blockDim.x < m ? a[i0 + q * blockDim.x] : k0;
#pragma unroll
    for (int q = 0; q < 8; q++) diff |= ks[q] ^ k0;
  }
  diff = warp_or64(diff);
  if (lane == 0) S.red[warp] = diff;
  __syncthreads();
  diff = 0;
  for (int w = 0; w < kEncWarps; w++) diff |= S.red[w];
  __syncthreads();
  uint32_t seg = ((m + kEncWarps - 1) / kEncWarps + 31u) & ~31u;
  uint32_t s0 = min(warp * seg, m), s1 = min(s0 + seg, m);
  for (int shift = 0; shift < 64; shift += 8) {
    if (((diff >> shift) & 0xFFull) == 0) continue;
    for (int i = t; i < kEncWarps * 256; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (uint32_t i0 = s0 + lane; i0 < s1; i0 += 32 * 8) {
      uint64_t ks[8];
#pragma unroll
      for (int q = 0; q < 8; q++) ks[q] = i0 + 32 * q < s1 ? a[i0 + 32 * q] : 0ull;
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (i0 + 32 * q < s1) atomicAdd(&hist[warp * 256 + (uint32_t)((ks[q] >> shift) & 0xFF)], 1u);
    }
    __syncthreads();
    {  // offsets: digit-major, then warp order (stability); thread t < 256 owns digit t
      uint32_t tot = 0, inc = 0;
      if (t < 256) {
        for (int w = 0; w < kEncWarps; w++) tot += hist[w * 256 + t];
        inc = tot;
        for (int o = 1; o < 32; o <<= 1) {
          uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += u;
        }
        if (lane == 31) S.red32[warp] = inc;
      }
      __syncthreads();
      if (t < 256) {
        uint32_t run = inc - tot;
        for (int w = 0; w < warp; w++) run += S.red32[w];
        for (int w = 0; w < kEncWarps; w++) {
          uint32_t c = hist[w * 256 + t];
          hist[w * 256 + t] = run;
          run += c;
        }
      }
    }
    __syncthreads();
    for (uint32_t base = s0; base < s1; base += 32 * 8) {
      uint64_t ks[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t i = base + q * 32 + lane;
        ks[q] = i < s1 ? a[i] : 0ull;
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t i = base + q * 32 + lane;
        uint32_t act = __ballot_sync(0xffffffffu, i < s1);
        if (i < s1) {
          uint32_t dg = (uint32_t)((ks[q] >> shift) & 0xFF);
          uint32_t peers = __match_any_sync(act, dg);
          uint32_t r = __popc(peers & ((1u << lane) - 1u));
          b[hist[warp * 256 + dg] + r] = ks[q];
          __syncwarp(act);
          if (r == 0) hist[warp * 256 + dg] += __popc(peers);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    uint64_t* tmp = a;
    a = b;
    b = tmp;
  }
  return a;
}

struct DictView {
  bool smem;
  const uint64_t* sorted;  // card values ascending
  uint32_t card;
  const uint64_t* tkey = nullptr;  // scratch hash table (keys) and ranks, 2^lg slots
  const uint32_t* trank = nullptr;
  uint32_t lg = 0;
};

__device__ inline uint32_t dict_hash_slot(const uint64_t* hk, uint64_t x) {
  uint32_t h = (uint32_t)((x * 0x9E3779B97F4A7C15ull) >> 53);
  for (uint32_t probe = 0; probe < kHashCap; probe++) {
    uint64_t cur = hk[h];
    if (cur == x || cur == kEmpty64) return h;
    h = (h + 1) & (kHashCap - 1);
  }
  return 0;
}

__device__ inline uint32_t dict_rank(const EncSmem& S, const DictView& dv, uint64_t x) {
  if (dv.smem) {
    if (x == kEmpty64) return S.max_rank;
    return S.big.dict.hval[dict_hash_slot(S.big.dict.hkey, x)];
  }
  if (x == kEmpty64) return S.max_rank;
  uint32_t cap = 1u << dv.lg;
  uint32_t h = (uint32_t)((x * 0x9E3779B97F4A7C15ull) >> (64 - dv.lg));
  for (uint32_t probe = 0; probe < cap && dv.tkey[h] != x; probe++) h = (h + 1) & (cap - 1);
  return dv.trank[h];
}

// Insert x into the smem hash (no-op once the table has overflowed).
__device__ __forceinline__ void dict_insert(DictArea& D, EncSmem& S, uint64_t x) {
  if (*(volatile uint32_t*)&S.ovf) return;
  if (x == kEmpty64) {
    if (atomicExch(&S.has_max, 1u) == 0) atomicAdd(&S.card, 1u);
    return;
  }
  uint32_t h = (uint32_t)((x * 0x9E3779B97F4A7C15ull) >> 53);
  for (uint32_t probe = 0; probe < kHashCap; probe++) {
    uint64_t cur = D.hkey[h];
    if (cur == kEmpty64) {
      unsigned long long old = atomicCAS((unsigned long long*)&D.hkey[h], kEmpty64, x);
      if (old == kEmpty64) {
        if (atomicAdd(&S.card, 1u) >= kHashLimit) S.ovf = 1;
        return;
      }
      cur = old;
    }
    if (cur == x) return;
    h = (h + 1) & (kHashCap - 1);
  }
  S.ovf = 1;
}

// lb_pre: the block's 17-bit bucket count when the statistics pass computed it
// (block == one adaptive window), else kNoLb.
// runs / starts (optional): the block's run starts, whose values are all its
// distinct ones (in a block of geometric runs of 16 an eighth of the work).
__device__ DictView dict_prepare(EncSmem& S, const uint64_t* v, uint32_t n, uint8_t* scratch, uint32_t lb_pre,
                                 const uint32_t* starts = nullptr, uint32_t runs = 0) {
  DictArea& D = S.big.dict;
  uint32_t max_card = n / 2 + 1;
  bool have_lb = lb_pre != kNoLb;
  if (have_lb && lb_pre > max_card) {  // the lower bound alone proves the bail
    if (threadIdx.x == 0) S.flag = 1;
    __syncthreads();
    DictView dv;
    dv.smem = false;
    dv.sorted = nullptr;
    dv.card = lb_pre;
    return dv;
  }
  for (uint32_t i = threadIdx.x; i < kHashCap; i += blockDim.x) {
    D.hkey[i] = kEmpty64;
    D.hval[i] = 0;
  }
  if (threadIdx.x == 0) {
    S.ovf = 0;
    S.card = 0;
    S.has_max = 0;
    S.flag = 0;
  }
  __syncthreads();
  // the shared-memory hash until it holds kHashLimit keys; the lower-bound
  // bitset is only built (below) for a block that overflows it
  auto insert_all = [&](uint32_t nv, auto at) {
    for (uint32_t base = 0; base < nv; base += blockDim.x * 8) {
      if (*(volatile uint32_t*)&S.ovf) break;
      uint64_t xs[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t iq = base + q * blockDim.x + threadIdx.x;
        xs[q] = iq < nv ? at(iq) : 0ull;
      }
      // the first probes of the eight values together: mostly the key is there
      uint64_t cur[8];
#pragma unroll
      for (int q = 0; q < 8; q++) cur[q] = D.hkey[(uint32_t)((xs[q] * 0x9E3779B97F4A7C15ull) >> 53)];
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (base + q * blockDim.x + threadIdx.x < nv && (cur[q] != xs[q] || xs[q] == kEmpty64)) dict_insert(D, S, xs[q]);
    }
  };
  if (starts) insert_all(runs, [&](uint32_t i) { return v[starts[i]]; });
  else insert_all(n, [&](uint32_t i) { return v[i]; });
  __syncthreads();
  DictView dv;
  if (!S.ovf) {
    uint32_t card = S.card;
    if (card > max_card) {
      if (threadIdx.x == 0) S.flag = 1;
      __syncthreads();
      dv.smem = true;
      dv.sorted = nullptr;
      dv.card = card;
      return dv;
    }
    if (threadIdx.x == 0) S.cnt32 = 0;
    __syncthreads();
    uint32_t P = pow2_at_least(max(card, 1u));
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) D.sorted[i] = kEmpty64;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kHashCap; i += blockDim.x)
      if (D.hkey[i] != kEmpty64) D.sorted[atomicAdd(&S.cnt32, 1u)] = D.hkey[i];
    __syncthreads();
    block_bitonic_sort(D.sorted, P);
    for (uint32_t r = threadIdx.x; r < card; r += blockDim.x) {
      uint64_t x = D.sorted[r];
      if (x == kEmpty64) S.max_rank = r;
      else D.hval[dict_hash_slot(D.hkey, x)] = r;
    }
    __syncthreads();
    dv.smem = true;
    dv.sorted = D.sorted;
    dv.card = card;
    return dv;
  }
  // Overflow: a lower bound on the cardinality may prove the bail outright:
  // the window's 17-bit bucket count when the statistics pass computed it,
  // and, when that does not prove it, the distinct buckets of a 2^20-bit set
  // (fewer for a short block) built in the block's scratch range with
  // fire-and-forget atomics, whose collisions stay few at any cardinality
  // near the bail threshold.
  {
    uint32_t lb = have_lb ? lb_pre : 0u;
    if (lb <= max_card) {
      uint32_t lgb = 20;
      while (lgb > 10 && (1ull << (lgb - 3)) > (uint64_t)n * kEncScratchPerValue) lgb--;
      const uint32_t words = (1u << lgb) / 32;
      uint32_t* bits = reinterpret_cast<uint32_t*>(scratch);
      for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) bits[i] = 0;
      __syncthreads();
      for (uint32_t base = 0; base < n; base += blockDim.x * 8) {
        uint64_t xs[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
          uint32_t iq = base + q * blockDim.x + threadIdx.x;
          xs[q] = iq < n ? v[iq] : 0ull;
        }
#pragma unroll
        for (int q = 0; q < 8; q++) {
          if (base + q * blockDim.x + threadIdx.x < n) {
            uint32_t h = (uint32_t)((xs[q] * 0xD6E8FEB86659FD93ull) >> (64 - lgb));
            atomicOr(&bits[h >> 5], 1u << (h & 31));
          }
        }
      }
      __syncthreads();
      uint32_t c = 0;
      for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) c += __popc(bits[i]);
      c = warp_sum(c);
      if ((threadIdx.x & 31) == 0) S.red32[threadIdx.x >> 5] = c;
      __syncthreads();
      uint32_t t = 0;
      for (int w = 0; w < kEncWarps; w++) t += S.red32[w];
      lb = t > lb ? t : lb;
    }
    __syncthreads();
    if (threadIdx.x == 0) S.cnt32 = lb;
    __syncthreads();
  }
  if (S.cnt32 > max_card) {
    if (threadIdx.x == 0) S.flag = 1;
    __syncthreads();
    dv.smem = false;
    dv.sorted = nullptr;
    dv.card = S.cnt32;
    return dv;
  }
  // Scratch path (more than kHashLimit distinct values): a u64 key hash table
  // T[cap] in scratch (cap = pow2 >= n, so the table stays at most about half
  // full for a dictionary that does not bail), the distinct keys compacted and
  // radix-sorted, and a rank table R[cap] beside T for the code lookups.
  // Scratch use: 12*cap + 16*max_card bytes <= 32*n.
  uint32_t cap = pow2_at_least(n), lg = 31 - __clz(cap);
  uint64_t* T = reinterpret_cast<uint64_t*>(scratch);
  uint32_t* R = reinterpret_cast<uint32_t*>(scratch + 8ull * cap);
  uint64_t* A = reinterpret_cast<uint64_t*>(scratch + 12ull * cap);
  uint64_t* B = A + max_card;
  for (uint32_t i = threadIdx.x; i < cap; i += blockDim.x) T[i] = kEmpty64;
  if (threadIdx.x == 0) {
    S.card = 0;
    S.cnt32 = 0;
    S.has_max = 0;
    S.flag = 0;
  }
  __syncthreads();
  for (uint32_t base = 0; base < n; base += blockDim.x * 8) {
    if (__any_sync(0xffffffffu, *(volatile uint32_t*)&S.flag)) break;  // warp-uniform exit
    uint64_t xs[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint32_t iq = base + q * blockDim.x + threadIdx.x;
      xs[q] = iq < n ? v[iq] : 0ull;
    }
    // first probes of the eight values in flight together, then the CASes
    uint32_t hs[8];
    uint64_t cur0[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      hs[q] = (uint32_t)((xs[q] * 0x9E3779B97F4A7C15ull) >> (64 - lg));
      cur0[q] = base + q * blockDim.x + threadIdx.x < n ? T[hs[q]] : 0ull;
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
      if (base + q * blockDim.x + threadIdx.x < n && xs[q] != kEmpty64 && cur0[q] == kEmpty64)
        cur0[q] = atomicCAS((unsigned long long*)&T[hs[q]], kEmpty64, xs[q]);
      else
        cur0[q] = cur0[q] == kEmpty64 ? 1ull : cur0[q];  // (not used: 1 never equals kEmpty64)
    }
    uint32_t mine = 0;  // distinct keys this lane added (counted once per warp below)
#pragma unroll
    for (int q = 0; q < 8; q++) {
      if (base + q * blockDim.x + threadIdx.x >= n) continue;
      uint64_t x = xs[q];
      if (x == kEmpty64) {
        if (atomicExch(&S.has_max, 1u) == 0) mine++;
        continue;
      }
      if (cur0[q] == kEmpty64) {  // the first-probe CAS inserted x
        mine++;
        continue;
      }
      if (cur0[q] == x) continue;
      uint32_t h = (hs[q] + 1) & (cap - 1);
      for (uint32_t probe = 1; probe < cap; probe++) {
        uint64_t cur = T[h];
        if (cur == kEmpty64) {
          cur = atomicCAS((unsigned long long*)&T[h], kEmpty64, x);
          if (cur == kEmpty64) {
            mine++;
            break;
          }
        }
        if (cur == x) break;
        h = (h + 1) & (cap - 1);
      }
    }
    mine = warp_sum(mine);
    if ((threadIdx.x & 31) == 0 && mine && atomicAdd(&S.card, mine) + mine > max_card) S.flag = 1;
  }
  __syncthreads();
  dv.smem = false;
  dv.tkey = T;
  dv.trank = R;
  dv.lg = lg;
  if (S.flag) {  // cardinality > n/2 + 1
    dv.card = S.card;
    dv.sorted = nullptr;
    return dv;
  }
  uint32_t card = S.card, has_max = S.has_max;
  for (uint32_t i0 = threadIdx.x; i0 < cap; i0 += blockDim.x * 8) {
    uint64_t ks[8];
#pragma unroll
    for (int q = 0; q < 8; q++) ks[q] = i0 + q * blockDim.x < cap ? T[i0 + q * blockDim.x] : kEmpty64;
#pragma unroll
    for (int q = 0; q < 8; q++) {  // one counter update per warp and step
      bool ok = ks[q] != kEmpty64;
      uint32_t m = __ballot_sync(0xffffffffu, ok);
      uint32_t base_i = 0;
      if ((threadIdx.x & 31) == 0 && m) base_i = atomicAdd(&S.cnt32, (uint32_t)__popc(m));
      base_i = __shfl_sync(0xffffffffu, base_i, 0);
      if (ok) A[base_i + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = ks[q];
    }
  }
  __syncthreads();
  uint64_t* srt = block_radix_sort(S, A, B, card - has_max);
  if (has_max && threadIdx.x == 0) srt[card - 1] = kEmpty64;
  if (threadIdx.x == 0) S.max_rank = card - 1;
  __syncthreads();
  for (uint32_t r0 = threadIdx.x; r0 + has_max < card; r0 += blockDim.x * 8) {
    uint64_t xs[8];
    uint32_t hs[8];
    uint64_t cur[8];
#pragma unroll
    for (int q = 0; q < 8; q++) xs[q] = r0 + q * blockDim.x + has_max < card ? srt[r0 + q * blockDim.x] : 0ull;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      hs[q] = (uint32_t)((xs[q] * 0x9E3779B97F4A7C15ull) >> (64 - lg));
      cur[q] = r0 + q * blockDim.x + has_max < card ? T[hs[q]] : 0ull;
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint32_t r = r0 + q * blockDim.x;
      if (r + has_max >= card) break;
      uint32_t h = hs[q];
      if (cur[q] != xs[q]) {
        h = (h + 1) & (cap - 1);
        for (uint32_t probe = 1; probe < cap && T[h] != xs[q]; probe++) h = (h + 1) & (cap - 1);
      }
      R[h] = r;
    }
  }
  __syncthreads();
  dv.card = card;
  dv.sorted = srt;
  return dv;
}

// Byte length of the dictionary value blob and its tag (reference dict.rs:40-61).
__device__ uint64_t dict_values_len(EncSmem& S, const DictView& dv, uint32_t* tag) {
  const uint64_t* s = dv.sorted;
  uint64_t raw = 8ull * dv.card;
  uint64_t delta = 8 + block_for(S, nullptr, dv.card, false, [&](uint32_t i) {
                     return zigzag64(s[i] - (i ? s[i - 1] : s[0]));
                   });
  if (delta < raw) {
    *tag = 1;
    return delta;
  }
  *tag = 0;
  return raw;
}

// ---------------------------------------------------------------------------
// RLE run starts (reference rle.rs:10-42).  Requires S.neq_k (transitions per
// sub-block).  Returns the starts, in the first 16 bytes per value of the
// block's scratch.
// ---------------------------------------------------------------------------
__device__ uint32_t* rle_starts(EncSmem& S, const uint64_t* v, uint32_t n, uint8_t* scratch) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* st = reinterpret_cast<uint32_t*>(scratch);
  uint32_t nsub = (n + kSub - 1) / kSub;
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.subsz[k] = S.neq_k[k];
  if (threadIdx.x == 0) st[0] = 0;
  block_offsets(S, nsub, 1);
  // eight rows in flight while the eight before them are compared
  uint64_t xs[8], nx[8];
  auto load = [&](uint32_t k, uint32_t j0, uint64_t (&x)[8]) {
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint32_t i = k * kSub + (j0 + q) * 32 + lane;
      x[q] = k < nsub && i < n ? v[i] : 0ull;
    }
  };
  load(warp, 0, nx);
  for (uint32_t k = warp; k < nsub; k += kEncWarps) {
    uint32_t base = k * kSub, before = S.subsz[k];
    uint64_t carry = base ? v[base - 1] : v[0];
    for (uint32_t j0 = 0; j0 < 32; j0 += 8) {
#pragma unroll
      for (int q = 0; q < 8; q++) xs[q] = nx[q];
      if (j0 < 24) load(k, j0 + 8, nx);
      else load(k + kEncWarps, 0, nx);
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t idx = base + (j0 + q) * 32 + lane;
        uint64_t x = xs[q];
        uint64_t rot = __shfl_sync(0xffffffffu, x, (lane + 31) & 31);
        bool tr = idx < n && x != (lane ? rot : carry);  // the block's first value equals its carry
        carry = rot;
        uint32_t m = __ballot_sync(0xffffffffu, tr);
        if (tr) st[before + __popc(m & ((1u << lane) - 1u))] = idx;
        before += __popc(m);
      }
    }
  }
  __syncthreads();
  return st;
}

// ---------------------------------------------------------------------------
// Entropy stage of the Balanced candidate pool (reference entropy/rans.rs:25-108
// behind the rANS tag of entropy/mod.rs:49-60): static 12-bit frequencies,
// four interleaved states sharing one byte stream, L = 2^23.  A coded part is
// [2][varint(m)][varint(symbols)][(symbol, varint(freq))...][4 x u32 states]
// [bytes].  The encoder runs backward over the input and its state chains
// are sequential, so four lanes run them (rans_run) while the other warps
// stage the next 4096 input bytes in shared memory.
// ---------------------------------------------------------------------------
constexpr uint32_t kRansM = 4096, kRansL = 1u << 23;

// Histogram of byte_at(0 .. m) and the normalised frequencies (rans.rs:25-48:
// f = max(1, c * 4096 / m); while the sum exceeds 4096 the largest f > 1 loses
// one, ties to the highest symbol; a short sum goes to the largest f, ties to
// the highest symbol).  Returns the header length after the tag byte.
template <class B>
__device__ uint32_t rans_plan(RansArea& R, uint32_t m, B byte_at) {
  int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int i = t; i < 256; i += blockDim.x) R.hist[i] = 0;
  __syncthreads();
  for (uint32_t base = (uint32_t)warp * 32; base < m; base += blockDim.x) {
    uint32_t i = base + lane;
    uint32_t sym = i < m ? (uint32_t)byte_at(i) : 256u;
    uint32_t peers = __match_any_sync(0xffffffffu, sym);
    if (sym < 256 && lane == __ffs(peers) - 1) atomicAdd(&R.hist[sym], (uint32_t)__popc(peers));
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t f[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint32_t c = R.hist[lane + 32 * j];
      uint32_t q = (uint32_t)(((uint64_t)c * kRansM) / m);
      f[j] = c ? (q ? q : 1u) : 0u;
      sum += f[j];
    }
    sum = warp_sum(sum);
    while (sum > kRansM) {
      uint32_t key = 0;
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (f[j] > 1) key = max(key, (f[j] << 8) | (uint32_t)(lane + 32 * j));
      key = warp_max(key);
      uint32_t sym = key & 255u;
#pragma unroll
      for (int j = 0; j < 8; j++)
        if ((uint32_t)(lane + 32 * j) == sym) f[j]--;
      sum--;
    }
    if (sum < kRansM) {
      uint32_t key = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) key = max(key, (f[j] << 8) | (uint32_t)(lane + 32 * j));
      key = warp_max(key);
      uint32_t sym = key & 255u;
#pragma unroll
      for (int j = 0; j < 8; j++)
        if ((uint32_t)(lane + 32 * j) == sym) f[j] += kRansM - sum;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) R.fc[lane + 32 * j].x = f[j];
    // A lower bound on the coded bytes: any static model codes the sequence
    // in at least its empirical entropy (Gibbs), and a byte-renormalising
    // four-state coder emits at most 32 bits less (the states' growth from
    // 2^23 to below 2^31) and loses under 2^-11 bits a symbol to the state
    // rounding; a margin of 64 bits covers the floating-point sum.
    double e = 0.0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      uint32_t c = R.hist[lane + 32 * j];
      if (c) e += (double)c * log2((double)m / (double)c);
    }
    for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    double bits = e * (1.0 - 1e-9) - 0.001 * (double)m - 96.0;
    __syncwarp();
    if (lane == 0) {
      R.bound = bits > 0.0 ? (uint32_t)(bits / 8.0) : 0u;
      uint32_t c = 0, present = 0, h = 0;
      for (int sym = 0; sym < 256; sym++) {
        uint32_t fs = R.fc[sym].x;
        R.fc[sym].y = c;
        c += fs;
        if (fs) {
          present++;
          h += 1 + varint_len(fs);
        }
      }
      R.hdr = varint_len(m) + varint_len(present) + h;
    }
  }
  __syncthreads();
  uint32_t hdr = R.hdr;
  __syncthreads();
  return hdr;
}

// Header of a coded part (after its tag byte), from the planned frequencies.
__device__ void rans_put_header(const RansArea& R, uint32_t m, uint8_t* out) {
  uint32_t present = 0;
  for (int sym = 0; sym < 256; sym++) present += R.fc[sym].x ? 1u : 0u;
  uint32_t pos = put_varint(out, m);
  pos += put_varint(out + pos, present);
  for (int sym = 0; sym < 256; sym++)
    if (R.fc[sym].x) {
      out[pos++] = (uint8_t)sym;
      pos += put_varint(out + pos, R.fc[sym].x);
    }
}

// The constants of coding a symbol of frequency f >= 1 and cumulative
// frequency c on a state x < 2^31, x' = ((x / f) << 12) + x % f + c: with
// q = x / f that is x + q * (4096 - f) + c, and q is a multiplication by a
// rounded-up reciprocal (Granlund and Montgomery, "Division by invariant
// integers using multiplication", 1994): for 2^(s-1) < f <= 2^s and
// r = ceil(2^(31+s) / f) < 2^32, q = (x * r) >> (31 + s) for every x < 2^31.
// f = 1 takes r = 2^32 - 1 and a shift of 32, which give q = x - 1, and the
// missing 4095 goes to c.  {f << 19 (renormalisation limit), r, 4096 - f with
// the shift past 32 in the high half, c}.
__device__ __forceinline__ uint4 rans_enc(uint32_t f, uint32_t c) {
  if (f <= 1) return make_uint4(1u << 19, 0xFFFFFFFFu, 4095u, c + 4095u);  // (an absent symbol is never coded)
  uint32_t s = 32 - __clz(f - 1);
  uint32_t r = (uint32_t)(((1ull << (31 + s)) + f - 1) / f);
  return make_uint4(f << 19, r, (kRansM - f) | (s - 1) << 16, c);
}

// Destination of a bit-packed stream of `len` bytes that a block stages for
// rANS: its scratch range (32 B per value) when it fits, else the shared
// big area, free once the ALP-RD dictionary is in S.dict8 (a sub-block pads
// to 1024 values, so a block of fewer than 257 values can exceed its range;
// such a stream is at most varint(n) + 9 + 128 * 64 bytes).
__device__ __forceinline__ uint8_t* stage_dst(EncSmem& S, uint8_t* scr, uint32_t n, uint64_t len) {
  return len <= 32ull * n ? scr : reinterpret_cast<uint8_t*>(&S.big);
}
static_assert(sizeof(BigArea) >= 3 + 9 + 128 * 64, "staged bit-packed stream of a short block");

// The encoder pass over byte_at(m - 1 .. 0) with the planned frequencies.
// Returns the number of stream bytes; WRITE stores them ending at `wend` and
// the four final states in the 16 bytes before the first of them.
//
// The four states code every fourth byte and touch each other only through
// the order of their renormalisation bytes in the stream, so lanes 0..3 of
// warp 0 run one state each, and two votes a step give every lane the place
// of its (at most two) bytes.  What bounds it is a state's dependent chain:
// two comparisons, two selections, the reciprocal's high product, a shift and
// a multiply-add a symbol, issued by one warp (about 50 ns a step of four
// symbols).  One thread running the four chains with divisions took 90 ns a
// byte: compressing 1,000,003 f32 readings and as many f64 prices at
// Balanced-in-pool took 136 ms, with this 21 ms.
template <bool WRITE, class B>
__device__ uint32_t rans_run(RansArea& R, uint32_t m, B byte_at, uint8_t* wend) {
  int t = threadIdx.x, warp = t >> 5, l = t & 31;
  if (t < 256) R.enc[t] = rans_enc(R.fc[t].x, R.fc[t].y);
  uint32_t nch = (m + kRansChunk - 1) / kRansChunk;
  auto fill = [&](uint32_t c, int slot) {  // warps 1.. stage chunk c
    uint32_t lo = c * kRansChunk, hi = min(lo + kRansChunk, m);
    for (uint32_t i = lo + (uint32_t)(t - 32); i < hi; i += blockDim.x - 32) R.buf[slot][i - lo] = (uint8_t)byte_at(i);
  };
  if (warp && nch) fill(nch - 1, 0);
  __syncthreads();
  uint32_t x = kRansL, e = 0;
  uint8_t* p = wend;
  for (uint32_t k = 0; k < nch; k++) {
    uint32_t c = nch - 1 - k;
    if (warp && c > 0) fill(c - 1, (int)((k + 1) & 1));
    if (warp == 0) {
      const uint8_t* bb = R.buf[k & 1];
      const uint32_t cnt = min(kRansChunk, m - c * kRansChunk), sel = l & 3;
      // lanes 4.. repeat the states of lanes 0..3 and write nothing, so a vote
      // holds its four bits in every nibble
      const uint32_t above = ((0xFu << sel << 1) & 0xFu) * 0x11u;
      auto step = [&](const uint4 f, bool act) {
        const uint32_t s1 = x >> 8, s2 = x >> 16;
        const bool b1 = act && x >= f.x, b2 = act && s1 >= f.x;  // a byte leaves, a second one
        if (WRITE) {
          const uint32_t m1 = __ballot_sync(0xffffffffu, b1), m2 = __ballot_sync(0xffffffffu, b2);
          const uint32_t mm = (m1 & 0x0Fu) | (m2 & 0xF0u);
          uint8_t* q = p - __popc(mm & above);  // after the bytes of the states above
          if (b1 && l < 4) q[-1] = (uint8_t)x;
          if (b2 && l < 4) q[-2] = (uint8_t)s1;
          p -= __popc(mm);
        } else {
          e += (b1 ? 1u : 0u) + (b2 ? 1u : 0u);
        }
        uint32_t xs = b1 ? s1 : x;
        xs = b2 ? s2 : xs;
        const uint32_t y = xs + (__umulhi(xs, f.y) >> (f.z >> 16)) * (f.z & 0xFFFFu) + f.w;
        x = act ? y : x;
      };
      // groups of four symbols from the top: the ragged one, then singly down
      // to a multiple of four groups, then four at a time, the constants of a
      // batch fetched during the one before and its bytes one earlier still
      int g = (int)((cnt + 3) / 4) - 1;
      for (; g >= 0 && ((g & 3) != 3 || (uint32_t)(4 * g + 3) >= cnt); g--) {
        bool act = (uint32_t)(4 * g) + sel < cnt;
        step(R.enc[bb[4 * g + (act ? sel : 0u)]], act);
      }
      if (g >= 0) {
        const uint4* bw = reinterpret_cast<const uint4*>(bb);  // batch j: groups 4j .. 4j+3
        auto byte_of = [&](uint32_t w) { return (w >> (8 * sel)) & 255u; };
        int j = g >> 2;
        uint4 w = bw[j];
        uint4 e3 = R.enc[byte_of(w.w)], e2 = R.enc[byte_of(w.z)], e1 = R.enc[byte_of(w.y)], e0 = R.enc[byte_of(w.x)];
        w = bw[j > 0 ? j - 1 : 0];
        for (; j >= 0; j--) {
          const uint4 c3 = e3, c2 = e2, c1 = e1, c0 = e0;
          e3 = R.enc[byte_of(w.w)];
          e2 = R.enc[byte_of(w.z)];
          e1 = R.enc[byte_of(w.y)];
          e0 = R.enc[byte_of(w.x)];
          w = bw[j > 1 ? j - 2 : 0];
          step(c3, true);
          step(c2, true);
          step(c1, true);
          step(c0, true);
        }
      }
    }
    __syncthreads();
  }
  if (warp == 0) {
    e += __shfl_xor_sync(0xffffffffu, e, 1);
    e += __shfl_xor_sync(0xffffffffu, e, 2);
    if (WRITE) e = (uint32_t)(wend - p);
    if (WRITE && l < 4) put_u32(p - 16 + 4 * l, x);
    if (l == 0) R.emitted = e;
  }
  __syncthreads();
  uint32_t r = R.emitted;
  __syncthreads();
  return r;
}

// A lower bound of coded_len: the header, the states and the entropy bound.
template <class B>
__device__ uint32_t coded_min(RansArea& R, uint32_t m, B byte_at) {
  uint32_t h = rans_plan(R, m, byte_at);
  return 1 + h + 16 + R.bound;
}

// Length of code_residuals(byte_at(0 .. m)) with the rANS tag: the coded part
// entropy_pick keeps at lambda >= 2 (m > 0).
template <class B>
// Callers only ask whether the length is below `limit`: when the entropy
// bound already reaches it, the serial sizing pass is skipped and a length at
// or above the limit (the bound) comes back.
__device__ uint32_t coded_len(RansArea& R, uint32_t m, B byte_at, uint64_t limit = ~0ull) {
  uint32_t h = rans_plan(R, m, byte_at);
  uint32_t lo = 1 + h + 16 + R.bound;  // uniform: R is read after rans_plan's barrier
  if ((uint64_t)lo >= limit) return lo;
  return 1 + h + 16 + rans_run<false>(R, m, byte_at, nullptr);
}

// Writes the coded part of byte_at(0 .. m) whose length (tag included) is len.
template <class B>
__device__ void coded_write(RansArea& R, uint32_t m, B byte_at, uint8_t* out, uint32_t len) {
  rans_plan(R, m, byte_at);
  if (threadIdx.x == 0) {
    out[0] = 2;
    rans_put_header(R, m, out + 1);
  }
  rans_run<true>(R, m, byte_at, out + len);
}

// FLOAT_MULT's entropy form (float_mult.rs:66-98): LEB128(zigzag(k_i - k_{i-1}))
// with k_{-1} = 0, written to dst; returns the byte count.  Thread t writes a
// contiguous run of values at offsets from a block scan of their lengths.
__device__ uint32_t fm_delta_bytes(EncSmem& S, const uint64_t* v, uint32_t n, int sc, uint8_t* dst) {
  int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t seg = (n + blockDim.x - 1) / blockDim.x;
  uint32_t i0 = min((uint32_t)t * seg, n), i1 = min(i0 + seg, n);
  uint32_t len = 0;
  int64_t prev = i0 ? fm_k(v[i0 - 1], sc) : 0;
  for (uint32_t i = i0; i < i1; i++) {
    int64_t k = fm_k(v[i], sc);
    len += varint_len(zigzag64((uint64_t)k - (uint64_t)prev));
    prev = k;
  }
  uint32_t inc = warp_incl_scan(len);
  if (lane == 31) S.red32[warp] = inc;
  __syncthreads();
  uint32_t off = inc - len, tot = 0;
  for (int w = 0; w < kEncWarps; w++) {
    if (w < warp) off += S.red32[w];
    tot += S.red32[w];
  }
  prev = i0 ? fm_k(v[i0 - 1], sc) : 0;
  for (uint32_t i = i0; i < i1; i++) {
    int64_t k = fm_k(v[i], sc);
    off += put_varint(dst + off, zigzag64((uint64_t)k - (uint64_t)prev));
    prev = k;
  }
  __syncthreads();
  return tot;
}

// The entropy parts chosen for a block (Balanced in-pool), read by k_emit.
// Lengths include the rANS tag byte.
constexpr uint32_t kEntFm = 1, kEntRdCodes = 2, kEntRdRights = 4, kEntDictVals = 8, kEntDictCodes = 16;
struct EntRec {
  uint32_t flags;
  uint32_t fm;      // FLOAT_MULT coded deltas
  uint32_t rdc;     // ALP-RD coded codes
  uint32_t rdr;     // ALP-RD coded rights (the bit-packed rights bytes)
  uint32_t bt;      // BYTE_TRANSPOSE payload
  uint32_t dv;      // DICT coded transposed values
  uint32_t dc[2];   // DICT coded code planes
};
static_assert(sizeof(EntRec) == 32, "EntRec layout");

struct Cand {
  uint64_t len;
  bool ok;
};

// ---------------------------------------------------------------------------
// Competition, part 1: per-sub-block statistics.  One warp per 1024-value
// sub-block, one pass over the lane.  Quantities that depend on whether the
// sub-block opens a block (its first value's delta / XOR / equality with the
// previous value) are kept out of the internal sums and folded in by k_decide,
// so the statistics are computed before the block plan exists.
// ---------------------------------------------------------------------------
struct SubStats {
  uint64_t umin, umax, first, last, d;  // d = v[1] - v[0] of the sub-block
  int64_t smin, smax;
  uint64_t dzmin, dzmax;                // zigzag deltas of internal pairs (j >= 1)
  uint64_t e16min, e16max, e16dz;       // early-out samples j % 16 == 0
  uint64_t e64min, e64max, e64dz;       // early-out samples j % 64 == 0
  uint32_t xb, neq, cnt;                // internal XORZ bytes, internal transitions, values
  uint8_t stride_ok, alp_ok, alp_w, fm_pass;
  uint16_t alp_exc, pad16;
  uint32_t pad32;
};
static_assert(sizeof(SubStats) == 144, "SubStats layout");
struct FmStat {  // signed min / max of k = round(x * scale) per FLOAT_MULT scale
  int64_t kmin[7], kmax[7];
};

// Adaptive mode: a cluster of four CTAs of eight warps per 32,768-value window,
// so that a column of few windows runs on four times as many SMs.
constexpr int kStatsWarps = 8, kStatsCluster = 4;
static_assert(kStatsWarps * kStatsCluster * kSub == kBaseQuantum, "a cluster covers a window");

// Start and length of statistics item `item` (one 1024-value sub-block): with
// a fixed block size the sub-blocks restart at every block boundary.
__device__ inline uint32_t sub_range(uint64_t item, uint64_t n, uint64_t fixed_bs, uint64_t* s) {
  if (fixed_bs) {
    uint64_t spb = (fixed_bs + kSub - 1) / kSub;
    uint64_t b = item / spb, k = item % spb;
    uint64_t bstart = b * fixed_bs, bend = qmin(bstart + fixed_bs, n);
    *s = bstart + k * kSub;
    return (bstart < n && *s < bend) ? (uint32_t)qmin(kSub, bend - *s) : 0u;
  }
  *s = item * kSub;
  return *s < n ? (uint32_t)qmin(kSub, n - *s) : 0u;
}

// ALP statistics of every sub-block (alp.rs:49-166), for float lanes at Fast
// and above: one warp per sub-block, after k_sub_stats (whose records it
// completes).  The power-of-ten tables are copied to shared memory, since the
// (e, f) search reads them at a different index in every lane.
constexpr int kAlpWarps = 8;
constexpr uint16_t kAlpEfKnown = 0x8000;  // SubStats::pad16 holds e | f << 8 of a sub-block that passed
__device__ __forceinline__ void alp_stats(const uint32_t cta, const uint64_t* __restrict__ v, uint64_t n,
                                          const uint64_t* d_n, uint64_t fixed_bs, uint64_t items,
                                          SubStats* __restrict__ ss) {
  __shared__ uint64_t smp[kAlpWarps][32];
  __shared__ double pexp[19], pfrac[19];
  if (d_n) n = *d_n;
  if (threadIdx.x < 19) {
    pexp[threadIdx.x] = kExp10[threadIdx.x];
    pfrac[threadIdx.x] = kFrac10[threadIdx.x];
  }
  __syncthreads();
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t item = (uint64_t)cta * kAlpWarps + warp;
  if (item >= items) return;
  uint64_t s;
  uint32_t cnt = sub_range(item, n, fixed_bs, &s);
  if (!cnt) return;
  AlpSub a;
  bool ok = alp_subblock(v + s, cnt, smp[warp], pexp, pfrac, &a);
  if (lane == 0) {
    ss[item].alp_ok = ok ? 1 : 0;
    ss[item].alp_w = ok ? (uint8_t)a.w : 0;
    ss[item].alp_exc = ok ? (uint16_t)a.exc : 0;
    ss[item].pad16 = ok ? (uint16_t)(kAlpEfKnown | a.e | (a.f << 8)) : 0;  // the emitter reuses (e, f)
  }
}

// A lane's share of a sub-block's statistics.
struct StatAcc {
  uint64_t umn = kEmpty64, umx = 0, dzmn = kEmpty64, dzmx = 0;
  int64_t smn = INT64_MAX, smx = INT64_MIN;
  uint32_t nq = 0, xb = 0, fmfail = 0;
  int64_t kmn[7], kmx[7];
};
// FLOAT_MULT's scales still alive on value x: the failing ones' bits set, the
// others' digit ranges widened (float_mult.rs:45-64).
__device__ __forceinline__ void fm_value(uint64_t x, uint32_t alive, StatAcc& A) {
  double xd = as_f64(x);
  while (alive) {
    int q = __ffs(alive) - 1;
    alive &= alive - 1;
    double sc = kFmScales[q];
    double k = round_half_away(__dmul_rn(xd, sc));
    bool good = is_finite_f64(k) && fabs(k) < 9.0e18 && f64_bits(__ddiv_rn(k, sc)) == x;
    if (!good) {
      A.fmfail |= 1u << q;
    } else {
      int64_t ki = __double2ll_rz(k);
#pragma unroll
      for (int j = 0; j < 7; j++)
        if (j == q) {
          A.kmn[j] = ki < A.kmn[j] ? ki : A.kmn[j];
          A.kmx[j] = ki > A.kmx[j] ? ki : A.kmx[j];
        }
    }
  }
}
// LEB128 bytes of v, with one leading-zero count.
__device__ __forceinline__ uint32_t leb_len(uint32_t lo, uint32_t hi) {
  const uint32_t h = hi ? hi : lo | 1u;
  const uint32_t bits = (hi ? 64u : 32u) - __clz(h);
  return (bits + 6) * 37 >> 8;  // (bits + 6) / 7 for bits <= 64
}

// A whole sub-block's rows.  KIND: 0 u64 lane, 1 i64, 2 i32, 3 u32, 4 floats.
// Issue slots bound this pass (59 % busy, the integer pipe 52 %; 122 a row of
// 32 values and 350 us for 60,000,000 values before, now 96 and 267 us), so it
// carries no per-value test: value 0's predecessor is chosen to
// repeat the first delta (its XOR bytes and transition are taken off at the
// end), the signed kinds derive the unsigned range unless a sub-block mixes
// signs (then a second pass over its values, in L1), 4-byte columns compare
// 32-bit words.
template <int KIND, bool LB>
__device__ __forceinline__ void stats_rows(const uint64_t* __restrict__ sv, uint32_t* lbits, uint32_t alive,
                                           StatAcc& A) {
  const int lane = threadIdx.x & 31;
  constexpr bool W32 = KIND == 2 || KIND == 3;
  const uint64_t x0 = sv[0], d0 = sv[1] - x0;
  uint64_t carry = x0 - d0;
  uint32_t umn32 = 0xFFFFFFFFu, umx32 = 0;
  int32_t smn32 = INT32_MAX, smx32 = INT32_MIN;
  for (uint32_t r0 = 0; r0 < 32; r0 += 8) {
    uint64_t xs[8];  // eight independent loads in flight per lane
#pragma unroll
    for (int q = 0; q < 8; q++) xs[q] = sv[(r0 + q) * 32 + lane];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const uint64_t x = xs[q];
      uint64_t pv;
      if (W32) {
        const uint32_t rot = __shfl_sync(0xffffffffu, (uint32_t)x, (lane + 31) & 31);
        const uint64_t r64 = KIND == 2 ? (uint64_t)(int64_t)(int32_t)rot : (uint64_t)rot;
        pv = lane ? r64 : carry;
        carry = r64;
      } else {
        const uint64_t rot = __shfl_sync(0xffffffffu, x, (lane + 31) & 31);
        pv = lane ? rot : carry;
        carry = rot;
      }
      if (W32) {
        umn32 = min(umn32, (uint32_t)x);
        umx32 = max(umx32, (uint32_t)x);
        if (KIND == 2) {
          smn32 = min(smn32, (int32_t)(uint32_t)x);
          smx32 = max(smx32, (int32_t)(uint32_t)x);
        }
      } else if (KIND == 1) {
        A.smn = (int64_t)x < A.smn ? (int64_t)x : A.smn;
        A.smx = (int64_t)x > A.smx ? (int64_t)x : A.smx;
      } else {
        A.umn = u64min(A.umn, x);
        A.umx = u64max(A.umx, x);
      }
      const uint64_t dz = zigzag64(x - pv), xo = x ^ pv;
      A.dzmn = u64min(A.dzmn, dz);
      A.dzmx = u64max(A.dzmx, dz);
      A.xb += leb_len((uint32_t)xo, (uint32_t)(xo >> 32));
      if (xo) {
        A.nq++;
        if (LB) {  // a repeat's bucket is already set
          const uint32_t b = dict_lb_bucket(x);
          atomicOr(&lbits[b >> 5], 1u << (b & 31));
        }
      }
      if (KIND == 4 && alive) {
        fm_value(x, alive, A);
        alive &= ~__reduce_or_sync(0xffffffffu, A.fmfail);  // a scale that failed anywhere in the sub-block is out
      }
    }
  }
  if (lane == 0) {
    const uint64_t xo = x0 ^ (x0 - d0);
    A.xb -= leb_len((uint32_t)xo, (uint32_t)(xo >> 32));
    if (xo) A.nq--;
    if (LB) {
      const uint32_t b = dict_lb_bucket(x0);
      atomicOr(&lbits[b >> 5], 1u << (b & 31));
    }
  }
  if (KIND == 2) {
    A.smn = smn32;
    A.smx = smx32;
    A.umn = (uint64_t)(int64_t)(int32_t)umn32;  // sign extension keeps the unsigned order
    A.umx = (uint64_t)(int64_t)(int32_t)umx32;
  } else if (KIND == 3) {
    A.umn = umn32;
    A.umx = umx32;
  } else if (KIND == 1) {
    if (__any_sync(0xffffffffu, A.smn < 0) && __any_sync(0xffffffffu, A.smx >= 0)) {
      for (uint32_t r = 0; r < 32; r++) {
        const uint64_t x = sv[r * 32 + lane];
        A.umn = u64min(A.umn, x);
        A.umx = u64max(A.umx, x);
      }
    } else {
      A.umn = (uint64_t)A.smn;
      A.umx = (uint64_t)A.smx;
    }
  }
}
// The rows of a sub-block of fewer than 1,024 values.
__device__ __noinline__ void stats_partial(const uint64_t* __restrict__ sv, uint32_t cnt, bool lb, uint32_t* lbits,
                                           uint32_t alive, StatAcc& A) {
  const int lane = threadIdx.x & 31;
  for (uint32_t j0 = 0; j0 < cnt; j0 += 32) {
    const uint32_t j = j0 + lane;
    if (j < cnt) {
      const uint64_t x = sv[j], pv = j ? sv[j - 1] : x;
      A.umn = u64min(A.umn, x);
      A.umx = u64max(A.umx, x);
      A.smn = (int64_t)x < A.smn ? (int64_t)x : A.smn;
      A.smx = (int64_t)x > A.smx ? (int64_t)x : A.smx;
      if (j > 0) {
        const uint64_t dz = zigzag64(x - pv);
        A.dzmn = u64min(A.dzmn, dz);
        A.dzmx = u64max(A.dzmx, dz);
        A.xb += varint_len(x ^ pv);
        A.nq += x != pv ? 1u : 0u;
      }
      if (lb) {
        const uint32_t b = dict_lb_bucket(x);
        atomicOr(&lbits[b >> 5], 1u << (b & 31));
      }
      if (alive) fm_value(x, alive, A);
    }
    if (alive) alive &= ~__reduce_or_sync(0xffffffffu, A.fmfail);
  }
}

template <bool FLOATS>
__device__ __forceinline__ void sub_stats(
    const uint32_t cta, const uint64_t* __restrict__ v, uint64_t n, const uint64_t* d_n, uint64_t fixed_bs, uint64_t items, int dtype,
    int level, SubStats* __restrict__ ss, FmStat* __restrict__ fms, uint64_t* __restrict__ smp16, uint8_t* __restrict__ grow,
    uint32_t* __restrict__ winbits) {
  __shared__ uint32_t bitsA[512], bitsB[512];
  __shared__ uint32_t lbits[kLbBits / 32];  // dictionary cardinality lower bound (the CTA's share of the window)
  __shared__ uint32_t s_lbc, s_dc;
  __shared__ uint64_t s_first[kStatsWarps], s_last[kStatsWarps];
  __shared__ uint32_t s_neq[kStatsWarps], s_cnt[kStatsWarps];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (d_n) n = *d_n;
  const bool do_float = FLOATS && level >= 1;
  uint64_t item = (uint64_t)cta * kStatsWarps + warp;
  const uint64_t win = cta / kStatsCluster;
  uint64_t s = 0;
  uint32_t cnt = item < items ? sub_range(item, n, fixed_bs, &s) : 0u;
  // window probe sampling (adaptive): window-relative stride max(len/4096, 1)
  uint64_t wstart = win * kBaseQuantum;
  uint32_t wlen = fixed_bs ? 0u : (uint32_t)(wstart < n ? qmin(kBaseQuantum, n - wstart) : 0);
  uint32_t wstride = max(wlen / 4096u, 1u);
  const bool sgn = dtype_signed(dtype);
  if (!fixed_bs) {
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
      bitsA[i] = 0;
      bitsB[i] = 0;
    }
    for (int i = threadIdx.x; i < (int)(kLbBits / 32); i += blockDim.x) lbits[i] = 0;
    if (threadIdx.x == 0) s_lbc = s_dc = 0;
    __syncthreads();
  }
  SubStats R;
  StatAcc A;
#pragma unroll
  for (int q = 0; q < 7; q++) {
    A.kmn[q] = INT64_MAX;
    A.kmx[q] = INT64_MIN;
  }
  const uint64_t* sv = v + s;
  uint64_t d = cnt >= 2 ? sv[1] - sv[0] : 0;
  const uint32_t alive = do_float ? 0x7Fu : 0u;
  if (cnt < (uint32_t)kSub) {
    stats_partial(sv, cnt, !fixed_bs, lbits, alive, A);
  } else if (FLOATS) {
    if (fixed_bs) stats_rows<4, false>(sv, lbits, alive, A);
    else stats_rows<4, true>(sv, lbits, alive, A);
  } else if (dtype == DT_I64) {
    if (fixed_bs) stats_rows<1, false>(sv, lbits, 0, A);
    else stats_rows<1, true>(sv, lbits, 0, A);
  } else if (dtype == DT_I32) {
    if (fixed_bs) stats_rows<2, false>(sv, lbits, 0, A);
    else stats_rows<2, true>(sv, lbits, 0, A);
  } else if (dtype == DT_U32) {
    if (fixed_bs) stats_rows<3, false>(sv, lbits, 0, A);
    else stats_rows<3, true>(sv, lbits, 0, A);
  } else {
    if (fixed_bs) stats_rows<0, false>(sv, lbits, 0, A);
    else stats_rows<0, true>(sv, lbits, 0, A);
  }
  // Sampled statistics, kept out of the per-value loop (only a few lanes of a
  // row would take them): early-out samples at j % 16 / j % 64 == 0 (integer
  // lanes), the ALP-RD sample (float lanes) and the window probe samples
  // (stride wstride, and stride 32).
  uint64_t a16mn = kEmpty64, a16mx = 0, a16dz = 0, a64mn = kEmpty64, a64mx = 0, a64dz = 0;
  if (FLOATS) {
    if (smp16 && !fixed_bs)
      for (uint32_t j = 16u * lane; j < cnt; j += 512) smp16[(s + j) >> 4] = sv[j];
  } else {
    for (uint32_t j = 16u * lane; j < cnt; j += 512) {
      uint64_t x = sv[j], pv = j ? sv[j - 1] : 0ull;
      a16mn = u64min(a16mn, x);
      a16mx = u64max(a16mx, x);
      if (j > 0) a16dz = u64max(a16dz, zigzag64(x - pv));
      if ((j & 63) == 0) {
        a64mn = u64min(a64mn, x);
        a64mx = u64max(a64mx, x);
        if (j > 0) a64dz = u64max(a64dz, zigzag64(x - pv));
      }
    }
  }
  if (!fixed_bs && cnt) {
    uint32_t off = (uint32_t)(s - wstart) % wstride;
    for (uint32_t j = (off ? wstride - off : 0u) + wstride * lane; j < cnt; j += wstride * 32) {
      uint32_t bk = (uint32_t)(((sv[j] * 0x9E3779B97F4A7C15ull) >> 50) & 0x3FFF);
      atomicOr(&bitsA[bk >> 5], 1u << (bk & 31));
    }
    uint32_t jb = 32u * lane;  // window offset of the sub-block is a multiple of 1024
    if (jb < cnt) {
      uint32_t bk = (uint32_t)(((sv[jb] * 0x9E3779B97F4A7C15ull) >> 50) & 0x3FFF);
      atomicOr(&bitsB[bk >> 5], 1u << (bk & 31));
    }
  }
  R.umin = warp_min(A.umn);
  R.umax = warp_max(A.umx);
  R.smin = sgn ? warp_min_i64(A.smn) : 0;
  R.smax = sgn ? warp_max_i64(A.smx) : 0;
  R.dzmin = warp_min(A.dzmn);
  R.dzmax = warp_max(A.dzmx);
  R.e16min = R.e16max = R.e16dz = R.e64min = R.e64max = R.e64dz = 0;
  if (!FLOATS) {
    R.e16min = warp_min(a16mn);
    R.e16max = warp_max(a16mx);
    R.e16dz = warp_max(a16dz);
    R.e64min = warp_min(a64mn);
    R.e64max = warp_max(a64mx);
    R.e64dz = warp_max(a64dz);
  }
  R.xb = __reduce_add_sync(0xffffffffu, A.xb);
  R.neq = __reduce_add_sync(0xffffffffu, A.nq);
  // every internal delta equals d exactly when the zigzag deltas are all zigzag(d)
  R.stride_ok = (cnt < 2 || (R.dzmin == R.dzmax && R.dzmax == zigzag64(d))) ? 1 : 0;
  R.cnt = cnt;
  R.first = cnt ? sv[0] : 0;
  R.last = cnt ? sv[cnt - 1] : 0;
  R.d = d;
  R.fm_pass = do_float ? (uint8_t)(0x7Fu & ~__reduce_or_sync(0xffffffffu, A.fmfail)) : 0;
  R.alp_ok = 0;
  R.alp_w = 0;
  R.alp_exc = 0;
  R.pad16 = 0;
  R.pad32 = 0;
  if (FLOATS && do_float && item < items) {
#pragma unroll
    for (int q = 0; q < 7; q++) {
      if (!(R.fm_pass >> q & 1)) continue;  // only a passing scale's range is read
      int64_t a = warp_min_i64(A.kmn[q]), b = warp_max_i64(A.kmx[q]);
      if (lane == 0) {
        fms[item].kmin[q] = a;
        fms[item].kmax[q] = b;
      }
    }
  }
  if (lane == 0) {
    if (item < items) ss[item] = R;
    s_first[warp] = R.first;
    s_last[warp] = R.last;
    s_neq[warp] = R.neq;
    s_cnt[warp] = cnt;
  }
  if (fixed_bs) return;
  // Window probe (reference encoder.rs:166-176, 705-750): grow the block at
  // this window when the sampled distinct count is low or most consecutive
  // values repeat.  consec_eq = len - transitions (the first element counts
  // against itself).  Each CTA of the cluster joins a quarter of the bitsets;
  // the first takes the counts.
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  const uint32_t rank = cl.block_rank();
  {
    uint32_t c = 0, dc = 0;
    const uint32_t *lb[kStatsCluster], *ba[kStatsCluster], *bb[kStatsCluster];
#pragma unroll
    for (int k = 0; k < kStatsCluster; k++) {
      lb[k] = cl.map_shared_rank(lbits, k);
      ba[k] = cl.map_shared_rank(bitsA, k);
      bb[k] = cl.map_shared_rank(bitsB, k);
    }
    constexpr uint32_t kLbPart = kLbBits / 32 / kStatsCluster, kBitPart = 512 / kStatsCluster;
    for (uint32_t i = rank * kLbPart + threadIdx.x; i < (rank + 1) * kLbPart; i += blockDim.x)
      c += __popc(lb[0][i] | lb[1][i] | lb[2][i] | lb[3][i]);
    for (uint32_t i = rank * kBitPart + threadIdx.x; i < (rank + 1) * kBitPart; i += blockDim.x) {
      const uint32_t x = ba[0][i] | ba[1][i] | ba[2][i] | ba[3][i], y = bb[0][i] | bb[1][i] | bb[2][i] | bb[3][i];
      dc += __popc(x);
      winbits[win * kWinWords + i] = x;
      winbits[win * kWinWords + 512 + i] = y;
    }
    static_assert(kStatsCluster == 4, "four shares are joined");
    c = __reduce_add_sync(0xffffffffu, c);
    dc = __reduce_add_sync(0xffffffffu, dc);
    if (lane == 0 && c) atomicAdd(cl.map_shared_rank(&s_lbc, 0), c);
    if (lane == 0 && dc) atomicAdd(cl.map_shared_rank(&s_dc, 0), dc);
  }
  uint32_t tr = 0;
  if (rank == 0 && warp == 0) {  // a lane per sub-block of the window
    const int k = lane / kStatsWarps, w = lane % kStatsWarps;
    if (cl.map_shared_rank(s_cnt, k)[w]) {
      tr = cl.map_shared_rank(s_neq, k)[w];
      const uint64_t f = cl.map_shared_rank(s_first, k)[w];
      if (lane > 0 && f != (w ? cl.map_shared_rank(s_last, k)[w - 1]
                              : cl.map_shared_rank(s_last, k - 1)[kStatsWarps - 1]))
        tr++;
    }
    tr = __reduce_add_sync(0xffffffffu, tr);
  }
  cl.sync();  // the counts are in, and no CTA's shared memory is read any more
  if (rank == 0 && threadIdx.x == 0) {
    winbits[win * kWinWords + 1024] = s_lbc;
    if (wlen) {
      uint32_t consec = wlen - tr;
      grow[win] = (s_dc < 2048 || (uint64_t)consec * 2 > wlen) ? 1 : 0;
    }
  }
}

// ---------------------------------------------------------------------------
// Competition, part 2: one CTA per block.  Candidate sizes in closed form
// from the sub-block statistics, the integer early-out, the ALP-RD cut search,
// and the DICT / RLE passes for compressible blocks (encoder.rs:275-469).
// ---------------------------------------------------------------------------
__device__ uint32_t popc_bits_block(EncSmem& S, const uint32_t* bits) {
  uint32_t c = 0;
  for (int i = threadIdx.x; i < 512; i += blockDim.x) c += __popc(bits[i]);
  c = warp_sum(c);
  if ((threadIdx.x & 31) == 0) S.red32[threadIdx.x >> 5] = c;
  __syncthreads();
  uint32_t t = 0;
  for (int w = 0; w < kEncWarps; w++) t += S.red32[w];
  __syncthreads();
  return t;
}

// ---------------------------------------------------------------------------
// Selection::Sample (reference encoder.rs:470-620) at Fastest and Fast: the
// candidate modes are sized on a stratified sample of the block (8 runs of 64
// values spread over it, or the whole block up to 512 values) and the
// smallest estimate, first in SAMPLE_MODES order on ties, is the one encoded
// in full.  The in-pool members at these levels: Xorz, ForBitpack,
// DeltaBitpack, Alp and AlpRd (float columns), Dict, Rle; FloatMult and
// ByteTranspose are entropy modes (Balanced and above).
// ---------------------------------------------------------------------------
__device__ __noinline__ int sample_winner(EncSmem& S, const uint64_t* v, uint32_t n, int dtype, uint8_t* scr) {
  int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint64_t* smp = reinterpret_cast<uint64_t*>(&S.ra.buf[0][0]);  // 512 values (the rANS staging is idle)
  uint32_t m = n <= 512u ? n : 512u;
  for (uint32_t i = t; i < m; i += blockDim.x) {
    uint32_t src = i;
    if (n > 512u) {  // build_sample: run r starts at r * (n - 64) / 7
      uint32_t r = i >> 6;
      src = (uint32_t)((uint64_t)r * (n - 64u) / 7u) + (i & 63u);
    }
    smp[i] = v[src];
  }
  if (t == 0) {
    S.sc[0] = 0;            // XORZ bytes
    S.sc[1] = kEmpty64;     // unsigned min
    S.sc[2] = 0;            // unsigned max
    S.sc[3] = kEmpty64;     // signed min, as x ^ 2^63 (signed order in unsigned compares)
    S.sc[4] = 0;            // signed max, likewise
    S.sc[5] = kEmpty64;     // zigzag delta min
    S.sc[6] = 0;            // zigzag delta max
    S.cnt32 = 0;            // transitions
  }
  __syncthreads();
  const bool fl = dtype_float(dtype), sgn = dtype_signed(dtype);
  const uint64_t kBias = 0x8000000000000000ull;  // signed order as unsigned order
  {
    uint64_t xb = 0, umn = kEmpty64, umx = 0, bmn = kEmpty64, bmx = 0, dmn = kEmpty64, dmx = 0;
    uint32_t tr = 0;
    for (uint32_t i = t; i < m; i += blockDim.x) {
      uint64_t x = smp[i], pv = i ? smp[i - 1] : 0ull;
      xb += varint_len(x ^ pv);
      umn = u64min(umn, x);
      umx = u64max(umx, x);
      bmn = u64min(bmn, x ^ kBias);
      bmx = u64max(bmx, x ^ kBias);
      uint64_t dz = i ? zigzag64(x - pv) : 0ull;  // delta_bitpack: d_0 = 0
      dmn = u64min(dmn, dz);
      dmx = u64max(dmx, dz);
      tr += (i && x != pv) ? 1u : 0u;
    }
    xb = warp_sum(xb);
    umn = warp_min(umn);
    umx = warp_max(umx);
    bmn = warp_min(bmn);
    bmx = warp_max(bmx);
    dmn = warp_min(dmn);
    dmx = warp_max(dmx);
    tr = warp_sum(tr);
    if (lane == 0) {
      atomicAdd((unsigned long long*)&S.sc[0], (unsigned long long)xb);
      atomic_min_u64((unsigned long long*)&S.sc[1], umn);
      atomic_max_u64((unsigned long long*)&S.sc[2], umx);
      atomic_min_u64((unsigned long long*)&S.sc[3], bmn);
      atomic_max_u64((unsigned long long*)&S.sc[4], bmx);
      atomic_min_u64((unsigned long long*)&S.sc[5], dmn);
      atomic_max_u64((unsigned long long*)&S.sc[6], dmx);
      atomicAdd(&S.cnt32, tr);
    }
  }
  __syncthreads();
  uint64_t vl = varint_len(m);
  uint64_t est_xorz = S.sc[0];
  uint64_t est_for = vl + 9 + 128ull * bit_width64(sgn ? S.sc[4] - S.sc[3] : S.sc[2] - S.sc[1]);
  uint64_t est_delta = 8 + vl + 9 + 128ull * bit_width64(S.sc[6] - S.sc[5]);
  uint32_t transitions = S.cnt32;
  __syncthreads();
  int win = M_XORZ;
  uint64_t win_est = est_xorz;
  auto take = [&](int mode, uint64_t est) {
    if (est < win_est) {
      win_est = est;
      win = mode;
    }
  };
  take(M_FOR_BITPACK, est_for);
  take(M_DELTA_BITPACK, est_delta);
  if (fl) {
    // ALP (alp.rs:93-166): one sub-block
    if (warp == 0) {
      AlpSub a;
      bool ok = alp_subblock(smp, m, S.alp_smp[0], kExp10, kFrac10, &a);
      if (lane == 0) S.sc[7] = ok ? vl + 13 + 128ull * a.w + 10ull * a.exc : kEmpty64;
    }
    __syncthreads();
    uint64_t est_alp = S.sc[7];
    __syncthreads();
    if (est_alp != kEmpty64) take(M_ALP, est_alp);
    // ALP-RD (alp_rd.rs:132-206), bit-packed streams
    uint32_t lbw = rd_choose_cut(S, smp, m, nullptr, 0);
    if (lbw) {
      rd_top8(S, smp, m, lbw, scr);
      uint32_t rbw = 64 - lbw;
      uint64_t rmask = (1ull << rbw) - 1ull;
      if (t == 0) {
        S.sc[0] = 0;         // exception bytes
        S.sc[1] = kEmpty64;  // code min
        S.sc[2] = 0;         // code max
        S.sc[3] = kEmpty64;  // right min
        S.sc[4] = 0;         // right max
        S.cnt32 = 0;         // exceptions
      }
      __syncthreads();
      uint64_t eb = 0, cmn = kEmpty64, cmx = 0, rmn = kEmpty64, rmx = 0;
      uint32_t ne = 0;
      for (uint32_t i = t; i < m; i += blockDim.x) {
        uint64_t x = smp[i];
        int c = rd_code(S, x >> rbw);
        uint64_t code = c < 0 ? 0ull : (uint64_t)c;
        if (c < 0) {
          ne++;
          eb += varint_len(i) + 8;
        }
        cmn = u64min(cmn, code);
        cmx = u64max(cmx, code);
        rmn = u64min(rmn, x & rmask);
        rmx = u64max(rmx, x & rmask);
      }
      eb = warp_sum(eb);
      ne = warp_sum(ne);
      cmn = warp_min(cmn);
      cmx = warp_max(cmx);
      rmn = warp_min(rmn);
      rmx = warp_max(rmx);
      if (lane == 0) {
        atomicAdd((unsigned long long*)&S.sc[0], (unsigned long long)eb);
        atomic_min_u64((unsigned long long*)&S.sc[1], cmn);
        atomic_max_u64((unsigned long long*)&S.sc[2], cmx);
        atomic_min_u64((unsigned long long*)&S.sc[3], rmn);
        atomic_max_u64((unsigned long long*)&S.sc[4], rmx);
        atomicAdd(&S.cnt32, ne);
      }
      __syncthreads();
      uint64_t nexc = S.cnt32;
      uint64_t clen = vl + 9 + 128ull * bit_width64(S.sc[2] - S.sc[1]);
      uint64_t rlen = vl + 9 + 128ull * bit_width64(S.sc[4] - S.sc[3]);
      if (nexc * 4 <= m)
        take(M_ALP_RD, 2 + 8ull * S.dl + varint_len(nexc) + S.sc[0] + 1 + varint_len(clen) + clen + 1 + rlen);
      __syncthreads();
    }
  }
  // DICT (dict.rs:87-152), bit-packed codes
  DictView dv = dict_prepare(S, smp, m, scr, kNoLb);
  if (!S.flag) {
    uint32_t vtag;
    uint64_t vlen = dict_values_len(S, dv, &vtag);
    if (t == 0) {
      S.sc[1] = kEmpty64;
      S.sc[2] = 0;
    }
    __syncthreads();
    uint64_t rmn = kEmpty64, rmx = 0;
    for (uint32_t i = t; i < m; i += blockDim.x) {
      uint64_t r = dict_rank(S, dv, smp[i]);
      rmn = u64min(rmn, r);
      rmx = u64max(rmx, r);
    }
    rmn = warp_min(rmn);
    rmx = warp_max(rmx);
    if (lane == 0) {
      atomic_min_u64((unsigned long long*)&S.sc[1], rmn);
      atomic_max_u64((unsigned long long*)&S.sc[2], rmx);
    }
    __syncthreads();
    uint64_t clen = vl + 9 + 128ull * bit_width64(S.sc[2] - S.sc[1]);
    take(M_DICT, varint_len(dv.card) + 1 + varint_len(vlen) + vlen + 1 + clen);
  }
  __syncthreads();
  // RLE (rle.rs:10-42): completed runs beyond m/2 + 1 bail
  if (transitions <= m / 2 + 1) {
    if (t == 0) {
      uint32_t runs = transitions + 1, start = 0, lmn = 0xFFFFFFFFu, lmx = 0;
      for (uint32_t i = 1; i <= m; i++)
        if (i == m || smp[i] != smp[i - 1]) {
          uint32_t len = i - start;
          lmn = min(lmn, len);
          lmx = max(lmx, len);
          start = i;
        }
      S.sc[0] = varint_len(runs) + 8ull * runs + varint_len(runs) + 9 + 128ull * bit_width64((uint64_t)(lmx - lmn));
    }
    __syncthreads();
    take(M_RLE, S.sc[0]);
  }
  __syncthreads();
  return win;
}

// ENT: the Balanced in-pool competition, with the rANS-coded forms of
// FLOAT_MULT, ALP-RD and DICT and the BYTE_TRANSPOSE candidate; the chosen
// coded parts go to ent[b] for the emission.
template <bool ENT, bool SAMPLE>
__device__ __forceinline__ void decide(const uint32_t b, const uint64_t* __restrict__ lane, FrameDesc* frames,
                                       const uint32_t* __restrict__ nbp, uint64_t fixed_bs, int dtype, int level,
                                       const SubStats* __restrict__ ss, const FmStat* __restrict__ fms,
                                       const uint64_t* __restrict__ smp16, const uint32_t* __restrict__ winbits,
                                       uint8_t* __restrict__ scratch, EntRec* __restrict__ ent,
                                       RdRec* __restrict__ rdr, BlkRec* __restrict__ blk) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  EncSmem& S = *reinterpret_cast<EncSmem*>(smem_raw);
  if (b >= *nbp) return;
  FrameDesc fd = frames[b];
  const uint64_t* v = lane + fd.value_off;
  uint32_t n = fd.n;
  uint8_t* scr = scratch + fd.value_off * kEncScratchPerValue;
  bool fam_float = dtype_float(dtype);
  bool reduced = level == 0;
  bool sgn = dtype_signed(dtype);
  uint64_t lambda = level_lambda(level);
  uint64_t lb = lane_bytes(dtype);
  uint64_t decoded_bytes = (uint64_t)n * lb, raw_bytes = (uint64_t)n * 8;
  uint32_t nsub = (n + kSub - 1) / kSub;
  uint64_t g0 = fixed_bs ? (uint64_t)b * ((fixed_bs + kSub - 1) / kSub) : fd.value_off / kSub;
  int t = threadIdx.x, lane_id = t & 31, warp = t >> 5;
  uint32_t step = max(n / 2048u, 1u);
  EntRec er = {0, 0, 0, 0, 0, 0, {0, 0}};
  // Early-out samples from the statistics when the block is a full adaptive block.
  bool pre_e = !fixed_bs && (step == 16 || step == 64) && (fd.value_off % kBaseQuantum) == 0;
  if (t == 0) {
    S.xor_bytes = 0;
    S.umin = kEmpty64;
    S.umax = 0;
    S.e_vmin = kEmpty64;
    S.e_vmax = 0;
    S.e_dmax = 0;
    S.neq = 0;
    S.stride_bad = 0;
    S.fm_mask = 0x7F;
    S.alp_fail = 0;
    S.acc64 = 0;
    S.sc[1] = 0;
    S.sc[2] = 0;
    S.sc[4] = 0;
  }
  __syncthreads();
  uint64_t D = n >= 2 ? v[1] - v[0] : 0;
  // One sub-block per thread (at most 128); the lanes' results are reduced by
  // shuffles, so that a warp updates each shared quantity once (with an atomic
  // per sub-block, whose 64-bit minima are compare-and-swap loops, this took
  // 9 us of a 32,768-value block's 13).
  if (warp * 32 < (int)nsub) {
    const uint32_t k = t;
    const bool in = k < nsub;
    SubStats R;
    uint64_t pl = 0, fsz = 0, dsz = 0, asz = 0, xbytes = 0;
    uint64_t emn = kEmpty64, emx = 0, edz = 0, umn = kEmpty64, umx = 0;
    uint32_t nq = 0, pass = 0x7F;
    bool sbad = false, abad = false;
    if (in) {
      R = ss[g0 + k];
      if (k) pl = ss[g0 + k - 1].last;
      uint32_t wf = sgn ? bit_width64((uint64_t)R.smax - (uint64_t)R.smin) : bit_width64(R.umax - R.umin);
      uint64_t dzf = k ? zigzag64(R.first - pl) : 0;
      uint64_t dmn = R.cnt > 1 ? u64min(R.dzmin, dzf) : dzf, dmx = R.cnt > 1 ? u64max(R.dzmax, dzf) : dzf;
      fsz = 9 + 128ull * wf;
      dsz = 9 + 128ull * bit_width64(dmx - dmn);
      nq = R.neq + ((k && R.first != pl) ? 1u : 0u);
      S.neq_k[k] = nq;
      umn = S.item_min[k] = R.umin;
      umx = S.item_max[k] = R.umax;
      xbytes = R.xb + varint_len(R.first ^ pl);
      sbad = !(R.stride_ok && (R.cnt < 2 || R.d == D) && (k == 0 || R.first - pl == D));
      emn = step == 16 ? R.e16min : R.e64min;
      emx = step == 16 ? R.e16max : R.e64max;
      edz = step == 16 ? R.e16dz : R.e64dz;
      if (k) edz = u64max(edz, dzf);
      pass = R.fm_pass;
      abad = !R.alp_ok;
      asz = 13 + 128ull * R.alp_w + 10ull * R.alp_exc;
    }
    // the sizes fit 32 bits (a sub-block's parts stay below 20 KB)
    const uint32_t sfor = __reduce_add_sync(0xffffffffu, (uint32_t)fsz), sdel = __reduce_add_sync(0xffffffffu, (uint32_t)dsz);
    const uint32_t sxor = __reduce_add_sync(0xffffffffu, (uint32_t)xbytes), sneq = __reduce_add_sync(0xffffffffu, nq);
    umn = warp_min(umn);
    umx = warp_max(umx);
    const bool any_s = __any_sync(0xffffffffu, sbad);
    if (lane_id == 0) {
      atomicAdd((unsigned long long*)&S.sc[1], (unsigned long long)sfor);
      atomicAdd((unsigned long long*)&S.sc[2], (unsigned long long)sdel);
      atomicAdd(&S.xor_bytes, (unsigned long long)sxor);
      atomicAdd(&S.neq, sneq);
      atomic_min_u64(&S.umin, umn);
      atomic_max_u64(&S.umax, umx);
      if (any_s) atomicOr(&S.stride_bad, 1u);
    }
    if (pre_e && !fam_float) {  // only the integer early-out reads them
      emn = warp_min(emn);
      emx = warp_max(emx);
      edz = warp_max(edz);
      if (lane_id == 0) {
        atomic_min_u64(&S.e_vmin, emn);
        atomic_max_u64(&S.e_vmax, emx);
        atomic_max_u64(&S.e_dmax, edz);
      }
    }
    if (fam_float && !reduced) {
      const uint32_t salp = __reduce_add_sync(0xffffffffu, (uint32_t)asz), am = __reduce_and_sync(0xffffffffu, pass);
      const bool any_a = __any_sync(0xffffffffu, abad);
      if (lane_id == 0) {
        atomicAdd((unsigned long long*)&S.sc[4], (unsigned long long)salp);
        atomicAnd(&S.fm_mask, am);
        if (any_a) atomicOr(&S.alp_fail, 1u);
      }
    }
  }
  static_assert(kSubsMax <= kEncThreads, "one sub-block per thread");
  __syncthreads();
  uint64_t vl = varint_len(n);
  uint64_t sz_for = vl + S.sc[1], sz_delta = 8 + vl + S.sc[2], sz_alp = vl + S.sc[4];
  // Selection::Sample: the mode whose estimate on the block's sample is the
  // smallest; it alone is sized in full below (encoder.rs:574-620).
  int win = -1;
  if (SAMPLE) win = sample_winner(S, v, n, dtype, scr);

  // Integer early-out (encoder.rs:295-298, 655-683) with the block's features
  // (the sampled selection has none).
  bool eo = false;
  if (!SAMPLE && !fam_float) {
    uint32_t consec_eq = n - S.neq;
    bool repeats = (uint64_t)consec_eq * 2 > (uint64_t)n;
    uint32_t dstride = max(n / 4096u, 1u);
    uint32_t distinct;
    uint64_t wi = fd.value_off / kBaseQuantum;
    if (!fixed_bs && dstride == 8 && n == (uint32_t)kBaseQuantum) {
      distinct = popc_bits_block(S, winbits + wi * kWinWords);
    } else if (!fixed_bs && dstride == 32 && n == (uint32_t)kMaxBlock) {
      for (int i = t; i < 512; i += blockDim.x)
        S.distinct_bits[i] = winbits[wi * kWinWords + 512 + i] | winbits[(wi + 1) * kWinWords + 512 + i] |
                             winbits[(wi + 2) * kWinWords + 512 + i] | winbits[(wi + 3) * kWinWords + 512 + i];
      __syncthreads();
      distinct = popc_bits_block(S, S.distinct_bits);
    } else {
      for (int i = t; i < 512; i += blockDim.x) S.distinct_bits[i] = 0;
      __syncthreads();
      for (uint32_t i = t; (uint64_t)i * dstride < n; i += blockDim.x) {
        uint64_t h = v[(uint64_t)i * dstride] * 0x9E3779B97F4A7C15ull;
        uint32_t bk = (uint32_t)((h >> 50) & 0x3FFF);
        atomicOr(&S.distinct_bits[bk >> 5], 1u << (bk & 31));
      }
      __syncthreads();
      distinct = popc_bits_block(S, S.distinct_bits);
    }
    bool distinct_low = distinct < 2048;
    if (!(distinct_low || repeats || n < 256)) {
      if (!pre_e) {
        if (t == 0) {
          S.e_vmin = v[0];
          S.e_vmax = v[0];
          S.e_dmax = 0;
        }
        __syncthreads();
        for (uint32_t i = t; (uint64_t)i * step < n; i += blockDim.x) {
          uint32_t idx = i * step;
          uint64_t x = v[idx];
          atomic_min_u64(&S.e_vmin, x);
          atomic_max_u64(&S.e_vmax, x);
          if (idx >= step) atomic_max_u64(&S.e_dmax, zigzag64(x - v[idx - 1]));
        }
        __syncthreads();
      }
      uint32_t thr = (uint32_t)(lb * 8) - 4;
      uint32_t vw = bit_width64(S.e_vmax - S.e_vmin), dw = bit_width64(S.e_dmax);
      eo = vw >= thr && dw >= thr;
    }
  }
  if (eo) {
    if (t == 0) {
      frames[b].mode = M_RAW;
      frames[b].plen = (uint32_t)decoded_bytes;
      frames[b].aux = 0;
      atomicAdd(&g_wins[M_RAW], 1ull);
    }
    return;
  }

  Cand c_fm = {0, false}, c_alp = {0, false}, c_rd = {0, false};
  uint32_t fm_scale = 0, rd_lbw = 0;
  if (fam_float && (SAMPLE ? (win == M_ALP || win == M_ALP_RD) : !reduced)) {
    uint32_t mask = SAMPLE ? 0u : S.fm_mask;  // FLOAT_MULT is an entropy mode for the sampled pool
    if (mask) {  // FLOAT_MULT (float_mult.rs:66-98, bit-packed k)
      fm_scale = __ffs(mask) - 1;
      uint64_t my = 0;
      for (uint32_t k = t; k < nsub; k += blockDim.x) {
        const FmStat& F = fms[g0 + k];
        my += 9 + 128ull * bit_width64((uint64_t)F.kmax[fm_scale] - (uint64_t)F.kmin[fm_scale]);
      }
      my = warp_sum(my);
      if (lane_id == 0) S.red[warp] = my;
      __syncthreads();
      uint64_t tot = 0;
      for (int w = 0; w < kEncWarps; w++) tot += S.red[w];
      __syncthreads();
      c_fm.ok = true;
      c_fm.len = 2 + vl + tot;
      if (ENT) {  // FM_ENTROPY, kept when strictly smaller (float_mult.rs:80-92)
        uint32_t m = fm_delta_bytes(S, v, n, (int)fm_scale, scr);
        uint32_t el = coded_len(S.ra, m, [&](uint32_t i) { return (uint32_t)scr[i]; }, c_fm.len - 2);
        if (el < c_fm.len - 2) {
          c_fm.len = 2 + el;
          er.flags |= kEntFm;
          er.fm = el;
        }
      }
    }
    c_alp.ok = !S.alp_fail;  // ALP (alp.rs:93-166)
    c_alp.len = sz_alp;
    if (SAMPLE && win == M_ALP && reduced) {  // Fastest gathered no ALP statistics: size it here
      if (t == 0) {
        S.acc64 = 0;
        S.alp_fail = 0;
      }
      __syncthreads();
      for (uint32_t k = warp; k < nsub; k += kEncWarps) {
        uint32_t cnt = min((uint32_t)kSub, n - k * kSub);
        AlpSub a;
        bool ok = alp_subblock(v + (uint64_t)k * kSub, cnt, S.alp_smp[warp], kExp10, kFrac10, &a);
        if (lane_id == 0) {
          if (ok) atomicAdd(&S.acc64, (unsigned long long)(13 + 128ull * a.w + 10ull * a.exc));
          else atomicOr(&S.alp_fail, 1u);
        }
      }
      __syncthreads();
      c_alp.ok = !S.alp_fail;
      c_alp.len = vl + S.acc64;
    }
    // ALP-RD (alp_rd.rs:132-206, bit-packed streams)
    bool pre_s = smp16 && !fixed_bs && (step == 16 || step == 64) && (fd.value_off % kBaseQuantum) == 0;
    rd_lbw = (SAMPLE && win != M_ALP_RD) ? 0u
                                         : rd_choose_cut(S, v, n, pre_s ? smp16 + fd.value_off / 16 : nullptr,
                                                         step / 16);
    uint64_t rlen = vl;
    if (rd_lbw) {  // the rights' FoR layout: each sub-block's range of x & rmask
      uint64_t rmask = (1ull << (64 - rd_lbw)) - 1ull;
      if (t == 0) S.acc64 = 0;
      __syncthreads();
      for (uint32_t k = warp; k < nsub; k += kEncWarps) {
        uint32_t base = k * kSub, cnt = min((uint32_t)kSub, n - base);
        uint64_t mn;
        uint32_t w;
        warp_minmax(cnt, false, [&](uint32_t i) { return v[base + i] & rmask; }, &mn, &w);
        if (lane_id == 0) {
          S.w_b[k] = (uint8_t)w;
          S.submin[k] = mn;
          atomicAdd(&S.acc64, (unsigned long long)(9 + 128ull * w));
        }
      }
      __syncthreads();
      rlen += S.acc64;
      __syncthreads();
    }
    if (rd_lbw && !SAMPLE && !ENT) {
      // With the rights' exact size and the smallest possible rest of the
      // payload (a 2-byte header, varint(nexc), the tags and lengths, one
      // 9-byte header per code sub-block) and ALP-RD's decode penalty, it may
      // already reach the best score of the candidates sized so far, and
      // ALP-RD cannot win (strict <): its dictionary and exception pass is
      // skipped.
      uint64_t floor_len = 6 + vl + 9ull * nsub + rlen;
      uint64_t best = decoded_bytes + ((lambda * decode_weight(M_RAW) * decoded_bytes) >> 8);
      auto sc_of = [&](int m, uint64_t len) { return len + ((lambda * decode_weight(m) * decoded_bytes) >> 8); };
      if (S.umin == S.umax) best = u64min(best, sc_of(M_CONST, 8));
      if (n >= 2 && !S.stride_bad) best = u64min(best, sc_of(M_STRIDE, 16));
      if (!reduced) best = u64min(best, sc_of(M_XORZ, S.xor_bytes));
      best = u64min(best, sc_of(M_FOR_BITPACK, sz_for));
      best = u64min(best, sc_of(M_DELTA_BITPACK, sz_delta));
      if (c_fm.ok) best = u64min(best, sc_of(M_FLOAT_MULT, c_fm.len));
      if (c_alp.ok) best = u64min(best, sc_of(M_ALP, c_alp.len));
      if (sc_of(M_ALP_RD, floor_len) >= best) rd_lbw = 0;
      __syncthreads();
    }
    if (rd_lbw) {
      uint32_t rbw = 64 - rd_lbw;
      uint64_t rmask = (1ull << rbw) - 1ull;
      if (!rd_dict_pass(S, v, n, rd_lbw)) {
        __syncthreads();
        rd_top8(S, v, n, rd_lbw, scr);
        for (uint32_t k = warp; k < nsub; k += kEncWarps) {
          uint32_t base = k * kSub, cnt = min((uint32_t)kSub, n - base);
          uint32_t cmx = 0, cmn = 8, eb = 0, ne = 0;
          for (uint32_t i = lane_id; i < cnt; i += 32) {
            int c = rd_code(S, v[base + i] >> rbw);
            uint32_t code = c < 0 ? 0u : (uint32_t)c;
            if (c < 0) {
              ne++;
              eb += varint_len(base + i) + 8;
            }
            cmn = min(cmn, code);
            cmx = max(cmx, code);
          }
          cmn = __reduce_min_sync(0xffffffffu, cmn);
          cmx = __reduce_max_sync(0xffffffffu, cmx);
          ne = __reduce_add_sync(0xffffffffu, ne);
          eb = __reduce_add_sync(0xffffffffu, eb);
          if (lane_id == 0) {
            S.w_a[k] = (uint8_t)bit_width64((uint64_t)(cmx - cmn));
            S.w_c[k] = (uint8_t)cmn;
            S.rd_ne[k] = ne;
            S.rd_eb[k] = eb;
          }
        }
        __syncthreads();
      }
      // sums, and the layout for the emission
      if (t == 0) {
        S.acc64 = 0;
        S.cnt32 = 0;
        S.sc[5] = 0;
      }
      __syncthreads();
      for (uint32_t k = t; k < nsub; k += blockDim.x) {
        atomicAdd(&S.cnt32, S.rd_ne[k]);
        atomicAdd(&S.acc64, (unsigned long long)S.rd_eb[k]);
        atomicAdd((unsigned long long*)&S.sc[5], (unsigned long long)(9 + 128ull * S.w_a[k]));
        RdRec r;
        r.rmin = S.submin[k];
        r.eb = S.rd_eb[k];
        r.ne = (uint16_t)S.rd_ne[k];
        r.cw = S.w_a[k];
        r.rw = S.w_b[k];
        r.cmin = S.w_c[k];
        rdr[g0 + k] = r;
      }
      if (t < 8) blk[b].dict8[t] = S.dict8[t];
      if (t == 8) blk[b].dl = S.dl;
      __syncthreads();
      uint64_t nexc = S.cnt32, excb = S.acc64, clen = vl + S.sc[5];
      c_rd.ok = nexc * 4 <= n;
      auto code_at = [&](uint32_t i) {
        int c = rd_code(S, v[i] >> rbw);
        return (uint32_t)(c < 0 ? 0 : c);
      };
      uint8_t* rdst = nullptr;
      uint32_t rb = 0;
      if (ENT && c_rd.ok) {
        // With the entropy bounds of both parts in place of their coded
        // lengths the payload may already reach the best score of the
        // candidates before it: the serial sizing passes (a quarter of a step
        // per byte of codes and rights) are skipped.
        rdst = stage_dst(S, scr, n, rlen);
        rb = (uint32_t)block_for(S, rdst, n, false, [&](uint32_t i) { return v[i] & rmask; });
        uint64_t cmin = u64min(clen, coded_min(S.ra, n, code_at));
        uint64_t rmin = u64min(rlen, coded_min(S.ra, rb, [&](uint32_t i) { return (uint32_t)rdst[i]; }));
        uint64_t floor_len = 2 + 8ull * S.dl + varint_len(nexc) + excb + 1 + varint_len(cmin) + cmin + 1 + rmin;
        uint64_t best = decoded_bytes + ((lambda * decode_weight(M_RAW) * decoded_bytes) >> 8);
        auto sc_of = [&](int m, uint64_t len) { return len + ((lambda * decode_weight(m) * decoded_bytes) >> 8); };
        if (S.umin == S.umax) best = u64min(best, sc_of(M_CONST, 8));
        if (n >= 2 && !S.stride_bad) best = u64min(best, sc_of(M_STRIDE, 16));
        if (!reduced) best = u64min(best, sc_of(M_XORZ, S.xor_bytes));
        best = u64min(best, sc_of(M_FOR_BITPACK, sz_for));
        best = u64min(best, sc_of(M_DELTA_BITPACK, sz_delta));
        if (c_fm.ok) best = u64min(best, sc_of(M_FLOAT_MULT, c_fm.len));
        if (c_alp.ok) best = u64min(best, sc_of(M_ALP, c_alp.len));
        if (sc_of(M_ALP_RD, floor_len) >= best) c_rd.ok = false;
      }
      if (ENT && c_rd.ok) {  // T_ENT codes / rights, kept when strictly smaller (alp_rd.rs:176-200)
        uint32_t cl = coded_len(S.ra, n, code_at, clen);
        if (cl < clen) {
          clen = cl;
          er.flags |= kEntRdCodes;
          er.rdc = cl;
        }
        uint32_t rl = coded_len(S.ra, rb, [&](uint32_t i) { return (uint32_t)rdst[i]; }, rlen);
        if (rl < rlen) {
          rlen = rl;
          er.flags |= kEntRdRights;
          er.rdr = rl;
        }
      }
      c_rd.len = 2 + 8ull * S.dl + varint_len(nexc) + excb + 1 + varint_len(clen) + clen + 1 + rlen;
      __syncthreads();
    }
  }

  // Selection up to ALP-RD (encoder.rs:301-344), then the compressibility gate.
  int best_mode = M_RAW;
  uint64_t best_len = decoded_bytes;
  uint64_t best_score = best_len + ((lambda * decode_weight(M_RAW) * decoded_bytes) >> 8);
  auto consider = [&](int m, uint64_t len) {
    uint64_t sc = len + ((lambda * decode_weight(m) * decoded_bytes) >> 8);
    if (sc < best_score) {
      best_score = sc;
      best_mode = m;
      best_len = len;
    }
  };
  if (S.umin == S.umax) consider(M_CONST, 8);
  if (n >= 2 && !S.stride_bad) consider(M_STRIDE, 16);
  if (SAMPLE) {  // the sample's winner, sized in full (DICT / RLE below)
    if (win == M_XORZ) consider(M_XORZ, S.xor_bytes);
    if (win == M_FOR_BITPACK) consider(M_FOR_BITPACK, sz_for);
    if (win == M_DELTA_BITPACK) consider(M_DELTA_BITPACK, sz_delta);
    if (win == M_ALP && c_alp.ok) consider(M_ALP, c_alp.len);
    if (win == M_ALP_RD && c_rd.ok) consider(M_ALP_RD, c_rd.len);
  } else {
    if (!reduced) consider(M_XORZ, S.xor_bytes);
    consider(M_FOR_BITPACK, sz_for);
    consider(M_DELTA_BITPACK, sz_delta);
    if (c_fm.ok) consider(M_FLOAT_MULT, c_fm.len);
    if (c_alp.ok) consider(M_ALP, c_alp.len);
    if (c_rd.ok) consider(M_ALP_RD, c_rd.len);
  }
  bool block_compressible = best_len * 20 < raw_bytes * 19;  // encoder.rs:394,644-646

  if (ENT && block_compressible) {
    // BYTE_TRANSPOSE (encoder.rs:414-420) when the exponent-field range is at
    // most 64 or most consecutive values repeat (encoder.rs:705-750)
    if (t == 0) {
      S.exp_lo = 0x7FF;
      S.exp_hi = 0;
    }
    __syncthreads();
    uint32_t elo = 0x7FF, ehi = 0;
    for (uint32_t i = t; i < n; i += blockDim.x) {
      uint32_t ex = (uint32_t)(v[i] >> 52) & 0x7FFu;
      elo = min(elo, ex);
      ehi = max(ehi, ex);
    }
    elo = warp_min(elo);
    ehi = warp_max(ehi);
    if (lane_id == 0) {
      atomicMin(&S.exp_lo, elo);
      atomicMax(&S.exp_hi, ehi);
    }
    __syncthreads();
    bool repeats = (uint64_t)(n - S.neq) * 2 > (uint64_t)n;
    if (S.exp_hi - S.exp_lo <= 64 || repeats) {
      // BYTE_TRANSPOSE wins only below best_score less its decode penalty
      uint64_t pen = (lambda * decode_weight(M_BYTE_TRANSPOSE) * decoded_bytes) >> 8;
      uint32_t bl = coded_len(S.ra, 8 * n, [&](uint32_t i) {
        uint32_t pl = i / n;
        return (uint32_t)(v[i - pl * n] >> (8 * pl)) & 255u;
      }, best_score > pen ? best_score - pen : 0ull);
      er.bt = bl;
      consider(M_BYTE_TRANSPOSE, bl);
    }
  }

  if (SAMPLE ? (win == M_DICT || win == M_RLE) : (block_compressible && !reduced)) {
    // DICT (dict.rs:87-152, bit-packed codes).  The dictionary is sorted, so
    // a sub-block's code range is [rank(min), rank(max)].
    bool one_win = !fixed_bs && (fd.value_off % kBaseQuantum) == 0 && n <= (uint32_t)kBaseQuantum;
    uint32_t lb_pre = one_win ? winbits[(fd.value_off / kBaseQuantum) * kWinWords + 1024] : kNoLb;
    bool want_dict = !SAMPLE || win == M_DICT;
    // A DICT payload holds at least 22 bytes (card, value tag and length, 8
    // value bytes, code tag, varint(n) and one 9-byte sub-block header): when
    // that and DICT's decode penalty already reach the best score, it cannot
    // win (strict <) and its passes are skipped.
    if (!SAMPLE && best_score <= 22 + ((lambda * decode_weight(M_DICT) * decoded_bytes) >> 8)) want_dict = false;
    // RLE's floor: the run values, two varint(runs) and a 9-byte header per
    // 1,024 run lengths
    const uint32_t neq = S.neq, runs = neq + 1;
    const uint64_t rle_floor = 2 * varint_len(runs) + 8ull * runs + 9ull * ((runs + kSub - 1) / kSub) +
                               ((lambda * decode_weight(M_RLE) * decoded_bytes) >> 8);
    const bool want_rle = (!SAMPLE || win == M_RLE) && neq <= n / 2 + 1 && (SAMPLE || best_score > rle_floor);
    uint32_t* st = want_rle ? rle_starts(S, v, n, scr) : nullptr;
    DictView dv;
    if (want_dict) {
      dv = dict_prepare(S, v, n, scr, lb_pre, st, runs);
      if (!dv.smem) st = nullptr;  // a large dictionary is built over the run starts
    }
    if (want_dict && !S.flag) {
      uint32_t vtag;
      uint64_t vlen = dict_values_len(S, dv, &vtag);
      if (ENT) {  // TRANSPOSE values, kept when strictly smaller (dict.rs:52-59)
        const uint64_t* sv = dv.sorted;
        uint32_t card = dv.card;
        uint32_t tl = coded_len(S.ra, 8 * card, [&](uint32_t i) {
          uint32_t pl = i / card;
          return (uint32_t)(sv[i - pl * card] >> (8 * pl)) & 255u;
        }, vlen);
        if (tl < vlen) {
          vlen = tl;
          vtag = 2;
          er.flags |= kEntDictVals;
          er.dv = tl;
        }
      }
      uint64_t my = 0;
      for (uint32_t k = t; k < nsub; k += blockDim.x) {
        uint32_t r0 = dict_rank(S, dv, S.item_min[k]), r1 = dict_rank(S, dv, S.item_max[k]);
        my += 9 + 128ull * bit_width64((uint64_t)(r1 - r0));
      }
      my = warp_sum(my);
      if (lane_id == 0) S.red[warp] = my;
      __syncthreads();
      uint64_t clen = vl;
      for (int w = 0; w < kEncWarps; w++) clen += S.red[w];
      __syncthreads();
      if (ENT && dv.card <= 65536u) {  // CODES_ENTROPY byte planes, kept when strictly smaller (dict.rs:128-145)
        uint32_t nb = dv.card <= 256u ? 1u : 2u;
        uint64_t el = 1;
        uint32_t pls[2] = {0, 0};
        for (uint32_t pl = 0; pl < nb; pl++) {
          pls[pl] = coded_len(S.ra, n, [&](uint32_t i) { return (dict_rank(S, dv, v[i]) >> (8 * pl)) & 255u; },
                              clen);
          el += varint_len(pls[pl]) + pls[pl];
        }
        if (el < clen) {
          clen = el;
          er.flags |= kEntDictCodes;
          er.dc[0] = pls[0];
          er.dc[1] = pls[1];
        }
      }
      consider(M_DICT, varint_len(dv.card) + 1 + varint_len(vlen) + vlen + 1 + clen);
      // a small dictionary is kept for the emission, in the half of the block's
      // scratch that the run starts below do not use
      if (dv.smem && best_mode == M_DICT) {
        uint64_t* keep = reinterpret_cast<uint64_t*>(scr + 16ull * n);
        for (uint32_t i = t; i < dv.card; i += blockDim.x) keep[i] = dv.sorted[i];
        if (t == 0) {
          blk[b].card = dv.card;
          blk[b].vtag = vtag;
          blk[b].vlen = vlen;
        }
      } else if (t == 0) {
        blk[b].card = 0;
      }
    }
    __syncthreads();
    // RLE (rle.rs:10-42)
    if (want_rle && (SAMPLE || best_score > rle_floor)) {
      if (!st) st = rle_starts(S, v, n, scr);
      uint64_t lens = block_for(S, nullptr, runs, false, [&](uint32_t r) {
        return (uint64_t)((r + 1 < runs ? st[r + 1] : n) - st[r]);
      });
      consider(M_RLE, varint_len(runs) + 8ull * runs + lens);
      if (best_mode == M_RLE) {  // for the emission: the starts stay in the block's scratch
        if (t == 0) blk[b].card = runs;
        for (uint32_t k = t; k < (runs + kSub - 1) / kSub; k += blockDim.x) {
          rdr[g0 + k].rmin = S.submin[k];
          rdr[g0 + k].rw = S.w_a[k];
        }
      }
    }
  }
  if (t == 0) {
    frames[b].mode = (uint32_t)best_mode;
    frames[b].plen = (uint32_t)best_len;
    frames[b].aux = best_mode == M_FLOAT_MULT ? fm_scale : best_mode == M_ALP_RD ? rd_lbw : 0;
    atomicAdd(&g_wins[best_mode], 1ull);
    if (ENT) ent[b] = er;
  }
}

// ---------------------------------------------------------------------------
// Emission kernel: writes the frame header and the winner's payload.  A CTA
// takes sub-blocks [k0, k1) of a block: a window's (32), or half of them when
// a column has fewer windows than the GPU has places for CTAs, so a column of
// a few blocks is spread over more SMs and a grown block over four CTAs.  Where
// every sub-block goes follows from the statistics' and the competition's
// records.  The CTA with the block's first sub-block (`lead`) writes what is
// not a sub-block's; it alone emits the modes whose parts depend on a pass
// over the block (a large dictionary, entropy-coded parts).
// ---------------------------------------------------------------------------
__device__ void emit_raw(const uint64_t* v, uint32_t n, int dtype, uint8_t* out, uint32_t k0, uint32_t k1) {
  const uint32_t i1 = min(n, k1 * kSub);
  uint32_t lb = lane_bytes(dtype);
#pragma unroll 8
  for (uint32_t i = k0 * kSub + threadIdx.x; i < i1; i += blockDim.x) {
    uint64_t x = v[i];
    if (dtype == DT_F32) put_u32(out + 4ull * i, f64bits_to_f32bits(x));
    else if (lb == 4) put_u32(out + 4ull * i, (uint32_t)x);
    else put_u64(out + 8ull * i, x);
  }
}

// S.subsz[k] holds each sub-block's LEB128 byte offset on entry.
__device__ void emit_xorz(EncSmem& S, const uint64_t* v, uint32_t n, uint8_t* out, uint32_t k0, uint32_t k1) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t k = k0 + warp; k < k1; k += kEncWarps) {
    uint32_t base = k * kSub, cnt = min((uint32_t)kSub, n - base);
    uint8_t* dst = out + S.subsz[k];
    uint64_t carry = base ? v[base - 1] : 0ull;
    for (uint32_t j0 = 0; j0 < 32; j0 += 8) {
      uint64_t xs[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t li = (j0 + q) * 32 + lane;
        xs[q] = li < cnt ? v[base + li] : 0ull;
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t li = (j0 + q) * 32 + lane;
        bool ok = li < cnt;
        uint64_t rot = __shfl_sync(0xffffffffu, xs[q], (lane + 31) & 31);
        uint64_t x = ok ? xs[q] ^ (lane ? rot : carry) : 0ull;
        carry = rot;
        uint32_t sz = ok ? varint_len(x) : 0u;
        uint32_t inc = warp_incl_scan(sz);
        if (ok) put_varint(dst + inc - sz, x);
        dst += __shfl_sync(0xffffffffu, inc, 31);
      }
    }
  }
}

__device__ __noinline__ void emit_alp(EncSmem& S, const uint64_t* v, uint32_t n, const SubStats* ss, uint8_t* out, uint32_t k0,
                         uint32_t k1) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t nsub = (n + kSub - 1) / kSub;
  __shared__ int64_t s_fill[kSubsMax];
  __shared__ double s_pexp[19], s_pfrac[19];  // the (e, f) search reads them at per-lane indices
  if (threadIdx.x < 19) {
    s_pexp[threadIdx.x] = kExp10[threadIdx.x];
    s_pfrac[threadIdx.x] = kFrac10[threadIdx.x];
  }
  __syncthreads();
  // the statistics' (e, f), width and exception count of every sub-block, or
  // (Sample at Fastest) all of them searched again by the lead CTA
  const bool known = ss && (ss[0].pad16 & kAlpEfKnown);
  if (!known) {
    if (k0) return;
    k1 = nsub;
  }
  for (uint32_t k = k0 + warp; k < k1; k += kEncWarps) {
    uint32_t cnt = min((uint32_t)kSub, n - k * kSub);
    AlpSub a;
    if (known) {
      const uint16_t ef = ss[k].pad16;
      a.e = ef & 0xFF;
      a.f = (ef >> 8) & 0x7F;
      alp_subblock_ef(v + (uint64_t)k * kSub, cnt, a.e, a.f, s_pexp, s_pfrac, &a);
    } else {
      alp_subblock(v + (uint64_t)k * kSub, cnt, S.alp_smp[warp], s_pexp, s_pfrac, &a);  // succeeded in the competition
    }
    if (lane == 0) {
      S.alp_ef[k][0] = (uint8_t)a.e;
      S.alp_ef[k][1] = (uint8_t)a.f;
      S.w_c[k] = (uint8_t)a.w;
      S.alp_exc[k] = (uint16_t)a.exc;
      S.submin[k] = (uint64_t)a.mn;
      s_fill[k] = a.filler;
      if (!known) S.subsz[k] = 13 + 128u * a.w + 10u * a.exc;
    }
  }
  if (known)
    for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.subsz[k] = 13 + 128u * ss[k].alp_w + 10u * ss[k].alp_exc;
  block_offsets(S, nsub, varint_len(n));
  if (threadIdx.x == 0 && k0 == 0) put_varint(out, n);
  for (uint32_t k = k0 + warp; k < k1; k += kEncWarps) {
    uint32_t base = k * kSub, cnt = min((uint32_t)kSub, n - base);
    uint8_t* d = out + S.subsz[k];
    int e = S.alp_ef[k][0], f = S.alp_ef[k][1];
    uint32_t w = S.w_c[k];
    int64_t mn = (int64_t)S.submin[k], fill = s_fill[k];
    const uint64_t* sv = v + base;
    // Digits (exceptions and padding take the filler digit), FastLanes packed:
    // a FoR sub-block at d + 4 whose width byte and minimum the ALP header
    // holds the other way round.
    warp_for_pack(d + 4, (uint32_t)kSub, (uint64_t)mn, w, [&](uint32_t i) {
      int64_t dd;
      return (uint64_t)(i < cnt && alp_roundtrips(sv[i], e, f, &dd) ? dd : fill);
    });
    __syncwarp();
    if (lane == 0) {
      put_u8(d, e);
      put_u8(d + 1, f);
      put_u16(d + 2, S.alp_exc[k]);
      put_u64(d + 4, (uint64_t)mn);
      put_u8(d + 12, w);
    }
    // Exceptions in position order.
    uint8_t* xp = d + 13 + 128u * w;
    uint32_t before = 0;
    for (uint32_t j = 0; S.alp_exc[k] && j < 32; j++) {
      uint32_t li = j * 32 + lane;
      bool ok = li < cnt;
      int64_t dd;
      bool ex = ok && !alp_roundtrips(sv[li], e, f, &dd);
      uint32_t m = __ballot_sync(0xffffffffu, ex);
      if (ex) {
        uint8_t* q = xp + 10u * (before + __popc(m & ((1u << lane) - 1u)));
        put_u16(q, li);
        put_u64(q + 2, sv[li]);
      }
      before += __popc(m);
    }
  }
}

// ALP-RD from the competition's records: every part's place is known, so a
// warp writes its sub-block's exceptions, codes and rights one after another
// while the values are in L1.  (Counting the left parts again, then a pass for
// each part's sizes and each part's bytes, took 238 us for 1,048,576 prices.)
__device__ __noinline__ void emit_alprd(EncSmem& S, const uint64_t* v, uint32_t n, uint32_t lbw, const RdRec* rec,
                           const BlkRec& B, uint8_t* scr, uint8_t* out, const EntRec* er, uint32_t k0, uint32_t k1) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t nsub = (n + kSub - 1) / kSub;
  const uint32_t rbw = 64 - lbw;
  const uint64_t rmask = (1ull << rbw) - 1ull;
  if (threadIdx.x < 8) S.dict8[threadIdx.x] = B.dict8[threadIdx.x];
  if (threadIdx.x == 0) {
    S.dl = B.dl;
    S.cnt32 = 0;
  }
  __syncthreads();
  // offsets of the exceptions (relative), the codes' and the rights' sub-blocks
  uint32_t ne = 0;
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) {
    S.subsz[k] = rec[k].eb;
    ne += rec[k].ne;
  }
  ne = __reduce_add_sync(0xffffffffu, ne);
  if (lane == 0 && ne) atomicAdd(&S.cnt32, ne);
  __syncthreads();
  const uint32_t nexc = S.cnt32, vl = varint_len(n);
  const uint32_t head = 2 + 8 * S.dl + varint_len(nexc);
  block_offsets(S, nsub, head);
  const uint32_t cpos = S.subsz[nsub];  // the codes' tag
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.rd_eb[k] = S.subsz[k];
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.subsz[k] = 9 + 128u * rec[k].cw;
  block_offsets(S, nsub, vl);
  uint32_t clen = S.subsz[nsub];
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.rd_ne[k] = S.subsz[k];  // within the codes
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) S.subsz[k] = 9 + 128u * rec[k].rw;
  block_offsets(S, nsub, vl);
  const bool ccoded = er && (er->flags & kEntRdCodes), rcoded = er && (er->flags & kEntRdRights);
  if (ccoded) clen = er->rdc;
  const uint32_t c0 = cpos + 1 + varint_len(clen), rpos = c0 + clen;  // the codes; the rights' tag
  if (threadIdx.x == 0 && k0 == 0) {
    uint32_t pos = 0;
    put_u8(out + pos++, lbw);
    put_u8(out + pos++, S.dl);
    for (uint32_t j = 0; j < S.dl; j++, pos += 8) put_u64(out + pos, S.dict8[j]);
    put_varint(out + pos, nexc);
    put_u8(out + cpos, ccoded ? 1 : 0);
    put_varint(out + cpos + 1, clen);
    if (!ccoded) put_varint(out + c0, n);
    put_u8(out + rpos, rcoded ? 1 : 0);
    if (!rcoded) put_varint(out + rpos + 1, n);
  }
  auto code_at = [&](uint32_t i) -> uint64_t {
    int c = rd_code(S, v[i] >> rbw);
    return c < 0 ? 0ull : (uint64_t)c;
  };
  for (uint32_t k = k0 + warp; k < k1; k += kEncWarps) {
    const uint32_t base = k * kSub, cnt = min((uint32_t)kSub, n - base);
    const RdRec r = rec[k];
    if (!ccoded) warp_for_pack(out + c0 + S.rd_ne[k], cnt, r.cmin, r.cw, [&](uint32_t i) { return code_at(base + i); });
    if (!rcoded)
      warp_for_pack(out + rpos + 1 + S.subsz[k], cnt, r.rmin, r.rw, [&](uint32_t i) { return v[base + i] & rmask; });
    uint32_t off = S.rd_eb[k];
    for (uint32_t j0 = 0; r.ne && j0 < 32; j0 += 8) {
      uint64_t xs[8];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t li = (j0 + q) * 32 + lane;
        xs[q] = li < cnt ? v[base + li] : 0ull;
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        uint32_t li = (j0 + q) * 32 + lane;
        bool ex = li < cnt && rd_code(S, xs[q] >> rbw) < 0;
        if (!__any_sync(0xffffffffu, ex)) continue;
        uint32_t sz = ex ? varint_len(base + li) + 8 : 0u;
        uint32_t inc = warp_incl_scan(sz);
        if (ex) {
          uint8_t* d = out + off + inc - sz;
          uint32_t vlb = put_varint(d, base + li);
          put_u64(d + vlb, xs[q] >> rbw);
        }
        off += __shfl_sync(0xffffffffu, inc, 31);
      }
    }
  }
  if (ccoded) coded_write(S.ra, n, [&](uint32_t i) { return (uint32_t)code_at(i); }, out + c0, clen);
  if (rcoded) {  // the bit-packed rights, coded
    auto right_of = [&](uint32_t i) { return v[i] & rmask; };
    uint8_t* rdst = stage_dst(S, scr, n, block_for(S, nullptr, n, false, right_of));
    uint32_t rb = (uint32_t)block_for(S, rdst, n, false, right_of);
    coded_write(S.ra, rb, [&](uint32_t i) { return (uint32_t)rdst[i]; }, out + rpos + 1, er->rdr);
  }
}

// The small dictionary that the competition kept (ascending), as the shared
// hash table of dict_prepare.
__device__ DictView dict_restore(EncSmem& S, const uint64_t* keep, uint32_t card) {
  DictArea& D = S.big.dict;
  for (uint32_t i = threadIdx.x; i < kHashCap; i += blockDim.x) D.hkey[i] = kEmpty64;
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < card; r += blockDim.x) {
    const uint64_t x = keep[r];
    D.sorted[r] = x;
    if (x == kEmpty64) {
      S.max_rank = r;
      continue;
    }
    uint32_t h = (uint32_t)((x * 0x9E3779B97F4A7C15ull) >> 53);
    while (atomicCAS((unsigned long long*)&D.hkey[h], kEmpty64, x) != kEmpty64) h = (h + 1) & (kHashCap - 1);
    D.hval[h] = r;
  }
  __syncthreads();
  DictView dv;
  dv.smem = true;
  dv.sorted = D.sorted;
  dv.card = card;
  return dv;
}

__device__ __noinline__ void emit_dict(EncSmem& S, const uint64_t* v, uint32_t n, const SubStats* ss, const BlkRec& B, uint8_t* scr,
                          uint8_t* out, const EntRec* er, uint32_t k0, uint32_t k1) {
  const bool kept = B.card != 0;
  if (!kept && k0) return;
  DictView dv;
  uint32_t vtag;
  uint64_t vlen;
  if (kept) {
    dv = dict_restore(S, reinterpret_cast<const uint64_t*>(scr + 16ull * n), B.card);
    vtag = B.vtag;
    vlen = B.vlen;
  } else {
    dv = dict_prepare(S, v, n, scr, kNoLb);
    vlen = dict_values_len(S, dv, &vtag);
    k1 = (n + kSub - 1) / kSub;
  }
  if (er && (er->flags & kEntDictVals)) {
    vtag = 2;
    vlen = er->dv;
  }
  const uint32_t card = dv.card;
  uint64_t pos = varint_len(card) + 1 + varint_len(vlen);
  const uint64_t* s = dv.sorted;
  if (k0 == 0) {
    if (threadIdx.x == 0) {
      uint32_t q = put_varint(out, card);
      put_u8(out + q, vtag);
      put_varint(out + q + 1, vlen);
    }
    if (vtag == 0) {
      for (uint32_t i = threadIdx.x; i < card; i += blockDim.x) put_u64(out + pos + 8ull * i, s[i]);
    } else if (vtag == 1) {
      if (threadIdx.x == 0) put_u64(out + pos, s[0]);
      block_for(S, out + pos + 8, card, false, [&](uint32_t i) { return zigzag64(s[i] - (i ? s[i - 1] : s[0])); });
    } else {
      coded_write(S.ra, 8 * card, [&](uint32_t i) {
        uint32_t pl = i / card;
        return (uint32_t)(s[i - pl * card] >> (8 * pl)) & 255u;
      }, out + pos, (uint32_t)vlen);
    }
  }
  __syncthreads();
  pos += vlen;
  if (er && (er->flags & kEntDictCodes)) {  // nplanes, then varint(len) + coded plane each
    uint32_t nb = card <= 256u ? 1u : 2u;
    if (threadIdx.x == 0) {
      put_u8(out + pos, 1);
      put_u8(out + pos + 1, nb);
    }
    pos += 2;
    for (uint32_t pl = 0; pl < nb; pl++) {
      uint32_t len = er->dc[pl];
      if (threadIdx.x == 0) put_varint(out + pos, len);
      pos += varint_len(len);
      coded_write(S.ra, n, [&](uint32_t i) { return (dict_rank(S, dv, v[i]) >> (8 * pl)) & 255u; }, out + pos, len);
      pos += len;
    }
    return;
  }
  if (threadIdx.x == 0 && k0 == 0) put_u8(out + pos, 0);
  // The dictionary is sorted, so a sub-block's codes run from the rank of its
  // smallest value to the rank of its largest (the statistics' unsigned
  // min / max): the FoR widths and bases without a pass over the codes.
  uint32_t nsub = (n + kSub - 1) / kSub;
  for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) {
    uint32_t r0 = dict_rank(S, dv, ss[k].umin), r1 = dict_rank(S, dv, ss[k].umax);
    S.w_a[k] = (uint8_t)bit_width64((uint64_t)(r1 - r0));
    S.submin[k] = r0;
  }
  __syncthreads();
  block_for_write(S, out + pos + 1, n, [&](uint32_t i) { return (uint64_t)dict_rank(S, dv, v[i]); }, k0, k1);
}

// RLE from the competition's run starts: the CTA's share of the run values and
// of the 1,024-run chunks of the lengths, whose layout is in the block's
// records.
__device__ __noinline__ void emit_rle(EncSmem& S, const uint64_t* v, uint32_t n, const RdRec* rec, const BlkRec& B,
                                      const uint8_t* scr, uint8_t* out, uint32_t part, uint32_t parts) {
  const uint32_t* st = reinterpret_cast<const uint32_t*>(scr);
  const uint32_t runs = B.card, vl = varint_len(runs), nch = (runs + kSub - 1) / kSub;
  auto len_at = [&](uint32_t r) { return (uint64_t)((r + 1 < runs ? st[r + 1] : n) - st[r]); };
  if (threadIdx.x == 0 && part == 0) put_varint(out, runs);
  const uint32_t per = (runs + parts - 1) / parts, r0 = min(part * per, runs), r1 = min(r0 + per, runs);
  for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) put_u64(out + vl + 8ull * r, v[st[r]]);
  for (uint32_t k = threadIdx.x; k < nch; k += blockDim.x) {
    S.w_a[k] = rec[k].rw;
    S.submin[k] = rec[k].rmin;
  }
  __syncthreads();
  const uint32_t cper = (nch + parts - 1) / parts, c0 = min(part * cper, nch);
  block_for_write(S, out + vl + 8ull * runs, runs, len_at, c0, min(c0 + cper, nch));
}

// w2b: the block of each window (adaptive plan); split: CTAs per window.
constexpr uint32_t kWinSubs = kBaseQuantum / kSub;
template <bool ENT>
__device__ __forceinline__ void emit_unit(const uint32_t cta, const uint64_t* __restrict__ lane,
                                          const FrameDesc* __restrict__ frames, const uint32_t* __restrict__ nbp,
                                          const uint32_t* __restrict__ w2b, uint32_t split, uint64_t fixed_bs,
                                          int dtype, const SubStats* __restrict__ ss, const FmStat* __restrict__ fms,
                                          const RdRec* __restrict__ rdr, const BlkRec* __restrict__ blk,
                                          uint8_t* __restrict__ scratch, uint8_t* __restrict__ outbuf,
                                          uint64_t out_cap, const EntRec* __restrict__ ent) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  EncSmem& S = *reinterpret_cast<EncSmem*>(smem_raw);
  const uint32_t unit = cta / split, part = cta % split;
  uint32_t b, win;  // the block, and the unit's window within it
  if (fixed_bs) {
    const uint32_t per = (uint32_t)((fixed_bs + kBaseQuantum - 1) / kBaseQuantum);
    b = unit / per;
    win = unit % per;
  } else {
    b = w2b[unit];
    win = 0;
  }
  if (b >= *nbp) return;
  FrameDesc fd = frames[b];
  if (!fixed_bs) win = unit - (uint32_t)(fd.value_off / kBaseQuantum);
  if (fd.payload_off + fd.plen > out_cap) return;  // the caller sees the total and reports the shortfall
  const uint64_t* v = lane + fd.value_off;
  uint32_t n = fd.n;
  const uint32_t nsub = (n + kSub - 1) / kSub, cut = kWinSubs / split;
  uint32_t k0 = win * kWinSubs + part * cut, k1 = min(k0 + cut, nsub);
  const int m = (int)fd.mode;
  const uint32_t parts = (nsub + cut - 1) / cut;
  if (ENT || m == M_CONST || m == M_STRIDE) {  // whole blocks
    if (k0) return;
    k1 = nsub;
  }
  if (k0 >= k1) return;
  const bool lead = k0 == 0;
  uint8_t* scr = scratch + fd.value_off * kEncScratchPerValue;
  uint8_t* hdr = outbuf + fd.payload_off - 9;
  uint8_t* out = outbuf + fd.payload_off;
  if (threadIdx.x == 0 && lead) {
    put_u8(hdr, fd.mode);
    put_u32(hdr + 1, n);
    put_u32(hdr + 5, fd.plen);
  }
  bool sgn = dtype_signed(dtype);
  // FoR / DELTA / FLOAT_MULT / XORZ sub-block layouts come from the statistics
  // pass (the same numbers the competition sized the frame with).
  uint64_t g0 = fixed_bs ? (uint64_t)b * ((fixed_bs + kSub - 1) / kSub) : fd.value_off / kSub;
  EntRec er = {0, 0, 0, 0, 0, 0, {0, 0}};
  if (ENT) er = ent[b];
  const EntRec* erp = ENT ? &er : nullptr;
  if (m == M_FOR_BITPACK || m == M_DELTA_BITPACK || m == M_FLOAT_MULT || m == M_XORZ) {
    for (uint32_t k = threadIdx.x; k < nsub; k += blockDim.x) {
      const SubStats& R = ss[g0 + k];
      uint64_t pl = k ? ss[g0 + k - 1].last : 0;
      uint32_t w = 0;
      uint64_t mn = 0;
      if (m == M_FOR_BITPACK) {
        w = sgn ? bit_width64((uint64_t)R.smax - (uint64_t)R.smin) : bit_width64(R.umax - R.umin);
        mn = sgn ? (uint64_t)R.smin : R.umin;
      } else if (m == M_DELTA_BITPACK) {
        uint64_t dzf = k ? zigzag64(R.first - pl) : 0;
        uint64_t dmn = R.cnt > 1 ? u64min(R.dzmin, dzf) : dzf, dmx = R.cnt > 1 ? u64max(R.dzmax, dzf) : dzf;
        w = bit_width64(dmx - dmn);
        mn = dmn;
      } else if (m == M_FLOAT_MULT) {
        const FmStat& F = fms[g0 + k];
        w = bit_width64((uint64_t)F.kmax[fd.aux] - (uint64_t)F.kmin[fd.aux]);
        mn = (uint64_t)F.kmin[fd.aux];
      } else {
        S.subsz[k] = R.xb + varint_len(R.first ^ pl);
      }
      S.w_a[k] = (uint8_t)w;
      S.submin[k] = mn;
    }
    if (m == M_XORZ) block_offsets(S, nsub, 0);
    __syncthreads();
  }
  switch (fd.mode) {
    case M_RAW: emit_raw(v, n, dtype, out, k0, k1); break;
    case M_CONST:
      if (threadIdx.x == 0) put_u64(out, v[0]);
      break;
    case M_STRIDE:
      if (threadIdx.x == 0) {
        put_u64(out, v[0]);
        put_u64(out + 8, v[1] - v[0]);
      }
      break;
    case M_XORZ: emit_xorz(S, v, n, out, k0, k1); break;
    case M_FOR_BITPACK: block_for_write(S, out, n, [&](uint32_t i) { return v[i]; }, k0, k1); break;
    case M_DELTA_BITPACK:
      if (threadIdx.x == 0 && lead) put_u64(out, v[0]);
      block_for_write(S, out + 8, n, [&](uint32_t i) { return zigzag64(v[i] - (i ? v[i - 1] : v[0])); }, k0, k1);
      break;
    case M_FLOAT_MULT: {
      int s = (int)fd.aux;
      bool coded = ENT && (er.flags & kEntFm);
      if (threadIdx.x == 0 && lead) {
        put_u8(out, coded ? 1 : 0);
        put_u8(out + 1, s);
      }
      if (coded) {
        uint32_t mb = fm_delta_bytes(S, v, n, s, scr);
        coded_write(S.ra, mb, [&](uint32_t i) { return (uint32_t)scr[i]; }, out + 2, er.fm);
      } else {
        block_for_write(S, out + 2, n, [&](uint32_t i) { return (uint64_t)fm_k(v[i], s); }, k0, k1);
      }
      break;
    }
    case M_BYTE_TRANSPOSE:  // transpose.rs:10-32 (Balanced in-pool only)
      if (ENT)
        coded_write(S.ra, 8 * n, [&](uint32_t i) {
          uint32_t pl = i / n;
          return (uint32_t)(v[i - pl * n] >> (8 * pl)) & 255u;
        }, out, fd.plen);
      break;
    case M_ALP: emit_alp(S, v, n, ss ? ss + g0 : nullptr, out, k0, k1); break;
    case M_ALP_RD: emit_alprd(S, v, n, fd.aux, rdr + g0, blk[b], scr, out, erp, k0, k1); break;
    case M_DICT: emit_dict(S, v, n, ss + g0, blk[b], scr, out, erp, k0, k1); break;
    case M_RLE: emit_rle(S, v, n, rdr + g0, blk[b], scr, out, ENT ? 0 : k0 / cut, ENT ? 1 : parts); break;
    default: break;
  }
}

// ---------------------------------------------------------------------------
// Window probe, block planning and frame offsets.
// ---------------------------------------------------------------------------

// Block plan (reference encoder.rs:154-178): fills frames[].value_off / .n and
// (adaptive) each window's block.
constexpr int kPlanThreads = 1024;
__device__ __forceinline__ void plan_blocks(const uint32_t cta, const uint32_t ctas, const uint8_t* __restrict__ grow,
                                            uint64_t n, const uint64_t* d_n, uint64_t fixed_bs, FrameDesc* frames,
                                            uint32_t* nb, uint32_t* __restrict__ w2b) {
  const uint64_t bound = n;
  if (d_n) n = *d_n;
  if (fixed_bs) {
    uint64_t nblk = (n + fixed_bs - 1) / fixed_bs;
    for (uint64_t i = (uint64_t)cta * blockDim.x + threadIdx.x; i < nblk; i += (uint64_t)ctas * blockDim.x) {
      FrameDesc f;
      f.value_off = i * fixed_bs;
      f.n = (uint32_t)qmin(fixed_bs, n - f.value_off);
      f.payload_off = 0;
      f.plen = 0;
      f.mode = 0;
      f.aux = 0;
      frames[i] = f;
    }
    if (cta == 0 && threadIdx.x == 0) *nb = (uint32_t)nblk;
    return;
  }
  // Adaptive: the block starts form a chain over the 32768-value windows
  // (grow -> +4 windows, else +1).  As a scan: the state before window w is
  // the number of windows still covered by the current block (0 = w starts a
  // block), and window w maps it by f_w(s) = s ? s - 1 : (grow[w] ? 3 : 0).
  // The maps compose (4 entries of 2 bits), so one CTA scans them in chunks
  // of 4096 windows, then compacts the starts into the frame table.
  if (cta) return;
  constexpr int kPer = 4, kWarps = kPlanThreads / 32;
  __shared__ uint32_t s_wmap[kWarps], s_wcnt[kWarps];
  __shared__ uint32_t s_state, s_count;
  int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint64_t nwin = (n + kBaseQuantum - 1) / kBaseQuantum;
  if (nwin <= 32) {  // a short column: one warp, a lane per window, no barrier
    if (warp) return;
    const uint32_t gm = __ballot_sync(0xffffffffu, lane < nwin && grow[lane]);
    uint32_t starts = 0;
    for (uint32_t w = 0; w < nwin; w += gm >> w & 1u ? 4 : 1) starts |= 1u << w;
    if (lane < nwin) {
      const uint32_t b = __popc(starts & ((2u << lane) - 1u)) - 1;
      w2b[lane] = b;
      if (starts >> lane & 1u) {
        FrameDesc f;
        f.value_off = lane * (uint64_t)kBaseQuantum;
        f.n = (uint32_t)(qmin(f.value_off + (gm >> lane & 1u ? kMaxBlock : kBaseQuantum), n) - f.value_off);
        f.payload_off = 0;
        f.plen = 0;
        f.mode = 0;
        f.aux = 0;
        frames[b] = f;
      }
    }
    for (uint64_t w = nwin + lane; w * kBaseQuantum < bound; w += 32) w2b[w] = kEmpty32;  // no block
    if (lane == 0) *nb = __popc(starts);
    return;
  }
  if (t == 0) {
    s_state = 0;
    s_count = 0;
  }
  __syncthreads();
  auto apply = [](uint32_t m, uint32_t st) { return (m >> (2 * st)) & 3u; };
  auto compose = [&](uint32_t g, uint32_t f) {  // g after f
    uint32_t r = 0;
#pragma unroll
    for (uint32_t st = 0; st < 4; st++) r |= apply(g, apply(f, st)) << (2 * st);
    return r;
  };
  const uint32_t kId = 0u | (1u << 2) | (2u << 4) | (3u << 6);
  for (uint64_t w0 = 0; w0 < nwin; w0 += (uint64_t)kPlanThreads * kPer) {
    uint64_t wb = w0 + (uint64_t)t * kPer;
    uint8_t g[kPer];
    uint32_t m = kId;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      g[q] = wb + q < nwin ? grow[wb + q] : 0;
      uint32_t f = wb + q < nwin ? ((g[q] ? 3u : 0u) | (0u << 2) | (1u << 4) | (2u << 6)) : kId;
      m = compose(f, m);
    }
    // inclusive scan of the maps in window order
    uint32_t inc = m;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc = compose(inc, u);
    }
    if (lane == 31) s_wmap[warp] = inc;
    __syncthreads();
    uint32_t pre = kId;  // maps of the warps before this one
    for (int k = 0; k < warp; k++) pre = compose(s_wmap[k], pre);
    uint32_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = kId;
    uint32_t st = apply(compose(ex, pre), s_state);  // state before window wb
    uint32_t starts = 0;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      if (wb + q < nwin && st == 0) starts |= 1u << q;
      if (wb + q < nwin) st = st ? st - 1 : (g[q] ? 3u : 0u);
    }
    uint32_t c = __popc(starts), ci = c;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t u = __shfl_up_sync(0xffffffffu, ci, o);
      if (lane >= o) ci += u;
    }
    if (lane == 31) s_wcnt[warp] = ci;
    __syncthreads();
    uint32_t base = s_count;
    for (int k = 0; k < warp; k++) base += s_wcnt[k];
    base += ci - c;
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      if (wb + q < nwin) w2b[wb + q] = base + __popc(starts >> q & 1u) - 1;
      if (!(starts >> q & 1u)) continue;
      uint64_t s0 = (wb + q) * (uint64_t)kBaseQuantum;
      uint64_t end = g[q] ? qmin(s0 + kMaxBlock, n) : qmin(s0 + kBaseQuantum, n);
      FrameDesc f;
      f.value_off = s0;
      f.n = (uint32_t)(end - s0);
      f.payload_off = 0;
      f.plen = 0;
      f.mode = 0;
      f.aux = 0;
      frames[base++] = f;
    }
    __syncthreads();
    if (t == kPlanThreads - 1) {  // the last thread holds the chunk's final state
      s_state = st;
      uint32_t tot = 0;
      for (int k = 0; k < kWarps; k++) tot += s_wcnt[k];
      s_count += tot;
    }
    __syncthreads();
  }
  if (t == 0) *nb = s_count;
  for (uint64_t w = nwin + t; w * kBaseQuantum < bound; w += kPlanThreads) w2b[w] = kEmpty32;  // no block
}

__global__ void k_frame_sizes(const FrameDesc* __restrict__ frames, const uint32_t* __restrict__ nbp, uint32_t maxb,
                              uint64_t* __restrict__ sizes) {
  uint32_t nb = *nbp;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < maxb; i += gridDim.x * blockDim.x)
    sizes[i] = i < nb ? 9ull + frames[i].plen : 0ull;
}
__global__ void k_frame_apply(FrameDesc* frames, const uint32_t* __restrict__ nbp, const uint64_t* __restrict__ offs,
                              const uint64_t* __restrict__ base_p) {
  uint32_t nb = *nbp;
  uint64_t base = *base_p;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x)
    frames[i].payload_off = base + offs[i] + 9;
}

// ---------------------------------------------------------------------------
// The kernels: of one lane (the arguments are the launch's), and of a group of
// lanes, where map[CTA] names the lane and the CTA's place among the lane's.
// A group's launch takes as long as its longest lane or as their sum needs on
// the whole chip: 192 columns of 1,024 to 1,048,576 values in 2,183 launches
// and 256 waits took 5.6 ms, in 50 launches and 5 waits 1.2 ms.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kAlpWarps * 32) k_alp_stats(const uint64_t* __restrict__ v, uint64_t n,
                                                              const uint64_t* d_n, uint64_t fixed_bs, uint64_t items,
                                                              SubStats* __restrict__ ss) {
  alp_stats(blockIdx.x, v, n, d_n, fixed_bs, items, ss);
}
template <bool FLOATS>
__global__ void __cluster_dims__(kStatsCluster, 1, 1) __launch_bounds__(kStatsWarps * 32, FLOATS ? 3 : 5) k_sub_stats(
    const uint64_t* __restrict__ v, uint64_t n, const uint64_t* d_n, uint64_t fixed_bs, uint64_t items, int dtype,
    int level, SubStats* __restrict__ ss, FmStat* __restrict__ fms, uint64_t* __restrict__ smp16, uint8_t* __restrict__ grow,
    uint32_t* __restrict__ winbits) {
  sub_stats<FLOATS>(blockIdx.x, v, n, d_n, fixed_bs, items, dtype, level, ss, fms, smp16, grow, winbits);
}
template <bool ENT, bool SAMPLE>
__global__ void __launch_bounds__(kEncThreads, 2) k_decide(const uint64_t* __restrict__ lane, FrameDesc* frames,
                                                        const uint32_t* __restrict__ nbp, uint64_t fixed_bs,
                                                        int dtype, int level, const SubStats* __restrict__ ss,
                                                        const FmStat* __restrict__ fms,
                                                        const uint64_t* __restrict__ smp16,
                                                        const uint32_t* __restrict__ winbits,
                                                        uint8_t* __restrict__ scratch, EntRec* __restrict__ ent,
                                                        RdRec* __restrict__ rdr, BlkRec* __restrict__ blk) {
  decide<ENT, SAMPLE>(blockIdx.x, lane, frames, nbp, fixed_bs, dtype, level, ss, fms, smp16, winbits, scratch, ent, rdr,
                      blk);
}
template <bool ENT>
__global__ void __launch_bounds__(kEncThreads, 2) k_emit(const uint64_t* __restrict__ lane,
                                                      const FrameDesc* __restrict__ frames,
                                                      const uint32_t* __restrict__ nbp,
                                                      const uint32_t* __restrict__ w2b, uint32_t split,
                                                      uint64_t fixed_bs, int dtype,
                                                      const SubStats* __restrict__ ss,
                                                      const FmStat* __restrict__ fms,
                                                      const RdRec* __restrict__ rdr, const BlkRec* __restrict__ blk,
                                                      uint8_t* __restrict__ scratch, uint8_t* __restrict__ outbuf,
                                                      uint64_t out_cap, const EntRec* __restrict__ ent) {
  emit_unit<ENT>(blockIdx.x, lane, frames, nbp, w2b, split, fixed_bs, dtype, ss, fms, rdr, blk, scratch, outbuf,
                 out_cap, ent);
}
__global__ void __launch_bounds__(kPlanThreads)
    k_plan(const uint8_t* __restrict__ grow, uint64_t n, const uint64_t* d_n, uint64_t fixed_bs, FrameDesc* frames,
           uint32_t* nb, uint32_t* __restrict__ w2b) {
  plan_blocks(blockIdx.x, gridDim.x, grow, n, d_n, fixed_bs, frames, nb, w2b);
}

__global__ void __launch_bounds__(kAlpWarps * 32) k_group_alp(const EncLane* __restrict__ lanes,
                                                              const uint32_t* __restrict__ map) {
  const uint32_t m = map[blockIdx.x];
  const EncLane& L = lanes[m >> 16];
  alp_stats(m & 0xFFFF, L.v, L.n, L.d_n, L.fixed_bs, L.items, (SubStats*)L.ss);
}
template <bool FLOATS>
__global__ void __cluster_dims__(kStatsCluster, 1, 1) __launch_bounds__(kStatsWarps * 32, FLOATS ? 3 : 5)
    k_group_stats(const EncLane* __restrict__ lanes, const uint32_t* __restrict__ map, int level) {
  const uint32_t m = map[blockIdx.x];
  const EncLane& L = lanes[m >> 16];
  sub_stats<FLOATS>(m & 0xFFFF, L.v, L.n, L.d_n, L.fixed_bs, L.items, L.dtype, level, (SubStats*)L.ss, (FmStat*)L.fms,
                    L.smp16, L.grow, L.winbits);
}
template <bool ENT, bool SAMPLE>
__global__ void __launch_bounds__(kEncThreads, 2)
    k_group_decide(const EncLane* __restrict__ lanes, const uint32_t* __restrict__ map, int level) {
  const uint32_t m = map[blockIdx.x];
  const EncLane& L = lanes[m >> 16];
  decide<ENT, SAMPLE>(m & 0xFFFF, L.v, L.frames, L.nb, L.fixed_bs, L.dtype, level, (const SubStats*)L.ss,
                      (const FmStat*)L.fms, L.smp16, L.winbits, L.scratch, (EntRec*)L.ent, (RdRec*)L.rdr,
                      (BlkRec*)L.blk);
}
template <bool ENT>
__global__ void __launch_bounds__(kEncThreads, 2)
    k_group_emit(const EncLane* __restrict__ lanes, const uint32_t* __restrict__ map) {
  const uint32_t m = map[blockIdx.x];
  const EncLane& L = lanes[m >> 16];
  emit_unit<ENT>(m & 0xFFFF, L.v, L.frames, L.nb, L.w2b, 1, L.fixed_bs, L.dtype, (const SubStats*)L.ss,
                 (const FmStat*)L.fms, (const RdRec*)L.rdr, (const BlkRec*)L.blk, L.scratch, L.out, L.out_cap,
                 (const EntRec*)L.ent);
}
__global__ void __launch_bounds__(kPlanThreads) k_group_plan(const EncLane* __restrict__ lanes) {
  const EncLane& L = lanes[blockIdx.x];
  plan_blocks(0, 1, L.grow, L.n, L.d_n, L.fixed_bs, L.frames, L.nb, L.w2b);
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
static size_t enc_smem_bytes() { return sizeof(EncSmem); }

void launch_plan(const uint8_t* grow, uint64_t n, const uint64_t* d_n, uint64_t fixed_bs, FrameDesc* frames,
                 uint32_t* nb, uint32_t* w2b, cudaStream_t st) {
  unsigned g = 1;
  if (fixed_bs) g = (unsigned)qmin(((n + fixed_bs - 1) / fixed_bs + kPlanThreads - 1) / kPlanThreads, 4096);
  if (g == 0) g = 1;
  k_plan<<<g, kPlanThreads, 0, st>>>(grow, n, d_n, fixed_bs, frames, nb, w2b);
  count_launches(1);
}

uint64_t sub_stats_items(uint64_t n, uint64_t fixed_bs) {
  if (fixed_bs) return ((n + fixed_bs - 1) / fixed_bs) * ((fixed_bs + kSub - 1) / kSub);
  return ((n + kBaseQuantum - 1) / kBaseQuantum) * (uint64_t)(kBaseQuantum / kSub);
}
uint64_t sub_stats_bytes() { return sizeof(SubStats); }
uint64_t fm_stats_bytes() { return sizeof(FmStat); }

void launch_sub_stats(const uint64_t* lane, uint64_t n, const uint64_t* d_n, uint64_t fixed_bs, int dtype, int level,
                      void* ss, void* fms, uint64_t* smp16, uint8_t* grow, uint32_t* winbits, cudaStream_t st) {
  uint64_t items = sub_stats_items(n, fixed_bs);
  if (!items) return;
  const uint64_t per = kStatsWarps * kStatsCluster;
  const unsigned g = (unsigned)((items + per - 1) / per * kStatsCluster);
  if (dtype_float(dtype)) {
    k_sub_stats<true><<<g, kStatsWarps * 32, 0, st>>>(lane, n, d_n, fixed_bs, items, dtype, level, (SubStats*)ss, (FmStat*)fms,
                                                       smp16, grow, winbits);
    if (level >= 1) {
      k_alp_stats<<<(unsigned)((items + kAlpWarps - 1) / kAlpWarps), kAlpWarps * 32, 0, st>>>(lane, n, d_n, fixed_bs, items,
                                                                                            (SubStats*)ss);
      count_launches(1);
    }
  } else
    k_sub_stats<false><<<g, kStatsWarps * 32, 0, st>>>(lane, n, d_n, fixed_bs, items, dtype, level, (SubStats*)ss,
                                                        (FmStat*)fms, nullptr, grow, winbits);
  count_launches(1);
}

static int enc_smem_ready() {
  const int sm = (int)enc_smem_bytes();
  static std::atomic<unsigned long long> smem_set{0};
  once_per_device(smem_set, [sm] {
    auto set = [sm](auto* kernel) { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm); };
    set(k_decide<false, false>);
    set(k_decide<true, false>);
    set(k_decide<false, true>);
    set(k_emit<false>);
    set(k_emit<true>);
    set(k_group_decide<false, false>);
    set(k_group_decide<true, false>);
    set(k_group_decide<false, true>);
    set(k_group_emit<false>);
    set(k_group_emit<true>);
  });
  return sm;
}

void launch_decide(const uint64_t* lane, FrameDesc* frames, const uint32_t* nb, uint32_t max_blocks, uint64_t fixed_bs,
                   int dtype, int level, const void* ss, const void* fms, const uint64_t* smp16,
                   const uint32_t* winbits, uint8_t* scratch, void* ent, void* rdr, void* blk, bool sample,
                   cudaStream_t st) {
  const int sm = enc_smem_ready();
  if (max_blocks) {
    if (ent)
      k_decide<true, false><<<max_blocks, kEncThreads, sm, st>>>(lane, frames, nb, fixed_bs, dtype, level,
                                                          (const SubStats*)ss, (const FmStat*)fms, smp16, winbits,
                                                          scratch, (EntRec*)ent, (RdRec*)rdr, (BlkRec*)blk);
    else if (sample)
      k_decide<false, true><<<max_blocks, kEncThreads, sm, st>>>(lane, frames, nb, fixed_bs, dtype, level,
                                                                 (const SubStats*)ss, (const FmStat*)fms, smp16,
                                                                 winbits, scratch, nullptr, (RdRec*)rdr, (BlkRec*)blk);
    else
      k_decide<false, false><<<max_blocks, kEncThreads, sm, st>>>(lane, frames, nb, fixed_bs, dtype, level,
                                                                  (const SubStats*)ss, (const FmStat*)fms, smp16,
                                                                  winbits, scratch, nullptr, (RdRec*)rdr, (BlkRec*)blk);
  }
  count_launches(max_blocks ? 1 : 0);
}

static uint64_t emit_units(uint64_t n, uint64_t fixed_bs, uint64_t max_blocks) {
  return fixed_bs ? max_blocks * ((fixed_bs + kBaseQuantum - 1) / kBaseQuantum) : (n + kBaseQuantum - 1) / kBaseQuantum;
}

// Two CTAs per window while the windows alone leave places free (two CTAs of
// an SM's registers): 1,048,576 prices' 32 windows emit on 64 SMs.
void launch_emit(const uint64_t* lane, const FrameDesc* frames, const uint32_t* nb, uint32_t max_blocks,
                 const uint32_t* w2b, uint64_t n, uint64_t fixed_bs, int dtype, const void* ss, const void* fms,
                 const void* rdr, const void* blk, uint8_t* scratch, uint8_t* out, uint64_t out_cap, const void* ent,
                 cudaStream_t st) {
  if (max_blocks) {
    const uint64_t units = emit_units(n, fixed_bs, max_blocks);
    const uint32_t split = units < 2 * 148 && !ent ? 2 : 1;
    const unsigned g = (unsigned)(units * split);
    if (ent)
      k_emit<true><<<g, kEncThreads, enc_smem_bytes(), st>>>(lane, frames, nb, w2b, split, fixed_bs, dtype,
                                                             (const SubStats*)ss, (const FmStat*)fms, (const RdRec*)rdr,
                                                             (const BlkRec*)blk, scratch, out, out_cap,
                                                             (const EntRec*)ent);
    else
      k_emit<false><<<g, kEncThreads, enc_smem_bytes(), st>>>(lane, frames, nb, w2b, split, fixed_bs, dtype,
                                                              (const SubStats*)ss, (const FmStat*)fms,
                                                              (const RdRec*)rdr, (const BlkRec*)blk, scratch, out,
                                                              out_cap, nullptr);
  }
  count_launches(max_blocks ? 1 : 0);
}

uint64_t rd_rec_bytes() { return sizeof(RdRec); }
uint64_t blk_rec_bytes() { return sizeof(BlkRec); }
uint64_t ent_rec_bytes() { return sizeof(EntRec); }

unsigned long long* device_win_counters() {
  void* p = nullptr;
  cudaGetSymbolAddress(&p, g_wins);
  return reinterpret_cast<unsigned long long*>(p);
}

}  // namespace qb

#include "qb_scan.cuh"

namespace qb {
// A nested lane's varint(length) and header at *nest.pos, for frames of
// `total` bytes; returns the offset of the first frame.
__device__ inline uint64_t nest_base(const NestedLane& nest, uint64_t pos, uint64_t total) {
  return pos + varint_len(16 + total) + 16;
}
__device__ inline void nest_write(const NestedLane& nest, uint64_t pos, uint64_t total) {
  const uint64_t at = nest_base(nest, pos, total);
  if (at <= nest.cap) {
    put_varint(nest.out + pos, 16 + total);
    for (int i = 0; i < 16; i++) nest.out[at - 16 + i] = nest.hdr.b[i];
    for (int i = 0; nest.d_n && i < 8; i++) nest.out[at - 8 + i] = (uint8_t)(*nest.d_n >> (8 * i));
  }
  *nest.pos = at + total;
}
__global__ void k_nest_base(NestedLane nest, const uint64_t* __restrict__ total, uint64_t* __restrict__ base) {
  if (threadIdx.x || blockIdx.x) return;
  const uint64_t pos = *nest.pos;
  *base = nest_base(nest, pos, *total);
  nest_write(nest, pos, *total);
}

// At most kSmallWords frames in one CTA of 1,024 threads: k_frame_sizes, the
// exclusive scan and k_frame_apply in one launch.
__device__ __forceinline__ void frame_offsets_small(FrameDesc* frames, const uint32_t* __restrict__ nbp,
                                                    uint64_t* __restrict__ base_p, uint64_t* __restrict__ total,
                                                    const NestedLane& nest) {
  __shared__ uint64_t wsum[32];
  uint32_t nb = *nbp, t = threadIdx.x, l = t & 31, warp = t >> 5;
  uint64_t base = nest.pos ? *nest.pos : *base_p;
  uint64_t v[kSmallPer], s = 0;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    uint32_t i = t * kSmallPer + k;
    v[k] = i < nb ? 9ull + frames[i].plen : 0ull;
    s += v[k];
  }
  uint64_t inc = s;
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if ((int)l >= o) inc += u;
  }
  if (l == 31) wsum[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint64_t x = wsum[l];
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t u = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)l >= o) x += u;
    }
    wsum[l] = x;
    if (l == 31) *total = x;
  }
  __syncthreads();
  if (nest.pos) {
    const uint64_t pos = base;
    base = nest_base(nest, pos, wsum[31]);
    if (t == 0) nest_write(nest, pos, wsum[31]);
  }
  uint64_t run = (warp ? wsum[warp - 1] : 0ull) + inc - s;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    uint32_t i = t * kSmallPer + k;
    if (i < nb) frames[i].payload_off = base + run + 9;
    run += v[k];
  }
}

__global__ void __launch_bounds__(1024) k_frame_offsets_small(FrameDesc* frames, const uint32_t* __restrict__ nbp,
                                                              uint64_t* __restrict__ base_p,
                                                              uint64_t* __restrict__ total, NestedLane nest) {
  frame_offsets_small(frames, nbp, base_p, total, nest);
}
// A column's lanes one after another: a limb's stream begins where the one
// before it ends.
__global__ void __launch_bounds__(1024) k_group_offsets(const EncLane* __restrict__ lanes,
                                                        const EncCol* __restrict__ cols) {
  const EncCol& C = cols[blockIdx.x];
  for (int k = 0; k < max(C.nl, 1); k++) {
    const EncLane& L = lanes[C.lane0 + k];
    frame_offsets_small(L.frames, L.nb, C.res, C.nl ? C.vmin + 4 : C.res + 1, L.nest);
    __syncthreads();
  }
}

// All lanes of a group of columns whose lanes launch_begin_cols has written.
void launch_encode_group(const EncGroup& G, int level, bool ent, bool sample, cudaStream_t st) {
  const int sm = enc_smem_ready();
  if (G.nfstats) k_group_stats<true><<<G.nfstats, kStatsWarps * 32, 0, st>>>(G.lanes, G.fstats, level);
  if (G.nistats) k_group_stats<false><<<G.nistats, kStatsWarps * 32, 0, st>>>(G.lanes, G.istats, level);
  if (G.nalp && level >= 1) k_group_alp<<<G.nalp, kAlpWarps * 32, 0, st>>>(G.lanes, G.alp);
  k_group_plan<<<G.nlanes, kPlanThreads, 0, st>>>(G.lanes);
  if (ent) k_group_decide<true, false><<<G.nblocks, kEncThreads, sm, st>>>(G.lanes, G.blocks, level);
  else if (sample) k_group_decide<false, true><<<G.nblocks, kEncThreads, sm, st>>>(G.lanes, G.blocks, level);
  else k_group_decide<false, false><<<G.nblocks, kEncThreads, sm, st>>>(G.lanes, G.blocks, level);
  k_group_offsets<<<G.ncols, 1024, 0, st>>>(G.lanes, G.cols);
  if (ent) k_group_emit<true><<<G.nunits, kEncThreads, sm, st>>>(G.lanes, G.units);
  else k_group_emit<false><<<G.nunits, kEncThreads, sm, st>>>(G.lanes, G.units);
  count_launches(4 + (G.nfstats != 0) + (G.nistats != 0) + (G.nalp && level >= 1));
}
// CTAs of a lane in the group's launches, as map entries of lane `lane`.
static void map_ctas(std::vector<uint32_t>& map, uint32_t lane, uint64_t ctas) {
  for (uint64_t k = 0; k < ctas; k++) map.push_back(lane << 16 | (uint32_t)k);
}
void map_lane(EncMaps& M, uint32_t lane, uint64_t n, uint64_t fixed_bs, int dtype, uint64_t max_blocks) {
  const uint64_t items = sub_stats_items(n, fixed_bs), per = kStatsWarps * kStatsCluster;
  map_ctas(dtype_float(dtype) ? M.fstats : M.istats, lane, (items + per - 1) / per * kStatsCluster);
  if (dtype_float(dtype)) map_ctas(M.alp, lane, (items + kAlpWarps - 1) / kAlpWarps);
  map_ctas(M.blocks, lane, max_blocks);
  map_ctas(M.units, lane, emit_units(n, fixed_bs, max_blocks));
}

void launch_frame_offsets(FrameDesc* frames, const uint32_t* nb, uint32_t max_blocks, uint64_t* base,
                          uint64_t* sizes_tmp, uint64_t* tile_tmp, uint64_t* total, const NestedLane& nest,
                          cudaStream_t st) {
  if (max_blocks == 0) {  // a lane without values: its header alone
    if (!nest.pos) return;
    cudaMemsetAsync(total, 0, 8, st);
    k_nest_base<<<1, 32, 0, st>>>(nest, total, base);
    count_launches(1);
    return;
  }
  if (max_blocks <= kSmallWords) {
    k_frame_offsets_small<<<1, 1024, 0, st>>>(frames, nb, base, total, nest);
    count_launches(1);
    return;
  }
  unsigned g = (unsigned)qmin((max_blocks + 255) / 256, 1024);
  k_frame_sizes<<<g, 256, 0, st>>>(frames, nb, max_blocks, sizes_tmp);
  scan_exclusive_u64(sizes_tmp, sizes_tmp, max_blocks, tile_tmp, total, st);
  if (nest.pos) k_nest_base<<<1, 32, 0, st>>>(nest, total, base);
  k_frame_apply<<<g, 256, 0, st>>>(frames, nb, sizes_tmp, base);
  count_launches((nest.pos ? 3 : 2) + scan_launches(max_blocks));
}
}  // namespace qb
