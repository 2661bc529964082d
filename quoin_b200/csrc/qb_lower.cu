// Column lowering and validity handling on the device: typed values -> u64
// lane with null compaction (reference lib.rs:389-403,446-454,
// validity.rs:122-127), the decimal limb split (decimal.rs:174-212,339-377)
// and the validity run-length blob (validity.rs:40-70).
#include "qb_common.cuh"
#include "qb_kernels.h"
#include "qb_scan.cuh"

namespace qb {

__device__ inline uint64_t lower_one(const uint8_t* base, uint64_t i, int dtype) {
  switch (dtype) {
    case DT_I32: return (uint64_t)(int64_t)reinterpret_cast<const int32_t*>(base)[i];
    case DT_U32: return (uint64_t)reinterpret_cast<const uint32_t*>(base)[i];
    case DT_F32: return f32bits_to_f64bits(reinterpret_cast<const uint32_t*>(base)[i]);
    default: return reinterpret_cast<const uint64_t*>(base)[i];
  }
}

__device__ inline uint32_t bm_word_at(const uint8_t* bm, uint64_t w, uint64_t n) {
  uint64_t nbytes = (n + 7) / 8;
  uint32_t bits = 0;
  if (w * 4 + 4 <= nbytes) bits = ld_u32(bm + w * 4);
  else
    for (int k = 0; w * 4 + k < nbytes; k++) bits |= (uint32_t)bm[w * 4 + k] << (8 * k);
  uint64_t rem = n - w * 32;
  if (rem < 32) bits &= (1u << rem) - 1u;
  return bits;
}

// A warp lowers 8 bitmap words (256 positions) per step: lanes 0-7 fetch the
// words and their ranks, every lane loads its 8 values up front, then each
// valid value goes to lane[rank].
__device__ __forceinline__ void lower_words(const uint8_t* __restrict__ values, int dtype,
                                            const uint8_t* __restrict__ bm, const uint64_t* __restrict__ word_rank,
                                            uint64_t n, uint64_t* __restrict__ lane) {
  uint64_t nw = (n + 31) / 32;
  int l = threadIdx.x & 31;
  uint32_t below = (1u << l) - 1u;
  uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t w0 = warp * 8; w0 < nw; w0 += nwarps * 8) {
    uint32_t mybits = 0;
    uint64_t myrank = 0;
    if (bm && l < 8 && w0 + l < nw) {
      mybits = bm_word_at(bm, w0 + l, n);
      myrank = word_rank[w0 + l];
    }
    uint64_t vals[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint64_t i = (w0 + q) * 32 + l;
      vals[q] = i < n ? lower_one(values, i, dtype) : 0ull;
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
      uint64_t i = (w0 + q) * 32 + l;
      uint32_t bits = __shfl_sync(0xffffffffu, mybits, q);
      uint64_t rank = __shfl_sync(0xffffffffu, myrank, q);
      if (i >= n) continue;
      if (!bm) lane[i] = vals[q];
      else if ((bits >> l) & 1u) lane[rank + __popc(bits & below)] = vals[q];
    }
  }
}

__global__ void k_lower(const uint8_t* __restrict__ values, int dtype, const uint8_t* __restrict__ bm,
                        const uint64_t* __restrict__ word_rank, uint64_t n, uint64_t* __restrict__ lane) {
  lower_words(values, dtype, bm, word_rank, n, lane);
}

static unsigned grid_for_words(uint64_t n) {
  uint64_t nw = (n + 31) / 32;
  uint64_t g = (nw + 7) / 8;
  if (g > 148ull * 32) g = 148ull * 32;
  return g ? (unsigned)g : 1u;
}
static unsigned grid_for_lower(uint64_t n) {
  uint64_t nw = (n + 31) / 32;
  uint64_t g = (nw + 63) / 64;  // 8 warps x 8 words per block step
  if (g > 148ull * 32) g = 148ull * 32;
  return g ? (unsigned)g : 1u;
}

void launch_lower(const void* values, int dtype, const uint8_t* bm, const uint64_t* word_rank, uint64_t n,
                  uint64_t* lane, cudaStream_t st) {
  if (n) k_lower<<<grid_for_lower(n), 256, 0, st>>>((const uint8_t*)values, dtype, bm, word_rank, n, lane);
  count_launches(n ? 1 : 0);
}

// ---------------------------------------------------------------------------
// Decimal: signed minimum over valid values, then limbs of (v - vmin).
// ---------------------------------------------------------------------------
template <int NL>
struct Limbs {
  uint64_t l[NL];
};
template <int NL>
__device__ __forceinline__ bool lt_signed(const Limbs<NL>& a, const Limbs<NL>& b) {  // reference decimal.rs:254-269
  bool lt = (int64_t)a.l[NL - 1] < (int64_t)b.l[NL - 1], eq = a.l[NL - 1] == b.l[NL - 1];
#pragma unroll
  for (int i = NL - 2; i >= 0; i--) {
    lt = lt || (eq && a.l[i] < b.l[i]);
    eq = eq && a.l[i] == b.l[i];
  }
  return lt;
}
template <int NL>
__device__ __forceinline__ Limbs<NL> most_positive() {
  Limbs<NL> r;
#pragma unroll
  for (int i = 0; i < NL; i++) r.l[i] = i == NL - 1 ? 0x7FFFFFFFFFFFFFFFull : ~0ull;
  return r;
}
// The CTA's minimum, in every lane of warp 0 (256 or 1,024 threads).
template <int NL>
__device__ Limbs<NL> block_min(Limbs<NL> m, Limbs<NL>* s_v) {
  auto warp = [&](Limbs<NL> x) {
    for (int o = 16; o; o >>= 1) {
      Limbs<NL> y;
#pragma unroll
      for (int i = 0; i < NL; i++) y.l[i] = __shfl_xor_sync(0xffffffffu, x.l[i], o);
      if (lt_signed(y, x)) x = y;
    }
    return x;
  };
  m = warp(m);
  if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = m;
  __syncthreads();
  m = (threadIdx.x & 31) < blockDim.x / 32 ? s_v[threadIdx.x & 31] : most_positive<NL>();
  return warp(m);
}

// Minima of the CTAs' shares, then of those (one CTA).  No valid value leaves
// the largest one, which the split then never subtracts from.  One thread of a
// CTA comparing its 256 candidates and one thread the CTAs' took 290 us for
// 10,000,019 Decimal128 values; reading them takes 25 us at the copy rate.
constexpr int kVminParts = 148 * 6;
template <int NL>
__device__ __forceinline__ void vmin_partial(const uint64_t* __restrict__ values, const uint8_t* __restrict__ bm,
                                             uint64_t n, uint64_t* __restrict__ tmp) {
  __shared__ Limbs<NL> s_v[32];
  Limbs<NL> best = most_positive<NL>();
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * step) {
    Limbs<NL> x[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint64_t i = i0 + u * step;
      x[u] = most_positive<NL>();
      if (i < n && (!bm || ((bm[i >> 3] >> (i & 7)) & 1))) {
#pragma unroll
        for (int k = 0; k < NL; k++) x[u].l[k] = values[i * NL + k];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (lt_signed(x[u], best)) best = x[u];
  }
  best = block_min(best, s_v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NL; k++) tmp[blockIdx.x * NL + k] = best.l[k];
}
template <int NL>
__global__ void __launch_bounds__(256) k_decimal_vmin_partial(const uint64_t* __restrict__ values,
                                                              const uint8_t* __restrict__ bm, uint64_t n,
                                                              uint64_t* __restrict__ tmp) {
  vmin_partial<NL>(values, bm, n, tmp);
}
template <int NL>
__device__ __forceinline__ void vmin_final(const uint64_t* __restrict__ tmp, int nparts, bool any,
                                           uint64_t* __restrict__ vmin) {
  __shared__ Limbs<NL> s_v[32];
  Limbs<NL> m = most_positive<NL>();
  for (int b = threadIdx.x; b < nparts; b += blockDim.x) {
    Limbs<NL> x;
#pragma unroll
    for (int k = 0; k < NL; k++) x.l[k] = tmp[b * NL + k];
    if (lt_signed(x, m)) m = x;
  }
  m = block_min(m, s_v);
  if (threadIdx.x < 4) {
    uint64_t v = 0;
#pragma unroll
    for (int k = 0; k < NL; k++)
      if (k == (int)threadIdx.x && any) v = m.l[k];
    vmin[threadIdx.x] = v;
  }
}
template <int NL>
__global__ void __launch_bounds__(1024) k_decimal_vmin_final(const uint64_t* __restrict__ tmp, int nparts, bool any,
                                                             uint64_t* __restrict__ vmin) {
  vmin_final<NL>(tmp, nparts, any, vmin);
}

uint64_t decimal_vmin_tmp_words() { return 4ull * kVminParts; }

// any: whether there is a valid value (0 for the minimum otherwise).
void launch_decimal_vmin(const uint8_t* values, int nlimbs, const uint8_t* bm, uint64_t n, bool any,
                         uint64_t* vmin_tmp, uint64_t* vmin, cudaStream_t st) {
  const int parts = (int)qmin((n + 1023) / 1024 + 1, kVminParts);
  const uint64_t* v = reinterpret_cast<const uint64_t*>(values);
  if (nlimbs == 2) {
    k_decimal_vmin_partial<2><<<parts, 256, 0, st>>>(v, bm, n, vmin_tmp);
    k_decimal_vmin_final<2><<<1, 1024, 0, st>>>(vmin_tmp, parts, any, vmin);
  } else {
    k_decimal_vmin_partial<4><<<parts, 256, 0, st>>>(v, bm, n, vmin_tmp);
    k_decimal_vmin_final<4><<<1, 1024, 0, st>>>(vmin_tmp, parts, any, vmin);
  }
  count_launches(2);
}

// A decimal container's bytes before its validity blob (decimal.rs:56-85):
// 19 given bytes and the limbs of vmin; *d_pos = their count.
__global__ void k_put_decimal_header(uint8_t* dst, Bytes19 head, int nl, const uint64_t* __restrict__ vmin,
                                     uint64_t* d_pos) {
  const int t = threadIdx.x;
  if (t < 19) dst[t] = head.b[t];
  if (t < 8 * nl) dst[19 + t] = (uint8_t)(vmin[t >> 3] >> (8 * (t & 7)));
  if (t == 0) *d_pos = 19 + 8ull * nl;
}
void launch_put_decimal_header(uint8_t* dst, const Bytes19& head, int nl, const uint64_t* vmin, uint64_t* d_pos,
                               cudaStream_t st) {
  k_put_decimal_header<<<1, 32, 0, st>>>(dst, head, nl, vmin, d_pos);
  count_launches(1);
}

// limbs[k * stride + j] = limb k of (v_i - vmin) for the j-th valid value i.
__device__ __forceinline__ void split_words(const uint8_t* __restrict__ values, int nl, const uint8_t* __restrict__ bm,
                                            const uint64_t* __restrict__ word_rank, uint64_t n,
                                            const uint64_t* __restrict__ vmin, uint64_t* __restrict__ limbs,
                                            uint64_t stride) {
  uint64_t nw = (n + 31) / 32, nbytes = (n + 7) / 8;
  int l = threadIdx.x & 31;
  uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint64_t vm[4];
  for (int k = 0; k < 4; k++) vm[k] = vmin[k];
  for (uint64_t w = warp; w < nw; w += nwarps) {
    uint64_t i = w * 32 + l;
    uint64_t j = i;
    bool valid = i < n;
    if (bm) {
      uint32_t byte = (w * 4 + (l >> 3) < nbytes) ? bm[w * 4 + (l >> 3)] : 0u;
      uint32_t bits = 0;
      for (int k = 0; k < 4; k++) bits |= __shfl_sync(0xffffffffu, byte, k * 8) << (8 * k);
      valid = valid && ((bits >> l) & 1u);
      j = word_rank[w] + __popc(bits & ((1u << l) - 1u));
    }
    if (!valid) continue;
    const uint64_t* p = reinterpret_cast<const uint64_t*>(values + i * 8ull * nl);
    uint64_t borrow = 0;
    for (int k = 0; k < nl; k++) {  // reference decimal.rs:281-293 (sub with borrow)
      uint64_t a = p[k], b = vm[k];
      uint64_t d1 = a - b;
      uint64_t b1 = a < b;
      uint64_t d2 = d1 - borrow;
      uint64_t b2 = d1 < borrow;
      limbs[k * stride + j] = d2;
      borrow = b1 | b2;
    }
  }
}

__global__ void k_decimal_split(const uint8_t* __restrict__ values, int nl, const uint8_t* __restrict__ bm,
                                const uint64_t* __restrict__ word_rank, uint64_t n, const uint64_t* __restrict__ vmin,
                                uint64_t* __restrict__ limbs, uint64_t stride) {
  split_words(values, nl, bm, word_rank, n, vmin, limbs, stride);
}

void launch_decimal_split(const uint8_t* values, int nlimbs, const uint8_t* bm, const uint64_t* word_rank,
                          uint64_t n, const uint64_t* vmin, uint64_t* limbs, uint64_t limb_stride, cudaStream_t st) {
  if (n) k_decimal_split<<<grid_for_words(n), 256, 0, st>>>(values, nlimbs, bm, word_rank, n, vmin, limbs, limb_stride);
  count_launches(n ? 1 : 0);
}

// ---------------------------------------------------------------------------
// Validity blob: the smaller of [1] ++ LEB128 alternating run lengths
// (starting with a null run) or [0] ++ the raw bitmap bytes.
// ---------------------------------------------------------------------------
// Transition mask of word w: bit j set when bit (32w + j) differs from its
// predecessor (the bit before position 0 is taken as 0, i.e. a null).
__device__ inline uint32_t trans_mask(const uint8_t* bm, uint64_t w, uint64_t n) {
  uint32_t b = bm_word_at(bm, w, n);
  uint32_t prev = w ? (bm_word_at(bm, w - 1, n) >> 31) : 0u;
  uint32_t t = b ^ ((b << 1) | prev);
  uint64_t rem = n - w * 32;
  if (rem < 32) t &= (1u << rem) - 1u;
  return t;
}

__global__ void k_vb_last(const uint8_t* __restrict__ bm, uint64_t n, uint64_t* __restrict__ last) {
  uint64_t nw = (n + 31) / 32;
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t t = trans_mask(bm, w, n);
    last[w] = t ? w * 32 + (31 - __clz(t)) : 0ull;
  }
}
__global__ void k_vb_sizes(const uint8_t* __restrict__ bm, uint64_t n, const uint64_t* __restrict__ prevpos,
                           uint64_t* __restrict__ sizes) {
  uint64_t nw = (n + 31) / 32;
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t t = trans_mask(bm, w, n);
    uint64_t prev = prevpos[w], bytes = 0;
    while (t) {
      uint64_t p = w * 32 + (__ffs(t) - 1);
      t &= t - 1;
      bytes += varint_len(p - prev);
      prev = p;
    }
    sizes[w] = bytes;
  }
}
// state[0] = last transition (max-scan grand), state[1] = bytes of runs that
// end at a transition (sum-scan grand); writes the blob and its length.
__global__ void k_vb_write(const uint8_t* __restrict__ bm, uint64_t n, const uint64_t* __restrict__ prevpos,
                           const uint64_t* __restrict__ offs, const uint64_t* __restrict__ state,
                           uint8_t* __restrict__ out, uint64_t* __restrict__ blob_len) {
  uint64_t nw = (n + 31) / 32, raw_len = (n + 7) / 8;
  uint64_t t_last = state[0];
  uint64_t rle_len = state[1] + varint_len(n - t_last);
  bool rle = rle_len < raw_len;
  uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, gsz = (uint64_t)gridDim.x * blockDim.x;
  if (gtid == 0) {
    out[0] = rle ? 1 : 0;
    *blob_len = 1 + (rle ? rle_len : raw_len);
  }
  if (rle) {
    for (uint64_t w = gtid; w < nw; w += gsz) {
      uint32_t t = trans_mask(bm, w, n);
      uint64_t prev = prevpos[w], pos = 1 + offs[w];
      while (t) {
        uint64_t p = w * 32 + (__ffs(t) - 1);
        t &= t - 1;
        uint64_t v = p - prev;
        do {
          uint8_t b = (uint8_t)(v & 0x7f);
          v >>= 7;
          out[pos++] = v ? (b | 0x80) : b;
        } while (v);
        prev = p;
      }
    }
    if (gtid == 0) {
      uint64_t v = n - t_last, pos = 1 + state[1];
      do {
        uint8_t b = (uint8_t)(v & 0x7f);
        v >>= 7;
        out[pos++] = v ? (b | 0x80) : b;
      } while (v);
    }
  } else {
    for (uint64_t i = gtid; i < raw_len; i += gsz) out[1 + i] = bm[i];
  }
}

// Number of bit transitions of the bitmap (added to *count).  The RLE blob
// holds one LEB128 run length per transition plus the final run, each at least
// a byte, so transitions + 1 >= ceil(n/8) proves the RAW blob is chosen.
__global__ void k_bitmap_transitions(const uint8_t* __restrict__ bm, uint64_t n, unsigned long long* count) {
  uint64_t nw = (n + 31) / 32;
  uint32_t c = 0;
  for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += (uint64_t)gridDim.x * blockDim.x)
    c += __popc(trans_mask(bm, w, n));
  c = warp_sum(c);
  __shared__ uint32_t part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += part[k];
    if (t) atomicAdd(count, t);
  }
}
// A short column's bitmap (at most kSmallWords 32-bit words, or such a stretch
// of a longer one from word w0 on) in one CTA of
// 1,024 threads: every word's exclusive valid rank, the valid count (returned)
// and the 0/1 transition count (optional) -- k_word_popcount, the rank scan and
// k_bitmap_transitions in one launch, since short columns pay per launch.
struct SmallWords {
  uint32_t w[kSmallPer];   // the thread's consecutive words
  uint32_t tm[kSmallPer];  // their transition masks (trans_mask)
  uint32_t first, per;     // the first of them, words a thread
};
__device__ inline uint32_t small_end(uint64_t n, uint32_t w0) {
  return (uint32_t)qmin((n + 31) / 32, (uint64_t)w0 + kSmallWords);
}
__device__ inline SmallWords small_words(const uint8_t* __restrict__ bm, uint64_t n, uint32_t w0 = 0) {
  SmallWords s;
  const uint32_t nw = small_end(n, w0);
  s.per = (nw - w0 + 1023) / 1024;
  s.first = w0 + threadIdx.x * s.per;
  uint32_t prev = s.first && s.first <= nw ? bm_word_at(bm, s.first - 1, n) >> 31 : 0u;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) s.w[k] = k < s.per && s.first + k < nw ? bm_word_at(bm, s.first + k, n) : 0u;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    s.tm[k] = 0;
    if (k < s.per && s.first + k < nw) {
      uint32_t t = s.w[k] ^ ((s.w[k] << 1) | prev);
      const uint64_t rem = n - 32ull * (s.first + k);
      if (rem < 32) t &= (1u << rem) - 1u;
      s.tm[k] = t;
    }
    prev = s.w[k] >> 31;
  }
  return s;
}
// Ranks (from rank0 on), the valid count with rank0 (returned) and the number
// of transitions.
__device__ uint64_t valid_small(const SmallWords& S, uint64_t n, uint64_t* __restrict__ rank, uint32_t* trans,
                                uint32_t w0 = 0, uint64_t rank0 = 0) {
  __shared__ uint64_t wsum[32];
  __shared__ uint32_t wtr[32], s_tr;
  uint32_t nw = small_end(n, w0), t = threadIdx.x, l = t & 31, warp = t >> 5;
  uint32_t s = 0, tr = 0;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    s += __popc(S.w[k]);
    tr += __popc(S.tm[k]);
  }
  const uint64_t inc = warp_incl_scan(s);
  tr = __reduce_add_sync(0xffffffffu, tr);
  if (l == 31) wsum[warp] = inc;
  if (l == 0) wtr[warp] = tr;
  __syncthreads();
  if (warp == 0) {
    wsum[l] = warp_incl_scan(wsum[l]);  // inclusive over warps
    uint32_t y = __reduce_add_sync(0xffffffffu, wtr[l]);
    if (l == 0) s_tr = y;
  }
  __syncthreads();
  uint64_t run = rank0 + (warp ? wsum[warp - 1] : 0ull) + inc - s;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    if (k < S.per && S.first + k < nw) rank[S.first + k] = run;
    run += __popc(S.w[k]);
  }
  *trans = s_tr;
  return rank0 + wsum[31];
}
__global__ void __launch_bounds__(1024) k_valid_small(const uint8_t* __restrict__ bm, uint64_t n,
                                                      uint64_t* __restrict__ rank, uint64_t* __restrict__ total,
                                                      unsigned long long* __restrict__ trans) {
  uint32_t tr;
  const uint64_t nv = valid_small(small_words(bm, n), n, rank, &tr);
  if (threadIdx.x == 0) {
    *total = nv;
    *trans = tr;
  }
}

void launch_valid_small(const uint8_t* bm, uint64_t n, uint64_t* rank, uint64_t* total, unsigned long long* trans,
                        cudaStream_t st) {
  k_valid_small<<<1, 1024, 0, st>>>(bm, n, rank, total, trans);
  count_launches(1);
}

// Bits [bit_off, bit_off + n) of a validity bitmap (LSB first) re-packed from
// bit 0, trailing bits of the last byte cleared (the Arrow slice re-pack of
// arrow.rs:29-52, on the device).  The source holds ceil((bit_off + n) / 8)
// bytes; nothing past them is read.
__global__ void k_bitmap_repack(const uint8_t* __restrict__ src, uint64_t bit_off, uint64_t n,
                                uint8_t* __restrict__ dst) {
  uint64_t nb = (n + 7) / 8, src_bytes = (bit_off + n + 7) / 8;
  uint32_t sh = (uint32_t)(bit_off & 7);
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nb; i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t s0 = (bit_off >> 3) + i;
    uint32_t v = src[s0] >> sh;
    if (sh && s0 + 1 < src_bytes) v |= (uint32_t)src[s0 + 1] << (8 - sh);
    if (i == nb - 1 && (n & 7)) v &= (1u << (n & 7)) - 1u;
    dst[i] = (uint8_t)v;
  }
}

void launch_bitmap_repack(const uint8_t* src, uint64_t bit_off, uint64_t n, uint8_t* dst, cudaStream_t st) {
  uint64_t nb = (n + 7) / 8;
  if (!nb) return;
  unsigned g = (unsigned)((nb + 255) / 256 < 4096 ? (nb + 255) / 256 : 4096);
  k_bitmap_repack<<<g, 256, 0, st>>>(src, bit_off, n, dst);
  count_launches(1);
}

void launch_bitmap_transitions(const uint8_t* bm, uint64_t n, unsigned long long* count, cudaStream_t st) {
  uint64_t nw = (n + 31) / 32;
  unsigned g = (unsigned)qmin((nw + 255) / 256, 148ull * 8);
  if (g == 0) g = 1;
  k_bitmap_transitions<<<g, 256, 0, st>>>(bm, n, count);
  count_launches(1);
}

// The RAW validity blob straight into the stream: varint(1 + ceil(n/8)), tag
// 0, the bitmap bytes (validity.rs:40-70); *d_base = the stream offset after it.
__global__ void k_put_validity_raw(uint8_t* dst, uint64_t dst_off, const uint8_t* __restrict__ bm, uint64_t raw_len,
                                   uint64_t* d_base) {
  uint64_t len = 1 + raw_len;
  uint32_t vl = varint_len(len);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    uint64_t v = len;
    uint32_t k = 0;
    do {
      uint8_t b = (uint8_t)(v & 0x7f);
      v >>= 7;
      dst[k++] = v ? (b | 0x80) : b;
    } while (v);
    dst[vl] = 0;
    *d_base = dst_off + vl + len;
  }
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < raw_len; i += (uint64_t)gridDim.x * blockDim.x)
    dst[vl + 1 + i] = bm[i];
}
void launch_put_validity_raw(uint8_t* dst, uint64_t dst_off, const uint8_t* bm, uint64_t n, uint64_t* d_base,
                             cudaStream_t st) {
  k_put_validity_raw<<<148 * 4, 256, 0, st>>>(dst, dst_off, bm, (n + 7) / 8, d_base);
  count_launches(1);
}

uint64_t validity_tmp_words(uint64_t n) {
  uint64_t nw = (n + 31) / 32;
  return 3 * nw + scan_tiles(nw) + 8;
}

// The validity blob of a short column in one CTA of 1,024 threads: the three
// passes above (last transitions + max scan, run bytes + sum scan, write) with
// block scans in place of the grid scans.  place(blob length) gives the blob's
// destination.  A longer bitmap goes stretch by stretch, first for the blob's
// size and then to write it.
struct VbRuns {
  uint64_t last, bytes;  // the last transition so far and the bytes of the runs that end at one
};
// This stretch's runs: in *r the totals, *prev and the result are the last
// transition and the run bytes before this thread's words.
__device__ uint64_t vb_scan(const SmallWords& S, VbRuns* r, uint64_t* prev0) {
  __shared__ uint64_t wa[32], wb[32];
  uint32_t t = threadIdx.x, l = t & 31, warp = t >> 5;
  uint64_t mx = 0;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    uint32_t w = S.first + k;
    if (S.tm[k]) mx = (uint64_t)w * 32 + (31 - __clz(S.tm[k]));  // words ascend: the thread's last transition
  }
  // exclusive max scan of the threads' last transitions (positions ascend, 0 = none yet)
  uint64_t inc = mx;
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if ((int)l >= o) inc = u > inc ? u : inc;
  }
  uint64_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
  if (l == 0) ex = 0;
  if (l == 31) wa[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint64_t x = wa[l];
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t u = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)l >= o) x = u > x ? u : x;
    }
    wa[l] = x;
  }
  __syncthreads();
  const uint64_t before = warp ? wa[warp - 1] : 0ull;
  *prev0 = qmax(r->last, qmax(ex, before));
  r->last = qmax(r->last, wa[31]);
  // bytes of the runs that end at this thread's transitions, then their offsets
  uint64_t prev = *prev0, s = 0;
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    uint32_t tt = S.tm[k];
    uint32_t w = S.first + k;
    while (tt) {
      uint64_t p = (uint64_t)w * 32 + (__ffs(tt) - 1);
      tt &= tt - 1;
      s += varint_len(p - prev);
      prev = p;
    }
  }
  const uint64_t inc2 = warp_incl_scan(s);
  if (l == 31) wb[warp] = inc2;
  __syncthreads();
  if (warp == 0) wb[l] = warp_incl_scan(wb[l]);
  __syncthreads();
  const uint64_t at = r->bytes + (warp ? wb[warp - 1] : 0ull) + inc2 - s;
  r->bytes += wb[31];
  return at;
}
__device__ inline uint64_t vb_leb(uint8_t* out, uint64_t pos, uint64_t v) {
  do {
    uint8_t b = (uint8_t)(v & 0x7f);
    v >>= 7;
    out[pos++] = v ? (b | 0x80) : b;
  } while (v);
  return pos;
}
__device__ inline void vb_put(const SmallWords& S, uint64_t prev, uint64_t pos, uint8_t* out) {
#pragma unroll
  for (uint32_t k = 0; k < kSmallPer; k++) {
    uint32_t tt = S.tm[k];
    uint32_t w = S.first + k;
    while (tt) {
      uint64_t p = (uint64_t)w * 32 + (__ffs(tt) - 1);
      tt &= tt - 1;
      pos = vb_leb(out, pos, p - prev);
      prev = p;
    }
  }
}
__device__ inline void vb_raw(const uint8_t* __restrict__ bm, uint64_t n, uint8_t* out) {
  if (threadIdx.x == 0) out[0] = 0;
#pragma unroll 4
  for (uint64_t i = threadIdx.x; i < (n + 7) / 8; i += 1024) out[1 + i] = bm[i];
}
template <class P>
__device__ void vb_small(const SmallWords& S, const uint8_t* __restrict__ bm, uint64_t n, bool raw, P place) {
  const uint64_t raw_len = (n + 7) / 8;
  if (raw) {  // proven by the transitions
    vb_raw(bm, n, place(1 + raw_len));
    return;
  }
  VbRuns r = {0, 0};
  uint64_t prev;
  uint64_t at = vb_scan(S, &r, &prev);
  const uint64_t rle_len = r.bytes + varint_len(n - r.last);
  const bool rle = rle_len < raw_len;
  uint8_t* out = place(1 + (rle ? rle_len : raw_len));
  if (!rle) {
    vb_raw(bm, n, out);
    return;
  }
  if (threadIdx.x == 0) {
    out[0] = 1;
    vb_leb(out, 1 + r.bytes, n - r.last);
  }
  vb_put(S, prev, 1 + at, out);
}
template <class P>
__device__ void vb_long(const uint8_t* __restrict__ bm, uint64_t n, bool raw, P place) {
  const uint32_t nw = (uint32_t)((n + 31) / 32);
  const uint64_t raw_len = (n + 7) / 8;
  VbRuns r = {0, 0};
  uint64_t prev;
  for (uint32_t w0 = 0; !raw && w0 < nw; w0 += kSmallWords) {
    vb_scan(small_words(bm, n, w0), &r, &prev);
    __syncthreads();
  }
  const uint64_t rle_len = r.bytes + varint_len(n - r.last);
  const bool rle = !raw && rle_len < raw_len;
  uint8_t* out = place(1 + (rle ? rle_len : raw_len));
  if (!rle) {
    vb_raw(bm, n, out);
    return;
  }
  if (threadIdx.x == 0) {
    out[0] = 1;
    vb_leb(out, 1 + r.bytes, n - r.last);
  }
  r = {0, 0};
  for (uint32_t w0 = 0; w0 < nw; w0 += kSmallWords) {
    const SmallWords S = small_words(bm, n, w0);
    const uint64_t at = vb_scan(S, &r, &prev);
    vb_put(S, prev, 1 + at, out);
    __syncthreads();
  }
}
__global__ void __launch_bounds__(1024) k_vb_small(const uint8_t* __restrict__ bm, uint64_t n,
                                                   uint8_t* __restrict__ out, uint64_t* __restrict__ blob_len) {
  vb_small(small_words(bm, n), bm, n, false, [&](uint64_t len) {
    if (threadIdx.x == 0) *blob_len = len;
    return out;
  });
}
// A short nullable column's stream up to its first frame, without the host: a
// call that waited for the valid count before it could go on paid 25 us of the
// 96 that a 65,537-value page took; with this kernel and the one-warp plan the
// page takes 72.
__global__ void __launch_bounds__(1024) k_begin_small(const uint8_t* __restrict__ bm, uint64_t n,
                                                      uint64_t* __restrict__ rank, uint64_t* __restrict__ total,
                                                      uint8_t* dst, Bytes16 hdr, uint64_t* __restrict__ d_base) {
  const SmallWords S = small_words(bm, n);
  uint32_t trans;
  const uint64_t nv = valid_small(S, n, rank, &trans);
  const int t = threadIdx.x;
  if (t < 16) dst[t] = t == 5 ? (nv < n ? 1 : 0) : hdr.b[t];
  if (t == 0) {
    *total = nv;
    if (nv == n) *d_base = 16;
  }
  if (nv == n) return;  // all valid: no bitmap in the stream
  vb_small(S, bm, n, trans + 1ull >= (n + 7) / 8, [&](uint64_t len) {
    const uint32_t vl = varint_len(len);
    if (t == 0) {
      uint64_t v = len;
      for (uint32_t k = 0; k < vl; k++, v >>= 7) dst[16 + k] = (uint8_t)((v & 0x7f) | (k + 1 < vl ? 0x80u : 0u));
      *d_base = 16 + vl + len;
    }
    return dst + 16 + vl;
  });
}
void launch_begin_small(const uint8_t* bm, uint64_t n, uint64_t* rank, uint64_t* total, uint8_t* dst, Bytes16 hdr,
                        uint64_t* d_base, cudaStream_t st) {
  k_begin_small<<<1, 1024, 0, st>>>(bm, n, rank, total, dst, hdr, d_base);
  count_launches(1);
}

// ---------------------------------------------------------------------------
// A group of columns of one batch call (EncCol): what the kernels above do for
// a column, for all of them in one launch each.  One column's launches of 2-8 us
// and its wait for the valid count were most of what a short column cost.
// ---------------------------------------------------------------------------
// CTAs a column: 192 columns of up to 1,048,576 values take 1,282 us with 32
// (a long column's lowering then is 128 dependent steps), 1,211 with 64 and
// 1,207 with 128 (more CTAs that find nothing to do).
constexpr int kColParts = 64;
__global__ void __launch_bounds__(256) k_cols_vmin(const EncCol* __restrict__ cols) {
  const EncCol& C = cols[blockIdx.y];
  const uint64_t* v = reinterpret_cast<const uint64_t*>(C.values);
  if (C.nl == 2) vmin_partial<2>(v, C.bm, C.n, C.parts);
  else if (C.nl == 4) vmin_partial<4>(v, C.bm, C.n, C.parts);
}
__global__ void __launch_bounds__(1024) k_cols_begin(const EncCol* __restrict__ cols) {
  const EncCol& C = cols[blockIdx.x];
  const int t = threadIdx.x, nl = C.nl;
  const uint64_t n = C.n;
  const uint32_t nw = (uint32_t)((n + 31) / 32);
  uint64_t nv = n, trans = 0;
  for (uint32_t w0 = 0; C.bm && w0 < nw; w0 += kSmallWords) {
    uint32_t tr;
    if (w0 == 0) nv = 0;
    nv = valid_small(small_words(C.bm, n, w0), n, C.rank, &tr, w0, nv);
    trans += tr;
    __syncthreads();
  }
  const uint64_t head = nl ? 19 + 8ull * nl : 16;
  uint8_t* dst = C.dst;
  if (t < (nl ? 19 : 16)) dst[t] = t == 5 ? C.hdr[5] | (nv < n ? 1 : 0) : C.hdr[t];
  if (nl) {
    if (nl == 2) vmin_final<2>(C.parts, kColParts, nv != 0, C.vmin);
    else vmin_final<4>(C.parts, kColParts, nv != 0, C.vmin);
    __syncthreads();
    if (t < 8 * nl) dst[19 + t] = (uint8_t)(C.vmin[t >> 3] >> (8 * (t & 7)));
  }
  if (t == 0) {
    C.res[0] = head;
    C.res[1] = 0;
    C.res[2] = nv;
  }
  if (nv == n) return;  // all valid: no bitmap in the stream
  auto place = [&](uint64_t len) {
    const uint32_t vl = varint_len(len);
    if (t == 0) {
      vb_leb(dst, head, len);
      C.res[0] = head + vl + len;
    }
    return dst + head + vl;
  };
  const bool raw = trans + 1 >= (n + 7) / 8;
  if (nw <= kSmallWords) vb_small(small_words(C.bm, n), C.bm, n, raw, place);
  else vb_long(C.bm, n, raw, place);
}
__global__ void __launch_bounds__(256) k_cols_lower(const EncCol* __restrict__ cols) {
  const EncCol& C = cols[blockIdx.y];
  if (C.nl) split_words(C.values, C.nl, C.bm, C.rank, C.n, C.vmin, C.lane, C.stride);
  else if (C.lane) lower_words(C.values, C.dtype, C.bm, C.rank, C.n, C.lane);
}
uint64_t enc_col_part_words() { return 4ull * kColParts; }
void launch_begin_cols(const EncCol* cols, int ncols, bool decimals, cudaStream_t st) {
  if (decimals) k_cols_vmin<<<dim3(kColParts, ncols), 256, 0, st>>>(cols);
  k_cols_begin<<<ncols, 1024, 0, st>>>(cols);
  k_cols_lower<<<dim3(kColParts, ncols), 256, 0, st>>>(cols);
  count_launches(decimals ? 3 : 2);
}

void launch_validity_blob(const uint8_t* bm, uint64_t n, uint64_t* tmp, uint64_t* tile_tmp, uint8_t* out,
                          uint64_t* blob_len, cudaStream_t st) {
  uint64_t nw = (n + 31) / 32;
  if (nw <= kSmallWords) {
    k_vb_small<<<1, 1024, 0, st>>>(bm, n, out, blob_len);
    count_launches(1);
    return;
  }
  uint64_t* last = tmp;
  uint64_t* sizes = tmp + nw;
  uint64_t* state = tmp + 2 * nw;  // [0] t_last, [1] bytes
  unsigned g = (unsigned)qmin((nw + 255) / 256, 148ull * 16);
  if (g == 0) g = 1;
  k_vb_last<<<g, 256, 0, st>>>(bm, n, last);
  scan_exclusive<ScanMax>(last, last, nw, tile_tmp, state, st);
  k_vb_sizes<<<g, 256, 0, st>>>(bm, n, last, sizes);
  scan_exclusive<ScanSum>(sizes, sizes, nw, tile_tmp, state + 1, st);
  k_vb_write<<<g, 256, 0, st>>>(bm, n, last, sizes, state, out, blob_len);
  count_launches(3 + 2 * scan_launches(nw));
}

void launch_scan_sum(const uint64_t* in, uint64_t* out, uint64_t n, uint64_t* tile_tmp, uint64_t* grand,
                     cudaStream_t st) {
  scan_exclusive<ScanSum>(in, out, n ? n : 1, tile_tmp, grand, st);
  count_launches(scan_launches(n));
}

void launch_write_bytes(uint8_t* dst, const uint8_t* src_dev, uint64_t len, cudaStream_t st) {
  if (len) cudaMemcpyAsync(dst, src_dev, len, cudaMemcpyDeviceToDevice, st);
}

__global__ void k_put_header(uint8_t* dst, Bytes16 hdr, uint64_t* d_base) {
  if (threadIdx.x < 16) dst[threadIdx.x] = hdr.b[threadIdx.x];
  if (threadIdx.x == 0 && d_base) *d_base = 16;
}
void launch_put_header(uint8_t* dst, Bytes16 hdr, uint64_t* d_base, cudaStream_t st) {
  k_put_header<<<1, 32, 0, st>>>(dst, hdr, d_base);
  count_launches(1);
}

__global__ void k_put_validity(uint8_t* dst, uint64_t dst_off, const uint8_t* __restrict__ blob,
                               const uint64_t* __restrict__ blob_len, uint64_t* d_base) {
  uint64_t len = *blob_len;
  uint32_t vl = varint_len(len);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    uint64_t v = len;
    uint32_t k = 0;
    do {
      uint8_t b = (uint8_t)(v & 0x7f);
      v >>= 7;
      dst[k++] = v ? (b | 0x80) : b;
    } while (v);
    *d_base = dst_off + vl + len;
  }
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x)
    dst[vl + i] = blob[i];
}
void launch_put_validity(uint8_t* dst, uint64_t dst_off, const uint8_t* blob, const uint64_t* blob_len,
                         uint64_t* d_base, cudaStream_t st) {
  k_put_validity<<<148 * 4, 256, 0, st>>>(dst, dst_off, blob, blob_len, d_base);
  count_launches(1);
}

}  // namespace qb
