// K1 per-peak search of one (tile, hypothesis) work item, shared by the staged K1 kernel and the fused search.
//
// The tile's postings and its coarse-bin CSR are in shared memory.  A fragment's key is f32bits(f) - f32bits(fmin)
// (mass_bits wide); its coarse bin is the top cbin_bits of the key, and the posting holds the remaining low key bits
// and the local row: (key mod 2^(mass_bits - cbin_bits)) << row_bits | row, sorted within each bin, the bin given
// by the posting's position (cbin_off).  Lanes stride over the spectrum's peaks x fragment charges: the tolerance
// window [a, bd] of peak mass p*z (Sage f32 bounds) is the key range [bits(a)-base, bits(bd)-base] (clamped to the
// fragment range); in each coarse bin it touches (one, or two at a bin edge) a binary search finds its first
// posting, and every posting in range whose row lies in [rlo, rhi) adds one to cnt[hoff + row].  Exactly the
// reference's brute-force count (kernels.cu:195-232).
#pragma once
#include "common.cuh"

namespace vk {

constexpr int K1_BM_LOG = 6;                         // log2 of the presence-bitmap bits per coarse bin
constexpr int K1_BM_WORDS = (1 << K1_BM_LOG) / 32;   // u32 words of a coarse bin's bitmap

// cnt[hoff + l] is the count of tile row l (rows rlo <= l < rhi only).  With isum != nullptr, every match also adds
// the peak's weight round(intensity * wscale) (u32, wscale = 2^24 / TIC of the spectrum) to isum[hoff + l]: the
// summed matched intensity as a fixed-point fraction of the TIC, accumulated with integer atomics (deterministic).
__device__ __forceinline__ void k1_item_per_peak(const uint32_t* post, const uint16_t* cb, uint32_t* cnt, int64_t hoff,
                                                 int rlo, int rhi,
                                                 int64_t p0, int64_t p1, int maxfz, const float* pk_mass,
                                                 float tol_lo, float tol_hi, int tol_da, const vk_tindex& ix,
                                                 int lane, uint32_t* isum = nullptr, const float* pk_int = nullptr,
                                                 float wscale = 0.f) {
  const int row_bits = ix.row_bits;
  const uint32_t rowmask = (1u << row_bits) - 1u;
  const int low_bits = ix.mass_bits - ix.cbin_bits;
  const uint32_t lowmask = (1u << low_bits) - 1u;
  const float fmin = __uint_as_float(ix.fmin_bits), fmax = __uint_as_float(ix.fmax_bits);
  const uint32_t krange = ix.fmax_bits - ix.fmin_bits;
  for (int64_t p = p0 + lane; p < p1; p += 32) {
    const float pm = pk_mass[p];
    const uint32_t wgt = isum ? __float2uint_rn(__fmul_rn(pk_int[p], wscale)) : 0u;
    for (int z = 1; z < maxfz; ++z) {
      const float m = __fmul_rn(pm, (float)z);
      const float a = vk::tol_bound(m, tol_lo, tol_da), bd = vk::tol_bound(m, tol_hi, tol_da);
      if (!(bd >= fmin && a <= fmax)) continue;
      const uint32_t ka = a <= fmin ? 0u : __float_as_uint(a) - ix.fmin_bits;
      const uint32_t kb = bd >= fmax ? krange : __float_as_uint(bd) - ix.fmin_bits;
      const uint32_t ba = ka >> low_bits, bb = kb >> low_bits;
      for (uint32_t bin = ba; bin <= bb; ++bin) {
        const uint32_t lo_key = bin == ba ? (ka & lowmask) << row_bits : 0u;
        const uint32_t hi_key = bin == bb ? ((kb & lowmask) << row_bits) | rowmask : 0xffffffffu;
        int e = cb[bin];
        const int e1 = cb[bin + 1];
        int R = e1;
        while (e < R) {
          const int M = (e + R) >> 1;
          if (post[M] < lo_key) e = M + 1; else R = M;
        }
        for (; e < e1; ++e) {
          const uint32_t v = post[e];
          if (v > hi_key) break;
          const int l = (int)(v & rowmask);
          if (l >= rlo && l < rhi) {
            atomicAdd(&cnt[hoff + l], 1u);
            if (isum) atomicAdd(&isum[hoff + l], wgt);
          }
        }
      }
    }
  }
}

// ---- filtered per-item search (staged K1) ----
//
// The tolerance window of a peak does not depend on the tile, so its key range is computed once per pass
// (k1_window_keys, by vk_k1_peak_keys) instead of once per (tile, hypothesis) item, together with a 32-bit filter
// word (k1_filter_word).  Every tile has a presence bitmap, built with the index (vk_tindex_bitmap) and staged with
// the tile: 2^K1_BM_LOG bits per coarse bin, bit s of bin b set when a posting of the bin has (low key) >>
// (low_bits - K1_BM_LOG) == s.  A window whose bits are all clear holds no posting and is dropped after one
// shared-memory word; the windows that may match are compacted into a per-warp queue (ballot) and searched
// exactly, one per lane, so the bin lookup and binary search run with every lane busy and only for them.  The
// counts are those of k1_item_per_peak: the bitmap only skips windows that hold no posting.

// Key range [ka, kb] of the tolerance window of fragment mass pm * z (Sage f32 bounds, both edges included), clamped
// to the index's fragment range; ka > kb when the window misses the range.
__device__ __forceinline__ uint2 k1_window_keys(float pm, int z, float tol_lo, float tol_hi, int tol_da,
                                                const vk_tindex& ix) {
  const float fmin = __uint_as_float(ix.fmin_bits), fmax = __uint_as_float(ix.fmax_bits);
  const float m = __fmul_rn(pm, (float)z);
  const float a = vk::tol_bound(m, tol_lo, tol_da), bd = vk::tol_bound(m, tol_hi, tol_da);
  if (!(bd >= fmin && a <= fmax)) return make_uint2(1u, 0u);
  const uint32_t ka = a <= fmin ? 0u : __float_as_uint(a) - ix.fmin_bits;
  const uint32_t kb = bd >= fmax ? ix.fmax_bits - ix.fmin_bits : __float_as_uint(bd) - ix.fmin_bits;
  return make_uint2(ka, kb);
}

// Bits per coarse bin actually used: 2^min(K1_BM_LOG, low_bits); a posting's bit is its top bits (row_bits +
// low_bits = 32).
__device__ __forceinline__ int k1_bm_bits(const vk_tindex& ix) {
  const int low_bits = ix.mass_bits - ix.cbin_bits;
  return low_bits < K1_BM_LOG ? low_bits : K1_BM_LOG;
}

// Bitmap position of key k: bin * 2^K1_BM_LOG + (low key >> (low_bits - bits)); monotone in k, below
// 2^(cbin_bits + K1_BM_LOG).
__device__ __forceinline__ uint32_t k1_bm_pos(uint32_t k, int low_bits, int bshift) {
  return ((k >> low_bits) << K1_BM_LOG) | ((k & ((1u << low_bits) - 1u)) >> bshift);
}

// One thread per coarse bin builds the bin's 64 bits in a register (the index build calls this per tile).
__device__ __forceinline__ void k1_build_bitmap(const uint32_t* post, const uint16_t* cb, int nb, int bits,
                                                uint32_t* bm) {
  const int top = 32 - bits;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    unsigned long long v = 0ull;
    const int e1 = cb[b + 1];
    for (int e = cb[b]; e < e1; ++e) v |= 1ull << (post[e] >> top);
    uint32_t* w = bm + (size_t)b * K1_BM_WORDS;
    w[0] = (uint32_t)v;
    w[1] = (uint32_t)(v >> 32);
  }
}

// Filter word of window [ka, kb]: the bitmap position of ka in bits 0..19 and the span to kb's position in bits
// 20..31, capped at 4095 (such wide windows always go to the exact search); K1_NO_WINDOW when ka > kb.
constexpr uint32_t K1_NO_WINDOW = 0xffffffffu;
__device__ __forceinline__ uint32_t k1_filter_word(uint2 k, const vk_tindex& ix) {
  if (k.x > k.y) return K1_NO_WINDOW;
  const int low_bits = ix.mass_bits - ix.cbin_bits;
  const int bshift = low_bits - k1_bm_bits(ix);
  const uint32_t ga = k1_bm_pos(k.x, low_bits, bshift), gb = k1_bm_pos(k.y, low_bits, bshift);
  return ga | (min(gb - ga, 4095u) << 20);
}

// true when the window of filter word f may hold a posting of the tile with bitmap bm (bm_mask + 1 words, a power of
// two, and one readable word behind them).  Branch-free: the window's bits lie in two neighbouring words, whichever
// side of a word edge they start on (a tenth of the windows straddle one, so some lane of nearly every warp does);
// windows of more than 32 bits go to the exact search.
__device__ __forceinline__ bool k1_filter_pass(const uint32_t* bm, uint32_t bm_mask, uint32_t f) {
  const uint32_t d = f >> 20, w = (f >> 5) & bm_mask;
  const uint32_t v = __funnelshift_r(bm[w], bm[w + 1], f);   // from the window's first bit on
  return f != K1_NO_WINDOW && (d >= 32u || (v & ~(0xfffffffeu << (d & 31u))) != 0u);
}

// Count the postings with key in [ka, kb] whose row lies in [rlo, rlo + rows) (one lane, one window): one lower bound
// in the first coarse bin, then one scan to the end of the last bin, in which a posting above the window ends it.
template <bool ISUM>
__device__ __forceinline__ void k1_count_range(const uint32_t* post, const uint16_t* cb, uint32_t* hw, uint32_t* iw,
                                               int rlo, uint32_t rows, uint32_t ka, uint32_t kb, uint32_t wgt,
                                               int row_bits, int low_bits) {
  const uint32_t rowmask = (1u << row_bits) - 1u, lowmask = (1u << low_bits) - 1u;
  const uint32_t ba = ka >> low_bits, bb = kb >> low_bits;
  const uint32_t lo_key = (ka & lowmask) << row_bits, hi_key = ((kb & lowmask) << row_bits) | rowmask;
  int e = cb[ba], end = cb[ba + 1], last = 0;   // postings from `last` on are in the window's last bin
  for (int span = end - e; span > 0;) {
    const int half = span >> 1;
    if (post[e + half] < lo_key) {
      e += half + 1;
      span -= half + 1;
    } else {
      span = half;
    }
  }
  if (bb != ba) {
    last = cb[bb];
    end = cb[bb + 1];
  }
  for (; e < end; ++e) {
    const uint32_t v = post[e];
    if (v > hi_key && e >= last) break;
    const uint32_t l = v & rowmask;
    if (l - (uint32_t)rlo < rows) {
      atomicAdd(&hw[l], 1u);
      if (ISUM) atomicAdd(&iw[l], wgt);
    }
  }
}

constexpr int K1_AHEAD = 2;    // filter words per lane tested at once, and as many more in flight
constexpr int K1_QUEUE = 32 * (K1_AHEAD + 1);   // u32 entries per warp: (charge - 1) << 16 | peak index

// A warp's next filter words: the first 32 * K1_AHEAD of an item are loaded while the item before it is worked on.
struct K1Words {
  uint32_t f[K1_AHEAD];
  // words [base, base + 32 * K1_AHEAD) of an item of n; src: the item's first word plus the lane
  __device__ __forceinline__ void load(const uint32_t* __restrict__ src, int n, int base, int lane) {
#pragma unroll
    for (int u = 0; u < K1_AHEAD; ++u) f[u] = base + 32 * u + lane < n ? __ldg(src + base + 32 * u) : K1_NO_WINDOW;
  }
};

// One (tile, hypothesis) item by one warp.  For fragment charges z <= n_kz, keys[(z - 1) * kstride + p] holds the
// window keys of peak p and filt[...] its filter word; higher charges are computed here.  q: this warp's queue.
// words: the item's first charge-1 filter words (n_kz >= 1); on return the next item's (next_n peaks from next_p0).
template <bool ISUM>
__device__ __forceinline__ void k1_item_filtered(const uint32_t* post, const uint16_t* cb, const uint32_t* bm,
                                                 uint32_t bm_mask, uint32_t* hw, uint32_t* iw, int rlo, int rhi,
                                                 int64_t p0, int n, int maxfz, const uint2* __restrict__ keys,
                                                 const uint32_t* __restrict__ filt, int n_kz, int64_t kstride,
                                                 const float* __restrict__ pk_mass, float tol_lo, float tol_hi,
                                                 int tol_da, const vk_tindex& ix, int lane, uint32_t* q,
                                                 const float* __restrict__ pk_int, float wscale, K1Words& words,
                                                 int64_t next_p0, int next_n) {
  const int row_bits = ix.row_bits, low_bits = ix.mass_bits - ix.cbin_bits;
  const unsigned lt = (1u << lane) - 1u;
  int nq = 0;
  auto search = [&](uint32_t e) {
    const int zi = (int)(e >> 16);
    const int64_t p = p0 + (e & 0xffffu);
    const uint2 k = zi < n_kz ? __ldg(keys + (int64_t)zi * kstride + p)
                              : k1_window_keys(pk_mass[p], zi + 1, tol_lo, tol_hi, tol_da, ix);
    const uint32_t wgt = ISUM ? __float2uint_rn(__fmul_rn(__ldg(pk_int + p), wscale)) : 0u;
    k1_count_range<ISUM>(post, cb, hw, iw, rlo, (uint32_t)(rhi - rlo), k.x, k.y, wgt, row_bits, low_bits);
  };
  auto test = [&](const K1Words& w, uint32_t tag) {   // tag: charge and this lane's first peak
#pragma unroll
    for (int u = 0; u < K1_AHEAD; ++u) {
      const bool pass = k1_filter_pass(bm, bm_mask, w.f[u]);
      const unsigned bal = __ballot_sync(0xffffffffu, pass);
      if (pass) q[nq + __popc(bal & lt)] = tag + 32u * u;
      nq += __popc(bal);
    }
    if (nq >= 32) {   // full rounds of 32 from the end; the rest stays in front
      __syncwarp();
      do {
        nq -= 32;
        search(q[nq + lane]);
      } while (nq >= 32);
      __syncwarp();
    }
  };
  for (int z = 1; z < maxfz; ++z) {
    const uint32_t zt = ((uint32_t)(z - 1) << 16) + (uint32_t)lane;
    K1Words cur;
    if (z <= n_kz) {
      const uint32_t* __restrict__ src = filt + (int64_t)(z - 1) * kstride + p0 + lane;
      if (z == 1) cur = words; else cur.load(src, n, 0, lane);
      for (int base = 0; base < n; base += 32 * K1_AHEAD) {
        K1Words nx;
        nx.load(src, n, base + 32 * K1_AHEAD, lane);
        test(cur, zt + base);
        cur = nx;
      }
    } else {
      for (int base = 0; base < n; base += 32 * K1_AHEAD) {
#pragma unroll
        for (int u = 0; u < K1_AHEAD; ++u) {
          const int i = base + 32 * u + lane;
          cur.f[u] = i < n ? k1_filter_word(k1_window_keys(pk_mass[p0 + i], z, tol_lo, tol_hi, tol_da, ix), ix)
                           : K1_NO_WINDOW;
        }
        test(cur, zt + base);
      }
    }
  }
  if (n_kz > 0) words.load(filt + next_p0 + lane, next_n, 0, lane);
  __syncwarp();
  if (lane < nq) search(q[lane]);
}


}  // namespace vk
