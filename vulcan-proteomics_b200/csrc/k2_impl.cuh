// K2 exact rescoring body (Sage score_candidate semantics, reference vulcan/gpu/kernels.cu:240-376).
//
// Three launch shapes, with the same per-candidate arithmetic (the f32 sums are sequential in ion order: b ions k
// ascending, fragment charge ascending, then y ions), which is the reference's operation for operation, so the
// outputs are bit-identical: a CTA per spectrum for the closed scoring of dense lists (k2_dense_body), a warp per
// spectrum for the shifted scoring (k2_body), a thread per candidate for sparse lists (k2_cands_k).  The first two
// stage the spectrum's first 512 mass-sorted peaks in shared memory with a bucket table of start indices (one lookup
// and a short walk replace the reference's binary search; same index found).
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace vk {

constexpr int K2_WARPS = 8;

struct K2Out {
  double* hs;
  float* sb;
  float* sy;
  float* ppm;
  int16_t* mb;
  int16_t* my;
  int16_t* lb;
  int16_t* ly;
};

struct RunLen {
  int start, length, last, longest;
};

// Longest run of consecutive matched ion indices (kernels.cu:252-258)
__device__ __forceinline__ void run_matched(RunLen& r, int idx) {
  if (r.last == idx) return;
  if (r.start + r.length == idx) {
    r.length += 1;
  } else {
    r.start = idx;
    r.length = 1;
  }
  r.longest = max(r.longest, r.length);
  r.last = idx;
}

__device__ __forceinline__ int lower_bound_smem(const float* v, int n, float x) {
  int lo = 0, hi = n;
  while (lo < hi) {
    int m = (lo + hi) >> 1;
    if (v[m] < x) lo = m + 1; else hi = m;
  }
  return lo;
}

// Bucket table of a spectrum's sorted peak masses: start[b] = first peak j with bucket(sm[j]) >= b, where
// bucket(x) = clamp((int)((x - m0) * inv_w), 0, K2_BUCKETS - 1) is monotone in x.  For a bound a with bucket b,
// every peak >= a has bucket >= b, so the first peak >= a is found by starting at start[b] and stepping while
// sm[j] < a: the same index the binary search returns, in one lookup and a short walk.
constexpr int K2_BUCKETS = 512;

__device__ __forceinline__ int k2_bucket(float x, float m0, float inv_w) {
  const float t = __fmul_rn(__fsub_rn(x, m0), inv_w);
  return t <= 0.f ? 0 : (t >= (float)(K2_BUCKETS - 1) ? K2_BUCKETS - 1 : (int)t);
}

struct PeakTable {
  const float* sm;
  const float* si;
  const uint16_t* start;
  int np;
  float m0, inv_w;

  __device__ __forceinline__ float mass(int j) const { return sm[j]; }
  __device__ __forceinline__ float inten(int j) const { return si[j]; }
  __device__ __forceinline__ int bucket(float x) const { return k2_bucket(x, m0, inv_w); }
  __device__ __forceinline__ int first_ge(float a) const {
    int j = start[bucket(a)];
    while (j < np && sm[j] < a) ++j;
    return j;
  }
};

// Build the table for the warp's spectrum (peaks already in shared memory).
__device__ __forceinline__ PeakTable build_table(const float* sm, const float* si, uint16_t* start, int np, int lane) {
  PeakTable t;
  t.sm = sm;
  t.si = si;
  t.start = start;
  t.np = np;
  t.m0 = np > 0 ? sm[0] : 0.f;
  float span = np > 0 ? __fsub_rn(sm[np - 1], t.m0) : 0.f;
  t.inv_w = span > 0.f ? __fdiv_rn((float)K2_BUCKETS, span) : 0.f;
  for (int j = lane; j < np; j += 32) {
    int b = t.bucket(sm[j]);
    int bp = j > 0 ? t.bucket(sm[j - 1]) : -1;
    for (int q = bp + 1; q <= b; ++q) start[q] = (uint16_t)j;
  }
  int blast = np > 0 ? t.bucket(sm[np - 1]) : -1;
  for (int q = blast + 1 + lane; q < K2_BUCKETS; q += 32) start[q] = (uint16_t)np;
  __syncwarp();
  return t;
}

// A spectrum's mass-sorted peaks read where they lie (global memory); first_ge is the lower bound by binary search,
// the index the bucket table also finds.  For candidate-parallel scoring of sparse candidate lists.
struct GlobalPeaks {
  const float* sm;
  const float* si;
  int np;

  __device__ __forceinline__ float mass(int j) const { return sm[j]; }
  __device__ __forceinline__ float inten(int j) const { return si[j]; }
  __device__ __forceinline__ int first_ge(float a) const {
    int lo = 0, hi = np;
    while (lo < hi) {
      const int m = (lo + hi) >> 1;
      if (__ldg(sm + m) < a) lo = m + 1; else hi = m;
    }
    return lo;
  }
};

// A candidate's sums, counts and longest runs.
struct K2Val {
  float sb, sy, ppm;
  int mb, my, lb, ly;
};

// Hyperscore and outputs of candidate c; lnf(n) is lnfact(n).
template <class L>
__device__ __forceinline__ void k2_write(const K2Val& v, L&& lnf, const K2Out& out, int64_t c) {
  const double i2 = (double)__fadd_rn(v.sb, 1.0f) * (double)__fadd_rn(v.sy, 1.0f);
  double hs = log(i2) + lnf(v.mb) + lnf(v.my);
  if (!isfinite(hs)) hs = 255.0;
  out.hs[c] = hs;
  out.sb[c] = v.sb;
  out.sy[c] = v.sy;
  out.ppm[c] = __fdiv_rn(v.ppm, __fadd_rn(v.sb, v.sy));
  out.mb[c] = (int16_t)v.mb;
  out.my[c] = (int16_t)v.my;
  out.lb[c] = (int16_t)v.lb;
  out.ly[c] = (int16_t)v.ly;
}

template <bool SHIFT, class PT>
__device__ __forceinline__ K2Val k2_score(const SmemFrag& fp, const PT& pt, int r,
                                          int maxfz, const int64_t* seq_off, const uint8_t* len,
                                          const uint64_t* mask, const float* mass32, const uint8_t* res,
                                          float tol_lo, float tol_hi, float shift) {
  const int np = pt.np;
  const uint8_t* sq = res + seq_off[r];
  int L = len[r];
  uint64_t mk = mask[r];
  float sb = 0.f, sy = 0.f, ppm = 0.f;
  int mb = 0, my = 0;
  RunLen rb = {0, 0, 0, 0}, ry = {0, 0, 0, 0};
  const int da = fp.tol_da;
  int n_alt = 1;
  // per ion kind and index: matched intensity and match count of the unshifted / shifted fragment
  float hit_u[2][SHIFT ? VK_K2_MAXLEN : 1], hit_s[2][SHIFT ? VK_K2_MAXLEN : 1];
  unsigned char cnt_u[2][SHIFT ? VK_K2_MAXLEN : 1], cnt_s[2][SHIFT ? VK_K2_MAXLEN : 1];
  if (SHIFT) {
    n_alt = shift != 0.f ? 2 : 1;
    if (n_alt == 2) {
      for (int k = 0; k < (SHIFT ? VK_K2_MAXLEN : 1); ++k) {
        hit_u[0][k] = hit_u[1][k] = hit_s[0][k] = hit_s[1][k] = 0.f;
        cnt_u[0][k] = cnt_u[1][k] = cnt_s[0][k] = cnt_s[1][k] = 0;
      }
    }
  }
  for (int kind = 0; kind < 2; ++kind) {
    float cum = kind == 0 ? nterm_of(fp, mk) : __fsub_rn(mass32[r], nterm_of(fp, mk));
    for (int k = 0; k + 1 < L; ++k) {
      float rm = resmass(fp, sq[k], k, mk);
      cum = kind == 0 ? __fadd_rn(cum, rm) : __fsub_rn(cum, rm);
      for (int z = 1; z < maxfz; ++z) {
        int best = -1;
        float mx = 0.f, best_mz = 0.f;
        for (int alt = 0; alt < n_alt; ++alt) {
          int best_a = -1;
          float mx_a = 0.f;
          float base = alt == 0 ? cum : __fadd_rn(cum, shift);
          float mz = z == 1 ? base : __fdiv_rn(base, (float)z);   // x / 1 == x exactly
          float a = tol_bound(mz, tol_lo, da), bd = tol_bound(mz, tol_hi, da);
          for (int j = pt.first_ge(a); j < np && pt.mass(j) <= bd; ++j) {
            float it = pt.inten(j);
            if (it >= mx) { mx = it; best = j; best_mz = mz; }
            if (SHIFT && it >= mx_a) { mx_a = it; best_a = j; }
          }
          if (SHIFT && n_alt == 2 && best_a >= 0 && k < VK_K2_MAXLEN) {
            if (alt == 0) { hit_u[kind][k] = __fadd_rn(hit_u[kind][k], pt.inten(best_a)); cnt_u[kind][k] += 1; }
            else { hit_s[kind][k] = __fadd_rn(hit_s[kind][k], pt.inten(best_a)); cnt_s[kind][k] += 1; }
          }
        }
        if (best >= 0) {
          float pmass = pt.mass(best), pint = pt.inten(best);
          float num = __fmul_rn(__fmul_rn(pint, fabsf(__fsub_rn(best_mz, pmass))), 2.0e6f);
          ppm = __fadd_rn(ppm, __fdiv_rn(num, __fadd_rn(best_mz, pmass)));
          if (kind == 0) { mb += 1; sb = __fadd_rn(sb, pint); run_matched(rb, k); }
          else { my += 1; sy = __fadd_rn(sy, pint); run_matched(ry, k); }
        }
      }
    }
  }
  if (SHIFT && n_alt == 2) {
    // best site of the delta (kernels.cu:343-363): b_k shifted iff k >= site, y_k iff k < site
    int Lk = min(L - 1, VK_K2_MAXLEN);
    float sum_bu = 0.f, sum_ys = 0.f, sum_bs = 0.f, sum_yu = 0.f;
    int n_bu = 0, n_ys = 0, n_bs = 0, n_yu = 0;
    for (int k = 0; k < Lk; ++k) {
      sum_bs = __fadd_rn(sum_bs, hit_s[0][k]); n_bs += cnt_s[0][k];
      sum_yu = __fadd_rn(sum_yu, hit_u[1][k]); n_yu += cnt_u[1][k];
    }
    double best_hs = -1e300;
    for (int site = 0; site < L; ++site) {
      if (site > 0 && site - 1 < Lk) {
        int k = site - 1;
        sum_bu = __fadd_rn(sum_bu, hit_u[0][k]); n_bu += cnt_u[0][k];
        sum_bs = __fsub_rn(sum_bs, hit_s[0][k]); n_bs -= cnt_s[0][k];
        sum_ys = __fadd_rn(sum_ys, hit_s[1][k]); n_ys += cnt_s[1][k];
        sum_yu = __fsub_rn(sum_yu, hit_u[1][k]); n_yu -= cnt_u[1][k];
      }
      float sb2 = __fadd_rn(sum_bu, sum_bs), sy2 = __fadd_rn(sum_yu, sum_ys);
      int mb2 = n_bu + n_bs, my2 = n_yu + n_ys;
      double h2 = log((double)__fadd_rn(fmaxf(sb2, 0.f), 1.0f) * (double)__fadd_rn(fmaxf(sy2, 0.f), 1.0f)) +
                  lnfact(mb2) + lnfact(my2);
      if (h2 > best_hs) { best_hs = h2; mb = mb2; my = my2; sb = fmaxf(sb2, 0.f); sy = fmaxf(sy2, 0.f); }
    }
  }
  return K2Val{sb, sy, ppm, mb, my, rb.longest, ry.longest};
}

// ------------------------------------------------------------------------------------------ dense lists, closed
//
// One CTA of KD_WARPS warps per spectrum at a time, one lane per candidate.  Most ions of a candidate meet no peak, and
// the lanes that do meet one differ from ion to ion, so a warp takes its candidates in two loops instead of one lookup
// per ion:
//   * walk (the ion index uniform over the warp): the running f32 masses of the b and y ions, each tested with one
//     fused multiply-add and one bit of a presence bitmap (KD_BITS buckets of 1/KD_SCALE Th, wrapping around; a peak
//     sets every bucket from which an ion could reach it, so a clear bit means no peak in the ion's window); the
//     ions whose bit is set are marked in a mask and their masses listed in shared memory;
//   * lookup: the listed ions of all the warp's candidates, 32 at a time with every lane busy: tolerance window, first
//     peak by a table of start indices, most intense peak, its ppm term; then every lane adds its own ions' results,
//     b then y in ion order.  The arithmetic is k2_score's, so the outputs are bit-identical to it.
// Residues come four at a time from aligned words (single bytes at the ends of the table), their masses
// from one table of mono + delta, lnfact of small counts from a table built by the same function.  With fragment
// charges above 1 each lane looks its own ions up, charge by charge.
//   * left: a candidate of more than KD_MAXLEN residues, or with more marked ions than its lists hold, is scored when
//     the warp's others are: one at a time by the whole warp (kd_score_warp), or by k2_score side by side where more
//     than KD_SLOW of 32 are, because a lane that scores alone leaves 31 idle for some 50 us, and an SM holds 24 of
//     these warps.  Measured, left to a lane each -> now: 3,000 spectra of 2 rows of 70-119 residues 0.211 -> 0.064 ms,
//     of 8 0.248 -> 0.172, of 40 0.359 -> 0.357; 8 rows of 50-65 residues at fragment charges up to 3 0.310 -> 0.166,
//     300 1.95 -> 0.93.  14 for KD_SLOW: 0.244 for 12 rows of 70-119 residues instead of 0.265, but 0.269 for 40 rows
//     of 50-65 at 0.5 Da instead of 0.242.  A warp for each candidate of spectra of up to 3, without the walk: 8-20%
//     faster where all spectra are such, but 0.334 ms instead of 0.289 where they have 2 to 6 (two codes on an SM).
//
// What bounds it: instruction issue and the latency of a warp's dependent steps (0.54 instructions a cycle and
// scheduler; HBM is at 15% with cold caches).  Of 0.341 ms for 20,000 spectra (3.0M candidates) the tables take 0.09
// when nothing hides them, the walk 0.13, the lookup 0.08, the hyperscore and the outputs 0.04.  The warp-per-spectrum
// kernel with a lookup per ion before it ran 4,700 instructions per 32 candidates at 20.7 active lanes; this one runs
// 2,100 at 25.6.  Measured (device time per launch, before -> now): 5.92M candidates of 40,000 spectra 1.590 -> 0.645
// ms, 10,001 spectra of up to 1,000 candidates at 20 ppm 1.412 -> 0.324, fragment charges up to 3 1.078 -> 0.308, 32
// spectra 0.030 -> 0.0096.
// 3 warps per CTA at 8 CTAs per SM: 2, 4 and 6 warps took 12-16% longer on the 40,000 spectra (a spectrum's 148
// candidates are 4.6 warps' worth; wider CTAs idle in their second round, narrower ones build the table with fewer).
// Testing an ion's charges right after its mass, instead of four ions at a time, cost the overlap of the tests (0.70
// and 0.36 ms); words that stop at each row's own end, with single bytes after them, 0.70.
constexpr int KD_WARPS = 3;
constexpr int KD_CTAS = 8;           // CTAs per SM (80 registers, 27 KB)
constexpr int KD_LIST = 20;          // list slots per lane and kind (a group of four ions starts with four free)
constexpr int KD_BITS = 8192;        // presence buckets
constexpr float KD_SCALE = 4.0f;     // buckets per Th: 2,048 Th before they wrap
constexpr int KD_LNF = 32;           // tabulated lnfact arguments
constexpr int KD_MAXLEN = 65;        // residues whose 64 ions fit a mask
constexpr int KD_SLOW = 8;           // of 32 candidates, those left that the warp takes one after another
constexpr int16_t KD_LEFT = -1;      // the longest run of a candidate that is left
constexpr int KD_QUEUE = 256;        // ions looked up per round of a warp (a lane has at most 2 * KD_LIST)
static_assert(KD_QUEUE >= 2 * KD_LIST, "a lane's ions fit a round");

struct K2DenseSmem {
  float2 peak[VK_K2_MAXPK + 1];      // (mass, intensity), a NaN mass after the last
  double lnf[KD_LNF];
  uint32_t bits[KD_BITS / 32];
  uint16_t start[K2_BUCKETS];        // first peak of 16 presence buckets (4 Th), from the first peak's on
  float res[64];                     // residue mass by (letter & 31) | modified << 5
  float ion[KD_WARPS][2][KD_LIST][32];   // listed ions' masses (b, y); after the lookup their peaks' intensities
  float term[KD_WARPS][KD_QUEUE];        // ppm terms of the ions of a lookup round
  uint16_t queue[KD_WARPS][KD_QUEUE];    // their places in ion
};

// Unwrapped bucket of mass m in the low bits: m * KD_SCALE rounded to an integer, monotone in m while its magnitude
// stays below 2^21 (KD_SAFE); the low 13 bits are the bucket.
constexpr float KD_SAFE = 2097152.0f / KD_SCALE;
__device__ __forceinline__ uint32_t kd_bucket(float m) {
  return __float_as_uint(__fmaf_rn(m, KD_SCALE, 12582912.0f));
}
__device__ __forceinline__ uint32_t kd_flag(const uint32_t* bits, float m) {
  const uint32_t q = kd_bucket(m);
  const uint32_t word = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(bits) +
                                                           ((q >> 3) & (KD_BITS / 8 - 4)));   // bits[(q >> 5) % words]
  return __funnelshift_r(word, 0u, q) & 1u;   // shift by q mod 32
}

// Ion masses that may have peak x in their tolerance window: [lo, hi] widened by 1e-6 of the masses, above the
// rounding of the bounds, of this inversion and of the walk's approximate division by the charge.
__device__ __forceinline__ float2 kd_reach(float x, float tol_lo, float tol_hi, int da) {
  if (da) return make_float2((x - tol_hi) - 1e-6f * (fabsf(x) + fabsf(tol_hi)),
                             (x - tol_lo) + 1e-6f * (fabsf(x) + fabsf(tol_lo)));
  const float up = 1.f + tol_hi * 1e-6f, dn = 1.f + tol_lo * 1e-6f;
  if (!(x > 0.f) || !(up > 0.5f && up < 2.f) || !(dn > 0.5f && dn < 2.f))
    return make_float2(-CUDART_INF_F, CUDART_INF_F);
  return make_float2(__fdividef(x, up) - 2e-6f * x, __fdividef(x, dn) + 2e-6f * x);
}

// Residues of a row, four per word, from aligned words of the residue table.  Words up to `end` -- the end of any row,
// so inside the table -- are read whole, whatever row their bytes belong to; past it (the row whose end that is) and
// before the table's first byte, only the row's own bytes are.
struct RowWords {
  const uint8_t* at;      // the next word
  const uint8_t* end;
  uint32_t cur, shift;
  int left;               // bytes of the row from `at` on

  static __device__ __forceinline__ uint32_t bytes(const uint8_t* a, int from, int to) {
    uint32_t v = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j >= from && j < to) v |= (uint32_t)__ldg(a + j) << (8 * j);
    return v;
  }
  __device__ __forceinline__ void begin(const uint8_t* table, const uint8_t* row, int len, const uint8_t* last_end) {
    const int skip = (int)(reinterpret_cast<uintptr_t>(row) & 3);
    at = row - skip;
    end = last_end;
    shift = 8u * (uint32_t)skip;
    left = len + skip;
    cur = at >= table && at + 4 <= end ? __ldg(reinterpret_cast<const uint32_t*>(at)) : bytes(at, skip, left);
    at += 4;
    left -= 4;
  }
  __device__ __forceinline__ uint32_t next() {   // the next four bytes: residues of the row, then whatever follows
    uint32_t nx = 0u;
    if (left > 0) nx = at + 4 <= end ? __ldg(reinterpret_cast<const uint32_t*>(at)) : bytes(at, 0, left);
    const uint32_t r = __funnelshift_r(cur, nx, shift);
    cur = nx;
    at += 4;
    left -= 4;
    return r;
  }
};

// Index of mass x into the start table whose first entry is bucket q0: monotone in x, clamped at both ends.
__device__ __forceinline__ int kd_start(float x, uint32_t q0) {
  const float t = fmaxf(__fmaf_rn(x, KD_SCALE, 12582912.0f), 8388608.0f);   // positive: its bits order like it
  return min(max((int)(__float_as_uint(t) - q0), 0) >> 4, K2_BUCKETS - 1);
}

// The spectrum's table in the form k2_score takes.
struct DensePeaks {
  const K2DenseSmem& S;
  int np;
  uint32_t q0;
  __device__ __forceinline__ float mass(int j) const { return S.peak[j].x; }
  __device__ __forceinline__ float inten(int j) const { return S.peak[j].y; }
  __device__ __forceinline__ int first_ge(float a) const {
    int j = S.start[kd_start(a, q0)];
    while (S.peak[j].x < a) ++j;   // ends at the NaN after the last peak
    return j;
  }
};

// The most intense peak (the last of equals) in the tolerance window of fragment m/z mz: its mass and intensity, a
// NaN intensity when there is none.
__device__ __forceinline__ float2 kd_match(const K2DenseSmem& S, uint32_t q0, float mz, float tol_lo, float tol_hi,
                                           int da) {
  const float a = tol_bound(mz, tol_lo, da), bd = tol_bound(mz, tol_hi, da);
  const float2* pk = &S.peak[S.start[kd_start(a, q0)]];
  float2 x = *pk;
  while (x.x < a) x = *++pk;   // ends at the NaN after the last peak
  float2 best = make_float2(0.f, CUDART_NAN_F);
  while (x.x <= bd) {
    if (x.y >= 0.f && !(x.y < best.y)) best = x;
    x = *++pk;
  }
  return best;
}

__device__ __forceinline__ float kd_term(float mz, float2 peak) {
  const float num = __fmul_rn(__fmul_rn(peak.y, fabsf(__fsub_rn(mz, peak.x))), 2.0e6f);
  return __fdiv_rn(num, __fadd_rn(mz, peak.x));
}

static __device__ __noinline__ K2Val kd_score_serial(const SmemFrag* fp, const K2DenseSmem* S, int np, uint32_t q0,
                                                     int r, int maxfz, const int64_t* seq_off,
                                                     const uint8_t* len, const uint64_t* mask, const float* mass32,
                                                     const uint8_t* res, float tol_lo, float tol_hi) {
  const DensePeaks pt{*S, np, q0};
  return k2_score<false, DensePeaks>(*fp, pt, r, maxfz, seq_off, len, mask, mass32, res, tol_lo, tol_hi, 0.f);
}

// One candidate by the whole warp: its ion masses summed by two lanes, the ions of every charge looked up 32 at a time,
// the matches added up in k2_score's order.  Every lane returns the candidate's values.
static __device__ __noinline__ K2Val kd_score_warp(const SmemFrag* fp, K2DenseSmem* S, int warp, uint32_t q0,
                                                   const uint8_t* seq, int len, int maxfz, uint64_t mask, float mass,
                                                   float tol_lo, float tol_hi) {
  const int lane = threadIdx.x & 31, n = len - 1, nz = maxfz - 1, half = n * nz;
  K2Val v{0.f, 0.f, 0.f, 0, 0, 0, 0};
  if (n <= 0 || nz <= 0) return v;
  float* rm = &S->ion[warp][0][0][0];   // n <= 254 residue masses, then the b and the y ions
  float* ions = rm + 256;
  for (int k = lane; k < n; k += 32) rm[k] = resmass(*fp, seq[k], k, mask);
  __syncwarp();
  if (lane < 2) {
    const float nt = nterm_of(*fp, mask), sign = lane ? -1.f : 1.f;
    float c = lane ? __fsub_rn(mass, nt) : nt;
    float* to = ions + 256 * lane;
#pragma unroll 4
    for (int k = 0; k < n; ++k) to[k] = c = __fadd_rn(c, __fmul_rn(sign, rm[k]));   // (x - r is x + -r)
  }
  __syncwarp();
  RunLen rb = {0, 0, 0, 0}, ry = {0, 0, 0, 0};
  for (int t0 = 0; t0 < 2 * half; t0 += 32) {
    const int t = t0 + lane, kind = t >= half, i = t - kind * half, k = i / nz, z = i - k * nz + 1;
    float2 peak = make_float2(0.f, CUDART_NAN_F);
    float term = 0.f;
    if (t < 2 * half) {
      const float base = ions[256 * kind + k], mz = z == 1 ? base : __fdiv_rn(base, (float)z);
      peak = kd_match(*S, q0, mz, tol_lo, tol_hi, fp->tol_da);
      term = kd_term(mz, peak);
    }
    for (unsigned hit = __ballot_sync(VK_FULL, peak.y >= 0.f); hit; hit &= hit - 1u) {
      const int l = __ffs(hit) - 1, at = __shfl_sync(VK_FULL, kind << 16 | k, l);
      const float pint = __shfl_sync(VK_FULL, peak.y, l);
      v.ppm = __fadd_rn(v.ppm, __shfl_sync(VK_FULL, term, l));
      if (at >> 16) {
        v.my += 1;
        v.sy = __fadd_rn(v.sy, pint);
        run_matched(ry, at & 0xffff);
      } else {
        v.mb += 1;
        v.sb = __fadd_rn(v.sb, pint);
        run_matched(rb, at);
      }
    }
  }
  v.lb = rb.longest;
  v.ly = ry.longest;
  return v;
}

__device__ __forceinline__ double kd_lnfact(const K2DenseSmem& S, int n) {
  return n < KD_LNF ? S.lnf[n] : lnfact(n);
}

// Longest run of consecutive matched ion indices (run_matched: ion 0 starts no run).
__device__ __forceinline__ int kd_longest(uint64_t hit) {
  int n = 0;
  if ((hit >> 32) == 0ull) {
    for (uint32_t x = (uint32_t)hit & ~1u; x; x &= x << 1) ++n;
  } else {
    for (uint64_t x = hit & ~1ull; x; x &= x << 1) ++n;
  }
  return n;
}

// The walk over the warp's candidates (see above): marks and lists the ions of n_max steps that may match at a charge
// below maxfz (at most z_max in the warp).  Sets `over` where a list may have overflowed.
__device__ __forceinline__ void kd_walk(K2DenseSmem& S, int warp, int lane, int n_ion, int n_max, int maxfz, int z_max,
                                        RowWords& w, uint64_t mask, float b, float y, uint64_t& mark_b,
                                        uint64_t& mark_y, bool& over) {
  uint32_t mod_lo = (uint32_t)mask, mod_hi = (uint32_t)(mask >> 32);
  uint32_t mb = 0u, my = 0u, mb_lo = 0u, my_lo = 0u;   // marks of the current 32 ions, of the 32 before them
  float* list_b = &S.ion[warp][0][0][lane];
  float* list_y = &S.ion[warp][1][0][lane];
  for (int k0 = 0; k0 < n_max; k0 += 4) {
    const bool in = k0 < n_ion;
    if (k0 > KD_LIST - 4) {   // (k0 ions fill at most k0 slots) the group needs four free ones
      if (k0 == 32) {
        mb_lo = mb;
        my_lo = my;
        mb = my = 0u;
      }
      const int n_b = __popc(mb) + __popc(mb_lo), n_y = __popc(my) + __popc(my_lo);
      over |= in && max(n_b, n_y) > KD_LIST - 4;
      list_b = &S.ion[warp][0][min(n_b, KD_LIST - 4)][lane];
      list_y = &S.ion[warp][1][min(n_y, KD_LIST - 4)][lane];
    }
    // byte offsets into the residue table, one per residue; past the row's end whatever follows: those ions land
    // behind the lists' valid part and their marks are cleared by the caller
    const uint32_t four = ((in ? w.next() : 0u) & 0x1f1f1f1fu) << 2 |
                          (((mod_lo & 15u) * 0x00204081u) & 0x01010101u) << 7;
    mod_lo = __funnelshift_r(mod_lo, mod_hi, 4);
    mod_hi >>= 4;
    float bv[4], yv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float rm = *reinterpret_cast<const float*>(reinterpret_cast<const char*>(S.res) +
                                                       ((four >> (8 * j)) & 0xffu));
      bv[j] = b = __fadd_rn(b, rm);
      yv[j] = y = __fsub_rn(y, rm);
    }
    uint32_t fb[4], fy[4];   // eight independent tests in flight
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      fb[j] = kd_flag(S.bits, bv[j]);
      fy[j] = kd_flag(S.bits, yv[j]);
    }
    for (int z = 2; z < z_max; ++z) {
      const uint32_t on = z < maxfz;
      const float rz = __fdividef(1.f, (float)z);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        fb[j] |= on & kd_flag(S.bits, __fmul_rn(bv[j], rz));
        fy[j] |= on & kd_flag(S.bits, __fmul_rn(yv[j], rz));
      }
    }
    uint32_t pb = 0u, py = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (in) {        // kept only when the slot moves on
        *list_b = bv[j];
        *list_y = yv[j];
      }
      list_b += fb[j] * 32u;
      list_y += fy[j] * 32u;
      pb += fb[j] << j;
      py += fy[j] << j;
    }
    mb |= pb << (k0 & 31);
    my |= py << (k0 & 31);
  }
  mark_b = n_max > 32 ? (uint64_t)mb << 32 | mb_lo : mb;
  mark_y = n_max > 32 ? (uint64_t)my << 32 | my_lo : my;
}

// A candidate's row, loaded ahead of its scoring.
struct DenseRow {
  const uint8_t* seq;
  uint64_t mask;
  float mass;
  int len, maxfz;

  // ions to walk; none of an empty row (whose offset may lie anywhere: its residues are not looked at)
  __device__ __forceinline__ int ions() const { return len <= KD_MAXLEN && maxfz > 1 ? max(len - 1, 0) : 0; }
};

__device__ __forceinline__ DenseRow kd_row(int64_t c, const int32_t* c_row, const int8_t* c_maxfz,
                                           const int64_t* seq_off, const uint8_t* len, const uint64_t* mask,
                                           const float* mass32, const uint8_t* res) {
  DenseRow d;
  const int row = c_row[c];
  d.maxfz = c_maxfz[c];
  d.seq = res + seq_off[row];
  d.len = len[row];
  d.mask = mask[row];
  d.mass = mass32[row];
  return d;
}

// The row's first word.  Words up to the row end of the warp's last lane with ions are read whole (candidates come in
// row order, so that is nearly all of them).
__device__ __forceinline__ void kd_begin(RowWords& w, const DenseRow& d, bool live, const uint8_t* res) {
  const unsigned lanes = __ballot_sync(VK_FULL, live && d.ions() > 0);
  if (!lanes) return;
  const unsigned long long mine = reinterpret_cast<unsigned long long>(d.seq + d.len);
  const unsigned long long last = __shfl_sync(VK_FULL, mine, 31 - __clz(lanes));
  if (live && d.ions() > 0) w.begin(res, d.seq, d.len, reinterpret_cast<const uint8_t*>(last));
}

// Scores the warp's candidates (lanes with `live` hold one each).  True in lanes whose candidate is left to kd_left.
__device__ __forceinline__ bool kd_score(K2DenseSmem& S, const DensePeaks& pt, int warp, int lane, bool live,
                                         const DenseRow& d, RowWords& w, const SmemFrag& fp, float tol_lo, float tol_hi,
                                         const K2Out& out, int64_t c) {
  const bool fits = live && d.len <= KD_MAXLEN;
  const int n_ion = live ? d.ions() : 0;
  const int n_max = __reduce_max_sync(VK_FULL, n_ion);
  const int z_max = __reduce_max_sync(VK_FULL, fits ? d.maxfz : 0);
  uint64_t mark_b, mark_y;   // ions that may match
  bool over = false;
  const float nt = nterm_of(fp, d.mask), y0 = __fsub_rn(d.mass, nt);
  kd_walk(S, warp, lane, n_ion, n_max, d.maxfz, z_max, w, d.mask, nt, y0, mark_b, mark_y, over);
  const uint64_t valid = n_ion < 64 ? (1ull << n_ion) - 1ull : ~0ull;
  mark_b &= valid;
  mark_y &= valid;
  K2Val v{0.f, 0.f, 0.f, 0, 0, 0, 0};
  uint64_t hit_b = 0ull, hit_y = 0ull;
  if (z_max <= 2) {
    const int n_b = __popcll(mark_b), n = over || !fits ? 0 : n_b + __popcll(mark_y);
    const int end = (int)warp_incl_scan_i32(n), begin = end - n, total = __shfl_sync(VK_FULL, end, 31);
    float* ion = &S.ion[warp][0][0][0];
    for (int base = 0; base < total;) {   // the ions of as many whole lanes as a round holds: usually all
      const bool mine = begin >= base && end <= base + KD_QUEUE && n > 0;
      const int stop = __reduce_max_sync(VK_FULL, mine ? end : 0);
      if (mine)
        for (int i = 0; i < n; ++i)
          S.queue[warp][begin - base + i] = (uint16_t)((i < n_b ? i : KD_LIST + i - n_b) * 32 + lane);
      __syncwarp();
      for (int t = lane; t < stop - base; t += 32) {
        const int at = S.queue[warp][t];
        const float mz = ion[at];
        const float2 peak = kd_match(S, pt.q0, mz, tol_lo, tol_hi, fp.tol_da);
        ion[at] = peak.y;
        S.term[warp][t] = kd_term(mz, peak);
      }
      __syncwarp();
      if (mine) {
        const float* term = &S.term[warp][begin - base];
        const float* at = &S.ion[warp][0][0][lane];
        for (uint64_t todo = mark_b; todo; todo &= todo - 1ull, at += 32, ++term) {
          const float pint = *at;
          if (pint >= 0.f) {
            v.ppm = __fadd_rn(v.ppm, *term);
            v.mb += 1;
            v.sb = __fadd_rn(v.sb, pint);
            hit_b |= todo ^ (todo & (todo - 1ull));
          }
        }
        at = &S.ion[warp][1][0][lane];
        for (uint64_t todo = mark_y; todo; todo &= todo - 1ull, at += 32, ++term) {
          const float pint = *at;
          if (pint >= 0.f) {
            v.ppm = __fadd_rn(v.ppm, *term);
            v.my += 1;
            v.sy = __fadd_rn(v.sy, pint);
            hit_y |= todo ^ (todo & (todo - 1ull));
          }
        }
      }
      base = stop;
      __syncwarp();
    }
  }
  if (!live) return false;
  if (!fits || over) {
    out.lb[c] = KD_LEFT;
    return true;
  } else {
    if (z_max > 2) {
      uint64_t todo = mark_b;
      bool in_y = todo == 0ull;
      if (in_y) todo = mark_y;
      const float* next = &S.ion[warp][in_y][0][lane];
      while (todo) {   // the lane's marked ions, b then y
        const uint64_t rest = todo & (todo - 1ull), bit = todo ^ rest;
        todo = rest;
        const float base = *next;
        next += 32;
        for (int z = 1; z < d.maxfz; ++z) {
          const float mz = z == 1 ? base : __fdiv_rn(base, (float)z);   // x / 1 == x exactly
          const float2 peak = kd_match(S, pt.q0, mz, tol_lo, tol_hi, fp.tol_da);
          if (!(peak.y >= 0.f)) continue;
          v.ppm = __fadd_rn(v.ppm, kd_term(mz, peak));
          if (in_y) {
            v.my += 1;
            v.sy = __fadd_rn(v.sy, peak.y);
            hit_y |= bit;
          } else {
            v.mb += 1;
            v.sb = __fadd_rn(v.sb, peak.y);
            hit_b |= bit;
          }
        }
        if (!todo && !in_y) {
          todo = mark_y;
          in_y = true;
          next = &S.ion[warp][1][0][lane];
        }
      }
    }
    v.lb = kd_longest(hit_b);
    v.ly = kd_longest(hit_y);
  }
  k2_write(v, [&](int n) { return kd_lnfact(S, n); }, out, c);
  return false;
}

// The warp's candidates that kd_score left: one after another by the whole warp where few of 32 are, else side by side.
__device__ __forceinline__ void kd_left(const SmemFrag* fp, K2DenseSmem* S, int np, uint32_t q0, int warp, int64_t c0,
                                        int64_t c1, const int32_t* c_row, const int8_t* c_maxfz,
                                        const int64_t* seq_off, const uint8_t* len, const uint64_t* mask,
                                        const float* mass32, const uint8_t* res, float tol_lo, float tol_hi,
                                        const K2Out& out) {
  const int lane = threadIdx.x & 31;
  for (int64_t cw = c0 + warp * 32; cw < c1; cw += KD_WARPS * 32) {
    const int64_t c = cw + lane;
    const bool mine = c < c1 && out.lb[c] == KD_LEFT;
    unsigned todo = __ballot_sync(VK_FULL, mine);
    if (!todo) continue;
    K2Val v{0.f, 0.f, 0.f, 0, 0, 0, 0};
    if (__popc(todo) <= KD_SLOW) {
      for (; todo; todo &= todo - 1u) {
        const int l = __ffs(todo) - 1, r = c_row[cw + l];
        const K2Val one = kd_score_warp(fp, S, warp, q0, res + seq_off[r], len[r], c_maxfz[cw + l], mask[r], mass32[r],
                                        tol_lo, tol_hi);
        if (lane == l) v = one;
      }
    } else if (mine) {
      v = kd_score_serial(fp, S, np, q0, c_row[c], c_maxfz[c], seq_off, len, mask, mass32, res, tol_lo, tol_hi);
    }
    if (mine) k2_write(v, [&](int n) { return kd_lnfact(*S, n); }, out, c);
    __syncwarp();
  }
}

// CTA-per-spectrum driver of the closed scoring.  spec_ids == nullptr: spectrum bs uses peaks of spectrum bs.
__device__ __forceinline__ void k2_dense_body(K2DenseSmem& S, const SmemFrag& fp, int n_spec, const int64_t* cand_off,
                                              const int32_t* c_row, const int8_t* c_maxfz, const int32_t* spec_ids,
                                              const int64_t* pk_off, const float* pk_mass, const float* pk_int,
                                              const int64_t* seq_off, const uint8_t* len, const uint64_t* mask,
                                              const float* mass32, const uint8_t* res, float tol_lo, float tol_hi,
                                              const K2Out& out) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int NT = KD_WARPS * 32;
  const int da = fp.tol_da;
  for (int i = tid; i < 64; i += NT) {
    const int letter = (i & 31) - 1;
    S.res[i] = letter >= 0 && letter < 26 ? __fadd_rn(fp.mono[letter], i & 32 ? fp.var[letter] : fp.stat[letter]) : 0.f;
  }
  if (warp == KD_WARPS - 1) S.lnf[lane] = lnfact(lane);
  static_assert(KD_LNF == 32, "one entry per lane");
  for (int bs = blockIdx.x; bs < n_spec; bs += gridDim.x) {
    const int s = spec_ids ? spec_ids[bs] : bs;
    const int64_t c0 = cand_off[bs], c1 = cand_off[bs + 1], p0 = pk_off[s], p1 = pk_off[s + 1];
    if (c0 >= c1) continue;    // uniform over the CTA
    const int np = (int)min((int64_t)VK_K2_MAXPK, p1 - p0);
    DenseRow d{};              // this thread's first candidate, loaded while the table is built
    const bool some = c0 + tid < c1;
    if (some) d = kd_row(c0 + tid, c_row, c_maxfz, seq_off, len, mask, mass32, res);
    __syncthreads();           // the previous spectrum's readers are done
    for (int j = tid; j < np; j += NT) S.peak[j] = make_float2(pk_mass[p0 + j], pk_int[p0 + j]);
    if (tid == 0) S.peak[max(np, 0)] = make_float2(CUDART_NAN_F, 0.f);
    for (int j = tid; j < KD_BITS / 32; j += NT) S.bits[j] = 0u;
    __syncthreads();
    const float first = np > 0 ? S.peak[0].x : 0.f, last = np > 0 ? S.peak[np - 1].x : 0.f;
    const DensePeaks pt{S, np, kd_bucket(first)};
    for (int j = tid; j < np; j += NT) {
      const float x = S.peak[j].x;
      const float2 rg = kd_reach(x, tol_lo, tol_hi, da);
      uint32_t qa = 0u, n = KD_BITS;   // the first bucket and how many
      if (rg.x > -KD_SAFE && rg.y < KD_SAFE) {
        qa = kd_bucket(rg.x);
        n = min(kd_bucket(rg.y) - qa + 1u, (uint32_t)KD_BITS);
      }
      while (n > 0u) {
        const uint32_t m = min(n, 32u - (qa & 31u));
        atomicOr(&S.bits[(qa >> 5) & (KD_BITS / 32 - 1)], (0xffffffffu >> (32u - m)) << (qa & 31u));
        qa += m;
        n -= m;
      }
      const int b = kd_start(x, pt.q0);
      const int bp = j > 0 ? kd_start(S.peak[j - 1].x, pt.q0) : -1;
      for (int q = bp + 1; q <= b; ++q) S.start[q] = (uint16_t)j;
    }
    const int blast = np > 0 ? kd_start(last, pt.q0) : -1;
    for (int q = blast + 1 + tid; q < K2_BUCKETS; q += NT) S.start[q] = (uint16_t)max(np, 0);
    RowWords w{};
    kd_begin(w, d, some, res);
    __syncthreads();
    bool left = false;
    for (int64_t cw = c0 + warp * 32; cw < c1; cw += NT) {   // uniform over the warp
      const int64_t c = cw + lane;
      left |= kd_score(S, pt, warp, lane, c < c1, d, w, fp, tol_lo, tol_hi, out, c);
      __syncwarp();
      const bool more = c + NT < c1;
      if (more) d = kd_row(c + NT, c_row, c_maxfz, seq_off, len, mask, mass32, res);
      kd_begin(w, d, more, res);
    }
    if (__any_sync(VK_FULL, left))
      kd_left(&fp, &S, np, pt.q0, warp, c0, c1, c_row, c_maxfz, seq_off, len, mask, mass32, res, tol_lo, tol_hi, out);
  }
}

// Grid of a dense kernel: up to KD_WAVES CTAs per resident slot, each taking every grid-th spectrum -- enough CTAs
// that the slots finish together (one per slot: 62 us instead of 44 on 5,000 spectra, 428 instead of 370 on 10,001),
// few enough that a CTA's residue and lnfact tables serve several spectra.
constexpr int KD_WAVES = 8;
template <class F>
int k2_dense_grid(F kernel, int n_spec, int* err) {
  int per_sm = 0, dev = 0, n_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, KD_WARPS * 32, 0);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  *err = (int)e;
  if (e != cudaSuccess) return 0;
  const int most = (per_sm > 1 ? per_sm : 1) * n_sm * KD_WAVES;
  return most < n_spec ? most : n_spec;
}

// Warp-per-spectrum driver of the shifted scoring.  spec_ids == nullptr: spectrum bs uses peaks of spectrum bs.
__device__ __forceinline__ void k2_body(const SmemFrag& fp, int n_spec, const int64_t* cand_off,
                                        const int32_t* c_row, const int8_t* c_maxfz, const int32_t* spec_ids,
                                        const int64_t* pk_off, const float* pk_mass, const float* pk_int,
                                        const int64_t* seq_off, const uint8_t* len, const uint64_t* mask,
                                        const float* mass32, const uint8_t* res, float tol_lo, float tol_hi,
                                        const float* c_shift, const K2Out& out) {
  __shared__ float s_mass[K2_WARPS][VK_K2_MAXPK];
  __shared__ float s_int[K2_WARPS][VK_K2_MAXPK];
  __shared__ uint16_t s_start[K2_WARPS][K2_BUCKETS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int bs = blockIdx.x * K2_WARPS + warp; bs < n_spec; bs += gridDim.x * K2_WARPS) {
    int s = spec_ids ? spec_ids[bs] : bs;
    int64_t p0 = pk_off[s];
    int np = (int)min((int64_t)VK_K2_MAXPK, pk_off[s + 1] - p0);
    float* sm = s_mass[warp];
    float* si = s_int[warp];
    __syncwarp();
    for (int j = lane; j < np; j += 32) {
      sm[j] = pk_mass[p0 + j];
      si[j] = pk_int[p0 + j];
    }
    __syncwarp();
    const PeakTable pt = build_table(sm, si, s_start[warp], np, lane);
    int64_t c1 = cand_off[bs + 1];
    for (int64_t c = cand_off[bs] + lane; c < c1; c += 32) {
      k2_write(k2_score<true, PeakTable>(fp, pt, c_row[c], c_maxfz[c], seq_off, len, mask, mass32, res, tol_lo, tol_hi,
                                         c_shift[c]),
               lnfact, out, c);
    }
  }
}

}  // namespace vk
