// FP64 grouped GEMM of the block-sparse hot path on sm_103a, on the tensor cores.
//
// GB300 retires about 2 FP64 multiply-adds per clock per SM, in its FP64 tensor instruction too (and
// as few with half the lanes off), but 1035 FP16 ones through mma.sync (all measured); every
// contraction here was bound by the FP64 pipe.  The kernel therefore splits FP64 operands into exact
// FP16 digits (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59 (2012)
// 95, in the fixed-point form used on tensor cores by Mukunoki, Ozaki, Ogita and Imamura, ISC 2020):
//   * a row of op(A), or a column of op(B), inside one K chunk of one term is scaled by a power of
//     two to magnitude < 127 / 128 and cut off at 63 fractional bits (entries down to 2^-10 of the
//     largest keep all 53 bits of theirs), then written as 8 balanced base-256 digits, |d_i| <= 128;
//   * digit products of one level l = i + j <= 7 (36 of the 64 pairs) are summed in FP32 by mma.sync
//     m16n8k16.  Every partial sum is an integer of at most 8 * 2^14 * 80 < 2^24, so the sums are
//     exact in any order; the dropped levels and the cut operands are below 2^-60.5 of the product of
//     the two scales for each k;
//   * per output and chunk the eight level sums are combined in integers, converted to FP64 and added
//     by one fma: one FP64 instruction where the direct form needs one per k;
//   * that error is relative to the largest entries of the row and the column, an FP64 sum's to
//     S = sum_k |a_ik| |b_kj|, which is far smaller where they are graded oppositely along k.  So
//     one more product sums the magnitudes that the first two digits give, |256 d_0 + d_1| (an entry
//     is within 0.502 of it: 80 products overstate S by at most 2.7e6 of the units of 2^-30).  From
//     kTrusted on, S is thus above 2^-7.5 of the scales and the error below K 2^-53 S, the bound of
//     K FP64 multiply-adds.  An output below it, other than one of a row or column of zeros, is computed
//     by plain FP64 multiply-adds: none at Gaussian operands, below 1% in an environment's products at
//     converged VUMPS states of XXZ D = 512.  (The first digit alone sees 0.3 to 6% of those as
//     too small, an environment's entries off its diagonal being some 0.3% of those on it: H_AC 36 us.)
// Relative error of the H_AC apply (2-norm, against a double-double reference): 0.9e-16 to 1.1e-16 over
// XXZ D = 32 to 1024 and Hubbard D = 64 to 1024, where the direct form had 1.4e-16 (D = 64) to 5.3e-16
// (XXZ D = 1024); at XXZ D = 512 0.9e-16 after 4.1e-16, at Hubbard D = 1024 1.0e-16 after 4.7e-16.
// Seven digits (28 products) without that test took 16.9 us instead of 18.8 (XXZ D = 512), but lost what is
// small: a thick restart's rotation had 1.1e-15 in the lowest Ritz vector where the direct form has 3e-16
// (now 2e-17), and VUMPS sweeps from starts 1e-16 apart had energies 1e-11 apart after one sweep (now
// 1e-14, as with the direct form).
// A chunk with an entry that is not finite, or with a row or column whose largest magnitude is outside
// 2^-423 .. 2^477 (where the scaled sums could leave the FP64 range), is computed by plain FP64
// fused multiply-adds, so infinities, NaN and extreme scales keep their FP64 results; so is one whose
// op(A) has at most one entry per row, or op(B) per column (copies by an identity stay exact).
//
// mma.sync rather than tcgen05: the operands are split in registers on the fly (no operand packs that
// could go stale, no extra pass over memory), blocks are ragged with edges from 1 to 82, and the eight
// level sums of a 16 x 8 sub-tile fit a warp's registers, where a 128-row instruction would compute
// mostly padding.  What bounds it (XXZ D = 512 H_AC, ncu): integer pipe 28%, tensor pipe 19%, FP64 pipe
// 12% busy, i.e. the latency of the chain load - split - multiply - combine of one to three chunks per
// CTA; throughput alone would take about 6 us.
//
// Work split: a table entry is an output tile (<= 32 x 32, or <= 16 x 16 where a stage has too few
// tiles; edges are multiples of 16 and 8, balanced over the block, so that a 68 x 68 block computes
// 80 x 72 instead of 96 x 96) and a contiguous share of its K chunks.  With one share the tile is
// written directly; otherwise every CTA stores its partial tile and the last CTA of the tile to
// finish (an atomic ticket after a memory fence; nobody waits) sums the partials in share order and
// writes the tile.  Deterministic for a given plan; the first write also performs the reference's
// memset of `out`, VUMPS_helpers.hpp:69.
//
// H_AC apply, direct FP64 form -> this one: XXZ D = 64 23.2 -> 7.0 us, XXZ D = 512 59.4 -> 18.8 us,
// Hubbard D = 1024 163.7 -> 47.4 us; four-stage transfer matrix at XXZ D = 512 73.8 -> 35.4 us.
// Dividing the work between warps that split and warps that multiply, in a persistent CTA per SM, gained 8
// to 9% on the H_AC applies (with seven digits), but lost 11% on the projected transfer matrix at Hubbard
// D = 1024: the SM's issue slots (some 10,000 warp instructions a chunk) are the limit, not the overlap.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "imps_internal.h"
#include "imps_status.h"

using imps::Term;
using imps::Tile;

namespace {

constexpr int NS = 8;     // digits per operand
constexpr int kLowExp = 600, kHighExp = 1500;  // biased exponents of rows the split form takes
constexpr float kTrusted = 9e6f;  // least magnitude sum, in units of 2^-30 of the scales, of an output that the digits give

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(addr)
               : "memory");
}

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// x / 2^(E - 1022) as a fixed-point integer with 63 fractional bits (cut off towards zero), |x| below 127 / 128 of
// that scale, plus a bias that makes every base-256 digit non-negative: byte i holds digit d_{7-i} + 128.
__device__ __forceinline__ uint64_t fixed_digits(double x, int E) {
  const uint32_t lo = (uint32_t)__double2loint(x);
  const int32_t hi = __double2hiint(x);
  const int e = (int)((2u * (uint32_t)hi) >> 21);
  // the significand in bits 62..10, with the sign as ones' complement; an entry below the normal range is
  // far below the row's scale, as is zero
  const uint32_t sg = (uint32_t)(hi >> 31);
  const uint32_t th = __funnelshift_l(lo, ((uint32_t)hi & 0x000fffffu) | 0x00100000u, 10) ^ sg, tl = (lo << 10) ^ sg;
  const int64_t s = (int64_t)(((uint64_t)th << 32) | tl);
  return (uint64_t)(s >> min(E - e, 63)) + (0x8080808080808080ull + (sg & 1u));
}

// the eight digits of two entries (k, k + 1) as packed FP16: 1024 + u, less 1024 and the bias
__device__ __forceinline__ void digit_pairs(uint64_t x, uint64_t y, uint32_t (&d)[NS]) {
  const uint32_t xl = (uint32_t)x, yl = (uint32_t)y, xh = (uint32_t)(x >> 32), yh = (uint32_t)(y >> 32);
  const uint32_t m = 0x64646464u;
  const uint32_t p[4] = {__byte_perm(xl, yl, 0x5140), __byte_perm(xl, yl, 0x7362), __byte_perm(xh, yh, 0x5140),
                         __byte_perm(xh, yh, 0x7362)};
#pragma unroll
  for (int i = 0; i < NS; ++i) {
    d[NS - 1 - i] = __byte_perm(p[i / 2], m, i & 1 ? 0x4342 : 0x4140);
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&d[NS - 1 - i]),
                              __half2half2(__ushort_as_half(0x6480)));  // 1152
    d[NS - 1 - i] = *reinterpret_cast<const uint32_t*>(&h);
  }
}

// One operand's chunk in the registers of four warps: entry (r, k) of op(A) (rows m) or op(B)^T (rows
// n) is at r * sr + k * sk (one of the strides is 1).  A thread holds the pairs of k at
// 2 * (lane / 8 + 4 i) of row 8 w + lane % 8: 64 contiguous bytes per row or column of a warp's load,
// and digit stores that hit 32 banks.  One mapping for both orders keeps the code short: most CTAs
// run few chunks, and with two mappings a fifth of the stalls were instruction fetches.
template <int KI>
__device__ __forceinline__ void load_operand(double (&v)[4 * KI], const double* p, int sr, int sk, int nrow, int len,
                                             int w, int lane) {
  const int r = 8 * w + (lane & 7), k0 = 2 * (lane >> 3);
  const double* pr = p + (int64_t)r * sr + (int64_t)k0 * sk;
  const int left = r < nrow ? len - k0 : 0;
#pragma unroll
  for (int s = 0; s < KI; ++s)
    if (16 * s < len)  // the same for the whole warp; entries of later K steps are not looked at
#pragma unroll
      for (int i = 2 * s; i < 2 * s + 2; ++i)
#pragma unroll
        for (int q = 0; q < 2; ++q) v[2 * i + q] = 8 * i + q < left ? pr[(8 * i + q) * (int64_t)sk] : 0.0;
}

// what a chunk's operands hold (flags of a chunk; side 0: rows of op(A), side 1: columns of op(B))
enum : int {
  kUnsplittable = 1,             // an entry that is not finite, a scale outside the split form's range
  kOne = 2, kSeveral = 4,        // side 0 has a row with one entry that is not zero, with several
  kOneB = 8, kSeveralB = 16      // side 1
};

// digits of the held entries into the planes dg[NS][TILE][RS bytes] and the rows' biased exponents into
// ex[TILE] (0 for a row of zeros); returns the row's flags
template <int KI, int TILE>
__device__ __forceinline__ int store_digits(const double (&v)[4 * KI], int steps, int* ex, unsigned char* dg, int w,
                                            int lane) {
  constexpr int RS = 32 * KI + 16, PL = TILE * RS;
  uint32_t m = 0, any = 0, sum = 0;  // largest exponent field, all low words, the sum of the exponent fields
#pragma unroll
  for (int s = 0; s < KI; ++s)
    if (s < steps)
#pragma unroll
      for (int i = 4 * s; i < 4 * s + 4; ++i) {
        const uint32_t e2 = 2u * (uint32_t)__double2hiint(v[i]);
        m = max(m, e2);
        sum += e2 >> 21;
        any |= (uint32_t)__double2loint(v[i]);
      }
  any |= m;
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {
    m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    any |= __shfl_xor_sync(0xffffffffu, any, o);
  }
  // the next power of two, or the one after it for a largest entry above 127 / 128 of it, whose first digit
  // could be 128
  const int E = any == 0 ? 1023 : (int)((m + (1u << 15)) >> 21), r = 8 * w + (lane & 7);
  if (lane < 8) ex[r] = any == 0 ? 0 : E;
  unsigned char* d = dg + r * RS + 4 * (lane >> 3);
#pragma unroll
  for (int i = 0; i < 2 * KI; ++i)
    if (i / 2 < steps) {
      uint32_t dp[NS];
      digit_pairs(fixed_digits(v[2 * i], E), fixed_digits(v[2 * i + 1], E), dp);
#pragma unroll
      for (int s = 0; s < NS; ++s) *reinterpret_cast<uint32_t*>(d + 16 * i + s * PL) = dp[s];
    }
  const int top = (int)(m >> 21);
  return (any != 0 && (top < kLowExp || top > kHighExp) ? kUnsplittable : 0) |
         (sum > (m >> 21) ? kSeveral : any != 0 ? kOne : 0);
}

// a chunk's operands: entry (r, k) of op(A) (rows m) or op(B)^T (rows n) at r * sr + k * sk
struct Chunk {
  const double *a, *b;
  int asr, ask, bsr, bsk, len;
  double alpha;
};

// a warp's k of a chunk: all of them, in a 16 x 16 tile those of every other K step
template <int TILE>
__device__ __forceinline__ int nth_k(int i, int ks0) { return TILE == 16 ? 32 * (i >> 4) + 16 * ks0 + (i & 15) : i; }
template <int TILE>
__device__ __forceinline__ int num_k(int len, int ks0) {
  return TILE == 16 ? (len >> 5) * 16 + min(16, max(0, (len & 31) - 16 * ks0)) : len;
}

template <int TILE, bool SCALED>
__device__ __forceinline__ void plain_sums(const Chunk& ch, const double* const (&a)[2], const double* const (&b)[2],
                                           int ks0, double (&facc)[4]) {
  const int n = num_k<TILE>(ch.len, ks0);
#pragma unroll 2
  for (int i = 0; i < n; ++i) {
    const int64_t k = nth_k<TILE>(i, ks0);
    double x[2] = {a[0][k * ch.ask], a[1][k * ch.ask]};
    const double y[2] = {b[0][k * ch.bsk], b[1][k * ch.bsk]};
    if (SCALED) {
      x[0] *= ch.alpha;
      x[1] *= ch.alpha;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) facc[q] = fma(x[q >> 1], y[q & 1], facc[q]);
  }
}

// a warp's m16 x n8 sub-tile of a chunk in plain FP64, added to facc; rows and columns past the tile's edge
// repeat its last ones and are not written
template <int TILE>
__device__ __forceinline__ void plain_products(const Chunk& ch, int mt, int nt, int m0, int n0, int ks0, int lane,
                                               double (&facc)[4]) {
  const double *a[2], *b[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    a[h] = ch.a + (int64_t)min(m0 + (lane >> 2) + 8 * h, mt - 1) * ch.asr;
    b[h] = ch.b + (int64_t)min(n0 + 2 * (lane & 3) + h, nt - 1) * ch.bsr;
  }
  // two loops: FP64 multiplications under a predicate that is off take their time all the same (one-site
  // transfer matrix of the identity, XXZ D = 512: 43 us, 32 so)
  if (ch.alpha == 1.0) plain_sums<TILE, false>(ch, a, b, ks0, facc);
  else plain_sums<TILE, true>(ch, a, b, ks0, facc);
}

// one output of a chunk in plain FP64 by eight lanes (sub: the lane's number among them), in each of them
template <int TILE, bool SCALED>
__device__ __forceinline__ double plain_output(const Chunk& ch, int m, int n, int ks0, int sub) {
  const double *a = ch.a + (int64_t)m * ch.asr, *b = ch.b + (int64_t)n * ch.bsr;
  const int nk = num_k<TILE>(ch.len, ks0);
  double s = 0.0;
#pragma unroll 2
  for (int i = sub; i < nk; i += 8) {
    const int64_t k = nth_k<TILE>(i, ks0);
    double x = a[k * ch.ask];
    if (SCALED) x *= ch.alpha;
    s = fma(x, b[k * ch.bsk], s);
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// the products of a warp's m16 x n8 sub-tile over the chunk's K steps (16 x 16 tiles: every other one), added
// to facc
// |256 d_0 + d_1| of two entries, to FP16
__device__ __forceinline__ uint32_t magnitude(uint32_t d0, uint32_t d1) {
  const __half2 h = __hfma2(*reinterpret_cast<const __half2*>(&d0), __half2half2(__ushort_as_half(0x5c00)),  // 256
                            *reinterpret_cast<const __half2*>(&d1));
  return *reinterpret_cast<const uint32_t*>(&h) & 0x7fff7fffu;
}

template <int KI, int TILE>
__device__ __forceinline__ void chunk_products(const unsigned char* da, const unsigned char* db, const int* ea,
                                               const int* eb, unsigned char* list, const Chunk& ch, int mt, int nt,
                                               int m0, int n0, int ks0, int lane, double (&facc)[4]) {
  constexpr int RS = 32 * KI + 16, PL = TILE * RS;
  const int steps = (ch.len + 15) >> 4;
  float acc[NS][4], mag[4] = {0.f, 0.f, 0.f, 0.f};  // level sums; magnitude sums
#pragma unroll
  for (int l = 0; l < NS; ++l)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[l][q] = 0.f;
  // ldmatrix lane addresses: A rows 0-15 x (k 0-7, 8-15); B rows (n) 0-7 x (k 0-7, 8-15)
  const uint32_t aa = smem_addr(da) + (m0 + (lane & 15)) * RS + (lane >> 4) * 16;
  const uint32_t ba = smem_addr(db) + (n0 + (lane & 7)) * RS + ((lane >> 3) & 1) * 16;
  for (int ks = ks0; ks < steps; ks += TILE == 16 ? 2 : 1) {
    uint32_t b[NS][2], ma[4];
#pragma unroll
    for (int s = 0; s < NS; ++s) ldsm2(b[s], ba + s * PL + ks * 32);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      uint32_t a[4];
      ldsm4(a, aa + i * PL + ks * 32);
#pragma unroll
      for (int s = 0; s + i < NS; ++s) mma_f16(acc[i + s], a, b[s][0], b[s][1]);
      if (i == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) ma[q] = a[q];
      if (i == 1) {
#pragma unroll
        for (int q = 0; q < 4; ++q) ma[q] = magnitude(ma[q], a[q]);
        mma_f16(mag, ma, magnitude(b[0][0], b[1][0]), magnitude(b[0][1], b[1][1]));
      }
    }
  }
  double w[4];
  bool bad[4];
  int nbad = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    int L[NS];
#pragma unroll
    for (int l = 0; l < NS; ++l) L[l] = __float2int_rn(acc[l][q]);
    // sum of L[l] 2^(-8 l) in units of 2^-56, as hi 2^32 + lo, and its highest 64 bits as w 2^(32 - z)
    int64_t hi = ((int64_t)((L[0] << 8) + L[1]) << 16) + ((L[2] << 8) + L[3]);
    const int64_t lo = ((int64_t)((L[4] << 8) + L[5]) << 16) + ((int64_t)L[6] << 8) + L[7];
    hi += lo >> 32;
    const int z = min(__clzll(hi ^ (hi >> 63)) - 1, 32);
    const double v = (double)((hi << z) + (int64_t)(((uint64_t)(uint32_t)lo << z) >> 32));
    // times 2^(ea + eb - 2044 - 70 + 32 - z), by the exponent field (in range: see kLowExp, kHighExp)
    const int m = m0 + (lane >> 2) + (q & 2 ? 8 : 0), n = n0 + 2 * (lane & 3) + (q & 1);
    const int sa = ea[m], sb = eb[n], s = sa + sb - 2082 - z;
    w[q] = v == 0.0 ? 0.0 : __hiloint2double(__double2hiint(v) + (s << 20), __double2loint(v));
    bad[q] = mag[q] < kTrusted && sa != 0 && sb != 0 && m < mt && n < nt;
    nbad += __popc(__ballot_sync(0xffffffffu, bad[q]));
  }
  // outputs that the digits do not hold well enough: all at once (256 cycles of the FP64 pipe for every k), or
  // four at a time (eight for every k and 200)
  if (nbad > 0) {
    const int nk = num_k<TILE>(ch.len, ks0);
    if (nbad * (8 * nk + 200) > 1024 * nk) {
      plain_products<TILE>(ch, mt, nt, m0, n0, ks0, lane, facc);
      return;
    }
    int at = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t all = __ballot_sync(0xffffffffu, bad[q]);
      if (bad[q]) list[at + __popc(all & ((1u << lane) - 1))] = (unsigned char)(4 * lane + q);
      at += __popc(all);
    }
    __syncwarp();
    for (int r = 0; r < nbad; r += 4) {
      const int id = list[min(r + (lane >> 3), nbad - 1)], l = id >> 2;
      const int m = m0 + (l >> 2) + (id & 2 ? 8 : 0), n = n0 + 2 * (l & 3) + (id & 1);
      const double s = ch.alpha == 1.0 ? plain_output<TILE, false>(ch, m, n, ks0, lane & 7)
                                       : plain_output<TILE, true>(ch, m, n, ks0, lane & 7);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int to = __shfl_sync(0xffffffffu, id, 8 * g);
        const double x = __shfl_sync(0xffffffffu, s, 8 * g);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (to == 4 * lane + q) w[q] = x;
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) facc[q] = fma(bad[q] ? 1.0 : ch.alpha, w[q], facc[q]);
}

template <int KI, int TILE>
__global__ void __launch_bounds__(TILE * 8, TILE == 32 ? 2 : 4)
grouped_gemm_f64_kernel(const Tile* __restrict__ tiles, const Term* __restrict__ terms,
                        const __grid_constant__ imps_planes planes, double* ws, int* cnt) {
  constexpr int RS = 32 * KI + 16, PL = TILE * RS;
  constexpr int NW = TILE / 8;  // warps per operand
  extern __shared__ __align__(16) unsigned char digits[];
  __shared__ int ex[2 * TILE];
  __shared__ int flags[2];  // of an even and an odd chunk
  __shared__ int last;
  __shared__ unsigned char lists[TILE / 4][128];  // outputs of a warp that plain FP64 has to compute
  imps::allow_successor();
  const imps_dslots& slots = planes.s[blockIdx.y];
  if (threadIdx.x == 0) flags[0] = flags[1] = 0;
  __syncthreads();
  const Tile tl = tiles[blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // one half of the warps splits op(A), the other op(B), eight rows each (rows past the tile's edge
  // are left as they are: they reach no output that is written); then each warp takes one 16 x 8
  // sub-tile, in a 16 x 16 tile with every other K step
  const int side = warp / NW, w4 = warp % NW;
  const bool tall = tl.mt > 16;
  const int m0 = TILE == 32 && tall ? (warp & 1) * 16 : 0;
  const int n0 = TILE == 16 ? (warp & 1) * 8 : (tall ? warp >> 1 : warp) * 8;
  const int ks0 = TILE == 16 ? warp >> 1 : 0;
  const bool mine = n0 < tl.nt, splits = 8 * w4 < (side ? tl.nt : tl.mt);
  double facc[4] = {0.0, 0.0, 0.0, 0.0};

  Chunk cur{}, prev{};
  double v[4 * KI];
  bool direct = false;  // the split chunk is to be computed by plain FP64
  int t = tl.t0, c = tl.c0;
  if (tl.nch > 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(terms + t));
  imps::wait_for_predecessor();  // the tables are the plan's own; operands may be its predecessor's results
  // iteration it: load chunk it, multiply chunk it - 1 under the loads, split chunk it
  for (int it = 0;; ++it) {
    if (it < tl.nch) {
      Term tm = terms[t];
      while (c * tm.kc >= tm.k) {  // this term is done
        c = 0;
        tm = terms[++t];
      }
      const int k0 = c * tm.kc;
      ++c;
      cur.len = min((int)tm.kc, tm.k - k0);
      cur.alpha = tm.alpha;
      cur.asr = tm.a_t ? tm.a_ld : 1;
      cur.ask = tm.a_t ? 1 : tm.a_ld;
      cur.bsr = tm.b_t ? 1 : tm.b_ld;
      cur.bsk = tm.b_t ? tm.b_ld : 1;
      cur.a = slots.p[tm.a_slot] + tm.a_off + (int64_t)tl.m0 * cur.asr + (int64_t)k0 * cur.ask;
      cur.b = slots.p[tm.b_slot] + tm.b_off + (int64_t)tl.n0 * cur.bsr + (int64_t)k0 * cur.bsk;
      if (splits)
        load_operand<KI>(v, side ? cur.b : cur.a, side ? cur.bsr : cur.asr, side ? cur.bsk : cur.ask,
                         side ? tl.nt : tl.mt, cur.len, w4, lane);
    }
    if (it > 0) {
      if (mine && 16 * ks0 < prev.len) {
        if (direct)
          plain_products<TILE>(prev, tl.mt, tl.nt, m0, n0, ks0, lane, facc);
        else
          chunk_products<KI, TILE>(digits, digits + NS * PL, ex, ex + TILE, lists[warp], prev, tl.mt, tl.nt, m0, n0,
                                   ks0, lane, facc);
      }
      if (it == tl.nch) break;
      __syncthreads();  // the previous chunk's digits are no longer read
    } else if (tl.nch == 0) {
      break;
    }
    if (splits) {
      const int f = store_digits<KI, TILE>(v, (cur.len + 15) >> 4, ex + TILE * side, digits + side * NS * PL, w4, lane);
      const int fs = (f & kUnsplittable) | (side ? (f & (kOne | kSeveral)) * (kOneB / kOne) : f & (kOne | kSeveral));
      if (lane < 8 && 8 * w4 + lane < (side ? tl.nt : tl.mt)) atomicOr(&flags[it & 1], fs);
    }
    __syncthreads();
    // An operand whose rows (columns) hold one entry each at most selects and scales the other's
    // entries: plain FP64 gives each product its own 53 bits.
    const int f = flags[it & 1];
    direct = (f & kUnsplittable) || (f & (kOne | kSeveral)) == kOne || (f & (kOneB | kSeveralB)) == kOneB;
    if (threadIdx.x == 0) flags[(it + 1) & 1] = 0;  // written again after the next barrier
    prev = cur;
  }
  bool writes = mine;
  if (TILE == 16) {  // the two halves of the K steps
    __shared__ double half[64 * 4];
    if (ks0 == 1)
#pragma unroll
      for (int q = 0; q < 4; ++q) half[q * 64 + threadIdx.x - 64] = facc[q];
    __syncthreads();
    writes = mine && ks0 == 0;
    if (ks0 == 0)
#pragma unroll
      for (int q = 0; q < 4; ++q) facc[q] += half[q * 64 + threadIdx.x];
  }

  if (tl.nparts > 1) {
    constexpr int WT = TILE * TILE / 4;  // threads that hold outputs
    // partial tile -> workspace; the last CTA of the tile sums all partials in share order
    ws += blockIdx.y * planes.ws_len;
    cnt += blockIdx.y * planes.cnt_len;
    double* wp = ws + ((int64_t)tl.ws_unit + tl.part) * (TILE * TILE) + threadIdx.x;
    if (writes)
#pragma unroll
      for (int q = 0; q < 4; ++q) wp[q * WT] = facc[q];
    __syncthreads();
    if (threadIdx.x == 0) {  // the barrier orders the CTA's stores before this thread's fences
      __threadfence();
      last = atomicAdd(cnt + tl.cnt_idx, 1) == tl.nparts - 1;
      __threadfence();
    }
    __syncthreads();
    if (!last) return;
    const double* wr = ws + (int64_t)tl.ws_unit * (TILE * TILE) + threadIdx.x;
    if (writes) {
#pragma unroll
      for (int q = 0; q < 4; ++q) facc[q] = 0.0;
#pragma unroll 4
      for (int p = 0; p < tl.nparts; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) facc[q] += __ldcg(wr + p * (TILE * TILE) + q * WT);
    }
    if (threadIdx.x == 0) cnt[tl.cnt_idx] = 0;  // re-armed for the next launch of this stage
  }
  if (!writes) return;
  double* C = slots.p[tl.c_slot] + tl.c_off;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int m = m0 + (lane >> 2) + (q & 2 ? 8 : 0), n = n0 + 2 * (lane & 3) + (q & 1);
    if (m >= tl.mt || n >= tl.nt) continue;
    double* p = C + (tl.m0 + m) + (int64_t)(tl.n0 + n) * tl.c_ld;
    *p = tl.accumulate ? *p + facc[q] : facc[q];
  }
}

template <int TILE>
constexpr int smem_bytes(int ki) { return 2 * NS * TILE * (32 * ki + 16); }

using KernelFn = void (*)(const Tile*, const Term*, imps_planes, double*, int*);
template <int TILE>
KernelFn kernel_of(int ki) {
  switch (ki) {
    case 1: return grouped_gemm_f64_kernel<1, TILE>;
    case 2: return grouped_gemm_f64_kernel<2, TILE>;
    case 3: return grouped_gemm_f64_kernel<3, TILE>;
    case 4: return grouped_gemm_f64_kernel<4, TILE>;
    case 5: return grouped_gemm_f64_kernel<5, TILE>;
    default: return nullptr;
  }
}

template <int TILE>
int setup() {
  for (int ki = 1; ki <= imps::kMaxKSteps; ++ki)
    if (cudaFuncSetAttribute((const void*)kernel_of<TILE>(ki), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem_bytes<TILE>(ki)) != cudaSuccess)
      return IMPS_ERR_CUDA;
  return IMPS_OK;
}

}  // namespace

int imps_f64_setup() {
  const int rc = setup<16>();
  return rc ? rc : setup<32>();
}

int imps_launch_grouped_f64(const void* d_tiles, int ntiles, const void* d_terms, imps_dslots slots, int tile,
                            int ksteps, int splits, double* ws, int* cnt, void* stream) {
  imps_planes one{};
  one.s[0] = slots;
  one.n = 1;
  return imps_launch_grouped_f64(d_tiles, ntiles, d_terms, one, tile, ksteps, splits, ws, cnt, stream);
}

int imps_launch_grouped_f64(const void* d_tiles, int ntiles, const void* d_terms, const imps_planes& planes, int tile,
                            int ksteps, int splits, double* ws, int* cnt, void* stream, bool after_tables) {
  if (ntiles <= 0) return IMPS_OK;
  if (planes.n < 1 || planes.n > 2 || splits < 1 || (splits > 1 && (!ws || !cnt)) || (tile != 16 && tile != 32))
    return IMPS_ERR_BAD_ARG;
  KernelFn fn = tile == 16 ? kernel_of<16>(ksteps) : kernel_of<32>(ksteps);
  if (!fn) return IMPS_ERR_BAD_ARG;
  imps::count_launch();
  const int smem = tile == 16 ? smem_bytes<16>(ksteps) : smem_bytes<32>(ksteps);
  if (after_tables) {
    fn<<<dim3(ntiles, planes.n), dim3(tile * 8), smem, (cudaStream_t)stream>>>((const Tile*)d_tiles,
                                                                               (const Term*)d_terms, planes, ws, cnt);
    return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
  }
  const cudaError_t e = imps::launch_overlapped(fn, dim3(ntiles, planes.n), dim3(tile * 8), smem, (cudaStream_t)stream,
                                                (const Tile*)d_tiles, (const Term*)d_terms, planes, ws, cnt);
  return e == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}
