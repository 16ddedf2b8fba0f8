// Tensor-core (tcgen05, sm_103a) execution of planner stages in split-BF16 precision.
//
// Every FP64 operand x is split as x = hi + mid + lo with hi, mid, lo in BF16; a product is
// formed from the six terms hi*hi + hi*mid + mid*hi + hi*lo + mid*mid + lo*hi (the dropped
// terms are O(2^-24) relative), accumulated in FP32 in tensor memory, and written back to
// the FP64 output.  Operands are packed once into the canonical UMMA layout (K-major, no
// swizzle: 8 rows x 16 bytes core matrices; LBO = stride between the two 8-element K
// chunks, SBO = stride between 8-row groups = 128 B):
//     packed[kstep][split][chunk][row group][8 rows][8 bf16]
// so that the two K-steps of one pipeline stage are one contiguous bulk copy.
//
// Kernel roles (256 threads, one CTA per output tile of <= 128 x 128):
//   warp 0 lane 0 : producer, cp.async.bulk global -> shared, mbarrier complete_tx
//   warp 1 lane 0 : MMA issuer, tcgen05.mma.cta_group::1.kind::f16 into TMEM, tcgen05.commit
//   warps 0-7     : epilogue, tcgen05.ld 32x32b -> FP64 global
// Every mbarrier wait is bounded; on timeout the CTA records an error, drains what it
// issued (bounded), frees its TMEM and returns.
//
// What bounds it: the chain of the longest tile, 40 K steps of 6 matrix instructions at 64 cycles each
// whatever their N, some 270 cycles of barriers a stage, and the epilogue.  So two CTAs share an SM, the
// longest tiles start first and the launches overlap; the issuing warp runs its loop as one (a lone lane spent
// 830 cycles a K step, on descriptors, table reads and the abort flag; now 500); and eight warps write the
// outputs, widened by integer operations at stepped pointers (11,400 -> 3,900 cycles for 96 columns).  A
// operands hold their own rows only.  H_AC apply at Hubbard D = 1024 (209 tiles): 50.1 us with one CTA of
// four stages per SM in table order and the pack kernel's former stores, 28.4 with two, 20.7 now.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <map>
#include <tuple>
#include <vector>

#include "imps_status.h"
#include "imps_tc.h"

namespace imps {

namespace {

constexpr int TC_M = 128;        // UMMA M (rows of every tile, zero padded)
constexpr int TC_NMAX = 128;     // max UMMA N per tile
constexpr int TC_NSTAGE = 8;     // most pipeline stages
constexpr int TC_THREADS = 256;
constexpr int PIPE_BYTES = 98304;  // of the pipeline's stages
// pipeline + alignment slack + headroom so that every descriptor-addressed access stays inside this
// CTA's allocation; two CTAs fit an SM
constexpr int SMEM_BYTES = 106496;  // 104 KB
static_assert(PIPE_BYTES + TC_M * 16 + 1024 <= SMEM_BYTES, "tcgen05 pipeline does not fit");
constexpr uint32_t WAIT_LIMIT = 1u << 24;

struct TcTerm {
  int64_t a_off, b_off;  // bf16 element offsets into the packed buffer
  int32_t ksteps;        // padded K / 16
  int32_t pad;
};

struct TcTile {
  int64_t c_off;
  int32_t c_ld, m, n, npad;
  int32_t t0, t1;
  int16_t c_slot, accumulate;
  int16_t mpad;             // rows of A as packed
  int8_t kstage, nstage;    // K steps of a pipeline stage, stages
};

struct PackJob {
  int64_t src_off;
  int64_t dst_off;  // bf16 elements
  int32_t src_ld;
  int32_t trans;    // stored matrix is op()^T
  int32_t role;     // 0: A (rows = M), 1: B (rows = N)
  int32_t rows, k;  // valid rows of this tile slice, valid K
  int32_t rpad, kpad;
  int32_t r0;       // first row (A: m0, B: n0) of the slice
  int32_t slot;
  int32_t pad;
  double alpha;
};

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// bounded wait for the phase with the given parity; returns false on timeout, or once *abort is set (it is
// looked at only while the phase is not there)
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const int* abort = nullptr) {
  const uint32_t a = smem_u32(bar);
  for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if (abort && *(const volatile int*)abort) return false;
  }
  return false;
}

__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (tcgen05)
  // base offset 0, LBO mode relative, layout type 0 = no swizzle
  return d;
}

// kind::f16 instruction descriptor: D fp32, A/B bf16, both K-major, N>>3 @17, M>>4 @24
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------------------------ kernels
// One job per blockIdx.x; its padded rpad x kpad operand in items of eight k of a row, lanes along the
// rows: an item's BF16 values of one split are the 16 bytes of one core matrix row, so a warp stores
// 512 contiguous bytes per split.  The FP64 value is rounded once to FP32 and split there into hi + mid
// + lo BF16 terms: each difference xf - bf16(xf) is exact in FP32, so the three terms carry all 24
// significand bits of xf (relative error 2^-24, the order of the dropped lo*lo-type products) while the
// FP64 pipe, slow on this GPU, sees one conversion per element, its bound.  Hubbard D = 1024 H_AC: 17.7
// us a launch on average with one element per thread, its index divided by rpad and three scattered
// 2-byte stores; 10.0 now.
__global__ void __launch_bounds__(256) pack_kernel(const PackJob* __restrict__ jobs,
                                                   const __grid_constant__ imps_dslots slots, __nv_bfloat16* out) {
  imps::allow_successor();
  const PackJob jb = jobs[blockIdx.x];
  const double* S = slots.p[jb.slot] + jb.src_off;
  const int rpad = jb.rpad, lane = threadIdx.x & 31;
  const float alpha = (float)jb.alpha;
  const int split_elems = rpad * 16;
  // entry (row, k) of the operand's row-major form: at row * sr + k * sk
  const bool kfast = (jb.role == 0) == (jb.trans != 0);
  const int64_t sr = kfast ? jb.src_ld : 1, sk = kfast ? 1 : jb.src_ld;
  const int octets = jb.kpad >> 3, wide = (rpad + 31) >> 5;  // items: octet * wide + row group of 32
  imps::wait_for_predecessor();
  for (int it = blockIdx.y * 8 + (threadIdx.x >> 5); it < octets * wide; it += gridDim.y * 8) {
    const int oct = it / wide, r = (it - oct * wide) * 32 + lane;
    if (r >= rpad) continue;
    const int k0 = oct * 8;
    float xf[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
      xf[e] = r < jb.rows && k0 + e < jb.k
                  ? __double2float_rn(S[(int64_t)(jb.r0 + r) * sr + (int64_t)(k0 + e) * sk]) * alpha
                  : 0.0f;
    __nv_bfloat162 w[3][4];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const __nv_bfloat16 hi = __float2bfloat16_rn(xf[e]);
      const float x1 = xf[e] - __bfloat162float(hi);
      const __nv_bfloat16 mid = __float2bfloat16_rn(x1);
      const float x2 = x1 - __bfloat162float(mid);
      const __nv_bfloat16 lo = __float2bfloat16_rn(x2);
      __nv_bfloat16* p[3] = {&w[0][e >> 1].x, &w[1][e >> 1].x, &w[2][e >> 1].x};
      p[0][e & 1] = hi;
      p[1][e & 1] = mid;
      p[2][e & 1] = lo;
    }
    __nv_bfloat16* d = out + jb.dst_off + (int64_t)(oct >> 1) * 3 * split_elems + (int64_t)(oct & 1) * rpad * 8 + r * 8;
#pragma unroll
    for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(d + q * split_elems) = *reinterpret_cast<const uint4*>(w[q]);
  }
}

// (double)x by integer operations where x is normal or zero: the conversion runs on the FP64 pipe, 64 cycles a
// warp
__device__ __forceinline__ double widen(float x) {
  const uint32_t b = __float_as_uint(x), mag = b & 0x7fffffffu;
  if (mag - 0x00800000u < 0x7f000000u)
    return __hiloint2double((int)((b & 0x80000000u) | ((mag >> 3) + 0x38000000u)), (int)(b << 29));
  return mag == 0 ? __hiloint2double((int)b, 0) : (double)x;
}

__global__ void __launch_bounds__(TC_THREADS, 2)
tc_gemm_kernel(const TcTile* __restrict__ tiles, const TcTerm* __restrict__ terms, const __nv_bfloat16* packed,
               const __grid_constant__ imps_dslots slots, int* err) {
  imps::allow_successor();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[TC_NSTAGE];
  __shared__ __align__(8) uint64_t empty_bar[TC_NSTAGE];
  __shared__ __align__(8) uint64_t done_bar;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  const TcTile tl = tiles[blockIdx.x];
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t ncols = 128;  // TMEM columns (power of two >= npad)
  if (threadIdx.x == 0) {
    for (int s = 0; s < TC_NSTAGE; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    __syncwarp();  // thread 0 comes from the barriers' initialisation
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  imps::wait_for_predecessor();  // the packed operands are its predecessor's
  const int nterm = tl.t1 - tl.t0;
  const uint32_t idesc = idesc_bf16(TC_M, tl.npad);
  // one split of one K-step.  A holds mpad rows: the rows of an MMA past them read what follows in shared
  // memory, and their outputs are not written
  const uint32_t a_split_bytes = (uint32_t)tl.mpad * 32;
  const uint32_t b_split_bytes = (uint32_t)tl.npad * 32;
  const int kstage = tl.kstage, nstage = tl.nstage;
  const uint32_t a_stage_bytes = kstage * 3 * a_split_bytes, stage_bytes = a_stage_bytes + kstage * 3 * b_split_bytes;
  int issued = 0;  // stages filled (by the producer)

  if (warp == 0 && lane == 0 && nterm > 0) {
    // ---------------- producer
    asm volatile("fence.proxy.async;" ::: "memory");  // the packs were written through the generic proxy
    int s = 0;
    uint32_t u = 0;  // stage, and how often it has been filled before
    bool ok = true;
    TcTerm next = terms[tl.t0];
    const uint32_t a_step = 3 * a_split_bytes, b_step = 3 * b_split_bytes;  // of one K step
    for (int t = tl.t0; t < tl.t1 && ok; ++t) {
      const TcTerm tm = next;
      if (t + 1 < tl.t1) next = terms[t + 1];  // on its way meanwhile
      const uint8_t* ga = (const uint8_t*)(packed + tm.a_off);
      const uint8_t* gb = (const uint8_t*)(packed + tm.b_off);
      for (int ks = 0; ks < tm.ksteps; ks += kstage) {
        if (u > 0 && !mbar_wait(&empty_bar[s], (u & 1) ^ 1, &abort_s)) { ok = false; break; }
        const int nk = min(kstage, tm.ksteps - ks);
        const uint32_t abytes = nk * a_step, bbytes = nk * b_step;
        uint8_t* sa = smem + s * stage_bytes;
        uint8_t* sb = sa + a_stage_bytes;
        mbar_expect_tx(&full_bar[s], abytes + bbytes);
        bulk_g2s(sa, ga, abytes, &full_bar[s]);
        bulk_g2s(sb, gb, bbytes, &full_bar[s]);
        ga += abytes;
        gb += bbytes;
        ++issued;
        if (++s == nstage) { s = 0; ++u; }
      }
    }
    if (!ok) { atomicExch(err, 1); abort_s = 1; }
  } else if (warp == 1 && nterm > 0) {
    // ---------------- MMA issuer: the whole warp runs the loop, one elected lane issues
    const bool leader = elect_one();
    const uint32_t a_step = a_split_bytes >> 4, b_step = b_split_bytes >> 4, stage_step = stage_bytes >> 4;
    // descriptors of a stage's first core matrices; the others' lie whole multiples of a split further
    const uint64_t ad0 = smem_desc(smem_u32(smem), tl.mpad * 16, 128);
    const uint64_t bd0 = smem_desc(smem_u32(smem) + a_stage_bytes, tl.npad * 16, 128);
    int s = 0, next = terms[tl.t0].ksteps;
    uint32_t accum = 0, u = 0;
    bool ok = true;
    for (int t = tl.t0; t < tl.t1 && ok; ++t) {
      const int ksteps = next;
      if (t + 1 < tl.t1) next = terms[t + 1].ksteps;  // on its way meanwhile
      for (int ks = 0; ks < ksteps; ks += kstage) {
        if (!mbar_wait(&full_bar[s], u & 1, &abort_s)) { ok = false; break; }
        tc_fence_after();
        if (leader) {
          const int nk = min(kstage, ksteps - ks);
          uint64_t ad = ad0 + s * stage_step, bd = bd0 + s * stage_step;
          for (int k = 0; k < nk; ++k, ad += 3 * a_step, bd += 3 * b_step) {
            // split pairs (a, b): hh, hm, mh, hl, mm, lh
            const uint64_t am = ad + a_step, al = am + a_step, bm = bd + b_step, bl = bm + b_step;
            mma_bf16(tmem, ad, bd, idesc, accum);
            accum = 1;
            mma_bf16(tmem, ad, bm, idesc, 1);
            mma_bf16(tmem, am, bd, idesc, 1);
            mma_bf16(tmem, ad, bl, idesc, 1);
            mma_bf16(tmem, am, bm, idesc, 1);
            mma_bf16(tmem, al, bd, idesc, 1);
          }
          mma_commit(&empty_bar[s]);  // frees the stage once these MMAs have read it
        }
        if (++s == nstage) { s = 0; ++u; }
      }
    }
    if (leader) {
      if (!ok) { atomicExch(err, 1); abort_s = 1; }
      mma_commit(&done_bar);  // arrives when every MMA issued above has completed
    }
    __syncwarp();
  }
  __syncthreads();  // role lanes rejoin their warps before the warp-collective TMEM loads
  // ---------------- epilogue
  double* C = slots.p[tl.c_slot] + tl.c_off;
  bool have = nterm > 0;
  if (have) {
    if (!mbar_wait(&done_bar, 0)) { atomicExch(err, 1); have = false; }
    tc_fence_after();
  }
  have = __all_sync(0xffffffffu, have);
  __syncwarp();
  // warps w and w + 4 take the rows of TMEM lanes 32 (w % 4) .., every other 16 columns each
  const int row = (warp & 3) * 32 + lane;
  const bool acc = tl.accumulate != 0;
  const int64_t ldc = tl.c_ld;
  double* p = C + row + (warp >> 2) * 16 * ldc;
  for (int c0 = (warp >> 2) * 16; c0 < tl.npad; c0 += 32) {
    float v[16];
    if (have) {
      tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = 0.f;
    }
    if (row < tl.m) {
      if (!acc && c0 + 16 <= tl.n) {
#pragma unroll
        for (int i = 0; i < 16; ++i) p[i * ldc] = widen(v[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (c0 + i < tl.n) p[i * ldc] = acc ? p[i * ldc] + widen(v[i]) : widen(v[i]);
      }
    }
    p += 32 * ldc;
  }
  // producer drains its copies if it aborted (bounded), then TMEM is released
  if (warp == 0 && lane == 0 && abort_s) {
    for (int i = max(0, issued - nstage); i < issued; ++i) mbar_wait(&full_bar[i % nstage], (i / nstage) & 1);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

}  // namespace

// ------------------------------------------------------------------ host side
struct TcStage {
  std::vector<TcTile> tiles;
  std::vector<TcTerm> terms;
  std::vector<PackJob> dyn_jobs;  // packed before every run of the stage
  TcTile* d_tiles = nullptr;
  TcTerm* d_terms = nullptr;
  PackJob* d_dyn = nullptr;
};

struct TcPlan {
  std::vector<TcStage> stages;         // parallel to Plan::stages
  std::vector<PackJob> static_jobs;    // packed at prepare time
  PackJob* d_static = nullptr;
  __nv_bfloat16* packed = nullptr;
  int64_t packed_elems = 0;
  int* d_err = nullptr;
  bool static_valid = false;
  std::vector<char> dynamic_slot;
  const Stage* first_stage = nullptr;
};

static int round_up(int x, int m) { return (x + m - 1) / m * m; }

int tc_create(TcPlan** out, const Plan& P, cudaStream_t st) {
  TcPlan* T = new TcPlan();
  T->dynamic_slot.assign(P.slots.size(), 0);
  T->dynamic_slot[P.n_in] = 1;
  for (const Stage& S : P.stages)
    for (const OutBlock& o : S.outs) T->dynamic_slot[o.c_slot] = 1;
  std::map<std::tuple<int, int64_t, int, int, int, int, int, int, double>, int64_t> seen;
  int64_t off = 0;
  bool too_large = false;  // the pack kernel indexes one operand slice with 32-bit integers
  auto pack_for = [&](int slot, int64_t src, int ld, int trans, int role, int r0, int rows, int k, int rpad,
                      double alpha, std::vector<PackJob>& jobs) -> int64_t {
    const int kpad = round_up(std::max(k, 1), 16);
    if ((int64_t)rpad * kpad * 3 >= ((int64_t)1 << 31)) too_large = true;
    auto key = std::make_tuple(slot, src, ld, trans, role, r0, rows, k, alpha);
    auto it = seen.find(key);
    if (it != seen.end()) return it->second;
    PackJob j{};
    j.src_off = src; j.dst_off = off; j.src_ld = ld; j.trans = trans; j.role = role;
    j.rows = rows; j.k = k; j.rpad = rpad; j.kpad = kpad; j.r0 = r0; j.slot = slot; j.alpha = alpha;
    jobs.push_back(j);
    seen[key] = off;
    const int64_t o = off;
    off += (int64_t)3 * rpad * kpad;
    return o;
  };
  for (const Stage& S : P.stages) {
    TcStage ts;
    for (const OutBlock& o : S.outs) {
      for (int m0 = 0; m0 < std::max(o.M, 1); m0 += TC_M)
        for (int n0 = 0; n0 < std::max(o.N, 1); n0 += TC_NMAX) {
          TcTile tl{};
          tl.c_off = o.c_off + m0 + (int64_t)n0 * o.c_ld;
          tl.c_ld = std::max(o.c_ld, 1);
          tl.m = std::min(TC_M, o.M - m0);
          tl.n = std::min(TC_NMAX, o.N - n0);
          tl.npad = std::max(16, round_up(tl.n, 16));
          tl.mpad = (int16_t)std::max(8, round_up(tl.m, 8));
          // two K steps a stage (one: 18.4 us for the kernel at Hubbard D = 1024 instead of 16.1, as a stage
          // costs its barriers some 270 cycles), as many stages as fit: 2 of 128 x 128 to 8 of 48 x 16
          tl.kstage = 2;
          tl.nstage = (int8_t)std::min(TC_NSTAGE, PIPE_BYTES / (tl.kstage * 3 * 32 * (tl.mpad + tl.npad)));
          tl.c_slot = o.c_slot;
          tl.accumulate = o.accumulate;
          tl.t0 = (int)ts.terms.size();
          if (tl.m <= 0 || tl.n <= 0) continue;
          for (int t = o.t0; t < o.t1; ++t) {
            const Term& tm = S.terms[t];
            if (tm.k <= 0) continue;
            std::vector<PackJob>& ja = T->dynamic_slot[tm.a_slot] ? ts.dyn_jobs : T->static_jobs;
            std::vector<PackJob>& jb = T->dynamic_slot[tm.b_slot] ? ts.dyn_jobs : T->static_jobs;
            TcTerm tt{};
            tt.a_off = pack_for(tm.a_slot, tm.a_off, tm.a_ld, tm.a_t, 0, m0, tl.m, tm.k, tl.mpad, tm.alpha, ja);
            tt.b_off = pack_for(tm.b_slot, tm.b_off, tm.b_ld, tm.b_t, 1, n0, tl.n, tm.k, tl.npad, 1.0, jb);
            tt.ksteps = round_up(tm.k, 16) / 16;
            ts.terms.push_back(tt);
          }
          tl.t1 = (int)ts.terms.size();
          ts.tiles.push_back(tl);
        }
    }
    // the tiles with the most matrix instructions first
    auto work = [&](const TcTile& t) {
      int64_t k = 0;
      for (int e = t.t0; e < t.t1; ++e) k += ts.terms[e].ksteps;
      return k * t.npad;
    };
    std::stable_sort(ts.tiles.begin(), ts.tiles.end(),
                     [&](const TcTile& a, const TcTile& b) { return work(a) > work(b); });
    T->stages.push_back(std::move(ts));
  }
  T->packed_elems = off;
  auto up = [&](void** d, const void* h, size_t bytes) -> int {
    if (bytes == 0) return IMPS_OK;
    if (cudaMalloc(d, bytes) != cudaSuccess) return IMPS_ERR_OOM;
    if (cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice) != cudaSuccess) return IMPS_ERR_CUDA;
    return IMPS_OK;
  };
  int rc = too_large ? IMPS_ERR_TOO_LARGE : IMPS_OK;
  for (TcStage& ts : T->stages) {
    if (rc) break;
    if ((rc = up((void**)&ts.d_tiles, ts.tiles.data(), ts.tiles.size() * sizeof(TcTile)))) break;
    if ((rc = up((void**)&ts.d_terms, ts.terms.data(), ts.terms.size() * sizeof(TcTerm)))) break;
    if ((rc = up((void**)&ts.d_dyn, ts.dyn_jobs.data(), ts.dyn_jobs.size() * sizeof(PackJob)))) break;
  }
  if (!rc) rc = up((void**)&T->d_static, T->static_jobs.data(), T->static_jobs.size() * sizeof(PackJob));
  if (!rc && cudaMalloc(&T->packed, std::max<int64_t>(T->packed_elems, 8) * sizeof(__nv_bfloat16)) != cudaSuccess)
    rc = IMPS_ERR_OOM;
  if (!rc && cudaMalloc(&T->d_err, sizeof(int)) != cudaSuccess) rc = IMPS_ERR_OOM;
  if (!rc) cudaMemsetAsync(T->d_err, 0, sizeof(int), st);
  if (!rc) {
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) {
      fprintf(stderr, "imps_gb300: tcgen05 kernel setup failed: %s\n", cudaGetErrorString(e));
      rc = IMPS_ERR_CUDA;
    }
  }
  if (rc) { tc_destroy(T); return rc; }
  T->first_stage = P.stages.empty() ? nullptr : &P.stages[0];
  *out = T;
  return IMPS_OK;
}

int tc_destroy(TcPlan* T) {
  if (!T) return IMPS_OK;
  for (TcStage& ts : T->stages) { cudaFree(ts.d_tiles); cudaFree(ts.d_terms); cudaFree(ts.d_dyn); }
  cudaFree(T->d_static);
  cudaFree(T->packed);
  cudaFree(T->d_err);
  delete T;
  return IMPS_OK;
}

int tc_invalidate(TcPlan* T) {
  if (T) T->static_valid = false;
  return IMPS_OK;
}

static int launch_pack(const PackJob* d_jobs, int n, const imps_dslots& slots, __nv_bfloat16* out, cudaStream_t st) {
  if (n <= 0) return IMPS_OK;
  imps::count_launch();
  const cudaError_t e = imps::launch_overlapped(pack_kernel, dim3(n, 2), dim3(256), 0, st, d_jobs, slots, out);
  return e == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int tc_run_stage(TcPlan* T, const Stage& S, const imps_dslots& slots, cudaStream_t st) {
  // locate the stage index by address (stages are stored in the same order)
  size_t si = (size_t)(&S - T->first_stage);
  if (!T->first_stage || si >= T->stages.size()) return IMPS_ERR_BAD_ARG;
  if (!T->static_valid) {
    int rc = launch_pack(T->d_static, (int)T->static_jobs.size(), slots, T->packed, st);
    if (rc) return rc;
    T->static_valid = true;
  }
  TcStage& ts = T->stages[si];
  int rc = launch_pack(ts.d_dyn, (int)ts.dyn_jobs.size(), slots, T->packed, st);
  if (rc) return rc;
  if (!ts.tiles.empty()) {
    imps::count_launch();
    const cudaError_t e = imps::launch_overlapped(tc_gemm_kernel, dim3((unsigned)ts.tiles.size()), dim3(TC_THREADS),
                                                  SMEM_BYTES, st, ts.d_tiles, ts.d_terms, T->packed, slots, T->d_err);
    if (e != cudaSuccess) return IMPS_ERR_CUDA;
  }
  return IMPS_OK;
}

int tc_error_flag(TcPlan* T, int* flag) {
  if (!T || !flag) return IMPS_ERR_BAD_ARG;
  if (cudaMemcpy(flag, T->d_err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return IMPS_ERR_CUDA;
  return IMPS_OK;
}

}  // namespace imps
