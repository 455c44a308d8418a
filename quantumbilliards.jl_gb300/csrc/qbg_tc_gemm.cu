// Complex FP32 GEMM on the 5th-generation tensor cores (tcgen05, sm_103a).
//
//   C = alpha A B + beta C,  A: M x K, B: K x N, C: M x N complex64,
//   column-major, batched by blockIdx.z.
//
// Mapping of the complex product onto one real product D = A' B'^T:
//   A'[i][2k] = Re A(i,k), A'[i][2k+1] = Im A(i,k)                 (M x 2K)
//   B'[j][2k] = Re B(k,j), B'[j][2k+1] = -Im B(k,j)                 (rows 0..BN-1)
//   B'[BN+j][2k] = Im B(k,j), B'[BN+j][2k+1] = Re B(k,j)            (rows BN..2BN-1)
//   Re C(i,j) = D[i][j],  Im C(i,j) = D[i][BN+j].
// FP32 accuracy from TF32 units (3xTF32): every operand x is split as
// x = big + small with big = tf32(x), small = tf32(x - big), and
// D += A_big B_big + A_big B_small + A_small B_big (the dropped small*small
// term is ~2^-22 relative).
//
// One CTA (16 staging warps and one that issues) computes a tile of 128 x 32 or
// 128 x up to 128 complex (tcgen05.mma.cta_group::1.kind::tf32, M = 128, K = 8).
// The staging warps write the operands to shared memory in the canonical K-major layout without
// swizzle (8-row x 16-byte core matrices; LBO = 128 B between the two core
// matrices along K, SBO = 256 B between 8-row groups), in two stages of 16
// complex k; lane 0 of the last warp issues the
// MMAs and commits each stage to its own mbarrier; the accumulators live in
// TMEM and are read back with tcgen05.ld.32x32b. C is fetched into
// registers before the k loop. Every mbarrier wait is bounded: on timeout the
// kernel records an error, waits (bounded) for its own MMAs, frees its TMEM and
// returns without writing C.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <cstdlib>
#include <cstdint>
#include <mutex>
#include <vector>
#include "qbg_common.cuh"
#include "qbg_handles.cuh"
#include "qbg_linalg.cuh"

namespace qbg {
namespace {

constexpr int TC_BM = 128;        // rows of C per CTA
constexpr int TC_BN = 32;         // complex columns of C per CTA (real N = 64)
constexpr int TC_BK = 16;         // complex k per stage (real K = 32 = 4 MMA steps of 8)
constexpr int TC_KSTEPS = 4;
constexpr int TC_A_STEP = TC_BM * 8;        // floats per operand block per MMA step (4 KB)
// the staged kernel's tile widths: 32 complex columns (48 KB stages, two CTAs per
// SM) or up to 128 (96 KB stages, one)
template <bool WIDE> struct TS {
  static constexpr int BN = WIDE ? 128 : TC_BN, NB = BN / 32;  // columns, B elements per thread
  static constexpr int B_STEP = 2 * BN * 8;                    // floats of one half (big, small) of a step
  static constexpr int STAGE = 2 * TC_KSTEPS * (TC_A_STEP + B_STEP);
  static constexpr uint32_t TMEM = 4 * BN;                     // Re and Im of two accumulators
};
constexpr long long TC_SPIN_LIMIT = 1ll << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// x = big + small + O(2^-23 |x|), both rounded to tf32 (nearest, ties away from zero)
// on the integer unit: the conversion instruction's throughput showed as a stall of the
// staging warps (0.84 of 8.4 cycles an instruction, 0.65 so). A NaN leaves big finite
// (0x7fffffff wraps to -0) and stays in small, whose rounding is applied as a
// floating-point correction (exact: r - s is the rounding error of s); an
// infinity gives big = inf, small = NaN.
__device__ __forceinline__ void tf32_split(float x, float& big, float& small) {
  big = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  const float s = x - big;
  const float r = __uint_as_float((__float_as_uint(s) + 0x1000u) & 0xffffe000u);
  small = s + (r - s);
}

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
  const uint64_t lbo = 128, sbo = 256;
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= ((lbo >> 4) & 0x3FFFu) << 16;
  d |= ((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture family
  return d;                 // base offset 0, layout type 0 (no swizzle)
}

// instruction descriptor: D f32, A/B tf32, both K-major, N = 64, M = 128
constexpr uint32_t TC_IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t TC_IDESC2 = (1u << 4) | (2u << 7) | (2u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);  // N = 128

__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Poll limit of the pipeline waits (not of the drains that follow a give-up):
// TC_SPIN_LIMIT unless lowered by qbg_set_tc_wait_limit, which lets a test make
// a wait run out on purpose and check the error path. One copy per device.
__device__ long long g_tc_wait_polls = TC_SPIN_LIMIT;

// bounded wait: gives up after ~0.5 s of SM clock (1e9 cycles) or `polls` polls
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t mbar, uint32_t parity,
                                                  long long polls = TC_SPIN_LIMIT) {
  if (polls > 0 && mbar_try(mbar, parity)) return true;
  const long long t0 = clock64();
  for (long long it = 1; it < polls; ++it) {
    if (mbar_try(mbar, parity)) return true;
    if (clock64() - t0 > 1000000000ll) break;
  }
  return false;
}


// Operand staging by TC_T = 512 threads: each holds 4 complex k of one row of
// the A tile (one MMA step) and one element of the B tile in registers between
// the global load and the shared-memory store. A warp's B elements are 4
// consecutive k of 8 columns (whole 32-byte sectors; with the lane order below
// each half-warp's 8-byte store covers 128 consecutive bytes).
constexpr int TC_T = 512;
template <bool WIDE> struct TcRegs {
  cxf a[4];             // A(m0 + row, k0 + 4 grp + q)
  cxf b[TS<WIDE>::NB];  // B(k0 + bk, n0 + bj + 32 q)
};
struct TcPos {
  int row, grp, bk, bj;
};

__device__ __forceinline__ TcPos tc_pos(int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  return TcPos{tid & 127, tid >> 7, 4 * (warp & 3) + 2 * (lane >> 4) + (lane & 1), 8 * (warp >> 2) + ((lane >> 1) & 7)};
}

// pa, pb: this thread's first A element and its B elements of the tile; kleft =
// K - k0. Rows past M and columns past N repeat the last one (their results are
// not stored); k past K are zeros.
template <bool WIDE>
__device__ __forceinline__ void tc_load(TcRegs<WIDE>& r, const TcPos& t, const cxf* __restrict__ pa, long long lda,
                                        const cxf* const* pb, int k0, int kleft) {
  if (kleft >= TC_BK) {
#pragma unroll
    for (int q = 0; q < 4; ++q) r.a[q] = pa[q * lda];
#pragma unroll
    for (int q = 0; q < TS<WIDE>::NB; ++q) r.b[q] = pb[q][k0];
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) r.a[q] = 4 * t.grp + q < kleft ? pa[q * lda] : cxf(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < TS<WIDE>::NB; ++q) r.b[q] = t.bk < kleft ? pb[q][k0] : cxf(0.f, 0.f);
  }
}

// 16-byte row segment (k = 4c .. 4c+3) of core matrices in the K-major layout
__device__ __forceinline__ int kmaj4(int row, int c) { return (row >> 3) * 64 + c * 32 + (row & 7) * 4; }

__device__ __forceinline__ void split4(float x0, float x1, float x2, float x3, float4& big, float4& small) {
  tf32_split(x0, big.x, small.x);
  tf32_split(x1, big.y, small.y);
  tf32_split(x2, big.z, small.z);
  tf32_split(x3, big.w, small.w);
}

// nn: columns of the tile, a multiple of 8
template <bool WIDE>
__device__ __forceinline__ void tc_store(const TcRegs<WIDE>& r, const TcPos& t, float* sAb, float* sAs, float* sB,
                                         int nn) {
  // A'[i][2k] = Re, A'[i][2k+1] = Im; pair p of the step's complex k is its 16-byte segment p
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float4 big, small;
    split4(r.a[2 * p].re, r.a[2 * p].im, r.a[2 * p + 1].re, r.a[2 * p + 1].im, big, small);
    const int off = t.grp * TC_A_STEP + kmaj4(t.row, p);
    *reinterpret_cast<float4*>(sAb + off) = big;
    *reinterpret_cast<float4*>(sAs + off) = small;
  }
  // B'[j] = (Re, -Im) and B'[nn + j] = (Im, Re) along k; big, then small, per step
  constexpr int BS = TS<WIDE>::B_STEP;
  const int lo = (t.bk >> 2) * 2 * BS + 2 * (t.bk & 1), seg = (t.bk >> 1) & 1;
#pragma unroll
  for (int q = 0; q < TS<WIDE>::NB; ++q) {
    const int j = t.bj + 32 * q;
    if (WIDE && j >= nn) break;
    float br, bi, sr, si;
    tf32_split(r.b[q].re, br, sr);
    tf32_split(r.b[q].im, bi, si);
    const int o0 = lo + kmaj4(j, seg), o1 = lo + kmaj4(nn + j, seg);
    *reinterpret_cast<float2*>(sB + o0) = make_float2(br, -bi);
    *reinterpret_cast<float2*>(sB + BS + o0) = make_float2(sr, -si);
    *reinterpret_cast<float2*>(sB + o1) = make_float2(bi, br);
    *reinterpret_cast<float2*>(sB + BS + o1) = make_float2(si, sr);
  }
}

}  // namespace

// Warps 0..15 stage the operands, warp 16 issues the MMAs: while the tensor cores
// read one of the two shared-memory stages, the others store the next tile, and
// the loads of the two tiles after it are in flight in registers. full[s] counts
// the staging warps, empty[s] completes with the MMAs that read stage s.
// Accumulators: A_big B_big, and A_big B_small + A_small B_big, added by the
// epilogue. On the 32-column tile the two products of A_big are one MMA of N = 128
// (B' = [big | small] of a step; an N = 64 MMA takes no less time).
// Bound at the solves' sizes (K = 256, few tiles): the chain of one k-tile, load,
// split, store and MMA. A product of 256 x 96 x 256 for 10 operators takes 16.5 us
// (128 threads that also issued three N = 64 MMAs a step: 25 us); one disk of 48
// nodes of N = 2048: 60.7 -> 56.9 ms, 16 streamed nodes of N = 5002: 165.5 -> 152 ms.
// The wide tile restages A a quarter as often and gives the same bits
// (when each is taken: staged_wide).
template <bool WIDE>
__global__ void __launch_bounds__(TC_T + 32, WIDE ? 1 : 2) k_tc_cgemm(int M, int N, int K, cxf alpha, const cxf* __restrict__ A,
                                                           long long lda, long long sA, const cxf* B, long long ldb,
                                                           long long sB, cxf beta, cxf* C, long long ldc,
                                                           long long sC, int batch2, long long sA2, long long sB2,
                                                           long long sC2, int* err) {
  using P = TS<WIDE>;
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  float* stage_base = reinterpret_cast<float*>(tc_smem);  // [2][sAb | sAs | sB]
  uint64_t* mbar = reinterpret_cast<uint64_t*>(stage_base + 2 * P::STAGE);  // full[2], empty[2], done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbar + 5);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool stager = warp < TC_T / 32;
  const int m0 = blockIdx.x * TC_BM, n0 = blockIdx.y * P::BN;
  const int nn = WIDE ? min((N - n0 + 7) & ~7, P::BN) : P::BN;
  const long long bo = blockIdx.z / batch2, bi = blockIdx.z % batch2;  // outer, inner batch index
  const cxf* Ab = A + bo * sA + bi * sA2;
  const cxf* Bb = B + bo * sB + bi * sB2;
  cxf* Cb = C + bo * sC + bi * sC2;

  if (!stager) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(P::TMEM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const uint32_t mb = smem_u32(mbar);
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < 5; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mb + 8 * q), "r"(q < 2 ? TC_T / 32 : 1) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = (*reinterpret_cast<volatile int*>(err) != 0) ? 1 : 0;
  }
  const TcPos pos = tc_pos(tid & (TC_T - 1));
  const int ktiles = (K + TC_BK - 1) / TC_BK;
  TcRegs<WIDE> regs[2];
  const cxf* pa = Ab + min(m0 + pos.row, M - 1) + (long long)(4 * pos.grp) * lda;
  const cxf* pb[P::NB];
#pragma unroll
  for (int q = 0; q < P::NB; ++q) pb[q] = Bb + pos.bk + (long long)min(n0 + pos.bj + 32 * q, N - 1) * ldb;
  const long long step = TC_BK * lda;
  if (stager) {
    tc_load<WIDE>(regs[0], pos, pa, lda, pb, 0, K);
    tc_load<WIDE>(regs[1], pos, pa += step, lda, pb, TC_BK, K - TC_BK);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const bool go = *abort_flag == 0;

  // C of this thread (row = TMEM lane tid & 127, 8 of the tile's columns), fetched now so that its
  // latency hides behind the k loop; the wide tile fetches its first 8 after it
  const int i = m0 + pos.row, jc = n0 + 8 * pos.grp;
  const bool use_beta = !(beta.re == 0.f && beta.im == 0.f);
  cxf cold[8];
  auto fetch = [&](int j0) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      cold[j] = (use_beta && i < M && j0 + j < N) ? Cb[(long long)i + (long long)(j0 + j) * ldc] : cxf(0.f, 0.f);
  };
  if (stager && go) {
    if (!WIDE) fetch(jc);
#pragma unroll 2
    for (int kt = 0; kt < ktiles; ++kt) {
      const int st = kt & 1;
      float* sAb = stage_base + st * P::STAGE;
      float* sAs = sAb + TC_KSTEPS * TC_A_STEP;
      float* sBt = sAs + TC_KSTEPS * TC_A_STEP;
      if (kt >= 2 && !mbar_wait_bounded(mb + 16 + 8 * st, (uint32_t)(((kt >> 1) - 1) & 1), g_tc_wait_polls)) {
        atomicExch(abort_flag, 1);  // the MMAs of tile kt-2 still read this stage
        break;
      }
      tc_store<WIDE>(st ? regs[1] : regs[0], pos, sAb, sAs, sBt, nn);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mb + 8 * st) : "memory");
      if (kt + 2 < ktiles) {
        pa += step;
        const int k0 = (kt + 2) * TC_BK;
        if (st) tc_load<WIDE>(regs[1], pos, pa, lda, pb, k0, K - k0);
        else tc_load<WIDE>(regs[0], pos, pa, lda, pb, k0, K - k0);
      }
    }
    if (WIDE) fetch(jc);
  } else if (!stager && lane == 0) {
    const uint32_t idn = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(2 * nn >> 3) << 17) | ((128u >> 4) << 24);
    for (int kt = 0; kt < ktiles && go; ++kt) {
      const int st = kt & 1;
      const uint32_t sAb = smem_u32(stage_base + st * P::STAGE);
      const uint32_t sAs = sAb + 4 * TC_KSTEPS * TC_A_STEP, sBt = sAs + 4 * TC_KSTEPS * TC_A_STEP;
      if (!mbar_wait_bounded(mb + 8 * st, (uint32_t)((kt >> 1) & 1), g_tc_wait_polls)) {
        atomicExch(abort_flag, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int s = 0; s < TC_KSTEPS; ++s) {
        const uint64_t dab = smem_desc(sAb + 4 * s * TC_A_STEP), das = smem_desc(sAs + 4 * s * TC_A_STEP);
        const uint64_t db = smem_desc(sBt + 8 * s * P::B_STEP);
        if constexpr (WIDE) {
          mma_tf32(tmem, dab, db, idn, (kt | s) != 0);
          mma_tf32(tmem + 2 * P::BN, dab, smem_desc(sBt + 8 * s * P::B_STEP + 4 * P::B_STEP), idn, (kt | s) != 0);
          mma_tf32(tmem + 2 * P::BN, das, db, idn, 1);
        } else {
          mma_tf32(tmem, dab, db, TC_IDESC2, (kt | s) != 0);
          mma_tf32(tmem + 2 * P::BN, das, db, TC_IDESC, 1);
        }
      }
      mma_commit(mb + 16 + 8 * st);
    }
    // every MMA issued must be observed done before TMEM is read or released
    mma_commit(mb + 32);
    if (!mbar_wait_bounded(mb + 32, 0)) atomicExch(abort_flag, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (*abort_flag || ktiles == 0) {
    if (tid == 0 && *abort_flag) atomicExch(err, 1);
  } else if (stager) {
    // warp w reads TMEM lanes 32 (w mod 4) .., columns 8 grp .. of Re and Im of both
    // accumulators (the wide tile: and every 32 columns from there)
#pragma unroll 1
    for (int c0 = 8 * pos.grp; c0 < nn; c0 += 32) {
      if (c0 > 8 * pos.grp) fetch(n0 + c0);
      const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
      float v[4][8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t x[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
                     : "r"(taddr + (uint32_t)((q >> 1) * 2 * P::BN + (q & 1) * nn)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) v[q][j] = __uint_as_float(x[j]);
      }
      if (i < M) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (n0 + c0 + j < N) {
            cxf c = alpha * cxf(v[0][j] + v[2][j], v[1][j] + v[3][j]);
            if (use_beta) c += beta * cold[j];
            Cb[(long long)i + (long long)(n0 + c0 + j) * ldc] = c;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (!stager) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P::TMEM) : "memory");
  }
}

namespace {
__device__ __forceinline__ void pk_expect(uint32_t mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void pk_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(mbar)
      : "memory");
}
}  // namespace

// ---------------------------------------------------------------------------
// Wide packed GEMM for large products (the LU's trailing updates): one CTA
// computes a 128 x 128 complex tile as one real M = 128, N = 256 MMA per k
// step (B' rows 0..127 = (Re, -Im) of the tile's columns, 128..255 =
// (Im, Re)), so an A tile read from L2 feeds four times the MMA work of the
// 128 x 32 tile. Accumulator: 256 TMEM columns (Re C in 0..127, Im C in
// 128..255). Operands are packed (split into big and small TF32 parts) in
// tiles of 4 KS complex k (KS MMA k steps), one bulk copy per operand and
// stage, through a four-stage ring:
//   PAW tile (b, mt, kt): [big | small] x KS MMA steps x 128 rows x 8 real k (8 KS KB)
//   PBW tile (b, nt, kt): [big | small] x KS MMA steps x 256 B' rows x 8 real k (16 KS KB)
// The epilogue reads the accumulator in 32-column chunks and updates C
// (beta C read there, not prefetched). Every wait is bounded; on a timeout thread
// 0 records the error, waits (bounded) for the copies and MMAs it issued, and the
// CTA frees its TMEM and returns without writing C.
// ---------------------------------------------------------------------------
constexpr int PW_BN = 128;                                  // complex columns per CTA (real N = 256)
constexpr int PW_NST = 4;                                   // stages in the ring
constexpr int PW_B_STEP = 2 * PW_BN * 8;                    // floats per B' block per MMA step (8 KB)
constexpr uint32_t PW_TMEM_COLS = 256;
// KS MMA k steps (4 KS complex k) per stage: KS = 2, 48 KB stages, one CTA per
// SM; KS = 1, 24 KB stages, two CTAs per SM (96 KB of stages and 256 TMEM
// columns each), so one CTA's epilogue and pipeline fill overlap the other's MMAs
template <int KS> struct PW {
  static constexpr int BK = 4 * KS;                           // complex k per stage
  static constexpr int A_TILE = 2 * KS * TC_A_STEP;           // floats
  static constexpr int B_TILE = 2 * KS * PW_B_STEP;
  static constexpr int STAGE = A_TILE + B_TILE;
  static constexpr int CTAS = KS == 1 ? 2 : 1;                // resident CTAs per SM
};
// instruction descriptor: D f32, A/B tf32, both K-major, N = 256, M = 128
constexpr uint32_t PW_IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_tf32_w(uint32_t dtmem, uint64_t da, uint64_t db, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(da), "l"(db), "r"(PW_IDESC), "r"(acc));
}

// grid (MT, KTW, batch * batch2), 128 threads: thread = row of the tile
template <int KS>
__global__ void __launch_bounds__(128) k_tc_pack_aw(const cxf* __restrict__ A, long long lda, long long sA,
                                                    long long sA2, int batch2, int M, int K, float* __restrict__ PA) {
  constexpr int PW_BK = PW<KS>::BK, PW_KSTEPS = KS, PW_A_TILE = PW<KS>::A_TILE;
  const int tid = threadIdx.x;
  const int mt = blockIdx.x, kt = blockIdx.y, MT = gridDim.x, KT = gridDim.y;
  const long long z = blockIdx.z, bo = z / batch2, bi = z % batch2;
  const cxf* Ab = A + bo * sA + bi * sA2;
  const int gi = mt * TC_BM + tid, k0 = kt * PW_BK;
  const bool rowok = gi < M;
  cxf a[PW_BK];
#pragma unroll
  for (int kc = 0; kc < PW_BK; ++kc) {
    const int gk = k0 + kc;
    a[kc] = (rowok && gk < K) ? Ab[(long long)gi + (long long)gk * lda] : cxf(0.f, 0.f);
  }
  float* tile = PA + ((z * MT + mt) * (long long)KT + kt) * PW_A_TILE;
#pragma unroll
  for (int p = 0; p < PW_BK / 2; ++p) {
    float4 big, small;
    split4(a[2 * p].re, a[2 * p].im, a[2 * p + 1].re, a[2 * p + 1].im, big, small);
    const int off = (p >> 1) * TC_A_STEP + kmaj4(tid, p & 1);
    *reinterpret_cast<float4*>(tile + off) = big;
    *reinterpret_cast<float4*>(tile + PW_KSTEPS * TC_A_STEP + off) = small;
  }
}

// grid (NTW, KTW, batch * batch2), 128 threads: 2 KS (column, k pair) items each
template <int KS>
__global__ void __launch_bounds__(128) k_tc_pack_bw(const cxf* __restrict__ B, long long ldb, long long sB,
                                                    long long sB2, int batch2, int N, int K, float* __restrict__ PB) {
  constexpr int PW_BK = PW<KS>::BK, PW_KSTEPS = KS, PW_B_TILE = PW<KS>::B_TILE;
  const int tid = threadIdx.x;
  const int nt = blockIdx.x, kt = blockIdx.y, NT = gridDim.x, KT = gridDim.y;
  const long long z = blockIdx.z, bo = z / batch2, bi = z % batch2;
  const cxf* Bb = B + bo * sB + bi * sB2;
  const int n0 = nt * PW_BN, k0 = kt * PW_BK;
  float* tile = PB + ((z * NT + nt) * (long long)KT + kt) * PW_B_TILE;
#pragma unroll
  for (int q = 0; q < 2 * KS; ++q) {
    const int item = tid + 128 * q;
    const int j = item & (PW_BN - 1), p = item >> 7;  // j fastest: consecutive columns per warp
    const int gj = n0 + j, gk = k0 + 2 * p;
    const bool colok = gj < N;
    const cxf v0 = (colok && gk < K) ? Bb[(long long)gk + (long long)gj * ldb] : cxf(0.f, 0.f);
    const cxf v1 = (colok && gk + 1 < K) ? Bb[(long long)(gk + 1) + (long long)gj * ldb] : cxf(0.f, 0.f);
    const int base = (p >> 1) * PW_B_STEP;
    float4 big, small;
    split4(v0.re, -v0.im, v1.re, -v1.im, big, small);
    *reinterpret_cast<float4*>(tile + base + kmaj4(j, p & 1)) = big;
    *reinterpret_cast<float4*>(tile + PW_KSTEPS * PW_B_STEP + base + kmaj4(j, p & 1)) = small;
    split4(v0.im, v0.re, v1.im, v1.re, big, small);
    *reinterpret_cast<float4*>(tile + base + kmaj4(PW_BN + j, p & 1)) = big;
    *reinterpret_cast<float4*>(tile + PW_KSTEPS * PW_B_STEP + base + kmaj4(PW_BN + j, p & 1)) = small;
  }
}

// grid (MT, NTW, batch * batch2), 128 threads
template <int KS>
__global__ void __launch_bounds__(128, PW<KS>::CTAS) k_tc_cgemm_pkw(int M, int N, int KT, cxf alpha,
                                                                   const float* __restrict__ PA,
                                                                   const float* __restrict__ PB, cxf beta, cxf* C,
                                                                   long long ldc, long long sC, int batch2,
                                                                   long long sC2, int* err) {
  constexpr int PW_KSTEPS = KS, PW_A_TILE = PW<KS>::A_TILE, PW_B_TILE = PW<KS>::B_TILE, PW_STAGE = PW<KS>::STAGE;
  extern __shared__ __align__(1024) unsigned char pw_smem[];
  float* stages = reinterpret_cast<float*>(pw_smem);  // [PW_NST][A tile | B tile]
  uint64_t* full = reinterpret_cast<uint64_t*>(stages + PW_NST * PW_STAGE);  // [PW_NST]
  uint64_t* empty = full + PW_NST;                                          // [PW_NST]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + PW_NST);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int mt = blockIdx.x, nt = blockIdx.y, MT = gridDim.x, NT = gridDim.y;
  const long long z = blockIdx.z, bo = z / batch2, bi = z % batch2;
  const int m0 = mt * TC_BM, n0 = nt * PW_BN;
  cxf* Cb = C + bo * sC + bi * sC2;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(PW_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < PW_NST; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(full + s)) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(empty + s)) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = (*reinterpret_cast<volatile int*>(err) != 0) ? 1 : 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (tid == 0 && *abort_flag == 0) {
    const float* pa = PA + (z * MT + mt) * (long long)KT * PW_A_TILE;
    const float* pb = PB + (z * NT + nt) * (long long)KT * PW_B_TILE;
    const uint32_t sbase = smem_u32(stages);
    auto issue = [&](int t) {
      const int s = t % PW_NST;
      const uint32_t fb = smem_u32(full + s);
      pk_expect(fb, (uint32_t)(PW_STAGE * sizeof(float)));
      pk_bulk(sbase + (uint32_t)(s * PW_STAGE * sizeof(float)), pa + (long long)t * PW_A_TILE,
              (uint32_t)(PW_A_TILE * sizeof(float)), fb);
      pk_bulk(sbase + (uint32_t)((s * PW_STAGE + PW_A_TILE) * sizeof(float)), pb + (long long)t * PW_B_TILE,
              (uint32_t)(PW_B_TILE * sizeof(float)), fb);
    };
    int issued = 0, consumed = 0, committed = 0, freed = 0;
    bool good = true;
    for (; issued < KT && issued < PW_NST; ++issued) issue(issued);
    for (int kt = 0; kt < KT && good; ++kt) {
      const int s = kt % PW_NST;
      if (!mbar_wait_bounded(smem_u32(full + s), (uint32_t)((kt / PW_NST) & 1), g_tc_wait_polls)) {
        good = false;
        break;
      }
      ++consumed;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float* sA = stages + s * PW_STAGE;
      const float* sB = sA + PW_A_TILE;
#pragma unroll
      for (int q = 0; q < PW_KSTEPS; ++q) {
        const uint64_t dab = smem_desc(smem_u32(sA + q * TC_A_STEP));
        const uint64_t das = smem_desc(smem_u32(sA + PW_KSTEPS * TC_A_STEP + q * TC_A_STEP));
        const uint64_t dbb = smem_desc(smem_u32(sB + q * PW_B_STEP));
        const uint64_t dbs = smem_desc(smem_u32(sB + PW_KSTEPS * PW_B_STEP + q * PW_B_STEP));
        mma_tf32_w(tmem, das, dbb, (kt | q) != 0);
        mma_tf32_w(tmem, dab, dbs, 1);
        mma_tf32_w(tmem, dab, dbb, 1);
      }
      mma_commit(smem_u32(empty + s));
      ++committed;
      if (kt >= 1 && issued < KT) {  // refill the stage of tile kt - 1 once its MMAs are done
        const int t = kt - 1;
        if (!mbar_wait_bounded(smem_u32(empty + t % PW_NST), (uint32_t)((t / PW_NST) & 1), g_tc_wait_polls)) {
          good = false;
          break;
        }
        ++freed;
        issue(issued);
        ++issued;
      }
    }
    for (; good && freed < committed; ++freed)
      if (!mbar_wait_bounded(smem_u32(empty + freed % PW_NST), (uint32_t)((freed / PW_NST) & 1), g_tc_wait_polls))
        good = false;
    if (!good) {
      *abort_flag = 1;
      atomicExch(err, 1);
      for (int t = consumed; t < issued; ++t)
        mbar_wait_bounded(smem_u32(full + t % PW_NST), (uint32_t)((t / PW_NST) & 1));
      for (int t = freed; t < committed; ++t)
        mbar_wait_bounded(smem_u32(empty + t % PW_NST), (uint32_t)((t / PW_NST) & 1));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (*abort_flag == 0 && KT > 0) {
    const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
    const int i = m0 + warp * 32 + lane;
    const bool use_beta = !(beta.re == 0.f && beta.im == 0.f);
#pragma unroll 1
    for (int ch = 0; ch < PW_BN / 32; ++ch) {
      uint32_t re[32], im[32];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
          "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
          : "=r"(re[0]), "=r"(re[1]), "=r"(re[2]), "=r"(re[3]), "=r"(re[4]), "=r"(re[5]), "=r"(re[6]), "=r"(re[7]),
            "=r"(re[8]), "=r"(re[9]), "=r"(re[10]), "=r"(re[11]), "=r"(re[12]), "=r"(re[13]), "=r"(re[14]),
            "=r"(re[15]), "=r"(re[16]), "=r"(re[17]), "=r"(re[18]), "=r"(re[19]), "=r"(re[20]), "=r"(re[21]),
            "=r"(re[22]), "=r"(re[23]), "=r"(re[24]), "=r"(re[25]), "=r"(re[26]), "=r"(re[27]), "=r"(re[28]),
            "=r"(re[29]), "=r"(re[30]), "=r"(re[31])
          : "r"(taddr + (uint32_t)(ch * 32)));
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
          "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
          : "=r"(im[0]), "=r"(im[1]), "=r"(im[2]), "=r"(im[3]), "=r"(im[4]), "=r"(im[5]), "=r"(im[6]), "=r"(im[7]),
            "=r"(im[8]), "=r"(im[9]), "=r"(im[10]), "=r"(im[11]), "=r"(im[12]), "=r"(im[13]), "=r"(im[14]),
            "=r"(im[15]), "=r"(im[16]), "=r"(im[17]), "=r"(im[18]), "=r"(im[19]), "=r"(im[20]), "=r"(im[21]),
            "=r"(im[22]), "=r"(im[23]), "=r"(im[24]), "=r"(im[25]), "=r"(im[26]), "=r"(im[27]), "=r"(im[28]),
            "=r"(im[29]), "=r"(im[30]), "=r"(im[31])
          : "r"(taddr + (uint32_t)(PW_BN + ch * 32)));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (i < M) {
        cxf cold[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int gj = n0 + ch * 32 + j;
          cold[j] = (use_beta && gj < N) ? Cb[(long long)i + (long long)gj * ldc] : cxf(0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int gj = n0 + ch * 32 + j;
          if (gj < N) {
            cxf v = alpha * cxf(__uint_as_float(re[j]), __uint_as_float(im[j]));
            if (use_beta) v += beta * cold[j];
            Cb[(long long)i + (long long)gj * ldc] = v;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PW_TMEM_COLS) : "memory");
  }
}

// device error flag of the tensor-core GEMM (one per device, found by symbol)
__device__ int g_tc_err;

template <bool WIDE>
static size_t tc_smem_bytes() { return sizeof(float) * (size_t)(2 * TS<WIDE>::STAGE) + 64; }
template <int KS>
static size_t pw_smem_bytes() { return sizeof(float) * (size_t)(PW_NST * PW<KS>::STAGE) + 16 * PW_NST + 64; }

namespace {
constexpr int TC_MAX_DEV = 64;
std::mutex g_tc_mu;
int* g_tc_err_addr[TC_MAX_DEV] = {};
bool g_tc_attr[TC_MAX_DEV] = {};
std::atomic<int> g_engine{GEMM_ENGINE_TCGEN05};
std::atomic<bool> g_pk_enabled{true};  // packed-operand path of tc_gemm_c64
// packed path: QBG_GEMM_WIDE in the environment, 0 leaves every product to the
// staged kernel, 1 one packed CTA per SM (48 KB stages), 2 (default) two per
// SM (24 KB stages; C2 factor phase 28.1 -> 26.7 ms against 1)
std::atomic<int> g_pkw_mode{[] {
  const char* e = std::getenv("QBG_GEMM_WIDE");
  return (e && *e) ? std::max(0, std::min(std::atoi(e), 2)) : 2;
}()};

int tc_device_setup(int** err_out) {
  int dev = 0;
  QBG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= TC_MAX_DEV) {
    set_error("device ordinal %d out of range", dev);
    return QBG_ECUDA;
  }
  std::lock_guard<std::mutex> lk(g_tc_mu);
  if (!g_tc_attr[dev]) {
    QBG_CUDA(cudaFuncSetAttribute(k_tc_cgemm<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)tc_smem_bytes<false>()));
    QBG_CUDA(cudaFuncSetAttribute(k_tc_cgemm<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)tc_smem_bytes<true>()));
    QBG_CUDA(cudaFuncSetAttribute(k_tc_cgemm_pkw<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)pw_smem_bytes<2>()));
    QBG_CUDA(cudaFuncSetAttribute(k_tc_cgemm_pkw<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)pw_smem_bytes<1>()));
    void* a = nullptr;
    QBG_CUDA(cudaGetSymbolAddress(&a, g_tc_err));
    g_tc_err_addr[dev] = static_cast<int*>(a);
    g_tc_attr[dev] = true;
  }
  *err_out = g_tc_err_addr[dev];
  return QBG_OK;
}

// Packing scratch, one buffer per (device, stream): the GEMMs of one stream
// run in order, so a stream reuses its buffer without waiting; a larger
// request replaces it (the old block goes back to the pool behind the stream's
// work). The owner of a stream returns its buffer with tc_release_scratch
// before destroying the stream.
struct PackScratch {
  int dev;
  cudaStream_t st;
  void* p;
  size_t bytes;
};
std::mutex g_pack_mu;
std::vector<PackScratch> g_pack;

int pack_scratch(cudaStream_t st, size_t bytes, void** out) {
  int dev = 0;
  QBG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_pack_mu);
  for (auto& e : g_pack)
    if (e.dev == dev && e.st == st) {
      if (e.bytes < bytes) {
        void* q = nullptr;
        QBG_TRY(dmalloc(&q, bytes));
        dfree(e.p, st);
        e.p = q;
        e.bytes = bytes;
      }
      *out = e.p;
      return QBG_OK;
    }
  void* q = nullptr;
  QBG_TRY(dmalloc(&q, bytes));
  g_pack.push_back({dev, st, q, bytes});
  *out = q;
  return QBG_OK;
}
}  // namespace

int tc_error_ptr(int** p) { return tc_device_setup(p); }

void tc_release_scratch(cudaStream_t st) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  std::lock_guard<std::mutex> lk(g_pack_mu);
  for (size_t q = 0; q < g_pack.size(); ++q)
    if (g_pack[q].dev == dev && g_pack[q].st == st) {
      dfree(g_pack[q].p, st);
      g_pack.erase(g_pack.begin() + (long)q);
      return;
    }
}

void set_gemm_engine(int e) {
  g_engine.store(e == GEMM_ENGINE_SIMT ? GEMM_ENGINE_SIMT : GEMM_ENGINE_TCGEN05);
  g_pk_enabled.store(e != GEMM_ENGINE_TCGEN05_STAGED);
}
int gemm_engine() { return g_engine.load(); }

// The staged kernel's tile width. Time of a tile of K = 256, in units of 16.5 us:
// the 32-column form takes 1 with a CTA to an SM and 1.75 with two (28.9 us); the
// wide one 1.37, 1.63 and 1.85 at 64, 96 and 128 columns (22.6, 26.8 and 31 us),
// one to an SM. Measured, narrow against wide: 256 x 96 for 2 operators 16.5 /
// 26.8 us, 4096 x 96 for 2 28.9 / 26.8, 768 x 96 for 96 150 / 107, 1000 x 1000
// for 2 52 / 33. Both give the same bits.
static bool staged_wide(int MT, int NT, int N, int nb) {
  const double cn = (double)MT * NT * nb, waves = std::ceil((double)MT * ((N + 127) / 128) * nb / 152);
  const double narrow = cn <= 152 ? 1.0 : 1.75 * std::max(1.0, cn / 304);
  return waves * (1.1 + 0.75 * std::min(N, 128) / 128) < narrow;
}

int tc_gemm_c64(int M, int N, int K, cxf alpha, const cxf* A, long long lda, long long sA, const cxf* B,
                long long ldb, long long sB, cxf beta, cxf* C, long long ldc, long long sC, int batch,
                cudaStream_t st, int batch2, long long sA2, long long sB2, long long sC2, bool allow_packed) {
  if (M <= 0 || N <= 0 || batch <= 0 || batch2 <= 0) return QBG_OK;
  if (K <= 0 || (long long)batch * batch2 > 65535) {
    set_error("tc_gemm_c64: K = %d, batch = %d x %d out of range", K, batch, batch2);
    return QBG_EINVAL;
  }
  int* derr = nullptr;
  if (int s = tc_device_setup(&derr)) return s;
  const int MT = (M + TC_BM - 1) / TC_BM, NT = (N + TC_BN - 1) / TC_BN;
  const int nb = batch * batch2;
  // Packed operands (split once, streamed by bulk copies) where a packed tile is
  // read often enough, each A tile by NTW CTAs and each B tile by MT, and the CTAs
  // fill the device more than once. K = 256, packed against staged (wide): 768 x 768
  // for 96 operators 703 / 702 us, 1280 x 1280 for 2, 6 and 24 58 / 60, 117 / 126 and
  // 422 / 490, 4700 x 4700 for 2 425 / 565, 1500 x 1500 for 1 49 / 33
  const int wide = g_pkw_mode.load();  // 0 off, 1 one CTA per SM (KS = 2), 2 two CTAs per SM (KS = 1)
  const int NTW = (N + PW_BN - 1) / PW_BN;
  if (allow_packed && g_pk_enabled.load() && wide > 0 && K >= 32 && MT >= 10 && NTW >= 10 &&
      (long long)MT * NTW * nb > 152) {
    auto run = [&](auto ks) -> int {
      constexpr int KS = decltype(ks)::value;
      const int KTW = (K + PW<KS>::BK - 1) / PW<KS>::BK;
      const size_t pa = (size_t)nb * MT * KTW * PW<KS>::A_TILE, pb = (size_t)nb * NTW * KTW * PW<KS>::B_TILE;
      void* scr = nullptr;
      QBG_TRY(pack_scratch(st, sizeof(float) * (pa + pb), &scr));
      float* PA = static_cast<float*>(scr);
      float* PB = PA + pa;
      k_tc_pack_aw<KS><<<dim3(MT, KTW, nb), 128, 0, st>>>(A, lda, sA, sA2, batch2, M, K, PA);
      QBG_LAUNCH_CHECK("k_tc_pack_aw");
      k_tc_pack_bw<KS><<<dim3(NTW, KTW, nb), 128, 0, st>>>(B, ldb, sB, sB2, batch2, N, K, PB);
      QBG_LAUNCH_CHECK("k_tc_pack_bw");
      k_tc_cgemm_pkw<KS><<<dim3(MT, NTW, nb), 128, pw_smem_bytes<KS>(), st>>>(M, N, KTW, alpha, PA, PB, beta, C,
                                                                               ldc, sC, batch2, sC2, derr);
      QBG_LAUNCH_CHECK("k_tc_cgemm_pkw");
      return QBG_OK;
    };
    return wide == 2 ? run(std::integral_constant<int, 1>{}) : run(std::integral_constant<int, 2>{});
  }
  if (staged_wide(MT, NT, N, nb)) {
    k_tc_cgemm<true><<<dim3(MT, (N + 127) / 128, nb), TC_T + 32, tc_smem_bytes<true>(), st>>>(
        M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch2, sA2, sB2, sC2, derr);
  } else {
    k_tc_cgemm<false><<<dim3(MT, NT, nb), TC_T + 32, tc_smem_bytes<false>(), st>>>(
        M, N, K, alpha, A, lda, sA, B, ldb, sB, beta, C, ldc, sC, batch2, sA2, sB2, sC2, derr);
  }
  QBG_LAUNCH_CHECK("k_tc_cgemm");
  return QBG_OK;
}

// runtime pipeline-wait limit (polls; < 0 restores the built-in limit) and
// reset of the sticky error flag, on the current device
int tc_set_wait_limit(long long polls) {
  int* derr = nullptr;
  if (int s = tc_device_setup(&derr)) return s;
  const long long v = polls < 0 ? TC_SPIN_LIMIT : polls;
  QBG_CUDA(cudaDeviceSynchronize());
  QBG_CUDA(cudaMemcpyToSymbol(g_tc_wait_polls, &v, sizeof(v)));
  return QBG_OK;
}

int tc_clear_error() {
  int* derr = nullptr;
  if (int s = tc_device_setup(&derr)) return s;
  QBG_CUDA(cudaDeviceSynchronize());
  QBG_CUDA(cudaMemset(derr, 0, sizeof(int)));
  return QBG_OK;
}

int tc_check(cudaStream_t st) {
  int* derr = nullptr;
  if (int s = tc_device_setup(&derr)) return s;
  QBG_CUDA(cudaStreamSynchronize(st));
  int h = 0;
  QBG_CUDA(cudaMemcpy(&h, derr, sizeof(int), cudaMemcpyDeviceToHost));
  if (h != 0) {
    // sticky for the process, like a CUDA context error: every handle sees it
    set_error("tensor-core GEMM: an mbarrier wait gave up; results discarded");
    return QBG_ECUDA;
  }
  return QBG_OK;
}

}  // namespace qbg
