// Attention kernels of layers 1 and 2 as CTA-tiled tcgen05 kernels.
//
// A tile is up to 128 consecutive entries of the compacted list of undirected pairs inside the 4.5 A cutoff, grouped by the end with
// the smaller index (the "receiver" i; j is the partner).  Both filters depend on the pair only -- on its length and on the
// invariants of the difference of the two `ev` rows -- so one evaluation serves (i <- j) and (j <- i), forward and reverse.  Per
// tile and layer, both filters of all pairs come out of ONE chain of tcgen05.mma instructions with the accumulators in tensor memory:
//
//     w[e, 0:256] = Phi[e, 0:64] * C[0:64, 0:256]  +  hs_f[e, 0:32] * K2_f[0:32, 0:128]   (f = 0, 1)
//
// Phi are 64 Chebyshev polynomials of t(r) (see common.cuh): the radial filter MLPs are smooth functions of the edge length
// alone, so their 2 x 128 outputs are contracted from a 64-term expansion on the tensor cores instead of being gathered
// from a table (4 KB per edge and layer through L2 before); hs_f is the hidden layer of the spherical filter.  FP32 accuracy
// comes from the two-term FP16 split used throughout the library (x = hi + lo / 2048; products hi*hi into one accumulator,
// hi*lo + lo*hi into a second one).  Operands sit in shared memory in the 8 x 8 core-matrix order without swizzle; the
// 96 KB weight image is resident for the whole kernel.  Four warps issue the MMAs, one per scheduler and accumulator; completion arrives on
// an mbarrier (tcgen05.commit) on which every thread waits for itself; every wait is bounded and reports through an error word
// instead of hanging.
//
// After the MMA the filter tile is moved from tensor memory to shared memory (row = edge) and the edge loop runs in the
// "lane = 4 features" layout of the other attention kernels: sender rows are read with coalesced 512-byte loads, logits are
// 8-lane reductions.  A warp owns a run of consecutive pairs and adds its partial sums to the receiver's row with vector
// reductions in global memory (a receiver's pairs can span warps, tiles and CTAs); the partner's share of a pair goes out as one
// reduction per row.  Those cost less than the second evaluation they replace: the L2 takes 5.4 TB/s of 512-byte row reductions
// (3.2 TB/s once the target exceeds it), and a pair sends 0.6 KB forward and 2.7 KB in reverse.
//
// What binds the kernels: the latency of four warps per scheduler (their 128 registers fill the register file).  Per 128 pairs the reverse
// kernel issues 65 k warp instructions (16 k cycles of the 43 k a tile takes), moves 24 k wavefronts through the load / store pipe, 7 k
// through the tensor cores' and keeps the way to the L2 busy for 18 k cycles (410 KB of reductions, which leave an SM at 21 to 26 bytes
// per cycle); the forward kernel 28 k instructions (7 k cycles of 17.6 k), 12 k and 2 k wavefronts (counters at 98,304 atoms).  None is
// near its limit, and forms with more warps, fewer registers or two independent tiles per SM ended within 15 % of it or above.
// 98,304 atoms (1.97 M pairs), forward / reverse, ms per launch: 1.99 / 5.12 with every pair evaluated at both ends, 1.16 / 2.85 with one
// evaluation per pair, entry loops that sum four pairs' logits together and one thread that issues, 1.00 / 2.47 as it stands.
//
// The reverse kernel forms dw in the same loop, writes it straight into shared memory as the (FP16-split) A operand of a
// second MMA chain against the SAME weight image read with the other major-ness,
//
//     [dPhi | dhs_f][e, :] = dw_f[e, 0:128] * [C_f^T | K2_f^T],
//
// and finishes the radial derivative (sum_m dPhi[e,m] T_m'(t) dt/dr) and the spherical hidden layer per edge.
#include <cuda_fp16.h>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "kernels.h"

namespace so3lr {

namespace {

constexpr int TE = 128;                       // edges per tile = rows of every MMA
constexpr int kLboA = 2064;                   // bytes between 8-column chunks of an A operand: 128 rows x 16 B + 16 B of padding
constexpr int kAHalf = 16 * kLboA;            // one FP16 matrix of 128 rows x 128 columns
constexpr int kWStride = 132;                 // floats per row of the filter tile
constexpr int kFwRec = 36;                    // floats per forward record: j | i | cutoff / nbar | - | Y[24] | padding (bank spread)
constexpr int kFwThreads = 512;
constexpr int kBwRec = 52;                    // floats per reverse record (48 used; 52 spreads consecutive rows over the banks)
constexpr int kBwThreads = 512;
constexpr float kInvNbar = 1.0f / kAvgNumNeighbors;
constexpr float kRc2 = kCutoffSr * kCutoffSr;
constexpr float kLoScale = 2048.f, kLoInv = 1.f / 2048.f;
constexpr int kTmemCols = 512;
constexpr int kWaitSpins = 1 << 22;

// shared-memory map (bytes)
constexpr int kOffImg = 0;                                   // weight image: C hi | C lo | K2 hi [2] | K2 lo [2]
constexpr int kOffA = kTcImageBytes;                         // A operand (hi | lo); the forward kernel reuses it as filter tile
constexpr int kARegion = TE * kWStride * 4;                  // 67584 >= 2 * kAHalf
static_assert(kARegion >= 2 * kAHalf, "A region");
constexpr int kOffFwRec = kOffA + kARegion;
constexpr int kSphFloats = 4 * 136;           // first spherical layer: 8 floats per hidden unit, 8 more after every 16 units (banks)
constexpr int kOffFwSph = kOffFwRec + TE * kFwRec * 4;
constexpr int kOffFwMisc = kOffFwSph + kSphFloats * 4;
constexpr int kOffFwStIJ = kOffFwMisc + 64;                  // staged inputs of the next tile: (i, j) | displacement
constexpr int kOffFwStD = kOffFwStIJ + TE * 8;
constexpr int kSmemFwd = kOffFwStD + TE * 16;
// reverse kernel: the filter tile holds 64 edges at a time
constexpr int kOffBwW = kOffA + kARegion;
constexpr int kOffBwRec = kOffBwW + 64 * kWStride * 4;
constexpr int kOffBwSph = kOffBwRec + TE * kBwRec * 4;
constexpr int kOffBwMisc = kOffBwSph + kSphFloats * 4;
constexpr int kOffBwStIJ = kOffBwMisc + 64;                  // staged inputs of the next tile: (i, j) | displacement
constexpr int kOffBwStD = kOffBwStIJ + TE * 8;
constexpr int kSmemBwd = kOffBwStD + TE * 16;
static_assert(kSmemFwd <= 232448 && kSmemBwd <= 232448, "shared memory budget of one CTA per SM");

__device__ __forceinline__ float invw(int l) {
  return l == 0 ? 0.5773502691896258f : (l == 1 ? 0.4472135954999579f : (l == 2 ? 0.3779644730092272f : 0.3333333333333333f));
}
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// float4 arithmetic as two packed operations (fma.rn.f32x2 / mul.rn.f32x2) on the halves
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 f4_fma(float a, float4 b, float4 c) {
  const float2 a2 = make_float2(a, a);
  const float2 l = __ffma2_rn(a2, lo2(b), lo2(c)), h = __ffma2_rn(a2, hi2(b), hi2(c));
  return make_float4(l.x, l.y, h.x, h.y);
}
__device__ __forceinline__ float4 f4_scale(float a, float4 b) {
  const float2 a2 = make_float2(a, a);
  const float2 l = __fmul2_rn(a2, lo2(b)), h = __fmul2_rn(a2, hi2(b));
  return make_float4(l.x, l.y, h.x, h.y);
}
__device__ __forceinline__ float4 f4_mul(float4 a, float4 b) {
  const float2 l = __fmul2_rn(lo2(a), lo2(b)), h = __fmul2_rn(hi2(a), hi2(b));
  return make_float4(l.x, l.y, h.x, h.y);
}
__device__ __forceinline__ float4 f4_mad(float4 a, float4 b, float4 c) {
  const float2 l = __ffma2_rn(lo2(a), lo2(b), lo2(c)), h = __ffma2_rn(hi2(a), hi2(b), hi2(c));
  return make_float4(l.x, l.y, h.x, h.y);
}
__device__ __forceinline__ float4 f4_zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float dot3(float4 a, float4 b, float4 c) {
  const float2 s = __ffma2_rn(__fmul2_rn(hi2(a), hi2(b)), hi2(c), __fmul2_rn(__fmul2_rn(lo2(a), lo2(b)), lo2(c)));
  return s.x + s.y;
}
__device__ __forceinline__ float dot2(float4 a, float4 b) {
  const float2 s = __ffma2_rn(hi2(a), hi2(b), __fmul2_rn(lo2(a), lo2(b)));
  return s.x + s.y;
}
// Eight sums over the eight lanes of a group at once: lane cg of the group gets the sum of v[cg].  Seven exchanges, in three dependent
// steps, where eight separate butterfly sums take 24.
__device__ __forceinline__ float transpose_sum8(const float (&v)[8], int cg) {
  float s[4], t[2];
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = ((cg & 4) ? v[k + 4] : v[k]) + __shfl_xor_sync(0xffffffffu, (cg & 4) ? v[k] : v[k + 4], 4);
#pragma unroll
  for (int k = 0; k < 2; ++k) t[k] = ((cg & 2) ? s[k + 2] : s[k]) + __shfl_xor_sync(0xffffffffu, (cg & 2) ? s[k] : s[k + 2], 2);
  return ((cg & 1) ? t[1] : t[0]) + __shfl_xor_sync(0xffffffffu, (cg & 1) ? t[0] : t[1], 1);
}
__device__ __forceinline__ bool f4_nonzero(float4 a) { return a.x != 0.f || a.y != 0.f || a.z != 0.f || a.w != 0.f; }

// (x, y) -> FP16 pair hi and FP16 pair of the residuals scaled by 2048
__device__ __forceinline__ void split2(float x, float y, unsigned& hi, unsigned& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn((x - hf.x) * kLoScale, (y - hf.y) * kLoScale);
  hi = *reinterpret_cast<const unsigned*>(&h);
  lo = *reinterpret_cast<const unsigned*>(&l);
}
// eight consecutive K entries of one operand row -> one 16-byte chunk of the hi matrix and one of the lo matrix
__device__ __forceinline__ void store_chunk(unsigned char* a_hi, int chunk, int row, const float* v) {
  uint4 h, l;
  split2(v[0], v[1], h.x, l.x); split2(v[2], v[3], h.y, l.y); split2(v[4], v[5], h.z, l.z); split2(v[6], v[7], h.w, l.w);
  unsigned char* p = a_hi + chunk * kLboA + row * 16;
  *reinterpret_cast<uint4*>(p) = h;
  *reinterpret_cast<uint4*>(p + kAHalf) = l;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// instruction descriptor, kind::f16: FP16 operands, FP32 accumulator, A K-major, B K-major or MN-major, M = 128
__device__ __forceinline__ uint32_t make_idesc(int n, int b_mn_major) {
  return (1u << 4) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TE >> 4) << 24);
}
// A whole warp runs the issue code; `on` is set in one lane, which issues.  Descriptors then are the same in all lanes and stay in uniform
// registers: 43 cycles from one MMA to the next instead of 53 where a single thread has branched off.
__device__ __forceinline__ void umma_if(uint32_t on, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(on) : "memory");
}
// ... that writes the accumulator rows [64 half, 64 half + 64) only
__device__ __forceinline__ void umma_half_if(uint32_t on, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, int half) {
  const uint32_t off_lo = half ? 0xffffffffu : 0u, off_hi = ~off_lo;
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%6, %6, %7, %7}, p;\n\t"
      "}\n" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(on), "r"(off_lo), "r"(off_hi) : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t on, uint32_t mbar) {
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
      "}\n" ::"r"(mbar), "r"(on) : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t on;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n" : "=r"(on));
  return on;
}
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  for (int it = 0; it < kWaitSpins; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n" : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// fire-and-forget vector add in global memory (no value comes back to the warp)
__device__ __forceinline__ void red_add_v4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Every thread that goes on to read what the MMAs left waits for itself.  After a wait that ran out the CTA's later ones return at once:
// the kernel carries on to its end with an error word set.
__device__ __forceinline__ void wait_mma(uint32_t mbar, uint32_t parity, volatile int* failed, int* err) {
  if (!*failed && !mbar_wait(mbar, parity)) { *failed = 1; atomicExch(err, 1); }
  tc_fence_after();
}

// main + cross / 2048 of 16 columns (cross accumulators sit 256 columns above the main ones)
__device__ __forceinline__ void tmem_ld16_combined(uint32_t taddr, float* v) {
  uint32_t a[16], b[16];      // both loads in flight before the one wait
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]), "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]), "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15]),
        "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7]), "=r"(b[8]), "=r"(b[9]), "=r"(b[10]), "=r"(b[11]), "=r"(b[12]), "=r"(b[13]), "=r"(b[14]), "=r"(b[15])
      : "r"(taddr), "r"(taddr + 256)
      : "memory");
  const float2 s2 = make_float2(kLoInv, kLoInv);
#pragma unroll
  for (int k = 0; k < 16; k += 2) {
    const float2 r = __ffma2_rn(make_float2(__uint_as_float(b[k]), __uint_as_float(b[k + 1])), s2,
                                make_float2(__uint_as_float(a[k]), __uint_as_float(a[k + 1])));
    v[k] = r.x; v[k + 1] = r.y;
  }
}
__device__ __forceinline__ void tmem_ld8_combined(uint32_t taddr, float* v) {
  uint32_t a[8], b[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]),
        "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]), "=r"(b[4]), "=r"(b[5]), "=r"(b[6]), "=r"(b[7])
      : "r"(taddr), "r"(taddr + 256)
      : "memory");
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = fmaf(__uint_as_float(b[k]), kLoInv, __uint_as_float(a[k]));
}

// A pair's ev rows, a quarter per thread of four neighbouring ones: request (`begin`), then the invariants of their difference in all four
struct PairInvariants {
  float4 i0, j0, i1, j1;
  int q;
  __device__ __forceinline__ void begin(const float* evi, const float* evj, int quarter) {
    q = quarter;
    i0 = ld4(evi + 4 * q); j0 = ld4(evj + 4 * q);
    i1 = f4_zero(); j1 = f4_zero();
    if (q < 2) { i1 = ld4(evi + 16 + 4 * q); j1 = ld4(evj + 16 + 4 * q); }
  }
  __device__ __forceinline__ void finish(float (&s)[4]) const {
    const float dv[8] = {j0.x - i0.x, j0.y - i0.y, j0.z - i0.z, j0.w - i0.w, j1.x - i1.x, j1.y - i1.y, j1.z - i1.z, j1.w - i1.w};
    s[0] = s[1] = s[2] = s[3] = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {      // components 4 q + c (degrees 1..3, and 15 of degree 4), then 16 + 4 q + (c - 4) of degree 4
      const float x2 = dv[c] * dv[c];
      if (c >= 4) { s[3] += x2; continue; }
      const int l = degree_of(4 * q + c);
#pragma unroll
      for (int g = 0; g < 4; ++g) s[g] += l == g ? x2 : 0.f;
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      s[l] += __shfl_xor_sync(0xffffffffu, s[l], 1);
      s[l] += __shfl_xor_sync(0xffffffffu, s[l], 2);
      s[l] *= invw(l);
    }
  }
};

// Column order of the Chebyshev block of the A operand: column k < 32 holds T_{2k}, column 32 + k holds T_{2k+1} (the rows of
// the coefficient image are permuted to match).  Two threads share an edge: `odd` = 0 writes the even terms (chunks 0..3),
// 1 the odd ones (chunks 4..7).  Each runs two independent recurrences of step 4, T_{m+4} = 2 T_4 T_m - T_{m-4}, so the
// dependent chain is 16 long instead of 64.
__device__ __forceinline__ void store_chebyshev_half(unsigned char* a_hi, int row, float r, bool valid, int odd) {
  const float x = expf(-kChebHalfGamma * r);
  const float t = fmaf(kChebA, x, kChebB);
  const float T2 = fmaf(2.f * t, t, -1.f), T3 = fmaf(2.f * t, T2, -t), T4x2 = 2.f * fmaf(2.f * T2, T2, -1.f);
  // chain A: m = odd, odd + 4, ...   chain B: m = odd + 2, odd + 6, ...   (prev holds T at the index 4 below cur; T_{-m} = T_m)
  float a_cur = odd ? t : 1.f, a_prev = odd ? T3 : 0.5f * T4x2;
  float b_cur = odd ? T3 : T2, b_prev = odd ? t : T2;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
      v[q] = valid ? a_cur : 0.f;
      v[q + 1] = valid ? b_cur : 0.f;
      const float2 nx = __ffma2_rn(make_float2(T4x2, T4x2), make_float2(a_cur, b_cur), make_float2(-a_prev, -b_prev));
      a_prev = a_cur; a_cur = nx.x;
      b_prev = b_cur; b_cur = nx.y;
    }
    store_chunk(a_hi, 4 * odd + c, row, v);
  }
}
// first-layer weights of hidden unit u of filter f in shared memory: the four weights, the bias, padding
__device__ __forceinline__ int sph_at(int f, int u) { return (f * 32 + u) * 8 + (2 * f + (u >> 4)) * 8; }
// One of four neighbouring threads of a pair: two of the eight chunks of both hidden layers
__device__ __forceinline__ void store_spherical_hidden_quarter(unsigned char* a_hi, int row, const float* s, const float* sph, int quarter) {
  const float* base = sph + sph_at(quarter >> 1, 16 * (quarter & 1));
#pragma unroll
  for (int c8 = 0; c8 < 2; ++c8) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float* p = base + (8 * c8 + q) * 8;
      const float4 k = ld4(p);
      const float z = fmaf(s[0], k.x, fmaf(s[1], k.y, fmaf(s[2], k.z, fmaf(s[3], k.w, p[4]))));
      v[q] = __fdividef(z, 1.f + __expf(-z));
    }
    store_chunk(a_hi, 8 + 2 * quarter + c8, row, v);
  }
}

// Descriptors differ only in their start-address field (bits 0..13, in units of 16 bytes): desc(addr) = base + (addr >> 4).
// The issuing thread keeps everything in registers -- shared-memory loads inside the issue loop wait behind the operand
// traffic of the MMAs already running and throttle the chain.
__device__ __forceinline__ uint64_t desc_base(uint32_t lbo, uint32_t sbo) {
  return ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}

// Forward kernel, K-major weight image (rows = output features, 8 consecutive K entries per 16 bytes; the core matrices of
// one K chunk are contiguous over the rows, the layout the tensor cores fetch fastest):
//   CT hi | CT lo : [256 features][64 terms], core (n/8, k/8) at (k/8) * 4096 + (n/8) * 128           (2 x 32 KB)
//   K2T_f hi | lo : [128 features][32 hidden], core (n/8, k/8) at (k/8) * 2048 + (n/8) * 128          (4 x 8 KB)
// w = Phi * C + hs_f * K2_f: main accumulators in TMEM columns [0, 256), cross accumulators in [256, 512)
// The Chebyshev steps (part 0) read chunks 0..7 of A only, the steps of the spherical hidden layers (part 1) chunks 8..15: part 0 is
// issued as soon as the two threads per entry that write the Chebyshev terms are through, while the others still evaluate the hidden
// layers.  Four warps share the work, one per filter and accumulator (`cross`: hi * lo + lo * hi): the issue of a chain waits behind the
// load / store queue of its scheduler.
__device__ __forceinline__ void issue_forward_mma(uint32_t on, uint32_t tmem, uint32_t a_hi, uint32_t img, int f, int cross, int part) {
  const uint64_t da = desc_base(kLboA, 128) + (a_hi >> 4), dal = da + (kAHalf >> 4);
  const uint64_t dc = desc_base(4096, 128) + ((img + f * 2048) >> 4), dcl = dc + (32768 >> 4);
  const uint64_t dk = desc_base(2048, 128) + ((img + 65536 + f * 8192) >> 4), dkl = dk + (16384 >> 4);
  const uint32_t id128 = make_idesc(128, 0), d = tmem + 128 * f + 256 * cross;
  // K steps 1 and 3 hold the Chebyshev terms of order 32..63 (even terms, then odd terms, 32 columns each).  Their coefficients
  // are below 2^-12 of the filter scale (the expansion converges geometrically), so their hi * lo cross terms are below 2^-23 of
  // it, like the lo * lo terms that are dropped everywhere: those steps issue the hi * hi product only.
#pragma unroll
  for (int ks = 0; ks < 6; ++ks) {
    if ((ks >= 4) != (part == 1)) continue;
    const int chunk = ks < 4 ? 2 * ks : 8 + 4 * f + 2 * (ks - 4);
    const uint64_t ah = da + chunk * (kLboA >> 4), al = dal + chunk * (kLboA >> 4);
    const uint64_t bh = ks < 4 ? dc + ks * (2 * 4096 >> 4) : dk + (ks - 4) * (2 * 2048 >> 4);
    const uint64_t bl = ks < 4 ? dcl + ks * (2 * 4096 >> 4) : dkl + (ks - 4) * (2 * 2048 >> 4);
    if (!cross) {
      umma_if(on, d, ah, bh, id128, ks > 0);
    } else if (ks != 1 && ks != 3) {
      umma_if(on, d, ah, bl, id128, ks > 0);
      umma_if(on, d, al, bh, id128, 1);
    }
  }
}

// Reverse kernel, one image for both directions, per filter f (24,576 bytes each; hi of f = 0, 1 then lo of f = 0, 1): the 96
// rows [64 Chebyshev terms | 32 hidden units] by the 128 features of the filter, core (row / 8, feature / 8) at
// (feature / 8) * 1536 + (row / 8) * 128 with the 8 features of a core row contiguous.
// Forward product (B read MN-major: N = features, K = rows): w_f = [Phi | hs_f] * [C_f ; K2_f], main accumulators in TMEM
// columns [128 f, 128 f + 128), cross 256 columns above.
constexpr int kRevImgFilter = 16 * 1536;
// part 0: the four Chebyshev steps, part 1: the two steps of the filter's hidden layer (see issue_forward_mma)
__device__ __forceinline__ void issue_filter_mma(uint32_t on, uint32_t tmem, uint32_t a_hi, uint32_t img, int f, int cross, int part) {
  const uint64_t da = desc_base(kLboA, 128) + (a_hi >> 4), dal = da + (kAHalf >> 4);
  const uint64_t db = desc_base(128, 1536) + ((img + f * kRevImgFilter) >> 4), dbl = db + (2 * kRevImgFilter >> 4);
  const uint32_t id128 = make_idesc(128, 1);
  const uint32_t d = tmem + 128 * f + 256 * cross;
#pragma unroll
  for (int ks = 0; ks < 6; ++ks) {      // K = 16 rows per step: Chebyshev chunks 0..7 of A, then the two chunks pairs of hs_f
    if ((ks >= 4) != (part == 1)) continue;
    const int chunk = ks < 4 ? 2 * ks : 8 + 4 * f + 2 * (ks - 4);
    const uint64_t ah = da + chunk * (kLboA >> 4), al = dal + chunk * (kLboA >> 4);
    const uint64_t bh = db + ks * (2 * 128 >> 4), bl = dbl + ks * (2 * 128 >> 4);
    if (!cross) {
      umma_if(on, d, ah, bh, id128, ks > 0);
    } else if (ks != 1 && ks != 3) {      // Chebyshev terms of order >= 32: no cross terms (see issue_forward_mma)
      umma_if(on, d, ah, bl, id128, ks > 0);
      umma_if(on, d, al, bh, id128, 1);
    }
  }
}

// accumulators of filter f, rows of a warp's group (warps 0..7 rows 0..63, warps 8..15 rows 64..127) -> filter tile: the four warps of the
// group that can read them, 64 columns each
__device__ __forceinline__ void tmem_to_tile(uint32_t tmem, int f, int warp, int lane, float* wt) {
  const int q = warp & 3, col = 64 * ((warp >> 2) & 1);
  if ((q >> 1) != (warp >> 3)) return;
  float* p = wt + (32 * q + lane) * kWStride + col;
#pragma unroll
  for (int c = 0; c < 64; c += 16) {      // 16 columns at a time: the sender rows in flight hold most of the registers
    float v[16];
    tmem_ld16_combined(tmem + ((uint32_t)(32 * q) << 16) + 128 * f + col + c, v);
#pragma unroll
    for (int k = 0; k < 16; k += 4) st4(p + c + k, make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]));
  }
}

// ------------------------------------------------------------------------------------------------------------------
// compacted edge list
// ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool edge_valid(int j, int n, float dx, float dy, float dz, float& r2) {
  r2 = dx * dx + dy * dy + dz * dz;
  return j >= 0 && j < n && r2 < kRc2 && r2 > 0.f;
}
// One entry per undirected pair: of (i <- j) and (j <- i) the list keeps the one in the row of the smaller index (rows [0, n_rows) hold
// every pair with at least one end below n_rows).  Caller-supplied lists keep the entry that comes before its partner
// (`partner`, see match_pairs_kernel), or all of them when *asym is set.
// One pass (kReserve): the rows of a CTA are counted, the CTA reserves its stretch of the list with one addition to *total (zero
// beforehand), and the rows are written from a second look at them in the L1.  A row's entries stay together and so do the rows of a CTA;
// the order of the stretches is the order in which the CTAs got there.  No result depends on it, but the gathers of neighbouring tiles
// do once the rows exceed the L2: at 98,304 atoms the attention kernels lose 8 % / 3 % (forward / reverse).  Long lists therefore take
// two passes (kCount, kFill) around a scan of the CTAs' counts, which keep the rows in order.
constexpr int kCompactRows = 16;
// The line: a force evaluation of water (6 A long range) in order / in order of arrival takes 404 / 400 us at 1,536 atoms, 964 / 963 at
// 6,144, 1,125 / 1,125 at 8,193, 1,498 / 1,497 at 12,288, 2,857 / 2,879 at 24,576, 5,275 / 5,363 at 49,152, 10,242 / 10,530 at 98,304: the
// two launches more cost 4 us where launches bind, nothing from 6,000 atoms on, and the order pays from about 16,000.
constexpr int kOrderedRows = 8192;
enum CompactPass { kReserve, kCount, kFill };
template <int PASS>
__global__ void __launch_bounds__(32 * kCompactRows) compact_rows_kernel(int n_rows, int n, const int* __restrict__ row_ptr,
                                                                         const int* __restrict__ nbr_j, const float* dR,
                                                                         const int* partner, const int* asym,
                                                                         int* total, int* blocks, int* __restrict__ ve_i,
                                                                         int* __restrict__ ve_j, float4* __restrict__ ve_d, int2* __restrict__ ve_orig) {
  grid_dep_sync();
  __shared__ int start[kCompactRows + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * kCompactRows + warp;
  const int e0 = i < n_rows ? row_ptr[i] : 0, e1 = i < n_rows ? row_ptr[i + 1] : 0;
  const bool all = asym && *asym != 0;
  auto look = [&](int e, int& j, int& pe, float4& d) -> bool {
    if (e >= e1) return false;
    j = nbr_j[e];
    if (!partner && j <= i) return false;
    float r2;
    d.x = dR[3 * (size_t)e]; d.y = dR[3 * (size_t)e + 1]; d.z = dR[3 * (size_t)e + 2];
    if (!edge_valid(j, n, d.x, d.y, d.z, r2)) return false;
    d.w = sqrtf(r2);
    if (partner && !all) { pe = partner[e]; return e < pe; }
    return true;
  };
  if (PASS == kReserve && blockIdx.x == 0 && threadIdx.x == 0) total[1] = total[2] = 0;      // the tile queue
  int count = 0, j = -1, pe = -1;
  float4 d = f4_zero();
  for (int eb = e0; eb < e1; eb += 32) count += __popc(__ballot_sync(0xffffffffu, look(eb + lane, j, pe, d)));
  if (lane == 0) start[warp + 1] = count;
  __syncthreads();
  if (threadIdx.x == 0) {
    int sum = 0;
    for (int w = 0; w < kCompactRows; ++w) { const int c = start[w + 1]; start[w + 1] = sum; sum += c; }
    if (PASS == kCount) blocks[blockIdx.x] = sum;
    else start[0] = PASS == kFill ? blocks[blockIdx.x] : (sum ? atomicAdd(total, sum) : 0);
  }
  if (PASS == kCount) return;
  __syncthreads();
  int base = start[0] + start[warp + 1];
  for (int eb = e0; eb < e1; eb += 32) {
    const int e = eb + lane;
    const bool valid = look(e, j, pe, d);
    const unsigned m = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      const int q = base + __popc(m & ((1u << lane) - 1u));
      ve_i[q] = i; ve_j[q] = j;
      ve_d[q] = d;
      if (ve_orig) ve_orig[q] = make_int2(e, pe);
    }
    base += __popc(m);
  }
}
// counts -> exclusive offsets, and their sum; one CTA (an eighth of a million atoms per 8 counts of a thread)
__global__ void __launch_bounds__(1024) scan_blocks_kernel(int n, int* blocks, int* total) {
  grid_dep_sync();
  __shared__ int warp_sum_[32];
  const int tid = threadIdx.x, lane = tid & 31, per = (n + 1023) / 1024;
  const int b0 = min(tid * per, n), b1 = min(b0 + per, n);
  int sum = 0;
  for (int b = b0; b < b1; ++b) sum += blocks[b];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
  if (lane == 31) warp_sum_[tid >> 5] = incl;
  __syncthreads();
  if (tid < 32) {
    int v = warp_sum_[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const int t = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += t; }
    warp_sum_[lane] = v;
  }
  __syncthreads();
  int at = incl - sum + (tid >= 32 ? warp_sum_[(tid >> 5) - 1] : 0);
  for (int b = b0; b < b1; ++b) { const int c = blocks[b]; blocks[b] = at; at += c; }
  if (tid == 1023) { total[0] = at; total[1] = total[2] = 0; }      // the sum, the tile queue
}
// Every entry (i <- j, d) inside the cutoff of a caller-supplied list finds its reversed entry (j <- i, -d): the k-th of several equal
// entries of a row takes the k-th match.  *asym is set when an entry has none or the numbers of equal entries differ.  One warp per row.
__global__ void __launch_bounds__(256) match_pairs_kernel(int n_rows, const int* __restrict__ row_ptr, const int* __restrict__ nbr_j,
                                                          const float* __restrict__ dR, int* __restrict__ partner, int* __restrict__ asym) {
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n_rows) return;
  const int e0 = row_ptr[i], e1 = row_ptr[i + 1];
  for (int e = e0 + (threadIdx.x & 31); e < e1; e += 32) {
    const int j = nbr_j[e];
    float r2, q2;
    const float dx = dR[3 * (size_t)e], dy = dR[3 * (size_t)e + 1], dz = dR[3 * (size_t)e + 2];
    if (!edge_valid(j, n_rows, dx, dy, dz, r2)) { partner[e] = -1; continue; }
    const float tol = 1e-5f * sqrtf(r2) + 1e-6f;
    int rank = 0, mult = 0, match = 0, pe = -1;
    for (int p = e0; p < e1; ++p) {
      if (nbr_j[p] != j) continue;
      const float x = dR[3 * (size_t)p], y = dR[3 * (size_t)p + 1], z = dR[3 * (size_t)p + 2];
      if (!edge_valid(j, n_rows, x, y, z, q2) || fabsf(x - dx) > tol || fabsf(y - dy) > tol || fabsf(z - dz) > tol) continue;
      ++mult;
      rank += p < e;
    }
    for (int p = row_ptr[j]; p < row_ptr[j + 1]; ++p) {
      if (nbr_j[p] != i) continue;
      const float x = dR[3 * (size_t)p], y = dR[3 * (size_t)p + 1], z = dR[3 * (size_t)p + 2];
      if (!edge_valid(i, n_rows, x, y, z, q2) || fabsf(x + dx) > tol || fabsf(y + dy) > tol || fabsf(z + dz) > tol) continue;
      if (match == rank) pe = p;
      ++match;
    }
    partner[e] = pe;
    if (match != mult) atomicExch(asym, 1);
  }
}
// the matches have to be mutual (displacements that agree within the tolerance only pairwise could break that)
__global__ void __launch_bounds__(256) check_mutual_kernel(int n_rows, const int* __restrict__ row_ptr, const int* __restrict__ partner, int* asym) {
  const int total = row_ptr[n_rows];
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const int p = partner[e];
    if (p >= 0 && (p == e || partner[p] != e)) { atomicExch(asym, 1); return; }
  }
}
// entries of the directed list: a pair whose ends both own a row stands for two of them
__global__ void __launch_bounds__(256) count_directed_kernel(int n_rows, const int* __restrict__ n_listed, const int* __restrict__ ve_j,
                                                             const int* __restrict__ asym, unsigned long long* total) {
  const int n_entries = *n_listed;
  const bool both = !(asym && *asym != 0);
  unsigned long long c = 0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n_entries; e += (long long)gridDim.x * blockDim.x)
    c += both && ve_j[e] < n_rows ? 2 : 1;
  if (c) atomicAdd(total, c);
}
// Entries per warp of a tile (8 fill the 128 rows): the same number of rounds over the grid, with the entries spread evenly.  A tile's
// time is its chain of phases plus the edge loops, which are as long as a warp's share: a short list runs one thin tile per CTA
// instead of full tiles on a few of them, and the last round of a longer one is not half empty.
__device__ __forceinline__ int entries_per_warp(long long n_edges, int grid) {
  const long long rounds = (n_edges + (long long)TE * grid - 1) / ((long long)TE * grid);
  return (int)((n_edges + 16 * rounds * grid - 1) / (16 * rounds * grid));
}
// Which tiles a CTA takes.  Short lists: an equal share of consecutive tiles.  Long lists: the tiles in the order in which CTAs come free (CTA b
// starts with tiles b and grid + b).  SMs differ by several per cent in the time of a tile (their distance from the L2 slices that hold its
// rows), so equal shares end with the slowest; and all CTAs work in one stretch of the list at a time, whose rows stay in the L2.  A
// tile's inputs are staged beneath the tile before it, so during each tile the one behind the next is asked for.  `queue`: tiles handed
// out beyond the first two of every CTA | CTAs that are through; both zero at the start of a launch: the build of the list clears them,
// and the last CTA to finish puts them back.
// Forward / reverse, us a launch, tiles per CTA: queue | equal shares | a queue of runs of two tiles, which ends with a whole tile too many where
// the share is odd.  2.2: 43.3 / 80.5 | 41.8 / 79.9 | 52.3 / 101.7, 5.2: 76.2 / 155.1 | 75.0 / 154.6 | -, 7.3: 89.5 / 206.1 | 90.0 / 207.1 | -,
// 8.3: 99.4 / 230.4 | 99.9 / 232.6 | 108.5 / 252.6, 14.4: 156 / 374 | 158 / 376 | 166 / 397, 25.8: 264 / 638 | 264 / 681 | 263 / 641,
// 104: 1,003 / 2,474 | 1,028 / 2,698 | 1,003 / 2,501.  The line stands behind the crossing (6): below it the queue's first question costs.
constexpr int kQueuedTiles = 8;                // tiles per CTA from which on the queue is used
struct TileWalk {
  int tile, next, end;      // this tile, the one behind it; tiles from `end` on are not this CTA's
  bool queued;
  SO3LR_HD TileWalk(int n, int grid, int b) {
    const int share = n / grid, more = n - share * grid;
    queued = share >= kQueuedTiles;
    tile = queued ? b : b * share + (b < more ? b : more);
    end = queued ? n : tile + share + (b < more);
    next = tile;
  }
  SO3LR_HD int second(int grid) const { return grid + tile; }
  SO3LR_HD static int handed(int grid, int ticket) { return 2 * grid + ticket; }
  // `handed_out`: two words in shared memory, taken in turns (`turn`): a warp may still look up the next tile when another one is at the end of
  // this one and writes the tile that follows
  SO3LR_HD void look_ahead(const int* handed_out, uint32_t turn) { next = queued ? handed_out[turn] : tile + 1; }
  // one thread per CTA, behind its last tile
  __device__ __forceinline__ void finish(int* queue) const {
    if (queued && atomicAdd(queue + 1, 1) == (int)gridDim.x - 1) { atomicExch(queue, 0); atomicExch(queue + 1, 0); }
  }
};
// `body(full)` with full = true_type where a warp's share is the whole run its loops are unrolled for (the run of a long list: branches
// on the share inside the loops cost 4 % there), false_type where it is shorter
template <class Body>
__device__ __forceinline__ void edge_loops(int share, Body&& body, int run = 8) {
  if (share == run) body(std::true_type{});
  else body(std::false_type{});
}

// ------------------------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------------------------
// 16 warps.  Per tile: (1) preparation of the A operand and the records: Chebyshev terms by two threads per pair, geometry by a third (the
// fourth's warps issue the MMAs), then the hidden layers by four neighbouring threads per pair; (2) the MMA chains of the two filters, while
// every warp already has the sender rows of its 8 pairs in flight; (3) per filter: tensor memory -> shared tile, then the edge loop.
__global__ void __launch_bounds__(kFwThreads, 1) attn_fwd_tc_kernel(const unsigned char* __restrict__ img_g, const float* __restrict__ sph1_k,
                                                                    const float* __restrict__ sph1_b, int n_recv,
                                                                    const int* n_listed, const int* ve_i,
                                                                    const int* ve_j, const float4* ve_d,
                                                                    const float* qkv, const float* ev_in,
                                                                    float* __restrict__ xa, float* __restrict__ ev1, int* __restrict__ err,
                                                                    long long* __restrict__ dbg, const int* asym, int* queue) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  float* rec = reinterpret_cast<float*>(smem + kOffFwRec);
  float* sph = reinterpret_cast<float*>(smem + kOffFwSph);
  float* wt = reinterpret_cast<float*>(smem + kOffA);
  int* st_ij = reinterpret_cast<int*>(smem + kOffFwStIJ);
  float4* st_d = reinterpret_cast<float4*>(smem + kOffFwStD);
  unsigned long long* mbar_p = reinterpret_cast<unsigned long long*>(smem + kOffFwMisc);
  uint32_t* tmem_p = reinterpret_cast<uint32_t*>(smem + kOffFwMisc + 16);
  volatile int* failed = reinterpret_cast<volatile int*>(smem + kOffFwMisc + 20);
  int* handed_out = reinterpret_cast<int*>(smem + kOffFwMisc + 32);
  for (int k = tid; k < kTcImageBytes / 16; k += kFwThreads) reinterpret_cast<uint4*>(smem + kOffImg)[k] = reinterpret_cast<const uint4*>(img_g)[k];
  for (int k = tid; k < 512; k += kFwThreads) {      // [filter][hidden unit][w0 w1 w2 w3 b - - -]
    const int q = k & 7, c = (k >> 3) & 31, f = k >> 8;
    sph[sph_at(f, c) + q] = q < 4 ? sph1_k[f * 128 + q * 32 + c] : (q == 4 ? sph1_b[f * 32 + c] : 0.f);
  }
  const uint32_t mbar0 = smem_u32(mbar_p);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(mbar0));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *failed = 0;
  }
  grid_dep_sync();
  const long long n_edges = *n_listed;
  if (n_edges <= 0) return;
  const int rpw = entries_per_warp(n_edges, gridDim.x), tr = 16 * rpw;      // entries per warp / per tile
  TileWalk walk((int)((n_edges + tr - 1) / tr), (int)gridDim.x, (int)blockIdx.x);
  if (walk.tile >= walk.end) return;
  const int pad_i = ve_i[n_edges - 1];
  // partners below n_scat receive the pair's other direction (j <- i)
  const int n_scat = asym && *asym != 0 ? 0 : n_recv;
  const int half = warp >> 3;            // the rows of this warp's pairs: [64 half, 64 half + 8 rpw)
  // list entry of a tile row within the tile, -1 for a padding row
  auto entry_of = [&](int row) { return (row & 63) < 8 * rpw ? (row & 63) + (row >> 6) * 8 * rpw : -1; };
  // (i, j) and displacement of one tile's pairs into the staging buffers (threads 256..383): in flight beneath the tile before
  auto stage_tile = [&](int tile) {
    if (tid < 256 || tid >= 384 || tile >= walk.end) return;
    const int row = tid - 256, k = entry_of(row);
    const long long e = (long long)tile * tr + k;
    if (k >= 0 && e < n_edges) {
      cp_async4(st_ij + 2 * row, ve_i + e); cp_async4(st_ij + 2 * row + 1, ve_j + e);
      cp_async16(st_d + row, ve_d + e);
    } else {
      st_ij[2 * row] = pad_i; st_ij[2 * row + 1] = pad_i;
      st_d[row] = make_float4(1.f, 0.f, 0.f, 1.f);
    }
  };
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_p)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  stage_tile(walk.tile);
  if (tid == 0) handed_out[0] = walk.second((int)gridDim.x);
  cp_async_wait_all();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_p, 0);
  const uint32_t on = elect_one();
  const bool issues = warp >= 12;      // one warp per scheduler, of those with the shortest preparation
  const uint32_t a_hi = smem_u32(smem + kOffA), img = smem_u32(smem + kOffImg);
  const int col = 4 * lane;
  const int deg = degree_of(lane < kMTot ? lane : 0);
  const int k0 = 64 * half + rpw * (warp & 7);      // this warp's rows of the tile in the edge loop
  auto sync_group = [&] { asm volatile("bar.sync %0, 256;" ::"r"(2 + half) : "memory"); };
  uint32_t parity = 0;
#ifdef SO3LR_TC_TIMING
  long long tph[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  long long tc0 = clock64();
  if (dbg && tid == 32 && blockIdx.x == 0) dbg[8] = 0;
#define TC_MARK(k) do { if (dbg && (tid & 31) == 0) { const long long c = clock64(); tph[k] += c - tc0; tc0 = c; } } while (0)
#define TC_TILE(slot) do { if (dbg && tid == 32 && blockIdx.x == 0) ++dbg[slot]; } while (0)
#else
#define TC_MARK(k) do { } while (0)
#define TC_TILE(slot) do { } while (0)
#endif
  for (; walk.tile < walk.end; walk.tile = walk.next) {
    const long long entry0 = (long long)walk.tile * tr;
    int run = 0;
    // ---- per-edge preparation ----
    {
      const int hrow = 8 * warp + (lane >> 2);
      PairInvariants I;      // requested first, used last
      I.begin(ev_in + (size_t)st_ij[2 * hrow] * kMTot, ev_in + (size_t)st_ij[2 * hrow + 1] * kMTot, lane & 3);
      const int row = tid & 127, role = tid >> 7;
      const int entry = entry_of(row);
      const bool valid = entry >= 0 && entry0 + entry < n_edges;
      const float4 d = st_d[row];
      const float r = d.w;
      if (role < 2) {
        // once these 256 threads are through, their share of the MMA chains starts beneath the rest of the preparation
        store_chebyshev_half(smem + kOffA, row, r, valid, role);
        fence_async_smem();
        asm volatile("bar.arrive 1, 384;" ::: "memory");
      } else if (role == 2) {
        const float ir = 1.f / r;
        float cut, dcut;
        phys_cutoff(r, cut, dcut);
        float Y[kMTot];
        sph_harm_24(d.x * ir, d.y * ir, d.z * ir, Y);
        float* rp = rec + row * kFwRec;
        st4(rp, make_float4(__int_as_float(st_ij[2 * row + 1]), __int_as_float(st_ij[2 * row]), valid ? cut * kInvNbar : 0.f, 0.f));
#pragma unroll
        for (int c = 0; c < 6; ++c) st4(rp + 4 + 4 * c, make_float4(Y[4 * c], Y[4 * c + 1], Y[4 * c + 2], Y[4 * c + 3]));
      }
      float s[4];
      I.finish(s);
      store_spherical_hidden_quarter(smem + kOffA, hrow, s, sph, lane & 3);
      if (issues) {
        asm volatile("bar.sync 1, 384;" ::: "memory");
        tc_fence_after();
        issue_forward_mma(on, tmem, a_hi, img, (warp >> 1) & 1, warp & 1, 0);
      }
    }
    TC_MARK(0);
    // the partners' q / k rows of filter 0 for this warp's pairs and the first receiver's rows: in flight while the tensor cores run.  The
    // indices are in the staging buffer since the previous tile, so the warps ask for them before the barrier; those that issue the MMAs do
    // after it, because an MMA waits behind the loads in its scheduler's queue
    float4 qj[8], kj[8], qi, ki, vi;
    int cur_i, jr[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) jr[u] = st_ij[2 * ((k0 + u) & (TE - 1)) + 1];      // past this warp's share: not used
    cur_i = st_ij[2 * k0];
    auto request_rows = [&] {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float* pj = qkv + (size_t)jr[u] * kProj + col;
        qj[u] = ld4(pj);
        kj[u] = ld4(pj + kF);
      }
      const float* pi = qkv + (size_t)cur_i * kProj + col;
      qi = ld4(pi); ki = ld4(pi + kF); vi = ld4(pi + 2 * kF);
    };
    if (!issues) request_rows();
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    TC_MARK(1);
    walk.look_ahead(handed_out, parity);
    if (issues) {
      tc_fence_after();
      issue_forward_mma(on, tmem, a_hi, img, (warp >> 1) & 1, warp & 1, 1);
      umma_commit_if(on, mbar0);
      request_rows();
    }
    stage_tile(walk.next);
    if (tid == kFwThreads - 1 && walk.queued) run = TileWalk::handed((int)gridDim.x, atomicAdd(queue, 1));
    wait_mma(mbar0, parity, failed, err);
    parity ^= 1;
    TC_MARK(2);
    // ---- filter 0: invariant logits, feature sums ----
    tmem_to_tile(tmem, 0, warp, lane, wt);
    tc_fence_before();
    sync_group();
    TC_MARK(3);
    edge_loops(rpw, [&](auto full) {
      // logits x cutoff of both directions: a of (i <- j), b of (j <- i); b's message goes out at once, a's are summed per receiver.
      // The value rows are requested as the q / k registers of a pair come free.
      float a[8];
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        const float* rp = rec + (k0 + h) * kFwRec;
        if (full && __float_as_int(rp[1]) == __float_as_int(rp[3 * kFwRec + 1])) {      // four pairs of one receiver: their sums together
          if (__float_as_int(rp[1]) != cur_i) {
            cur_i = __float_as_int(rp[1]);
            const float* pi = qkv + (size_t)cur_i * kProj + col;
            qi = ld4(pi); ki = ld4(pi + kF); vi = ld4(pi + 2 * kF);
          }
          float v[8];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 w = ld4(wt + (k0 + h + u) * kWStride + col);
            v[2 * u] = dot3(qi, w, kj[h + u]);
            v[2 * u + 1] = dot3(qj[h + u], w, ki);
          }
          const float d = transpose_sum8(v, lane & 7) * rp[((lane & 7) >> 1) * kFwRec + 2];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = __float_as_int(rp[u * kFwRec]);
            a[h + u] = __shfl_sync(0xffffffffu, d, (lane & 24) + 2 * u);
            const float b = __shfl_sync(0xffffffffu, d, (lane & 24) + 2 * u + 1);
            if (j < n_scat) red_add_v4(xa + (size_t)j * kF + col, f4_scale(b, vi));
            qj[h + u] = ld4(qkv + (size_t)j * kProj + 2 * kF + col);
          }
          continue;
        }
#pragma unroll
        for (int u = h; u < h + 4; ++u) {
          if (!full && u >= rpw) break;
          const float4 r0 = ld4(rec + (k0 + u) * kFwRec);
          const int j = __float_as_int(r0.x), i = __float_as_int(r0.y);
          if (i != cur_i) {
            cur_i = i;
            const float* pi = qkv + (size_t)cur_i * kProj + col;
            qi = ld4(pi); ki = ld4(pi + kF); vi = ld4(pi + 2 * kF);
          }
          const float4 w = ld4(wt + (k0 + u) * kWStride + col);
          a[u] = group8_sum(dot3(qi, w, kj[u])) * r0.z;
          const float b = group8_sum(dot3(qj[u], w, ki)) * r0.z;
          if (j < n_scat && r0.z != 0.f) red_add_v4(xa + (size_t)j * kF + col, f4_scale(b, vi));
          qj[u] = ld4(qkv + (size_t)j * kProj + 2 * kF + col);
        }
      }
      float4 accx = f4_zero();
      cur_i = __float_as_int(rec[k0 * kFwRec + 1]);
      if (full && cur_i == __float_as_int(rec[(k0 + 7) * kFwRec + 1])) {
#pragma unroll
        for (int u = 0; u < 8; ++u) accx = f4_fma(a[u], qj[u], accx);
      } else {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (!full && u >= rpw) break;
          const int i = __float_as_int(rec[(k0 + u) * kFwRec + 1]);
          if (i != cur_i) {
            if (f4_nonzero(accx)) red_add_v4(xa + (size_t)cur_i * kF + col, accx);
            cur_i = i;
            accx = f4_zero();
          }
          accx = f4_fma(a[u], qj[u], accx);
        }
      }
      if (f4_nonzero(accx)) red_add_v4(xa + (size_t)cur_i * kF + col, accx);
    });
    // rows of filter 1: in flight across the barrier and the second tile copy
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float* pj = qkv + (size_t)__float_as_int(rec[((k0 + u) & (TE - 1)) * kFwRec]) * kProj + 3 * kF + col;
      qj[u] = ld4(pj);
      kj[u] = ld4(pj + kF);
    }
    cur_i = __float_as_int(rec[k0 * kFwRec + 1]);
    qi = ld4(qkv + (size_t)cur_i * kProj + 3 * kF + col);
    ki = ld4(qkv + (size_t)cur_i * kProj + 4 * kF + col);
    TC_MARK(4);
    sync_group();
    TC_MARK(5);
    // ---- filter 1: equivariant logits, spherical-harmonic sums ----
    tmem_to_tile(tmem, 1, warp, lane, wt);
    tc_fence_before();
    sync_group();
    TC_MARK(6);
    edge_loops(rpw, [&](auto full) {
      float accev = 0.f;
      const float sgn = deg == 0 || deg == 2 ? -1.f : 1.f;      // Y_lm(-u) = (-1)^l Y_lm(u)
      auto new_receiver = [&](int i) {
        if (lane < kMTot && accev != 0.f) atomicAdd(ev1 + (size_t)cur_i * kMTot + lane, accev);
        cur_i = i;
        accev = 0.f;
        qi = ld4(qkv + (size_t)cur_i * kProj + 3 * kF + col);
        ki = ld4(qkv + (size_t)cur_i * kProj + 4 * kF + col);
      };
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        const float* rp = rec + (k0 + h) * kFwRec;
        if (full && __float_as_int(rp[1]) == __float_as_int(rp[3 * kFwRec + 1])) {
          if (__float_as_int(rp[1]) != cur_i) new_receiver(__float_as_int(rp[1]));
          float v[8];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 w = ld4(wt + (k0 + h + u) * kWStride + col);
            v[2 * u] = dot3(qi, w, kj[h + u]);
            v[2 * u + 1] = dot3(qj[h + u], w, ki);
          }
          const float d = transpose_sum8(v, lane & 7) * rp[((lane & 7) >> 1) * kFwRec + 2];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = __float_as_int(rp[u * kFwRec]);
            const float ym = lane < kMTot ? rp[u * kFwRec + 4 + lane] : 0.f;
            accev = fmaf(__shfl_sync(0xffffffffu, d, 8 * deg + 2 * u), ym, accev);
            const float bd = __shfl_sync(0xffffffffu, d, 8 * deg + 2 * u + 1);
            if (lane < kMTot && j < n_scat) atomicAdd(ev1 + (size_t)j * kMTot + lane, sgn * bd * ym);
          }
          continue;
        }
#pragma unroll
        for (int u = h; u < h + 4; ++u) {
          if (!full && u >= rpw) break;
          const float4 r0 = ld4(rec + (k0 + u) * kFwRec);
          const int j = __float_as_int(r0.x), i = __float_as_int(r0.y);
          if (i != cur_i) new_receiver(i);
          const float4 w = ld4(wt + (k0 + u) * kWStride + col);
          const float a = group8_sum(dot3(qi, w, kj[u])) * r0.z;
          const float b = group8_sum(dot3(qj[u], w, ki)) * r0.z;
          const float ym = lane < kMTot ? rec[(k0 + u) * kFwRec + 4 + lane] : 0.f;
          accev = fmaf(__shfl_sync(0xffffffffu, a, 8 * deg), ym, accev);
          const float bd = __shfl_sync(0xffffffffu, b, 8 * deg);
          if (lane < kMTot && j < n_scat && r0.z != 0.f) atomicAdd(ev1 + (size_t)j * kMTot + lane, sgn * bd * ym);
        }
      }
      if (lane < kMTot && accev != 0.f) atomicAdd(ev1 + (size_t)cur_i * kMTot + lane, accev);
    });
    cp_async_wait_all();
    if (tid == kFwThreads - 1 && walk.queued) handed_out[parity] = run;
    __syncthreads();
    TC_MARK(7);
    TC_TILE(8);
  }
#ifdef SO3LR_TC_TIMING
  if (dbg && tid == 32 && blockIdx.x == 0) { for (int q = 0; q < 8; ++q) dbg[q] = tph[q]; }
  if (dbg && (tid & 31) == 0 && blockIdx.x == 0) { for (int q = 0; q < 8; ++q) dbg[160 + 8 * warp + q] = tph[q]; }
#endif
  if (tid == kFwThreads - 1) walk.finish(queue);
  cp_async_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

}  // namespace

namespace {

// ------------------------------------------------------------------------------------------------------------------
// reverse
// ------------------------------------------------------------------------------------------------------------------
// [dPhi | dhs_f] = dw_f * [C_f^T | K2_f^T] (the same image read K-major: N = 96 rows, K = features): main accumulators in TMEM
// columns [128 f, 128 f + 96), cross 256 columns above
__device__ __forceinline__ void issue_reverse_mma(uint32_t on, uint32_t tmem, uint32_t a_hi, uint32_t img, int f, int half, int cross) {
  const uint64_t da = desc_base(kLboA, 128) + (a_hi >> 4), dal = da + (kAHalf >> 4);
  const uint64_t db = desc_base(1536, 128) + ((img + f * kRevImgFilter) >> 4), dbl = db + (2 * kRevImgFilter >> 4);
  const uint32_t id96 = make_idesc(96, 0);
  const uint32_t d = tmem + 128 * f + 256 * cross;
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {      // K = 16 features per step
    const uint64_t ah = da + ks * (2 * kLboA >> 4), al = dal + ks * (2 * kLboA >> 4);
    const uint64_t bh = db + ks * (2 * 1536 >> 4), bl = dbl + ks * (2 * 1536 >> 4);
    if (!cross) {
      umma_half_if(on, d, ah, bh, id96, ks > 0, half);
    } else {
      umma_half_if(on, d, ah, bl, id96, ks > 0, half);
      umma_half_if(on, d, al, bh, id96, 1, half);
    }
  }
}

// Sender-side q / k rows of four consecutive tile rows for the reverse edge loop of filter F (lane = 4 features)
// (for every row of the four: past a warp's share these are rows of other warps, whose values are not used)
struct RevLoads {
  float4 qj[4], kj[4];
  template <int F>
  __device__ __forceinline__ void fetch(int u, const float* rec, int row, int lane, const float* __restrict__ qkv) {
    const float* pj = qkv + (size_t)__float_as_int(rec[(row & (TE - 1)) * kBwRec]) * kProj + F * 3 * kF + 4 * lane;
    qj[u] = ld4(pj);
    kj[u] = ld4(pj + kF);
  }
};
// A receiver's q / k rows and the sums of their cotangents, which a warp carries through its pairs
struct Receiver {
  float4 q, k, gq, gk;
  int i;
  template <int F>
  __device__ __forceinline__ void start(int receiver, int lane, const float* __restrict__ qkv) {
    i = receiver;
    const float* pi = qkv + (size_t)i * kProj + F * 3 * kF + 4 * lane;
    q = ld4(pi);
    k = ld4(pi + kF);
    gq = f4_zero(); gk = f4_zero();
  }
  template <int F>
  __device__ __forceinline__ void flush(int lane, float* __restrict__ g_qkv) const {
    float* gi = g_qkv + (size_t)i * kProj + F * 3 * kF + 4 * lane;
    if (f4_nonzero(gq)) red_add_v4(gi, gq);
    if (f4_nonzero(gk)) red_add_v4(gi + kF, gk);
  }
};
template <int F>
__device__ __forceinline__ void reverse_prefetch(RevLoads& L, const float* rec, int row0, int lane, const float* __restrict__ qkv) {
#pragma unroll
  for (int u = 0; u < 4; ++u) L.fetch<F>(u, rec, row0 + u, lane, qkv);
}

// Value path of the invariant filter, split off the edge loop so that it runs while the tensor cores are busy.
// Before the loop (rows [row0, row0 + nu), nu <= 8, of one warp): cotangents of the invariant logits of both directions of every edge,
// daA_h = <g_xa[i], v[j]>_h and daB_h = <g_xa[j], v[i]>_h, into record fields 24..27 and 28..31.
template <bool FULL>
__device__ __forceinline__ void value_logit_cotangents(float* rec, int row0, int nu, int lane, const float* __restrict__ qkv,
                                                       const float* __restrict__ g_xa) {
  const int col = 4 * lane, grp = lane >> 3, cg = lane & 7;
  int cur_i = -1;
  float4 v_i = f4_zero(), gx_i = f4_zero();
#pragma unroll
  for (int k0 = 0; k0 < 8; k0 += 4) {
    float4 vj[4], gxj[4];
    int ii[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float* rp = rec + ((row0 + k0 + u) & (TE - 1)) * kBwRec;
      const int j = __float_as_int(rp[0]);
      ii[u] = __float_as_int(rp[1]);
      vj[u] = ld4(qkv + (size_t)j * kProj + 2 * kF + col);
      gxj[u] = ld4(g_xa + (size_t)j * kF + col);
    }
    if (FULL && ii[0] == ii[3]) {      // four pairs of one receiver
      if (ii[0] != cur_i) {
        cur_i = ii[0];
        v_i = ld4(qkv + (size_t)cur_i * kProj + 2 * kF + col);
        gx_i = ld4(g_xa + (size_t)cur_i * kF + col);
      }
      float v[8];
#pragma unroll
      for (int u = 0; u < 4; ++u) { v[2 * u] = dot2(gx_i, vj[u]); v[2 * u + 1] = dot2(gxj[u], v_i); }
      rec[(row0 + k0 + (cg >> 1)) * kBwRec + 24 + 4 * (cg & 1) + grp] = transpose_sum8(v, cg);
      continue;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (!FULL && k0 + u >= nu) break;
      if (ii[u] != cur_i) {
        cur_i = ii[u];
        v_i = ld4(qkv + (size_t)cur_i * kProj + 2 * kF + col);
        gx_i = ld4(g_xa + (size_t)cur_i * kF + col);
      }
      const float daA = group8_sum(dot2(gx_i, vj[u])), daB = group8_sum(dot2(gxj[u], v_i));
      if (cg == 0) {
        float* rp = rec + (row0 + k0 + u) * kBwRec;
        rp[24 + grp] = daA;
        rp[28 + grp] = daB;
      }
    }
  }
}

// two unit vectors that span the plane across u, without a branch at either pole (Duff et al., J. Comput. Graph. Tech. 6, 2017)
__device__ __forceinline__ void tangent_frame(float ux, float uy, float uz, float* e1, float* e2) {
  const float s = copysignf(1.f, uz), a = -1.f / (s + uz), b = ux * uy * a;
  e1[0] = fmaf(s * ux * ux, a, 1.f); e1[1] = s * b; e1[2] = -s * ux;
  e2[0] = b; e2[1] = fmaf(uy * uy, a, s); e2[2] = -uy;
}
// What one end's cotangent of ev contributes to a pair, ahead of the logits: dl[l] = sum_m g_lm Y_lm (cotangent of the equivariant logit)
// and, per degree, the two components across the pair of the transposed harmonics (field + 2 l of the record): the angular force is
// their sum weighted with the logits.
template <int L>
__device__ __forceinline__ void angular_degree(const float* g, const float* Y, const float* u, const float* e1, const float* e2, float sign,
                                               float* dl, float* t) {
  constexpr int m0 = L * L - 1;
  float d = 0.f;
#pragma unroll
  for (int m = 0; m < 2 * L + 1; ++m) d = fmaf(g[m0 + m], Y[m0 + m], d);
  float gx = 0.f, gy = 0.f, gz = 0.f;
  sph_harm_vjp_degree<L>(u[0], u[1], u[2], g + m0, gx, gy, gz);
  dl[L - 1] = sign * d;
  t[2 * (L - 1)] = sign * fmaf(gx, e1[0], fmaf(gy, e1[1], gz * e1[2]));
  t[2 * (L - 1) + 1] = sign * fmaf(gx, e2[0], fmaf(gy, e2[1], gz * e2[2]));
}
// `odd`: sign of the odd degrees, Y_lm(-u) = (-1)^l Y_lm(u)
__device__ __forceinline__ void angular_end(const float* __restrict__ gev, float ux, float uy, float uz, float odd, float* rp_dl, float* rp_t) {
  float g[kMTot];
#pragma unroll
  for (int c = 0; c < 6; ++c) st4(g + 4 * c, ld4(gev + 4 * c));
  const float u[3] = {ux, uy, uz};
  float Y[kMTot], e1[3], e2[3], dl[4], t[8];
  sph_harm_24(ux, uy, uz, Y);
  tangent_frame(ux, uy, uz, e1, e2);
  angular_degree<1>(g, Y, u, e1, e2, odd, dl, t);
  angular_degree<2>(g, Y, u, e1, e2, 1.f, dl, t);
  angular_degree<3>(g, Y, u, e1, e2, odd, dl, t);
  angular_degree<4>(g, Y, u, e1, e2, 1.f, dl, t);
  st4(rp_dl, make_float4(dl[0], dl[1], dl[2], dl[3]));
  st4(rp_t, make_float4(t[0], t[1], t[2], t[3]));
  st4(rp_t + 4, make_float4(t[4], t[5], t[6], t[7]));
}

// After the loop: cotangents of the value rows, gv_i = sum over its pairs (cutoff x logit of edge j<-i)_h g_xa[j] (fields 28..31) and,
// pair by pair, gv_j += (cutoff x logit of edge i<-j)_h g_xa[i] (fields 24..27)
template <bool FULL>
__device__ __forceinline__ void value_cotangent(const float* rec, int row0, int nu, int lane, const float* __restrict__ g_xa,
                                                float* __restrict__ g_qkv, int n_scat) {
  const int col = 4 * lane, grp = lane >> 3;
  auto record = [&](int k) { return rec + ((row0 + k) & (TE - 1)) * kBwRec; };
  float4 gxj[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) gxj[u] = ld4(g_xa + (size_t)__float_as_int(record(u)[0]) * kF + col);
  int cur_i = __float_as_int(record(0)[1]);
  float4 gv = f4_zero(), gxi = ld4(g_xa + (size_t)cur_i * kF + col);
  if (FULL && cur_i == __float_as_int(record(7)[1])) {      // eight pairs of one receiver
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float* rp = record(u);
      const int j = __float_as_int(rp[0]);
      gv = f4_fma(rp[28 + grp], gxj[u], gv);
      if (j < n_scat) red_add_v4(g_qkv + (size_t)j * kProj + 2 * kF + col, f4_scale(rp[24 + grp], gxi));
    }
    red_add_v4(g_qkv + (size_t)cur_i * kProj + 2 * kF + col, gv);
    return;
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    if (!FULL && u >= nu) break;
    const float* rp = record(u);
    const float4 r0 = ld4(rp);
    const int j = __float_as_int(r0.x), i = __float_as_int(r0.y);
    if (i != cur_i) {
      if (f4_nonzero(gv)) red_add_v4(g_qkv + (size_t)cur_i * kProj + 2 * kF + col, gv);
      cur_i = i;
      gv = f4_zero();
      gxi = ld4(g_xa + (size_t)cur_i * kF + col);
    }
    gv = f4_fma(rp[28 + grp], gxj[u], gv);
    if (j < n_scat && r0.z != 0.f) red_add_v4(g_qkv + (size_t)j * kProj + 2 * kF + col, f4_scale(rp[24 + grp], gxi));
  }
  if (f4_nonzero(gv)) red_add_v4(g_qkv + (size_t)cur_i * kProj + 2 * kF + col, gv);
}

// dw of one pair as A operand of the second MMA chain: row = pair, columns 4 lane .. 4 lane + 3 of the hi and the lo matrix
__device__ __forceinline__ void store_dw(unsigned char* a_hi, int row, int lane, float4 dw) {
  uint2 h, l;
  split2(dw.x, dw.y, h.x, l.x); split2(dw.z, dw.w, h.y, l.y);
  unsigned char* p = a_hi + (lane >> 1) * kLboA + row * 16 + (lane & 1) * 8;
  *reinterpret_cast<uint2*>(p) = h;
  *reinterpret_cast<uint2*>(p + kAHalf) = l;
}
// Reverse edge loop of filter F over nu <= 4 tile rows [row0, row0 + nu) of one warp: logits of both directions of every edge,
// cotangents of this receiver's q / k rows (added to g_qkv with vector reductions when the receiver changes), dw into the
// A operand of the second MMA chain, the cutoff part of d/dr into the records.  The cotangents of the logits come from the
// records (fields 24.. for the invariant filter, 16.. for the equivariant one); cutoff x logit takes their place.
// NEXT: the rows of the four pairs that follow are requested as these come free.
template <int F, bool FULL, bool NEXT>
__device__ __forceinline__ void reverse_edges4(RevLoads& L, Receiver& S, float* rec, const float* wt, int wrow0, int row0, int nu,
                                               unsigned char* a_hi, int lane, const float* __restrict__ qkv, float* __restrict__ g_qkv, int n_scat) {
  constexpr int kField = F ? 16 : 24;
  const int col = 4 * lane, grp = lane >> 3, cg = lane & 7;
  const int first_i = __float_as_int(rec[row0 * kBwRec + 1]);
  if (first_i != S.i) {
    S.flush<F>(lane, g_qkv);
    S.start<F>(first_i, lane, qkv);
  }
  if (FULL && first_i == __float_as_int(rec[(row0 + 3) * kBwRec + 1])) {
    // four pairs of one receiver (five runs of six): no branches between the rows, the eight logits summed together; lane cg of a head's
    // group then holds row cg / 2, direction cg & 1
    float v[8];
    float4 w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      w[u] = ld4(wt + (wrow0 + u) * kWStride + col);
      v[2 * u] = dot3(S.q, w[u], L.kj[u]);
      v[2 * u + 1] = dot3(L.qj[u], w[u], S.k);
    }
    float* mp = rec + (row0 + (cg >> 1)) * kBwRec;
    const int dir = cg & 1;
    const float sc = mp[2], dcn = mp[3], da = mp[kField + 4 * dir + grp];
    const float D = transpose_sum8(v, cg);
    mp[kField + 4 * dir + grp] = sc * D;
    const float dD = sc * da;
    float gc = dcn * da * D;      // cutoff part of d/dr, summed over the directions and heads
    gc += __shfl_xor_sync(0xffffffffu, gc, 1);
    gc += __shfl_xor_sync(0xffffffffu, gc, 8);
    gc += __shfl_xor_sync(0xffffffffu, gc, 16);
    if (grp == 0 && dir == 0) mp[12] += gc;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float dDA = __shfl_sync(0xffffffffu, dD, (lane & 24) + 2 * u), dDB = __shfl_sync(0xffffffffu, dD, (lane & 24) + 2 * u + 1);
      const float4 aw = f4_scale(dDA, w[u]), bw = f4_scale(dDB, w[u]);
      S.gq = f4_mad(aw, L.kj[u], S.gq);
      S.gk = f4_mad(bw, L.qj[u], S.gk);
      const int j = __float_as_int(rec[(row0 + u) * kBwRec]);
      if (j < n_scat) {
        float* gj = g_qkv + (size_t)j * kProj + F * 3 * kF + col;
        red_add_v4(gj, f4_mul(bw, S.k));
        red_add_v4(gj + kF, f4_mul(aw, S.q));
      }
      store_dw(a_hi, row0 + u, lane, f4_fma(dDA, f4_mul(S.q, L.kj[u]), f4_scale(dDB, f4_mul(L.qj[u], S.k))));
      if (NEXT) L.fetch<F>(u, rec, row0 + 4 + u, lane, qkv);
    }
    return;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (!FULL && u >= nu) break;
    const int row = row0 + u;
    float* rp = rec + row * kBwRec;
    const float4 r0 = ld4(rp);
    const int j = __float_as_int(r0.x), i = __float_as_int(r0.y);
    const float sc = r0.z, dcn = r0.w;
    if (i != S.i) {      // rare: a run of four rows mostly stays with one receiver
      S.flush<F>(lane, g_qkv);
      S.start<F>(i, lane, qkv);
    }
    const float4 w = ld4(wt + (wrow0 + u) * kWStride + col);
    const float4 pA = f4_mul(S.q, L.kj[u]), pB = f4_mul(L.qj[u], S.k);      // serve both the logits and dw
    const float DA = group8_sum(dot2(w, pA)), DB = group8_sum(dot2(w, pB));
    const float daA = rp[kField + grp], daB = rp[kField + 4 + grp];
    __syncwarp();      // the eight lanes of a head have read its cotangents: the logits take their place
    if (cg == 0) { rp[kField + grp] = sc * DA; rp[kField + 4 + grp] = sc * DB; }
    const float dDA = sc * daA, dDB = sc * daB;
    const float4 aw = f4_scale(dDA, w), bw = f4_scale(dDB, w);
    S.gq = f4_mad(aw, L.kj[u], S.gq);
    S.gk = f4_mad(bw, L.qj[u], S.gk);
    if (j < n_scat && sc != 0.f) {      // the partner's shares: gq_j = dDB w k_i, gk_j = dDA w q_i
      float* gj = g_qkv + (size_t)j * kProj + F * 3 * kF + col;
      red_add_v4(gj, f4_mul(bw, S.k));
      red_add_v4(gj + kF, f4_mul(aw, S.q));
    }
    store_dw(a_hi, row, lane, f4_fma(dDA, pA, f4_scale(dDB, pB)));
    if (NEXT) L.fetch<F>(u, rec, row0 + 4 + u, lane, qkv);
    // cutoff part of d/dr, summed over the four heads
    float gc = dcn * fmaf(daA, DA, daB * DB);
    gc += __shfl_xor_sync(0xffffffffu, gc, 8);
    gc += __shfl_xor_sync(0xffffffffu, gc, 16);
    if (lane == 0) rp[12] += gc;
  }
}
// ... over a warp's nu <= 8 pairs
template <int F>
__device__ __forceinline__ void reverse_edges(RevLoads& L, float* rec, const float* wt, int wrow0, int row0, int nu, unsigned char* a_hi, int lane,
                                              const float* __restrict__ qkv, float* __restrict__ g_qkv, int n_scat, Receiver& S) {
  if (nu == 8) {
    reverse_edges4<F, true, true>(L, S, rec, wt, wrow0, row0, 4, a_hi, lane, qkv, g_qkv, n_scat);
    reverse_edges4<F, true, false>(L, S, rec, wt, wrow0 + 4, row0 + 4, 4, a_hi, lane, qkv, g_qkv, n_scat);
  } else {
    for (int k = 0; k < nu; k += 4) {
      if (k) reverse_prefetch<F>(L, rec, row0 + k, lane, qkv);
      reverse_edges4<F, false, false>(L, S, rec, wt, wrow0 + k, row0 + k, nu - k, a_hi, lane, qkv, g_qkv, n_scat);
    }
  }
  S.flush<F>(lane, g_qkv);
}

// record fields (floats): 0 j | 1 i | 2 cutoff / nbar | 3 its r-derivative | 4-7 invariants | 8-10 unit vector | 11 1/r |
// 12 d/dr (cutoff part) | 13 r | 14 1 for a list entry, 0 for a padding row | 16-19, 20-23 cotangents of the equivariant logits of edge
// (i<-j) and (j<-i), after that filter's loop the logits x cutoff | 24-27, 28-31 the same of the invariant logits |
// 32-39, 40-47 transposed harmonics of both ends' cotangents of ev across the pair, two components per degree (angular_end)
//
// 16 warps in two groups: the pairs of rows 0..63 belong to warps 0..7, those of rows 64..127 to warps 8..15.  Per tile: (1) all prepare the
// records and the A operand: Chebyshev terms by two threads per pair, the ev cotangents of the two ends by two others, then the hidden layers
// by four neighbouring threads per pair; (2) MMA chain w = Phi C + hs K2 (both filters, all rows), beneath it the value path's logit
// cotangents; (3) per filter and group: tensor memory -> filter tile (64 rows), reverse edge loop, dw into the A operand, MMA chain
// [dPhi | dhs] = dw [C^T | K2^T] of the group's rows (the other rows' results switched off).  The groups take turns with the filter tile:
// the edge loops are bound by their row reductions (an SM sends 21 to 26 bytes per cycle), so while one group runs its loop the other goes
// through the value path, the wait for its MMAs and the copy of its accumulators; (4) per pair the radial derivative and the spherical
// hidden layer (the first filter's beneath the second filter's last chain); (5) force on the receiver, cotangent of ev.
// PER_ENTRY (caller-supplied lists): `F` is the gradient with respect to the source list's displacement vectors (3 floats per
// source entry, added to), `ve_orig` maps compacted entries to source entries, and the launch returns at once when *gate != 0.
template <bool PER_ENTRY>
__global__ void __launch_bounds__(kBwThreads, 1) attn_bwd_tc_kernel(const unsigned char* __restrict__ img_g, const float* __restrict__ sph1_k,
                                                                    const float* __restrict__ sph1_b, int n_recv,
                                                                    const int* n_listed, const int* ve_i,
                                                                    const int* ve_j, const float4* ve_d,
                                                                    const float* qkv, const float* ev_in,
                                                                    const float* g_xa, const float* gev1,
                                                                    float* __restrict__ g_qkv, float* __restrict__ gev_in,
                                                                    float* F, float* __restrict__ virial,
                                                                    int* __restrict__ err, long long* __restrict__ dbg,
                                                                    const int2* ve_orig, const int* gate, int* queue,
                                                                    int n_own) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  float* rec = reinterpret_cast<float*>(smem + kOffBwRec);
  float* sph = reinterpret_cast<float*>(smem + kOffBwSph);
  float* wt = reinterpret_cast<float*>(smem + kOffBwW);
  unsigned long long* mbar_p = reinterpret_cast<unsigned long long*>(smem + kOffBwMisc);
  uint32_t* tmem_p = reinterpret_cast<uint32_t*>(smem + kOffBwMisc + 48);
  int* handed_out = reinterpret_cast<int*>(smem + kOffBwMisc + 56);
  volatile int* failed = reinterpret_cast<volatile int*>(smem + kOffBwMisc + 52);
  for (int k = tid; k < kTcImageBytes / 16; k += kBwThreads) reinterpret_cast<uint4*>(smem + kOffImg)[k] = reinterpret_cast<const uint4*>(img_g)[k];
  for (int k = tid; k < 512; k += kBwThreads) {      // [filter][hidden unit][w0 w1 w2 w3 b - - -]
    const int q = k & 7, c = (k >> 3) & 31, f = k >> 8;
    sph[sph_at(f, c) + q] = q < 4 ? sph1_k[f * 128 + q * 32 + c] : (q == 4 ? sph1_b[f * 32 + c] : 0.f);
  }
  const uint32_t mbar = smem_u32(mbar_p);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(mbar));
    for (int k = 1; k < 5; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(mbar + 8 * k));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *failed = 0;
  }
  grid_dep_sync();
  if (PER_ENTRY && gate && *gate != 0) return;
  const long long n_edges = *n_listed;
  if (n_edges <= 0) return;
  const int rpw = entries_per_warp(n_edges, gridDim.x), tr = 16 * rpw;      // entries per warp / per tile
  TileWalk walk((int)((n_edges + tr - 1) / tr), (int)gridDim.x, (int)blockIdx.x);
  if (walk.tile >= walk.end) return;
  const int pad_i = ve_i[n_edges - 1];
  int* st_ij = reinterpret_cast<int*>(smem + kOffBwStIJ);
  float4* st_d = reinterpret_cast<float4*>(smem + kOffBwStD);
  const int half = warp >> 3;                   // the rows of this warp's pairs: [64 half, 64 half + 8 rpw)
  const int row0 = 64 * half + rpw * (warp & 7);
  // list entry of a tile row within the tile, -1 for a padding row
  auto entry_of = [&](int row) { return (row & 63) < 8 * rpw ? (row & 63) + (row >> 6) * 8 * rpw : -1; };
  // (i, j) and displacement of one tile's pairs into the staging buffers (threads 384..511): in flight beneath the tile before
  auto stage_tile = [&](int t) {
    if (tid < 384 || t >= walk.end) return;
    const int row = tid - 384, k = entry_of(row);
    const long long e = (long long)t * tr + k;
    if (k >= 0 && e < n_edges) {
      cp_async4(st_ij + 2 * row, ve_i + e); cp_async4(st_ij + 2 * row + 1, ve_j + e);
      cp_async16(st_d + row, ve_d + e);
    } else {
      st_ij[2 * row] = pad_i; st_ij[2 * row + 1] = pad_i;
      st_d[row] = make_float4(1.f, 0.f, 0.f, 1.f);
    }
  };
  stage_tile(walk.tile);
  if (tid == 0) handed_out[0] = walk.second((int)gridDim.x);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_p)), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  cp_async_wait_all();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_p, 0);
  const uint32_t a_hi = smem_u32(smem + kOffA), img = smem_u32(smem + kOffImg);
  unsigned char* a_ptr = smem + kOffA;
  const int deg = degree_of(lane < kMTot ? lane : 0);
  const int quad = warp & 3;                    // TMEM lane quadrant of this warp
  const int n_scat = n_recv;                    // partners below it own a row: they receive their share of a pair here
  uint32_t parity = 0;
  const uint32_t on = elect_one();
#ifdef SO3LR_TC_TIMING
  long long bph[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  long long bc0 = clock64();
  if (dbg && tid == 32 && blockIdx.x == 0) dbg[24] = 0;
#define BW_MARK(k) do { if (dbg && (tid & 31) == 0) { const long long c = clock64(); bph[k] += c - bc0; bc0 = c; } } while (0)
#else
#define BW_MARK(k) do { } while (0)
#endif
  for (; walk.tile < walk.end; walk.tile = walk.next) {
    const long long entry0 = (long long)walk.tile * tr;
    int run = 0;
    float dev8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // ---- per-edge preparation ----
    {
      const int hrow = 8 * warp + (lane >> 2), q = lane & 3;
      PairInvariants I;      // requested first, used last
      I.begin(ev_in + (size_t)st_ij[2 * hrow] * kMTot, ev_in + (size_t)st_ij[2 * hrow + 1] * kMTot, q);
      const int row = tid & 127, role = tid >> 7;
      const int k = entry_of(row);
      const bool valid = k >= 0 && entry0 + k < n_edges;
      const float4 d = st_d[row];
      const float r = d.w;
      if (role < 2) {
        // once these 256 threads are through, the Chebyshev steps of both filters' MMA chains start beneath the rest
        store_chebyshev_half(a_ptr, row, r, valid, role);
        fence_async_smem();
        if (warp < 4) {
          asm volatile("bar.sync 1, 256;" ::: "memory");
          tc_fence_after();
          issue_filter_mma(on, tmem, a_hi, img, warp >> 1, warp & 1, 0);
        } else {
          asm volatile("bar.arrive 1, 256;" ::: "memory");
        }
      } else {
        const int i = st_ij[2 * row], j = st_ij[2 * row + 1];
        const float ir = 1.f / r;
        const float ux = d.x * ir, uy = d.y * ir, uz = d.z * ir;
        float* rp = rec + row * kBwRec;
        if (role == 2) {
          float cut, dcut;
          phys_cutoff(r, cut, dcut);
          st4(rp, make_float4(__int_as_float(j), __int_as_float(i), valid ? cut * kInvNbar : 0.f, valid ? dcut * kInvNbar : 0.f));
          st4(rp + 8, make_float4(ux, uy, uz, ir));
          st4(rp + 12, make_float4(0.f, r, valid ? 1.f : 0.f, 0.f));
        }
        angular_end(gev1 + (size_t)(role == 2 ? i : j) * kMTot, ux, uy, uz, role == 2 ? 1.f : -1.f, rp + 8 + 4 * role, rp + 16 + 8 * role);
      }
      float s[4];
      I.finish(s);
      if (q == 0) st4(rec + hrow * kBwRec + 4, make_float4(s[0], s[1], s[2], s[3]));
      store_spherical_hidden_quarter(a_ptr, hrow, s, sph, q);
    }
    BW_MARK(0);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    BW_MARK(1);
    walk.look_ahead(handed_out, parity);
    stage_tile(walk.next);
    if (tid == 256 && walk.queued) run = TileWalk::handed((int)gridDim.x, atomicAdd(queue, 1));
    if (warp < 4) {
      tc_fence_after();
      issue_filter_mma(on, tmem, a_hi, img, warp >> 1, warp & 1, 1);
      umma_commit_if(on, mbar);
    }
    // while the tensor cores run: the value path's logit cotangents (8 rows per warp), then the sender rows of the first edge run
    edge_loops(rpw, [&](auto full) { value_logit_cotangents<full>(rec, row0, rpw, lane, qkv, g_xa); });
    RevLoads L;
    Receiver S;
    S.start<0>(__float_as_int(rec[row0 * kBwRec + 1]), lane, qkv);
    reverse_prefetch<0>(L, rec, row0, lane, qkv);
    wait_mma(mbar, parity, failed, err);
    BW_MARK(2);
    // this thread's shares of its row's cotangents of the invariants and of the radial derivative, both filters
    float ds0 = 0.f, ds1 = 0.f, ds2 = 0.f, ds3 = 0.f, drad = 0.f;
    // accumulators of filter f, rows of this group -> filter tile: the four warps of the group that can read them, 64 columns each
    auto copy_half = [&](int f) {
      if ((quad >> 1) != half) return;
      const int col = 64 * ((warp >> 2) & 1);
      float* p = wt + (32 * (quad & 1) + lane) * kWStride + col;
#pragma unroll
      for (int c = 0; c < 64; c += 16) {
        float v[16];
        tmem_ld16_combined(tmem + ((uint32_t)(32 * quad) << 16) + 128 * f + col + c, v);
#pragma unroll
        for (int k = 0; k < 16; k += 4) st4(p + c + k, make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]));
      }
    };
    auto sync_group = [&] { asm volatile("bar.sync %0, 256;" ::"r"(4 + half) : "memory"); };
    // dw of filter f stands in this group's rows: their chain of second MMAs, main and cross products by one warp each
    auto second_chain = [&](int f) {
      fence_async_smem();
      tc_fence_before();
      sync_group();
      const int first = half ? 8 : 2;      // warps that do not copy accumulators
      if (warp == first || warp == first + 1) {
        tc_fence_after();
        issue_reverse_mma(on, tmem, a_hi, img, f, half, warp - first);
        umma_commit_if(on, mbar + 8 * (1 + 2 * f + half));
      }
    };
    // per pair, once the second MMA chain of filter f is through: radial derivative and spherical hidden layer (all four threads of a row)
    auto finish_filter = [&](int f) {
      const int row = tid & 127, role = tid >> 7;
      const float* rp = rec + row * kBwRec;
      const uint32_t lane_base = tmem + ((uint32_t)(32 * quad) << 16) + 128 * f;
      {
        // thread (odd, upper) takes the terms m = 2c + odd of c in [16 upper, 16 upper + 16): columns 32 odd + c.  T_m' = m U_{m-1}, and
        // U_{n+2} = 2 T_2 U_n - U_{n-2} from (U_{-2}, U_0) or (U_{-3}, U_{-1}), in the upper half from (U_30, U_32) or (U_29, U_31),
        // which follow from t by doubling: T_2n = 2 T_n^2 - 1, U_{2n-1} = 2 T_n U_{n-1}, U_n = t U_{n-1} + T_n, U_{n-2} = t U_{n-1} - T_n
        const int odd = role & 1, upper = role >> 1;
        const float r = rp[13];
        const float x = expf(-kChebHalfGamma * r);
        const float t = fmaf(kChebA, x, kChebB), t2 = 2.f * t;
        const float dtdr = -kChebA * kChebHalfGamma * x;
        const float T2 = fmaf(t2, t, -1.f), T2x2 = 2.f * T2;
        float v[16];
        tmem_ld16_combined(lane_base + 32 * odd + 16 * upper, v);
        float up = odd ? -1.f : -t2, uc = odd ? 1.f : 0.f;
        if (upper) {
          const float T4 = fmaf(T2x2, T2, -1.f), T8 = fmaf(2.f * T4, T4, -1.f), T16 = fmaf(2.f * T8, T8, -1.f), T32 = fmaf(2.f * T16, T16, -1.f);
          const float U31 = 16.f * (((T16 * T8) * (T4 * T2)) * t2);
          const float U30 = fmaf(t, U31, -T32), U32 = fmaf(t, U31, T32);
          up = odd ? U30 : fmaf(t2, U30, -U31);
          uc = odd ? U32 : U31;
        }
        float acc = 0.f;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          const int m = 2 * c + odd + 32 * upper;
          acc = fmaf(v[c] * (float)m, uc, acc);
          const float un = fmaf(T2x2, uc, -up);
          up = uc; uc = un;
        }
        drad = fmaf(acc, dtdr, drad);
      }
      // spherical hidden layer, reverse: the four threads of a row take eight hidden units each
      {
        float v[8];
        tmem_ld8_combined(lane_base + 64 + 8 * role, v);
        const float4 s4 = ld4(rp + 4);
#pragma unroll
        for (int c8 = 0; c8 < 8; ++c8) {
          const int c = 8 * role + c8;
          const float* p = sph + sph_at(f, c);
          const float4 k = ld4(p);
          const float z = fmaf(s4.x, k.x, fmaf(s4.y, k.y, fmaf(s4.z, k.z, fmaf(s4.w, k.w, p[4]))));
          const float sg = __fdividef(1.f, 1.f + __expf(-z));
          const float dz = v[c8] * sg * (1.f + z * (1.f - sg));
          ds0 = fmaf(dz, k.x, ds0); ds1 = fmaf(dz, k.y, ds1); ds2 = fmaf(dz, k.z, ds2); ds3 = fmaf(dz, k.w, ds3);
        }
      }
    };
    // The filter tile goes from the first group to the second and back, twice (named barriers 2: to the second group, 3: to the first).
    // ---- filter 0 ----
    if (half) asm volatile("bar.sync 2, 512;" ::: "memory");
    copy_half(0);
    tc_fence_before();
    sync_group();
    BW_MARK(3);
    reverse_edges<0>(L, rec, wt, row0 - 64 * half, row0, rpw, a_ptr, lane, qkv, g_qkv, n_scat, S);
    BW_MARK(4);
    if (half) asm volatile("bar.arrive 3, 512;" ::: "memory");
    else asm volatile("bar.arrive 2, 512;" ::: "memory");
    second_chain(0);
    edge_loops(rpw, [&](auto full) { value_cotangent<full>(rec, row0, rpw, lane, g_xa, g_qkv, n_scat); });
    S.start<1>(__float_as_int(rec[row0 * kBwRec + 1]), lane, qkv);
    reverse_prefetch<1>(L, rec, row0, lane, qkv);
    wait_mma(mbar + 8 * (1 + half), parity, failed, err);      // the next loop overwrites the operand that this chain reads
    BW_MARK(5);
    // ---- filter 1 ----
    if (half) asm volatile("bar.sync 2, 512;" ::: "memory");
    else asm volatile("bar.sync 3, 512;" ::: "memory");
    copy_half(1);
    tc_fence_before();
    sync_group();
    BW_MARK(3);
    reverse_edges<1>(L, rec, wt, row0 - 64 * half, row0, rpw, a_ptr, lane, qkv, g_qkv, n_scat, S);
    BW_MARK(4);
    if (!half) asm volatile("bar.arrive 2, 512;" ::: "memory");
    second_chain(1);
    if (lane < kMTot) {      // ev differences of this warp's rows of the final flush: requested now, used after the last MMA
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float* rp = rec + ((row0 + k) & (TE - 1)) * kBwRec;
        const int j = __float_as_int(rp[0]), i = __float_as_int(rp[1]);
        dev8[k] = ev_in[(size_t)j * kMTot + lane] - ev_in[(size_t)i * kMTot + lane];
      }
    }
    wait_mma(mbar + 8, parity, failed, err);
    wait_mma(mbar + 16, parity, failed, err);
    finish_filter(0);
    wait_mma(mbar + 24, parity, failed, err);
    wait_mma(mbar + 32, parity, failed, err);
    parity ^= 1;
    BW_MARK(5);
    finish_filter(1);
    {
      // the filter tile is free (both groups' last chains follow their loops): it takes the four threads' shares
      const int row = tid & 127, role = tid >> 7;
      st4(wt + (role * TE + row) * 4, make_float4(ds0, ds1, ds2, ds3));
      wt[(4 * 4 + role) * TE + row] = drad;
    }
    tc_fence_before();
    __syncthreads();
    BW_MARK(6);
    // ---- force on the receiver (threads 0..127); cotangent of ev (8 rows per warp) ----
    if (tid < 128) {
      const float* rp = rec + tid * kBwRec;
      const bool listed = rp[14] != 0.f;
      const int i = listed ? __float_as_int(rp[1]) : -1;
      const float4 uu = ld4(rp + 8);
      float e1[3], e2[3], t1 = 0.f, t2 = 0.f;
      tangent_frame(uu.x, uu.y, uu.z, e1, e2);
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const float a = rp[16 + l], b = rp[20 + l];
        t1 = fmaf(a, rp[32 + 2 * l], fmaf(b, rp[40 + 2 * l], t1));
        t2 = fmaf(a, rp[33 + 2 * l], fmaf(b, rp[41 + 2 * l], t2));
      }
      t1 *= uu.w; t2 *= uu.w;
      const float4 ang = make_float4(fmaf(t1, e1[0], t2 * e2[0]), fmaf(t1, e1[1], t2 * e2[1]), fmaf(t1, e1[2], t2 * e2[2]), 0.f);
      const float* dr = wt + 4 * 4 * TE + tid;
      const float g_r = rp[12] + ((dr[0] + dr[TE]) + (dr[2 * TE] + dr[3 * TE]));
      float fsx = listed ? fmaf(g_r, uu.x, ang.x) : 0.f, fsy = listed ? fmaf(g_r, uu.y, ang.y) : 0.f, fsz = listed ? fmaf(g_r, uu.z, ang.z) : 0.f;
      if (virial && listed) {
        // both ends' halves on the receiver's row, unless the partner's is not summed here (rows below n_own are)
        const float hr = (__float_as_int(rp[0]) < n_own ? 1.f : 0.5f) * rp[13];
        const float wx = hr * uu.x, wy = hr * uu.y, wz = hr * uu.z;
        float* w = virial + 6 * (size_t)i;
        atomicAdd(w, wx * fsx); atomicAdd(w + 1, wy * fsy); atomicAdd(w + 2, wz * fsz);
        atomicAdd(w + 3, 0.5f * (wy * fsz + wz * fsy)); atomicAdd(w + 4, 0.5f * (wx * fsz + wz * fsx));
        atomicAdd(w + 5, 0.5f * (wx * fsy + wy * fsx));
      }
      if (PER_ENTRY) {
        // half of the pair's force on the receiver goes to this entry of the source list, the other half with the opposite sign to the
        // reversed entry
        if (listed) {
          const int2 eo = ve_orig[entry0 + entry_of(tid)];
          float *g = F + 3 * (size_t)eo.x, *h = F + 3 * (size_t)eo.y;
          g[0] += 0.5f * fsx; g[1] += 0.5f * fsy; g[2] += 0.5f * fsz;
          h[0] -= 0.5f * fsx; h[1] -= 0.5f * fsy; h[2] -= 0.5f * fsz;
        }
      } else {
      // the rows of a tile are sorted by receiver: sum each run of equal receivers inside the warp (segmented scan) and let its
      // last lane add the total, instead of up to 32 additions to one address; the partners differ and get theirs one by one
      const int jp = __float_as_int(rp[0]);
      if (listed && jp < n_scat) {
        atomicAdd(F + 3 * (size_t)jp, -fsx); atomicAdd(F + 3 * (size_t)jp + 1, -fsy); atomicAdd(F + 3 * (size_t)jp + 2, -fsz);
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float tx = __shfl_up_sync(0xffffffffu, fsx, o), ty = __shfl_up_sync(0xffffffffu, fsy, o), tz = __shfl_up_sync(0xffffffffu, fsz, o);
        const int ti = __shfl_up_sync(0xffffffffu, i, o);
        if (lane >= o && ti == i) { fsx += tx; fsy += ty; fsz += tz; }
      }
      const int inext = __shfl_down_sync(0xffffffffu, i, 1);
      if (listed && (lane == 31 || inext != i)) {
        atomicAdd(F + 3 * (size_t)i, fsx); atomicAdd(F + 3 * (size_t)i + 1, fsy); atomicAdd(F + 3 * (size_t)i + 2, fsz);
      }
      }
    }
    edge_loops(rpw, [&](auto full) {
      const float sc = -2.f * invw(deg);
      auto share = [&](int k) {      // derivative with respect to the receiver's component; the partner's is its negative
        const float* dp = wt + 4 * (row0 + k) + deg;
        return sc * ((dp[0] + dp[TE * 4]) + (dp[2 * TE * 4] + dp[3 * TE * 4])) * dev8[k];
      };
      int cur_i = __float_as_int(rec[row0 * kBwRec + 1]);
      float acc = 0.f;
      if (full && cur_i == __float_as_int(rec[(row0 + 7) * kBwRec + 1])) {      // eight pairs of one receiver
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float t = share(k);
          const int j = __float_as_int(rec[(row0 + k) * kBwRec]);
          acc += t;
          if (lane < kMTot && j < n_scat) atomicAdd(gev_in + (size_t)j * kMTot + lane, -t);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (!full && k >= rpw) break;
          const float* rp = rec + (row0 + k) * kBwRec;
          const int i = __float_as_int(rp[1]);
          if (i != cur_i) {
            if (lane < kMTot && acc != 0.f) atomicAdd(gev_in + (size_t)cur_i * kMTot + lane, acc);
            cur_i = i; acc = 0.f;
          }
          const float t = share(k);
          const int j = __float_as_int(rp[0]);
          acc += t;
          if (lane < kMTot && j < n_scat && rp[14] != 0.f) atomicAdd(gev_in + (size_t)j * kMTot + lane, -t);
        }
      }
      if (lane < kMTot && acc != 0.f) atomicAdd(gev_in + (size_t)cur_i * kMTot + lane, acc);
    });
    cp_async_wait_all();
    if (tid == 256 && walk.queued) handed_out[parity] = run;
    __syncthreads();
    BW_MARK(7);
    TC_TILE(24);
  }
#ifdef SO3LR_TC_TIMING
  if (dbg && tid == 32 && blockIdx.x == 0) { for (int q = 0; q < 8; ++q) dbg[16 + q] = bph[q]; }
  if (dbg && (tid & 31) == 0 && blockIdx.x == 0) { for (int q = 0; q < 8; ++q) dbg[32 + 8 * warp + q] = bph[q]; }
#endif
  if (tid == 256) walk.finish(queue);
  cp_async_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

}  // namespace

// ------------------------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------------------------
int configure_attention_tc_kernels() {
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(attn_fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemFwd));
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(attn_bwd_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBwd));
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(attn_bwd_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBwd));
  return kOk;
}

int valid_edges_reserve(ValidEdges* V, int n_rows, long long capacity) {
  if (!V->total) SO3LR_CUDA_CHECK(dev_alloc(&V->total, 3));      // and the tile queue
  const int n_blocks = (n_rows + kCompactRows - 1) / kCompactRows;
  if (n_blocks > V->block_cap) {
    dev_free(V->blocks);
    V->blocks = nullptr; V->block_cap = 0;
    SO3LR_CUDA_CHECK(dev_alloc(&V->blocks, (size_t)n_blocks));
    V->block_cap = n_blocks;
  }
  if (capacity > V->capacity) {
    if (V->i) dev_free(V->i);
    if (V->j) dev_free(V->j);
    if (V->d) dev_free(V->d);
    V->i = V->j = nullptr; V->d = nullptr; V->capacity = 0;
    if (capacity < 1) capacity = 1;
    SO3LR_CUDA_CHECK(dev_alloc(&V->i, (size_t)capacity));
    SO3LR_CUDA_CHECK(dev_alloc(&V->j, (size_t)capacity));
    SO3LR_CUDA_CHECK(dev_alloc(&V->d, (size_t)capacity));
    V->capacity = capacity;
  }
  return kOk;
}

void valid_edges_free(ValidEdges* V) {
  dev_free(V->total); dev_free(V->blocks); dev_free(V->i); dev_free(V->j); dev_free(V->d); dev_free(V->orig); dev_free(V->partner);
  *V = ValidEdges{};
}

int valid_edges_build(ValidEdges* V, cudaStream_t s, int n_rows, int n, const int* row_ptr, const int* nbr_j, const float* dR, int* asym,
                      long long n_source, bool total_cleared) {
  V->asym = nullptr;
  V->n_rows = n_rows;
  if (n_rows <= 0) return kOk;
  if (!V->total) return kInvalidArgument;
  if (!total_cleared) SO3LR_CUDA_CHECK(cudaMemsetAsync(V->total, 0, sizeof(int), s));
  const int blocks = (n_rows + 7) / 8;
  if (asym) {
    if (n_source > V->capacity) return kInvalidArgument;
    if (V->orig_cap < V->capacity) {
      dev_free(V->orig); dev_free(V->partner);
      V->orig = nullptr; V->partner = nullptr; V->orig_cap = 0;
      SO3LR_CUDA_CHECK(dev_alloc(&V->orig, (size_t)V->capacity));
      SO3LR_CUDA_CHECK(dev_alloc(&V->partner, (size_t)V->capacity));
      V->orig_cap = V->capacity;
    }
    V->asym = asym;
    { match_pairs_kernel<<<blocks, 256, 0, s>>>(n_rows, row_ptr, nbr_j, dR, V->partner, asym); count_launch(); }
    { check_mutual_kernel<<<sm_count() * 8, 256, 0, s>>>(n_rows, row_ptr, V->partner, asym); count_launch(); }
  }
  const int* partner = asym ? V->partner : nullptr;
  int2* orig = asym ? V->orig : nullptr;
  const int n_blocks = (n_rows + kCompactRows - 1) / kCompactRows, threads = 32 * kCompactRows;
  if (n_blocks > V->block_cap) return kInvalidArgument;
  if (n_rows < kOrderedRows) {
    { launch_chained(compact_rows_kernel<kReserve>, n_blocks, threads, 0, s, n_rows, n, row_ptr, nbr_j, dR, partner, asym, V->total, nullptr, V->i, V->j, V->d, orig); count_launch(); }
  } else {
    { launch_chained(compact_rows_kernel<kCount>, n_blocks, threads, 0, s, n_rows, n, row_ptr, nbr_j, dR, partner, asym, nullptr, V->blocks, nullptr, nullptr, nullptr, nullptr); count_launch(); }
    { launch_chained(scan_blocks_kernel, 1, 1024, 0, s, n_blocks, V->blocks, V->total); count_launch(); }
    { launch_chained(compact_rows_kernel<kFill>, n_blocks, threads, 0, s, n_rows, n, row_ptr, nbr_j, dR, partner, asym, nullptr, V->blocks, V->i, V->j, V->d, orig); count_launch(); }
  }
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

int valid_edges_count_directed(const ValidEdges& V, long long* n_host) {
  *n_host = 0;
  if (!V.total || V.n_rows <= 0) return kOk;
  SO3LR_CUDA_CHECK(cudaDeviceSynchronize());
  unsigned long long* t = nullptr;
  SO3LR_CUDA_CHECK(dev_alloc(&t, 1));
  unsigned long long h = 0;
  cudaError_t e = cudaMemset(t, 0, sizeof(h));
  if (e == cudaSuccess) {
    { count_directed_kernel<<<sm_count(), 256>>>(V.n_rows, V.total, V.j, V.asym, t); count_launch(); }
    e = cudaMemcpy(&h, t, sizeof(h), cudaMemcpyDeviceToHost);
  }
  dev_free(t);
  SO3LR_CUDA_CHECK(e);
  *n_host = (long long)h;
  return kOk;
}

// The walks of all CTAs over n tiles whose times are all alike, CTAs coming free in the order of their numbers
long long tile_walk_longest(int n, int grid) {
  struct Cta { TileWalk walk; int handed_out[2]; int tiles; };
  std::vector<Cta> ctas;
  for (int b = 0; b < grid; ++b) {
    Cta c{TileWalk(n, grid, b), {0, 0}, 0};
    c.handed_out[0] = c.walk.second(grid);
    ctas.push_back(c);
  }
  std::vector<char> seen(n > 0 ? n : 0, 0);
  long long walked = 0;
  int tickets = 0, longest = 0;
  for (bool any = true; any;) {
    any = false;
    for (Cta& c : ctas) {
      if (c.walk.tile >= c.walk.end) continue;
      any = true;
      if (c.walk.tile < 0 || c.walk.tile >= n || seen[c.walk.tile]++) return -1;
      const uint32_t turn = c.tiles & 1;
      c.walk.look_ahead(c.handed_out, turn);
      if (c.walk.queued) c.handed_out[turn ^ 1] = TileWalk::handed(grid, tickets++);
      c.walk.tile = c.walk.next;
      if (++c.tiles > longest) longest = c.tiles;
      ++walked;
    }
  }
  return walked == n ? longest : -1;
}

// development aid of builds with -DSO3LR_TC_TIMING: SO3LR_B200_TC_DEBUG=1 makes the first CTA of both kernels record the cycles of each phase and
// the number of its tiles
static long long* tc_debug_buffer() {
  static long long* buf = [] {
    long long* p = nullptr;
    if (std::getenv("SO3LR_B200_TC_DEBUG")) {
      cudaMalloc((void**)&p, 288 * sizeof(long long)); cudaMemset(p, 0, 288 * sizeof(long long));
    }
    return p;
  }();
  return buf;
}
void tc_debug_print() {
  long long* d = tc_debug_buffer();
  if (!d) return;
  long long h[288];
  cudaDeviceSynchronize();
  cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  if (h[24]) std::fprintf(stderr, "tc bwd phases (cycles per tile, %lld tiles): prep %lld | sync %lld | mma1 %lld | sync+tmem->tile %lld | edge loop %lld | sync+mma2 %lld | epilogue %lld | phase C %lld\n",
               h[24], h[16] / h[24], h[17] / h[24], h[18] / h[24], h[19] / h[24], h[20] / h[24], h[21] / h[24], h[22] / h[24], h[23] / h[24]);
  if (h[24])
    for (int w = 0; w < 16; ++w) {
      std::fprintf(stderr, "  bwd warp %2d:", w);
      for (int q = 0; q < 8; ++q) std::fprintf(stderr, " %6lld", h[32 + 8 * w + q] / h[24]);
      std::fprintf(stderr, "\n");
    }
  if (h[8])
    for (int w = 0; w < 16; ++w) {
      std::fprintf(stderr, "  fwd warp %2d:", w);
      for (int q = 0; q < 8; ++q) std::fprintf(stderr, " %6lld", h[160 + 8 * w + q] / h[8]);
      std::fprintf(stderr, "\n");
    }
  if (h[8]) std::fprintf(stderr, "tc fwd phases (cycles per tile, %lld tiles): prep %lld | sync %lld | mma+wait %lld | tmem0 %lld | loop0 %lld | sync %lld | tmem1 %lld | loop1 %lld\n",
               h[8], h[0] / h[8], h[1] / h[8], h[2] / h[8], h[3] / h[8], h[4] / h[8], h[5] / h[8], h[6] / h[8], h[7] / h[8]);
}
int launch_attn_fwd_tc(cudaStream_t s, const LayerDev& L, const ValidEdges& V, int n_recv, const float* qkv, const float* x_in,
                       const float* ev_in, float* xa, float* ev1, int* err, bool preset) {
  if (n_recv <= 0) return kOk;
  if (n_recv != V.n_rows) return kInvalidArgument;
  // the kernel adds the attention sums onto the skip connection
  if (!preset) {
    SO3LR_CUDA_CHECK(cudaMemcpyAsync(xa, x_in, (size_t)n_recv * kF * sizeof(float), cudaMemcpyDeviceToDevice, s));
    SO3LR_CUDA_CHECK(cudaMemcpyAsync(ev1, ev_in, (size_t)n_recv * kMTot * sizeof(float), cudaMemcpyDeviceToDevice, s));
  }
  { launch_chained(attn_fwd_tc_kernel, sm_count(), kFwThreads, kSmemFwd, s, L.tc_img_fwd, L.sph1_k, L.sph1_b, n_recv, V.total, V.i, V.j, V.d, qkv, ev_in, xa, ev1, err, tc_debug_buffer(), V.asym, V.total + 1); count_launch(); }
  return kOk;
}

int launch_attn_bwd_tc(cudaStream_t s, const LayerDev& L, const ValidEdges& V, int n_recv, const float* qkv, const float* ev_in,
                       const float* g_xa, const float* gev1, float* g_qkv, float* gev_in, float* F, float* virial, int n_own, int* err,
                       bool gev_preset, bool gq_preset) {
  if (n_recv <= 0) return kOk;
  if (n_recv != V.n_rows) return kInvalidArgument;
  // the kernel adds into the receivers' rows: cotangents of q/k/v start at zero, that of ev at the skip term
  if (!gq_preset) SO3LR_CUDA_CHECK(cudaMemsetAsync(g_qkv, 0, (size_t)n_recv * kProj * sizeof(float), s));
  if (!gev_preset) SO3LR_CUDA_CHECK(cudaMemcpyAsync(gev_in, gev1, (size_t)n_recv * kMTot * sizeof(float), cudaMemcpyDeviceToDevice, s));
  { launch_chained(attn_bwd_tc_kernel<false>, sm_count(), kBwThreads, kSmemBwd, s, L.tc_img, L.sph1_k, L.sph1_b, n_recv, V.total, V.i, V.j, V.d, qkv, ev_in, g_xa, gev1,
                                                              g_qkv, gev_in, F, virial, err, tc_debug_buffer(), nullptr, nullptr, V.total + 1, n_own); count_launch(); }
  return kOk;
}

int launch_attn_bwd_tc_graph(cudaStream_t s, const LayerDev& L, const ValidEdges& V, int n_recv, const float* qkv, const float* ev_in,
                             const float* g_xa, const float* gev1, float* g_qkv, float* gev_in, float* g_dR, int* err, const int* asym) {
  if (n_recv <= 0) return kOk;
  if (n_recv != V.n_rows || !V.orig) return kInvalidArgument;
  { launch_chained(attn_bwd_tc_kernel<true>, sm_count(), kBwThreads, kSmemBwd, s, L.tc_img, L.sph1_k, L.sph1_b, n_recv, V.total, V.i, V.j, V.d, qkv, ev_in, g_xa, gev1,
                                                             g_qkv, gev_in, g_dR, nullptr, err, nullptr, V.orig, asym, V.total + 1, 0); count_launch(); }
  return kOk;
}

}  // namespace so3lr
