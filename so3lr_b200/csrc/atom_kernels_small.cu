// Per-atom dense blocks and output heads for short atom lists.
//
// The tensor-core kernels (dense_tc.cu) work on 128 atoms per CTA: a molecule or a small box fills one tile or a dozen of them, and
// its time is the chain of dependent phases of one tile (operand stores, 24 MMAs, commit, accumulator loads, barriers: about 2.5 us
// per 128 x 128 contraction), whatever the number of atoms in it.  Here a CTA takes AT = 2 .. 16 atoms, so that the list spreads over all
// SMs, and a contraction is 128 x 128 / 4 FP32 multiply-adds per thread and atom: thread (p, c) forms the p-th quarter of the sum over
// the inputs for output column c, with its 32 kernel elements requested before the barrier that precedes their use (they do not
// depend on the data).  The quarters meet in shared memory, where one warp per atom (lane = 4 features) adds them up and evaluates
// everything between two contractions without further barriers: bias, silu, residual, LayerNorm by shuffles.
// Bound by the kernels' way from the L2 into each SM (272 KB per CTA and block) and, from AT = 8 on, by the FP32 pipe.  Measured
// (post-attention block reverse / forward, head block forward / reverse): 192 atoms 37.2 / 27.5, 17.5 / 17.0 us on dense_tc.cu, 7.1 / 7.1,
// 6.0 / 5.2 us here; 1,536 atoms 37.0 / 28.1, 17.6 / 17.1 against 15.0 / 14.5, 10.8 / 9.9 us.  A force evaluation of 2,340 atoms, next to
// the limit of 16 atoms per SM, takes 527 us with these kernels and 627 us with the others; the limit is the registers of AT = 16.
#include "kernels.h"

namespace so3lr {

namespace {

constexpr int NTHR = 640;      // 20 warps: 4 x 128 partial sums (the fifth group idles), 640 projection outputs, 5 x 128 reverse projections
constexpr int NP = 4;          // parts of a 128-long sum
constexpr int KP = kF / NP;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// the model's weights only (see grid_dep_sync)
__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 fma4(float s, float4 b, float4 c) {
  return make_float4(fmaf(s, b.x, c.x), fmaf(s, b.y, c.y), fmaf(s, b.z, c.z), fmaf(s, b.w, c.w));
}
__device__ __forceinline__ float sum4(float4 a) { return (a.x + a.y) + (a.z + a.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, a.y * b.y) + fmaf(a.z, b.z, a.w * b.w); }
__device__ __forceinline__ float4 silu4(float4 a) { return make_float4(silu_f(a.x), silu_f(a.y), silu_f(a.z), silu_f(a.w)); }
__device__ __forceinline__ float4 dsilu4(float4 a) { return make_float4(dsilu_f(a.x), dsilu_f(a.y), dsilu_f(a.z), dsilu_f(a.w)); }
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float inv_weight(int l) {
  return l == 0 ? 0.5773502691896258f : (l == 1 ? 0.4472135954999579f : (l == 2 ? 0.3779644730092272f : 0.3333333333333333f));
}

// K kernel elements of one output column, `ld` floats apart
template <int K>
__device__ __forceinline__ void load_w(float (&w)[32], const float* __restrict__ W, int ld) {
#pragma unroll
  for (int k = 0; k < K; ++k) w[k] = __ldg(W + (size_t)k * ld);
}
// acc[a] += sum_k w[k] x[a][k], x rows `ld` floats apart in shared memory (all lanes of a warp read the same address, or the 32
// inputs of their head); even and odd inputs are summed apart (packed arithmetic) and joined by the caller
template <int AT, int K>
__device__ __forceinline__ void dot_rows(float2 (&acc)[AT], const float (&w)[32], const float* x, int ld) {
#pragma unroll
  for (int k = 0; k < K; k += 4) {
    const float2 wa = make_float2(w[k], w[k + 1]), wb = make_float2(w[k + 2], w[k + 3]);
#pragma unroll
    for (int a = 0; a < AT; ++a) {
      const float4 v = ld4(x + a * ld + k);
      acc[a] = __ffma2_rn(wb, make_float2(v.z, v.w), __ffma2_rn(wa, make_float2(v.x, v.y), acc[a]));
    }
  }
}
template <int AT>
__device__ __forceinline__ void zero_acc(float2 (&acc)[AT]) {
#pragma unroll
  for (int a = 0; a < AT; ++a) acc[a] = make_float2(0.f, 0.f);
}
// partial sums of part p, column c of `width` -> red[p][a][c]
template <int AT>
__device__ __forceinline__ void put_partials(float* red, const float2 (&acc)[AT], int p, int c, int width) {
#pragma unroll
  for (int a = 0; a < AT; ++a) red[(p * AT + a) * width + c] = acc[a].x + acc[a].y;
}
// one 128 x 128 contraction of the rows in `act`: kernel elements already in w
template <int AT>
__device__ __forceinline__ void contract(float* red, const float (&w)[32], const float* act) {
  const int p = threadIdx.x >> 7, c = threadIdx.x & 127;
  if (p < NP) {
    float2 acc[AT];
    zero_acc<AT>(acc);
    dot_rows<AT, KP>(acc, w, act + KP * p, kF);
    put_partials<AT>(red, acc, p, c, kF);
  }
}
__device__ __forceinline__ void load_w128(float (&w)[32], const float* __restrict__ W) {
  const int p = threadIdx.x >> 7, c = threadIdx.x & 127;
  if (p < NP) load_w<KP>(w, W + (size_t)KP * p * kF + c, kF);
}
// columns 4 lane .. 4 lane + 3 of row a, summed over the parts
template <int AT, int PARTS>
__device__ __forceinline__ float4 get_sum(const float* red, int a, int lane) {
  float4 s = ld4(red + a * kF + 4 * lane);
#pragma unroll
  for (int p = 1; p < PARTS; ++p) s = add4(s, ld4(red + (p * AT + a) * kF + 4 * lane));
  return s;
}
// normalised row (no affine) and 1 / standard deviation
__device__ __forceinline__ float4 normalise(float4 x, float& rstd) {
  const float mean = wsum(sum4(x)) * (1.f / kF);
  x = make_float4(x.x - mean, x.y - mean, x.z - mean, x.w - mean);
  rstd = rsqrtf(wsum(dot4(x, x)) * (1.f / kF) + kLnEps);
  return make_float4(x.x * rstd, x.y * rstd, x.z * rstd, x.w * rstd);
}
// cotangent of a LayerNorm's input from gy = cotangent x scale
__device__ __forceinline__ float4 normalise_vjp(float4 gy, float4 xh, float rstd) {
  const float s1 = wsum(sum4(gy)) * (1.f / kF), s2 = wsum(dot4(gy, xh)) * (1.f / kF);
  return make_float4(rstd * (gy.x - s1 - xh.x * s2), rstd * (gy.y - s1 - xh.y * s2), rstd * (gy.z - s1 - xh.z * s2), rstd * (gy.w - s1 - xh.w * s2));
}
// sums over the components of each degree (lane m < 24 holds component m)
__device__ __forceinline__ float4 degree_sums(float v, int deg) {
  return make_float4(wsum(deg == 0 ? v : 0.f), wsum(deg == 1 ? v : 0.f), wsum(deg == 2 ? v : 0.f), wsum(deg == 3 ? v : 0.f));
}
__device__ __forceinline__ float pick(float4 v, int l) { return l == 0 ? v.x : (l == 1 ? v.y : (l == 2 ? v.z : v.w)); }

// The blocks' definitions, inputs and outputs are those of dense_tc.cu.
template <int AT>
__global__ void __launch_bounds__(NTHR, 1) post_fwd_small_kernel(LayerDev L, int n, const float* xa, const float* ev1,
                                                                 float* __restrict__ z1_out, float* __restrict__ x3_out, float* __restrict__ gate_out,
                                                                 float* __restrict__ x4_out, float* __restrict__ ev2_out,
                                                                 const float* __restrict__ projT, float* __restrict__ qkv_next,
                                                                 float* __restrict__ x4_copy, float* __restrict__ ev2_copy) {
  extern __shared__ __align__(16) float sm[];
  float* act = sm;                // [AT][128]
  float* red = sm + AT * kF;      // [4][AT][128]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col = 4 * lane;
  const int atom = blockIdx.x * AT + warp;
  const bool own = warp < AT && atom < n;
  const size_t ra = (size_t)atom * kF + col;
  const int deg = degree_of(lane < kMTot ? lane : 0);
  float w[32];
  load_w128(w, L.res1_k);
  grid_dep_sync();
  float4 xr = zero4(), inv = zero4();
  float e = 0.f;
  if (warp < AT) {
    const float4 x = own ? ld4(xa + ra) : zero4();
    if (own && lane < kMTot) e = ev1[(size_t)atom * kMTot + lane];
    float rstd;
    const float4 xh = normalise(x, rstd), sc = ldg4(L.ln1_s + col), bi = ldg4(L.ln1_b + col);
    xr = add4(mul4(xh, sc), bi);
    st4(act + warp * kF + col, silu4(xr));
    inv = degree_sums(e * e, deg);
    inv = make_float4(inv.x * inv_weight(0), inv.y * inv_weight(1), inv.z * inv_weight(2), inv.w * inv_weight(3));
  }
  __syncthreads();
  contract<AT>(red, w, act);
  load_w128(w, L.res2_k);
  __syncthreads();
  if (warp < AT) {
    const float4 z = add4(get_sum<AT, NP>(red, warp, lane), ldg4(L.res1_b + col));
    if (own) st4(z1_out + ra, z);
    st4(act + warp * kF + col, silu4(z));
  }
  __syncthreads();
  contract<AT>(red, w, act);
  load_w128(w, L.ex_xx);
  __syncthreads();
  if (warp < AT) {
    xr = add4(xr, add4(get_sum<AT, NP>(red, warp, lane), ldg4(L.res2_b + col)));
    st4(act + warp * kF + col, xr);
    const float4 w0 = ldg4(L.ex_xg + 4 * col), w1 = ldg4(L.ex_xg + 4 * col + 4), w2 = ldg4(L.ex_xg + 4 * col + 8), w3 = ldg4(L.ex_xg + 4 * col + 12);
    float4 g = fma4(xr.x, w0, fma4(xr.y, w1, fma4(xr.z, w2, fma4(xr.w, w3, zero4()))));
    g = make_float4(wsum(g.x), wsum(g.y), wsum(g.z), wsum(g.w));
    g = add4(g, make_float4(L.ex_bg[0], L.ex_bg[1], L.ex_bg[2], L.ex_bg[3]));
    g = fma4(inv.x, ldg4(L.ex_ig), fma4(inv.y, ldg4(L.ex_ig + 4), fma4(inv.z, ldg4(L.ex_ig + 8), fma4(inv.w, ldg4(L.ex_ig + 12), g))));
    if (own) {
      if (lane == 0) st4(gate_out + (size_t)atom * 4, g);
      if (lane < kMTot) {
        const float ev2 = e * (1.f + pick(g, deg));
        ev2_out[(size_t)atom * kMTot + lane] = ev2;
        if (ev2_copy) ev2_copy[(size_t)atom * kMTot + lane] = ev2;
      }
    }
  }
  __syncthreads();
  contract<AT>(red, w, act);
  if (projT) load_w<32>(w, projT + (size_t)(tid >> 5) * 1024 + (tid & 31), 32);
  __syncthreads();
  if (warp < AT) {
    float4 y = add4(get_sum<AT, NP>(red, warp, lane), ldg4(L.ex_bx + col));
    y = fma4(inv.x, ldg4(L.ex_ix + col), fma4(inv.y, ldg4(L.ex_ix + kF + col), fma4(inv.z, ldg4(L.ex_ix + 2 * kF + col), fma4(inv.w, ldg4(L.ex_ix + 3 * kF + col), y))));
    const float4 x3 = add4(xr, y);
    float rstd;
    const float4 xh = normalise(x3, rstd);
    const float4 x4 = add4(mul4(xh, ldg4(L.ln2_s + col)), ldg4(L.ln2_b + col));
    if (own) {
      st4(x3_out + ra, x3); st4(x4_out + ra, x4);
      if (x4_copy) st4(x4_copy + ra, x4);
    }
    st4(act + warp * kF + col, x4);
  }
  if (!projT) return;
  __syncthreads();
  {      // q/k/v rows of the next layer: thread = output column, 32 inputs of its head
    float2 acc[AT];
    zero_acc<AT>(acc);
    dot_rows<AT, 32>(acc, w, act + 32 * (warp & 3), kF);
    const int rows = n - (int)blockIdx.x * AT;
#pragma unroll
    for (int a = 0; a < AT; ++a)
      if (a < rows) qkv_next[(size_t)(blockIdx.x * AT + a) * kProj + tid] = acc[a].x + acc[a].y;
  }
}

template <int AT>
__global__ void __launch_bounds__(NTHR, 1) post_bwd_small_kernel(LayerDev L, int n, const float* xa, const float* ev1,
                                                                 const float* z1, const float* x3,
                                                                 const float* gate, const float* g4,
                                                                 const float* gev2, float* g_xa, float* __restrict__ gev1,
                                                                 const float* __restrict__ proj, float* g_qkv_up,
                                                                 float* __restrict__ gev1_copy) {
  extern __shared__ __align__(16) float sm[];
  float* act = sm;                        // [AT][128]
  float* red = act + AT * kF;             // [5][AT][128]
  float* gq = red + 5 * AT * kF;          // [AT][640] (with `proj` only)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col = 4 * lane;
  const int row0 = blockIdx.x * AT, atom = row0 + warp;
  const bool own = warp < AT && atom < n;
  const size_t ra = (size_t)atom * kF + col;
  const int deg = degree_of(lane < kMTot ? lane : 0);
  float w[32];
  float4 g3 = zero4(), gg = zero4(), vx3 = zero4(), vz = zero4(), vxa = zero4();
  float e = 0.f, ge2 = 0.f, gt = 0.f;
  if (proj) load_w<32>(w, proj + (size_t)((tid >> 7) * 4 + ((tid >> 5) & 3)) * 1024 + lane, 32);      // thread (projection, column): 32 outputs of its head
  else load_w128(w, L.ex_xxT);
  grid_dep_sync();
  // this thread's shares of the CTA's g_qkv rows (16-byte pieces, NTHR apart): all requested at once, and cleared for the next attention
  // layer behind the barrier.  A load and the clearing store of its piece in turn serialise: 8 us a launch at 1,536 atoms
  constexpr int kPieces = (AT * (kProj / 4) + NTHR - 1) / NTHR;
  auto piece = [&](int u) { return tid + u * NTHR; };
  auto listed = [&](int u) { return piece(u) < AT * (kProj / 4) && row0 + piece(u) / (kProj / 4) < n; };
  if (proj) {
    float4 v[kPieces];
#pragma unroll
    for (int u = 0; u < kPieces; ++u) v[u] = listed(u) ? ld4(g_qkv_up + (size_t)row0 * kProj + 4 * piece(u)) : zero4();
#pragma unroll
    for (int u = 0; u < kPieces; ++u)
      if (piece(u) < AT * (kProj / 4)) st4(gq + 4 * piece(u), v[u]);
  }
  if (own) {
    g3 = ld4((proj ? g_xa : g4) + ra);
    vx3 = ld4(x3 + ra); vz = ld4(z1 + ra); vxa = ld4(xa + ra);
    if (lane < kMTot) {
      e = ev1[(size_t)atom * kMTot + lane];
      ge2 = gev2[(size_t)atom * kMTot + lane];
      gt = gate[(size_t)atom * 4 + deg];
    }
  }
  if (proj) {
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kPieces; ++u)
      if (listed(u)) st4(g_qkv_up + (size_t)row0 * kProj + 4 * piece(u), zero4());
    float2 acc[AT];
    zero_acc<AT>(acc);
    dot_rows<AT, 32>(acc, w, gq + 32 * warp, kProj);
    put_partials<AT>(red, acc, tid >> 7, tid & 127, kF);
    load_w128(w, L.ex_xxT);
    __syncthreads();
  }
  if (warp < AT) {
    if (proj) g3 = add4(g3, get_sum<AT, 5>(red, warp, lane));
    float rstd;
    const float4 xh = normalise(vx3, rstd);
    g3 = normalise_vjp(mul4(g3, ldg4(L.ln2_s + col)), xh, rstd);
    st4(act + warp * kF + col, g3);
    gg = degree_sums(ge2 * e, deg);
    float4 gi = make_float4(wsum(dot4(g3, ldg4(L.ex_ix + col))), wsum(dot4(g3, ldg4(L.ex_ix + kF + col))),
                            wsum(dot4(g3, ldg4(L.ex_ix + 2 * kF + col))), wsum(dot4(g3, ldg4(L.ex_ix + 3 * kF + col))));
    gi = add4(gi, make_float4(dot4(gg, ldg4(L.ex_ig)), dot4(gg, ldg4(L.ex_ig + 4)), dot4(gg, ldg4(L.ex_ig + 8)), dot4(gg, ldg4(L.ex_ig + 12))));
    if (own && lane < kMTot) {
      const float v = ge2 * (1.f + gt) + pick(gi, deg) * 2.f * e * inv_weight(deg);
      gev1[(size_t)atom * kMTot + lane] = v;
      if (gev1_copy) gev1_copy[(size_t)atom * kMTot + lane] = v;
    }
  }
  __syncthreads();
  contract<AT>(red, w, act);
  load_w128(w, L.res2_kT);
  __syncthreads();
  if (warp < AT) {
    g3 = add4(g3, get_sum<AT, NP>(red, warp, lane));
    g3 = add4(g3, make_float4(dot4(gg, ldg4(L.ex_xg + 4 * col)), dot4(gg, ldg4(L.ex_xg + 4 * col + 4)), dot4(gg, ldg4(L.ex_xg + 4 * col + 8)),
                              dot4(gg, ldg4(L.ex_xg + 4 * col + 12))));
    st4(act + warp * kF + col, g3);
  }
  __syncthreads();
  contract<AT>(red, w, act);
  load_w128(w, L.res1_kT);
  __syncthreads();
  if (warp < AT) st4(act + warp * kF + col, mul4(get_sum<AT, NP>(red, warp, lane), dsilu4(vz)));
  __syncthreads();
  contract<AT>(red, w, act);
  __syncthreads();
  if (warp < AT) {
    float rstd;
    const float4 xh = normalise(vxa, rstd), sc = ldg4(L.ln1_s + col), bi = ldg4(L.ln1_b + col);
    const float4 x1 = add4(mul4(xh, sc), bi);
    const float4 gx1 = add4(g3, mul4(get_sum<AT, NP>(red, warp, lane), dsilu4(x1)));
    const float4 o = normalise_vjp(mul4(gx1, sc), xh, rstd);
    if (own) st4(g_xa + ra, o);
  }
}

template <int AT>
__global__ void __launch_bounds__(NTHR, 1) heads_fwd_small_kernel(ModelDev M, int n, const int* __restrict__ Z, const float* x,
                                                                  float* __restrict__ ze, float* __restrict__ zq, float* __restrict__ zh,
                                                                  float* __restrict__ e_nn, float* __restrict__ q_raw, float* __restrict__ hv) {
  extern __shared__ __align__(16) float sm[];
  float* act = sm;                        // [AT][128]
  float* red_e = act + AT * kF;           // [4][AT][128]
  float* red_q = red_e + NP * AT * kF;    // [4][AT][128]
  float* red_h = red_q + NP * AT * kF;    // [8][AT][64]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col = 4 * lane;
  const int atom = blockIdx.x * AT + warp;
  const bool own = warp < AT && atom < n;
  const int p8 = tid >> 6, c64 = tid & 63;      // eight parts of a 64-column contraction
  float w[32];
  load_w128(w, M.e_reg_k);
  grid_dep_sync();
  if (warp < AT) st4(act + warp * kF + col, own ? ld4(x + (size_t)atom * kF + col) : zero4());
  const int z = own ? Z[atom] : 0;
  const int z_e = z < 0 ? 0 : (z >= kZEmbed ? kZEmbed - 1 : z), z_h = z < 0 ? 0 : (z >= kZHead ? kZHead - 1 : z);
  __syncthreads();
  contract<AT>(red_e, w, act);
  load_w128(w, M.q_reg_k);
  contract<AT>(red_q, w, act);
  if (p8 < 8) {
    load_w<16>(w, M.h_reg_k + (size_t)16 * p8 * 64 + c64, 64);
    float2 acc[AT];
    zero_acc<AT>(acc);
    dot_rows<AT, 16>(acc, w, act + 16 * p8, kF);
    put_partials<AT>(red_h, acc, p8, c64, 64);
    load_w<8>(w, M.h_fin_k + (size_t)8 * p8 * 64 + c64, 64);
  }
  __syncthreads();
  if (warp < AT) {
    const float4 ve = add4(get_sum<AT, NP>(red_e, warp, lane), ldg4(M.e_reg_b + col));
    const float4 vq = add4(get_sum<AT, NP>(red_q, warp, lane), ldg4(M.q_reg_b + col));
    const float se = wsum(dot4(silu4(ve), ldg4(M.e_fin_k + col))), sq = wsum(dot4(silu4(vq), ldg4(M.q_fin_k + col)));
    float h0 = M.h_reg_b[lane], h1 = M.h_reg_b[32 + lane];
#pragma unroll
    for (int p = 0; p < 8; ++p) { h0 += red_h[(p * AT + warp) * 64 + lane]; h1 += red_h[(p * AT + warp) * 64 + 32 + lane]; }
    if (own) {
      st4(ze + (size_t)atom * kF + col, ve);
      st4(zq + (size_t)atom * kF + col, vq);
      zh[(size_t)atom * 64 + lane] = h0; zh[(size_t)atom * 64 + 32 + lane] = h1;
      if (lane == 0) {
        e_nn[atom] = (se + M.e_fin_b) * M.e_scale[z_e] + M.e_offset[z_e];
        q_raw[atom] = sq + M.q_fin_b + M.q_embed[z_h];
      }
    }
    act[warp * kF + lane] = silu_f(h0); act[warp * kF + 32 + lane] = silu_f(h1);
  }
  __syncthreads();
  if (p8 < 8) {
    float2 acc[AT];
    zero_acc<AT>(acc);
    dot_rows<AT, 8>(acc, w, act + 8 * p8, kF);
    put_partials<AT>(red_h, acc, p8, c64, 64);
  }
  __syncthreads();
  if (warp < AT) {
    float h0 = M.h_fin_b[lane], h1 = M.h_fin_b[32 + lane];
#pragma unroll
    for (int p = 0; p < 8; ++p) { h0 += red_h[(p * AT + warp) * 64 + lane]; h1 += red_h[(p * AT + warp) * 64 + 32 + lane]; }
    const float s = wsum(fmaf(h0, M.h_embed1[z_h * 64 + lane], h1 * M.h_embed1[z_h * 64 + 32 + lane]));
    if (own && lane == 0) hv[atom] = M.h_embed0[z_h] + s * 0.125f;
  }
}

template <int AT>
__global__ void __launch_bounds__(NTHR, 1) heads_bwd_small_kernel(ModelDev M, int n, const int* __restrict__ Z, const float* ze,
                                                                  const float* zq, const float* zh,
                                                                  const float* hv, const float* ge,
                                                                  const float* gq, const float* gh, float* __restrict__ gx) {
  extern __shared__ __align__(16) float sm[];
  float* act_e = sm;                      // [AT][128]
  float* act_q = act_e + AT * kF;         // [AT][128]
  float* act_h = act_q + AT * kF;         // [AT][64]
  float* red = act_h + AT * 64;           // [4][AT][128] ([8][AT][64] first)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col = 4 * lane;
  const int atom = blockIdx.x * AT + warp;
  const bool own = warp < AT && atom < n;
  const int p = tid >> 7, c = tid & 127, p8 = tid >> 6, c64 = tid & 63;
  float w[32];
  float dh0 = 0.f, dh1 = 0.f;
  if (p8 < 8) load_w<8>(w, M.h_fin_kT + (size_t)8 * p8 * 64 + c64, 64);
  grid_dep_sync();
  if (warp < AT) {
    float4 ae = zero4(), aq = zero4();
    float k0 = 0.f, k1 = 0.f;
    if (own) {
      const int z = Z[atom];
      const int z_e = z < 0 ? 0 : (z >= kZEmbed ? kZEmbed - 1 : z), z_h = z < 0 ? 0 : (z >= kZHead ? kZHead - 1 : z);
      const float ce = ge[atom] * M.e_scale[z_e], cq = gq[atom], ch = gh[atom] * (hv[atom] < 0.f ? -0.125f : 0.125f);
      k0 = ch * M.h_embed1[z_h * 64 + lane]; k1 = ch * M.h_embed1[z_h * 64 + 32 + lane];
      dh0 = dsilu_f(zh[(size_t)atom * 64 + lane]); dh1 = dsilu_f(zh[(size_t)atom * 64 + 32 + lane]);
      ae = fma4(ce, mul4(ldg4(M.e_fin_k + col), dsilu4(ld4(ze + (size_t)atom * kF + col))), ae);
      aq = fma4(cq, mul4(ldg4(M.q_fin_k + col), dsilu4(ld4(zq + (size_t)atom * kF + col))), aq);
    }
    st4(act_e + warp * kF + col, ae);
    st4(act_q + warp * kF + col, aq);
    act_h[warp * 64 + lane] = k0; act_h[warp * 64 + 32 + lane] = k1;
  }
  __syncthreads();
  if (p8 < 8) {
    float2 acc[AT];
    zero_acc<AT>(acc);
    dot_rows<AT, 8>(acc, w, act_h + 8 * p8, 64);
    put_partials<AT>(red, acc, p8, c64, 64);
  }
  float2 acc[AT];
  zero_acc<AT>(acc);
  if (p < NP) {
    load_w128(w, M.e_reg_kT);
    dot_rows<AT, KP>(acc, w, act_e + KP * p, kF);
    load_w128(w, M.q_reg_kT);
    dot_rows<AT, KP>(acc, w, act_q + KP * p, kF);
    load_w<16>(w, M.h_reg_kT + (size_t)16 * p * kF + c, kF);
  }
  __syncthreads();
  if (warp < AT) {
    float h0 = 0.f, h1 = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) { h0 += red[(q * AT + warp) * 64 + lane]; h1 += red[(q * AT + warp) * 64 + 32 + lane]; }
    act_h[warp * 64 + lane] = h0 * dh0; act_h[warp * 64 + 32 + lane] = h1 * dh1;
  }
  __syncthreads();
  if (p < NP) {
    dot_rows<AT, 16>(acc, w, act_h + 16 * p, 64);
    put_partials<AT>(red, acc, p, c, kF);
  }
  __syncthreads();
  if (own) st4(gx + (size_t)atom * kF + col, get_sum<AT, NP>(red, warp, lane));
}

template <int AT> constexpr int smem_post_fwd() { return (1 + NP) * AT * kF * 4; }
template <int AT> constexpr int smem_post_bwd() { return (6 * kF + kProj) * AT * 4; }
template <int AT> constexpr int smem_heads_fwd() { return (kF + 2 * NP * kF + 8 * 64) * AT * 4; }
template <int AT> constexpr int smem_heads_bwd() { return (2 * kF + 64 + NP * kF) * AT * 4; }

template <int AT>
int configure() {
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(post_fwd_small_kernel<AT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_post_fwd<AT>()));
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(post_bwd_small_kernel<AT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_post_bwd<AT>()));
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(heads_fwd_small_kernel<AT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_heads_fwd<AT>()));
  SO3LR_CUDA_CHECK(cudaFuncSetAttribute(heads_bwd_small_kernel<AT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_heads_bwd<AT>()));
  return kOk;
}

// the smallest tile that still gives every CTA its own SM
int atoms_per_cta(int n) { return (n + sm_count() - 1) / sm_count(); }

}  // namespace

bool dense_small_applies(int n) { return n <= 16 * sm_count(); }

int configure_dense_small_kernels() {
  int rc = configure<2>();
  if (!rc) rc = configure<4>();
  if (!rc) rc = configure<6>();
  if (!rc) rc = configure<8>();
  if (!rc) rc = configure<10>();
  if (!rc) rc = configure<12>();
  if (!rc) rc = configure<16>();
  return rc;
}

#define SO3LR_SMALL_DISPATCH(n, CALL) \
  do { \
    const int at_ = atoms_per_cta(n); \
    if (at_ <= 2) { constexpr int AT = 2; CALL; } \
    else if (at_ <= 4) { constexpr int AT = 4; CALL; } \
    else if (at_ <= 6) { constexpr int AT = 6; CALL; } \
    else if (at_ <= 8) { constexpr int AT = 8; CALL; } \
    else if (at_ <= 10) { constexpr int AT = 10; CALL; } \
    else if (at_ <= 12) { constexpr int AT = 12; CALL; } \
    else { constexpr int AT = 16; CALL; } \
    count_launch(); \
  } while (0)

void launch_atom_post_fwd_small(cudaStream_t s, const LayerDev& L, int n, const float* xa, const float* ev1, float* z1, float* x3, float* gate,
                                float* x4, float* ev2, const float* projT, float* qkv_next, float* x4_copy, float* ev2_copy) {
  if (n <= 0) return;
  SO3LR_SMALL_DISPATCH(n, (launch_chained(post_fwd_small_kernel<AT>, (n + AT - 1) / AT, NTHR, smem_post_fwd<AT>(), s, L, n, xa, ev1, z1, x3, gate, x4, ev2, projT, qkv_next, x4_copy, ev2_copy)));
}
void launch_atom_post_bwd_small(cudaStream_t s, const LayerDev& L, int n, const float* xa, const float* ev1, const float* z1, const float* x3,
                                const float* gate, const float* g4, const float* gev2, float* g_xa, float* gev1, const float* proj,
                                float* g_qkv_up, float* gev1_copy) {
  if (n <= 0) return;
  SO3LR_SMALL_DISPATCH(n, (launch_chained(post_bwd_small_kernel<AT>, (n + AT - 1) / AT, NTHR, smem_post_bwd<AT>(), s, L, n, xa, ev1, z1, x3, gate, g4, gev2, g_xa, gev1, proj, g_qkv_up, gev1_copy)));
}
void launch_heads_fwd_small(cudaStream_t s, const ModelDev& M, int n, const int* Z, const float* x, float* ze, float* zq, float* zh, float* e_nn,
                            float* q_raw, float* hv) {
  if (n <= 0) return;
  SO3LR_SMALL_DISPATCH(n, (launch_chained(heads_fwd_small_kernel<AT>, (n + AT - 1) / AT, NTHR, smem_heads_fwd<AT>(), s, M, n, Z, x, ze, zq, zh, e_nn, q_raw, hv)));
}
void launch_heads_bwd_small(cudaStream_t s, const ModelDev& M, int n, const int* Z, const float* ze, const float* zq, const float* zh,
                            const float* hv, const float* ge, const float* gq, const float* gh, float* gx) {
  if (n <= 0) return;
  SO3LR_SMALL_DISPATCH(n, (launch_chained(heads_bwd_small_kernel<AT>, (n + AT - 1) / AT, NTHR, smem_heads_bwd<AT>(), s, M, n, Z, ze, zq, zh, hv, ge, gq, gh, gx)));
}

}  // namespace so3lr
