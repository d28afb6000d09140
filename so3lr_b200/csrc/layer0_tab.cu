// First SO3krates layer through per-species-pair tables.
//
// The inputs of layer 0 are constants of the atom's element: x0 = embedding[Z], ev0 = 0.  Its q/k/v rows therefore
// depend on the element only and the attention logits of an edge depend on (Z_i, Z_j, r) only:
//     D_h(Z_i, Z_j, r) = sum_{t in h} q_{Z_i}[t] k_{Z_j}[t] w(r)[t],
// where w(r) is the tabulated radial filter (cubic Hermite, four rows per interval: value, slope, value difference, far
// slope).  The interpolant is linear in those rows, so contracting them with q*k once per element pair gives a table of
// 4 x 8 numbers per interval (4 heads of the invariant branch, 4 degrees of the equivariant branch) that reproduces the
// generic kernel's logits (up to the order of additions) at 128 bytes of table traffic per edge instead of 4 KB of filter
// rows plus 1.5 KB of neighbour rows.
//   forward : lane = list entry; per edge a table lookup, the cutoff, the spherical harmonics; per-element sums of the
//             invariant coefficients are combined with the element's v row at the end
//   backward: only forces leave layer 0.  A thread per compacted pair evaluates both directions from the per-atom contractions
//             GV[j][element][head] = sum_{t in head} g_xa[j][t] v_element[t] (450 -> 167 us at 98,304 atoms against a lane per list
//             entry, which stays for the attention generations that build no pair list).  Caller-supplied lists: a thread per
//             entry, its own direction only, which is the entry's exact gradient on a list of any form.
#include <algorithm>
#include <vector>

#include "kernels.h"

namespace so3lr {

namespace {

constexpr float kInvNbar = 1.0f / kAvgNumNeighbors;
constexpr float kRc2 = kCutoffSr * kCutoffSr;
constexpr int SP = kMaxTabSpecies;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

__device__ __forceinline__ void hermite_weights(float r, int& g, float4& hv, float4& hd) {
  float t = r * (1.0f / kTableH);
  g = (int)t;
  g = g > kTableGrid - 2 ? kTableGrid - 2 : g;
  t -= (float)g;
  const float t2 = t * t, t3 = t2 * t;
  hv = make_float4(1.f, t3 - 2.f * t2 + t, -2.f * t3 + 3.f * t2, t3 - t2);      // applied to (v0, h m0, v1 - v0, h m1)
  const float ih = 1.0f / kTableH;
  hd = make_float4(0.f, (3.f * t2 - 4.f * t + 1.f) * ih, (-6.f * t2 + 6.f * t) * ih, (3.f * t2 - 2.f * t) * ih);
}

// 32 per-lane partials -> lane L holds the total of entry L
__device__ __forceinline__ float warp_transpose_reduce32(float (&v)[32], int lane) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float send = (lane & 16) ? v[i] : v[i + 16], keep = (lane & 16) ? v[i + 16] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float send = (lane & 8) ? v[i] : v[i + 8], keep = (lane & 8) ? v[i + 8] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float send = (lane & 4) ? v[i] : v[i + 4], keep = (lane & 4) ? v[i + 4] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float send = (lane & 2) ? v[i] : v[i + 2], keep = (lane & 2) ? v[i + 2] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  }
  const float send = (lane & 1) ? v[0] : v[1], keep = (lane & 1) ? v[1] : v[0];
  return keep + __shfl_xor_sync(0xffffffffu, send, 1);
}

// table[(a * SP + b)][interval][32]: the four interval rows of the radial table (value, slope, value difference, far
// slope) contracted with q_a * k_b per head: entry 8 * row + 4 * filter + head.  Sums are formed in double precision.  The intervals
// are spread over kTableSplit CTAs per element pair: with one CTA a water box (4 pairs) used 4 SMs and took 0.81 ms.
constexpr int kTableSplit = 32;
__global__ void build_pair_table_kernel(const float* __restrict__ radial, const float* __restrict__ qkv_sp, int n_sp,
                                        float* __restrict__ table) {
  const int a = blockIdx.y / n_sp, b = blockIdx.y % n_sp;
  const float* qa = qkv_sp + (size_t)a * kProj;
  const float* kb = qkv_sp + (size_t)b * kProj;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < (kTableGrid - 1) * 32; idx += gridDim.x * blockDim.x) {
    const int iv = idx >> 5, o = idx & 31;
    const int grp = o & 3, filt = (o >> 2) & 1, row = o >> 3;
    const float* w = radial + ((size_t)iv * 4 + row) * 256 + filt * kF + 32 * grp;
    const float* q = qa + (filt ? 3 * kF : 0) + 32 * grp;
    const float* k = kb + (filt ? 4 * kF : kF) + 32 * grp;
    double s = 0.0;
    for (int t = 0; t < 32; ++t) s += (double)q[t] * (double)k[t] * (double)w[t];
    table[((size_t)(a * SP + b) * (kTableGrid - 1) + iv) * 32 + o] = (float)s;
  }
}

__global__ void __launch_bounds__(256) layer0_fwd_tab_kernel(SpeciesTables T, const float* __restrict__ embed, int n_recv, int n,
                                                             const int* __restrict__ row_ptr, const int* __restrict__ nbr_j,
                                                             const float* dR, const int* __restrict__ Z,
                                                             float* __restrict__ xa, float* __restrict__ ev1) {
  grid_dep_sync();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n_recv) return;
  const int Zi = Z[i];
  const int zi = T.slot[Zi < 0 ? 0 : (Zi > 118 ? 118 : Zi)];
  float A[32], EV[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) { A[k] = 0.f; EV[k] = 0.f; }
  const int e0 = row_ptr[i], e1 = row_ptr[i + 1];
  for (int e = e0 + lane; e < e1; e += 32) {
    const int j = nbr_j[e];
    const float dx = dR[3 * (size_t)e], dy = dR[3 * (size_t)e + 1], dz = dR[3 * (size_t)e + 2];
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (j < 0 || j >= n || !(r2 < kRc2) || !(r2 > 0.f)) continue;
    const float r = sqrtf(r2), ir = 1.f / r;
    float cut, dcut;
    phys_cutoff(r, cut, dcut);
    const float sc = cut * kInvNbar;
    int g; float4 hv, hd;
    hermite_weights(r, g, hv, hd);
    const int Zj = Z[j];
    const int zj = T.slot[Zj < 0 ? 0 : (Zj > 118 ? 118 : Zj)];
    const float* row = T.table + ((size_t)(zi * SP + zj) * (kTableGrid - 1) + g) * 32;
    const float4 v0a = ld4(row), v0b = ld4(row + 4), m0a = ld4(row + 8), m0b = ld4(row + 12);
    const float4 v1a = ld4(row + 16), v1b = ld4(row + 20), m1a = ld4(row + 24), m1b = ld4(row + 28);   // "v1" = value difference
    float a1[4], a2[4];
    a1[0] = sc * (hv.x * v0a.x + hv.y * m0a.x + hv.z * v1a.x + hv.w * m1a.x);
    a1[1] = sc * (hv.x * v0a.y + hv.y * m0a.y + hv.z * v1a.y + hv.w * m1a.y);
    a1[2] = sc * (hv.x * v0a.z + hv.y * m0a.z + hv.z * v1a.z + hv.w * m1a.z);
    a1[3] = sc * (hv.x * v0a.w + hv.y * m0a.w + hv.z * v1a.w + hv.w * m1a.w);
    a2[0] = sc * (hv.x * v0b.x + hv.y * m0b.x + hv.z * v1b.x + hv.w * m1b.x);
    a2[1] = sc * (hv.x * v0b.y + hv.y * m0b.y + hv.z * v1b.y + hv.w * m1b.y);
    a2[2] = sc * (hv.x * v0b.z + hv.y * m0b.z + hv.z * v1b.z + hv.w * m1b.z);
    a2[3] = sc * (hv.x * v0b.w + hv.y * m0b.w + hv.z * v1b.w + hv.w * m1b.w);
#pragma unroll
    for (int z = 0; z < SP; ++z) {
      const float m = (zj == z) ? 1.f : 0.f;
#pragma unroll
      for (int h = 0; h < 4; ++h) A[4 * z + h] = fmaf(m, a1[h], A[4 * z + h]);
    }
    float Y[kMTot];
    sph_harm_24(dx * ir, dy * ir, dz * ir, Y);
#pragma unroll
    for (int m = 0; m < kMTot; ++m) EV[m] = fmaf(a2[degree_of(m)], Y[m], EV[m]);
  }
  const float At = warp_transpose_reduce32(A, lane);     // lane 4z + h: sum of a1_h over neighbours of element z
  const float Et = warp_transpose_reduce32(EV, lane);    // lane m: ev component m
  const int col = 4 * lane, hL = lane >> 3;
  float4 acc = ld4(embed + (size_t)(Zi < 0 ? 0 : (Zi >= kZEmbed ? kZEmbed - 1 : Zi)) * kF + col);
#pragma unroll
  for (int z = 0; z < SP; ++z) {
    const float c = __shfl_sync(0xffffffffu, At, 4 * z + hL);
    if (z < T.n_species) {
      const float4 v = ld4(T.v_sp + (size_t)z * kF + col);
      acc.x = fmaf(c, v.x, acc.x); acc.y = fmaf(c, v.y, acc.y); acc.z = fmaf(c, v.z, acc.z); acc.w = fmaf(c, v.w, acc.w);
    }
  }
  *reinterpret_cast<float4*>(xa + (size_t)i * kF + col) = acc;
  if (lane < kMTot) ev1[(size_t)i * kMTot + lane] = Et;
}

// GV[a][z][h] = sum_{t in head h} g_xa[a][t] * v_z[t]
__global__ void __launch_bounds__(256) layer0_gv_kernel(SpeciesTables T, int n, const float* g_xa, float* __restrict__ GV) {
  grid_dep_sync();
  const int lane = threadIdx.x & 31;
  const int a = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (a >= n) return;
  const float4 g = ld4(g_xa + (size_t)a * kF + 4 * lane);
  float out = 0.f;   // lane 4z + h keeps GV[a][z][h]
#pragma unroll
  for (int z = 0; z < SP; ++z) {
    float s = 0.f;
    if (z < T.n_species) {
      const float4 v = ld4(T.v_sp + (size_t)z * kF + 4 * lane);
      s = g.x * v.x + g.y * v.y + g.z * v.z + g.w * v.w;
    }
    s = group8_sum(s);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float sh = __shfl_sync(0xffffffffu, s, 8 * h);
      if (lane == 4 * z + h) out = sh;
    }
  }
  GV[(size_t)a * (4 * SP) + lane] = out;
}

// One direction (receiver of element zr, sender of element zs) of a pair's table entry: adds to the derivative with respect to r and
// returns the equivariant logits x cutoff.  d1, d2: cotangents of the invariant and of the equivariant coefficients.
__device__ __forceinline__ void table_reverse(const SpeciesTables& T, int zr, int zs, int g, float4 hv, float4 hd, float sc, float dcn, float4 d1,
                                              const float (&d2)[4], float& gr, float (&a2)[4]) {
  const float* row = T.table + ((size_t)(zr * SP + zs) * (kTableGrid - 1) + g) * 32;
  const float4 v0a = ld4(row), v0b = ld4(row + 4), m0a = ld4(row + 8), m0b = ld4(row + 12);
  const float4 v1a = ld4(row + 16), v1b = ld4(row + 20), m1a = ld4(row + 24), m1b = ld4(row + 28);
  const float D1[4] = {hv.x * v0a.x + hv.y * m0a.x + hv.z * v1a.x + hv.w * m1a.x, hv.x * v0a.y + hv.y * m0a.y + hv.z * v1a.y + hv.w * m1a.y,
                       hv.x * v0a.z + hv.y * m0a.z + hv.z * v1a.z + hv.w * m1a.z, hv.x * v0a.w + hv.y * m0a.w + hv.z * v1a.w + hv.w * m1a.w};
  const float D2[4] = {hv.x * v0b.x + hv.y * m0b.x + hv.z * v1b.x + hv.w * m1b.x, hv.x * v0b.y + hv.y * m0b.y + hv.z * v1b.y + hv.w * m1b.y,
                       hv.x * v0b.z + hv.y * m0b.z + hv.z * v1b.z + hv.w * m1b.z, hv.x * v0b.w + hv.y * m0b.w + hv.z * v1b.w + hv.w * m1b.w};
  const float E1[4] = {hd.x * v0a.x + hd.y * m0a.x + hd.z * v1a.x + hd.w * m1a.x, hd.x * v0a.y + hd.y * m0a.y + hd.z * v1a.y + hd.w * m1a.y,
                       hd.x * v0a.z + hd.y * m0a.z + hd.z * v1a.z + hd.w * m1a.z, hd.x * v0a.w + hd.y * m0a.w + hd.z * v1a.w + hd.w * m1a.w};
  const float E2[4] = {hd.x * v0b.x + hd.y * m0b.x + hd.z * v1b.x + hd.w * m1b.x, hd.x * v0b.y + hd.y * m0b.y + hd.z * v1b.y + hd.w * m1b.y,
                       hd.x * v0b.z + hd.y * m0b.z + hd.z * v1b.z + hd.w * m1b.z, hd.x * v0b.w + hd.y * m0b.w + hd.z * v1b.w + hd.w * m1b.w};
  const float d1v[4] = {d1.x, d1.y, d1.z, d1.w};
  float dsc = 0.f, dder = 0.f;
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    dsc = fmaf(d1v[h], D1[h], fmaf(d2[h], D2[h], dsc));
    dder = fmaf(d1v[h], E1[h], fmaf(d2[h], E2[h], dder));
    a2[h] = sc * D2[h];
  }
  gr += dcn * dsc + sc * dder;
}
__device__ __forceinline__ int element_slot(const SpeciesTables& T, int z) { return T.slot[z < 0 ? 0 : (z > 118 ? 118 : z)]; }
__device__ __forceinline__ void load_ev(const float* __restrict__ p, float (&v)[kMTot]) {
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const float4 q = ld4(p + 4 * c);
    v[4 * c] = q.x; v[4 * c + 1] = q.y; v[4 * c + 2] = q.z; v[4 * c + 3] = q.w;
  }
}
// Force on atom i of the pair (i, j), d = (dx, dy, dz) from i to j: both directions (BOTH), or the derivative of the direction (i <- j)
// with respect to d alone.
template <bool BOTH>
__device__ __forceinline__ float3 pair_reverse(const SpeciesTables& T, int i, int j, float dx, float dy, float dz, float r, const int* __restrict__ Z,
                                               const float* __restrict__ GV, const float* __restrict__ gev1) {
  const float ir = 1.f / r, ux = dx * ir, uy = dy * ir, uz = dz * ir;
  float cut, dcut;
  phys_cutoff(r, cut, dcut);
  const float sc = cut * kInvNbar, dcn = dcut * kInvNbar;
  int g; float4 hv, hd;
  hermite_weights(r, g, hv, hd);
  const int zi = element_slot(T, Z[i]), zj = element_slot(T, Z[j]);
  float Y[kMTot], gi[kMTot], gj[kMTot];
  sph_harm_24(ux, uy, uz, Y);
  load_ev(gev1 + (size_t)i * kMTot, gi);
  if (BOTH) load_ev(gev1 + (size_t)j * kMTot, gj);
  float dA2[4] = {0.f, 0.f, 0.f, 0.f}, dB2[4] = {0.f, 0.f, 0.f, 0.f}, a2A[4], a2B[4], gr = 0.f;
#pragma unroll
  for (int m = 0; m < kMTot; ++m) {
    dA2[degree_of(m)] = fmaf(gi[m], Y[m], dA2[degree_of(m)]);
    if (BOTH) dB2[degree_of(m)] = fmaf(gj[m], Y[m], dB2[degree_of(m)]);
  }
  dB2[0] = -dB2[0]; dB2[2] = -dB2[2];       // Y_lm(-u) = (-1)^l Y_lm(u)
  table_reverse(T, zi, zj, g, hv, hd, sc, dcn, ld4(GV + (size_t)i * (4 * SP) + 4 * zj), dA2, gr, a2A);
  if (BOTH) table_reverse(T, zj, zi, g, hv, hd, sc, dcn, ld4(GV + (size_t)j * (4 * SP) + 4 * zi), dB2, gr, a2B);
  float gY[kMTot];
#pragma unroll
  for (int m = 0; m < kMTot; ++m) {
    const int l = degree_of(m);
    const float sgn = (l == 0 || l == 2) ? -1.f : 1.f;
    gY[m] = BOTH ? a2A[l] * gi[m] + sgn * a2B[l] * gj[m] : a2A[l] * gi[m];
  }
  float gux, guy, guz;
  sph_harm_24_vjp(ux, uy, uz, gY, gux, guy, guz);
  const float gd = gux * ux + guy * uy + guz * uz;
  return make_float3(gr * ux + (gux - gd * ux) * ir, gr * uy + (guy - gd * uy) * ir, gr * uz + (guz - gd * uz) * ir);
}

// Forces from the full list, a warp per receiver (with the attention kernels that do not build the compacted pair list).
__global__ void __launch_bounds__(256) layer0_bwd_tab_kernel(SpeciesTables T, int n_recv, int n, const int* __restrict__ row_ptr,
                                                             const int* __restrict__ nbr_j, const float* __restrict__ dR,
                                                             const int* __restrict__ Z, const float* __restrict__ GV,
                                                             const float* __restrict__ gev1, float* __restrict__ F,
                                                             float* __restrict__ virial) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n_recv) return;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  VirialAcc va;
  const int e0 = row_ptr[i], e1 = row_ptr[i + 1];
  for (int e = e0 + lane; e < e1; e += 32) {
    const int j = nbr_j[e];
    const float dx = dR[3 * (size_t)e], dy = dR[3 * (size_t)e + 1], dz = dR[3 * (size_t)e + 2];
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (j < 0 || j >= n || !(r2 < kRc2) || !(r2 > 0.f)) continue;
    const float3 f = pair_reverse<true>(T, i, j, dx, dy, dz, sqrtf(r2), Z, GV, gev1);
    fx += f.x; fy += f.y; fz += f.z;
    if (virial) va.add(0.5f, dx, dy, dz, f.x, f.y, f.z);
  }
  fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz);
  if (lane == 0) { F[3 * (size_t)i] += fx; F[3 * (size_t)i + 1] += fy; F[3 * (size_t)i + 2] += fz; }
  if (virial) va.flush_warp(virial, (size_t)i, lane);
}

// Forces from the compacted pair list (one entry per undirected pair, sorted by its receiver): a thread per pair, so that every lane
// has one (the full list's rows hold the skin too and leave 45 % of the lanes without work, and every pair was evaluated at both ends).
// Equal receivers inside a warp are summed before they go out; the partner gets its share if it owns a row.  Rows of `virial` below
// n_own add up to the total, in any distribution: every warp adds its sum to one of them.
__global__ void __launch_bounds__(128) layer0_bwd_pairs_kernel(SpeciesTables T, int n_recv, const int* n_listed,
                                                               const int* ve_i, const int* ve_j,
                                                               const float4* ve_d, const int* __restrict__ Z,
                                                               const float* GV, const float* gev1,
                                                               float* __restrict__ F, float* __restrict__ virial, int n_own) {
  grid_dep_sync();
  const int lane = threadIdx.x & 31;
  const long long n_pairs = *n_listed;
  const long long warp0 = (long long)blockIdx.x * 4 + (threadIdx.x >> 5), step = (long long)gridDim.x * 128;
  VirialAcc va;
  for (long long e0 = 32 * warp0; e0 < n_pairs; e0 += step) {
    const long long e = e0 + lane;
    int i = -1, j = -1;
    float3 f = make_float3(0.f, 0.f, 0.f);
    if (e < n_pairs) {
      i = ve_i[e]; j = ve_j[e];
      const float4 d = ve_d[e];
      f = pair_reverse<true>(T, i, j, d.x, d.y, d.z, d.w, Z, GV, gev1);
      if (virial) va.add(0.5f * ((i < n_own ? 1.f : 0.f) + (j < n_own ? 1.f : 0.f)), d.x, d.y, d.z, f.x, f.y, f.z);
      if (j < n_recv) { atomicAdd(F + 3 * (size_t)j, -f.x); atomicAdd(F + 3 * (size_t)j + 1, -f.y); atomicAdd(F + 3 * (size_t)j + 2, -f.z); }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float tx = __shfl_up_sync(0xffffffffu, f.x, o), ty = __shfl_up_sync(0xffffffffu, f.y, o), tz = __shfl_up_sync(0xffffffffu, f.z, o);
      const int ti = __shfl_up_sync(0xffffffffu, i, o);
      if (lane >= o && ti == i) { f.x += tx; f.y += ty; f.z += tz; }
    }
    const int inext = __shfl_down_sync(0xffffffffu, i, 1);
    if (i >= 0 && (lane == 31 || inext != i)) {
      atomicAdd(F + 3 * (size_t)i, f.x); atomicAdd(F + 3 * (size_t)i + 1, f.y); atomicAdd(F + 3 * (size_t)i + 2, f.z);
    }
  }
  if (virial && n_own > 0 && 32 * warp0 < n_pairs) {
    const float a = warp_sum(va.xx), b = warp_sum(va.yy), c = warp_sum(va.zz), d = warp_sum(va.yz), e = warp_sum(va.xz), h = warp_sum(va.xy);
    if (lane == 0) {
      float* w = virial + 6 * (size_t)(warp0 % n_own);
      atomicAdd(w, a); atomicAdd(w + 1, b); atomicAdd(w + 2, c); atomicAdd(w + 3, d); atomicAdd(w + 4, e); atomicAdd(w + 5, h);
    }
  }
}

// Gradient with respect to every displacement of a caller-supplied list (added to g_dR); the list may be of any form.
__global__ void __launch_bounds__(128) layer0_bwd_entries_kernel(SpeciesTables T, int n, long long n_entries, const int* __restrict__ idx_i,
                                                                 const int* __restrict__ idx_j, const float* __restrict__ dR,
                                                                 const int* __restrict__ Z, const float* __restrict__ GV,
                                                                 const float* __restrict__ gev1, float* __restrict__ g_dR) {
  const long long e = (long long)blockIdx.x * 128 + threadIdx.x;
  if (e >= n_entries) return;
  const int i = idx_i[e], j = idx_j[e];
  const float dx = dR[3 * e], dy = dR[3 * e + 1], dz = dR[3 * e + 2];
  const float r2 = dx * dx + dy * dy + dz * dz;
  if (i < 0 || i >= n || j < 0 || j >= n || !(r2 < kRc2) || !(r2 > 0.f)) return;
  const float3 f = pair_reverse<false>(T, i, j, dx, dy, dz, sqrtf(r2), Z, GV, gev1);
  g_dR[3 * e] += f.x; g_dR[3 * e + 1] += f.y; g_dR[3 * e + 2] += f.z;
}

// the elements as a kernel argument: a copy from the host's stack would need a wait, and a context of one evaluation (a batch of a
// dataset) builds its tables in the middle of it
struct SpeciesList {
  int slot[119], z[SP];
};
__global__ void set_species_kernel(SpeciesList L, int* __restrict__ slot, int* __restrict__ z) {
  if (threadIdx.x < 119) slot[threadIdx.x] = L.slot[threadIdx.x];
  if (threadIdx.x < SP) z[threadIdx.x] = L.z[threadIdx.x];
}

}  // namespace

static int build_tables(cudaStream_t st, const ModelDev& M, const std::vector<int>& sp, SpeciesTables* T) {
  if (!T->table) SO3LR_CUDA_CHECK(dev_alloc(&T->table, (size_t)SP * SP * (kTableGrid - 1) * 32));
  if (!T->v_sp) SO3LR_CUDA_CHECK(dev_alloc(&T->v_sp, (size_t)SP * kF));
  if (!T->slot) SO3LR_CUDA_CHECK(dev_alloc(&T->slot, 119));
  if (!T->qkv_sp) SO3LR_CUDA_CHECK(dev_alloc(&T->qkv_sp, (size_t)SP * kProj));
  if (!T->x_sp) SO3LR_CUDA_CHECK(dev_alloc(&T->x_sp, (size_t)SP * kF));
  if (!T->z_sp) SO3LR_CUDA_CHECK(dev_alloc(&T->z_sp, SP));
  const int ns = (int)sp.size();
  SpeciesList list{};
  for (int k = 0; k < ns; ++k) { list.slot[sp[k]] = k; list.z[k] = sp[k]; }
  set_species_kernel<<<1, 128, 0, st>>>(list, T->slot, T->z_sp);
  count_launch();
  launch_embed(st, M, T->z_sp, ns, T->x_sp);
  launch_proj_fwd(st, M.layer[0], T->x_sp, ns, T->qkv_sp);
  SO3LR_CUDA_CHECK(cudaMemcpy2DAsync(T->v_sp, kF * sizeof(float), T->qkv_sp + 2 * kF, kProj * sizeof(float), kF * sizeof(float), ns,
                                     cudaMemcpyDeviceToDevice, st));
  { build_pair_table_kernel<<<dim3(kTableSplit, ns * ns), 256, 0, st>>>(M.layer[0].table, T->qkv_sp, ns, T->table); count_launch(); }
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// (Re)builds the tables for the elements present in Z_host; returns kOk with T->n_species = 0 when more than
// kMaxTabSpecies elements occur (the caller then uses the generic kernels).  After a failure there are none: nothing is half built.
int species_tables_build(cudaStream_t st, const ModelDev& M, const int* Z_host, int n, SpeciesTables* T) {
  std::vector<int> sp;
  for (int a = 0; a < n; ++a) {
    int z = Z_host[a];
    z = z < 0 ? 0 : (z > 118 ? 118 : z);
    if (std::find(sp.begin(), sp.end(), z) == sp.end()) sp.push_back(z);
    if ((int)sp.size() > SP) break;
  }
  if ((int)sp.size() > SP || sp.empty()) { T->n_species = 0; return kOk; }
  std::sort(sp.begin(), sp.end());
  bool same = T->n_species == (int)sp.size();
  for (int k = 0; same && k < (int)sp.size(); ++k) same = T->species[k] == sp[k];
  if (same) return kOk;
  T->n_species = 0;
  const int rc = build_tables(st, M, sp, T);
  if (rc) { species_tables_free(T); return rc; }
  T->n_species = (int)sp.size();
  for (int k = 0; k < T->n_species; ++k) T->species[k] = sp[k];
  return kOk;
}

void species_tables_free(SpeciesTables* T) {
  dev_free(T->table); dev_free(T->v_sp); dev_free(T->slot); dev_free(T->qkv_sp); dev_free(T->x_sp); dev_free(T->z_sp);
  *T = SpeciesTables{};
}

void launch_layer0_fwd_tab(cudaStream_t s, const SpeciesTables& T, const ModelDev& M, int n_recv, int n, const int* row_ptr,
                           const int* nbr_j, const float* dR, const int* Z, float* xa, float* ev1) {
  if (n_recv <= 0) return;
  { launch_chained(layer0_fwd_tab_kernel, (n_recv + 7) / 8, 256, 0, s, T, M.embed_z, n_recv, n, row_ptr, nbr_j, dR, Z, xa, ev1); count_launch(); }
}

void launch_layer0_bwd_tab(cudaStream_t s, const SpeciesTables& T, int n_recv, int n_gv, int n, const int* row_ptr, const int* nbr_j,
                           const float* dR, const int* Z, const float* g_xa, const float* gev1, float* GV, float* F, float* virial) {
  if (n_recv <= 0) return;
  { launch_chained(layer0_gv_kernel, (n_gv + 7) / 8, 256, 0, s, T, n_gv, g_xa, GV); count_launch(); }
  { layer0_bwd_tab_kernel<<<(n_recv + 7) / 8, 256, 0, s>>>(T, n_recv, n, row_ptr, nbr_j, dR, Z, GV, gev1, F, virial); count_launch(); }
}

void launch_layer0_bwd_pairs(cudaStream_t s, const SpeciesTables& T, int n_recv, int n_gv, const ValidEdges& V, const int* Z, const float* g_xa,
                             const float* gev1, float* GV, float* F, float* virial, int n_own) {
  if (n_recv <= 0) return;
  { launch_chained(layer0_gv_kernel, (n_gv + 7) / 8, 256, 0, s, T, n_gv, g_xa, GV); count_launch(); }
  // the number of pairs stays on the device: four CTAs per SM walk over the list, fewer where the rows cannot fill them
  int blocks = (int)(((long long)n_recv * 24 + 127) / 128);
  if (blocks > 4 * sm_count()) blocks = 4 * sm_count();
  { launch_chained(layer0_bwd_pairs_kernel, blocks, 128, 0, s, T, n_recv, V.total, V.i, V.j, V.d, Z, GV, gev1, F, virial, n_own); count_launch(); }
}

void launch_layer0_bwd_entries(cudaStream_t s, const SpeciesTables& T, int n, long long n_entries, const int* idx_i, const int* idx_j,
                               const float* dR, const int* Z, const float* g_xa, const float* gev1, float* GV, float* g_dR) {
  if (n <= 0 || n_entries <= 0) return;
  { launch_chained(layer0_gv_kernel, (n + 7) / 8, 256, 0, s, T, n, g_xa, GV); count_launch(); }
  { layer0_bwd_entries_kernel<<<(unsigned)((n_entries + 127) / 128), 128, 0, s>>>(T, n, n_entries, idx_i, idx_j, dR, Z, GV, gev1, g_dR); count_launch(); }
}

}  // namespace so3lr
