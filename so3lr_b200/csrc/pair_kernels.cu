// Edge geometry + ZBL repulsion on the short-range graph, the fused long-range pair kernel (damped Coulomb +
// dispersion with analytic gradients) and the small per-graph reductions around them.
#include <algorithm>

#include "kernels.h"

namespace so3lr {

namespace {

__global__ void sr_geometry_zbl_kernel(ZblParams zbl, Cell cell, int n, long long n_edges, const int* __restrict__ edge_i,
                                       const int* __restrict__ nbr_j, const int* __restrict__ Z, const float* R,
                                       int dR_given, float* dR, float* __restrict__ e_atom,
                                       float* g_dR, const float* ge, float* __restrict__ F_direct, int n_owned,
                                       float* __restrict__ virial) {
  grid_dep_sync();
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_edges) return;
  const int i = edge_i[e], j = nbr_j[e];
  float dx = 0.f, dy = 0.f, dz = 0.f;
  const bool valid = i >= 0 && i < n && j >= 0 && j < n;
  if (dR_given) {
    dx = dR[3 * e]; dy = dR[3 * e + 1]; dz = dR[3 * e + 2];
  } else {
    if (valid) {
      dx = R[3 * (size_t)j] - R[3 * (size_t)i];
      dy = R[3 * (size_t)j + 1] - R[3 * (size_t)i + 1];
      dz = R[3 * (size_t)j + 2] - R[3 * (size_t)i + 2];
      min_image(cell, dx, dy, dz);
    }
    dR[3 * e] = dx; dR[3 * e + 1] = dy; dR[3 * e + 2] = dz;
  }
  float gx = 0.f, gy = 0.f, gz = 0.f;
  const float r2 = dx * dx + dy * dy + dz * dz;
  // n_owned >= 0: only the edges of owned receivers carry energy, and the receiver takes the pair's whole force
  // (the reversed edge belongs to the other atom's owner)
  if (valid && r2 > 0.f && r2 < kZblSwitchOff * kZblSwitchOff && (n_owned < 0 || i < n_owned)) {
    const float r = sqrtf(r2);
    float cut, dcut, ez, dez;
    phys_cutoff(r, cut, dcut);
    zbl_edge(zbl, r, cut, dcut, Z[i], Z[j], ez, dez);
    atomicAdd(e_atom + i, ez);
    const float s = (ge ? ge[i] : 1.f) * dez / r;
    gx = s * dx; gy = s * dy; gz = s * dz;
    if (virial) {     // every directed edge carries its own energy: dE/d eps += dR (x) g
      float* w = virial + 6 * (size_t)i;
      atomicAdd(w, dx * gx); atomicAdd(w + 1, dy * gy); atomicAdd(w + 2, dz * gz);
      atomicAdd(w + 3, dy * gz); atomicAdd(w + 4, dx * gz); atomicAdd(w + 5, dx * gy);
    }
    if (F_direct) {   // only edges shorter than 1.5 A get here: a handful per atom
      const float wi = n_owned >= 0 ? 2.f : 1.f;
      atomicAdd(F_direct + 3 * (size_t)i, wi * gx); atomicAdd(F_direct + 3 * (size_t)i + 1, wi * gy); atomicAdd(F_direct + 3 * (size_t)i + 2, wi * gz);
      if (n_owned < 0) {
        atomicAdd(F_direct + 3 * (size_t)j, -gx); atomicAdd(F_direct + 3 * (size_t)j + 1, -gy); atomicAdd(F_direct + 3 * (size_t)j + 2, -gz);
      }
    }
  }
  if (g_dR) { g_dR[3 * e] = gx; g_dR[3 * e + 1] = gy; g_dR[3 * e + 2] = gz; }
}

__global__ void force_scatter_kernel(int n, long long n_edges, const int* __restrict__ edge_i, const int* __restrict__ nbr_j,
                                     const float* __restrict__ g_dR, float* __restrict__ F) {
  long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_edges) return;
  const float gx = g_dR[3 * e], gy = g_dR[3 * e + 1], gz = g_dR[3 * e + 2];
  if (gx == 0.f && gy == 0.f && gz == 0.f) return;
  const int i = edge_i[e], j = nbr_j[e];
  if (i < 0 || i >= n || j < 0 || j >= n) return;
  // E depends on dR = R_j - R_i:  F_i = +g, F_j = -g
  atomicAdd(F + 3 * (size_t)i, gx); atomicAdd(F + 3 * (size_t)i + 1, gy); atomicAdd(F + 3 * (size_t)i + 2, gz);
  atomicAdd(F + 3 * (size_t)j, -gx); atomicAdd(F + 3 * (size_t)j + 1, -gy); atomicAdd(F + 3 * (size_t)j + 2, -gz);
}

// one warp per row i; lanes stride over the row's pairs
template <int MODE>
__global__ void __launch_bounds__(256) pair_lr_kernel(LrParams P, Cell cell, int n, const int* __restrict__ row_ptr,
                                                      const int* __restrict__ nbr_j, const int* __restrict__ Z,
                                                      const float* __restrict__ R, const float* __restrict__ q,
                                                      const float* __restrict__ h, const float* __restrict__ dR_lr,
                                                      float* __restrict__ g_dR_lr, float* __restrict__ e_atom,
                                                      float* __restrict__ F, float* __restrict__ gq, float* __restrict__ gh,
                                                      float* __restrict__ e_coul, float* __restrict__ e_disp, const float* __restrict__ ge,
                                                      float* __restrict__ virial) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n) return;
  VirialAcc va;
  const int e0 = row_ptr[i], e1 = row_ptr[i + 1];
  if (e0 == e1) return;
  const float qi = q[i], hi = h[i];
  const float alf_i = alpha_free(Z[i]), x_i = dispersion_x(Z[i]);
  const float gei = ge ? ge[i] : 1.f;
  float xi = 0.f, yi = 0.f, zi = 0.f;
  if (MODE == 0) { xi = R[3 * (size_t)i]; yi = R[3 * (size_t)i + 1]; zi = R[3 * (size_t)i + 2]; }
  float ec = 0.f, ed = 0.f, fx = 0.f, fy = 0.f, fz = 0.f, gqi = 0.f, ghi = 0.f;
  for (int e = e0 + lane; e < e1; e += 32) {
    const int j = nbr_j[e];
    float gx = 0.f, gy = 0.f, gz = 0.f;
    if (j >= 0 && j < n) {
      float dx, dy, dz;
      if (MODE == 0) {
        dx = R[3 * (size_t)j] - xi; dy = R[3 * (size_t)j + 1] - yi; dz = R[3 * (size_t)j + 2] - zi;
        min_image(cell, dx, dy, dz);
      } else {
        dx = dR_lr[3 * (size_t)e]; dy = dR_lr[3 * (size_t)e + 1]; dz = dR_lr[3 * (size_t)e + 2];
      }
      const float r2 = dx * dx + dy * dy + dz * dz;
      if (r2 > 0.f && (!P.has_cutoff || r2 < P.rc * P.rc)) {
        const float rinv = rsqrtf(r2), r = r2 * rinv;
        float chi, dchi;
        coulomb_chi(P, r, rinv, chi, dchi);
        const float qj = q[j], hj = h[j];
        const float pf = P.pair_factor;
        const float kq = pf * kKe;
        const float e_c = kq * qi * qj * chi;
        float e_d, dd_dr, dd_dhi, dd_dhj;
        const int Zj = Z[j];
        dispersion_pair_fast(P, r, alf_i, x_i, hi, alpha_free(Zj), dispersion_x(Zj), hj, e_d, dd_dr, dd_dhi, dd_dhj);
        e_d *= pf; dd_dr *= pf; dd_dhi *= pf; dd_dhj *= pf;
        ec += e_c; ed += e_d;
        gqi = fmaf(kq * qj, chi, gqi);
        ghi += dd_dhi;
        atomicAdd(gq + j, gei * kq * qi * chi);
        atomicAdd(gh + j, gei * dd_dhj);
        const float de_dr = gei * (kq * qi * qj * dchi + dd_dr);
        const float s = de_dr * rinv;
        gx = s * dx; gy = s * dy; gz = s * dz;   // dE/d(dR), dR = R_j - R_i
        if (MODE == 0) {
          if (virial) va.add(1.f, dx, dy, dz, gx, gy, gz);     // every listed pair carries its own share of the energy
          fx += gx; fy += gy; fz += gz;
          atomicAdd(F + 3 * (size_t)j, -gx); atomicAdd(F + 3 * (size_t)j + 1, -gy); atomicAdd(F + 3 * (size_t)j + 2, -gz);
        }
      }
    }
    if (MODE == 1) { g_dR_lr[3 * (size_t)e] = gx; g_dR_lr[3 * (size_t)e + 1] = gy; g_dR_lr[3 * (size_t)e + 2] = gz; }
  }
  ec = warp_sum(ec); ed = warp_sum(ed); gqi = warp_sum(gqi); ghi = warp_sum(ghi);
  if (MODE == 0) { fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz); }
  if (lane == 0) {
    if (e_atom) atomicAdd(e_atom + i, ec + ed);
    if (e_coul) atomicAdd(e_coul + i, ec);
    if (e_disp) atomicAdd(e_disp + i, ed);
    atomicAdd(gq + i, gei * gqi);
    atomicAdd(gh + i, gei * ghi);
    if (MODE == 0) { atomicAdd(F + 3 * (size_t)i, fx); atomicAdd(F + 3 * (size_t)i + 1, fy); atomicAdd(F + 3 * (size_t)i + 2, fz); }
  }
  if (MODE == 0 && virial) va.flush_warp(virial, (size_t)i, lane);
}

// The single-device long-range kernel with packed operands: per atom (x, y, z, q) and (h, alpha_free, alpha_free^2 / c6_free, -) so that a pair costs two
// 16-byte gathers, and a packed accumulator (Fx, Fy, Fz, dE/dq) so that the sender's share of a pair is one
// vector reduction (red.global.add.v4.f32) and one scalar one (dE/dh) instead of five scalar atomics.
__global__ void __launch_bounds__(256) pair_pack_kernel(int n, const float* R, const float* q,
                                                        const float* h, const int* __restrict__ Z,
                                                        float4* __restrict__ pq, float4* __restrict__ hz, float4* acc) {
  grid_dep_sync();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  pq[i] = make_float4(R[3 * (size_t)i], R[3 * (size_t)i + 1], R[3 * (size_t)i + 2], q[i]);
  hz[i] = make_float4(h[i], alpha_free(Z[i]), dispersion_x(Z[i]), 0.f);
  acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
// with e_atom also the per-atom energies: the sum of the network's, the repulsion's and the two pair terms' shares
__global__ void __launch_bounds__(256) pair_unpack_kernel(int n, const float4* acc, float* F, float* gq,
                                                          const float* e_nn, const float* e_zbl,
                                                          const float* e_coul, const float* e_disp, float* __restrict__ e_atom) {
  grid_dep_sync();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = acc[i];
  F[3 * (size_t)i] += a.x; F[3 * (size_t)i + 1] += a.y; F[3 * (size_t)i + 2] += a.z;
  gq[i] += a.w;
  if (e_atom) e_atom[i] = ((e_nn[i] + e_zbl[i]) + e_coul[i]) + e_disp[i];
}
__device__ __forceinline__ void red_add_f4(float4* p, float x, float y, float z, float w) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
// QUEUED (lists with a skin): the entries inside the cutoff (four of five at a 1 A skin) pass through a queue in shared memory, so that the
// arithmetic of the pair terms runs with full warps.  `split` warps share a row (see pair_row_split).
template <bool QUEUED>
__global__ void __launch_bounds__(256) pair_lr_packed_kernel(LrParams P, Cell cell, int n, int split, const int* __restrict__ row_ptr,
                                                             const int* __restrict__ nbr_j, const float4* pq,
                                                             const float4* hz, float4* __restrict__ acc,
                                                             float* __restrict__ gh, float* e_coul,
                                                             float* e_disp, float* __restrict__ virial) {
  __shared__ float4 queue_d[QUEUED ? 8 : 1][QUEUED ? 64 : 1];      // displacement and charge
  __shared__ int queue_j[QUEUED ? 8 : 1][QUEUED ? 64 : 1];
  grid_dep_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = (blockIdx.x * 8 + warp) / split, part = (blockIdx.x * 8 + warp) % split;
  if (i >= n) return;
  VirialAcc va;
  const int e0 = row_ptr[i] + 32 * part, e1 = row_ptr[i + 1];
  if (e0 >= e1) return;
  const float4 pi = pq[i];
  const float4 hzi = hz[i];
  const float qi = pi.w, hi = hzi.x;
  const float pf = P.pair_factor, kq = pf * kKe, rc2 = P.rc * P.rc;
  float ec = 0.f, ed = 0.f, fx = 0.f, fy = 0.f, fz = 0.f, gqi = 0.f, ghi = 0.f;
  auto pair = [&](int j, float dx, float dy, float dz, float qj) {
    const float4 hzj = hz[j];
    const float r2 = dx * dx + dy * dy + dz * dz;
    const float rinv = rsqrtf(r2), r = r2 * rinv;
    float chi, dchi;
    coulomb_chi(P, r, rinv, chi, dchi);
    float e_d, dd_dr, dd_dhi, dd_dhj;
    dispersion_pair_fast(P, r, hzi.y, hzi.z, hi, hzj.y, hzj.z, hzj.x, e_d, dd_dr, dd_dhi, dd_dhj);
    ec = fmaf(kq * qi * qj, chi, ec);
    ed = fmaf(pf, e_d, ed);
    gqi = fmaf(kq * qj, chi, gqi);
    ghi = fmaf(pf, dd_dhi, ghi);
    const float s = (kq * qi * qj * dchi + pf * dd_dr) * rinv;
    const float gx = s * dx, gy = s * dy, gz = s * dz;   // dE/d(dR), dR = R_j - R_i
    if (virial) va.add(1.f, dx, dy, dz, gx, gy, gz);
    fx += gx; fy += gy; fz += gz;
    red_add_f4(acc + j, -gx, -gy, -gz, kq * qi * chi);
    atomicAdd(gh + j, pf * dd_dhj);
  };
  int waiting = 0;
  for (int eb = e0; eb < e1; eb += 32 * split) {
    const int e = eb + lane;
    const int j = e < e1 ? nbr_j[e] : -1;
    bool inside = j >= 0 && j < n;
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (inside) {
      const float4 pj = pq[j];
      d = make_float4(pj.x - pi.x, pj.y - pi.y, pj.z - pi.z, pj.w);
      min_image(cell, d.x, d.y, d.z);
      const float r2 = d.x * d.x + d.y * d.y + d.z * d.z;
      inside = r2 > 0.f && !(P.has_cutoff && r2 >= rc2);
    }
    if (!QUEUED) {
      if (inside) pair(j, d.x, d.y, d.z, d.w);
      continue;
    }
    const unsigned m = __ballot_sync(0xffffffffu, inside);
    if (inside) {
      const int at = waiting + __popc(m & ((1u << lane) - 1u));
      queue_d[warp][at] = d;
      queue_j[warp][at] = j;
    }
    waiting += __popc(m);
    __syncwarp();
    if (waiting >= 32) {
      waiting -= 32;
      const float4 w = queue_d[warp][waiting + lane];
      pair(queue_j[warp][waiting + lane], w.x, w.y, w.z, w.w);
      __syncwarp();
    }
  }
  if (QUEUED && lane < waiting) {
    const float4 w = queue_d[warp][lane];
    pair(queue_j[warp][lane], w.x, w.y, w.z, w.w);
  }
  __syncwarp();
  ec = warp_sum(ec); ed = warp_sum(ed); gqi = warp_sum(gqi); ghi = warp_sum(ghi);
  fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz);
  if (lane == 0) {
    if (split == 1) { e_coul[i] += ec; e_disp[i] += ed; }      // only this warp writes the energies of row i
    else { atomicAdd(e_coul + i, ec); atomicAdd(e_disp + i, ed); }
    red_add_f4(acc + i, fx, fy, fz, gqi);
    atomicAdd(gh + i, ghi);
  }
  if (virial) va.flush_warp(virial, (size_t)i, lane, split > 1);
}
// Warps per row.  A short list leaves most of the chip idle with one: 1,536 atoms are 10 warps per SM, and a row of the ordered list holds up to
// 12 rounds of 32 pairs, each a chain of gathers and some 400 instructions (2 us).  As many warps as the average row has rounds and as 32
// per SM allow (what 62 registers a thread keep resident); never more than 12 (390 atoms in a list with both directions).
// The three launches of the pair terms without / with a 1 A skin, us, one warp a row -> this rule: 192 atoms 17.5 / 18.9 -> 13.3 / 13.4 (3 warps),
// 390: 24.7 / 27.6 -> 15.0 / 15.5 (6, 7), 600: 29.9 / 33.9 -> 17.6 / 18.1 (7), 1,536: 36.5 / 48.0 -> 24.1 / 25.8 (3); one warp from 2,369 atoms
// on: 38.0 / 50.0 at 2,400 (two warps there, two waves of blocks: 35.6 / 36.0).
int pair_row_split(int n, long long pairs) {
  const long long rounds = (pairs / n + 31) / 32, room = 32LL * sm_count() / n;
  return (int)std::max(1LL, std::min(rounds, room));
}

// Owned rows of an ordered list over owned atoms and ghosts (decomposed runs; ghosts carry the larger indices, so the list
// holds every pair of two owned atoms once and every owned-ghost pair in the owned atom's row).  A pair of two owned atoms
// books its whole energy on the row atom and scatters the other end's derivatives with atomics; a pair with a ghost end books
// half of the energy and the row atom's derivatives only (the ghost's owner does the same from its side).  gq, gh and F_add
// must hold the values to add to (zeros for gq, gh) when the kernel starts.
__global__ void __launch_bounds__(256) pair_lr_owned_kernel(LrParams P, Cell cell, int n_owned, int n, const int* __restrict__ row_ptr,
                                                            const int* __restrict__ nbr_j, const int* __restrict__ Z,
                                                            const float* __restrict__ R, const float* __restrict__ q,
                                                            const float* __restrict__ h, float* __restrict__ F_add,
                                                            float* __restrict__ gq, float* __restrict__ gh, float* __restrict__ e_coul,
                                                            float* __restrict__ e_disp, float* __restrict__ virial) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n_owned) return;
  const int e0 = row_ptr[i], e1 = row_ptr[i + 1];
  const float qi = q[i], hi = h[i];
  const float alf_i = alpha_free(Z[i]), x_i = dispersion_x(Z[i]);
  const float xi = R[3 * (size_t)i], yi = R[3 * (size_t)i + 1], zi = R[3 * (size_t)i + 2];
  float ec = 0.f, ed = 0.f, fx = 0.f, fy = 0.f, fz = 0.f, gqi = 0.f, ghi = 0.f;
  VirialAcc va;
  for (int e = e0 + lane; e < e1; e += 32) {
    const int j = nbr_j[e];
    if (j < 0 || j >= n) continue;
    float dx = R[3 * (size_t)j] - xi, dy = R[3 * (size_t)j + 1] - yi, dz = R[3 * (size_t)j + 2] - zi;
    min_image(cell, dx, dy, dz);
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (!(r2 > 0.f) || (P.has_cutoff && r2 >= P.rc * P.rc)) continue;
    const float rinv = rsqrtf(r2), r = r2 * rinv;
    float chi, dchi;
    coulomb_chi(P, r, rinv, chi, dchi);
    const float qj = q[j], hj = h[j];
    const int Zj = Z[j];
    float e_d, dd_dr, dd_dhi, dd_dhj;
    dispersion_pair_fast(P, r, alf_i, x_i, hi, alpha_free(Zj), dispersion_x(Zj), hj, e_d, dd_dr, dd_dhi, dd_dhj);
    const bool both = j < n_owned;
    const float w = both ? 1.f : 0.5f;                             // share of the pair energy booked on this row
    ec = fmaf(w * kKe * qi * qj, chi, ec);
    ed = fmaf(w, e_d, ed);
    gqi = fmaf(kKe * qj, chi, gqi);
    ghi += dd_dhi;
    const float s = (kKe * qi * qj * dchi + dd_dr) * rinv;   // dE_ij/d(dR), dR = R_j - R_i; F_i = +that, F_j = -that
    const float gx = s * dx, gy = s * dy, gz = s * dz;
    fx += gx; fy += gy; fz += gz;
    if (virial) va.add(w * s, dx, dy, dz, dx, dy, dz);
    if (both) {
      atomicAdd(gq + j, kKe * qi * chi);
      atomicAdd(gh + j, dd_dhj);
      atomicAdd(F_add + 3 * (size_t)j, -gx); atomicAdd(F_add + 3 * (size_t)j + 1, -gy); atomicAdd(F_add + 3 * (size_t)j + 2, -gz);
    }
  }
  ec = warp_sum(ec); ed = warp_sum(ed); gqi = warp_sum(gqi); ghi = warp_sum(ghi);
  fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz);
  if (lane == 0) {
    e_coul[i] = ec; e_disp[i] = ed;      // only this warp writes the energies of row i
    atomicAdd(gq + i, gqi); atomicAdd(gh + i, ghi);
    atomicAdd(F_add + 3 * (size_t)i, fx); atomicAdd(F_add + 3 * (size_t)i + 1, fy); atomicAdd(F_add + 3 * (size_t)i + 2, fz);
  }
  if (virial) va.flush_warp(virial, (size_t)i, lane);
}

// one CTA per graph: q = q_raw + (Q - sum q_raw) / n_g ; h = |hv|
__global__ void charge_conserve_kernel(int n_graphs, const int* __restrict__ graph_start, const float* q_raw,
                                       const float* __restrict__ total_charge, const float* hv,
                                       float* __restrict__ q, float* __restrict__ h) {
  grid_dep_sync();
  __shared__ float red[32];
  const int g = blockIdx.x;
  const int a0 = graph_start[g], a1 = graph_start[g + 1];
  float s = 0.f;
  for (int a = a0 + threadIdx.x; a < a1; a += blockDim.x) s += q_raw[a];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    v = warp_sum(v);
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const float Q = total_charge ? total_charge[g] : 0.f;
  // the shift is applied in double: rounded to float32 first, its relative error times the atom count would show up in sum q
  const double corr = a1 > a0 ? ((double)Q - (double)red[0]) / (double)(a1 - a0) : 0.0;
  for (int a = a0 + threadIdx.x; a < a1; a += blockDim.x) {
    q[a] = (float)((double)q_raw[a] + corr);
    h[a] = fabsf(hv[a]);
  }
}

// gq_raw = gq - mean_graph(gq)
__global__ void charge_conserve_bwd_kernel(int n_graphs, const int* __restrict__ graph_start, const float* gq,
                                           float* __restrict__ gq_raw) {
  grid_dep_sync();
  __shared__ float red[32];
  const int g = blockIdx.x;
  const int a0 = graph_start[g], a1 = graph_start[g + 1];
  float s = 0.f;
  for (int a = a0 + threadIdx.x; a < a1; a += blockDim.x) s += gq[a];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    v = warp_sum(v);
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const float mean = a1 > a0 ? red[0] / (float)(a1 - a0) : 0.f;
  for (int a = a0 + threadIdx.x; a < a1; a += blockDim.x) gq_raw[a] = gq[a] - mean;
}

// per-graph energy (double accumulation) and dipole sum_i q_i R_i; one CTA per graph
__global__ void graph_reduce_kernel(int n_graphs, const int* __restrict__ graph_start, const float* e_atom,
                                    const float* q, const float* R, double* __restrict__ e_graph,
                                    float* __restrict__ dipole) {
  grid_dep_sync();
  __shared__ double red[4][32];
  const int g = blockIdx.x;
  const int a0 = graph_start[g], a1 = graph_start[g + 1];
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int a = a0 + threadIdx.x; a < a1; a += blockDim.x) {
    v[0] += (double)e_atom[a];
    if (R) {
      float qa = q[a];
      v[1] += (double)(qa * R[3 * (size_t)a]); v[2] += (double)(qa * R[3 * (size_t)a + 1]); v[3] += (double)(qa * R[3 * (size_t)a + 2]);
    }
  }
  for (int k = 0; k < 4; ++k) {
    double s = v[k];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
    if (threadIdx.x == 0) e_graph[g] = s;
    else if (dipole) dipole[3 * g + threadIdx.x - 1] = (float)s;
  }
}

// ---- one structure with many atoms: the same three operations spread over many CTAs (sums in double, fixed order) ----
constexpr int kWideBlocks = 296;      // two CTAs per SM of a 148-SM part; a fixed count keeps the order of the double sums independent of the device
// One CTA takes 23 to 28 us for 12,000 atoms, the two wide launches 6.  The three sums of an evaluation (water, 6 A long range) wide / in
// one CTA: 216 / 208 us at 192 atoms, 284 / 280 at 768, 401 / 403 at 1,536, 688 / 694 at 3,072, 794 / 801 at 4,095, 967 / 986 at 6,144,
// 1,485 / 1,546 at 12,288.  They meet near 1,500 atoms; up to the line the one CTA costs 7 us (1 %) and is one launch less.
constexpr int kWideMinAtoms = 4096;

__device__ double block_sum_double_256(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < 8; ++w) s += sh[w];
  __syncthreads();
  return s;       // valid in thread 0
}

// partials[b][0] = sum a ; with R: partials[b][1..3] = sum q R
__global__ void __launch_bounds__(256) wide_partial_kernel(int n, const float* a, const float* q,
                                                           const float* R, double* __restrict__ partials) {
  grid_dep_sync();
  __shared__ double sh[8];
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    v[0] += (double)a[i];
    if (R) {
      const float qa = q[i];
      v[1] += (double)(qa * R[3 * (size_t)i]); v[2] += (double)(qa * R[3 * (size_t)i + 1]); v[3] += (double)(qa * R[3 * (size_t)i + 2]);
    }
  }
  for (int k = 0; k < (R ? 4 : 1); ++k) {
    const double s = block_sum_double_256(v[k], sh);
    if (threadIdx.x == 0) partials[4 * blockIdx.x + k] = s;
  }
}

__device__ double wide_total(const double* __restrict__ partials, int n_blocks, int k, double* sh) {
  // every CTA forms the same total from the same partials in the same order
  double v = 0.0;
  for (int b = threadIdx.x; b < n_blocks; b += 256) v += partials[4 * b + k];
  const double s = block_sum_double_256(v, sh);
  __shared__ double total;
  if (threadIdx.x == 0) total = s;
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(256) charge_conserve_wide_kernel(int n, const float* q_raw, const float* __restrict__ total_charge,
                                                                   const float* hv, float* __restrict__ q, float* __restrict__ h,
                                                                   const double* partials, int n_blocks) {
  grid_dep_sync();
  __shared__ double sh[8];
  const float Q = total_charge ? total_charge[0] : 0.f;
  // in double: a float32 shift carries a relative error of 6e-8, which times a million atoms is a visible net charge
  const double corr = ((double)Q - wide_total(partials, n_blocks, 0, sh)) / (double)n;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    q[i] = (float)((double)q_raw[i] + corr);
    h[i] = fabsf(hv[i]);
  }
}

__global__ void __launch_bounds__(256) charge_conserve_bwd_wide_kernel(int n, const float* gq, float* __restrict__ gq_raw,
                                                                       const double* partials, int n_blocks) {
  grid_dep_sync();
  __shared__ double sh[8];
  const float mean = (float)wide_total(partials, n_blocks, 0, sh) / (float)n;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) gq_raw[i] = gq[i] - mean;
}

__global__ void __launch_bounds__(256) graph_reduce_wide_kernel(const double* partials, int n_blocks, int with_dipole,
                                                                double* __restrict__ e_graph, float* __restrict__ dipole) {
  grid_dep_sync();
  __shared__ double sh[8];
  for (int k = 0; k < (with_dipole ? 4 : 1); ++k) {
    const double t = wide_total(partials, n_blocks, k, sh);
    if (threadIdx.x == 0) {
      if (k == 0) e_graph[0] = t;
      else if (dipole) dipole[k - 1] = (float)t;
    }
    __syncthreads();
  }
}

}  // namespace

void launch_sr_geometry_zbl(cudaStream_t s, const ModelDev& M, const Cell& cell, int n, long long n_edges, const int* edge_i,
                            const int* nbr_j, const int* Z, const float* R, int dR_given, float* dR, float* e_atom, float* g_dR, const float* ge,
                            float* F_direct, int n_owned, float* virial) {
  if (n_edges <= 0) return;
  unsigned blocks = (unsigned)((n_edges + 255) / 256);
  { launch_chained(sr_geometry_zbl_kernel, blocks, 256, 0, s, M.zbl, cell, n, n_edges, edge_i, nbr_j, Z, R, dR_given, dR, e_atom, g_dR, ge, F_direct, n_owned, virial); count_launch(); }
}

void launch_force_scatter(cudaStream_t s, int n, long long n_edges, const int* edge_i, const int* nbr_j, const float* g_dR, float* F) {
  if (n_edges <= 0) return;
  unsigned blocks = (unsigned)((n_edges + 255) / 256);
  { force_scatter_kernel<<<blocks, 256, 0, s>>>(n, n_edges, edge_i, nbr_j, g_dR, F); count_launch(); }
}

void launch_pair_lr(cudaStream_t s, const LrParams& P, const Cell& cell, int n, const int* row_ptr, const int* nbr_j,
                    const int* Z, const float* R, const float* q, const float* h, int mode, const float* dR_lr,
                    float* g_dR_lr, float* e_atom, float* F, float* gq, float* gh, float* e_coul, float* e_disp, const float* ge,
                    float* virial) {
  if (n <= 0) return;
  int blocks = (n + 7) / 8;
  if (mode == 0)
    { pair_lr_kernel<0><<<blocks, 256, 0, s>>>(P, cell, n, row_ptr, nbr_j, Z, R, q, h, dR_lr, g_dR_lr, e_atom, F, gq, gh, e_coul, e_disp, ge, virial); count_launch(); }
  else
    { pair_lr_kernel<1><<<blocks, 256, 0, s>>>(P, cell, n, row_ptr, nbr_j, Z, R, q, h, dR_lr, g_dR_lr, e_atom, F, gq, gh, e_coul, e_disp, ge, virial); count_launch(); }
}

void launch_pair_lr_packed(cudaStream_t s, const LrParams& P, const Cell& cell, int n, const int* row_ptr, const int* nbr_j, const int* Z,
                           const float* R, const float* q, const float* h, float* pack /* 12 n floats */, float* F, float* gq, float* gh,
                           float* e_coul, float* e_disp, float* virial, const float* e_nn, const float* e_zbl, float* e_atom, bool skin,
                           long long pairs) {
  if (n <= 0) return;
  float4* pq = reinterpret_cast<float4*>(pack);
  float4* acc = pq + n;
  float4* hz = acc + n;
  launch_chained(pair_pack_kernel, (n + 255) / 256, 256, 0, s, n, R, q, h, Z, pq, hz, acc);
  const int split = pair_row_split(n, pairs);
  const unsigned blocks = (unsigned)(((long long)n * split + 7) / 8);
  if (skin) launch_chained(pair_lr_packed_kernel<true>, blocks, 256, 0, s, P, cell, n, split, row_ptr, nbr_j, pq, hz, acc, gh, e_coul, e_disp, virial);
  else launch_chained(pair_lr_packed_kernel<false>, blocks, 256, 0, s, P, cell, n, split, row_ptr, nbr_j, pq, hz, acc, gh, e_coul, e_disp, virial);
  launch_chained(pair_unpack_kernel, (n + 255) / 256, 256, 0, s, n, acc, F, gq, e_nn, e_zbl, e_coul, e_disp, e_atom);
  count_launch(3);
}

void launch_pair_lr_owned(cudaStream_t s, const LrParams& P, const Cell& cell, int n_owned, int n, const int* row_ptr,
                          const int* nbr_j, const int* Z, const float* R, const float* q, const float* h, float* F_add,
                          float* gq, float* gh, float* e_coul, float* e_disp, float* virial) {
  if (n_owned <= 0) return;
  cudaMemsetAsync(gq, 0, (size_t)n_owned * sizeof(float), s);
  cudaMemsetAsync(gh, 0, (size_t)n_owned * sizeof(float), s);
  { pair_lr_owned_kernel<<<(n_owned + 7) / 8, 256, 0, s>>>(P, cell, n_owned, n, row_ptr, nbr_j, Z, R, q, h, F_add, gq, gh, e_coul, e_disp, virial); count_launch(); }
}

void launch_charge_conserve(cudaStream_t s, int n_graphs, const int* graph_start, const float* q_raw,
                            const float* total_charge, const float* hv, float* q, float* h, int n_atoms, double* scratch) {
  if (n_graphs <= 0) return;
  if (n_graphs == 1 && scratch && n_atoms >= kWideMinAtoms) {
    launch_chained(wide_partial_kernel, kWideBlocks, 256, 0, s, n_atoms, q_raw, nullptr, nullptr, scratch);
    launch_chained(charge_conserve_wide_kernel, kWideBlocks, 256, 0, s, n_atoms, q_raw, total_charge, hv, q, h, scratch, kWideBlocks);
    count_launch(2);
    return;
  }
  { launch_chained(charge_conserve_kernel, n_graphs, 256, 0, s, n_graphs, graph_start, q_raw, total_charge, hv, q, h); count_launch(); }
}
void launch_charge_conserve_bwd(cudaStream_t s, int n_graphs, const int* graph_start, const float* gq, float* gq_raw, int n_atoms,
                                double* scratch) {
  if (n_graphs <= 0) return;
  if (n_graphs == 1 && scratch && n_atoms >= kWideMinAtoms) {
    launch_chained(wide_partial_kernel, kWideBlocks, 256, 0, s, n_atoms, gq, nullptr, nullptr, scratch);
    launch_chained(charge_conserve_bwd_wide_kernel, kWideBlocks, 256, 0, s, n_atoms, gq, gq_raw, scratch, kWideBlocks);
    count_launch(2);
    return;
  }
  { launch_chained(charge_conserve_bwd_kernel, n_graphs, 256, 0, s, n_graphs, graph_start, gq, gq_raw); count_launch(); }
}
void launch_graph_reduce(cudaStream_t s, int n_graphs, const int* graph_start, const float* e_atom, const float* q,
                         const float* R, double* e_graph, float* dipole, int n_atoms, double* scratch) {
  if (n_graphs <= 0) return;
  if (n_graphs == 1 && scratch && n_atoms >= kWideMinAtoms) {
    launch_chained(wide_partial_kernel, kWideBlocks, 256, 0, s, n_atoms, e_atom, q, R, scratch);
    launch_chained(graph_reduce_wide_kernel, 1, 256, 0, s, scratch, kWideBlocks, R ? 1 : 0, e_graph, dipole);
    count_launch(2);
    return;
  }
  { launch_chained(graph_reduce_kernel, n_graphs, 256, 0, s, n_graphs, graph_start, e_atom, q, R, e_graph, dipole); count_launch(); }
}

}  // namespace so3lr
