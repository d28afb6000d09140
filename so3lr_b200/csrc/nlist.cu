// Cell-list neighbor lists on the GPU (replaces jax_md.partition.neighbor_list for the 4.5 A and 12 A graphs).
//
// Atoms are binned into cells no smaller than the list radius, sorted by cell with a stable radix sort (so the
// row contents are deterministic), and one warp per atom scans the 27 (or fewer) surrounding cells with a
// ballot-compaction into its row.  Two passes (count, fill) with an exclusive scan in between give exact rows.
// Distances use the minimum-image convention with the float32 operation order of common.cuh::min_image and
// d2 = (dx*dx + dy*dy) + dz*dz < r*r, evaluated without fused multiply-adds.
#include "kernels.h"

#include <cub/cub.cuh>

namespace so3lr {

struct Grid {
  int nc[3];        // cells per dimension
  int wrap[3];      // periodic wrap in that dimension
  float lo[3];      // free space: lower corner
  float inv_w[3];   // free space: 1 / cell width
  int n_atoms;      // candidates in all
};
struct NlistWorkspace {
  int* cell_of = nullptr;      // n
  int* cell_sorted = nullptr;  // n
  int* atom_sorted = nullptr;  // n   atom indices ordered by cell
  int* atom_iota = nullptr;    // n
  int* cell_start = nullptr;   // ncell_total + 1
  float4* pos_sorted = nullptr; // n: positions in cell order, w = atom index (bit pattern)
  int* row_count = nullptr;    // n + 1
  void* cub_tmp = nullptr;
  size_t cub_bytes = 0;
  long long* d_total = nullptr;
  long long* h_total = nullptr;  // pinned
  int n_cap = 0, cell_cap = 0;
  // spatial ordering of the atoms (Morton keys of the short-range cells)
  unsigned* key = nullptr;
  unsigned* key_sorted = nullptr;
  void* sort_tmp = nullptr;
  size_t sort_bytes = 0;
  int key_cap = 0;
  unsigned* masks = nullptr;   // votes of the row count for the fill
  size_t mask_cap = 0;
  int* ticket = nullptr;       // of the scan at the end of the count kernels
  // list under way between nlist_begin and nlist_end
  Grid G{};
  int n = 0, n_rows = 0, ordered = 0, allow_grow = 1, mask_stride = 0;
  bool by_graph = false, binned = false;
  float r_list = 0.f;
  const float* R = nullptr;
  const int *seg = nullptr, *graph_start = nullptr;
};

NlistWorkspace* nlist_workspace_create() { return new NlistWorkspace(); }
void nlist_workspace_destroy(NlistWorkspace* w) {
  if (!w) return;
  dev_free(w->cell_of); dev_free(w->cell_sorted); dev_free(w->atom_sorted); dev_free(w->atom_iota);
  dev_free(w->cell_start); dev_free(w->row_count); dev_free(w->cub_tmp); dev_free(w->d_total);
  dev_free(w->key); dev_free(w->key_sorted); dev_free(w->sort_tmp); dev_free(w->pos_sorted); dev_free(w->masks); dev_free(w->ticket);
  if (w->h_total) host_free(w->h_total);
  delete w;
}

// gives the vote buffer back (its next build asks for it again); false when there is none
bool nlist_drop_votes(NlistWorkspace* w) {
  if (!w || !w->masks) return false;
  dev_free(w->masks);
  w->masks = nullptr; w->mask_cap = 0;
  return true;
}

namespace {


__device__ __forceinline__ void cell_coords(const Cell& cell, const Grid& G, float x, float y, float z, int* c) {
  if (cell.periodic) {
    float s0 = x * cell.hinv[0] + y * cell.hinv[3] + z * cell.hinv[6];
    float s1 = x * cell.hinv[1] + y * cell.hinv[4] + z * cell.hinv[7];
    float s2 = x * cell.hinv[2] + y * cell.hinv[5] + z * cell.hinv[8];
    s0 -= floorf(s0); s1 -= floorf(s1); s2 -= floorf(s2);
    c[0] = min((int)(s0 * G.nc[0]), G.nc[0] - 1);
    c[1] = min((int)(s1 * G.nc[1]), G.nc[1] - 1);
    c[2] = min((int)(s2 * G.nc[2]), G.nc[2] - 1);
  } else {
    c[0] = min(max((int)((x - G.lo[0]) * G.inv_w[0]), 0), G.nc[0] - 1);
    c[1] = min(max((int)((y - G.lo[1]) * G.inv_w[1]), 0), G.nc[1] - 1);
    c[2] = min(max((int)((z - G.lo[2]) * G.inv_w[2]), 0), G.nc[2] - 1);
  }
}

__global__ void assign_cells_kernel(Cell cell, Grid G, int n, const float* __restrict__ R, int* __restrict__ cell_of,
                                    int* __restrict__ iota) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n) return;
  int c[3];
  cell_coords(cell, G, R[3 * (size_t)a], R[3 * (size_t)a + 1], R[3 * (size_t)a + 2], c);
  cell_of[a] = (c[2] * G.nc[1] + c[1]) * G.nc[0] + c[0];
  iota[a] = a;
}

__global__ void cell_bounds_kernel(int n, int n_cells, const int* __restrict__ cell_sorted, int* __restrict__ cell_start) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > n) return;
  int cur = k < n ? cell_sorted[k] : n_cells;
  int prev = k > 0 ? cell_sorted[k - 1] : -1;
  for (int c = prev + 1; c <= cur; ++c) cell_start[c] = k;
}

// positions in cell order (one coalesced 16-byte load per candidate in the row kernels)
__global__ void gather_sorted_positions_kernel(int n, const float* __restrict__ R, const int* __restrict__ atom_sorted,
                                               float4* __restrict__ pos_sorted) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int a = atom_sorted[k];
  pos_sorted[k] = make_float4(R[3 * (size_t)a], R[3 * (size_t)a + 1], R[3 * (size_t)a + 2], __int_as_float(a));
}

// What the count kernels of short lists do at their end in place of four more launches: the CTA that finishes last turns the row counts
// into offsets (32 bits) and leaves their 64-bit sum in row_ptr[n] (clamped) and in pinned host memory.
struct TailScan {
  int* ticket = nullptr;            // two words, zero before and after: CTAs that are through, whether a position is not finite
  int* row_ptr = nullptr;
  long long* total_host = nullptr;  // pinned; -1: a position is not finite
  bool check_finite = false;
};
// The line (16 rounds of one CTA): building and exporting the 4.5 A list of water with the device-wide scan / with the last CTA takes
// 108 / 88 us at 1,536 atoms, 178 / 166 at 8,193, 229 / 217 at 16,383, 273 / 271 at 24,576, 327 / 327 at 32,769, 520 / 542 at 65,535.
constexpr int kTailScanRows = 32768;
__device__ __forceinline__ void tail_scan(const TailScan& T, int n, const int* __restrict__ row_count) {
  if (!T.ticket) return;
  __shared__ int last;
  __shared__ long long part[8];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(T.ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // 2,048 counts at a time, eight consecutive ones per thread (two 16-byte loads and stores)
  const int tid = threadIdx.x, lane = tid & 31;
  long long at = 0;
  for (int base = 0; base < n; base += 2048) {
    const int k0 = base + 8 * tid;
    int c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (k0 + 8 <= n) {
      const int4 a = __ldcg(reinterpret_cast<const int4*>(row_count + k0)), b = __ldcg(reinterpret_cast<const int4*>(row_count + k0) + 1);
      c[0] = a.x; c[1] = a.y; c[2] = a.z; c[3] = a.w; c[4] = b.x; c[5] = b.y; c[6] = b.z; c[7] = b.w;
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) if (k0 + q < n) c[q] = __ldcg(row_count + k0 + q);
    }
    long long sum = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) sum += c[q];
    long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const long long t = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += t; }
    if (lane == 31) part[tid >> 5] = incl;
    __syncthreads();
    long long mine = at + incl - sum;
#pragma unroll
    for (int w = 0; w < 8; ++w) { if (w < (tid >> 5)) mine += part[w]; at += part[w]; }
    __syncthreads();
    int o[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) { o[q] = (int)mine; mine += c[q]; }
    if (k0 + 8 <= n) {
      reinterpret_cast<int4*>(T.row_ptr + k0)[0] = make_int4(o[0], o[1], o[2], o[3]);
      reinterpret_cast<int4*>(T.row_ptr + k0)[1] = make_int4(o[4], o[5], o[6], o[7]);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) if (k0 + q < n) T.row_ptr[k0 + q] = o[q];
    }
  }
  if (tid == 255) {
    T.row_ptr[n] = at > 2147483647LL ? 2147483647 : (int)at;
    *T.total_host = __ldcg(T.ticket + 1) != 0 ? -1 : at;
    T.ticket[0] = 0; T.ticket[1] = 0;
  }
}

// FILL = false: row_count[i] = number of neighbours.  FILL = true: write rows at row_ptr[i].
// The candidates of a row come in cell order.  Cells that are neighbours along the first axis are neighbours in the sorted array: up to
// three of them are walked as one range (the 5.5 A cells of the short-range list hold half a warp of atoms each).  In an orthorhombic
// box a cell further from the atom than the list's radius is left out: of the 27 cells of edge r, 20.6 remain on average.  The count
// leaves the warps' votes in `masks` (optional, mask_stride words per row), and the fill takes them instead of testing every candidate
// a second time; a row that needs more words is tested again.
template <bool FILL>
__device__ __forceinline__ void build_row(const Cell& cell, const Grid& G, int n, const float* __restrict__ R, float r_list, float r2max, int ordered,
                                          const int* __restrict__ seg, const float4* __restrict__ pos_sorted, const int* __restrict__ cell_start,
                                          int* __restrict__ row_count, const int* __restrict__ row_ptr, int* __restrict__ nbr_j,
                                          int* __restrict__ edge_i, long long capacity, unsigned* __restrict__ masks, int mask_stride) {
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= n) return;
  const float xi = R[3 * (size_t)i], yi = R[3 * (size_t)i + 1], zi = R[3 * (size_t)i + 2];
  const int segi = seg ? seg[i] : 0;
  int ci[3];
  cell_coords(cell, G, xi, yi, zi, ci);
  // squared distances from the atom to the neighbouring cells along each axis (lower bounds; 0 where they are not known)
  float gap2[3][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  const bool prune = cell.periodic && cell.ortho;
  if (prune) {
    const float x[3] = {xi, yi, zi};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (G.nc[k] < 3) continue;
      float s = x[k] * cell.hinv[4 * k];
      s -= floorf(s);
      const float t = s * G.nc[k] - (float)ci[k], w = fabsf(cell.h[4 * k]) / (float)G.nc[k];      // position inside the cell, its width
      const float margin = 1e-5f * fabsf(cell.h[4 * k]) + 1e-6f * fabsf(x[k]) + 1e-3f;                                   // roundings of positions and cells
      const float below = fmaxf(t * w - margin, 0.f), above = fmaxf((1.f - t) * w - margin, 0.f);
      gap2[k][0] = below * below; gap2[k][2] = above * above;
    }
  }
  const float reach2 = r_list * r_list;
  long long base = FILL ? row_ptr[i] : 0;
  int count = 0, word = 0;
  unsigned* mine = masks ? masks + (size_t)i * mask_stride : nullptr;
  auto range = [&](int s0, int s1) {
    for (int k0 = s0; k0 < s1; k0 += 32, ++word) {
      const int k = k0 + lane;
      unsigned m;
      int j = -1;
      if (FILL && mine && word < mask_stride) {
        m = mine[word];
        if ((m >> lane) & 1u) j = pos_sorted ? __float_as_int(pos_sorted[k].w) : k;
      } else {
        bool hit = false;
        if (k < s1) {
          const float4 pj = pos_sorted ? pos_sorted[k] : make_float4(R[3 * (size_t)k], R[3 * (size_t)k + 1], R[3 * (size_t)k + 2], __int_as_float(k));
          j = __float_as_int(pj.w);
          float dx = pj.x - xi, dy = pj.y - yi, dz = pj.z - zi;
          min_image(cell, dx, dy, dz);
          const float dd = dist2_rn(dx, dy, dz);
          hit = dd < r2max && (ordered ? j > i : j != i) && (!seg || seg[j] == segi);
        }
        m = __ballot_sync(0xffffffffu, hit);
        if (!FILL && mine && word < mask_stride && lane == 0) mine[word] = m;
      }
      if (FILL && ((m >> lane) & 1u)) {
        long long pos = base + count + __popc(m & ((1u << lane) - 1u));
        if (pos < capacity) { nbr_j[pos] = j; edge_i[pos] = i; }
      }
      count += __popc(m);
    }
  };
  if (!pos_sorted) {      // a single cell that was not binned: all atoms, in their order
    range(0, G.n_atoms);
    if (!FILL && lane == 0) row_count[i] = count;
    return;
  }
  const int lo0 = G.nc[0] > 1 ? -1 : 0, hi0 = G.nc[0] > 1 ? 1 : 0;
  const int lo1 = G.nc[1] > 1 ? -1 : 0, hi1 = G.nc[1] > 1 ? 1 : 0;
  const int lo2 = G.nc[2] > 1 ? -1 : 0, hi2 = G.nc[2] > 1 ? 1 : 0;
  for (int d2 = lo2; d2 <= hi2; ++d2) {
    int c2 = ci[2] + d2;
    if (G.wrap[2]) c2 = (c2 + G.nc[2]) % G.nc[2]; else if (c2 < 0 || c2 >= G.nc[2]) continue;
    for (int d1 = lo1; d1 <= hi1; ++d1) {
      int c1 = ci[1] + d1;
      if (G.wrap[1]) c1 = (c1 + G.nc[1]) % G.nc[1]; else if (c1 < 0 || c1 >= G.nc[1]) continue;
      const float g12 = (d1 < 0 ? gap2[1][0] : (d1 > 0 ? gap2[1][2] : 0.f)) + (d2 < 0 ? gap2[2][0] : (d2 > 0 ? gap2[2][2] : 0.f));
      if (g12 > reach2) continue;
      const int row = (c2 * G.nc[1] + c1) * G.nc[0];
      int open0 = -1, open1 = -1;      // range under way
      for (int d0 = lo0; d0 <= hi0; ++d0) {
        int c0 = ci[0] + d0;
        if (G.wrap[0]) c0 = (c0 + G.nc[0]) % G.nc[0]; else if (c0 < 0 || c0 >= G.nc[0]) continue;
        if (d0 != 0 && g12 + (d0 < 0 ? gap2[0][0] : gap2[0][2]) > reach2) continue;
        const int s0 = cell_start[row + c0], s1 = cell_start[row + c0 + 1];
        if (s0 == open1) { open1 = s1; continue; }
        if (open1 > open0) range(open0, open1);
        open0 = s0; open1 = s1;
      }
      if (open1 > open0) range(open0, open1);
    }
  }
  if (!FILL && lane == 0) row_count[i] = count;
}

// The row kernels of the short- and the long-range list of a rebuild do not depend on each other: the second may run beside the first (see
// RowsBeside).  It then has no wait at its start, but ends no earlier than the first: what follows waits for it alone.  Only the first
// of two lets its successor start: no kernel but the second takes its place while a list is being written.
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void end_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <bool FILL>
__global__ void __launch_bounds__(256) build_rows_kernel(Cell cell, Grid G, int n, const float* __restrict__ R, float r_list, float r2max,
                                                         int ordered, const int* __restrict__ seg,
                                                         const float4* __restrict__ pos_sorted, const int* __restrict__ cell_start,
                                                         int* __restrict__ row_count, const int* __restrict__ row_ptr,
                                                         int* __restrict__ nbr_j, int* __restrict__ edge_i, long long capacity,
                                                         unsigned* __restrict__ masks, int mask_stride, TailScan tail, bool first_of_two) {
  if (first_of_two) let_next_start();
  build_row<FILL>(cell, G, n, R, r_list, r2max, ordered, seg, pos_sorted, cell_start, row_count, row_ptr, nbr_j, edge_i, capacity, masks, mask_stride);
  if (!FILL) {
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tail.check_finite && i < n && (threadIdx.x & 31) < 3) {
      // a NaN is nobody's neighbour: without this test a structure of NaNs would be one of isolated atoms, with zero forces
      if (!isfinite(R[3 * (size_t)i + (threadIdx.x & 31)])) atomicExch(tail.ticket + 1, 1);
    }
    tail_scan(tail, n, row_count);
  }
  end_after_previous();
}

// batched free-space graphs: the candidates of atom i are the atoms of its own graph
template <bool FILL>
__global__ void __launch_bounds__(256) build_rows_graph_kernel(int n, const float* __restrict__ R, float r2max, int ordered,
                                                               const int* __restrict__ seg, const int* __restrict__ graph_start,
                                                               int* __restrict__ row_count, const int* __restrict__ row_ptr,
                                                               int* __restrict__ nbr_j, int* __restrict__ edge_i, long long capacity,
                                                               TailScan tail, bool first_of_two) {
  if (first_of_two) let_next_start();
  const int lane = threadIdx.x & 31;
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i < n) {
  const float xi = R[3 * (size_t)i], yi = R[3 * (size_t)i + 1], zi = R[3 * (size_t)i + 2];
  const int g = seg[i];
  const int s0 = graph_start[g], s1 = graph_start[g + 1];
  long long base = FILL ? row_ptr[i] : 0;
  int count = 0;
  for (int k0 = s0; k0 < s1; k0 += 32) {
    const int j = k0 + lane;
    bool hit = false;
    if (j < s1) {
      float dx = R[3 * (size_t)j] - xi, dy = R[3 * (size_t)j + 1] - yi, dz = R[3 * (size_t)j + 2] - zi;
      hit = dist2_rn(dx, dy, dz) < r2max && (ordered ? j > i : j != i);
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (FILL && hit) {
      long long pos = base + count + __popc(m & ((1u << lane) - 1u));
      if (pos < capacity) { nbr_j[pos] = j; edge_i[pos] = i; }
    }
    count += __popc(m);
  }
  if (!FILL && lane == 0) row_count[i] = count;
  }
  if (!FILL) tail_scan(tail, n, row_count);
  end_after_previous();
}

// 64-bit sum of the per-row counts.  The exclusive scan that follows runs in 32 bits (CSR offsets are int): this total, not
// the scan's last element, decides whether the list fits, so a sum beyond 2^31 is seen before any offset is used.
__global__ void __launch_bounds__(256) row_total_kernel(int n, const int* __restrict__ row_count, unsigned long long* __restrict__ total) {
  __shared__ unsigned long long red[8];
  unsigned long long v = 0;
  for (int k = blockIdx.x * 256 + threadIdx.x; k < n; k += gridDim.x * 256) v += (unsigned long long)(unsigned)row_count[k];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < 8; ++w) t += red[w];
    if (t) atomicAdd(total, t);
  }
}

__global__ void finish_scan_kernel(int n, int* __restrict__ row_ptr, const long long* __restrict__ total, long long capacity, int* overflow) {
  // row_ptr[0..n-1] hold the exclusive scan already; close it with the 64-bit total (clamped: a total beyond the int range
  // is rejected on the host before any row is filled)
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    const long long t = *total;
    row_ptr[n] = t > 2147483647LL ? 2147483647 : (int)t;
    if (overflow && t > capacity) *overflow = 1;
  }
}

__global__ void clamp_rows_kernel(int n, int* __restrict__ row_ptr, long long capacity) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k <= n && (long long)row_ptr[k] > capacity) row_ptr[k] = (int)capacity;
}

__device__ __forceinline__ unsigned spread3(unsigned v) {   // 10 bits -> every third bit
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000ffu;
  v = (v | (v << 8)) & 0x0300f00fu;
  v = (v | (v << 4)) & 0x030c30c3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}
__global__ void morton_keys_kernel(Cell cell, Grid G, int n, const float* __restrict__ R, unsigned* __restrict__ key,
                                   int* __restrict__ iota) {
  int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n) return;
  int c[3];
  cell_coords(cell, G, R[3 * (size_t)a], R[3 * (size_t)a + 1], R[3 * (size_t)a + 2], c);
  key[a] = spread3((unsigned)c[0]) | (spread3((unsigned)c[1]) << 1) | (spread3((unsigned)c[2]) << 2);
  iota[a] = a;
}

// Every capacity is zero while its arrays are replaced: one that is not there after a failed allocation is asked for again.
template <typename T>
int ensure(T** p, size_t n) {
  if (*p) dev_free(*p);
  *p = nullptr;
  SO3LR_CUDA_CHECK(dev_alloc(p, n));
  return kOk;
}
// arrays of one element per atom
int ensure_atoms(NlistWorkspace* w, int n) {
  if (n <= w->n_cap) return kOk;
  w->n_cap = 0;
  int st;
  if ((st = ensure(&w->cell_of, n)) || (st = ensure(&w->cell_sorted, n)) || (st = ensure(&w->atom_sorted, n)) || (st = ensure(&w->atom_iota, n)) ||
      (st = ensure(&w->row_count, (size_t)n + 1)) || (st = ensure(&w->pos_sorted, (size_t)n)))
    return st;
  w->n_cap = n;
  return kOk;
}
template <class... P, class... A>
void launch_rows(RowsBeside beside, void (*kernel)(P...), int blocks, cudaStream_t s, A&&... args) {
  const bool first = beside == RowsBeside::kFirst;
  if (beside == RowsBeside::kSecond) launch_early(kernel, blocks, 256, 0, s, args..., first);
  else kernel<<<blocks, 256, 0, s>>>(args..., first);
  count_launch();
}
int ensure_bytes(void** p, size_t* have, size_t need) {
  if (need <= *have) return kOk;
  if (*p) dev_free(*p);
  *p = nullptr; *have = 0;
  SO3LR_CUDA_CHECK(dev_alloc_bytes(p, need));
  *have = need;
  return kOk;
}

}  // namespace

int nlist_row_total(cudaStream_t s, int n, const int* row_count_dev, long long* total_host) {
  unsigned long long* d = nullptr;
  SO3LR_CUDA_CHECK(dev_alloc(&d, 1));
  SO3LR_CUDA_CHECK(cudaMemsetAsync(d, 0, sizeof(unsigned long long), s));
  int tb = (n + 255) / 256;
  if (tb > 1024) tb = 1024;
  if (n > 0) { row_total_kernel<<<tb, 256, 0, s>>>(n, row_count_dev, d); count_launch(); }
  unsigned long long t = 0;
  cudaError_t e = cudaMemcpyAsync(&t, d, sizeof(t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  dev_free(d);
  if (e != cudaSuccess) return kCudaError;
  *total_host = (long long)t;
  return t > 2147483000ULL ? kTooLarge : kOk;
}

int spatial_order(NlistWorkspace* w, cudaStream_t s, const Cell& cell, int n, const float* R, float cell_size, int* perm) {
  if (n <= 0 || !cell.periodic) return kInvalidArgument;
  if (n > w->key_cap) {
    int st;
    w->key_cap = 0;
    if ((st = ensure(&w->key, n))) return st;
    if ((st = ensure(&w->key_sorted, n))) return st;
    w->key_cap = n;
  }
  if (int rca = ensure_atoms(w, n)) return rca;
  Grid G{};
  for (int k = 0; k < 3; ++k) {
    double nx = cell.hinv[0 + k], ny = cell.hinv[3 + k], nz = cell.hinv[6 + k];
    double width = 1.0 / std::sqrt(nx * nx + ny * ny + nz * nz);
    int nc = (int)std::floor(width / (double)cell_size);
    if (nc < 1) nc = 1;
    if (nc > 1024) nc = 1024;
    G.nc[k] = nc; G.wrap[k] = 1;
  }
  { morton_keys_kernel<<<(n + 255) / 256, 256, 0, s>>>(cell, G, n, R, w->key, w->atom_iota); count_launch(); }
  size_t need = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, need, w->key, w->key_sorted, w->atom_iota, perm, n, 0, 30, s);
  if (int rcb = ensure_bytes(&w->sort_tmp, &w->sort_bytes, need)) return rcb;
  size_t tmp = w->sort_bytes;
  cub::DeviceRadixSort::SortPairs(w->sort_tmp, tmp, w->key, w->key_sorted, w->atom_iota, perm, n, 0, 30, s);
  count_launch(6);   // histogram, prefix, four 8-bit passes
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// Free space: up to here all atoms are tested.  An evaluation of a water cluster (12 A long range, lists made new) with cells / without takes
// 262 / 226 us at 96 atoms, 320 / 262 at 384, 421 / 357 at 1,023, 849 / 758 at 3,072, 984 / 893 at 4,095, 1,482 / 1,566 at 8,193: finding the
// cells costs the read-back of all positions.  The line lies below the crossing: the tests grow with the square of the atoms.
constexpr int kOneCellAtoms = 1024;

bool nlist_counts_in_one_kernel(int n) { return n <= kTailScanRows; }
// `beside` kSecond: the kernel enqueued last is another list's count (or, in nlist_end, fill), launched as kFirst, beside which this one's may
// run.  Short lists are bound by latency: the four row kernels of 1,536 atoms take 23, 26, 16 and 13 us one behind the other, the last
// CTA's scan of each among them.
int nlist_begin(NlistWorkspace* w, cudaStream_t s, const Cell& cell, int n, const float* R, float r_list, int ordered,
                const int* seg, const int* graph_start, NeighborListDev* out, int allow_grow, int* d_overflow, int n_rows, bool any_order,
                RowsBeside beside) {
  w->n_rows = 0;
  if (n <= 0) { out->count = 0; return kOk; }
  if (n_rows < 0 || n_rows > n) n_rows = n;
  // work of this list's own comes in between
  auto not_second = [&] { if (beside == RowsBeside::kSecond) beside = RowsBeside::kNo; };
  if (int rca = ensure_atoms(w, n)) return rca;
  if (!w->ticket) {
    SO3LR_CUDA_CHECK(dev_alloc(&w->ticket, 2));
    SO3LR_CUDA_CHECK(cudaMemsetAsync(w->ticket, 0, 2 * sizeof(int), s));
    not_second();
  }
  if (!w->d_total) SO3LR_CUDA_CHECK(dev_alloc(&w->d_total, 1));
  if (!w->h_total) SO3LR_CUDA_CHECK(host_alloc(&w->h_total, 1));
  if (n + 1 > out->row_cap) {
    if (out->row_ptr) dev_free(out->row_ptr);
    out->row_ptr = nullptr; out->row_cap = 0;
    SO3LR_CUDA_CHECK(dev_alloc(&out->row_ptr, ((size_t)n + 1)));
    out->row_cap = n + 1;
  }
  const float r2max = r_list * r_list;
  const bool by_graph = graph_start != nullptr && !cell.periodic;
  Grid G{};
  G.n_atoms = n;
  bool binned = false;
  int n_cells = 1;
  if (!by_graph) {
    if (cell.periodic) {
      // perpendicular widths of the cell: 1 / |column k of hinv|
      for (int k = 0; k < 3; ++k) {
        double nx = cell.hinv[0 + k], ny = cell.hinv[3 + k], nz = cell.hinv[6 + k];
        double width = 1.0 / std::sqrt(nx * nx + ny * ny + nz * nz);
        int nc = (int)std::floor(width / (double)r_list);
        if (nc < 3) nc = 1;          // fewer than 3 cells: one cell, minimum-image handles the rest
        if (nc > 1024) nc = 1024;
        G.nc[k] = nc; G.wrap[k] = 1;
      }
    } else if (any_order && n <= kOneCellAtoms) {
      // the entries of a row may come in any order: all atoms are candidates, without the bounding box (a read-back) and the cells
      for (int k = 0; k < 3; ++k) G.nc[k] = 1;
    } else {
      // bounding box on the host side would need a reduction; use a coarse device-free approach: the caller
      // passes free-space systems of moderate size, so read the positions back once per build.
      not_second();
      std::vector<float> h((size_t)n * 3);
      SO3LR_CUDA_CHECK(cudaMemcpyAsync(h.data(), R, h.size() * sizeof(float), cudaMemcpyDeviceToHost, s));
      SO3LR_CUDA_CHECK(cudaStreamSynchronize(s));
      float lo[3] = {1e30f, 1e30f, 1e30f}, hi[3] = {-1e30f, -1e30f, -1e30f};
      for (int a = 0; a < n; ++a)
        for (int k = 0; k < 3; ++k) { float v = h[3 * (size_t)a + k]; lo[k] = v < lo[k] ? v : lo[k]; hi[k] = v > hi[k] ? v : hi[k]; }
      for (int k = 0; k < 3; ++k) {
        float ext = hi[k] - lo[k];
        if (!(ext >= 0.f) || !std::isfinite(ext)) return kNotFinite;
        int nc = (int)std::floor(ext / r_list);
        if (nc < 1) nc = 1;
        if (nc > 512) nc = 512;
        G.nc[k] = nc; G.wrap[k] = 0; G.lo[k] = lo[k];
        G.inv_w[k] = nc / (ext > 0.f ? ext * 1.000001f : 1.f);
      }
    }
    n_cells = G.nc[0] * G.nc[1] * G.nc[2];
    binned = n_cells > 1;      // the atoms of a single cell come in their own order either way
    if (binned) {
      not_second();
      if (n_cells + 1 > w->cell_cap) {
        w->cell_cap = 0;
        if (int rcc = ensure(&w->cell_start, (size_t)n_cells + 1)) return rcc;
        w->cell_cap = n_cells + 1;
      }
      { assign_cells_kernel<<<(n + 255) / 256, 256, 0, s>>>(cell, G, n, R, w->cell_of, w->atom_iota); count_launch(); }
      int bits = 1;
      while ((1 << bits) < n_cells && bits < 31) ++bits;
      size_t need = 0;
      cub::DeviceRadixSort::SortPairs(nullptr, need, w->cell_of, w->cell_sorted, w->atom_iota, w->atom_sorted, n, 0, bits, s);
      size_t need2 = 0;
      cub::DeviceScan::ExclusiveSum(nullptr, need2, w->row_count, out->row_ptr, n, s);   // sized for the largest row count
      if (need2 > need) need = need2;
      if (int rcb = ensure_bytes(&w->cub_tmp, &w->cub_bytes, need)) return rcb;
      size_t tmp = w->cub_bytes;
      cub::DeviceRadixSort::SortPairs(w->cub_tmp, tmp, w->cell_of, w->cell_sorted, w->atom_iota, w->atom_sorted, n, 0, bits, s);
      count_launch(2 + (bits + 7) / 8);
      { cell_bounds_kernel<<<(n + 1 + 255) / 256, 256, 0, s>>>(n, n_cells, w->cell_sorted, w->cell_start); count_launch(); }
      { gather_sorted_positions_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, R, w->atom_sorted, w->pos_sorted); count_launch(); }
    }
  }
  if (!binned) {
    size_t need = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, need, w->row_count, out->row_ptr, n, s);
    if (int rcb = ensure_bytes(&w->cub_tmp, &w->cub_bytes, need)) return rcb;
  }
  const int blocks = (n_rows + 7) / 8;
  if (n_rows == 0) { out->count = 0; return kOk; }
  // votes of the count for the fill: room for 1.25 times the candidates of 27 cells (an atom in the middle of its cell has all of them
  // within the radius, also where cells are left out) and one partial word per range; for the 13 A list of water (12 A and the skin)
  // 269 words, 1.1 KB per atom.  Short of memory they are given back (see nlist_end) and the fill tests the candidates again.
  unsigned* masks = nullptr;
  int mask_stride = 0;
  if (!by_graph) {
    double cells = 1.0;
    for (int k = 0; k < 3; ++k) cells *= G.nc[k] > 1 ? 3.0 : 1.0;
    const double mean = cells * (double)n / (double)n_cells;
    mask_stride = (int)std::min(mean * 1.25 / 32.0 + 12.0, 1024.0);
    const size_t words = (size_t)n_rows * mask_stride;
    if (words > w->mask_cap) {
      if (w->masks) dev_free(w->masks);
      w->masks = nullptr; w->mask_cap = 0;
      if (dev_alloc(&w->masks, words) == cudaSuccess) w->mask_cap = words;
      else { w->masks = nullptr; cudaGetLastError(); }
    }
    masks = w->masks;
  }
  TailScan tail;
  if (n_rows <= kTailScanRows && allow_grow) { tail.ticket = w->ticket; tail.row_ptr = out->row_ptr; tail.total_host = w->h_total; }
  tail.check_finite = tail.ticket && !by_graph && !cell.periodic && !binned;      // in place of the bounding box's test of the extent
  if (by_graph)
    launch_rows(beside, build_rows_graph_kernel<false>, blocks, s, n_rows, R, r2max, ordered, seg, graph_start, w->row_count, nullptr, nullptr, nullptr, 0, tail);
  else
    launch_rows(beside, build_rows_kernel<false>, blocks, s, cell, G, n_rows, R, r_list, r2max, ordered, seg, binned ? w->pos_sorted : nullptr,
                w->cell_start, w->row_count, nullptr, nullptr, nullptr, 0, masks, mask_stride, tail);
  if (!tail.ticket) {
    SO3LR_CUDA_CHECK(cudaMemsetAsync(w->d_total, 0, sizeof(long long), s));
    { int tb = (n_rows + 255) / 256; if (tb > 1024) tb = 1024;
      row_total_kernel<<<tb, 256, 0, s>>>(n_rows, w->row_count, reinterpret_cast<unsigned long long*>(w->d_total)); count_launch(); }
    size_t tmp = w->cub_bytes;
    cub::DeviceScan::ExclusiveSum(w->cub_tmp, tmp, w->row_count, out->row_ptr, n_rows, s);
    count_launch(2);
    { finish_scan_kernel<<<1, 32, 0, s>>>(n_rows, out->row_ptr, w->d_total, out->capacity, allow_grow ? nullptr : d_overflow); count_launch(); }
    SO3LR_CUDA_CHECK(cudaMemcpyAsync(w->h_total, w->d_total, sizeof(long long), cudaMemcpyDeviceToHost, s));
  }
  w->G = G; w->n = n; w->n_rows = n_rows; w->ordered = ordered; w->allow_grow = allow_grow; w->mask_stride = mask_stride;
  w->by_graph = by_graph; w->binned = binned; w->r_list = r_list; w->R = R; w->seg = seg; w->graph_start = graph_start;
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

// the second half, once the stream has been waited for
int nlist_end(NlistWorkspace* w, cudaStream_t s, const Cell& cell, NeighborListDev* out, RowsBeside beside) {
  const int n_rows = w->n_rows;
  if (n_rows <= 0) return kOk;
  const int blocks = (n_rows + 7) / 8, allow_grow = w->allow_grow;
  const float r2max = w->r_list * w->r_list;
  const long long total = *w->h_total;
  if (total < 0) return kNotFinite;
  if (total > 2147483000LL) return kTooLarge;
  if (total > out->capacity) {
    if (!allow_grow) {
      out->count = out->capacity;   // rows are truncated; the overflow flag is set on the device
    } else {
      long long cap = total + total / 4 + 1024;
      if (out->nbr_j) dev_free(out->nbr_j);
      if (out->edge_i) dev_free(out->edge_i);
      out->nbr_j = nullptr; out->edge_i = nullptr; out->capacity = 0; out->count = 0;
      // the list itself goes before the votes
      for (int** p : {&out->nbr_j, &out->edge_i})
        if (dev_alloc(p, (size_t)cap) != cudaSuccess) {
          if (!nlist_drop_votes(w)) return kCudaError;
          SO3LR_CUDA_CHECK(dev_alloc(p, (size_t)cap));
        }
      out->capacity = cap;
    }
  }
  w->n_rows = 0;      // not before: a call that found no memory may be repeated
  if (total <= out->capacity) out->count = total;
  const bool truncated = total > out->capacity;
  if (w->by_graph)
    launch_rows(beside, build_rows_graph_kernel<true>, blocks, s, n_rows, w->R, r2max, w->ordered, w->seg, w->graph_start, nullptr, out->row_ptr,
                out->nbr_j, out->edge_i, out->capacity, TailScan{});
  else
    launch_rows(beside, build_rows_kernel<true>, blocks, s, cell, w->G, n_rows, w->R, w->r_list, r2max, w->ordered, w->seg,
                w->binned ? w->pos_sorted : nullptr, w->cell_start, nullptr, out->row_ptr, out->nbr_j, out->edge_i, out->capacity, w->masks,
                w->mask_stride, TailScan{});
  if (truncated) { clamp_rows_kernel<<<(n_rows + 1 + 255) / 256, 256, 0, s>>>(n_rows, out->row_ptr, out->capacity); count_launch(); }
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return truncated ? kOverflow : kOk;
}

int nlist_build(NlistWorkspace* w, cudaStream_t s, const Cell& cell, int n, const float* R, float r_list, int ordered,
                const int* seg, const int* graph_start, NeighborListDev* out, int allow_grow, int* d_overflow, int n_rows) {
  int rc = nlist_begin(w, s, cell, n, R, r_list, ordered, seg, graph_start, out, allow_grow, d_overflow, n_rows, false);
  if (rc) return rc;
  SO3LR_CUDA_CHECK(cudaStreamSynchronize(s));
  return nlist_end(w, s, cell, out);
}

}  // namespace so3lr
