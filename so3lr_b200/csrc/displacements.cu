// Pair displacements of caller-supplied lists and their transpose: what a caller of the graph-level evaluation does around it.
//
//   forward : d_e = R[j_e] - R[i_e], minimum image                      (so3lr/jaxmd_utils.py:57-66)
//   reverse : dE/dR[j_e] += g_e, dE/dR[i_e] -= g_e                      (the transpose of the two gathers under jax.grad)
//
// Both are bound by memory: the forward pass reads 8 and writes 12 bytes per entry, the reverse pass reads 20.  The list is walked
// once, coalesced; the atoms' rows (12-24 bytes each) stay in the L2.  A framework's generic index backward serialises on equal
// indices -- the padding of a list, a quarter of it, points at one atom -- and took 54 ms per call at 1,536 atoms (0.8 M entries)
// and 965 ms at 24,000 (12 M): the whole step 56.3 and 1,048 ms.  Here entries with a zero gradient are skipped, the receiver's
// share is summed over runs of equal indices inside a warp (lists come grouped by receiver) and every other share is one 16-byte
// vector reduction: the step takes 1.5 and 5.0 ms.
#include <algorithm>

#include "kernels.h"

namespace so3lr {

namespace {

template <typename T>
struct Lattice {
  T h[9], hi[9];
};
// rows of `cell` are the lattice vectors; the inverse is formed in double by one thread per CTA (no host copy of a device cell)
template <typename T>
__device__ void load_lattice(const T* __restrict__ cell, Lattice<T>& L) {
  if (threadIdx.x == 0) {
    double h[9];
    for (int k = 0; k < 9; ++k) { L.h[k] = cell[k]; h[k] = (double)cell[k]; }
    const double c0 = h[4] * h[8] - h[5] * h[7], c1 = h[5] * h[6] - h[3] * h[8], c2 = h[3] * h[7] - h[4] * h[6];
    const double id = 1.0 / (h[0] * c0 + h[1] * c1 + h[2] * c2);
    L.hi[0] = (T)(c0 * id); L.hi[1] = (T)((h[2] * h[7] - h[1] * h[8]) * id); L.hi[2] = (T)((h[1] * h[5] - h[2] * h[4]) * id);
    L.hi[3] = (T)(c1 * id); L.hi[4] = (T)((h[0] * h[8] - h[2] * h[6]) * id); L.hi[5] = (T)((h[2] * h[3] - h[0] * h[5]) * id);
    L.hi[6] = (T)(c2 * id); L.hi[7] = (T)((h[1] * h[6] - h[0] * h[7]) * id); L.hi[8] = (T)((h[0] * h[4] - h[1] * h[3]) * id);
  }
  __syncthreads();
}

// padding entries carry index n: like a clamped gather they read the last atom, so both ends coincide and d = 0; a negative index
// counts from the end
__device__ __forceinline__ int clamp_index(int k, int n) { return min(max(k < 0 ? k + n : k, 0), n - 1); }

template <typename T, typename O>
__global__ void __launch_bounds__(256) displacement_kernel(int n, const T* __restrict__ R, const T* __restrict__ cell, long long n_entries,
                                                           const int* __restrict__ idx_i, const int* __restrict__ idx_j, O* __restrict__ out) {
  __shared__ Lattice<T> L;
  if (cell) load_lattice(cell, L);
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < n_entries; e += (long long)gridDim.x * 256) {
    const int i = clamp_index(idx_i[e], n), j = clamp_index(idx_j[e], n);
    T d[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) d[c] = R[3 * (size_t)j + c] - R[3 * (size_t)i + c];
    if (cell) {
      T k[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) k[c] = rint(d[0] * L.hi[c] + d[1] * L.hi[3 + c] + d[2] * L.hi[6 + c]);
#pragma unroll
      for (int c = 0; c < 3; ++c) d[c] -= k[0] * L.h[c] + k[1] * L.h[3 + c] + k[2] * L.h[6 + c];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) out[3 * (size_t)e + c] = (O)d[c];
  }
}

__device__ __forceinline__ void add3(float* p, float x, float y, float z) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(x), "f"(y), "f"(z), "f"(0.f) : "memory");
}
__device__ __forceinline__ void add3(double* p, double x, double y, double z) {
  atomicAdd(p, x); atomicAdd(p + 1, y); atomicAdd(p + 2, z);
}

// acc: four values per atom (x, y, z, unused), so that a share is one aligned vector reduction
template <typename T, typename G>
__global__ void __launch_bounds__(256) displacement_vjp_kernel(int n, long long n_entries, const int* __restrict__ idx_i,
                                                               const int* __restrict__ idx_j, const G* __restrict__ g, T sign, T* __restrict__ acc) {
  const int lane = threadIdx.x & 31;
  const long long step = (long long)gridDim.x * 256;
  for (long long e0 = (long long)blockIdx.x * 256 + (threadIdx.x & ~31); e0 < n_entries; e0 += step) {
    const long long e = e0 + lane;
    int i = -1;
    T x = 0, y = 0, z = 0;
    if (e < n_entries) {
      i = clamp_index(idx_i[e], n);
      x = sign * (T)g[3 * (size_t)e]; y = sign * (T)g[3 * (size_t)e + 1]; z = sign * (T)g[3 * (size_t)e + 2];
    }
    bool any = x != (T)0 || y != (T)0 || z != (T)0;
    if (any) {
      const int j = clamp_index(idx_j[e], n);
      if (j != i) add3(acc + 4 * (size_t)j, x, y, z);
      else { x = 0; y = 0; z = 0; any = false; }         // both shares fall on one atom and cancel
    }
    if (!__ballot_sync(0xffffffffu, any)) continue;
    // sum over the run of equal receivers that ends at this lane (`head` = first lane of the run); the last lane of a run adds it
    const int iprev = __shfl_up_sync(0xffffffffu, i, 1);
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || iprev != i);
    const int head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T tx = __shfl_up_sync(0xffffffffu, x, o), ty = __shfl_up_sync(0xffffffffu, y, o), tz = __shfl_up_sync(0xffffffffu, z, o);
      if (lane - o >= head) { x += tx; y += ty; z += tz; }
    }
    const int inext = __shfl_down_sync(0xffffffffu, i, 1);
    if (i >= 0 && (lane == 31 || inext != i) && (x != (T)0 || y != (T)0 || z != (T)0)) add3(acc + 4 * (size_t)i, -x, -y, -z);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) take3_kernel(int n, const T* __restrict__ acc, T* __restrict__ out) {
  const int k = blockIdx.x * 256 + threadIdx.x;
  if (k < 3 * n) out[k] = acc[4 * (size_t)(k / 3) + k % 3];
}

// flags[0], flags[1]: set when the list is not grouped by ascending receiver
__global__ void __launch_bounds__(256) unsorted_kernel(long long n0, const int* __restrict__ i0, long long n1, const int* __restrict__ i1,
                                                       int* __restrict__ flags) {
  const long long total = n0 + n1;
  for (long long t = (long long)blockIdx.x * 256 + threadIdx.x; t < total; t += (long long)gridDim.x * 256) {
    const bool first = t < n0;
    const long long e = first ? t : t - n0;
    const int* p = first ? i0 : i1;
    if (e > 0 && p[e] < p[e - 1]) flags[first ? 0 : 1] = 1;
  }
}

unsigned grid_for(long long entries) {      // eight CTAs of 256 per SM fill the memory pipe; more only add launch work
  return (unsigned)std::max<long long>(1, std::min<long long>((entries + 255) / 256, (long long)sm_count() * 8));
}

}  // namespace

int displacements(cudaStream_t s, bool dbl, int n, const void* R, const void* cell, long long n_entries, const int* idx_i, const int* idx_j,
                  void* out, bool out_dbl) {
  if (n_entries == 0) return kOk;
  const unsigned blocks = grid_for(n_entries);
  if (!dbl && !out_dbl) displacement_kernel<float, float><<<blocks, 256, 0, s>>>(n, (const float*)R, (const float*)cell, n_entries, idx_i, idx_j, (float*)out);
  else if (dbl && !out_dbl) displacement_kernel<double, float><<<blocks, 256, 0, s>>>(n, (const double*)R, (const double*)cell, n_entries, idx_i, idx_j, (float*)out);
  else if (dbl) displacement_kernel<double, double><<<blocks, 256, 0, s>>>(n, (const double*)R, (const double*)cell, n_entries, idx_i, idx_j, (double*)out);
  else return kInvalidArgument;
  count_launch();
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

int displacements_vjp(cudaStream_t s, bool dbl, int n, long long n_entries, const int* idx_i, const int* idx_j, const void* g, bool g_dbl,
                      double sign, void* acc4, bool clear, void* out) {
  if (clear) SO3LR_CUDA_CHECK(cudaMemsetAsync(acc4, 0, (size_t)n * 4 * (dbl ? sizeof(double) : sizeof(float)), s));
  if (n_entries > 0) {
    const unsigned blocks = grid_for(n_entries);
    if (!dbl && !g_dbl) displacement_vjp_kernel<float, float><<<blocks, 256, 0, s>>>(n, n_entries, idx_i, idx_j, (const float*)g, (float)sign, (float*)acc4);
    else if (dbl && !g_dbl) displacement_vjp_kernel<double, float><<<blocks, 256, 0, s>>>(n, n_entries, idx_i, idx_j, (const float*)g, sign, (double*)acc4);
    else if (dbl) displacement_vjp_kernel<double, double><<<blocks, 256, 0, s>>>(n, n_entries, idx_i, idx_j, (const double*)g, sign, (double*)acc4);
    else return kInvalidArgument;
    count_launch();
  }
  if (out) {
    const unsigned blocks = (unsigned)((3LL * n + 255) / 256);
    if (dbl) take3_kernel<double><<<blocks, 256, 0, s>>>(n, (const double*)acc4, (double*)out);
    else take3_kernel<float><<<blocks, 256, 0, s>>>(n, (const float*)acc4, (float*)out);
    count_launch();
  }
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

int lists_unsorted(cudaStream_t s, long long n0, const int* i0, long long n1, const int* i1, int* flags2) {
  SO3LR_CUDA_CHECK(cudaMemsetAsync(flags2, 0, 2 * sizeof(int), s));
  if (n0 + n1 > 0) { unsorted_kernel<<<grid_for(n0 + n1), 256, 0, s>>>(n0, i0, n1, i1, flags2); count_launch(); }
  SO3LR_CUDA_CHECK(cudaGetLastError());
  return kOk;
}

}  // namespace so3lr
