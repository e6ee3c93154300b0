// Pieces of the multi-vector kernels (Krylov solvers).
#pragma once

#include <cstddef>
#include <cstdint>

namespace qcmg {

// Vector lists and coefficients passed to the kernels by value (up to
// kByValue entries): no host-to-device copy of a pointer array per call,
// which on small sectors costs more than the kernel.  Longer lists go
// through device arrays (the same kernels, instantiated on pointers).
constexpr int kByValue = 64;
struct VecList {
  const double* v[kByValue];
  __device__ const double* operator[](int k) const { return v[k]; }
};
struct MutVecList {
  double* v[kByValue];
  __device__ double* operator[](int k) const { return v[k]; }
};
struct CoefList {
  double c[kByValue];
  __device__ double operator[](int k) const { return c[k]; }
};

// Sums each of the V values of the 32 lanes; afterwards lane l holds the sum
// of value l / (32 / V): V - 1 additions and a few more, where a butterfly
// per value takes five each.
template <int V>
__device__ __forceinline__ double lane_sums(double (&a)[V], int lane) {
  int o = 16;
#pragma unroll
  for (int n = V; n > 1; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const double give = up ? a[i] : a[i + n / 2], keep = up ? a[i + n / 2] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  double s = a[0];
  for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// VEC consecutive doubles (16-byte loads for VEC = 2).
template <int VEC>
struct Pack {
  double e[VEC];
};
template <int VEC>
__device__ __forceinline__ Pack<VEC> load_pack(const double* p, size_t i) {
  Pack<VEC> r;
  if constexpr (VEC == 2) {
    const double2 t = reinterpret_cast<const double2*>(p)[i];
    r.e[0] = t.x;
    r.e[1] = t.y;
  } else {
    r.e[0] = p[i];
  }
  return r;
}
template <int VEC>
__device__ __forceinline__ void store_pack(double* p, size_t i, const Pack<VEC>& v) {
  if constexpr (VEC == 2)
    reinterpret_cast<double2*>(p)[i] = make_double2(v.e[0], v.e[1]);
  else
    p[i] = v.e[0];
}

constexpr int kDotThreads = 256;

// Block sums of up to MAXM accumulators per thread into part[k], k < m.
template <int MAXM>
__device__ __forceinline__ void block_sums(double (&acc)[MAXM], int m, double* part) {
  constexpr int V = MAXM <= 1 ? 1 : MAXM <= 2 ? 2 : MAXM <= 4 ? 4 : MAXM <= 8 ? 8 : MAXM <= 16 ? 16 : 32;
  __shared__ double red[kDotThreads / 32][V];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  double a[V];
#pragma unroll
  for (int k = 0; k < V; ++k) a[k] = k < MAXM ? acc[k] : 0.0;
  const double s = lane_sums<V>(a, lane);
  if (lane % (32 / V) == 0) red[wp][lane / (32 / V)] = s;
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += blockDim.x) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < kDotThreads / 32; ++q) t += red[q][k];
    part[k] = t;
  }
}

}  // namespace qcmg
