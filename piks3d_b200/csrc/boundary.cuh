// Plane kernels of an iteration (x ghosts, inlet / outlet, symmetry), FP64 or FP32 storage.
//
// What bounds them: memory round trips; each moves tens of MB. A thread takes one 16-byte piece of
// all four octants' rows at both ends of the box, so that eight loads are in flight per thread and the
// row lookup is done once (k_symmetry: of a node's eight rows, four loads for each plane that the
// node lies on). Per iteration on a 128^3 pack of 512 velocities, a thread per
// value / this: capture FP64 0.037 / 0.024, FP32 0.033 / 0.015; inlet and outlet 0.037 / 0.024, 0.033 /
// 0.015; symmetry 0.054 / 0.040, 0.046 / 0.025 ms (some 5 us of each are the launch).
#pragma once
#include <cuda_runtime.h>

#include "kernels.h"

namespace piks {
namespace boundary {

// (Nc8 is a multiple of 8: rows are whole pieces)
template <typename T>
struct alignas(16) Piece {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
};
template <typename T> __device__ __forceinline__ Piece<T> load(const T *p) { return *reinterpret_cast<const Piece<T> *>(p); }
template <typename T> __device__ __forceinline__ void store(T *p, const Piece<T> &x) { *reinterpret_cast<Piece<T> *>(p) = x; }

// octants with cx > 0 and with cx < 0 in the order of a ghost plane's rows
__device__ __forceinline__ int plus_x(int q) { return q == 0 ? 0 : q == 1 ? 3 : q == 2 ? 4 : 7; }
__device__ __forceinline__ int minus_x(int q) { return q == 0 ? 1 : q == 1 ? 2 : q == 2 ? 5 : 6; }

// Periodic x halo (solver.F90:535-560, one rank): the planes x = Nx (octants with cx > 0)
// and x = 1 (cx < 0) as they stand after the sweep become the ghost planes x = 0 and
// x = Nx+1 that the boundary conditions of the NEXT iteration read.
template <typename T>
__global__ void __launch_bounds__(256) k_capture(const T *h, T *ghostW, T *ghostE, const int32_t *plane_x1,
                                                 const int32_t *plane_xN, size_t rows, int Nc8) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int pieces = Nc8 / Piece<T>::N;
  const size_t r = idx / pieces;
  if (r >= rows) return;
  const int l = (int)(idx - r * pieces) * Piece<T>::N;
  const int nW = plane_xN[r], nE = plane_x1[r];
  Piece<T> w[4], e[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    w[q] = e[q] = Piece<T>{};
    if (nW >= 0) w[q] = load(h + ((size_t)nW * 8 + plus_x(q)) * Nc8 + l);
    if (nE >= 0) e[q] = load(h + ((size_t)nE * 8 + minus_x(q)) * Nc8 + l);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    store(ghostW + (r * 4 + q) * Nc8 + l, w[q]);
    store(ghostE + (r * 4 + q) * Nc8 + l, e[q]);
  }
}

// Inlet x = 1 and outlet x = Nx with the pressure jump (solver.F90:1832-1862), reading the
// ghost planes captured in the previous iteration.
template <typename T>
__global__ void __launch_bounds__(256) k_inlet_outlet(T *h, const T *ghostW, const T *ghostE, const int32_t *plane_x1,
                                                      const int32_t *plane_xN, const double *weight, double pressDrop,
                                                      size_t rows, int Nc8) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int pieces = Nc8 / Piece<T>::N;
  const size_t r = idx / pieces;
  if (r >= rows) return;
  const int l = (int)(idx - r * pieces) * Piece<T>::N;
  const int n1 = plane_x1[r], nN = plane_xN[r];
  Piece<T> w[4], e[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (n1 >= 0) w[q] = load(ghostW + (r * 4 + q) * Nc8 + l);
    if (nN >= 0) e[q] = load(ghostE + (r * 4 + q) * Nc8 + l);
  }
  T jump[Piece<T>::N];
#pragma unroll
  for (int v = 0; v < Piece<T>::N; ++v) jump[v] = (T)__dmul_rn(weight[l + v], pressDrop);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int v = 0; v < Piece<T>::N; ++v) { w[q].v[v] = w[q].v[v] + jump[v]; e[q].v[v] = e[q].v[v] - jump[v]; }
    if (n1 >= 0) store(h + ((size_t)n1 * 8 + plus_x(q)) * Nc8 + l, w[q]);
    if (nN >= 0) store(h + ((size_t)nN * 8 + minus_x(q)) * Nc8 + l, e[q]);
  }
}

// Specular symmetry planes y = 1, y = Ny, z = 1, z = Nz in the reference's order
// (solver.F90:1867-1918): four rows of the node are read and four written per plane, so that a node
// on an edge of the box sees the first plane's rows in the second.
template <typename T>
__global__ void __launch_bounds__(256) k_symmetry(T *h, const int32_t *node, const uint8_t *flag, size_t n, int Nc8) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int pieces = Nc8 / Piece<T>::N;
  const size_t s = idx / pieces;
  if (s >= n) return;
  const uint8_t f = flag[s];
  T *hp = h + (size_t)node[s] * 8 * Nc8 + (idx - s * pieces) * Piece<T>::N;
  // one plane: four rows are read and four written
  auto plane = [&](int a0, int b0, int a1, int b1, int a2, int b2, int a3, int b3) {
    const Piece<T> x0 = load(hp + (size_t)b0 * Nc8), x1 = load(hp + (size_t)b1 * Nc8), x2 = load(hp + (size_t)b2 * Nc8),
                   x3 = load(hp + (size_t)b3 * Nc8);
    store(hp + (size_t)a0 * Nc8, x0);
    store(hp + (size_t)a1 * Nc8, x1);
    store(hp + (size_t)a2 * Nc8, x2);
    store(hp + (size_t)a3 * Nc8, x3);
  };
  if (f & 1) plane(1, 2, 0, 3, 5, 6, 4, 7);
  if (f & 2) plane(2, 1, 3, 0, 6, 5, 7, 4);
  if (f & 4) plane(0, 4, 1, 5, 2, 6, 3, 7);
  if (f & 8) plane(4, 0, 5, 1, 6, 2, 7, 3);
}

template <typename T>
inline void launch_capture(const T *h, T *ghostW, T *ghostE, const DevState &s, cudaStream_t st) {
  const size_t rows = (size_t)s.Ny * s.Nz, threads = rows * (s.Nc8 / Piece<T>::N);
  k_capture<T><<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(h, ghostW, ghostE, s.plane_x1, s.plane_xN, rows, s.Nc8);
}
template <typename T>
inline void launch_inlet_outlet(T *h, const T *ghostW, const T *ghostE, const DevState &s, cudaStream_t st) {
  const size_t rows = (size_t)s.Ny * s.Nz, threads = rows * (s.Nc8 / Piece<T>::N);
  k_inlet_outlet<T><<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(h, ghostW, ghostE, s.plane_x1, s.plane_xN, s.w,
                                                                       s.pressDrop, rows, s.Nc8);
}
template <typename T>
inline void launch_symmetry(T *h, const DevState &s, cudaStream_t st) {
  if (!s.nsym) return;
  const size_t threads = (size_t)s.nsym * (s.Nc8 / Piece<T>::N);
  k_symmetry<T><<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(h, s.sym_node, s.sym_flag, (size_t)s.nsym, s.Nc8);
}

}  // namespace boundary
}  // namespace piks
