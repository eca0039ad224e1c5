// FP32 path of the source iteration: the distribution function, the wall slots, the
// 3-fold corner storage and the ghost planes are stored and swept in FP32; the moments
// (Rho, U), the diffuse-wall densities, the mass flux and the convergence test stay FP64
// (the moments and the flux reuse the FP64 arrays of DevState). The data flow is the one
// of kernels.cu (same tasks, roles, commits, wall programs and boundary order); only the
// arithmetic type differs, so the FP32 iterate approximates the FP64 one.
#include <cuda_runtime.h>

#include "boundary.cuh"
#include "kernels.h"
#include "piks_internal.h"

namespace piks {

namespace {

__constant__ WProg c32_prog[26];
__constant__ WPlan c32_plan[26];
bool g32_plan_ok = false;  // every program resolved (make_wall_plan)
__constant__ int8_t c32_prog_of[128];
__constant__ int c32_incoming[6][4];

__device__ __forceinline__ size_t hidx(int node, int o, int Nc8, int l) {
  return ((size_t)node * 8 + o) * (size_t)Nc8 + l;
}
__device__ __forceinline__ int plane_slot(int o) { return o >> 1; }
constexpr int kFwBit = 1 << 30;
__device__ __forceinline__ void cp_async16_cg(void *smem, const void *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int VPL>
__device__ __forceinline__ void ld32(const float *p, float (&v)[VPL]) {
  if constexpr (VPL == 4) {
    const float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else if constexpr (VPL == 2) {
    const float2 t = __ldcg(reinterpret_cast<const float2 *>(p));
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = __ldcg(p);
  }
}
template <int VPL>
__device__ __forceinline__ void st32(float *p, const float (&v)[VPL]) {
  if constexpr (VPL == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if constexpr (VPL == 2) *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
  else p[0] = v[0];
}

// Hyperplane sweep task (same task records as the FP64 kernel); upwind rows from h32/fw32.
template <int LPT, int VPL>
__global__ void __launch_bounds__(256)
k_sweep32(const DevState a, long t0, long ntask) {
  const long gl = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long slot = gl / LPT;
  const int sub = (int)(gl % LPT);
  const long ti = slot / a.nchunk;
  const int chunk = (int)(slot - ti * a.nchunk);
  if (ti >= ntask) return;
  const int Nc8 = a.Nc8;
  const int lfirst = chunk * LPT * VPL + sub * VPL;
  if (lfirst >= Nc8) return;
  const int4 *rec = reinterpret_cast<const int4 *>(a.tasks + (size_t)(t0 + ti) * 8);
  const int4 r0 = __ldg(rec), r1 = __ldg(rec + 1);
  const int m = r0.x, fl = r0.y;
  const int o = fl & 7;
  const bool fx = fl & 8, fy = fl & 16, fz = fl & 32;
  auto row = [&](int code, float (&v)[VPL]) {
    const float *base = (code & kFwBit) ? a.fw32 : a.h32;
    ld32<VPL>(base + (size_t)(code & ~kFwBit) * (size_t)Nc8 + lfirst, v);
  };
  float fold[VPL], x1[VPL], x2[VPL], y1[VPL], y2[VPL], z1[VPL], z2[VPL];
  row(m * 8 + o, fold);
  row(r0.z, x1);
  row(r1.x, y1);
  row(r1.z, z1);
  if (!fx) row(r0.w, x2);
  if (!fy) row(r1.y, y2);
  if (!fz) row(r1.w, z2);
  const double2 m01 = __ldg(reinterpret_cast<const double2 *>(a.mom) + 2 * (size_t)m);
  const double2 m23 = __ldg(reinterpret_cast<const double2 *>(a.mom) + 2 * (size_t)m + 1);
  const float rho = (float)m01.x, ux = (float)m01.y, uy = (float)m23.x, uz = (float)m23.y;
  const int cls = (fx ? 1 : 0) | (fy ? 2 : 0) | (fz ? 4 : 0);
  const float sxf = (o == 0 || o == 3 || o == 4 || o == 7) ? 1.f : -1.f;
  const float syf = (o == 0 || o == 1 || o == 4 || o == 5) ? 1.f : -1.f;
  const float szf = o < 4 ? 1.f : -1.f;
  const float mu = (float)a.mu;
  float out[VPL];
#pragma unroll
  for (int q = 0; q < VPL; ++q) {
    const float *vt = a.vtab32 + (size_t)(lfirst + q) * kVtab;
    const float cx = __ldg(vt + 0), cy = __ldg(vt + 1), cz = __ldg(vt + 2), wl = __ldg(vt + 3);
    const float feq = wl * (rho + (sxf * cx * ux + syf * cy * uy + szf * cz * uz));
    float num = mu * (feq - 0.5f * fold[q]);
    num += __ldg(vt + (fx ? 5 : 4)) * x1[q];
    if (!fx) num += __ldg(vt + 6) * x2[q];
    num += __ldg(vt + (fy ? 8 : 7)) * y1[q];
    if (!fy) num += __ldg(vt + 9) * y2[q];
    num += __ldg(vt + (fz ? 11 : 10)) * z1[q];
    if (!fz) num += __ldg(vt + 12) * z2[q];
    out[q] = num * __ldg(vt + 21 + cls);
  }
  st32<VPL>(a.h32 + ((size_t)m * 8 + o) * (size_t)Nc8 + lfirst, out);
}

__global__ void k_commit32(const DevState a) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)a.ncommit * a.Nc8) return;
  const int e = (int)(idx / a.Nc8), l = (int)(idx % a.Nc8);
  const int node = a.commit[3 * e], o = a.commit[3 * e + 1], src = a.commit[3 * e + 2];
  a.h32[hidx(node, o, a.Nc8, l)] = src < 8 ? a.h32[hidx(node, src, a.Nc8, l)]
                                           : a.fw32[hidx(a.bcorner[node - a.NF], o, a.Nc8, l)];
}

// Walls: extrapolation and re-emission in FP32, the wall densities summed in FP64 (a warp
// reduction) and the re-emitted value formed in FP64 before rounding.
template <int VPL, int LANES>
__global__ void __launch_bounds__(256) k_walls32(const DevState a, int begin, int end, int gbuf) {
  // LANES lanes per wall (32 / LANES walls per warp), VPL velocities per lane
  const int widx = begin + (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES);
  if (widx >= end) return;
  const int lane = threadIdx.x % LANES;
  const unsigned seg = LANES == 32 ? 0xffffffffu : (((1u << LANES) - 1u) << (threadIdx.x & 31 & ~(LANES - 1)));
  const int q = a.wall_order[widx];
  const int node = a.wall_node[q];
  const int corner = a.wall_corner[q];
  const WProg &P = c32_prog[c32_prog_of[a.wall_label[q]]];
  const float e1 = (float)a.wall_e[2 * q], e2 = (float)a.wall_e[2 * q + 1];
  const int Nc8 = a.Nc8;
  const int *nb = a.wall_nb + 6 * q;
  const int nface = P.nface;
  const int chunkw = LANES * VPL;
  auto far_ptr = [&](int code, int oo, int lf) -> const float * {
    if (e2 == 0.f) return nullptr;  // as in k_walls32_rows
    if (code >= 0) return a.h32 + hidx(code, oo, Nc8, lf);
    if (code == -1) return nullptr;
    const int cc = -code - 2;
    const float *plane = (cc & 1) ? a.ghostE32[gbuf] : a.ghostW32[gbuf];
    return plane + ((size_t)(cc >> 1) * 4 + plane_slot(oo)) * Nc8 + lf;
  };
  double rho0 = 0.0, rho1 = 0.0, rho2 = 0.0;
  for (int fi = 0; fi < nface; ++fi) {
    const int dir = P.face[fi].dir, st = P.face[fi].store;
    const int n1 = nb[2 * fi], code = nb[2 * fi + 1];
    double racc = 0.0;
    for (int l0 = 0; l0 < Nc8; l0 += chunkw) {
      const int lf = l0 + lane * VPL;
      const bool lv = lf < Nc8;
      float ext[4][VPL];
#pragma unroll
      for (int mm = 0; mm < 4; ++mm) {
        const int oo = c32_incoming[dir][mm] - 1;
        float nv[VPL], fv[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v) { nv[v] = 0.f; fv[v] = 0.f; }
        if (lv) {
          ld32<VPL>(a.h32 + hidx(n1, oo, Nc8, lf), nv);
          const float *fp = far_ptr(code, oo, lf);
          if (fp) ld32<VPL>(fp, fv);
        }
#pragma unroll
        for (int v = 0; v < VPL; ++v) ext[mm][v] = e1 * nv[v] + e2 * fv[v];
        if (lv) {
          if (st == ST_F) st32<VPL>(a.h32 + hidx(node, oo, Nc8, lf), ext[mm]);
          else if (st == ST_W) st32<VPL>(a.fw32 + hidx(corner, oo, Nc8, lf), ext[mm]);
        }
      }
      double tface[VPL];
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int l = lf + v;
        const double ca = !lv ? 0.0 : dir < 2 ? __ldg(a.cx + l) : dir < 4 ? __ldg(a.cy + l) : __ldg(a.cz + l);
        tface[v] = ca * (((double)ext[0][v] + (double)ext[1][v]) + (double)ext[2][v] + (double)ext[3][v]);
      }
#pragma unroll
      for (int v = 0; v < VPL; ++v) racc += tface[v];
    }
    // warp sum in FP64 (the FP32 path does not keep the reference's summation order)
    for (int off = LANES / 2; off > 0; off >>= 1) racc += __shfl_xor_sync(seg, racc, off, LANES);
    if (fi == 0) rho0 = racc; else if (fi == 1) rho1 = racc; else rho2 = racc;
  }
  rho0 /= a.DiffFlux; rho1 /= a.DiffFlux; rho2 /= a.DiffFlux;
  const double one_m = 1.0 - a.accom;
  int zface = -1;
  for (int fi = 0; fi < nface; ++fi) if (P.face[fi].store == ST_Z) zface = fi;
  for (int l0 = 0; l0 < Nc8; l0 += chunkw) {
    const int lf = l0 + lane * VPL;
    if (lf >= Nc8) continue;
    // re-emission in groups of four writes: the sources of a group are loaded before its
    // stores (no write of a wall program reads a slot that an earlier write stores)
    for (int r0 = 0; r0 < P.nwr; r0 += 4) {
      float src[4][VPL];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (r0 + k >= P.nwr) break;
        const WWrite &W = P.wr[r0 + k];
        const int so = W.src_o - 1;
        if (W.src_store == ST_F) ld32<VPL>(a.h32 + hidx(node, so, Nc8, lf), src[k]);
        else if (W.src_store == ST_W) ld32<VPL>(a.fw32 + hidx(corner, so, Nc8, lf), src[k]);
        else {
          float nv[VPL], fv[VPL];
          ld32<VPL>(a.h32 + hidx(nb[2 * zface], so, Nc8, lf), nv);
#pragma unroll
          for (int v = 0; v < VPL; ++v) fv[v] = 0.f;
          const float *fp = far_ptr(nb[2 * zface + 1], so, lf);
          if (fp) ld32<VPL>(fp, fv);
#pragma unroll
          for (int v = 0; v < VPL; ++v) src[k][v] = e1 * nv[v] + e2 * fv[v];
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (r0 + k >= P.nwr) break;
        const WWrite &W = P.wr[r0 + k];
        const int dso = W.dst_o - 1;
        const double rf = W.face == 0 ? rho0 : W.face == 1 ? rho1 : rho2;
        float val[VPL];
#pragma unroll
        for (int v = 0; v < VPL; ++v)
          val[v] = (float)(a.accom * __ldg(a.w + lf + v) * rf + one_m * (double)src[k][v]);
        if (W.dst_store == ST_F) st32<VPL>(a.h32 + hidx(node, dso, Nc8, lf), val);
        else st32<VPL>(a.fw32 + hidx(corner, dso, Nc8, lf), val);
      }
    }
  }
}

// Shared memory of a wall in k_walls32_rows, in floats: 12 near rows (then the extrapolated
// values) and 12 far rows where some wall has an e2; walls of 8 velocities start 32 bytes past a
// multiple of 128, so that the four walls of a quarter-warp request use different banks.
__host__ __device__ constexpr int wall32_floats(int Nc8, int far_rows) {
  return (12 + far_rows) * Nc8 + (Nc8 == 8 ? 8 : 0);
}

// The FP32 diffuse wall for octants of 4 * LANES velocities, LANES lanes per wall and four
// velocities per lane: all rows of a wall are asked for at once (cp.async into shared memory: a
// lane copies what it reads itself), every face is extrapolated, the densities are summed in FP64
// (four velocities in the lane, then the lanes), and the re-emission reads the extrapolated values
// on chip (WPlan); a face value is stored only where it is the slot's final content.
// What bounds it: the rows' bytes (1.1 GB a pass on a 128^3 pack of 300,000 walls, 512 velocities,
// 0.165 ms at the copy rate: 0.189 ms). A version with separate plan fields, a load round trip per
// face and mixed programs in a warp was bound by its instructions: 0.430 ms there, and 0.156 against
// 0.023 ms on a 96^3 pack of 64 velocities, where a warp now takes 16 walls instead of 4.
template <int LANES>
__global__ void __launch_bounds__(64, 18) k_walls32_rows(const DevState a, int begin, int end, int gbuf, int far_rows) {
  extern __shared__ __align__(16) float wall32_sm[];
  constexpr int Nc8 = LANES * 4;
  const int widx = begin + (int)blockIdx.x * (64 / LANES) + (int)threadIdx.x / LANES;
  if (widx >= end) return;  // whole segment
  const int lane = threadIdx.x % LANES, lf = lane * 4;
  const unsigned seg = ((1u << LANES) - 1u) << (threadIdx.x & 31 & ~(LANES - 1));
  float *E = wall32_sm + (int)threadIdx.x / LANES * wall32_floats(Nc8, far_rows) + lf;
  const int4 *rp = a.wall_rec + (size_t)widx * 4;
  const int4 r0 = __ldg(rp), nb0 = __ldg(rp + 2), nb1 = __ldg(rp + 3);
  const double2 ee = __ldg(reinterpret_cast<const double2 *>(rp + 1));
  const float e1 = (float)ee.x, e2 = (float)ee.y;
  const WPlan &P = c32_plan[c32_prog_of[r0.z]];
  const int nface = (int)P.nface;
  for (int fi = 0; fi < nface; ++fi) {
    const uint32_t F = P.face[fi];
    const int n1 = fi == 0 ? nb0.x : fi == 1 ? nb0.z : nb1.x, code = fi == 0 ? nb0.y : fi == 1 ? nb0.w : nb1.y;
    const float *np = a.h32 + hidx(n1, 0, Nc8, lf);
#pragma unroll
    for (int m = 0; m < 4; ++m) cp_async16_cg(E + (fi * 4 + m) * Nc8, np + (F >> (3 * m) & 7) * Nc8);
    // the second extrapolation point only matters when its coefficient does (wallExtOrder 1
    // makes it 0)
    if (e2 == 0.f || code == -1) continue;
    const int cc = -code - 2;
    const float *plane = (cc & 1) ? a.ghostE32[gbuf] : a.ghostW32[gbuf];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int oo = F >> (3 * m) & 7;
      cp_async16_cg(E + (12 + fi * 4 + m) * Nc8,
                    code >= 0 ? a.h32 + hidx(code, oo, Nc8, lf)
                              : plane + ((size_t)(cc >> 1) * 4 + plane_slot(oo)) * Nc8 + lf);
    }
  }
  cp_async_wait_all();
  float *hn = a.h32 + hidx(r0.x, 0, Nc8, lf), *wn = a.fw32 + hidx(r0.y, 0, Nc8, lf);
  double rho0 = 0.0, rho1 = 0.0, rho2 = 0.0;
  for (int fi = 0; fi < nface; ++fi) {
    const uint32_t F = P.face[fi];
    const int dir = F >> 12 & 7, code = fi == 0 ? nb0.y : fi == 1 ? nb0.w : nb1.y;
    const bool far = e2 != 0.f && code != -1;
    float *out = (F >> 15 & 3) == ST_F ? hn : wn;
    float ext[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float *e = E + (fi * 4 + m) * Nc8;
      const float4 nv = *reinterpret_cast<const float4 *>(e);
      float4 fv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (far) fv = *reinterpret_cast<const float4 *>(e + 12 * Nc8);
      ext[m][0] = e1 * nv.x + e2 * fv.x;
      ext[m][1] = e1 * nv.y + e2 * fv.y;
      ext[m][2] = e1 * nv.z + e2 * fv.z;
      ext[m][3] = e1 * nv.w + e2 * fv.w;
      st32<4>(e, ext[m]);
      if (F >> (17 + m) & 1) st32<4>(out + (F >> (3 * m) & 7) * Nc8, ext[m]);
    }
    // the four octants of a velocity summed in FP32 (one conversion per velocity rather than
    // four), the velocities and lanes in FP64
    const double2 *cp = reinterpret_cast<const double2 *>((dir < 2 ? a.cx : dir < 4 ? a.cy : a.cz) + lf);
    const double2 c01 = __ldg(cp), c23 = __ldg(cp + 1);
    const double ca[4] = {c01.x, c01.y, c23.x, c23.y};
    double tv[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) tv[v] = (double)__fadd_rn(__fadd_rn(__fadd_rn(ext[0][v], ext[1][v]), ext[2][v]), ext[3][v]);
    double racc;
    if (LANES == 2) {
      // velocities l and l + 4 first, then l and l + 2, then the two left
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        tv[v] = __dmul_rn(ca[v], tv[v]);
        tv[v] += __shfl_xor_sync(seg, tv[v], 1, LANES);
      }
      racc = (tv[0] + tv[2]) + (tv[1] + tv[3]);
    } else {
      racc = 0.0;
#pragma unroll
      for (int v = 0; v < 4; ++v) racc = __fma_rn(ca[v], tv[v], racc);
#pragma unroll
      for (int off = LANES / 2; off > 0; off >>= 1) racc += __shfl_xor_sync(seg, racc, off, LANES);
    }
    if (fi == 0) rho0 = racc; else if (fi == 1) rho1 = racc; else rho2 = racc;
  }
  // re-emission in FP32: accom * rho_face rounded once per face, then w * that + (1 - accom)
  // * the extrapolated value, with the weights rounded to FP32 (vtab32 column 3)
  const float af[3] = {(float)(a.accom * (rho0 / a.DiffFlux)), nface > 1 ? (float)(a.accom * (rho1 / a.DiffFlux)) : 0.f,
                       nface > 2 ? (float)(a.accom * (rho2 / a.DiffFlux)) : 0.f};
  const float one_m = (float)(1.0 - a.accom);
  float wl[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) wl[v] = __ldg(a.vtab32 + (size_t)(lf + v) * kVtab + 3);
  const int nwr = (int)P.nwr;
  for (int k = 0; k < nwr; ++k) {
    const uint32_t W = P.wr[k];
    const float4 sp = *reinterpret_cast<const float4 *>(E + (W & 15) * Nc8);
    const int f = W >> 8 & 3;
    const float rf = f == 0 ? af[0] : f == 1 ? af[1] : af[2];
    const float val[4] = {__fmaf_rn(rf, wl[0], __fmul_rn(one_m, sp.x)), __fmaf_rn(rf, wl[1], __fmul_rn(one_m, sp.y)),
                          __fmaf_rn(rf, wl[2], __fmul_rn(one_m, sp.z)), __fmaf_rn(rf, wl[3], __fmul_rn(one_m, sp.w))};
    st32<4>((W >> 10 & 1 ? hn : wn) + (W >> 4 & 7) * Nc8, val);
  }
}

// Moments in FP64 from FP32 values: LANES lanes over K nodes, two velocities per lane and pass
// (the FP32 path does not follow the reference's order), all rows of a pass in flight together.
// The lanes' 4 * K sums are added by halves: at each step a lane keeps one half of its sums and
// hands the other to its partner, so 9 exchanges serve two nodes of 32 lanes where a tree per sum
// takes 40; the pairs added are the tree's. What bounds
// it: the bytes of f (128^3 pack, 512 velocities: 0.342 ms with trees, 0.275 now, 0.263 at the copy
// rate). Octants of 8 velocities take 4 lanes a node (96^3 pack: 0.164 -> 0.026 ms; a whole warp had
// 28 idle lanes).
template <int LANES, int K, int NC8>
__global__ void __launch_bounds__(256) k_moments32(const DevState a) {
  const int node0 = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES) * K;
  if (node0 >= a.NF) return;  // whole segment
  const int lane = threadIdx.x % LANES;
  const unsigned seg = LANES == 32 ? 0xffffffffu : (((1u << (LANES & 31)) - 1u) << (threadIdx.x & 31 & ~(LANES - 1)));
  const int Nc8 = NC8 ? NC8 : a.Nc8;
  double acc[4 * K];
#pragma unroll
  for (int i = 0; i < 4 * K; ++i) acc[i] = 0.0;
  for (int l0 = lane * 2; l0 < Nc8; l0 += LANES * 2) {
    float2 f[K][8];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float *hp = a.h32 + (size_t)min(node0 + k, a.NF - 1) * 8 * Nc8 + l0;
#pragma unroll
      for (int o = 0; o < 8; ++o) f[k][o] = __ldcs(reinterpret_cast<const float2 *>(hp + (size_t)o * Nc8));
    }
    const double2 cx = __ldg(reinterpret_cast<const double2 *>(a.cx + l0)),
                  cy = __ldg(reinterpret_cast<const double2 *>(a.cy + l0)),
                  cz = __ldg(reinterpret_cast<const double2 *>(a.cz + l0));
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const double f1 = v ? f[k][0].y : f[k][0].x, f2 = v ? f[k][1].y : f[k][1].x, f3 = v ? f[k][2].y : f[k][2].x,
                     f4 = v ? f[k][3].y : f[k][3].x, f5 = v ? f[k][4].y : f[k][4].x, f6 = v ? f[k][5].y : f[k][5].x,
                     f7 = v ? f[k][6].y : f[k][6].x, f8 = v ? f[k][7].y : f[k][7].x;
        acc[4 * k] += ((f1 + f2) + (f3 + f4)) + ((f5 + f6) + (f7 + f8));
        acc[4 * k + 1] += (v ? cx.y : cx.x) * (((f1 - f2) + (f4 - f3)) + ((f5 - f6) + (f8 - f7)));
        acc[4 * k + 2] += (v ? cy.y : cy.x) * (((f1 + f2) - (f3 + f4)) + ((f5 + f6) - (f7 + f8)));
        acc[4 * k + 3] += (v ? cz.y : cz.x) * (((f1 + f2) + (f3 + f4)) - ((f5 + f6) + (f7 + f8)));
      }
  }
  int n = 4 * K, which = 0;
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) {
    if (n > 1) {
      n /= 2;
      const bool up = lane & off;
      if (up) which += n;
#pragma unroll
      for (int i = 0; i < n; ++i) {
        const double mine = up ? acc[i + n] : acc[i], theirs = up ? acc[i] : acc[i + n];
        acc[i] = mine + __shfl_xor_sync(seg, theirs, off, LANES);
      }
    } else {
      acc[0] += __shfl_xor_sync(seg, acc[0], off, LANES);
    }
  }
  constexpr int kSame = LANES / (4 * K);  // lanes left with the same sum
  if (lane % kSame == 0 && node0 + which / 4 < a.NF) a.mom[(size_t)node0 * 4 + which] = acc[0];
}

__global__ void k_widen(const float *src, double *dst, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = (double)src[i];
}

__global__ void k_narrow(const double *src, float *dst, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = (float)src[i];
}

inline unsigned nblocks(size_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

}  // namespace

void upload_tables_fp32() {
  int8_t prog_of[128];
  WProg progs[26];
  int n = 0;
  for (int lab = 0; lab < 128; ++lab) {
    prog_of[lab] = -1;
    const WProg *p = wall_program(lab);
    if (p) { progs[n] = *p; prog_of[lab] = (int8_t)n; ++n; }
  }
  cudaMemcpyToSymbol(c32_prog_of, prog_of, sizeof prog_of);
  cudaMemcpyToSymbol(c32_prog, progs, sizeof progs);
  cudaMemcpyToSymbol(c32_incoming, kIncoming, sizeof(int) * 24);
  WPlan plans[26];
  int ok = n == 26;
  for (int i = 0; i < n; ++i) ok &= make_wall_plan(progs[i], plans[i]) ? 1 : 0;
  g32_plan_ok = ok != 0;
  cudaMemcpyToSymbol(c32_plan, plans, sizeof plans);
}

void launch_sweep_hyperplane32(const DevState &s, long t0, long ntask, cudaStream_t st) {
  if (ntask <= 0) return;
  if (s.lpt == 32) k_sweep32<32, 2><<<nblocks((size_t)ntask * s.nchunk * 32, 256), 256, 0, st>>>(s, t0, ntask);
  else k_sweep32<8, 1><<<nblocks((size_t)ntask * s.nchunk * 8, 256), 256, 0, st>>>(s, t0, ntask);
}
void launch_commit32(const DevState &s, cudaStream_t st) {
  if (s.ncommit && s.Nc8 % 4 == 0) return launch_commit_rows(s, true, st);
  if (s.ncommit) k_commit32<<<nblocks((size_t)s.ncommit * s.Nc8, 256), 256, 0, st>>>(s);
}
void launch_capture32(const DevState &s, int buf, cudaStream_t st) {
  boundary::launch_capture<float>(s.h32, s.ghostW32[buf], s.ghostE32[buf], s, st);
}
namespace {
template <int LANES>
void launch_walls32_rows(const DevState &s, int begin, int end, int gbuf, cudaStream_t st) {
  const int walls = 64 / LANES, far_rows = s.wall_far ? 12 : 0;
  once_per_device(reinterpret_cast<const void *>(k_walls32_rows<LANES>), [](int) {
    cudaFuncSetAttribute(k_walls32_rows<LANES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(float) * wall32_floats(4 * LANES, 12) * (64 / LANES));
  });
  const size_t smem = sizeof(float) * (size_t)wall32_floats(s.Nc8, far_rows) * walls;
  k_walls32_rows<LANES><<<(end - begin + walls - 1) / walls, 64, smem, st>>>(s, begin, end, gbuf, far_rows);
}
}  // namespace
void launch_walls32(const DevState &s, int begin, int end, int gbuf, cudaStream_t st) {
  if (end <= begin) return;
  const size_t walls = (size_t)(end - begin);
  if (g32_plan_ok && s.Nc8 == 64) return launch_walls32_rows<16>(s, begin, end, gbuf, st);
  if (g32_plan_ok && s.Nc8 == 8) return launch_walls32_rows<2>(s, begin, end, gbuf, st);
  if (s.Nc8 % 64 == 0) k_walls32<4, 16><<<nblocks(walls * 16, 256), 256, 0, st>>>(s, begin, end, gbuf);
  else k_walls32<1, 32><<<nblocks(walls * 32, 256), 256, 0, st>>>(s, begin, end, gbuf);
}
void launch_inlet_outlet32(const DevState &s, int buf, cudaStream_t st) {
  boundary::launch_inlet_outlet<float>(s.h32, s.ghostW32[buf], s.ghostE32[buf], s, st);
}
void launch_symmetry32(const DevState &s, cudaStream_t st) {
  boundary::launch_symmetry<float>(s.h32, s, st);
}
void launch_moments32(const DevState &s, cudaStream_t st) {
  if (!s.NF) return;
  if (s.Nc8 == 8) k_moments32<4, 1, 8><<<nblocks((size_t)s.NF * 4, 256), 256, 0, st>>>(s);
  else if (s.Nc8 == 64) k_moments32<32, 2, 64><<<nblocks((size_t)(s.NF + 1) / 2 * 32, 256), 256, 0, st>>>(s);
  else k_moments32<32, 2, 0><<<nblocks((size_t)(s.NF + 1) / 2 * 32, 256), 256, 0, st>>>(s);
}
template <typename T>
__global__ void __launch_bounds__(256) k_gram(const char *base, size_t stride, int n, size_t count, double *partial) {
  constexpr int kMaxD = kMaxSnapSlots - 1, kMaxPairs = kMaxD * (kMaxD + 1) / 2;
  __shared__ double red[256];
  const int nd = n - 1, npair = nd * (nd + 1) / 2;
  double acc[kMaxPairs];
#pragma unroll
  for (int q = 0; q < kMaxPairs; ++q) acc[q] = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
    double x[kMaxSnapSlots], u[kMaxD];
#pragma unroll
    for (int j = 0; j < kMaxSnapSlots; ++j)
      x[j] = j < n ? (double)reinterpret_cast<const T *>(base + (size_t)j * stride)[i] : 0.0;
#pragma unroll
    for (int a = 0; a < kMaxD; ++a) u[a] = x[a + 1] - x[a];
    int q = 0;
#pragma unroll
    for (int a = 0; a < kMaxD; ++a)
#pragma unroll
      for (int b = a; b < kMaxD; ++b, ++q)
        if (b < nd) acc[q] += u[a] * u[b];
  }
  // block sums in a fixed tree order, pair by pair (acc is indexed over the kMaxD triangle,
  // the output over the nd triangle)
  int q = 0;
  for (int a = 0; a < nd; ++a)
    for (int b = a; b < nd; ++b, ++q) {
      const int qa = a * kMaxD - a * (a - 1) / 2 + (b - a);
      double v = 0.0;
#pragma unroll
      for (int k = 0; k < kMaxPairs; ++k)
        if (k == qa) v = acc[k];
      red[threadIdx.x] = v;
      __syncthreads();
      for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
      }
      if (threadIdx.x == 0) partial[(size_t)blockIdx.x * npair + q] = red[0];
      __syncthreads();
    }
}
template <typename T>
void gram_any(const T *base, size_t stride, int n, size_t count, double *partial, cudaStream_t st) {
  const int npair = (n - 1) * n / 2;
  if (!count) {
    cudaMemsetAsync(partial, 0, (size_t)kGramBlocks * npair * sizeof(double), st);
    return;
  }
  k_gram<T><<<kGramBlocks, 256, 0, st>>>(reinterpret_cast<const char *>(base), stride, n, count, partial);
}
void launch_gram(const double *base, size_t stride, int n, size_t count, double *partial, cudaStream_t st) {
  gram_any(base, stride, n, count, partial, st);
}
void launch_gram(const float *base, size_t stride, int n, size_t count, double *partial, cudaStream_t st) {
  gram_any(base, stride, n, count, partial, st);
}

struct Coefs { double c[kMaxSnapSlots]; };
template <typename T>
__global__ void k_combine(T *dst, const char *base, size_t stride, int n, Coefs cf, size_t count) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
    double v = 0.0;
    for (int j = 0; j < n; ++j) v += cf.c[j] * (double)reinterpret_cast<const T *>(base + (size_t)j * stride)[i];
    dst[i] = (T)v;
  }
}
template <typename T>
void combine_any(T *dst, const T *base, size_t stride, int n, const double *coef, size_t count, cudaStream_t st) {
  if (!count) return;
  Coefs cf{};
  for (int j = 0; j < n && j < kMaxSnapSlots; ++j) cf.c[j] = coef[j];
  k_combine<T><<<148 * 16, 256, 0, st>>>(dst, reinterpret_cast<const char *>(base), stride, n, cf, count);
}
void launch_combine(double *dst, const double *base, size_t stride, int n, const double *coef, size_t count,
                    cudaStream_t st) {
  combine_any(dst, base, stride, n, coef, count, st);
}
void launch_combine(float *dst, const float *base, size_t stride, int n, const double *coef, size_t count,
                    cudaStream_t st) {
  combine_any(dst, base, stride, n, coef, count, st);
}
void launch_widen(const float *src, double *dst, size_t n, cudaStream_t st) {
  if (n) k_widen<<<148 * 16, 256, 0, st>>>(src, dst, n);
}
void launch_narrow(const double *src, float *dst, size_t n, cudaStream_t st) {
  if (n) k_narrow<<<148 * 16, 256, 0, st>>>(src, dst, n);
}

}  // namespace piks
