// Cell kernels of the GB300 HemoCell step (sm_103a):
//   K2 spread          IBM phi2 force spreading with FORCE_LIMIT clamp; one
//                      vector atomic per node contribution (FP32); tags the
//                      stencil nodes for the interpolation
//   K3+K5 interp_advance  velocity interpolation from the tagged node
//                      velocities, Euler advance, nearest-node bin, wall deletion
//   K4 mechanics       RBC / PLT / WBC membrane forces, one CTA per cell
//   binning            tile CSR sorted by (tile, cell, vertex)
// Templated on T = double (plain form) or float (mixed form); positions are
// double in both forms.
#include <cmath>
#include <cstdint>

#include "hc_async.cuh"
#include "hc_d3q19.cuh"
#include "hc_newton.h"
#include "hc_posbits.h"

namespace hcd {

template <typename T>
__device__ __forceinline__ T tmax(T a, T b) {
  return a > b ? a : b;
}

template <typename T>
struct V3t {
  T x, y, z;
};
template <typename T>
__device__ __forceinline__ V3t<T> operator-(V3t<T> a, V3t<T> b) {
  return {a.x - b.x, a.y - b.y, a.z - b.z};
}
template <typename T>
__device__ __forceinline__ V3t<T> operator+(V3t<T> a, V3t<T> b) {
  return {a.x + b.x, a.y + b.y, a.z + b.z};
}
template <typename T>
__device__ __forceinline__ V3t<T> vscale(V3t<T> a, T s) {
  return {a.x * s, a.y * s, a.z * s};
}
template <typename T>
__device__ __forceinline__ V3t<T> vcross(V3t<T> a, V3t<T> b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
template <typename T>
__device__ __forceinline__ T vdot(V3t<T> a, V3t<T> b) {
  T r = a.x * b.x;
  r += a.y * b.y;
  r += a.z * b.z;
  return r;
}
// x == 0 and isfinite(x) on the bits of a double: a comparison would take an
// instruction of the FP64 pipe
__device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
__device__ __forceinline__ bool is_zero(double x) {
  return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool is_finite(float x) { return isfinite(x); }
__device__ __forceinline__ bool is_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// IBM phi2 kernel (core/immersedBoundaryMethod.h:37-41, :62-138).  The
// reference scans the 3x3x3 nodes around floor(p+0.5) and keeps the nonzero
// weights; phi2 vanishes beyond distance 1, so the kept nodes always lie in
// the 2x2x2 block {floor(p), floor(p)+1}^3, scanned here in the same
// (x, y, z) order.  Nodes off a non-periodic axis, zero weights and boundary
// nodes are skipped (slot node = -1); the weights are renormalised to one.
// FP64 evaluates phi2(p - q) exactly as the reference; FP32 takes the
// fractional part (float)(p - floor(p)) once, from the bits of the FP64
// coordinate (hc_posbits.h), and the rest in float.
template <typename T>
struct Kern {
  int node[8];  // the lattice holds fewer than 2^31 nodes (hc_create's size limit)
  T w[8];
};

// load(nodes) is called with the node of every slot, skipped or not (0 off the
// lattice), before the flags are waited for.
template <typename T, typename Load>
__device__ __forceinline__ void ibm_weights(const LbmView<T>& L, double px, double py, double pz, Kern<T>& K,
                                            const Load& load) {
  constexpr bool kF64 = sizeof(T) == 8;
  const double P[3] = {px, py, pz};
  const int dims[3] = {L.nx, L.ny, L.nz};
  T phi[3][2];
  int idx[3][2];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    long long qi;
    if (kF64) {
      // floor(P) from the bits of P as well: P - floor(P) is then the one FP64
      // instruction, and both weights are the bits of the expression below it
      // (1 - |P - (q + 1)| is exactly the fraction for P >= 1)
      int qs;
      double q0;
      if (hcpos::floor_bits(P[a], qs, q0)) {
        const T fr = T(P[a] - q0);
        phi[a][0] = T(1) - fr;
        phi[a][1] = fr;
        qi = qs;
      } else {
        q0 = floor(P[a]);
        phi[a][0] = tmax(T(1) - T(fabs(P[a] - q0)), T(0));
        phi[a][1] = tmax(T(1) - T(fabs(P[a] - (q0 + 1.0))), T(0));
        qi = (long long)q0;
      }
    } else {
      // floor(P) and the fraction (float)(P - floor(P)) from the bits of P,
      // the FP64 instructions only outside [1, 2^31)
      // A fraction within 2^-25 of one rounds to 1.0f; the lower node's
      // weight is then the rounded exact complement 1 - (P - floor(P)), not
      // zero, so that a vertex next to a wall keeps the FP64 form's
      // renormalised stencil.
      int qs;
      float w0, w1;
      if (hcpos::split_weights(P[a], qs, w0, w1)) {
        qi = qs;
      } else {
        const double q0 = floor(P[a]);
        const double fr = P[a] - q0;  // exact, as is 1 - fr
        w1 = (float)fr;
        w0 = w1 == 1.0f ? (float)(1.0 - fr) : 1.0f - w1;
        qi = (long long)q0;
      }
      phi[a][0] = (T)w0;
      phi[a][1] = (T)w1;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const long long q = qi + k;
      int wrapped;
      if (q < 0 || q >= dims[a]) {
        if (L.per[a]) {
          long long mm = q % dims[a];
          wrapped = (int)(mm < 0 ? mm + dims[a] : mm);
        } else {
          wrapped = -1;
        }
      } else {
        wrapped = (int)q;
      }
      idx[a][k] = wrapped;
    }
  }
  // the eight nodes' solid bits in one byte of the block's first node, in flight
  // together with what else the caller loads per node (with eight scattered
  // flags the FP32 force assembly of a 960-cell suspension took 134 us against
  // 127; before, with the other loads waiting for them, 139)
  uint32_t solid = 0;
  if (idx[0][0] >= 0 && idx[1][0] >= 0 && idx[2][0] >= 0) {
    const int base = idx[0][0] + L.nx * (idx[1][0] + L.ny * idx[2][0]);
    solid = HC_IN(L.status, base, L.N) ? L.corner[base] : 0xffu;
  } else {
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int ax = s >> 2, ay = (s >> 1) & 1, az = s & 1;
      if (idx[0][ax] < 0 || idx[1][ay] < 0 || idx[2][az] < 0) continue;
      const int nd = idx[0][ax] + L.nx * (idx[1][ay] + L.ny * idx[2][az]);
      if (!HC_IN(L.status, nd, L.N) || L.flag[nd] != 0) solid |= 1u << s;
    }
  }
  bool cut = false;  // a node that carries weight was left out
  int nodes[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    const int ax = s >> 2, ay = (s >> 1) & 1, az = s & 1;
    const bool off = idx[0][ax] < 0 || idx[1][ay] < 0 || idx[2][az] < 0;
    const int nd = off ? 0 : idx[0][ax] + L.nx * (idx[1][ay] + L.ny * idx[2][az]);
    const bool in = HC_IN(L.status, nd, L.N);
    nodes[s] = in ? nd : 0;
    cut |= off;
    K.w[s] = phi[0][ax] * phi[1][ay] * phi[2][az];
    K.node[s] = off || is_zero(K.w[s]) || !in ? -1 : nd;
  }
  load(nodes);
  T total = T(0);
#pragma unroll
  for (int s = 0; s < 8; ++s) {
    if (K.node[s] >= 0 && (solid >> s & 1u)) {
      K.node[s] = -1;
      cut = true;
    }
    if (K.node[s] < 0) K.w[s] = T(0);
    else if (!kF64) total += K.w[s];
  }
  // The weights of a whole stencil sum to one by themselves, to the rounding
  // of their products: FP64, whose pipe bounds the cell kernels, renormalises
  // only a stencil that lost a node (24 of its 60 instructions otherwise).  Random
  // coordinates up to 1000, rms in units of 2^-53 against exact weights: each
  // weight 0.115 off (renormalised 0.181), their sum 0.35 (0.82), the value
  // interpolated from a random field 0.64 (0.75).
  if (kF64 && cut) {
#pragma unroll
    for (int s = 0; s < 8; ++s) total += K.w[s];
  }
  if (total > T(0)) {
    const T coeff = T(1) / total;
#pragma unroll
    for (int s = 0; s < 8; ++s) K.w[s] *= coeff;
  }
}

// Bit s of corner[n]: slot s of the 2x2x2 block from node n on, wrapped at the
// lattice's ends, is a boundary node.  Of a slot beyond a non-periodic end the bit
// says nothing; the callers leave such a slot out by its index.
__global__ void k_corner_flags(const uint8_t* flag, uint8_t* corner, int nx, int ny, int nz) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x;
  if (X >= nx) return;
  for (int Z = blockIdx.z; Z < nz; Z += gridDim.z)
    for (int Y = blockIdx.y * blockDim.y + threadIdx.y; Y < ny; Y += gridDim.y * blockDim.y) {
      uint32_t bits = 0;
      for (int s = 0; s < 8; ++s) {
        const int x = X + (s >> 2) < nx ? X + (s >> 2) : 0, y = Y + (s >> 1 & 1) < ny ? Y + (s >> 1 & 1) : 0,
                  z = Z + (s & 1) < nz ? Z + (s & 1) : 0;
        if (flag[x + (long long)nx * (y + (long long)ny * z)] != 0) bits |= 1u << s;
      }
      corner[X + (long long)nx * (Y + (long long)ny * Z)] = (uint8_t)bits;
    }
}
cudaError_t launch_corner_flags(const uint8_t* flag, uint8_t* corner, int nx, int ny, int nz, cudaStream_t s) {
  const dim3 block(32, 8), grid((nx + 31) / 32, std::min((ny + 7) / 8, 65535), std::min(nz, 65535));
  k_corner_flags<<<grid, block, 0, s>>>(flag, corner, nx, ny, nz);
  return cudaGetLastError();
}

template <typename T>
__device__ __forceinline__ void ibm_weights(const LbmView<T>& L, double px, double py, double pz, Kern<T>& K) {
  ibm_weights(L, px, py, pz, K, [](const int*) {});
}
// The velocity at (px, py, pz): the lower x-side's four nodes, then the upper's.
template <typename T>
__device__ __forceinline__ V3t<T> ibm_velocity(const LbmView<T>& L, double px, double py, double pz) {
  Kern<T> K;
  V3t<T> u[8], v[2] = {};
  ibm_weights(L, px, py, pz, K, [&](const int* nd) {
#pragma unroll
    for (int s = 0; s < 8; ++s) FieldLayout<T>::load(L.unode, L.N, nd[s], u[s].x, u[s].y, u[s].z);
  });
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (K.node[j] < 0) continue;
    v[j >> 2].x += u[j].x * K.w[j];
    v[j >> 2].y += u[j].y * K.w[j];
    v[j >> 2].z += u[j].z * K.w[j];
  }
  return v[0] + v[1];
}
// Two neighbouring lanes share their stencils: of both vertices the even lane
// takes the lower x-side (slots 0 to 3) and the odd lane the upper one, whose
// nodes lie beside the lower's.  A load or atomic add of the warp then touches
// 16 pairs of neighbouring nodes instead of 32 nodes of 32 vertices (27 lines of
// 128 bytes for a turned red cell).  Force assembly of the 280-cell pipe: FP64
// 184.7 us before, 179.1 now; FP32 39.1 and 37.7.  side[0..3] of the even lane's
// vertex, side[4..7] of the odd lane's.
template <typename V>
__device__ __forceinline__ void pair_sides(const V own[8], V side[8]) {
  const bool odd = threadIdx.x & 1;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const V other = __shfl_xor_sync(0xffffffffu, odd ? own[j] : own[4 + j], 1);
    side[j] = odd ? other : own[j];
    side[4 + j] = odd ? own[4 + j] : other;
  }
}
// ibm_velocity by whole warps, the sums in the same order; a lane without a
// vertex (on clear) takes part with weights of zero.
template <typename T>
__device__ __forceinline__ V3t<T> pair_velocity(const LbmView<T>& L, double px, double py, double pz, bool on) {
  Kern<T> K;
  V3t<T> u[8], v[2] = {};
  ibm_weights(L, px, py, pz, K, [&](const int* own) {
    int nd[8];
    pair_sides(own, nd);
#pragma unroll
    for (int s = 0; s < 8; ++s) FieldLayout<T>::load(L.unode, L.N, nd[s], u[s].x, u[s].y, u[s].z);
  });
  T w[8];
  if (!on) {
#pragma unroll
    for (int s = 0; s < 8; ++s) K.w[s] = T(0);
  }
  pair_sides(K.w, w);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (is_zero(w[j])) continue;
    v[j >> 2].x += u[j].x * w[j];
    v[j >> 2].y += u[j].y * w[j];
    v[j >> 2].z += u[j].z * w[j];
  }
  // this lane's vertex is v[0] of an even lane, v[1] of an odd one
  const bool odd = threadIdx.x & 1;
  const V3t<T> own = odd ? v[1] : v[0], give = odd ? v[0] : v[1];
  const V3t<T> other = {__shfl_xor_sync(0xffffffffu, give.x, 1), __shfl_xor_sync(0xffffffffu, give.y, 1),
                        __shfl_xor_sync(0xffffffffu, give.z, 1)};
  return own + other;
}

// ---------------------------------------------------------------------------
// K2: spreadParticleForce (core/hemoCellParticleField.cpp:841-863) with the
// FORCE_LIMIT clamp written back (:847-852); the stencil nodes are tagged
// with the step stamp so the interpolation evaluates only those nodes.
template <typename T>
__global__ void __launch_bounds__(256) k_spread(const LbmView<T> L, const VertexView<T> vv, const T f_limit) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= vv.nvert || !vv.alive[vv.vcell[i]]) return;
  const uint32_t stamp = *L.stamp;
  const long long V = vv.V;
  T fx = vv.f[i], fy = vv.f[V + i], fz = vv.f[2 * V + i];
  T mag = fx * fx;
  mag += fy * fy;
  mag += fz * fz;
  mag = sqrt(mag);
  if (mag > f_limit) {
    const T s = f_limit / mag;
    fx *= s;
    fy *= s;
    fz *= s;
    vv.f[i] = fx;
    vv.f[V + i] = fy;
    vv.f[2 * V + i] = fz;
  }
  // the repulsion force is spread with the clamped force (:857-859)
  if (vv.frep_cell) {
    fx += vv.frep_cell[i];
    fy += vv.frep_cell[V + i];
    fz += vv.frep_cell[2 * V + i];
  }
  if (vv.frep_wall) {
    fx += vv.frep_wall[i];
    fy += vv.frep_wall[V + i];
    fz += vv.frep_wall[2 * V + i];
  }
  Kern<T> K;
  ibm_weights(L, vv.x[i], vv.x[V + i], vv.x[2 * V + i], K);
  T* F = const_cast<T*>(L.Fcur);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (K.node[j] < 0) continue;
    if (L.ntag) L.ntag[K.node[j]] = stamp;
    FieldLayout<T>::add(F, L.N, K.node[j], fx * K.w[j], fy * K.w[j], fz * K.w[j]);
  }
  pdl_trigger();
}

template <typename T>
cudaError_t launch_spread(const LbmView<T>& L, const VertexView<T>& vv, double f_limit, int bs, cudaStream_t s) {
  if (vv.nvert <= 0) return cudaSuccess;
  if (bs <= 0) bs = 128;
  return launch_kernel(k_spread<T>, dim3((vv.nvert + bs - 1) / bs), dim3(bs), 0, s, L.pdl, L, vv, (T)f_limit);
}

// ---------------------------------------------------------------------------
// CellInformation (helper/cellInfo.cpp:170-266), one CTA per cell: centroid,
// mean velocity, membrane area, enclosed volume (six-term sum over faces, on
// coordinates relative to the cell's vertex 0), largest distance between two
// of its vertices (stretch), bounding box.  out holds 16 doubles per cell:
// cx cy cz vx vy vz area volume stretch xmin xmax ymin ymax zmin zmax type
// (type -1 once the cell was deleted).
template <typename T>
__global__ void __launch_bounds__(256) k_cell_info(const VertexView<T> vv, const int* cell_type, const int* cell_voff,
                                                   const TypeDev* types, double* out) {
  __shared__ double red[32][16];
  const int cell = blockIdx.x;
  const TypeDev& t = types[cell_type[cell]];
  const int nv = t.nv, voff = cell_voff[cell];
  const long long V = vv.V;
  const double* X = vv.x;
  const double o[3] = {X[voff], X[V + voff], X[2 * V + voff]};
  double acc[16];
  for (int k = 0; k < 16; ++k) acc[k] = 0.0;
  acc[9] = acc[11] = acc[13] = 1e300;    // minima
  acc[10] = acc[12] = acc[14] = -1e300;  // maxima
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    for (int a = 0; a < 3; ++a) {
      const double p = X[a * V + voff + i];
      acc[a] += p;
      acc[3 + a] += (double)vv.v[a * V + voff + i];
      acc[9 + 2 * a] = fmin(acc[9 + 2 * a], p);
      acc[10 + 2 * a] = fmax(acc[10 + 2 * a], p);
    }
    double pi[3];
    for (int a = 0; a < 3; ++a) pi[a] = X[a * V + voff + i];
    for (int j = i + 1; j < nv; ++j) {
      double d2 = 0.0;
      for (int a = 0; a < 3; ++a) {
        const double d = pi[a] - X[a * V + voff + j];
        d2 += d * d;
      }
      acc[8] = fmax(acc[8], d2);
    }
  }
  for (int k = threadIdx.x; k < t.nf; k += blockDim.x) {
    double v[3][3];
    for (int c = 0; c < 3; ++c)
      for (int a = 0; a < 3; ++a) v[c][a] = X[a * V + voff + t.tris[3 * k + c]] - o[a];
    const double e1[3] = {v[1][0] - v[0][0], v[1][1] - v[0][1], v[1][2] - v[0][2]};
    const double e2[3] = {v[2][0] - v[0][0], v[2][1] - v[0][1], v[2][2] - v[0][2]};
    const double cx = e1[1] * e2[2] - e1[2] * e2[1], cy = e1[2] * e2[0] - e1[0] * e2[2],
                 cz = e1[0] * e2[1] - e1[1] * e2[0];
    acc[6] += 0.5 * sqrt(cx * cx + cy * cy + cz * cz);
    acc[7] += (-v[2][0] * v[1][1] * v[0][2] + v[1][0] * v[2][1] * v[0][2] + v[2][0] * v[0][1] * v[1][2] -
               v[0][0] * v[2][1] * v[1][2] - v[1][0] * v[0][1] * v[2][2] + v[0][0] * v[1][1] * v[2][2]) /
              6.0;
  }
  // block reduction: sums for 0-7, max for 8, 10, 12, 14, min for 9, 11, 13
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  for (int k = 0; k < 15; ++k) {
    double x = acc[k];
    for (int off = 16; off > 0; off >>= 1) {
      const double y = __shfl_down_sync(0xffffffffu, x, off);
      x = k < 8 ? x + y : ((k == 9 || k == 11 || k == 13) ? fmin(x, y) : fmax(x, y));
    }
    if (lane == 0) red[wid][k] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double r[15];
    for (int k = 0; k < 15; ++k) {
      r[k] = red[0][k];
      for (int w = 1; w < nw; ++w)
        r[k] = k < 8 ? r[k] + red[w][k] : ((k == 9 || k == 11 || k == 13) ? fmin(r[k], red[w][k]) : fmax(r[k], red[w][k]));
    }
    double* dst = out + 16 * (size_t)cell;
    for (int a = 0; a < 3; ++a) {
      dst[a] = r[a] / nv;
      dst[3 + a] = r[3 + a] / nv;
    }
    dst[6] = r[6];
    dst[7] = r[7];
    dst[8] = sqrt(r[8]);
    for (int k = 9; k < 15; ++k) dst[k] = r[k];
    dst[15] = vv.alive[cell] ? (double)cell_type[cell] : -1.0;
  }
}

template <typename T>
cudaError_t launch_cell_info(const VertexView<T>& vv, const int* cell_type, const int* cell_voff, const TypeDev* types,
                             int ncells, double* out, cudaStream_t s) {
  if (ncells <= 0) return cudaSuccess;
  k_cell_info<T><<<ncells, 256, 0, s>>>(vv, cell_type, cell_voff, types, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Repulsion.  k_rep_bin bins every vertex of a live cell at its node
// int(x + 0.5) (core/hemoCellParticleField.cpp:153-156), wrapped on periodic
// axes, and keeps its position relative to that node.  k_repulsion then
// gathers, per vertex, over the 27 nodes around its own: vertices of other
// cells closer than the cutoff push with kc * (rc / d) along the separation,
// counted twice when they share the node (the reference visits a node's own
// pairs in both orders, :678-694), and boundary nodes closer than the wall
// cutoff push with kw * (rw / d) (:891-918).  Node offsets of at most one in
// each axis make the separation (x_p - q_p) - (x_b - q_b) - d exact in the
// working precision and take the periodic image.  Each node's vertices are
// visited in ascending index order so the sums are deterministic.
//
// What bounds it: the chain of dependent loads (count, slots, cell, position) at
// each of the 27 nodes, of which all but a few hold no vertex or only the
// vertex's own cell.  So every node carries the cell of its vertices (or that
// there are several), the 27 are loaded at once, and the chain runs only at the
// nodes that another cell reaches; likewise the boundary nodes only where one of
// the 27 is one.  Those few (vertex, node) pairs are spread over the warp, four
// lanes to a vertex.  77,000 vertices at 25% haematocrit: 54 -> 26 us for the
// kernel, 86 -> 54 us for the step (one lane a vertex with the same tags: 36).
constexpr int REP_MIXED = -1;  // a node's vertices belong to several cells
template <typename T>
__global__ void k_rep_bin(const LbmView<T> L, const VertexView<T> vv, const RepView<T> R) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= vv.nvert) return;
  int q = -1;
  const int cell = vv.vcell[i];
  if (vv.alive[cell]) {
    const long long V = vv.V;
    const double P[3] = {vv.x[i], vv.x[V + i], vv.x[2 * V + i]};
    const int n[3] = {L.nx, L.ny, L.nz};
    int c[3];
    T r[3];
    bool in = true;
    for (int a = 0; a < 3; ++a) {
      long long v = hcpos::nearest(P[a]);  // floor(P + 0.5), exactly
      r[a] = (T)(P[a] - (double)v);
      if (v < 0 || v >= n[a]) {
        if (L.per[a]) {
          v %= n[a];
          if (v < 0) v += n[a];
        } else {
          in = false;
        }
      }
      c[a] = (int)v;
    }
    if (in) {
      q = c[0] + L.nx * (c[1] + L.ny * c[2]);
      R.rec[i] = {r[0], r[1], r[2], cell};
      if (R.node) {
        const int s = atomicAdd(&R.node[q].x, 1);
        if (s < REP_SLOTS) R.slot[(long long)q * REP_SLOTS + s] = i;
        else atomicOr(L.status, STATUS_REP_OVERFLOW);
        const int was = atomicCAS(&R.node[q].y, 0, cell + 1);
        if (was != 0 && was != cell + 1 && was != REP_MIXED) atomicExch(&R.node[q].y, REP_MIXED);
      }
    }
  }
  R.vq[i] = q;
}

// The node at offset d of node (X0, Y0, Z0), or -1 off a non-periodic axis.
template <typename T>
__device__ __forceinline__ int rep_node(const LbmView<T>& L, int X0, int Y0, int Z0, int dx, int dy, int dz) {
  int x = X0 + dx, y = Y0 + dy, z = Z0 + dz;
  if (x < 0 || x >= L.nx) {
    if (!L.per[0]) return -1;
    x = x < 0 ? x + L.nx : x - L.nx;
  }
  if (y < 0 || y >= L.ny) {
    if (!L.per[1]) return -1;
    y = y < 0 ? y + L.ny : y - L.ny;
  }
  if (z < 0 || z >= L.nz) {
    if (!L.per[2]) return -1;
    z = z < 0 ? z + L.nz : z - L.nz;
  }
  return x + L.nx * (y + L.ny * z);
}

// The push on vertex (rp, cell) at node q0 from the other cells' vertices at its
// node s, in ascending index order.
template <typename T>
__device__ __forceinline__ V3t<T> rep_push(const LbmView<T>& L, const RepView<T>& R, int q0, const RepRecord<T>& own,
                                           int s) {
  const int X0 = q0 % L.nx, Y0 = (q0 / L.nx) % L.ny, Z0 = q0 / (L.nx * L.ny);
  const int d[3] = {s % 3 - 1, s / 3 % 3 - 1, s / 9 - 1};
  const int qb = rep_node(L, X0, Y0, Z0, d[0], d[1], d[2]);
  const int cnt = min(R.node[qb].x, REP_SLOTS);
  const int* sl = R.slot + (long long)qb * REP_SLOTS;
  const T mult = s == 13 ? T(2) : T(1);
  V3t<T> f = {T(0), T(0), T(0)};
  auto push = [&](int b) {
    const RepRecord<T> o = R.rec[b];
    if (o.cell == own.cell) return;
    const V3t<T> dv = {(own.x - o.x) - T(d[0]), (own.y - o.y) - T(d[1]), (own.z - o.z) - T(d[2])};
    const T dist = sqrt(dv.x * dv.x + dv.y * dv.y + dv.z * dv.z);
    if (dist < R.rc) f = f + vscale(dv, mult * R.kc * (R.rc / dist) / dist);
  };
  // the first two at once (a node seldom holds more), the others by selection
  const int2 two = *reinterpret_cast<const int2*>(sl);
  if (cnt == 1) {
    push(two.x);
  } else if (cnt == 2) {
    push(min(two.x, two.y));
    push(max(two.x, two.y));
  } else {
    int last = -1;
    for (int k = 0; k < cnt; ++k) {
      int b = 0x7fffffff;
      for (int m = 0; m < cnt; ++m) {
        const int v = sl[m];
        if (v > last && v < b) b = v;
      }
      last = b;
      push(b);
    }
  }
  return f;
}

// Four lanes a vertex: each looks at every fourth of the 27 nodes, then the
// warp's (vertex, node) pairs are evaluated a lane each, 32 at a time.
constexpr int kRepBlock = 128, kRepVertices = 8, kRepWarps = kRepBlock / 32;
template <typename T>
__global__ void __launch_bounds__(kRepBlock) k_repulsion(const LbmView<T> L, const VertexView<T> vv,
                                                         const RepView<T> R) {
  pdl_wait();
  __shared__ RepRecord<T> s_own[kRepWarps][kRepVertices];
  __shared__ int s_node[kRepWarps][kRepVertices];
  __shared__ uint8_t s_pair[kRepWarps][kRepVertices * 32];  // vertex << 5 | node
  __shared__ T s_push[kRepWarps][32][3];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, v = lane >> 2, part = lane & 3;
  const int p = (blockIdx.x * kRepWarps + w) * kRepVertices + v;
  const bool in = p < vv.nvert;
  const long long V = vv.V;
  const int q0 = in ? R.vq[p] : -1;
  RepRecord<T> own = {T(0), T(0), T(0), 0};
  int X0 = 0, Y0 = 0, Z0 = 0;
  if (q0 >= 0) {
    own = R.rec[p];
    X0 = q0 % L.nx;
    Y0 = (q0 / L.nx) % L.ny;
    Z0 = q0 / (L.nx * L.ny);
  }
  const bool cells = R.fcell != nullptr, near_wall = R.fwall && q0 >= 0 && (R.bnode[q0] & 2);
  // bit s: node s = 9 (dz + 1) + 3 (dy + 1) + dx + 1 holds another cell
  unsigned others = 0;
  V3t<T> fw = {T(0), T(0), T(0)};
  if (q0 >= 0) {
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      const int s = 4 * k + part, dz = s / 9 - 1, dy = s / 3 % 3 - 1, dx = s % 3 - 1;
      if (s >= 27) continue;
      const int qb = rep_node(L, X0, Y0, Z0, dx, dy, dz);
      if (qb < 0) continue;
      if (cells) {
        const int o = R.node[qb].y;
        if (o != 0 && o != own.cell + 1) others |= 1u << s;
      }
      // bit 1 of the vertex's node: one of the 27 is a boundary node (bit 0)
      if (near_wall && (R.bnode[qb] & 1)) {
        const V3t<T> dv = {own.x - T(dx), own.y - T(dy), own.z - T(dz)};
        const T dist = sqrt(vdot(dv, dv));
        if (dist < R.rw) fw = fw + vscale(dv, R.kw * (R.rw / dist) / dist);
      }
    }
  }
  V3t<T> fc = {T(0), T(0), T(0)};
  if (cells) {
    others |= __shfl_xor_sync(0xffffffffu, others, 1);
    others |= __shfl_xor_sync(0xffffffffu, others, 2);
    const int n = __popc(others);
    int end = n;  // pairs up to this vertex's last
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += y;
    }
    const int total = __shfl_sync(0xffffffffu, end, 31), begin = end - n;
    if (part == 0) {
      s_own[w][v] = own;
      s_node[w][v] = q0;
      for (int k = begin; others; ++k, others &= others - 1) s_pair[w][k] = (uint8_t)(v << 5 | (__ffs(others) - 1));
    }
    for (int r = 0; r < total; r += 32) {
      __syncwarp();
      if (r + lane < total) {
        const int pair = s_pair[w][r + lane], u = pair >> 5;
        const V3t<T> f = rep_push(L, R, s_node[w][u], s_own[w][u], pair & 31);
        s_push[w][lane][0] = f.x;
        s_push[w][lane][1] = f.y;
        s_push[w][lane][2] = f.z;
      }
      __syncwarp();
      // the own pairs of this round, in the order of their nodes
      if (part == 0)
        for (int k = max(begin, r); k < min(end, r + 32); ++k)
          fc = fc + V3t<T>{s_push[w][k - r][0], s_push[w][k - r][1], s_push[w][k - r][2]};
    }
    if (in && part == 0) {
      R.fcell[p] = fc.x;
      R.fcell[V + p] = fc.y;
      R.fcell[2 * V + p] = fc.z;
    }
  }
  if (R.fwall) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      fw.x += __shfl_xor_sync(0xffffffffu, fw.x, o);
      fw.y += __shfl_xor_sync(0xffffffffu, fw.y, o);
      fw.z += __shfl_xor_sync(0xffffffffu, fw.z, o);
    }
    if (in && part == 0) {
      R.fwall[p] = fw.x;
      R.fwall[V + p] = fw.y;
      R.fwall[2 * V + p] = fw.z;
    }
  }
}

template <typename T>
cudaError_t launch_repulsion(const LbmView<T>& L, const VertexView<T>& vv, const RepView<T>& R, cudaStream_t s) {
  if (vv.nvert <= 0) return cudaSuccess;
  cudaError_t e = launch_kernel(k_rep_bin<T>, dim3((vv.nvert + 127) / 128), dim3(128), 0, s, L.pdl, L, vv, R);
  if (e != cudaSuccess) return e;
  constexpr int per = kRepWarps * kRepVertices;
  return launch_kernel(k_repulsion<T>, dim3((vv.nvert + per - 1) / per), dim3(kRepBlock), 0, s, L.pdl, L, vv, R);
}

// Tag the stencil nodes of every vertex (the interpolation run as a stage
// of its own, without the spread of the same step).
template <typename T>
__global__ void k_mark_nodes(const LbmView<T> L, const VertexView<T> vv) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= vv.nvert || !vv.alive[vv.vcell[i]]) return;
  const uint32_t stamp = *L.stamp;
  Kern<T> K;
  ibm_weights(L, vv.x[i], vv.x[vv.V + i], vv.x[2 * vv.V + i], K);
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (K.node[j] >= 0 && L.ntag) L.ntag[K.node[j]] = stamp;
}
template <typename T>
cudaError_t launch_mark_nodes(const LbmView<T>& L, const VertexView<T>& vv, cudaStream_t s) {
  if (vv.nvert <= 0) return cudaSuccess;
  return launch_kernel(k_mark_nodes<T>, dim3((vv.nvert + 255) / 256), dim3(256), 0, s, L.pdl, L, vv);
}

// External vertex forces (HemoCellStretch::applyForce adds them to the
// vertex force right before the spread, helper/hemoCellStretch.cpp:63-78).
template <typename T>
__global__ void k_add_vertex_forces(const VertexView<T> vv, const int* ids, const double* fext, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int i = ids[k];
  if (i < 0 || i >= vv.nvert) return;
  vv.f[i] += (T)fext[3 * k];
  vv.f[vv.V + i] += (T)fext[3 * k + 1];
  vv.f[2 * vv.V + i] += (T)fext[3 * k + 2];
}
template <typename T>
cudaError_t launch_add_vertex_forces(const VertexView<T>& vv, const int* ids, const double* fext, int n,
                                     cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_add_vertex_forces<T><<<(n + 127) / 128, 128, 0, s>>>(vv, ids, fext, n);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// K3+K5: interpolateFluidVelocity (core/hemoCellParticleField.cpp:819-839)
// from the node velocities of this step (L.unode), advanceParticles
// (:566-588, core/hemoCellParticle.h:188-203) and the per-vertex bin of
// update_pg (:137-168).  Thread 0 advances the device step stamp; no thread
// of this kernel reads it.
template <typename T>
__global__ void __launch_bounds__(256) k_interp_advance(const LbmView<T> L, const VertexView<T> vv, const TileGrid tg,
                                                        const int do_interp, const int do_advance) {
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *L.stamp += 1;
  if (i >= vv.nvert) return;
  const int cell = vv.vcell[i];
  if (!vv.alive[cell]) {
    vv.vnode[i] = -1;
    vv.vtile[i] = -1;
    return;
  }
  const long long V = vv.V;
  double px = vv.x[i], py = vv.x[V + i], pz = vv.x[2 * V + i];
  T vx, vy, vz;
  if (do_interp) {
    const V3t<T> u = ibm_velocity(L, px, py, pz);
    vx = u.x;
    vy = u.y;
    vz = u.z;
    vv.v[i] = vx;
    vv.v[V + i] = vy;
    vv.v[2 * V + i] = vz;
    if (!(is_finite(vx) && is_finite(vy) && is_finite(vz))) atomicOr(vv.status, 1u);
  } else {
    vx = vv.v[i];
    vy = vv.v[V + i];
    vz = vv.v[2 * V + i];
  }
  if (do_advance) {
    px += (double)vx;
    py += (double)vy;
    pz += (double)vz;
    vv.x[i] = px;
    vv.x[V + i] = py;
    vv.x[2 * V + i] = pz;
  }
  const double P[3] = {px, py, pz};
  const int dims[3] = {L.nx, L.ny, L.nz};
  int q[3];
  bool inside = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    long long qi = hcpos::nearest(P[a]);  // floor(P + 0.5), exactly
    if (qi < 0 || qi >= dims[a]) {
      if (L.per[a]) {
        long long mm = qi % dims[a];
        qi = mm < 0 ? mm + dims[a] : mm;
      } else {
        inside = false;
      }
    }
    q[a] = (int)qi;
  }
  if (!inside) {
    vv.vnode[i] = -1;
    vv.vtile[i] = -1;
    return;
  }
  const long long nd = (long long)q[0] + (long long)L.nx * ((long long)q[1] + (long long)L.ny * q[2]);
  vv.vnode[i] = (int)nd;
  vv.vtile[i] = q[0] / tg.tx + tg.ntx * (q[1] / tg.ty + tg.nty * (q[2] / tg.tz));
  if (do_advance && L.flag[nd] != 0) {
    vv.alive[cell] = 0;
    atomicOr(vv.status, 2u);
  }
  pdl_trigger();
}

template <typename T>
cudaError_t launch_interp_advance(const LbmView<T>& L, const VertexView<T>& vv, const TileGrid& tg, int do_interp,
                                  int do_advance, int bs, cudaStream_t s) {
  if (bs <= 0) bs = 128;
  const int n = vv.nvert > 0 ? vv.nvert : 1;  // one thread at least: it advances the stamp
  return launch_kernel(k_interp_advance<T>, dim3((n + bs - 1) / bs), dim3(bs), 0, s, L.pdl, L, vv, tg, do_interp,
                       do_advance);
}

// ---------------------------------------------------------------------------
// K4: constitutive models, one CTA per cell (grid-stride over the cell list).
// Saturation constants: config/constant_defaults.h:157-173.
constexpr double kMaxVol = 0.01, kMaxArea = 0.09, kMaxBend = 0.0555, kMaxPltBend = 2.467, kMaxLink = 9.0;
constexpr double kForceLimit = 50.0;

template <typename T>
__device__ __forceinline__ T vnorm(V3t<T> a) {
  return sqrt(vdot(a, a));
}
template <typename T>
__device__ __forceinline__ V3t<T> ld3(const T* s, int k) {
  return {s[3 * k], s[3 * k + 1], s[3 * k + 2]};
}
template <typename T>
__device__ __forceinline__ void add3(T* s, int k, V3t<T> v) {
  atomicAdd(s + 3 * k, v.x);
  atomicAdd(s + 3 * k + 1, v.y);
  atomicAdd(s + 3 * k + 2, v.z);
}
// Division and normalisation: IEEE in FP64 (the plain form follows the
// reference's arithmetic), fast reciprocal / rsqrt in the FP32 mixed form.
template <typename T>
__device__ __forceinline__ T fdiv(T a, T b) {
  return a / b;
}
template <>
__device__ __forceinline__ float fdiv<float>(float a, float b) {
  return __fdividef(a, b);
}
// v / |v| with |v| returned in len (len = 0 leaves v unnormalised)
template <typename T>
__device__ __forceinline__ V3t<T> normalized(V3t<T> v, T& len) {
  len = vnorm(v);
  if (len == T(0)) return v;
  return {v.x / len, v.y / len, v.z / len};
}
template <>
__device__ __forceinline__ V3t<float> normalized<float>(V3t<float> v, float& len) {
  const float d = vdot(v, v);
  if (d == 0.f) {
    len = 0.f;
    return v;
  }
  const float inv = rsqrtf(d);
  len = d * inv;
  return {v.x * inv, v.y * inv, v.z * inv};
}
template <typename T>
__device__ __forceinline__ T third(T a) {
  return a / T(3);
}
template <>
__device__ __forceinline__ float third<float>(float a) {
  return a * (1.0f / 3.0f);
}

template <typename T>
__device__ __forceinline__ V3t<T> unit_normal(V3t<T> a, V3t<T> b, V3t<T> c) {
  V3t<T> n = vcross(b - a, c - a);
  if constexpr (sizeof(T) == 8) {
    T inv, len;
    hcnewton::inv_length(vdot(n, n), inv, len);
    return vscale(n, inv);
  }
  const T l = vnorm(n);
  if (l != T(0)) return {n.x / l, n.y / l, n.z / l};
  return {T(0), T(0), T(0)};
}

// Doubles at the start of the force assembly's shared memory: one partial sum a
// warp of the largest block, the block's sum, the volume force and the same per area.
template <typename T>
constexpr int kMechThreads = sizeof(T) == 8 ? 384 : 768;
template <typename T>
constexpr int kSum = kMechThreads<T> / 32;
template <typename T>
constexpr int kVolumeForce = kSum<T> + 1;
template <typename T>
constexpr int kForcePerArea = kSum<T> + 2;
template <typename T>
constexpr int kMechHeader = kSum<T> + 3;
template <typename T>
__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    double s = lane < nw ? red[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) red[kSum<T>] = s;
  }
  __syncthreads();
  return red[kSum<T>];
}

template <typename T>
__device__ __forceinline__ T rest_value(const double* d, const float* f, int k);
template <>
__device__ __forceinline__ double rest_value<double>(const double* d, const float*, int k) {
  return d[k];
}
template <>
__device__ __forceinline__ float rest_value<float>(const double*, const float* f, int k) {
  return f[k];
}

// Cells on clusters of CTAs: rank r of a cluster owns a run of whole warps of
// the cell's vertices (and faces, edges): items [r c, (r + 1) c) with
// c = cluster_chunk(n, cluster size).
__host__ __device__ __forceinline__ int cluster_chunk(int n, int cluster) {
  return ((n + cluster - 1) / cluster + 31) / 32 * 32;
}
// The vertex-centric kernel's shared memory: positions, the own bending forces and
// the valences.  A cell on one CTA takes no more than its vertices: rounded up to
// whole warps, the largest types (4,731 vertices in FP64, 9,273 in FP32) would not fit.
__host__ __device__ __forceinline__ int gather_chunk(int nv, int cluster) {
  return cluster == 1 ? nv : cluster_chunk(nv, cluster);
}
template <typename T>
size_t mechanics_smem_bytes(int nv, int cluster) {
  return kMechHeader<T> * sizeof(double) + (3 * (size_t)nv + 3 * (size_t)gather_chunk(nv, cluster)) * sizeof(T) +
         (size_t)nv;
}
constexpr int kStagedHeader = 40;  // of the staged kernel, whose faces start on a 16-byte boundary
template <typename T>
__device__ __forceinline__ V3t<T> ld3_cluster(uint32_t a) {
  V3t<T> v;
  ld_cluster(a, v.x);
  ld_cluster(a + (uint32_t)sizeof(T), v.y);
  ld_cluster(a + 2u * (uint32_t)sizeof(T), v.z);
  return v;
}
template <typename Terms, typename T>
__device__ __forceinline__ V3t<T> ld3_terms(uint32_t a) {
  V3t<T> v;
  Terms::load(a, v.x);
  Terms::load(a + (uint32_t)sizeof(T), v.y);
  Terms::load(a + 2u * (uint32_t)sizeof(T), v.z);
  return v;
}
// the sum of a double over the ranks, in their order: the same bits in each
__device__ __forceinline__ double cluster_sum(const double* p, int cs) {
  double sum = 0.0;
  for (int r = 0; r < cs; ++r) {
    double part;
    ld_cluster(cluster_addr(smem_addr(p), (uint32_t)r), part);
    sum += part;
  }
  return sum;
}
// Where item k of an array cut into chunks lies: its address in the owner's
// shared memory.  magic = ceil(2^32 / chunk) makes the division exact for
// k * chunk < 2^32 (at most 19,000 faces in chunks of at most that many).
// ONE: the cell is one CTA's and every item its own.
template <bool ONE>
struct Chunked {
  uint32_t base, stride, magic;
  int chunk;
  __device__ __forceinline__ Chunked(const void* p, int chunk_, size_t stride_)
      : base(smem_addr(p)), stride((uint32_t)stride_), magic((uint32_t)((0x100000000ull + chunk_ - 1) / chunk_)),
        chunk(chunk_) {}
  __device__ __forceinline__ uint32_t owner(int k) const { return ONE ? 0u : __umulhi((uint32_t)k, magic); }
  __device__ __forceinline__ uint32_t within(int k, uint32_t own) const {
    return ONE ? (uint32_t)k : (uint32_t)k - own * (uint32_t)chunk;
  }
  __device__ __forceinline__ uint32_t at(int k, uint32_t own) const {
    const uint32_t a = base + within(k, own) * stride;
    return ONE ? a : cluster_addr(a, own);
  }
  __device__ __forceinline__ uint32_t at(int k) const { return at(k, owner(k)); }
  template <typename T>
  static __device__ __forceinline__ void load(uint32_t a, T& v) {
    if constexpr (ONE) ld_shared(a, v);
    else ld_cluster(a, v);
  }
  template <typename T>
  static __device__ __forceinline__ void load4(uint32_t a, T* v) {
    if constexpr (ONE) ld_shared4(a, v);
    else ld_cluster4(a, v);
  }
};
// six 16-bit indices in one 16-byte load (TypeDev)
struct Six {
  uint32_t w[4];
  __device__ __forceinline__ Six(const uint4* table, int i) {
    const uint4 v = table[i];
    w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
  }
  __device__ __forceinline__ int operator[](int j) const { return (int)(j & 1 ? w[j >> 1] >> 16 : w[j >> 1] & 0xffffu); }
};

// One CTA or cluster per cell (grid-stride over the cell list), vertex-centric: each
// thread owns vertices and sums, in a fixed order, every contribution the
// reference's face / edge / vertex loops deposit on them
// (rbcHighOrderModel.cpp:56-204, pltSimpleModel.cpp:59-205,
// wbcHighOrderModel.cpp:60-223).  Phase 1 sums the face volume terms and
// evaluates each vertex's own bending force into shared memory; after the
// block reduction of the volume, phase 2 gathers for each vertex: area and
// volume forces of its incident faces, link and membrane viscosity of its
// ring edges, the neighbours' bending reactions, the platelet dihedral terms
// of its incident and opposite edges, and its inner links.  No atomics: the
// forces are bit-reproducible.
template <typename T>
struct Face {
  V3t<T> n;  // unit normal
  T area;
  V3t<T> cen;
};

// platelet dihedral bending force of edge e (pltSimpleModel.cpp:156-182),
// +bfv on its end points, -bfv on the two outer points
template <typename T>
__device__ __forceinline__ V3t<T> plt_bending(const T* sx, const TypeDev& t, int e) {
  const int a = t.edges[2 * e], b = t.edges[2 * e + 1];
  const V3t<T> ev = ld3(sx, b) - ld3(sx, a);
  V3t<T> uv;
  if constexpr (sizeof(T) == 8) {
    T inv, len;
    hcnewton::inv_length(vdot(ev, ev), inv, len);
    uv = vscale(ev, inv);
  } else {
    const T L = vnorm(ev);
    uv = {ev.x / L, ev.y / L, ev.z / L};
  }
  const int* A = t.tris + 3 * t.bend_tris[2 * e];
  const int* B = t.tris + 3 * t.bend_tris[2 * e + 1];
  const V3t<T> V1 = unit_normal(ld3(sx, A[0]), ld3(sx, A[1]), ld3(sx, A[2]));
  const V3t<T> V2 = unit_normal(ld3(sx, B[0]), ld3(sx, B[1]), ld3(sx, B[2]));
  const T angle = atan2(vdot(vcross(V1, V2), uv), vdot(V1, V2));
  const T af = angle - rest_value<T>(t.edge_angle0, t.edge_angle0f, e);
  const T fm = (T)t.k_bend * (af + af / fabs(T(kMaxPltBend) - af * af));
  return vscale(V1 + V2, fm * T(0.5));
}

// spreadParticleForce of the next step for global vertex gi with the force
// just assembled (core/hemoCellParticleField.cpp:841-863): FORCE_LIMIT clamp
// (the stored force stays unclamped, as after the reference's constitutive
// model), plus the repulsion force, spread with the phi2 weights; the
// stencil nodes are tagged for the interpolation.  By whole warps, two lanes to
// a pair of vertices (pair_sides); a lane without a vertex (on clear) names any.
template <typename T>
__device__ __forceinline__ void spread_vertex(const MechView<T>& M, int gi, V3t<T> f, bool on) {
  const VertexView<T>& vv = M.vv;
  const long long V = vv.V;
  T mag = f.x * f.x;
  mag += f.y * f.y;
  mag += f.z * f.z;
  // the FP64 square root (ten FP64 instructions) only near or above the limit
  if (sizeof(T) == 4 || mag > T(0.999999) * M.f_limit * M.f_limit) {
    mag = sqrt(mag);
    if (mag > M.f_limit) f = vscale(f, M.f_limit / mag);
  }
  if (vv.frep_cell) f = f + V3t<T>{vv.frep_cell[gi], vv.frep_cell[V + gi], vv.frep_cell[2 * V + gi]};
  if (vv.frep_wall) f = f + V3t<T>{vv.frep_wall[gi], vv.frep_wall[V + gi], vv.frep_wall[2 * V + gi]};
  Kern<T> K;
  ibm_weights(M.L, vv.x[gi], vv.x[V + gi], vv.x[2 * V + gi], K);
  const uint32_t stamp = *M.L.stamp + (M.fuse_advance ? 1u : 0u);
  T* F = const_cast<T*>(M.L.Fcur);
  if (!on) {
#pragma unroll
    for (int s = 0; s < 8; ++s) K.node[s] = -1;
  }
  int node[8];
  T w[8];
  pair_sides(K.node, node);
  pair_sides(K.w, w);
  const V3t<T> other = {__shfl_xor_sync(0xffffffffu, f.x, 1), __shfl_xor_sync(0xffffffffu, f.y, 1),
                        __shfl_xor_sync(0xffffffffu, f.z, 1)};
  const bool odd = threadIdx.x & 1;
  const V3t<T> even_f = odd ? other : f, odd_f = odd ? f : other;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (node[j] < 0) continue;
    const V3t<T> g = vscale(j < 4 ? even_f : odd_f, w[j]);
    if (M.L.ntag) M.L.ntag[node[j]] = stamp;
    FieldLayout<T>::add(F, M.L.N, node[j], g.x, g.y, g.z);
  }
}

// Interpolation and advance of one cell's vertices by the CTA that then
// assembles its forces (the step's interpolate + advance stage fused in front
// of the constitutive model): velocity from the node velocities with the
// phi2 weights, Euler step, nearest node and tile, and the cell's deletion
// when a vertex reaches a wall node (core/hemoCellParticleField.cpp:566-588,
// :819-839).
// voff and alive are the cell's first vertex and its state before the step;
// `hit` is a shared flag the caller cleared before its last barrier.  Returns
// whether the cell is still alive; the deletion is written to the cell's state
// by thread 0.  Ends with a barrier: every vertex is advanced and binned.
// advance_range does vertices [k0, k1) of the cell, without the barrier.
template <typename T>
__device__ __forceinline__ void advance_range(const MechView<T>& M, int voff, int k0, int k1, bool alive, int& hit) {
  const VertexView<T>& vv = M.vv;
  const LbmView<T>& L = M.L;
  const long long V = vv.V;
  if (!alive) {
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
      vv.vnode[voff + k] = -1;
      vv.vtile[voff + k] = -1;
    }
    return;
  }
  // whole warps, whose last one's spare lanes follow its last vertex
  const int lane = threadIdx.x & 31;
  for (int kw = k0 + (int)threadIdx.x - lane; kw < k1; kw += blockDim.x) {
    const bool on = kw + lane < k1;
    const int i = voff + min(kw + lane, k1 - 1);
    double px = vv.x[i], py = vv.x[V + i], pz = vv.x[2 * V + i];
    const V3t<T> u = pair_velocity(L, px, py, pz, on);
    if (!on) continue;
    const T vx = u.x, vy = u.y, vz = u.z;
    vv.v[i] = vx;
    vv.v[V + i] = vy;
    vv.v[2 * V + i] = vz;
    if (!(is_finite(vx) && is_finite(vy) && is_finite(vz))) atomicOr(vv.status, STATUS_NONFINITE);
    px += (double)vx;
    py += (double)vy;
    pz += (double)vz;
    vv.x[i] = px;
    vv.x[V + i] = py;
    vv.x[2 * V + i] = pz;
    const double P[3] = {px, py, pz};
    const int dims[3] = {L.nx, L.ny, L.nz};
    int q[3];
    bool inside = true;
    for (int a = 0; a < 3; ++a) {
      long long qi = hcpos::nearest(P[a]);  // floor(P + 0.5), exactly
      if (qi < 0 || qi >= dims[a]) {
        if (L.per[a]) {
          const long long mm = qi % dims[a];
          qi = mm < 0 ? mm + dims[a] : mm;
        } else {
          inside = false;
        }
      }
      q[a] = (int)qi;
    }
    if (!inside) {
      vv.vnode[i] = -1;
      vv.vtile[i] = -1;
      continue;
    }
    const long long nd = (long long)q[0] + (long long)L.nx * ((long long)q[1] + (long long)L.ny * q[2]);
    vv.vnode[i] = (int)nd;
    vv.vtile[i] = q[0] / M.tg.tx + M.tg.ntx * (q[1] / M.tg.ty + M.tg.nty * (q[2] / M.tg.tz));
    if (L.flag[nd] != 0) hit = 1;
  }
}
// the rest areas and lengths of vertex i's slots
__device__ __forceinline__ void slot_rest(const TypeDev& t, int i, int, float a0[6], float l0[6]) {
  const float4 p = t.slot_f[3 * i], q = t.slot_f[3 * i + 1], r = t.slot_f[3 * i + 2];
  a0[0] = p.x, a0[1] = p.y, a0[2] = p.z, a0[3] = p.w, a0[4] = q.x, a0[5] = q.y;
  l0[0] = q.z, l0[1] = q.w, l0[2] = r.x, l0[3] = r.y, l0[4] = r.z, l0[5] = r.w;
}
__device__ __forceinline__ void slot_rest(const TypeDev& t, int i, int rn, double a0[6], double l0[6]) {
#pragma unroll
  for (int j = 0; j < 6; ++j)
    if (j < rn) {
      a0[j] = t.slot_a0[6 * i + j];
      l0[j] = t.slot_l0[6 * i + j];
    }
}

// The vertex-centric force assembly of one cell's vertices [v0, v1) and faces
// [f0, f1) by one rank of its cluster (variant 0; the staged variant falls back
// to it for FP32 cell types whose terms would not share an SM).  sx holds
// 3 nv T, the own bending forces and nv bytes of shared memory after `red`.
// Every rank of the cluster calls it: it holds the cluster's barriers.
template <typename T>
__device__ __forceinline__ void gather_cell(const MechView<T>& M, const TypeDev& t, int voff, bool alive, int cs,
                                            int rank, double* red, T* sx) {
  const VertexView<T>& vv = M.vv;
  const long long V = vv.V;
  const int tid = threadIdx.x, bs = blockDim.x;
  constexpr bool kF64 = sizeof(T) == 8;
  const int nv = t.nv, vch = gather_chunk(nv, cs), fch = cluster_chunk(t.nf, cs);
  const int v0 = min(rank * vch, nv), v1 = min(v0 + vch, nv);
  const int f0 = min(rank * fch, t.nf), f1 = min(f0 + fch, t.nf);
  T* sbf = sx + 3 * nv;  // own bending force per own vertex
  uint8_t* srn = reinterpret_cast<uint8_t*>(sbf + 3 * vch);  // valence per vertex
  if (!HC_IN(vv.status, (long long)voff + nv - 1, V)) return;  // the cell's vertices in the arrays (every rank returns)
  for (int k = tid; k < nv; k += bs) srn[k] = (uint8_t)(t.ring16[k].w & 0xffffu);
  // positions relative to the cell's vertex 0 (translation invariant forces;
  // the volume sum stays well conditioned far from the origin)
  const double r0x = vv.x[voff], r0y = vv.x[V + voff], r0z = vv.x[2 * V + voff];
  for (int k = tid; k < nv; k += bs) {
    sx[3 * k] = (T)(vv.x[voff + k] - r0x);
    sx[3 * k + 1] = (T)(vv.x[V + voff + k] - r0y);
    sx[3 * k + 2] = (T)(vv.x[2 * V + voff + k] - r0z);
  }
  __syncthreads();
  if (!alive) {
    for (int k = v0 + tid; k < v1; k += bs) {
      vv.f[voff + k] = T(0);
      vv.f[V + voff + k] = T(0);
      vv.f[2 * V + voff + k] = T(0);
    }
    return;
  }
  // --- phase 1: face volume terms, own bending force (rbcHighOrderModel.cpp:62-68, :127-157)
  double vol = 0.0;
  for (int k = f0 + tid; k < f1; k += bs) {
    const uint2 c = t.tris16[k];
    const V3t<T> v0 = ld3(sx, c.x & 0xffffu), v1 = ld3(sx, c.x >> 16), v2 = ld3(sx, c.y);
    if (kF64) {
      const double v210 = (double)v2.x * v1.y * v0.z, v120 = (double)v1.x * v2.y * v0.z;
      const double v201 = (double)v2.x * v0.y * v1.z, v021 = (double)v0.x * v2.y * v1.z;
      const double v102 = (double)v1.x * v0.y * v2.z, v012 = (double)v0.x * v1.y * v2.z;
      vol += (-v210 + v120 + v201 - v021 - v102 + v012);
    } else {
      // v0 . ((v1-v0) x (v2-v0)) == v0 . (v1 x v2): FP32 term, FP64 sum
      vol += (double)vdot(v0, vcross(v1 - v0, v2 - v0));
    }
  }
  if (t.model != 1) {
    for (int i = v0 + tid; i < v1; i += bs) {
      const Six rg(t.ring16, i);
      const int rn = rg[6];
      const V3t<T> xi = ld3(sx, i);
      V3t<T> sum = {T(0), T(0), T(0)};
#pragma unroll
      for (int j = 0; j < 6; ++j)
        if (j < rn) sum = sum + ld3(sx, rg[j]);
      const V3t<T> mid = {fdiv(sum.x, (T)rn), fdiv(sum.y, (T)rn), fdiv(sum.z, (T)rn)};
      const V3t<T> dev = mid - xi;
      V3t<T> pn = {T(0), T(0), T(0)};
      V3t<T> a = ld3(sx, rg[0]) - xi;
      const V3t<T> first = a;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        if (j >= rn) break;
        const V3t<T> b = (j + 1 < rn) ? ld3(sx, rg[j + 1]) - xi : first;
        T l;
        pn = pn + normalized(vcross(a, b), l);
        a = b;
      }
      T pl;
      pn = normalized(pn, pl);
      const T ndev = vdot(pn, dev);
      const T dDev = fdiv(ndev - rest_value<T>(t.patch_d0, t.patch_d0f, i), (T)t.edge_mean_eq);
      const V3t<T> bf = vscale(pn, (T)t.k_bend * (dDev + fdiv(dDev, fabs(T(kMaxBend) - dDev * dDev))));
      T* q = sbf + 3 * (i - v0);
      q[0] = bf.x;
      q[1] = bf.y;
      q[2] = bf.z;
    }
  }
  block_sum<T>(vol, red);  // red[kSum] = sum over the block
  cluster_sync(cs);
  const Chunked<false> bending(sbf, vch, 3 * sizeof(T));
  // volume constraint in FP64 (rbcHighOrderModel.cpp:100-104), by one thread
  if (tid == 0) {
    const double volume = cluster_sum(red + kSum<T>, cs) * (1.0 / 6.0);
    const double vfr = (volume - t.volume_eq) / t.volume_eq;
    const double vf = -t.k_volume * vfr / fabs(kMaxVol - vfr * vfr);
    red[kVolumeForce<T>] = vf;
    red[kForcePerArea<T>] = vf / t.area_mean_eq;
  }
  __syncthreads();
  const T vforce = (T)red[kVolumeForce<T>];
  const T vforce_per_area = (T)red[kForcePerArea<T>];
  const T area_mean = (T)t.area_mean_eq;
  const bool visc = (t.model != 0) || (t.eta_m != 0.0);
  // --- phase 2: gather per vertex
  for (int iw = v0 + (tid & ~31); iw < v1; iw += bs) {
    // whole warps, whose last one's spare lanes repeat its last vertex
    const int i = min(iw + (tid & 31), v1 - 1);
    const bool on = iw + (tid & 31) < v1;
    const Six rs(t.ring16, i);
    const int rn = rs[6];
    T a0s[6], l0s[6];
    slot_rest(t, i, rn, a0s, l0s);
    const V3t<T> xi = ld3(sx, i);
    V3t<T> f = {T(0), T(0), T(0)};
    V3t<T> vi = {T(0), T(0), T(0)};
    if (visc) vi = {vv.v[voff + i], vv.v[V + voff + i], vv.v[2 * V + voff + i]};
    int rot[6];
#pragma unroll
    for (int j = 0; j < 6; ++j) rot[j] = (rs[7] >> (2 * j)) & 3;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      if (j >= rn) break;
      const int r = rs[j];
      const int r1 = j + 1 < rn ? rs[j < 5 ? j + 1 : 0] : rs[0];
      // incident face (i, r, r1) in the reference's corner order: area force
      // on this corner and the face's volume force
      const V3t<T> xr = ld3(sx, r), xr1 = ld3(sx, r1);
      const V3t<T> c0 = rot[j] == 0 ? xi : (rot[j] == 1 ? xr1 : xr);
      const V3t<T> c1 = rot[j] == 0 ? xr : (rot[j] == 1 ? xi : xr1);
      const V3t<T> c2 = rot[j] == 0 ? xr1 : (rot[j] == 1 ? xr : xi);
      Face<T> F;
      {
        T nn;
        const V3t<T> n = normalized(vcross(c1 - c0, c2 - c0), nn);
        if (nn != T(0)) {
          F.area = T(0.5) * nn;
          F.n = n;
        } else {
          F.area = T(0);
          F.n = {T(0), T(0), T(0)};
        }
        F.cen = {third(c0.x + c1.x + c2.x), third(c0.y + c1.y + c2.y), third(c0.z + c1.z + c2.z)};
      }
      const T a0 = a0s[j];
      const T ar = fdiv(F.area - a0, a0);
      const T afm = (T)t.k_area * (ar + fdiv(ar, fabs(T(kMaxArea) - ar * ar)));
      f = f + vscale(F.cen - xi, afm);
      if (kF64) f = f + vscale(vscale(F.n, vforce), F.area / area_mean);
      else f = f + vscale(F.n, vforce_per_area * F.area);
      // ring edge (i, r): link force toward r when stretched, viscosity
      T L;
      const V3t<T> uv = normalized(xr - xi, L);
      const T l0 = l0s[j];
      const T ef = fdiv(L - l0, l0);
      f = f + vscale(uv, (T)t.k_link * (ef + fdiv(ef, fabs(T(kMaxLink) - ef * ef))));
      if (visc) {
        const V3t<T> vr = {vv.v[voff + r], vv.v[V + voff + r], vv.v[2 * V + voff + r]};
        V3t<T> fv = vscale(vscale(uv, vdot(vr - vi, uv)), (T)t.eta_m);
        const T mm = vnorm(fv);
        if (mm > T(kForceLimit / 4.0)) fv = vscale(fv, T(kForceLimit / 4.0) / mm);
        f = f + fv;
      }
      if (t.model != 1) {
        // neighbour's bending reaction -bf_r / n_r
        const T rnr = (T)srn[r];
        const V3t<T> b = ld3_cluster<T>(bending.at(r));
        f = f + V3t<T>{fdiv(-b.x, rnr), fdiv(-b.y, rnr), fdiv(-b.z, rnr)};
      } else {
        // platelet dihedral terms: end point of edge e, outer point of the opposite edge
        f = f + plt_bending(sx, t, t.vedge[6 * i + j]);
        f = f - plt_bending(sx, t, t.vopp[6 * i + j]);
      }
    }
    if (t.model != 1) f = f + ld3(sbf, i - v0);
    // inner links (pltSimpleModel.cpp:188-205, wbcHighOrderModel.cpp:202-223)
    for (int q = t.ni ? t.vinner_off[i] : 0, q1 = t.ni ? t.vinner_off[i + 1] : 0; q < q1; ++q) {
      const int e = t.vinner[q];
      const int o = t.inner[2 * e] == i ? t.inner[2 * e + 1] : t.inner[2 * e];
      const V3t<T> ev = ld3(sx, o) - xi;
      const T L = vnorm(ev);
      const V3t<T> uv = {ev.x / L, ev.y / L, ev.z / L};  // toward the partner
      if (t.model == 1) {
        const T l0 = rest_value<T>(t.inner_l0, t.inner_l0f, e);
        f = f + vscale(uv, (T)t.k_link * T(5) * ((L - l0) / l0));
      } else if (t.model == 2) {
        if (L < T(2) * (T)t.radius) f = f - vscale(vscale(uv, T(1) - L / (T(2) * (T)t.radius)), (T)t.k_cyto);
        if (L < T(2) * (T)t.core_radius)
          f = f - vscale(vscale(uv, T(1) - L / (T(2) * (T)t.core_radius)), (T)t.k_inner_rigid);
      }
    }
    if (on) {
      vv.f[voff + i] = f.x;
      vv.f[V + voff + i] = f.y;
      vv.f[2 * V + voff + i] = f.z;
    }
    if (M.fuse_spread) spread_vertex(M, voff + i, f, on);
  }
}

// The start of a cell's assembly, by every rank of its cluster: the type record
// into shared memory (set-up data, read before the programmatic wait), then with
// fuse_advance the interpolation and advance of the rank's vertices.  Returns
// whether the cell is alive; with fuse_advance the ranks are synchronised and
// every vertex is advanced.
template <typename T>
__device__ __forceinline__ bool begin_cell(const MechView<T>& M, int cell, int voff, int cs, int rank, TypeDev& t,
                                           int& hit) {
  const VertexView<T>& vv = M.vv;
  const int tid = threadIdx.x, lane = tid & 31;
  static_assert(sizeof(TypeDev) % 8 == 0, "copied in 8-byte words");
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(M.types + M.cell_type[cell]);
  for (int w = tid; w < (int)(sizeof(TypeDev) / 8); w += blockDim.x)
    reinterpret_cast<unsigned long long*>(&t)[w] = src[w];
  if (tid == 0) hit = 0;
  // Behind another type's launch: that one let this start after its own wait
  // for everything before it, and this one reads nothing that it writes.
  if (!M.after_prev) pdl_wait();
  if (M.before_next) pdl_trigger();
  bool alive = vv.alive[cell] != 0;
  __syncthreads();
  if (!M.fuse_advance) return alive;
  const int nv = t.nv, vch = cluster_chunk(nv, cs), v0 = min(rank * vch, nv);
  advance_range(M, voff, v0, min(v0 + vch, nv), alive, hit);
  cluster_sync(cs);
  // the ranks' flags together; rank 0 writes the cell's state, which every rank
  // read before the barrier
  int h = 0;
  for (int r = lane; r < cs; r += 32) h |= ld_cluster_int(cluster_addr(smem_addr(&hit), (uint32_t)r));
  const bool deleted = alive && __any_sync(0xffffffffu, h != 0);
  if (deleted && rank == 0 && tid == 0) {
    vv.alive[cell] = 0;
    atomicOr(vv.status, STATUS_CELL_DELETED);
  }
  return alive && !deleted;
}

// The end of a launch: the next kernel waits for this one alone, so this one may
// not end before the type's launch before it.
template <typename T>
__device__ __forceinline__ void end_launch(const MechView<T>& M) {
  if (M.after_prev && blockIdx.x == 0) pdl_wait();
  pdl_trigger();
}

template <typename T>
__global__ void __launch_bounds__(kMechThreads<T>) k_mechanics(const MechView<T> M) {
  extern __shared__ double smem_d[];
  __shared__ TypeDev tshared;
  __shared__ int hit;
  const int cs = (int)cluster_size(), rank = (int)cluster_rank();
  for (int ci = blockIdx.x / cs; ci < M.ncells; ci += gridDim.x / cs) {
    const int cell = M.cells[ci], voff = M.cell_voff[cell];
    const bool alive = begin_cell(M, cell, voff, cs, rank, tshared, hit);
    gather_cell(M, tshared, voff, alive, cs, rank, smem_d, reinterpret_cast<T*>(smem_d + kMechHeader<T>));
    cluster_sync(cs);  // no rank goes on or leaves while another reads its terms
  }
  end_launch(M);
}

// Staged variant (2): each cell on a cluster of 1 to 16 CTAs.  Rank r of the
// cluster owns a run of whole warps of the cell's vertices, faces and edges; it
// interpolates and advances its vertices, computes its faces' and edges' terms
// once into its own shared memory and gathers the forces of its vertices,
// reading the terms of other ranks through distributed shared memory.  Every
// rank holds all positions of the cell.
//
// What bounds it: in FP64 the FP64 pipe (two lanes an SM and cycle).  One CTA
// per cell left that pipe idle on every SM without a cell, and on all but one
// SM of a one-cell run; a vertex cost about 2100 FP64 instructions.  Here each
// face and edge is computed once, normalisation takes one reciprocal square
// root, saturation terms one reciprocal, the face's volume force is its cross
// product (area times unit normal), bending normals are the faces' and rest
// values come as reciprocals.  Area and link forces (and the membrane
// viscosity) act along the edges: a face gives each corner a third of its area
// scalar along both of the corner's edges, so a vertex needs one scalar per
// face and one per edge instead of two vectors.
//
// In FP32 latency bounds it: the chain of loads, barriers and reductions of one
// cell, two cells an SM (more CTAs or threads an SM leave the first-level cache
// too little room for the tables: 280 cells took 46 us, 52 to 59 with all of the
// SM's memory shared).  So the tables are 16-bit, one load a vertex instead of
// 18, and a cell on one CTA (ONE) reads its terms without a cluster's address
// mapping: 45.6 to 41.9 us for the pipe, 152 to 139 for 960 cells.  Splitting
// the last, nearly empty wave's cells over clusters made the latter 143.
//
// Shared layout after a header of 40 doubles: faces 4 words (cross product,
// area scalar) and 1 word (inverse length of the cross product) of the own
// chunk, own bending 4 vch (force, 1/valence), edge scalars ech, platelet
// dihedral 3 ech (platelets only), positions 3 nv.
template <typename T>
__host__ __device__ __forceinline__ size_t staged_smem_bytes(int model, int nv, int nf, int ne, int cluster) {
  const size_t words = 5 * (size_t)cluster_chunk(nf, cluster) + 4 * (size_t)cluster_chunk(nv, cluster) + 3 * (size_t)nv +
                       (size_t)cluster_chunk(ne, cluster) * (model == 1 ? 4 : 1);
  return kStagedHeader * sizeof(double) + words * sizeof(T);
}

// x + x / |limit - x^2|, the saturating response of every membrane term
__device__ __forceinline__ float saturating(float x, float limit) { return x + fdiv(x, fabsf(limit - x * x)); }
__device__ __forceinline__ double saturating(double x, double limit) {
  return fma(x, hcnewton::recip(fabs(fma(-x, x, limit))), x);
}
// (value - rest) / rest
__device__ __forceinline__ float strain(float v, const double*, const float* rest, const double*, int k) {
  const float r = rest[k];
  return fdiv(v - r, r);
}
__device__ __forceinline__ double strain(double v, const double* rest, const float*, const double* inv, int k) {
  return (v - rest[k]) * inv[k];
}
// 1 / n for a valence of 3 to 6
template <typename T>
__device__ __forceinline__ T inv_valence(int n) {
  return n == 6 ? T(1.0 / 6.0) : (n == 5 ? T(0.2) : (n == 4 ? T(0.25) : T(1.0 / 3.0)));
}
// a / b by a reciprocal: fast in both forms
__device__ __forceinline__ float quotient(float a, float b) { return fdiv(a, b); }
__device__ __forceinline__ double quotient(double a, double b) { return a * hcnewton::recip(b); }
// the same, rounded in FP32
__device__ __forceinline__ float ratio(float a, float b) { return a / b; }
__device__ __forceinline__ double ratio(double a, double b) { return quotient(a, b); }
template <typename T, bool ONE>
__global__ void __launch_bounds__(384, 2) k_mechanics_staged(const MechView<T> M) {
  extern __shared__ __align__(16) double smem_cluster[];
  __shared__ TypeDev t;
  __shared__ int hit;
  const int tid = threadIdx.x, bs = blockDim.x;
  const int cs = ONE ? 1 : (int)cluster_size(), rank = ONE ? 0 : (int)cluster_rank();
  const VertexView<T>& vv = M.vv;
  const long long V = vv.V;
  const int cell = M.cells[blockIdx.x / cs], voff = M.cell_voff[cell];
  bool alive = begin_cell(M, cell, voff, cs, rank, t, hit);
  const int nv = t.nv, nf = t.nf, ne = t.ne;
  const bool plt = t.model == 1, visc = (t.model != 0) || (t.eta_m != 0.0);
  const int vch = cluster_chunk(nv, cs), fch = cluster_chunk(nf, cs), ech = cluster_chunk(ne, cs);
  const int v0 = min(rank * vch, nv), v1 = min(v0 + vch, nv);
  const int f0 = min(rank * fch, nf), f1 = min(f0 + fch, nf);
  const int e0 = min(rank * ech, ne), e1 = min(e0 + ech, ne);
  double* red = smem_cluster;
  T* sface = reinterpret_cast<T*>(smem_cluster + kStagedHeader);
  T* sinv = sface + 4 * fch;
  T* sbf = sinv + fch;
  T* sedge = sbf + 4 * vch;
  T* splt = sedge + ech;
  T* sx = splt + (plt ? 3 * ech : 0);
  if (!HC_IN(vv.status, (long long)voff + nv - 1, V)) alive = false;
  if (!alive) {
    for (int k = v0 + tid; k < v1; k += bs) {
      if (!HC_IN(vv.status, voff + k, V)) break;
      vv.f[voff + k] = T(0);
      vv.f[V + voff + k] = T(0);
      vv.f[2 * V + voff + k] = T(0);
    }
    cluster_sync(cs);  // no rank leaves while another may still read its flag
    end_launch(M);
    return;
  }
  // positions relative to the cell's vertex 0
  const double r0x = vv.x[voff], r0y = vv.x[V + voff], r0z = vv.x[2 * V + voff];
  for (int k = tid; k < nv; k += bs) {
    sx[3 * k] = (T)(vv.x[voff + k] - r0x);
    sx[3 * k + 1] = (T)(vv.x[V + voff + k] - r0y);
    sx[3 * k + 2] = (T)(vv.x[2 * V + voff + k] - r0z);
  }
  __syncthreads();
  // --- own faces: six times the signed volume, area force, cross product
  double vol = 0.0;
  for (int k = f0 + tid; k < f1; k += bs) {
    const uint2 corner = t.tris16[k];
    const V3t<T> a = ld3(sx, corner.x & 0xffffu), b = ld3(sx, corner.x >> 16), c = ld3(sx, corner.y);
    const V3t<T> n = vcross(b - a, c - a);
    vol += (double)vdot(a, n);
    T inv, len;
    hcnewton::inv_length(vdot(n, n), inv, len);
    const T ar = strain(T(0.5) * len, t.tri_a0, t.tri_a0f, t.tri_ia0, k);
    T* q = sface + 4 * (k - f0);
    q[0] = n.x;
    q[1] = n.y;
    q[2] = n.z;
    q[3] = (T)t.k_area * saturating(ar, T(kMaxArea));
    sinv[k - f0] = inv;
  }
  // --- own edges: link and viscous force per edge vector, dihedral force
  for (int e = e0 + tid; e < e1; e += bs) {
    const uint32_t ends = t.edges16[e];
    const int a = (int)(ends & 0xffffu), b = (int)(ends >> 16);
    const V3t<T> d = ld3(sx, b) - ld3(sx, a);
    T inv, len;
    hcnewton::inv_length(vdot(d, d), inv, len);
    const T ef = strain(len, t.edge_l0, t.edge_l0f, t.edge_il0, e);
    T pull = (T)t.k_link * saturating(ef, T(kMaxLink));
    if (visc) {
      const V3t<T> va = {vv.v[voff + a], vv.v[V + voff + a], vv.v[2 * V + voff + a]};
      const V3t<T> vb = {vv.v[voff + b], vv.v[V + voff + b], vv.v[2 * V + voff + b]};
      const T fv = vdot(vb - va, d) * inv * (T)t.eta_m;
      const T lim = T(kForceLimit / 4.0);
      pull += fv > lim ? lim : (fv < -lim ? -lim : fv);
    }
    sedge[e - e0] = pull * inv;
    if (plt) {
      const V3t<T> pb = plt_bending(sx, t, e);
      T* p = splt + 3 * (e - e0);
      p[0] = pb.x;
      p[1] = pb.y;
      p[2] = pb.z;
    }
  }
  block_sum<T>(vol, red);  // red[kSum] = the own faces' sum
  cluster_sync(cs);
  using Terms = Chunked<ONE>;
  const Terms faces(sface, fch, 4 * sizeof(T)), edges(sedge, ech, sizeof(T)), dihedral(splt, ech, 3 * sizeof(T)),
      bending(sbf, vch, 4 * sizeof(T));
  const uint32_t inv_base = smem_addr(sinv);
  // --- volume constraint in FP64, by one thread of each rank, over the ranks'
  // sums in their order (the same bits in every rank); its warp's bending waits
  // for it, so there are no divisions in it (960 FP32 cells 127 us with, 122
  // without)
  if (tid == 0) {
    const double sum = ONE ? red[kSum<T>] : cluster_sum(red + kSum<T>, cs);
    const double vfr = (sum * (1.0 / 6.0) - t.volume_eq) * t.inv_volume_eq;
    red[kVolumeForce<T>] = -t.k_volume * vfr * hcnewton::recip(fabs(kMaxVol - vfr * vfr)) * t.inv_area_mean_eq;
  }
  // --- own bending forces, from the unit normals of the incident faces
  if (!plt) {
    for (int i = v0 + tid; i < v1; i += bs) {
      const Six ring(t.ring16, i), face(t.vface16, i);
      const int rn = ring[6];
      V3t<T> sum = {T(0), T(0), T(0)}, pn = {T(0), T(0), T(0)};
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        if (j >= rn) break;
        sum = sum + ld3(sx, ring[j]);
        const int k = face[j];
        const uint32_t owner = faces.owner(k);
        T q[4], s;
        Terms::load4(faces.at(k, owner), q);
        const uint32_t at = inv_base + (uint32_t)sizeof(T) * faces.within(k, owner);
        Terms::load(ONE ? at : cluster_addr(at, owner), s);
        pn = pn + vscale(V3t<T>{q[0], q[1], q[2]}, s);
      }
      T inv, len;
      hcnewton::inv_length(vdot(pn, pn), inv, len);
      // the mean's last place decides the deviation's fourth: in FP32 divided as
      // in the vertex-centric kernel, so that both agree
      const T part = inv_valence<T>(rn);
      V3t<T> dev = vscale(sum, part);
      if constexpr (sizeof(T) == 4) dev = {fdiv(sum.x, (T)rn), fdiv(sum.y, (T)rn), fdiv(sum.z, (T)rn)};
      dev = dev - ld3(sx, i);
      pn = vscale(pn, inv);
      const T d = quotient(vdot(pn, dev) - rest_value<T>(t.patch_d0, t.patch_d0f, i), (T)t.edge_mean_eq);
      const T s = (T)t.k_bend * saturating(d, T(kMaxBend));
      T* q = sbf + 4 * (i - v0);
      q[0] = pn.x * s;
      q[1] = pn.y * s;
      q[2] = pn.z * s;
      q[3] = part;
    }
  }
  cluster_sync(cs);
  const T push = T(0.5) * (T)red[kVolumeForce<T>];  // volume force per cross product
  // --- gather the own vertices' forces
  for (int iw = v0 + (tid & ~31); iw < v1; iw += bs) {
    // whole warps, whose last one's spare lanes repeat its last vertex
    const int i = min(iw + (tid & 31), v1 - 1);
    const bool on = iw + (tid & 31) < v1;
    const Six ring(t.ring16, i), face(t.vface16, i), edge(t.vedge16, i), opp(plt ? t.vopp16 : t.vedge16, i);
    const int rn = ring[6];
    const V3t<T> xi = ld3(sx, i);
    V3t<T> f = {T(0), T(0), T(0)}, n = {T(0), T(0), T(0)};
    T af[6], last = T(0);
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      if (j >= rn) break;
      T q[4];
      Terms::load4(faces.at(face[j]), q);
      n = n + V3t<T>{q[0], q[1], q[2]};
      af[j] = last = q[3];
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      if (j >= rn) break;
      const int r = ring[j], e = edge[j];
      T pull;
      Terms::load(edges.at(e), pull);
      // the edge's own scalar and a third of its two faces'
      const T c = pull + T(1.0 / 3.0) * (af[j] + (j == 0 ? last : af[j - 1]));
      f = f + vscale(ld3(sx, r) - xi, c);
      if (!plt) {
        T q[4];
        Terms::load4(bending.at(r), q);
        f = f - vscale(V3t<T>{q[0], q[1], q[2]}, q[3]);
      } else {
        f = f + ld3_terms<Terms, T>(dihedral.at(e)) - ld3_terms<Terms, T>(dihedral.at(opp[j]));
      }
    }
    f = f + vscale(n, push);
    if (!plt) f = f + V3t<T>{sbf[4 * (i - v0)], sbf[4 * (i - v0) + 1], sbf[4 * (i - v0) + 2]};
    for (int q = t.ni ? t.vinner_off[i] : 0, q1 = t.ni ? t.vinner_off[i + 1] : 0; q < q1; ++q) {
      const int e = t.vinner[q];
      const int o = t.inner[2 * e] == i ? t.inner[2 * e + 1] : t.inner[2 * e];
      const V3t<T> ev = ld3(sx, o) - xi;
      // the forces follow the small difference of two lengths: the rounded root and
      // quotients in FP32, as in the vertex-centric kernel (the same bits)
      T inv, len;
      V3t<T> uv;  // toward the partner
      if constexpr (sizeof(T) == 8) {
        hcnewton::inv_length(vdot(ev, ev), inv, len);
        uv = vscale(ev, inv);
      } else {
        len = vnorm(ev);
        uv = {ev.x / len, ev.y / len, ev.z / len};
      }
      if (plt) {
        const T l0 = rest_value<T>(t.inner_l0, t.inner_l0f, e);
        f = f + vscale(uv, (T)t.k_link * T(5) * ratio(len - l0, l0));
      } else if (t.model == 2) {
        const T d1 = T(2) * (T)t.radius, d2 = T(2) * (T)t.core_radius;
        if (len < d1) f = f - vscale(vscale(uv, T(1) - ratio(len, d1)), (T)t.k_cyto);
        if (len < d2) f = f - vscale(vscale(uv, T(1) - ratio(len, d2)), (T)t.k_inner_rigid);
      }
    }
    if (on) {
      vv.f[voff + i] = f.x;
      vv.f[V + voff + i] = f.y;
      vv.f[2 * V + voff + i] = f.z;
    }
    if (M.fuse_spread) spread_vertex(M, voff + i, f, on);
  }
  cluster_sync(cs);  // no rank leaves while another reads its terms
  end_launch(M);
}

template <typename T>
cudaError_t launch_mechanics_staged(const MechView<T>& M, int cluster, int bs, cudaStream_t s) {
  if (M.ncells <= 0) return cudaSuccess;
  return launch_cluster(cluster == 1 ? k_mechanics_staged<T, true> : k_mechanics_staged<T, false>, cluster, dim3(M.ncells * cluster), dim3(bs), M.dyn_smem, s, M.L.pdl,
                        M.carveout, M);
}
size_t mechanics_staged_bytes(int model, int nv, int nf, int ne, int cluster, bool f64) {
  return f64 ? staged_smem_bytes<double>(model, nv, nf, ne, cluster)
             : staged_smem_bytes<float>(model, nv, nf, ne, cluster);
}

// Scatter variant (selected by the tuner): one CTA per cell.  Pass A runs the faces
// (volume terms, area force); after the block reduction of the volume, pass B
// runs the volume force of every face, the bending of every vertex (RBC,
// WBC), every edge (link, membrane viscosity, platelet dihedral bending) and
// every inner link as one merged item loop.  Forces accumulate in shared
// memory and are written once.
template <typename T>
__global__ void __launch_bounds__(kMechThreads<T>) k_mechanics_scatter(const MechView<T> M) {
  pdl_wait();
  extern __shared__ double smem_d[];
  __shared__ TypeDev tshared;
  double* red = smem_d;
  T* sx = reinterpret_cast<T*>(smem_d + kMechHeader<T>);
  const VertexView<T>& vv = M.vv;
  const long long V = vv.V;
  const int tid = threadIdx.x, bs = blockDim.x;
  constexpr bool kF64 = sizeof(T) == 8;
  for (int ci = blockIdx.x; ci < M.ncells; ci += gridDim.x) {
    const int cell = M.cells[ci];
    __syncthreads();  // previous cell fully written out
    if (tid == 0) tshared = M.types[M.cell_type[cell]];
    __syncthreads();
    const TypeDev& t = tshared;
    const int nv = t.nv;
    const int voff = M.cell_voff[cell];
    T* sf = sx + 3 * nv;
    const bool alive = vv.alive[cell] != 0;
    const double r0x = vv.x[voff], r0y = vv.x[V + voff], r0z = vv.x[2 * V + voff];
    for (int k = tid; k < nv; k += bs) {
      sx[3 * k] = (T)(vv.x[voff + k] - r0x);
      sx[3 * k + 1] = (T)(vv.x[V + voff + k] - r0y);
      sx[3 * k + 2] = (T)(vv.x[2 * V + voff + k] - r0z);
      sf[3 * k] = T(0);
      sf[3 * k + 1] = T(0);
      sf[3 * k + 2] = T(0);
    }
    __syncthreads();
    if (alive) {
      // --- pass A: faces, volume terms and area force (rbcHighOrderModel.cpp:56-98)
      double vol = 0.0;
      for (int k = tid; k < t.nf; k += bs) {
        const int i0 = t.tris[3 * k], i1 = t.tris[3 * k + 1], i2 = t.tris[3 * k + 2];
        const V3t<T> v0 = ld3(sx, i0), v1 = ld3(sx, i1), v2 = ld3(sx, i2);
        V3t<T> n = vcross(v1 - v0, v2 - v0);
        if (kF64) {
          const double v210 = (double)v2.x * v1.y * v0.z, v120 = (double)v1.x * v2.y * v0.z;
          const double v201 = (double)v2.x * v0.y * v1.z, v021 = (double)v0.x * v2.y * v1.z;
          const double v102 = (double)v1.x * v0.y * v2.z, v012 = (double)v0.x * v1.y * v2.z;
          vol += (-v210 + v120 + v201 - v021 - v102 + v012);
        } else {
          // v0 . ((v1-v0) x (v2-v0)) == v0 . (v1 x v2): FP32 term, FP64 sum
          vol += (double)vdot(v0, n);
        }
        const T nn = vnorm(n);
        T area;
        if (nn != T(0)) {
          area = T(0.5) * nn;
          n = {n.x / nn, n.y / nn, n.z / nn};
        } else {
          area = T(0);
        }
        const T a0 = rest_value<T>(t.tri_a0, t.tri_a0f, k);
        const T ar = (area - a0) / a0;
        const T afm = (T)t.k_area * (ar + ar / fabs(T(kMaxArea) - ar * ar));
        const V3t<T> cen = {(v0.x + v1.x + v2.x) / T(3), (v0.y + v1.y + v2.y) / T(3), (v0.z + v1.z + v2.z) / T(3)};
        add3(sf, i0, vscale(cen - v0, afm));
        add3(sf, i1, vscale(cen - v1, afm));
        add3(sf, i2, vscale(cen - v2, afm));
      }
      const double volume = block_sum<T>(vol, red) * (1.0 / 6.0);
      // volume constraint in FP64 (rbcHighOrderModel.cpp:100-104)
      const double vfr = (volume - t.volume_eq) / t.volume_eq;
      const double vforce = -t.k_volume * vfr / fabs(kMaxVol - vfr * vfr);
      const T vforce_per_area = (T)(vforce / t.area_mean_eq);
      const bool visc = (t.model != 0) || (t.eta_m != 0.0);
      const int nb = (t.model != 1) ? nv : 0;
      const int e0 = t.nf + nb, e1 = e0 + t.ne, total = e1 + t.ni;
      // --- pass B: volume force, bending, edges, inner links
      for (int k = tid; k < total; k += bs) {
        if (k < t.nf) {
          // volume force per face (rbcHighOrderModel.cpp:103-124)
          const int i0 = t.tris[3 * k], i1 = t.tris[3 * k + 1], i2 = t.tris[3 * k + 2];
          const V3t<T> v0 = ld3(sx, i0), v1 = ld3(sx, i1), v2 = ld3(sx, i2);
          V3t<T> n = vcross(v1 - v0, v2 - v0);
          const T nn = vnorm(n);
          T area;
          if (nn != T(0)) {
            area = T(0.5) * nn;
            n = {n.x / nn, n.y / nn, n.z / nn};
          } else {
            area = T(0);
            n = {T(0), T(0), T(0)};
          }
          V3t<T> lvf;
          if (kF64) lvf = vscale(vscale(n, (T)vforce), area / (T)t.area_mean_eq);
          else lvf = vscale(n, vforce_per_area * area);
          add3(sf, i0, lvf);
          add3(sf, i1, lvf);
          add3(sf, i2, lvf);
        } else if (k < e0) {
          // bending per vertex (rbcHighOrderModel.cpp:127-166)
          const int i = k - t.nf;
          const int rn = t.ring_n[i];
          const int* rg = t.ring + 6 * i;
          const V3t<T> xi = ld3(sx, i);
          V3t<T> sum = {T(0), T(0), T(0)};
          for (int j = 0; j < rn; ++j) sum = sum + ld3(sx, rg[j]);
          const V3t<T> mid = {sum.x / (T)rn, sum.y / (T)rn, sum.z / (T)rn};
          const V3t<T> dev = mid - xi;
          V3t<T> pn = {T(0), T(0), T(0)};
          V3t<T> a = ld3(sx, rg[0]) - xi;
          const V3t<T> first = a;
          for (int j = 0; j < rn; ++j) {
            const V3t<T> b = (j + 1 < rn) ? ld3(sx, rg[j + 1]) - xi : first;
            V3t<T> tn = vcross(a, b);
            const T l = vnorm(tn);
            pn = pn + V3t<T>{tn.x / l, tn.y / l, tn.z / l};
            a = b;
          }
          const T pl = vnorm(pn);
          pn = {pn.x / pl, pn.y / pl, pn.z / pl};
          const T ndev = vdot(pn, dev);
          const T dDev = (ndev - rest_value<T>(t.patch_d0, t.patch_d0f, i)) / (T)t.edge_mean_eq;
          const V3t<T> bf = vscale(pn, (T)t.k_bend * (dDev + dDev / fabs(T(kMaxBend) - dDev * dDev)));
          add3(sf, i, bf);
          const V3t<T> nbf = {-bf.x / (T)rn, -bf.y / (T)rn, -bf.z / (T)rn};
          for (int j = 0; j < rn; ++j) add3(sf, rg[j], nbf);
        } else if (k < e1) {
          // link, membrane viscosity, platelet dihedral bending
          const int e = k - e0;
          const int a = t.edges[2 * e], b = t.edges[2 * e + 1];
          const V3t<T> p0 = ld3(sx, a), p1 = ld3(sx, b);
          const V3t<T> ev = p1 - p0;
          const T L = vnorm(ev);
          const V3t<T> uv = {ev.x / L, ev.y / L, ev.z / L};
          const T l0 = rest_value<T>(t.edge_l0, t.edge_l0f, e);
          const T ef = (L - l0) / l0;
          const T fs = (T)t.k_link * (ef + ef / fabs(T(kMaxLink) - ef * ef));
          const V3t<T> force = vscale(uv, fs);
          V3t<T> fa = force, fb = {-force.x, -force.y, -force.z};
          if (visc) {
            const V3t<T> va = {vv.v[voff + a], vv.v[V + voff + a], vv.v[2 * V + voff + a]};
            const V3t<T> vb = {vv.v[voff + b], vv.v[V + voff + b], vv.v[2 * V + voff + b]};
            V3t<T> fv = vscale(vscale(uv, vdot(vb - va, uv)), (T)t.eta_m);
            const T mm = vnorm(fv);
            if (mm > T(kForceLimit / 4.0)) fv = vscale(fv, T(kForceLimit / 4.0) / mm);
            fa = fa + fv;
            fb = fb - fv;
          }
          if (t.model == 1) {  // pltSimpleModel.cpp:156-182
            const int* A = t.tris + 3 * t.bend_tris[2 * e];
            const int* B = t.tris + 3 * t.bend_tris[2 * e + 1];
            const V3t<T> V1 = unit_normal(ld3(sx, A[0]), ld3(sx, A[1]), ld3(sx, A[2]));
            const V3t<T> V2 = unit_normal(ld3(sx, B[0]), ld3(sx, B[1]), ld3(sx, B[2]));
            const T angle = atan2(vdot(vcross(V1, V2), uv), vdot(V1, V2));
            const T af = angle - rest_value<T>(t.edge_angle0, t.edge_angle0f, e);
            const T fm = (T)t.k_bend * (af + af / fabs(T(kMaxPltBend) - af * af));
            const V3t<T> bfv = vscale(V1 + V2, fm * T(0.5));
            fa = fa + bfv;
            fb = fb + bfv;
            const V3t<T> nbv = {-bfv.x, -bfv.y, -bfv.z};
            add3(sf, t.bend_outer[2 * e], nbv);
            add3(sf, t.bend_outer[2 * e + 1], nbv);
          }
          add3(sf, a, fa);
          add3(sf, b, fb);
        } else {
          // inner links
          const int e = k - e1;
          const int a = t.inner[2 * e], b = t.inner[2 * e + 1];
          const V3t<T> ev = ld3(sx, b) - ld3(sx, a);
          const T L = vnorm(ev);
          const V3t<T> uv = {ev.x / L, ev.y / L, ev.z / L};
          if (t.model == 1) {  // pltSimpleModel.cpp:188-205
            const T l0 = rest_value<T>(t.inner_l0, t.inner_l0f, e);
            const T ef = (L - l0) / l0;
            const V3t<T> force = vscale(uv, (T)t.k_link * T(5) * ef);
            add3(sf, a, force);
            add3(sf, b, V3t<T>{-force.x, -force.y, -force.z});
          } else if (t.model == 2) {  // wbcHighOrderModel.cpp:202-223
            if (L < T(2) * (T)t.radius) {
              const V3t<T> force = vscale(vscale(uv, T(1) - L / (T(2) * (T)t.radius)), (T)t.k_cyto);
              add3(sf, a, V3t<T>{-force.x, -force.y, -force.z});
              add3(sf, b, force);
            }
            if (L < T(2) * (T)t.core_radius) {
              const V3t<T> force = vscale(vscale(uv, T(1) - L / (T(2) * (T)t.core_radius)), (T)t.k_inner_rigid);
              add3(sf, a, V3t<T>{-force.x, -force.y, -force.z});
              add3(sf, b, force);
            }
          }
        }
      }
    }
    __syncthreads();
    for (int k = tid; k < nv; k += bs) {
      vv.f[voff + k] = sf[3 * k];
      vv.f[V + voff + k] = sf[3 * k + 1];
      vv.f[2 * V + voff + k] = sf[3 * k + 2];
    }
  }
}

// Raise the kernels' dynamic shared-memory limits (done when a cell type is
// added, never inside a stream capture).  The attribute belongs to the kernel,
// not to a handle: it goes to the device's maximum, so that no handle lowers it
// beneath what another one launches with.  staged_limit receives the staged
// kernel's.
template <typename T>
cudaError_t prepare_mechanics(int smem_bytes, int* staged_limit) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  void (*kernels[4])(const MechView<T>) = {k_mechanics<T>, k_mechanics_scatter<T>, k_mechanics_staged<T, true>,
                                           k_mechanics_staged<T, false>};
  for (int k = 0; k < 4; ++k) {
    cudaFuncAttributes a;
    if ((e = cudaFuncGetAttributes(&a, kernels[k])) != cudaSuccess) return e;
    const int room = optin - (int)a.sharedSizeBytes;
    if (k < 2 && smem_bytes > room) return cudaErrorInvalidValue;
    e = cudaFuncSetAttribute(kernels[k], cudaFuncAttributeMaxDynamicSharedMemorySize, room);
    if (e != cudaSuccess) return e;
    if (k >= 2) *staged_limit = k == 2 ? room : std::min(*staged_limit, room);
  }
  e = cudaFuncSetAttribute(k_mechanics<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_mechanics_staged<T, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}

template <typename T>
bool mechanics_cluster_fits(bool staged, int cluster, int bs, int smem_bytes) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(bs);
  cfg.dynamicSmemBytes = smem_bytes;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)cluster;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, staged ? k_mechanics_staged<T, false> : k_mechanics<T>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n > 0;
}

// variant 0: vertex-centric gather (deterministic), 1: face/edge scatter with
// shared-memory atomics
template <typename T>
cudaError_t launch_mechanics(const MechView<T>& M, int cluster, int bs, int grid, int variant, cudaStream_t s) {
  if (M.ncells <= 0) return cudaSuccess;
  if (bs <= 0) bs = 256;
  if (bs > kMechThreads<T>) bs = kMechThreads<T>;
  if (grid <= 0 || grid > M.ncells) grid = M.ncells;
  if (variant == 1) return launch_kernel(k_mechanics_scatter<T>, dim3(grid), dim3(bs), M.dyn_smem, s, M.L.pdl, M);
  return launch_cluster(k_mechanics<T>, cluster, dim3(grid * cluster), dim3(bs), M.dyn_smem, s, M.L.pdl, M.carveout, M);
}

// device [3][Vcap] (T) -> [V][3] double
template <typename T>
__global__ void k_soa_to_aos(const T* src, double* dst, long long V, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  dst[3 * (long long)i] = (double)src[i];
  dst[3 * (long long)i + 1] = (double)src[V + i];
  dst[3 * (long long)i + 2] = (double)src[2 * V + i];
}
template <typename T>
cudaError_t launch_soa_to_aos(const T* src, double* dst, long long V, int n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_soa_to_aos<T><<<(n + 255) / 256, 256, 0, s>>>(src, dst, V, n);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Per-vertex nearest node and tile from the current positions (update_pg,
// core/hemoCellParticleField.cpp:137-168): bin = floor(x+0.5) wrapped on
// periodic axes; vertices of removed cells or off a non-periodic axis get -1.
template <typename T>
__global__ void k_bin_vertices(const LbmView<T> L, const VertexView<T> vv, const TileGrid tg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= vv.nvert) return;
  const long long V = vv.V;
  const double P[3] = {vv.x[i], vv.x[V + i], vv.x[2 * V + i]};
  const int dims[3] = {L.nx, L.ny, L.nz};
  int q[3];
  bool inside = vv.alive[vv.vcell[i]] != 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    long long qi = hcpos::nearest(P[a]);  // floor(P + 0.5), exactly
    if (qi < 0 || qi >= dims[a]) {
      if (L.per[a]) {
        long long mm = qi % dims[a];
        qi = mm < 0 ? mm + dims[a] : mm;
      } else {
        inside = false;
      }
    }
    q[a] = (int)qi;
  }
  if (!inside) {
    vv.vnode[i] = -1;
    vv.vtile[i] = -1;
    return;
  }
  vv.vnode[i] = q[0] + L.nx * (q[1] + L.ny * q[2]);
  vv.vtile[i] = q[0] / tg.tx + tg.ntx * (q[1] / tg.ty + tg.nty * (q[2] / tg.tz));
}
template <typename T>
cudaError_t launch_bin_vertices(const LbmView<T>& L, const VertexView<T>& vv, const TileGrid& tg, cudaStream_t s) {
  if (vv.nvert <= 0) return cudaSuccess;
  k_bin_vertices<T><<<(vv.nvert + 255) / 256, 256, 0, s>>>(L, vv, tg);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Binning CSR: counts per tile, exclusive scan, fill, per-tile sort by vertex
// id (vertex ids grow with (cell, vertex id)), then per-tile unique cells.
__global__ void k_bin_count(const int* vtile, int nvert, int* counts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nvert) return;
  const int t = vtile[i];
  if (t >= 0) atomicAdd(counts + t, 1);
}

// single-CTA exclusive scan of n ints into out[0..n]
__global__ void k_scan(const int* in, int n, int* out) {
  __shared__ int carry;
  __shared__ int warp_sums[32];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += blockDim.x) {
    const int i = base + threadIdx.x;
    int v = i < n ? in[i] : 0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
      const int nw = blockDim.x >> 5;
      int s = lane < nw ? warp_sums[lane] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
      }
      if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    const int incl = x + (wid > 0 ? warp_sums[wid - 1] : 0);
    if (i < n) out[i] = carry + incl - v;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry += incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}

__global__ void k_bin_fill(const int* vtile, int nvert, const int* offsets, int* cursor, int* tile_vertices) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nvert) return;
  const int t = vtile[i];
  if (t < 0) return;
  const int pos = offsets[t] + atomicAdd(cursor + t, 1);
  tile_vertices[pos] = i;
}

// One CTA per tile: rank sort of the segment in shared memory (keys are
// unique vertex ids; a segment beyond 2048 takes a sorting network in place),
// then the number of distinct cells in the sorted segment.
__global__ void k_bin_sort(const int* offsets, int* tile_vertices, const int* vcell, int* tile_cell_counts) {
  __shared__ int buf[2048];
  __shared__ int ncell;
  const int t = blockIdx.x;
  const int b = offsets[t], e = offsets[t + 1], len = e - b;
  if (threadIdx.x == 0) ncell = 0;
  if (len <= 0) {
    if (threadIdx.x == 0) tile_cell_counts[t] = 0;
    return;
  }
  if (len <= 2048) {
    for (int k = threadIdx.x; k < len; k += blockDim.x) buf[k] = tile_vertices[b + k];
    __syncthreads();
    int out[8];
    int cnt = 0;
    for (int k = threadIdx.x; k < len; k += blockDim.x) {
      const int key = buf[k];
      int r = 0;
      for (int j = 0; j < len; ++j) r += buf[j] < key;
      out[cnt++] = r;
    }
    __syncthreads();
    cnt = 0;
    int keys[8];
    for (int k = threadIdx.x; k < len; k += blockDim.x) keys[cnt++] = buf[k];
    __syncthreads();
    cnt = 0;
    for (int k = threadIdx.x; k < len; k += blockDim.x) {
      buf[out[cnt]] = keys[cnt];
      cnt++;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < len; k += blockDim.x) tile_vertices[b + k] = buf[k];
    int local = 0;
    for (int k = threadIdx.x; k < len; k += blockDim.x)
      local += (k == 0 || vcell[buf[k]] != vcell[buf[k - 1]]) ? 1 : 0;
    atomicAdd(&ncell, local);
    __syncthreads();
    if (threadIdx.x == 0) tile_cell_counts[t] = ncell;
  } else {
    // A segment beyond the shared buffer is sorted in place in global memory
    // by the whole CTA: Batcher's bitonic network in its all-ascending form
    // (each merge starts by comparing element i with its mirror in the block
    // of size k, then halves the stride), over the length padded to a power
    // of two with +infinity.  A pair whose upper element lies in the padding
    // already holds the smaller key below, so it is skipped, and no index
    // past the segment is touched.  O(len log^2 len) / blockDim.x steps.
    int* seg = tile_vertices + b;
    int p2 = 1;
    while (p2 < len) p2 <<= 1;
    for (int k = 2; k <= p2; k <<= 1) {
      for (int j = k >> 1; j >= 1; j >>= 1) {
        // the first pass of a merge pairs i with its mirror in the k-block,
        // the later ones with i + j
        for (int q = threadIdx.x; q < p2 / 2; q += blockDim.x) {
          const int i = (q / j) * 2 * j + (q % j);       // lower element of pair q
          const int u = (j == k >> 1) ? (i | (k - 1)) - (i & (k - 1)) : i + j;
          if (u < len) {
            const int a = seg[i], c = seg[u];
            if (a > c) {
              seg[i] = c;
              seg[u] = a;
            }
          }
        }
        __syncthreads();
      }
    }
    int local = 0;
    for (int k = threadIdx.x; k < len; k += blockDim.x)
      local += (k == 0 || vcell[seg[k]] != vcell[seg[k - 1]]) ? 1 : 0;
    atomicAdd(&ncell, local);
    __syncthreads();
    if (threadIdx.x == 0) tile_cell_counts[t] = ncell;
  }
}

__global__ void k_tile_cells(const int* offsets, const int* tile_vertices, const int* vcell, int ntiles,
                             const int* tile_cell_offsets, int* tile_cells, int max_cells) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  int o = tile_cell_offsets[t];
  for (int k = offsets[t]; k < offsets[t + 1]; ++k) {
    const int c = vcell[tile_vertices[k]];
    if (k == offsets[t] || c != vcell[tile_vertices[k - 1]]) {
      if (o < max_cells) tile_cells[o] = c;
      o++;
    }
  }
}

cudaError_t launch_bin_csr(const int* vtile, int nvert, int ntiles, int* counts, int* offsets, int* cursor,
                           int* tile_vertices, const int* vcell, int* tile_cell_counts, cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(counts, 0, sizeof(int) * ntiles, s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(cursor, 0, sizeof(int) * ntiles, s)) != cudaSuccess) return e;
  if (nvert > 0) k_bin_count<<<(nvert + 255) / 256, 256, 0, s>>>(vtile, nvert, counts);
  k_scan<<<1, 1024, 0, s>>>(counts, ntiles, offsets);
  if (nvert > 0) k_bin_fill<<<(nvert + 255) / 256, 256, 0, s>>>(vtile, nvert, offsets, cursor, tile_vertices);
  k_bin_sort<<<ntiles, 256, 0, s>>>(offsets, tile_vertices, vcell, tile_cell_counts);
  return cudaGetLastError();
}

cudaError_t launch_tile_cells(const int* offsets, const int* tile_vertices, const int* vcell, int ntiles,
                              int* tile_cell_counts, int* tile_cell_offsets, int* tile_cells, int max_cells,
                              cudaStream_t s) {
  k_scan<<<1, 1024, 0, s>>>(tile_cell_counts, ntiles, tile_cell_offsets);
  k_tile_cells<<<(ntiles + 255) / 256, 256, 0, s>>>(offsets, tile_vertices, vcell, ntiles, tile_cell_offsets,
                                                    tile_cells, max_cells);
  return cudaGetLastError();
}

cudaError_t launch_exclusive_scan(const int* in, int n, int* out, cudaStream_t s) {
  k_scan<<<1, 1024, 0, s>>>(in, n, out);
  return cudaGetLastError();
}

// Neighbour lists (the cells within the kernel halo of a tile): for tile t,
// the distinct cells with vertices in t or in one of its 26 neighbouring
// tiles (wrapped on periodic axes, cut at the others), ascending.  A 27-way
// merge of the tiles' ascending cell lists (tile_cell_offsets / tile_cells);
// `out` null counts only.
__device__ int tile_neighbour_cells(const TileGrid tg, int per_x, int per_y, int per_z, const int* tco,
                                    const int* tcells, int t, int* out) {
  const int tx = t % tg.ntx, ty = (t / tg.ntx) % tg.nty, tz = t / (tg.ntx * tg.nty);
  const int per[3] = {per_x, per_y, per_z};
  const int n3[3] = {tg.ntx, tg.nty, tg.ntz};
  int pos[27], end[27], tid[27], nl = 0;
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        int c[3] = {tx + dx, ty + dy, tz + dz};
        bool ok = true;
        for (int a = 0; a < 3; ++a) {
          if (c[a] < 0 || c[a] >= n3[a]) {
            if (per[a]) c[a] = (c[a] + n3[a]) % n3[a];
            else ok = false;
          }
        }
        if (!ok) continue;
        const int nt = c[0] + tg.ntx * (c[1] + tg.nty * c[2]);
        bool dup = false;  // a small periodic grid wraps onto the same tile
        for (int k = 0; k < nl; ++k)
          if (tid[k] == nt) dup = true;
        if (dup) continue;
        tid[nl] = nt;
        pos[nl] = tco[nt];
        end[nl] = tco[nt + 1];
        ++nl;
      }
  int count = 0, last = -1;
  for (;;) {
    int best = -1;
    for (int k = 0; k < nl; ++k)
      if (pos[k] < end[k] && (best < 0 || tcells[pos[k]] < best)) best = tcells[pos[k]];
    if (best < 0) break;
    for (int k = 0; k < nl; ++k)
      while (pos[k] < end[k] && tcells[pos[k]] == best) ++pos[k];
    if (best != last) {
      if (out) out[count] = best;
      ++count;
      last = best;
    }
  }
  return count;
}

__global__ void k_tile_neighbours(const TileGrid tg, int px, int py, int pz, const int* tco, const int* tcells,
                                  int ntiles, int* counts, const int* offsets, int* cells) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  if (offsets) tile_neighbour_cells(tg, px, py, pz, tco, tcells, t, cells + offsets[t]);
  else counts[t] = tile_neighbour_cells(tg, px, py, pz, tco, tcells, t, nullptr);
}

cudaError_t launch_tile_neighbours(const TileGrid& tg, const int per[3], const int* tile_cell_offsets,
                                   const int* tile_cells, int ntiles, int* counts, const int* offsets, int* cells,
                                   cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  k_tile_neighbours<<<(ntiles + 127) / 128, 128, 0, s>>>(tg, per[0], per[1], per[2], tile_cell_offsets, tile_cells,
                                                         ntiles, counts, offsets, cells);
  return cudaGetLastError();
}

cudaError_t launch_tile_sort(const int* offsets, int* tile_vertices, const int* vcell, int ntiles,
                             int* tile_cell_counts, cudaStream_t s) {
  k_bin_sort<<<ntiles, 256, 0, s>>>(offsets, tile_vertices, vcell, tile_cell_counts);
  return cudaGetLastError();
}

#define HC_CELL_INST(T)                                                                                        \
  template cudaError_t launch_spread<T>(const LbmView<T>&, const VertexView<T>&, double, int, cudaStream_t);   \
  template cudaError_t launch_mark_nodes<T>(const LbmView<T>&, const VertexView<T>&, cudaStream_t);            \
  template cudaError_t launch_cell_info<T>(const VertexView<T>&, const int*, const int*, const TypeDev*, int,   \
                                           double*, cudaStream_t);                                             \
  template cudaError_t launch_repulsion<T>(const LbmView<T>&, const VertexView<T>&, const RepView<T>&,          \
                                           cudaStream_t);                                                      \
  template cudaError_t launch_add_vertex_forces<T>(const VertexView<T>&, const int*, const double*, int,       \
                                                   cudaStream_t);                                              \
  template cudaError_t launch_interp_advance<T>(const LbmView<T>&, const VertexView<T>&, const TileGrid&, int, \
                                                int, int, cudaStream_t);                                       \
  template cudaError_t launch_mechanics<T>(const MechView<T>&, int, int, int, int, cudaStream_t);              \
  template cudaError_t launch_mechanics_staged<T>(const MechView<T>&, int, int, cudaStream_t);                \
  template size_t mechanics_smem_bytes<T>(int, int);                                                           \
  template cudaError_t prepare_mechanics<T>(int, int*);                                                        \
  template bool mechanics_cluster_fits<T>(bool, int, int, int);                                                \
  template cudaError_t launch_soa_to_aos<T>(const T*, double*, long long, int, cudaStream_t);                  \
  template cudaError_t launch_bin_vertices<T>(const LbmView<T>&, const VertexView<T>&, const TileGrid&,         \
                                              cudaStream_t);
HC_CELL_INST(double)
HC_CELL_INST(float)

}  // namespace hcd
