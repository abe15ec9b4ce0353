// Finite-difference advection-diffusion coupled to the LBGK velocity field:
// ASL's FDAdvectionDiffusion (src/num/aslFDAdvectionDiffusion.cxx:88-180,
// 209-226) for one component with a constant diffusion coefficient D,
//   c' = D lap(c) + c - divProduct(u, c)
//   (compressibility correction: c' /= 1 - div(u); c' += lap(c) |u(x)|^2 / 2)
// and, with setElectricFieldParameters (:66-74, 166-172), c' -= divAgradB(c q / k, phi),
// with the stencil operators of src/math/aslTemplateVE.cxx:164-280 on the
// templates d3q7 / d3q15 / d3q19 (laplacian and gradient coefficients of
// src/math/aslTemplates.cxx:134-186):
//   lap(c)            = sum_i LC_i c(x + e_i)
//   div(u)            = sum_d sum_i GC_i e_i,d u_d(x + e_i)
//   divProduct(u, c)  = sum_d sum_i GC_i e_i,d (u_d(x + e_i) + u_d(x)) (c(x + e_i) + c(x)) / 2
//   divAgradB(a, b)   = sum_i GC_i (a(x + e_i) + a(x)) (b(x + e_i) - b(x))
// The update writes the interior of a second buffer and the buffers swap
// (postProcessing), so ghost values persist in both: they are the
// boundary values (BCConstantValue on faces, src/num/aslBasicBC.cxx:51-57).
// The velocity is the bound LBGK's device velocity field (ASL layout, FP32,
// FP64 for FP64 storage), read on that domain's stream after its step.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>
#include <nvtx3/nvToolsExt.h>
#include "aslb.h"
#include "kernels.h"
#include "f32x2.cuh"
#include "lattice.cuh"
#include "launch.cuh"
#include "per_device.h"
#include "tma.cuh"

namespace aslb {
namespace {

// Template vectors: d3q7, d3q15 and d3q19 list their vectors in the order of
// the lattice tables (d3q7 is the first seven of d3q19). Coefficients by
// vector class: rest, axis, diagonal.
template <int Q>
struct FdTemplate {
  __host__ __device__ static constexpr int e(int i, int d) { return Q == 15 ? lat_c15(i, d) : lat_c27(i, d); }
  __host__ __device__ static constexpr double lc(int i) {
    return i == 0 ? (Q == 7 ? -6.0 : Q == 15 ? -14.0 / 3.0 : -4.0)
                  : (i <= 6 ? (Q == 7 ? 1.0 : Q == 15 ? 2.0 / 3.0 : 1.0 / 3.0) : (Q == 15 ? 1.0 / 12.0 : 1.0 / 6.0));
  }
  __host__ __device__ static constexpr double gc(int i) {
    return i == 0 ? 0.0
                  : (i <= 6 ? (Q == 7 ? 0.5 : Q == 15 ? 1.0 / 3.0 : 1.0 / 6.0) : (Q == 15 ? 1.0 / 24.0 : 1.0 / 12.0));
  }
};

struct FdGrid {
  int nx, ny, nz, gx, gy, gz;
  long long L;
};

// The update of one cell from its stencil values: cv(i) = c(x + e_i),
// uv(d, i) = u_d(x + e_i).
template <int Q, class T, bool U, bool E, class CV, class UV, class EV>
__device__ __forceinline__ T fd_cell(CV cvf, UV uvf, EV evf, T D, int cc) {
  using Tp = FdTemplate<Q>;
  T cv[Q];
#pragma unroll
  for (int i = 0; i < Q; ++i) cv[i] = cvf(i);
  T lap = T(0);
#pragma unroll
  for (int i = 0; i < Q; ++i) lap += T(Tp::lc(i)) * cv[i];
  T cnew = D * lap + cv[0];
  if (U) {
    T dp[3], dv[3], u0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) u0[d] = uvf(d, 0);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      T s = T(0), v = T(0);
#pragma unroll
      for (int i = 1; i < Q; ++i) {
        if (Tp::e(i, d) == 0) continue;
        const T ui = uvf(d, i);
        const T coef = T(Tp::gc(i) * Tp::e(i, d));
        s += T(0.5) * ((ui + u0[d]) * (cv[i] + cv[0])) * coef;
        v += coef * ui;
      }
      dp[d] = s;
      dv[d] = v;
    }
    cnew -= dp[0] + dp[1] + dp[2];
    if (cc) {
      cnew /= T(1) - (dv[0] + dv[1] + dv[2]);
      cnew += lap * (u0[0] * u0[0] + u0[1] * u0[1] + u0[2] * u0[2]) * T(0.5);
    }
  }
  if (E) {
    // electric term: - divAgradB(c q / k, phi) = - sum_i GC_i (a_i + a_0) (phi_i - phi_0),
    // a = c q / k (evf(0, i) = phi, evf(1, i) = k, evf(2, i) = q at x + e_i)
    const T a0 = cv[0] * evf(2, 0) / evf(1, 0), p0 = evf(0, 0);
    T s = T(0);
#pragma unroll
    for (int i = 1; i < Q; ++i) s += T(Tp::gc(i)) * (cv[i] * evf(2, i) / evf(1, i) + a0) * (evf(0, i) - p0);
    cnew -= s;
  }
  return cnew;
}

// 2.5-D tiling: a block of 32 x 8 threads owns a 32 (z) x 8 (y) column of
// cells and walks kFdPlanes x planes, keeping three planes of c (and u) with
// a one-cell halo in shared memory, so every value is read from HBM about
// once (the y/z halos of neighbouring tiles come from L2) and every
// neighbour read of the stencil is a shared-memory load. FP64, the electric
// term, and blocks beyond 32-bit element indices.
constexpr int kFdTZ = 32, kFdTY = 8, kFdPlanes = 32;

template <int Q, class T, bool U, bool E>
__global__ void __launch_bounds__(kFdTZ * kFdTY) k_fd_step(const T* __restrict__ c, T* __restrict__ cn,
                                                          const T* __restrict__ u, const T* __restrict__ ef,
                                                          FdGrid g, T D, int cc) {
  using Tp = FdTemplate<Q>;
  // fields per plane: c, then u (3) with a velocity, then phi, k, q with the electric term
  constexpr int UB = 1, EB = U ? 4 : 1;
  constexpr int W = kFdTZ + 2, H = kFdTY + 2, P = W * H, NF = 1 + (U ? 3 : 0) + (E ? 3 : 0);
  // three planes of the tile (dynamic: FP64 with velocity and electric fields
  // needs 56 KB)
  extern __shared__ __align__(16) unsigned char fd_smem[];
  wait_before();
  let_next();
  auto sm = reinterpret_cast<T(*)[NF][P]>(fd_smem);
  const int tz = threadIdx.x, ty = threadIdx.y, t = ty * kFdTZ + tz;
  const int z0 = blockIdx.x * kFdTZ, y0 = blockIdx.y * kFdTY;  // ghosted origin of the tile
  const int x0 = blockIdx.z * kFdPlanes + 1, x1 = min(g.nx, x0 + kFdPlanes - 1);
  const int z = z0 + tz + 1, y = y0 + ty + 1;
  const bool active = z <= g.nz && y <= g.ny;
  // each thread owns tile entries t and t + 256 (P <= 512): a plane is
  // fetched into registers one iteration ahead, so its HBM latency overlaps
  // the arithmetic of the current plane
  constexpr int NT = kFdTZ * kFdTY;
  static_assert(P <= 2 * NT, "two tile entries per thread");
  T r[2][NF];
  auto fetch = [&](int xp) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int e = t + k * NT;
      const int yy = y0 + e / W, zz = z0 + e % W;
      if (e < P && yy < g.gy && zz < g.gz) {
        const long long a = ((long long)xp * g.gy + yy) * g.gz + zz;
        r[k][0] = c[a];
        if (U) {
          r[k][UB % NF] = u[a];
          r[k][(UB + 1) % NF] = u[g.L + a];
          r[k][(UB + 2) % NF] = u[2 * g.L + a];
        }
        if (E) {
          r[k][EB % NF] = ef[a];
          r[k][(EB + 1) % NF] = ef[g.L + a];
          r[k][(EB + 2) % NF] = ef[2 * g.L + a];
        }
      }
    }
  };
  auto stash = [&](int xp) {
    const int slot = xp % 3;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int e = t + k * NT;
      if (e < P)
#pragma unroll
        for (int f = 0; f < NF; ++f) sm[slot][f][e] = r[k][f];
    }
  };
  fetch(x0 - 1);
  stash(x0 - 1);
  fetch(x0);
  stash(x0);
  fetch(x0 + 1);
  for (int x = x0; x <= x1; ++x) {
    stash(x + 1);  // into the slot plane x - 2 used; everyone passed the barrier below
    __syncthreads();
    if (x < x1) fetch(x + 2);
    if (active) {
      const int sl[3] = {(x + 2) % 3, x % 3, (x + 1) % 3};
      const int base = (ty + 1) * W + tz + 1;
      auto cvf = [&](int i) { return sm[sl[1 + Tp::e(i, 0)]][0][base + Tp::e(i, 1) * W + Tp::e(i, 2)]; };
      auto uvf = [&](int d, int i) { return sm[sl[1 + Tp::e(i, 0)]][U ? UB + d : 0][base + Tp::e(i, 1) * W + Tp::e(i, 2)]; };
      auto evf = [&](int f, int i) { return sm[sl[1 + Tp::e(i, 0)]][E ? EB + f : 0][base + Tp::e(i, 1) * W + Tp::e(i, 2)]; };
      cn[((long long)x * g.gy + y) * g.gz + z] = fd_cell<Q, T, U, E>(cvf, uvf, evf, D, cc);
    }
    __syncthreads();
  }
}

// FP32 step without the electric term: a block marches along x and reads
// every plane of its tile once.
//
// With e_i, GC_i the template and sum_i GC_i e_i = 0, the product divergence
//   divProduct = sum_i GC_i / 2 (c_i + c_0) (e_i . u_i + e_i . u_0)
// is 1/2 [div(c u) + c_0 div(u) + u_0 . grad(c)], so a step needs only linear
// stencil sums (laplacian and gradient of c, divergences of u and c u), and
// each plane's contribution to the outputs of the planes before, at and after
// it is a handful of in-plane sums. A thread owns KY x 2 cells (y, z) of the
// tile: per plane it reads the KY + 2 rows of its four columns once (two
// 8-byte shared loads per row and field: the tile's column 0 is the ghosted
// z0, so they are aligned), forms the sums of its two z cells in packed FP32,
// finishes the outputs of the previous plane and keeps, for the outputs of
// the next one, the five sums that its velocity will multiply.
//
// The gather over three planes that this replaces read 18.7 shared words per
// d3q19 cell and was bound by that stream of loads. Planes are staged by
// 4-byte asynchronous copies (ASL's rows have no alignment) into a ring of
// three slots, two planes ahead of the arithmetic, without registers.
// Work: items of `len` planes of a tile, all tiles of an x range before the
// next range, so that the blocks running together share their tiles' halo
// rows in L2 (tile by tile, the halos come from HBM again). Element indices are
// 32-bit: blocks of 2^32 cells or more take k_fd_step (with a 64-bit pointer per
// plane and field d3q19 took 0.0643 ms per step at 256x192x192 instead of
// 0.0618).
// KY: two, four for d3q7, whose cells carry fewer sums (512x256x256 FP32 with
// velocity, ms per step with two / four: d3q7 0.187 / 0.183, 0.062 / 0.049 at
// 256x192x192; d3q19 0.215 / 0.243).
template <int Q>
struct MarchConf {
  static constexpr int KY = Q == 7 ? 4 : 2, TY = 4;  // y cells per thread, warps
  static constexpr int NT = 32 * TY;            // threads
  static constexpr int TZ = 64, H = KY * TY + 2, W = TZ + 2, P = H * W;
  static constexpr int E = (P + NT - 1) / NT;   // staged entries per thread and field
  static constexpr int S = 3;                   // ring slots
};

template <int Q, bool U>
constexpr size_t fd_march_smem() {
  return (size_t)MarchConf<Q>::S * (U ? 4 : 1) * MarchConf<Q>::P * sizeof(float);
}

// One row's values at a thread's two cells: the value (m), the sum (s) and
// the difference (d) of its two z neighbours, of c, u_x, c u_x, u_y, c u_y,
// u_z, c u_z as far as the sums need them.
struct MarchRow {
  F2 cm, cs, cd, um, us, pm, ps, vm, vs, qm, qs, wm, wd, rd;
};

template <bool U, int P>
__device__ __forceinline__ MarchRow march_row(const float* b) {
  auto pair = [](const float* q) {
    const float2 v = *reinterpret_cast<const float2*>(q);
    return F2(v.x, v.y);
  };
  MarchRow r;
  const F2 c0 = pair(b), c1 = pair(b + 2);
  r.cm = F2(c0.hi(), c1.lo());
  r.cs = add_(c0, c1);
  r.cd = sub_(c1, c0);
  if constexpr (U) {
    const F2 u0 = pair(b + P), u1 = pair(b + P + 2);
    const F2 v0 = pair(b + 2 * P), v1 = pair(b + 2 * P + 2);
    const F2 w0 = pair(b + 3 * P), w1 = pair(b + 3 * P + 2);
    const F2 p0 = mul_(c0, u0), p1 = mul_(c1, u1), q0 = mul_(c0, v0), q1 = mul_(c1, v1);
    r.um = F2(u0.hi(), u1.lo());
    r.us = add_(u0, u1);
    r.pm = F2(p0.hi(), p1.lo());
    r.ps = add_(p0, p1);
    r.vm = F2(v0.hi(), v1.lo());
    r.vs = add_(v0, v1);
    r.qm = F2(q0.hi(), q1.lo());
    r.qs = add_(q0, q1);
    r.wm = F2(w0.hi(), w1.lo());
    r.wd = sub_(w1, w0);
    r.rd = sub_(mul_(c1, w1), mul_(c0, w0));
  }
  return r;
}

template <int Q, bool U, bool CC>
__global__ void __launch_bounds__(MarchConf<Q>::NT, 2)
    k_fd_march(const float* __restrict__ c, float* __restrict__ cn, const float* __restrict__ u, FdGrid g, float Df,
               int ntz, int tiles, int len, int items) {
  using Tp = FdTemplate<Q>;
  using R = MarchConf<Q>;
  constexpr int NF = U ? 4 : 1, P = R::P, W = R::W, NT = R::NT, KY = R::KY, S = R::S;
  constexpr float ga = (float)Tp::gc(1), gd = Q > 7 ? (float)Tp::gc(Q - 1) : 0.f;
  extern __shared__ __align__(16) float march_smem[];  // [S slots][NF][H][W]
  wait_before();
  let_next();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned plane = (unsigned)g.gy * (unsigned)g.gz;
  const F2 a = F2(ga), d = F2(gd), D = F2(Df), half = F2(0.5f), mhalf = F2(-0.5f), two = F2(2.f);
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int tile = item % tiles;
    const int xa = (item / tiles) * len + 1, xb = min(g.nx, xa + len - 1);
    const int z0 = (tile % ntz) * R::TZ, y0 = (tile / ntz) * (R::TY * KY);  // ghosted origin
    unsigned off[R::E];  // this thread's tile entries within a plane, ~0u off the grid
#pragma unroll
    for (int k = 0; k < R::E; ++k) {
      const int e = (int)threadIdx.x + k * NT;
      const int yy = y0 + e / W, zz = z0 + e % W;
      off[k] = (e < P && yy < g.gy && zz < g.gz) ? (unsigned)yy * (unsigned)g.gz + (unsigned)zz : ~0u;
    }
    auto fetch = [&](int xp) {
      if (xp <= xb + 1) {
        const unsigned pb = (unsigned)xp * plane;
        float* sp = march_smem + (xp % S) * NF * P + threadIdx.x;
#pragma unroll
        for (int k = 0; k < R::E; ++k) {
          if (off[k] == ~0u) continue;
          const unsigned at = pb + off[k];
          copy_async4(sp + k * NT, c + at);
          if constexpr (U) {
            copy_async4(sp + P + k * NT, u + at);
            copy_async4(sp + 2 * P + k * NT, u + g.L + at);
            copy_async4(sp + 3 * P + k * NT, u + 2 * g.L + at);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int z = z0 + 2 * lane + 1, y1 = y0 + w * KY + 1;
    // the previous plane's outputs less its centre, up to that plane's own
    // sums (with the correction cl and cd hold lap and div), and its centre
    // (cc, cu, cv, cw). The centre is added last, in one rounding of its size:
    // with the centre in acc from the start, three such roundings put a step
    // a fifth farther from the sums in double precision
    F2 acc[KY], cl[KY], cd[KY], cc[KY], cu[KY], cv[KY], cw[KY];
    // the current plane's sums for the next plane's outputs
    F2 sX[KY], sU[KY], sP[KY], sY[KY], sZ[KY];
    __syncthreads();  // every thread is done with the ring's previous run
    fetch(xa - 1);
    fetch(xa);
    for (int x = xa - 1; x <= xb + 1; ++x) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();  // plane x is in, plane x - 1 is done with
      fetch(x + 2);
      const float* b = march_smem + (x % S) * NF * P + (w * KY) * W + 2 * lane;
      MarchRow lo = march_row<U, P>(b), mid = march_row<U, P>(b + W);
#pragma unroll
      for (int r = 0; r < KY; ++r) {
        const MarchRow hi = march_row<U, P>(b + (r + 2) * W);
        // in-plane sums of c
        const F2 cross = add_(add_(lo.cm, hi.cm), mid.cs), corner = add_(lo.cs, hi.cs);
        const F2 dy = sub_(hi.cm, lo.cm), dyz = sub_(hi.cs, lo.cs), dzy = add_(lo.cd, hi.cd);
        // sums that this plane gives the planes before and after it: X with
        // opposite signs, the others alike
        auto across = [&](F2 m, F2 m0, F2 m1, F2 s, F2 s0, F2 s1) {
          F2 t = mul_(a, m);
          if (Q == 19) t = fma_(d, add_(add_(m0, m1), s), t);
          if (Q == 15) t = fma_(d, add_(s0, s1), t);
          return t;
        };
        F2 X = mul_(a, mid.cm);
        if (Q == 19) X = fma_(d, cross, X);
        if (Q == 15) X = fma_(d, corner, X);
        F2 Gy = F2(0.f), Gz = F2(0.f), Xu, Xp, Tu = F2(0.f), Tp_ = F2(0.f), v1, v2, q1, q2;
        if constexpr (U) {
          Xu = across(mid.um, lo.um, hi.um, mid.us, lo.us, hi.us);
          Xp = across(mid.pm, lo.pm, hi.pm, mid.ps, lo.ps, hi.ps);
          v1 = add_(sub_(hi.vm, lo.vm), mid.wd);
          q1 = add_(sub_(hi.qm, lo.qm), mid.rd);
          if (Q > 7) {
            v2 = add_(sub_(hi.vs, lo.vs), add_(lo.wd, hi.wd));
            q2 = add_(sub_(hi.qs, lo.qs), add_(lo.rd, hi.rd));
            Gy = mul_(d, Q == 19 ? dy : dyz);
            Gz = mul_(d, Q == 19 ? mid.cd : dzy);
            Tu = mul_(d, Q == 19 ? v1 : v2);
            Tp_ = mul_(d, Q == 19 ? q1 : q2);
          }
        }
        if (x > xa) {
          // outputs of plane x - 1: this plane's share
          F2 o = fma_(mul_(two, D), X, acc[r]), B;
          if constexpr (U) {
            B = add_(Tu, Xu);
            F2 f = fma_(cc[r], B, add_(Tp_, Xp));
            f = fma_(cu[r], X, f);
            if (Q > 7) f = fma_(cw[r], Gz, fma_(cv[r], Gy, f));
            o = fma_(mhalf, f, o);
          }
          o = add_(cc[r], o);
          if constexpr (CC) {
            o = div_(o, sub_(F2(1.f), add_(cd[r], B)));
            const F2 uu = fma_(cw[r], cw[r], fma_(cv[r], cv[r], mul_(cu[r], cu[r])));
            o = fma_(fma_(two, X, cl[r]), mul_(uu, half), o);
          }
          const int y = y1 + r;
          if (y <= g.ny) {
            float* out = cn + (size_t)((unsigned)(x - 1) * plane + (unsigned)y * (unsigned)g.gz + (unsigned)z);
            if (z <= g.nz) out[0] = o.lo();
            if (z < g.nz) out[1] = o.hi();
          }
        }
        if (x >= xa && x <= xb) {
          // outputs of plane x: the share of plane x - 1 and its own
          F2 L = fma_(F2((float)Tp::lc(0)), mid.cm, mul_(mul_(two, a), cross));
          if (Q == 19) L = fma_(mul_(two, d), corner, L);
          L = fma_(two, sX[r], L);
          F2 o = mul_(D, L);
          cc[r] = mid.cm;
          if constexpr (U) {
            F2 By = fma_(a, q1, sP[r]), Bu = fma_(a, v1, sU[r]);
            F2 gy = mul_(a, dy), gz = mul_(a, mid.cd);
            if (Q == 19) {
              By = fma_(d, q2, By);
              Bu = fma_(d, v2, Bu);
              gy = fma_(d, dyz, gy);
              gz = fma_(d, dzy, gz);
            }
            if (Q > 7) {
              gy = add_(gy, sY[r]);
              gz = add_(gz, sZ[r]);
            }
            F2 f = fma_(mid.cm, Bu, By);
            f = fma_(mid.vm, gy, sub_(f, mul_(mid.um, sX[r])));
            f = fma_(mid.wm, gz, f);
            o = fma_(mhalf, f, o);
            cu[r] = mid.um;
            cv[r] = mid.vm;
            cw[r] = mid.wm;
            if constexpr (CC) {
              cl[r] = L;
              cd[r] = Bu;
            }
          }
          acc[r] = o;
        }
        sX[r] = X;
        if constexpr (U) {
          sU[r] = sub_(Tu, Xu);
          sP[r] = sub_(Tp_, Xp);
          sY[r] = Gy;
          sZ[r] = Gz;
        }
        lo = mid;
        mid = hi;
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
}

// Face ghost layers (cells of the face with interior tangential indices).
template <class T>
__global__ void k_fd_face_value(T* __restrict__ c, FdGrid g, int axis, int layer, T value) {
  const int n1 = axis == 0 ? g.ny : g.nx, n2 = axis == 2 ? g.ny : g.nz;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n1 * n2) return;
  const int i = t / n2 + 1, j = t % n2 + 1;
  int x, y, z;
  if (axis == 0) { x = layer; y = i; z = j; }
  else if (axis == 1) { x = i; y = layer; z = j; }
  else { x = i; y = j; z = layer; }
  c[((long long)x * g.gy + y) * g.gz + z] = value;
}

// Conditions on c at a map (aslBasicBC.cxx:71-108, 271-350), thread t per
// guard cell (x, y, z, mask of fluid-neighbour directions of the template):
//   VALUE     c(x) = value
//   GRADIENT  c(x) = sum_k W_k (c(x + e_k) - (n . e_k / |e_k|) value) / sum_k W_k
//             when sum_k W_k > 0.1; W_k = (n . e_k / |e_k| + 1)^2 and
//             n . e_k / |e_k| precomputed per cell and direction (wt, nd).
template <int Q, class T>
__global__ void k_fd_map_bc(T* __restrict__ c, FdGrid g, const int4* __restrict__ cells, int n,
                            const double* __restrict__ wt, const double* __restrict__ nd, int gradient, T value) {
  using Tp = FdTemplate<Q>;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  wait_before();
  let_next();
  if (t >= n) return;
  const int4 an = cells[t];
  const long long a = ((long long)an.x * g.gy + an.y) * g.gz + an.z;
  if (!gradient) {
    c[a] = value;
    return;
  }
  T sum = T(0), counter = T(0);
#pragma unroll
  for (int k = 1; k < Q; ++k) {
    if (!((unsigned)an.w >> k & 1u)) continue;
    const long long q = ((long long)(an.x + Tp::e(k, 0)) * g.gy + an.y + Tp::e(k, 1)) * g.gz + an.z + Tp::e(k, 2);
    const T w = T(wt[(size_t)t * Q + k]);
    sum += (c[q] - T(nd[(size_t)t * Q + k]) * value) * w;
    counter += w;
  }
  if (counter > T(0.1)) c[a] = sum / counter;
}

}  // namespace
}  // namespace aslb

using namespace aslb;

struct aslb_fd_bc;

struct aslb_fd {
  FdGrid g{};
  int q = 7;
  int dtype = ASLB_F32;
  double D = 0;
  void* c[2] = {nullptr, nullptr};
  int cur = 0;
  const void* u = nullptr;  // bound velocity field (device), or none
  int cc = 0;
  cudaStream_t stream = nullptr, own = nullptr;
  aslb_lbgk* bound = nullptr;  // domain whose velocity and stream are used
  void* ef = nullptr;           // electric term: phi, k, q (3 L values), or none
  long long steps = 0;
  std::vector<aslb_fd_bc*> bcs;  // map conditions on c (detached on destroy)
};

struct aslb_fd_bc {
  aslb_fd* fd = nullptr;
  int gradient = 0;
  double value = 0;
  int n = 0;
  int4* cells = nullptr;
  double* wt = nullptr;
  double* nd = nullptr;
};

namespace aslb {
// The bound domain is being destroyed: fall back to no velocity.
void fd_detached(aslb_fd* f) {
  f->u = nullptr;
  f->stream = f->own;
  f->cc = 0;
  f->bound = nullptr;
}
}  // namespace aslb

namespace {
int fd_err(const char* what, cudaError_t e) {
  set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
  return ASLB_ERR_CUDA;
}
int fd_arg(const char* what) {
  set_last_error(std::string(what));
  return ASLB_ERR_ARG;
}
size_t fd_elem(const aslb_fd* f) { return f->dtype == ASLB_F64 ? 8 : 4; }

// Launch one instantiation with its dynamic shared memory (three tile planes
// of every field it stages), raising the device's limit where above 48 KB.
template <int Q, class T, bool U, bool E>
cudaError_t fd_launch_one(aslb_fd* f, dim3 grid, dim3 block, const T* c, T* cn, const T* u, const T* ef) {
  constexpr int NF = 1 + (U ? 3 : 0) + (E ? 3 : 0);
  constexpr size_t bytes = 3u * NF * (kFdTZ + 2) * (kFdTY + 2) * sizeof(T);
  if (bytes > 48 * 1024) {
    static PerDevice raised;
    int dev = 0, limit = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
      e = raised.get(dev, limit, [&](int& n) {
        n = (int)bytes;
        return cudaFuncSetAttribute(k_fd_step<Q, T, U, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, n);
      });
    if (e != cudaSuccess) return e;
  }
  return launch_after(k_fd_step<Q, T, U, E>, grid, block, bytes, f->stream, c, cn, u, ef, f->g, T(f->D), U ? f->cc : 0);
}

// The marching FP32 kernel on as many blocks as are resident.
template <int Q, bool U, bool CC>
cudaError_t fd_launch_march(aslb_fd* f) {
  using R = MarchConf<Q>;
  constexpr size_t bytes = fd_march_smem<Q, U>();
  auto kern = k_fd_march<Q, U, CC>;
  static PerDevice blocks;
  int dev = 0, sms = 0, resident = 0;  // blocks per SM
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess)
    e = blocks.get(dev, resident, [&](int& n) {
      cudaError_t r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      if (r == cudaSuccess) r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, R::NT, bytes);
      return r == cudaSuccess && n < 1 ? cudaErrorInvalidConfiguration : r;
    });
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int ntz = (f->g.nz + R::TZ - 1) / R::TZ, nty = (f->g.ny + R::TY * R::KY - 1) / (R::TY * R::KY);
  const int tiles = ntz * nty;
  const long long slots = (long long)resident * sms;
  // planes per item: one item per block while that keeps them short, else at
  // most 32 planes (an item reads two planes more than it writes)
  const long long share = ((long long)tiles * f->g.nx + slots - 1) / slots;
  const int len = (int)std::min<long long>({share, 32, f->g.nx});
  const int items = tiles * ((f->g.nx + len - 1) / len);
  return launch_after(kern, (unsigned)std::min<long long>(items, slots), R::NT, bytes, f->stream,
                      (const float*)f->c[f->cur], (float*)f->c[1 - f->cur], (const float*)f->u, f->g, (float)f->D, ntz,
                      tiles, len, items);
}

template <int Q, class T>
cudaError_t fd_launch(aslb_fd* f) {
  // FP32 without the electric term: the marching kernel, within its 32-bit
  // element indices; FP64 (whose sums would take twice the registers), the
  // electric term and larger blocks: the 32 x 8 tiles
  if constexpr (std::is_same<T, float>::value) {
    if (!f->ef && f->g.L < (1LL << 32)) {
      if (!f->u) return fd_launch_march<Q, false, false>(f);
      return f->cc ? fd_launch_march<Q, true, true>(f) : fd_launch_march<Q, true, false>(f);
    }
  }
  dim3 block(kFdTZ, kFdTY),
      grid((f->g.nz + kFdTZ - 1) / kFdTZ, (f->g.ny + kFdTY - 1) / kFdTY, (f->g.nx + kFdPlanes - 1) / kFdPlanes);
  const T* c = (const T*)f->c[f->cur];
  T* cn = (T*)f->c[1 - f->cur];
  const T* ef = (const T*)f->ef;
  const T* u = (const T*)f->u;
  if (u && ef) return fd_launch_one<Q, T, true, true>(f, grid, block, c, cn, u, ef);
  if (u) return fd_launch_one<Q, T, true, false>(f, grid, block, c, cn, u, nullptr);
  if (ef) return fd_launch_one<Q, T, false, true>(f, grid, block, c, cn, nullptr, ef);
  return fd_launch_one<Q, T, false, false>(f, grid, block, c, cn, nullptr, nullptr);
}

template <class T>
cudaError_t fd_step_t(aslb_fd* f) {
  switch (f->q) {
    case 7: return fd_launch<7, T>(f);
    case 15: return fd_launch<15, T>(f);
    case 19: return fd_launch<19, T>(f);
  }
  return cudaErrorInvalidValue;
}
}  // namespace

extern "C" {

int aslb_fd_create(int nx, int ny, int nz, int q, int dtype, double D, aslb_fd** out) {
  if (!out) return fd_arg("aslb_fd_create: null argument");
  *out = nullptr;
  if (nx < 1 || ny < 1 || nz < 1) return fd_arg("aslb_fd_create: sizes must be positive");
  if (q != 7 && q != 15 && q != 19) return fd_arg("aslb_fd_create: template must be d3q7, d3q15 or d3q19");
  if (dtype != ASLB_F32 && dtype != ASLB_F64) return fd_arg("aslb_fd_create: dtype must be F32 or F64");
  auto* f = new aslb_fd();
  f->g = FdGrid{nx, ny, nz, nx + 2, ny + 2, nz + 2, (long long)(nx + 2) * (ny + 2) * (nz + 2)};
  f->q = q;
  f->dtype = dtype;
  f->D = D;
  cudaError_t e = cudaStreamCreateWithFlags(&f->own, cudaStreamNonBlocking);
  f->stream = f->own;
  for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
    e = cudaMalloc(&f->c[b], f->g.L * fd_elem(f));
    if (e == cudaSuccess) e = cudaMemsetAsync(f->c[b], 0, f->g.L * fd_elem(f), f->stream);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
  if (e != cudaSuccess) {
    aslb_fd_destroy(f);
    return fd_err("aslb_fd_create", e);
  }
  *out = f;
  return ASLB_OK;
}

int aslb_fd_set_velocity(aslb_fd* f, aslb_lbgk* h, int compressibility_correction) {
  if (!f) return fd_arg("aslb_fd_set_velocity: null argument");
  if (f->bound) {
    cudaStreamSynchronize(f->stream);
    lbgk_detach_fd(f->bound, f);
    fd_detached(f);
  }
  if (!h) return ASLB_OK;
  int n[3], storage;
  void* u;
  cudaStream_t st;
  int r = lbgk_velocity_binding(h, n, &storage, &u, &st);
  if (r) return r;
  if (n[0] != f->g.nx || n[1] != f->g.ny || n[2] != f->g.nz)
    return fd_arg("aslb_fd_set_velocity: the domain has another size");
  if ((storage == ASLB_F64) != (f->dtype == ASLB_F64))
    return fd_arg("aslb_fd_set_velocity: the velocity field is FP64 only for FP64 storage; match the FD dtype");
  cudaStreamSynchronize(f->stream);
  f->u = u;
  f->stream = st;  // after the domain's step, in order
  f->cc = compressibility_correction ? 1 : 0;
  f->bound = h;
  lbgk_attach_fd(h, f);
  return ASLB_OK;
}

int aslb_fd_set_electric_field(aslb_fd* f, int dtype, const void* phi, const void* k, const void* q) {
  if (!f) return fd_arg("aslb_fd_set_electric_field: null argument");
  if (!phi && !k && !q) {
    if (f->ef) {
      cudaStreamSynchronize(f->stream);
      cudaFree(f->ef);
      f->ef = nullptr;
    }
    return ASLB_OK;
  }
  if (!phi || !k || !q || dtype != f->dtype)
    return fd_arg("aslb_fd_set_electric_field: phi, k and q are all needed, in the FD's dtype");
  const size_t bytes = (size_t)f->g.L * fd_elem(f);
  cudaError_t e = cudaSuccess;
  if (!f->ef) e = cudaMalloc(&f->ef, 3 * bytes);
  const void* src[3] = {phi, k, q};
  for (int i = 0; i < 3 && e == cudaSuccess; ++i)
    e = cudaMemcpyAsync((char*)f->ef + i * bytes, src[i], bytes, cudaMemcpyHostToDevice, f->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
  if (e != cudaSuccess) return fd_err("aslb_fd_set_electric_field", e);
  return ASLB_OK;
}

int aslb_fd_set_diffusion(aslb_fd* f, double D) {
  if (!f) return fd_arg("aslb_fd_set_diffusion: null argument");
  f->D = D;
  return ASLB_OK;
}

int aslb_fd_write(aslb_fd* f, int dtype, const void* host) {
  if (!f || !host || dtype != f->dtype) return fd_arg("aslb_fd_write: null argument or dtype differs from the FD's");
  const size_t bytes = f->g.L * fd_elem(f);
  cudaError_t e = cudaMemcpyAsync(f->c[0], host, bytes, cudaMemcpyHostToDevice, f->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(f->c[1], f->c[0], bytes, cudaMemcpyDeviceToDevice, f->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
  if (e != cudaSuccess) return fd_err("aslb_fd_write", e);
  f->cur = 0;
  return ASLB_OK;
}

int aslb_fd_read(aslb_fd* f, int dtype, void* host) {
  if (!f || !host || dtype != f->dtype) return fd_arg("aslb_fd_read: null argument or dtype differs from the FD's");
  cudaError_t e = cudaMemcpyAsync(host, f->c[f->cur], f->g.L * fd_elem(f), cudaMemcpyDeviceToHost, f->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
  if (e != cudaSuccess) return fd_err("aslb_fd_read", e);
  return ASLB_OK;
}

int aslb_fd_set_face_value(aslb_fd* f, unsigned wallmask, double value) {
  if (!f) return fd_arg("aslb_fd_set_face_value: null argument");
  cudaError_t e = cudaSuccess;
  for (int w = 0; w < 6 && e == cudaSuccess; ++w) {
    if (!(wallmask >> w & 1u)) continue;
    const int axis = w / 2;
    const int n[3] = {f->g.nx, f->g.ny, f->g.nz};
    const int layer = (w & 1) ? n[axis] + 1 : 0;
    const int cnt = (axis == 0 ? f->g.ny * f->g.nz : axis == 1 ? f->g.nx * f->g.nz : f->g.nx * f->g.ny);
    for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
      if (f->dtype == ASLB_F64)
        k_fd_face_value<double><<<(cnt + 255) / 256, 256, 0, f->stream>>>((double*)f->c[b], f->g, axis, layer, value);
      else
        k_fd_face_value<float><<<(cnt + 255) / 256, 256, 0, f->stream>>>((float*)f->c[b], f->g, axis, layer,
                                                                         (float)value);
      e = cudaGetLastError();
    }
  }
  if (e != cudaSuccess) return fd_err("aslb_fd_set_face_value", e);
  return ASLB_OK;
}

int aslb_fd_step(aslb_fd* f, int n) {
  nvtxRangePushA("aslb_fd_step");
  struct Pop { ~Pop() { nvtxRangePop(); } } pop;
  if (!f || n < 0) return fd_arg("aslb_fd_step: null argument or negative count");
  for (int s = 0; s < n; ++s) {
    cudaError_t e = f->dtype == ASLB_F64 ? fd_step_t<double>(f) : fd_step_t<float>(f);
    if (e != cudaSuccess) return fd_err("aslb_fd_step", e);
    f->cur = 1 - f->cur;
    f->steps++;
  }
  return ASLB_OK;
}

int aslb_fd_sync(aslb_fd* f) {
  if (!f) return fd_arg("aslb_fd_sync: null argument");
  cudaError_t e = cudaStreamSynchronize(f->stream);
  if (e != cudaSuccess) return fd_err("aslb_fd_sync", e);
  return ASLB_OK;
}

void* aslb_fd_device_field(aslb_fd* f) { return f ? f->c[f->cur] : nullptr; }

int aslb_fd_bc_create(aslb_fd* f, int kind, const float* map, double value, aslb_fd_bc** out) {
  if (!f || !map || !out) return fd_arg("aslb_fd_bc_create: null argument");
  *out = nullptr;
  if (kind != ASLB_FD_BC_VALUE_MAP && kind != ASLB_FD_BC_GRADIENT_MAP)
    return fd_arg("aslb_fd_bc_create: kind must be ASLB_FD_BC_VALUE_MAP or ASLB_FD_BC_GRADIENT_MAP");
  const FdGrid& g = f->g;
  const int q = f->q;
  auto e = [&](int k, int d) { return q == 15 ? lat_c15(k, d) : lat_c27(k, d); };
  auto gc = [&](int k) {
    return q == 7 ? FdTemplate<7>::gc(k) : q == 15 ? FdTemplate<15>::gc(k) : FdTemplate<19>::gc(k);
  };
  auto mat = [&](int x, int y, int z) -> double {  // the map, -0.9 off the grid (generateDCFullSafe)
    if (x < 0 || y < 0 || z < 0 || x >= g.gx || y >= g.gy || z >= g.gz) return -0.9;
    return map[((long long)x * g.gy + y) * g.gz + z];
  };
  std::vector<int4> cells;
  std::vector<double> wt, nd;
  for (int x = 0; x < g.gx; ++x)
    for (int y = 0; y < g.gy; ++y)
      for (int z = 0; z < g.gz; ++z) {
        const float m0 = map[((long long)x * g.gy + y) * g.gz + z];
        if (!(m0 <= 0.f && m0 > -0.9999f)) continue;
        unsigned mask = 0;
        double nrm[3] = {0, 0, 0};
        for (int k = 1; k < q; ++k) {
          const int qx = x + e(k, 0), qy = y + e(k, 1), qz = z + e(k, 2);
          const double mk = mat(qx, qy, qz);
          const bool in = qx >= 1 && qx <= g.nx && qy >= 1 && qy <= g.ny && qz >= 1 && qz <= g.nz;
          if (mk > 0.0 && in) mask |= 1u << k;
          for (int d = 0; d < 3; ++d) nrm[d] += gc(k) * e(k, d) * (float)mk;
        }
        if (kind == ASLB_FD_BC_GRADIENT_MAP) {
          const double len = std::sqrt(nrm[0] * nrm[0] + nrm[1] * nrm[1] + nrm[2] * nrm[2]);
          if (!(len > 0.0) || !mask) continue;  // no normal or no fluid neighbour: c stays
          for (int k = 0; k < q; ++k) {
            double w = 0, dn = 0;
            if (k > 0 && (mask >> k & 1u)) {
              const double cl = std::sqrt((double)(e(k, 0) * e(k, 0) + e(k, 1) * e(k, 1) + e(k, 2) * e(k, 2)));
              dn = (nrm[0] * e(k, 0) + nrm[1] * e(k, 1) + nrm[2] * e(k, 2)) / len / cl;
              w = (dn + 1.0) * (dn + 1.0);
            }
            wt.push_back(w);
            nd.push_back(dn);
          }
        }
        cells.push_back(make_int4(x, y, z, (int)mask));
      }
  auto* b = new aslb_fd_bc();
  b->fd = f;
  b->gradient = kind == ASLB_FD_BC_GRADIENT_MAP;
  b->value = value;
  b->n = (int)cells.size();
  cudaError_t err = cudaSuccess;
  if (b->n) {
    err = cudaMalloc((void**)&b->cells, cells.size() * sizeof(int4));
    if (err == cudaSuccess)
      err = cudaMemcpy(b->cells, cells.data(), cells.size() * sizeof(int4), cudaMemcpyHostToDevice);
    if (err == cudaSuccess && !wt.empty()) {
      err = cudaMalloc((void**)&b->wt, wt.size() * sizeof(double));
      if (err == cudaSuccess) err = cudaMalloc((void**)&b->nd, nd.size() * sizeof(double));
      if (err == cudaSuccess) err = cudaMemcpy(b->wt, wt.data(), wt.size() * sizeof(double), cudaMemcpyHostToDevice);
      if (err == cudaSuccess) err = cudaMemcpy(b->nd, nd.data(), nd.size() * sizeof(double), cudaMemcpyHostToDevice);
    }
  }
  if (err != cudaSuccess) {
    aslb_fd_bc_destroy(b);
    return fd_err("aslb_fd_bc_create", err);
  }
  f->bcs.push_back(b);
  *out = b;
  return ASLB_OK;
}

int aslb_fd_bc_execute(aslb_fd_bc* b) {
  if (!b) return fd_arg("aslb_fd_bc_execute: null argument");
  if (!b->fd) {
    set_last_error("aslb_fd_bc_execute: its FD solver was destroyed");
    return ASLB_ERR_STATE;
  }
  aslb_fd* f = b->fd;
  if (!b->n) return ASLB_OK;
  const unsigned blocks = (unsigned)((b->n + 255) / 256);
  const int q = f->q;
  if (f->dtype == ASLB_F64) {
    double* c = (double*)f->c[f->cur];
    if (q == 7) k_fd_map_bc<7, double><<<blocks, 256, 0, f->stream>>>(c, f->g, b->cells, b->n, b->wt, b->nd, b->gradient, b->value);
    else if (q == 15) k_fd_map_bc<15, double><<<blocks, 256, 0, f->stream>>>(c, f->g, b->cells, b->n, b->wt, b->nd, b->gradient, b->value);
    else k_fd_map_bc<19, double><<<blocks, 256, 0, f->stream>>>(c, f->g, b->cells, b->n, b->wt, b->nd, b->gradient, b->value);
  } else {
    float* c = (float*)f->c[f->cur];
    const float v = (float)b->value;
    if (q == 7) k_fd_map_bc<7, float><<<blocks, 256, 0, f->stream>>>(c, f->g, b->cells, b->n, b->wt, b->nd, b->gradient, v);
    else if (q == 15) k_fd_map_bc<15, float><<<blocks, 256, 0, f->stream>>>(c, f->g, b->cells, b->n, b->wt, b->nd, b->gradient, v);
    else k_fd_map_bc<19, float><<<blocks, 256, 0, f->stream>>>(c, f->g, b->cells, b->n, b->wt, b->nd, b->gradient, v);
  }
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return fd_err("aslb_fd_bc_execute", err);
  return ASLB_OK;
}

long long aslb_fd_bc_cells(aslb_fd_bc* b) { return b ? b->n : -1; }

int aslb_fd_bc_destroy(aslb_fd_bc* b) {
  if (!b) return ASLB_OK;
  if (b->fd) {
    cudaStreamSynchronize(b->fd->stream);
    auto& v = b->fd->bcs;
    v.erase(std::remove(v.begin(), v.end(), b), v.end());
  }
  cudaFree(b->cells);
  cudaFree(b->wt);
  cudaFree(b->nd);
  delete b;
  return ASLB_OK;
}

int aslb_fd_destroy(aslb_fd* f) {
  if (!f) return ASLB_OK;
  if (f->stream) cudaStreamSynchronize(f->stream);
  if (f->bound) lbgk_detach_fd(f->bound, f);
  for (aslb_fd_bc* b : f->bcs) b->fd = nullptr;
  if (f->ef) cudaFree(f->ef);
  for (void* p : f->c)
    if (p) cudaFree(p);
  if (f->own) cudaStreamDestroy(f->own);
  delete f;
  return ASLB_OK;
}

}  // extern "C"
