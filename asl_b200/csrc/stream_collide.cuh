// Fused AA-pattern stream-collide kernel (one interior cell per thread) and its
// launch helpers. Instantiated per lattice and storage in step_q<Q>_<type>.cu
// so the instantiations compile in parallel.
#pragma once
#include <algorithm>
#include <type_traits>
#include "kernels.h"
#include "collide.cuh"
#include "launch.cuh"

namespace aslb {

template <class S>
struct MacroT {
  using T = float;
};
template <>
struct MacroT<double> {
  using T = double;
};

// Storage offsets of the neighbours at displacement d in {-1,0,1} per axis
// (index d + 1), with periodic axes wrapping across the interior.
__device__ __forceinline__ void nb_offsets(const GridDesc& g, int x, int y, int z, int (&ox)[3], int (&oy)[3],
                                           int (&oz)[3]) {
  const int pl = (int)g.plane;
  ox[0] = -pl; ox[1] = 0; ox[2] = pl;
  oy[0] = -g.pitch; oy[1] = 0; oy[2] = g.pitch;
  oz[0] = -1; oz[1] = 0; oz[2] = 1;
  if (g.periodic & 1) {
    if (x == 1) ox[0] = (g.nx - 1) * pl;
    if (x == g.nx) ox[2] = -(g.nx - 1) * pl;
  }
  if (g.periodic & 2) {
    if (y == 1) oy[0] = (g.ny - 1) * g.pitch;
    if (y == g.ny) oy[2] = -(g.ny - 1) * g.pitch;
  }
  if (g.periodic & 4) {
    if (z == 1) oz[0] = g.nz - 1;
    if (z == g.nz) oz[2] = -(g.nz - 1);
  }
}

// Resident blocks of 256 threads per SM the register budget aims for. The
// plain FP32/FP16 kernels must keep enough loads in flight to saturate HBM:
// four blocks (64 registers) with fused links, whose per-direction slot
// selects keep the schedule compact; three (80 registers) without, where the
// compiler hoists all addresses and 64 registers would spill (two, 128
// registers, for D3Q27). Three (80 registers) for the closures, two for FP64.
template <int Q, class S, int CL, bool FUSED>
struct StepOccupancy {
  static constexpr int blocks = std::is_same<S, double>::value
                                    ? 2
                                    : (CL == CL_NONE ? (FUSED ? 4 : (Q == 27 ? 2 : 3)) : 3);
};

// Store one outgoing population unless its slot is elided (the slot keeps its
// bits). In the AA pattern a cell writes exactly the slots it read moments
// before, so the lines are still in L2 and a warp's partial store merges there
// without an HBM read.
template <class S>
__device__ __forceinline__ void store_slot(S* __restrict__ slot, typename Store<S>::C v, bool elided,
                                           const StepParams& p) {
  if (!elided) *slot = Store<S>::encode(v, p);
}

// Gather the Q incoming populations of cell s. MASKED: bounce bits select
// the bounce-back slot (this cell's own outgoing population: the upstream and
// own slots swap roles between representations). Offsets from the periodic
// wrap (nb_offsets): the slow path of cells on a periodic face.
template <int Q, class S, bool ODD, bool MASKED>
__device__ __forceinline__ void cell_load(const S* __restrict__ F, unsigned ds, unsigned s, const int (&ox)[3],
                                          const int (&oy)[3], const int (&oz)[3], uint32_t bounce,
                                          typename Store<S>::C (&f)[Q]) {
  using Lt = Lattice<Q>;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const bool b = MASKED && ((bounce >> i) & 1u);
    unsigned idx;
    if (ODD) {
      idx = b ? (unsigned)Lt::inv(i) * ds + s
              : (unsigned)i * ds + s + (unsigned)(ox[1 - Lt::c(i, 0)] + oy[1 - Lt::c(i, 1)] + oz[1 - Lt::c(i, 2)]);
    } else if (b) {
      idx = (unsigned)i * ds + s + (unsigned)(ox[1 - Lt::c(i, 0)] + oy[1 - Lt::c(i, 1)] + oz[1 - Lt::c(i, 2)]);
    } else {
      idx = (unsigned)Lt::inv(i) * ds + s;
    }
    f[i] = Store<S>::load_c(F + idx);
  }
}

// The same gather for a cell whose neighbours do not wrap: every slot is the
// cell's index plus a precomputed offset (p.slot).
template <int Q, class S, bool ODD, bool MASKED>
__device__ __forceinline__ void cell_load_flat(const S* __restrict__ F, unsigned s, const StepParams& p,
                                               uint32_t bounce, typename Store<S>::C (&f)[Q]) {
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const bool b = MASKED && ((bounce >> i) & 1u);
    // ODD: pull, or the opposite own slot when bounced; EVEN: the reverse
    const unsigned off = (ODD != b) ? p.slot[0][i] : p.slot[3][i];
    f[i] = Store<S>::load_c(F + (s + off));
  }
}

// Collide cell (x, y, z) at storage index s and write rho / u when asked;
// f becomes the outgoing populations.
template <int Q, class S, int CL>
__device__ __forceinline__ void cell_collide(const GridDesc& g, const StepParams& p,
                                             typename MacroT<S>::T* __restrict__ rho_out,
                                             typename MacroT<S>::T* __restrict__ u_out, int x, int y, int z,
                                             unsigned s, typename Store<S>::C (&f)[Q], typename Store<S>::C om0) {
  using C = typename Store<S>::C;
  C rho, u[3];
  const C cs2 = CL == CL_MLP ? C(p.cs2[s]) : C(0);
  collide_cell<Q, C, CL, Store<S>::kDev>(f, p, om0, cs2, rho, u);
  if (p.write_macro) {
    const long long a = aidx(g, x, y, z);
    if (p.write_rho) rho_out[a] = rho;
    if (p.write_vel) {
      u_out[a] = u[0];
      u_out[g.L + a] = u[1];
      u_out[2 * g.L + a] = u[2];
    }
  }
}

// Store the outgoing populations (elide bits keep the slot), wrap-aware.
template <int Q, class S, bool ODD, bool MASKED>
__device__ __forceinline__ void cell_store(S* __restrict__ F, const StepParams& p, unsigned ds, unsigned s,
                                           const int (&ox)[3], const int (&oy)[3], const int (&oz)[3],
                                           uint32_t elide, const typename Store<S>::C (&f)[Q]) {
  using Lt = Lattice<Q>;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    unsigned idx;
    if (ODD)
      idx = (unsigned)Lt::inv(i) * ds + s + (unsigned)(ox[1 + Lt::c(i, 0)] + oy[1 + Lt::c(i, 1)] + oz[1 + Lt::c(i, 2)]);
    else
      idx = (unsigned)i * ds + s;
    store_slot<S>(F + idx, f[i], MASKED && ((elide >> i) & 1u), p);
  }
}

// s, seen by the compiler as computed after v: addresses derived from the
// result cannot be hoisted above the collision that produced v (hoisted, the
// Q store addresses of a cell would stay live across it and spill).
__device__ __forceinline__ unsigned after(unsigned s, float v) {
  asm volatile("" : "+r"(s) : "f"(v));
  return s;
}
__device__ __forceinline__ unsigned after(unsigned s, F2 v) {
  asm volatile("" : "+r"(s) : "l"(v.v));
  return s;
}
__device__ __forceinline__ unsigned after(unsigned s, double v) {
  asm volatile("" : "+r"(s) : "d"(v));
  return s;
}

// The same stores for a cell whose neighbours do not wrap (p.slot).
template <int Q, class S, bool ODD, bool MASKED>
__device__ __forceinline__ void cell_store_flat(S* __restrict__ F, const StepParams& p, unsigned s, uint32_t elide,
                                                const typename Store<S>::C (&f)[Q]) {
  const unsigned sl = after(s, f[0]);
#pragma unroll
  for (int i = 0; i < Q; ++i)
    store_slot<S>(F + (sl + (ODD ? p.slot[2][i] : p.slot[1][i])), f[i], MASKED && ((elide >> i) & 1u), p);
}

// Whether any neighbour of a cell with coordinate v on a periodic axis of n
// interior cells wraps to the opposite face.
__device__ __forceinline__ bool wraps(int periodic_bit, int v, int n) { return periodic_bit && (v == 1 || v == n); }

// ---------------------------------------------------------------------------
// Cells on periodic faces, whose neighbours wrap to the opposite face, are
// skipped by the main blocks of a stream-collide launch (by their loop range,
// so the main loop has no branch) and advanced by extra blocks of the same
// launch, one cell per thread with the wrap-aware offsets (disjoint cells:
// the AA update of a cell touches only its own slots). The face cells lie on
// up to six planes, the two faces of every periodic axis. A cell on
// several planes belongs to the first that holds it. The face blocks come
// first in the grid (blockIdx.z < fz), so they run alongside the main blocks
// instead of after them.
struct FaceWork {
  int n;          // planes
  int axis[6];
  int coord[6];
  int start[7];   // prefix sums of the planes' cell counts
  int fz;         // grid z-slices of face blocks
};

template <int Q, class S, int CL, bool ODD, bool FUSED>
__device__ __forceinline__ void face_cell(S* __restrict__ F, const GridDesc& g, const StepParams& p,
                                          const FaceWork& fw, typename MacroT<S>::T* __restrict__ rho_out,
                                          typename MacroT<S>::T* __restrict__ u_out) {
  using C = typename Store<S>::C;
  const int threads = blockDim.x * blockDim.y;
  const long long blk = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const long long c = blk * threads + threadIdx.y * blockDim.x + threadIdx.x;
  if (c >= fw.start[fw.n]) return;
  int k = 0;
  while (c >= fw.start[k + 1]) ++k;
  const int r = (int)(c - fw.start[k]);
  const int axis = fw.axis[k];
  // in-plane coordinates: the two other axes in order
  const int nu = axis == 0 ? g.ny : g.nx;
  const int nv = axis == 2 ? g.ny : g.nz;
  (void)nu;
  const int u = r / nv + 1, v = r % nv + 1;
  const int x = axis == 0 ? fw.coord[k] : u;
  const int y = axis == 1 ? fw.coord[k] : (axis == 0 ? u : v);
  const int z = axis == 2 ? fw.coord[k] : v;
  for (int j = 0; j < k; ++j)
    if ((fw.axis[j] == 0 ? x : (fw.axis[j] == 1 ? y : z)) == fw.coord[j]) return;
  const unsigned s = (unsigned)sidx(g, x, y, z);
  uint2 m = make_uint2(0u, 0u);
  if (FUSED) m = p.mask[s];
  int ox[3], oy[3], oz[3];
  nb_offsets(g, x, y, z, ox, oy, oz);
  C f[Q];
  cell_load<Q, S, ODD, FUSED>(F, (unsigned)g.dstride, s, ox, oy, oz, m.x, f);
  cell_collide<Q, S, CL>(g, p, rho_out, u_out, x, y, z, s, f, step_omega<C>(p));
  cell_store<Q, S, ODD, FUSED>(F, p, (unsigned)g.dstride, s, ox, oy, oz, m.y, f);
}

// The face planes of a domain and the grid z-slices their cells need with
// blocks of `threads` threads on a gx x gy grid face. paired: the main kernel
// is the two-cells-per-thread kernel, which wraps a periodic z axis itself
// (its z faces would be single cells of every row, one sector each).
inline FaceWork face_work(const GridDesc& g, bool paired, int threads, int gx, int gy) {
  FaceWork fw{};
  const int n[3] = {g.nx, g.ny, g.nz};
  for (int a = 0; a < (paired ? 2 : 3); ++a)
    if ((g.periodic >> a) & 1)
      for (int side = 0; side < 2; ++side) {
        const int c = side ? n[a] : 1;
        if (side && c == 1) continue;
        const int cells = a == 0 ? g.ny * g.nz : (a == 1 ? g.nx * g.nz : g.nx * g.ny);
        fw.axis[fw.n] = a;
        fw.coord[fw.n] = c;
        fw.start[fw.n + 1] = fw.start[fw.n] + cells;
        ++fw.n;
      }
  const long long per_slice = (long long)threads * gx * gy;
  fw.fz = (int)((fw.start[fw.n] + per_slice - 1) / per_slice);
  return fw;
}

// ---------------------------------------------------------------------------
// Stream + collide, one interior cell per thread. ODD: representation A -> B
// (reads F[i][x - c_i], writes F[inv i][x + c_i]); EVEN: B -> A (reads
// F[inv i][x], writes F[i][x]). Element indices are 32-bit (Q * dstride < 2^32).
// FUSED: the domain has fused no-slip links (p.mask is read); chosen on the
// host so domains without them run the unmasked code. A block walks
// `planes` consecutive x planes; with fused links each thread loads the
// next plane's link words one iteration ahead (the population addresses
// depend on them, so they must not cost a second memory round trip).
constexpr int kOnePlanes = 4;
// Where the kernel says that `planes` is at most kOnePlanes. The compiler then
// orders the masked body's loads otherwise, for better or worse: 192x128x120
// porous box, us per step, without / with: D3Q19 FP64 plain 184 / 171,
// Smagorinsky 206 / 190, ASL's closure 190 / 204; D3Q19 FP32 learned 154 / 143,
// plain 131 / 137; D3Q15 FP32 ASL's closure 120 / 111; D3Q27 FP32 ASL's closure
// 217 / 200, Smagorinsky 199 / 210 (FP32: periodic in all axes).
template <int Q, class S, int CL>
constexpr bool kBoundPlanes = sizeof(S) == 8   ? Q == 19 && CL != CL_ASL_INTENT
                              : Q == 15        ? sizeof(S) == 2 || CL != CL_NONE
                              : Q == 19        ? CL == CL_MLP
                                               : CL == CL_ASL_INTENT || (sizeof(S) == 2 && CL == CL_SMAGORINSKY);
template <int Q, class S, int CL, bool ODD, bool FUSED>
__global__ void __launch_bounds__(256, StepOccupancy<Q, S, CL, FUSED>::blocks)
    k_stream_collide(S* __restrict__ F, const __grid_constant__ GridDesc g, const __grid_constant__ StepParams p,
                     const __grid_constant__ FaceWork fw, int planes, typename MacroT<S>::T* __restrict__ rho_out,
                     typename MacroT<S>::T* __restrict__ u_out) {
  using C = typename Store<S>::C;
  wait_before();
  let_next();
  if ((int)blockIdx.z < fw.fz) {
    face_cell<Q, S, CL, ODD, FUSED>(F, g, p, fw, rho_out, u_out);
    return;
  }
  const int z = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int x0 = (blockIdx.z - fw.fz) * planes + 1;
  int x1 = min(g.nx, x0 + planes - 1);
  if (FUSED && kBoundPlanes<Q, S, CL>) x1 = min(x1, x0 + kOnePlanes - 1);
  if (z > g.nz || y > g.ny) return;
  // cells whose neighbours wrap across a periodic face belong to the face
  // kernel; skipped by the loop's range, the loop body has no branch
  if (wraps(g.periodic & 2, y, g.ny) || wraps(g.periodic & 4, z, g.nz)) return;
  if (g.periodic & 1) {
    x0 = max(x0, 2);
    x1 = min(x1, g.nx - 1);
    if (x0 > x1) return;
  }
  const unsigned pl = (unsigned)g.plane;
  const unsigned s0 = (unsigned)sidx(g, x0, y, z);
  // fused no-slip links: a fluid cell reads bounce-back populations, a solid
  // cell skips the writes the condition would overwrite
  uint2 m = make_uint2(0u, 0u);
  if (FUSED) m = p.mask[s0];
  for (int x = x0; x <= x1; ++x) {
    const unsigned s = s0 + (unsigned)(x - x0) * pl;
    uint2 mn = make_uint2(0u, 0u);
    if (FUSED && x < x1) mn = p.mask[s + pl];
    C f[Q];
    cell_load_flat<Q, S, ODD, FUSED>(F, s, p, m.x, f);
    cell_collide<Q, S, CL>(g, p, rho_out, u_out, x, y, z, s, f, step_omega<C>(p));
    cell_store_flat<Q, S, ODD, FUSED>(F, p, s, m.y, f);
    m = mn;
  }
}

// Two cells per thread, z and z + 32 of the same row: a warp covers 64
// consecutive cells, and each thread has the loads of both cells in flight
// before it collides them. FP32 and FP16 storage: with fused links, and
// without them for the closures and for a periodic z axis, which
// wraps in the lane's own offsets (a row's first and last cell: as face cells
// they are one sector per population, and cost a fully periodic 160^3 FP32
// step 0.156 ms against 0.112). The plain step without links on a z axis that
// does not wrap is faster with one cell per thread (384x192x192 FP32 0.376 ms
// against 0.390). Fused links on a z axis that wraps: the plain step of D3Q15 /
// D3Q19 has a body with both (PZ), other steps take one cell per thread and z
// faces as single cells (porous box periodic in all axes, D3Q19, us per step, PZ
// / one cell / pairs left to the face blocks where either cell wraps: 192x128x120
// FP32 102 / 131 / 182, FP16 75 / 94 / 123; 64x48x33 7.2 / 11.1 / 10.0, 7.2 /
// 12.1 / 10.0).
// One-word masks where every cell's links fit in one: FP16 D3Q19 porous channel
// 320x208x256 0.357 ms with one word, 0.358 with two; D3Q15 0.319, 0.326.
// A block walks `planes` consecutive x planes; each thread loads the
// fused-link words of the next plane one iteration ahead, so that the
// population loads, whose addresses those words select, do not wait for a
// second memory round trip. x and y faces go to the face blocks.
constexpr int kPairPlanes = 2;
constexpr int kPairThreads = 128;
// Resident blocks of 128 threads: six (80 registers) for D3Q15 / D3Q19 with
// fused links, five (96) without (the compiler hoists the addresses), four
// (128) for D3Q27; the closures without links take five in the odd step (three
// bases keep fewer addresses live) and four in the even one, three to four in
// D3Q27.
template <int Q, int CL, bool MASKED, bool ODD>
constexpr int kPairBlocks = Q == 27 ? (CL == CL_NONE || (ODD && !MASKED) ? 4 : 3)
                                    : (CL == CL_NONE ? (MASKED ? 6 : 5) : (ODD && !MASKED ? 5 : 4));
// Whether the collision runs on the pair in packed FP32 (f32x2.cuh): where
// the link selects of D3Q15 / D3Q19 do not dominate, it halves the collision's
// instructions (160^3 periodic FP32, ms per step packed / scalar: plain 0.112
// / 0.134, Smagorinsky 0.138 / 0.155, learned closure at 128^3 0.064 / 0.082;
// D3Q27 with links 0.198 / 0.206; with links FP16 D3Q19 0.362 / 0.355).
template <int Q, int CL, bool MASKED>
constexpr bool kPairPack = CL != CL_NONE || !MASKED || Q == 27;
// Whether fused links take pairs. D3Q27's two cells leave too few registers in
// FP16 (more instructions per byte) and with the learned closure: 192x128x120
// porous box, us per step, pairs / one cell: FP16 plain 110 / 104, ASL's closure
// 132 / 114, Smagorinsky 133 / 117, learned 134 / 118; FP32 learned 204 / 154,
// but plain 140 / 144 and ASL's closure 155 / 168.
template <int Q, class S, int CL>
constexpr bool kPairLinks = Q != 27 || (sizeof(S) == 4 && CL != CL_MLP);
// Whether the body with links also wraps z (PZ).
template <int Q, int CL>
constexpr bool kPairWraps = Q != 27 && CL == CL_NONE;
// Whether a domain's step takes pairs. D3Q27 in FP32 where z does not wrap: the
// learned closure without links 140 / 132; Smagorinsky 158 / 150 with links and
// 128 / 125 without, but in rows that fill the lanes' 64 cells 209 / 211 and
// 175 / 176 (256x128x128).
template <int Q, class S, int CL>
inline bool takes_pairs(const GridDesc& g, bool fused) {
  const bool pz = g.periodic & 4;
  if (fused ? !kPairLinks<Q, S, CL> || (pz && !kPairWraps<Q, CL>) : !pz && CL == CL_NONE) return false;
  if (Q == 27 && !pz && (CL == CL_MLP || (CL == CL_SMAGORINSKY && g.nz % 64 != 0))) return false;
  return true;
}

// Offsets of a cell and of the cells below and above it along z: the slots at
// c_z = 0, at z - 1 and at z + 1, wrapped on a periodic z axis.
struct ZBase {
  unsigned at, below, above;
};
template <bool PZ>
__device__ __forceinline__ ZBase z_base(const GridDesc& g, unsigned s, int z) {
  ZBase r;
  r.at = r.below = r.above = s;
  if (PZ && (g.periodic & 4)) {
    if (z == 1) r.below += (unsigned)g.nz;
    if (z == g.nz) r.above -= (unsigned)g.nz;
  }
  return r;
}
__device__ __forceinline__ unsigned z_pick(const ZBase& b, int dz) { return dz == 0 ? b.at : (dz < 0 ? b.below : b.above); }

template <int Q, class S, bool ODD, bool MASKED, bool PZ>
__device__ __forceinline__ void pair_load(const S* __restrict__ F, const ZBase& b, const StepParams& p, uint32_t bounce,
                                          float (&f)[Q]) {
  using Lt = Lattice<Q>;
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    unsigned at;
    if (MASKED) {
      // ODD: pull, or the opposite own slot when bounced; EVEN: the reverse
      const bool bb = (bounce >> i) & 1u;
      const unsigned pull = (PZ ? z_pick(b, -Lt::c(i, 2)) : b.at) + p.slot[0][i];
      at = (ODD != bb) ? pull : b.at + p.slot[3][i];
    } else {
      at = ODD ? z_pick(b, -Lt::c(i, 2)) + p.slot[0][i] : b.at + p.slot[3][i];
    }
    f[i] = Store<S>::load_c(F + at);
  }
}
template <int Q, class S, bool ODD, bool MASKED, bool PZ>
__device__ __forceinline__ void pair_store(S* __restrict__ F, const ZBase& b0, const StepParams& p, uint32_t elide,
                                           const float (&f)[Q]) {
  using Lt = Lattice<Q>;
  ZBase b = b0;
  b.at = after(b.at, f[0]);
  if (!MASKED || PZ) {
    b.below = after(b.below, f[0]);
    b.above = after(b.above, f[0]);
  } else {
    b.below = b.above = b.at;
  }
#pragma unroll
  for (int i = 0; i < Q; ++i) {
    const unsigned at = ODD ? z_pick(b, Lt::c(i, 2)) + p.slot[2][i] : b.at + p.slot[1][i];
    store_slot<S>(F + at, f[i], MASKED && ((elide >> i) & 1u), p);
  }
}

// One pair: cells (x, y, za) and, with has_b, (x, y, za + 32) at storage
// indices sa and sa + 32, with their (bounce, elide) words.
template <int Q, class S, int CL, bool ODD, bool MASKED, bool PZ>
__device__ __forceinline__ void pair_step(S* __restrict__ F, const GridDesc& g, const StepParams& p, int x, int y,
                                          int za, bool has_b, unsigned sa, uint2 ma, uint2 mb,
                                          float* __restrict__ rho_out, float* __restrict__ u_out) {
  const unsigned sb = sa + 32u;
  const int zb = za + 32;
  const ZBase ba = z_base<!MASKED || PZ>(g, sa, za), bb = z_base<!MASKED || PZ>(g, sb, zb);
  float fa[Q], fb[Q];
  pair_load<Q, S, ODD, MASKED, PZ>(F, ba, p, ma.x, fa);
  if (has_b) pair_load<Q, S, ODD, MASKED, PZ>(F, bb, p, mb.x, fb);
  if constexpr (!kPairPack<Q, CL, MASKED>) {
    cell_collide<Q, S, CL>(g, p, rho_out, u_out, x, y, za, sa, fa, p.om0f);
    pair_store<Q, S, ODD, MASKED, PZ>(F, ba, p, ma.y, fa);
    if (has_b) {
      cell_collide<Q, S, CL>(g, p, rho_out, u_out, x, y, zb, sb, fb, p.om0f);
      pair_store<Q, S, ODD, MASKED, PZ>(F, bb, p, mb.y, fb);
    }
  } else {
    F2 f[Q], rho, u[3], cs2 = F2(0.f);
    if (CL == CL_MLP) cs2 = F2(p.cs2[sa], has_b ? p.cs2[sb] : 0.f);
#pragma unroll
    for (int i = 0; i < Q; ++i) f[i] = F2(fa[i], has_b ? fb[i] : 0.f);
    collide_cell<Q, F2, CL, Store<S>::kDev>(f, p, F2(p.om0f), cs2, rho, u);
    if (p.write_macro) {
      const long long a = aidx(g, x, y, za);
      auto put = [&](float* out, F2 v) {
        out[a] = v.lo();
        if (has_b) out[a + 32] = v.hi();
      };
      if (p.write_rho) put(rho_out, rho);
      if (p.write_vel) {
        put(u_out, u[0]);
        put(u_out + g.L, u[1]);
        put(u_out + 2 * g.L, u[2]);
      }
    }
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      fa[i] = f[i].lo();
      fb[i] = f[i].hi();
    }
    pair_store<Q, S, ODD, MASKED, PZ>(F, ba, p, ma.y, fa);
    if (has_b) pair_store<Q, S, ODD, MASKED, PZ>(F, bb, p, mb.y, fb);
  }
}

// FUSED: 0 no links, 1 the two-word masks, 2 the one-word masks. PZ: with links,
// the z axis wraps (three bases per cell: five blocks instead of six).
template <int Q, class S, int CL, bool ODD, int FUSED, bool PZ = false>
__global__ void __launch_bounds__(kPairThreads, kPairBlocks<Q, CL, FUSED != 0 && !PZ, ODD>)
    k_step_pair(S* __restrict__ F, const __grid_constant__ GridDesc g, const __grid_constant__ StepParams p,
                const __grid_constant__ FaceWork fw, int planes, float* __restrict__ rho_out,
                float* __restrict__ u_out) {
  wait_before();
  let_next();
  if ((int)blockIdx.z < fw.fz) {
    face_cell<Q, S, CL, ODD, FUSED != 0>(F, g, p, fw, rho_out, u_out);
    return;
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int za = blockIdx.x * (2 * blockDim.x) + 64 * w + lane + 1;
  const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int x0 = (blockIdx.z - fw.fz) * planes + 1;
  int x1 = min(g.nx, x0 + planes - 1);
  if (za > g.nz || y > g.ny) return;
  const bool has_b = za + 32 <= g.nz;
  // cells on a periodic x or y face belong to the face blocks; skipped by the
  // loop's range, the loop body has no branch
  if (wraps(g.periodic & 2, y, g.ny)) return;
  if (g.periodic & 1) {
    x0 = max(x0, 2);
    x1 = min(x1, g.nx - 1);
    if (x0 > x1) return;
  }
  const unsigned pl = (unsigned)g.plane;
  const unsigned s0 = (unsigned)sidx(g, x0, y, za);
  auto words = [&](unsigned s) {  // as stored: split when used
    uint2 v = make_uint2(0u, 0u);
    if (FUSED == 1) v = p.mask[s];
    if (FUSED == 2) v.x = p.mask32[s];
    return v;
  };
  auto split = [](uint2 v) { return FUSED == 2 ? link_words<Q>(v.x) : v; };
  uint2 wa = words(s0), wb = make_uint2(0u, 0u);
  if (has_b) wb = words(s0 + 32u);
  for (int x = x0; x <= x1; ++x) {
    const unsigned sa = s0 + (unsigned)(x - x0) * pl;
    uint2 na = make_uint2(0u, 0u), nb = make_uint2(0u, 0u);
    if (FUSED && x < x1) {
      na = words(sa + pl);
      if (has_b) nb = words(sa + pl + 32u);
    }
    // D3Q27 (the closures' and its own registers leave room for both bodies):
    // 64 cells without a link take the body without selects
    if (FUSED && (Q != 27 || __any_sync(__activemask(), wa.x | wa.y | wb.x | wb.y)))
      pair_step<Q, S, CL, ODD, true, PZ>(F, g, p, x, y, za, has_b, sa, split(wa), split(wb), rho_out, u_out);
    else
      pair_step<Q, S, CL, ODD, false, PZ>(F, g, p, x, y, za, has_b, sa, make_uint2(0u, 0u), make_uint2(0u, 0u), rho_out,
                                      u_out);
    wa = na;
    wb = nb;
  }
}

// FP16 storage without links, rows aligned: two neighbouring cells per thread,
// z and z + 1 (z odd), so that a population of the two that is not shifted
// along z is one 4-byte access: all of them in the even step, nine of nineteen
// in the odd one. Bound by the number of accesses (with one cell per thread a
// warp's 64-byte loads and stores are as many as FP32's 128-byte ones):
// 320x208x256 D3Q19, ms per step, 0.269 against 0.342. With fused links the
// two cells' selects undo it (0.49 against 0.355 for k_step_pair).
template <int Q, int CL, bool ODD>
__global__ void __launch_bounds__(kPairThreads, kPairBlocks<Q, CL, CL == CL_NONE, ODD>)
    k_step_half2(__half* __restrict__ F, const __grid_constant__ GridDesc g, const __grid_constant__ StepParams p,
                 const __grid_constant__ FaceWork fw, int planes, float* __restrict__ rho_out,
                 float* __restrict__ u_out) {
  using Lt = Lattice<Q>;
  wait_before();
  let_next();
  if ((int)blockIdx.z < fw.fz) {
    face_cell<Q, __half, CL, ODD, false>(F, g, p, fw, rho_out, u_out);
    return;
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int za = blockIdx.x * (2 * blockDim.x) + 64 * w + 2 * lane + 1;
  const int y = blockIdx.y * blockDim.y + threadIdx.y + 1;
  int x0 = (blockIdx.z - fw.fz) * planes + 1;
  int x1 = min(g.nx, x0 + planes - 1);
  if (za > g.nz || y > g.ny) return;
  const bool has_b = za < g.nz;
  if (wraps(g.periodic & 2, y, g.ny)) return;
  if (g.periodic & 1) {
    x0 = max(x0, 2);
    x1 = min(x1, g.nx - 1);
  }
  for (int x = x0; x <= x1; ++x) {
    const unsigned s = (unsigned)sidx(g, x, y, za);
    const ZBase ba = z_base<true>(g, s, za), bb = z_base<true>(g, s + 1u, za + 1);
    float fa[Q], fb[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const unsigned off = ODD ? p.slot[0][i] : p.slot[3][i];
      if (!ODD || Lt::c(i, 2) == 0) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(F + (s + off)));
        fa[i] = v.x;
        fb[i] = v.y;
      } else {
        fa[i] = __half2float(F[z_pick(ba, -Lt::c(i, 2)) + off]);
        fb[i] = has_b ? __half2float(F[z_pick(bb, -Lt::c(i, 2)) + off]) : 0.f;
      }
    }
    if constexpr (CL == CL_NONE) {
      cell_collide<Q, __half, CL>(g, p, rho_out, u_out, x, y, za, s, fa, p.om0f);
      if (has_b) cell_collide<Q, __half, CL>(g, p, rho_out, u_out, x, y, za + 1, s + 1u, fb, p.om0f);
    } else {
      F2 f[Q], rho, u[3], cs2 = F2(0.f);
      if (CL == CL_MLP) cs2 = F2(p.cs2[s], has_b ? p.cs2[s + 1u] : 0.f);
#pragma unroll
      for (int i = 0; i < Q; ++i) f[i] = F2(fa[i], fb[i]);
      collide_cell<Q, F2, CL, true>(f, p, F2(p.om0f), cs2, rho, u);
      if (p.write_macro) {
        const long long a = aidx(g, x, y, za);
        auto put = [&](float* out, F2 v) {
          out[a] = v.lo();
          if (has_b) out[a + 1] = v.hi();
        };
        if (p.write_rho) put(rho_out, rho);
        if (p.write_vel) {
          put(u_out, u[0]);
          put(u_out + g.L, u[1]);
          put(u_out + 2 * g.L, u[2]);
        }
      }
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        fa[i] = f[i].lo();
        fb[i] = f[i].hi();
      }
    }
    ZBase sa = ba, sb = bb;
    sa.at = after(sa.at, fa[0]);
    sa.below = after(sa.below, fa[0]);
    sa.above = after(sa.above, fa[0]);
    sb.at = sa.at + 1u;
    sb.below = after(sb.below, fb[0]);
    sb.above = after(sb.above, fb[0]);
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const unsigned off = ODD ? p.slot[2][i] : p.slot[1][i];
      const __half2 h = __floats2half2_rn(fa[i], fb[i]);
      if (!ODD || Lt::c(i, 2) == 0) {
        __half* at = F + (sa.at + off);
        if (has_b) *reinterpret_cast<__half2*>(at) = h;
        else *at = __low2half(h);
      } else {
        F[z_pick(sa, Lt::c(i, 2)) + off] = __low2half(h);
        if (has_b) F[z_pick(sb, Lt::c(i, 2)) + off] = __high2half(h);
      }
    }
  }
}

inline void step_launch_shape(const GridDesc& g, dim3& grid, dim3& block) {
  int tz = ((g.nz + 31) / 32) * 32;
  if (tz > 256) tz = 256;
  int ty = 256 / tz;
  block = dim3(tz, ty, 1);
  grid = dim3((g.nz + tz - 1) / tz, (g.ny + ty - 1) / ty, g.nx);
}

// x planes that a block walks: up to `most`, fewer where that would leave
// SMs without a block (a small domain's step is one block's chain of planes).
constexpr int kSms = 148;  // of a B200
inline int planes_per_block(const GridDesc& g, const dim3& grid, int most) {
  int planes = most;
  while (planes > 1 && (long long)grid.x * grid.y * ((g.nx + planes - 1) / planes) < 4 * kSms) planes /= 2;
  return planes;
}

// The one-cell stream-collide: the same blocks, several x planes each.
inline int plane_launch_shape(const GridDesc& g, dim3& grid, dim3& block) {
  step_launch_shape(g, grid, block);
  const int planes = planes_per_block(g, grid, kOnePlanes);
  grid.z = (g.nx + planes - 1) / planes;
  return planes;
}

// Launch of the TMA-staged variant (stream_collide_tma.cuh).
template <int Q, class S, int CL>
cudaError_t step_tma(const DomainDev& d, const StepParams& p, int parity_in, cudaStream_t st);

// Two-cells-per-thread shape: 32-thread groups cover 64 cells of a row.
inline int pair_launch_shape(const GridDesc& g, dim3& grid, dim3& block) {
  int tz = ((g.nz + 63) / 64) * 32;
  if (tz > kPairThreads) tz = kPairThreads;
  int ty = kPairThreads / tz;
  block = dim3(tz, ty, 1);
  grid = dim3((g.nz + 2 * tz - 1) / (2 * tz), (g.ny + ty - 1) / ty, g.nx);
  const int planes = planes_per_block(g, grid, kPairPlanes);
  grid.z = (g.nx + planes - 1) / planes;
  return planes;
}

template <int Q, class S, int CL>
cudaError_t step_q_s_cl(const DomainDev& d, const StepParams& p, int parity_in, cudaStream_t st) {
  if (d.variant == 1) return step_tma<Q, S, CL>(d, p, parity_in, st);
  dim3 grid, block;
  using M = typename MacroT<S>::T;
  const bool fused = p.mask != nullptr;
  S* F = (S*)d.F;
  M* rho = (M*)d.rho;
  M* u = (M*)d.u;
  if constexpr (std::is_same<S, __half>::value) {
    // even element offsets put z odd on a 4-byte boundary (packed rows need not)
    if (d.variant == 0 && !fused && (d.g.zoff + 1) % 2 == 0 && d.g.pitch % 2 == 0) {
      const int planes = pair_launch_shape(d.g, grid, block);
      const FaceWork fw = face_work(d.g, true, block.x * block.y, grid.x, grid.y);
      grid.z += fw.fz;
      return launch_after(parity_in == 0 ? k_step_half2<Q, CL, true> : k_step_half2<Q, CL, false>, grid, block, 0, st, F,
                          d.g, p, fw, planes, rho, u);
    }
  }
  if constexpr (!std::is_same<S, double>::value) {
    if (d.variant == 0 && takes_pairs<Q, S, CL>(d.g, fused)) {
      const int planes = pair_launch_shape(d.g, grid, block);
      const FaceWork fw = face_work(d.g, true, block.x * block.y, grid.x, grid.y);
      grid.z += fw.fz;
      auto go = [&](auto kern) { return launch_after(kern, grid, block, 0, st, F, d.g, p, fw, planes, rho, u); };
      const bool odd = parity_in == 0;
      if (!fused) return odd ? go(k_step_pair<Q, S, CL, true, 0>) : go(k_step_pair<Q, S, CL, false, 0>);
      if constexpr (kPairWraps<Q, CL>)
        if (d.g.periodic & 4) {
          if (!p.mask32) return odd ? go(k_step_pair<Q, S, CL, true, 1, true>) : go(k_step_pair<Q, S, CL, false, 1, true>);
          return odd ? go(k_step_pair<Q, S, CL, true, 2, true>) : go(k_step_pair<Q, S, CL, false, 2, true>);
        }
      if constexpr (kPairLinks<Q, S, CL>) {
        if (!p.mask32) return odd ? go(k_step_pair<Q, S, CL, true, 1>) : go(k_step_pair<Q, S, CL, false, 1>);
        return odd ? go(k_step_pair<Q, S, CL, true, 2>) : go(k_step_pair<Q, S, CL, false, 2>);
      }
    }
  }
  const int planes = plane_launch_shape(d.g, grid, block);
  const FaceWork fw = face_work(d.g, false, block.x * block.y, grid.x, grid.y);
  grid.z += fw.fz;
  auto go = [&](auto kern) { return launch_after(kern, grid, block, 0, st, F, d.g, p, fw, planes, rho, u); };
  if (parity_in == 0) return fused ? go(k_stream_collide<Q, S, CL, true, true>) : go(k_stream_collide<Q, S, CL, true, false>);
  return fused ? go(k_stream_collide<Q, S, CL, false, true>) : go(k_stream_collide<Q, S, CL, false, false>);
}

template <int Q, class S>
cudaError_t step_q_s(const DomainDev& d, const StepParams& p, int closure, int parity_in, cudaStream_t st) {
  switch (closure) {
    case CL_NONE: return step_q_s_cl<Q, S, CL_NONE>(d, p, parity_in, st);
    case CL_ASL_INTENT: return step_q_s_cl<Q, S, CL_ASL_INTENT>(d, p, parity_in, st);
    case CL_SMAGORINSKY: return step_q_s_cl<Q, S, CL_SMAGORINSKY>(d, p, parity_in, st);
    case CL_MLP:
      // The learned closure is built for the lattices and storages it is trained for.
      if constexpr ((Q == 19 || Q == 27) && !std::is_same<S, double>::value)
        return step_q_s_cl<Q, S, CL_MLP>(d, p, parity_in, st);
      else
        return cudaErrorNotSupported;
  }
  return cudaErrorInvalidValue;
}

template <int Q>
cudaError_t step_q(const DomainDev& d, const StepParams& p, int closure, int parity_in, cudaStream_t st) {
  switch (d.storage) {
    case ST_F32: return step_q_s<Q, float>(d, p, closure, parity_in, st);
    case ST_F16: return step_q_s<Q, __half>(d, p, closure, parity_in, st);
    case ST_F64: return step_q_s<Q, double>(d, p, closure, parity_in, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace aslb
