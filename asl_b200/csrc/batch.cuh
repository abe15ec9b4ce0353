// Batched stream-collide and boundary links (kernels and their launchers):
// many independent domains of different sizes and viscosities advanced by
// one launch per step (plus one per condition position), instead of one
// launch per domain and condition. Each domain keeps its own allocation and
// layout; a device table maps the launch's tiles (one x plane of one domain,
// its cells taken 256 at a time, z fastest across y rows) and links to
// domains. Each block of the persistent grid takes a contiguous run of tiles
// holding an equal share of the batch's cells (BatchWork), the blocks of a
// group of four interleaving its planes, so a block's domain changes rarely
// and neighbouring planes of a domain are streamed together.
// Instantiated per storage in batch_<type>.cu.
#pragma once
#include <climits>
#include "kernels.h"
#include "stream_collide.cuh"
#include "bc_links.cuh"

namespace aslb {

// Launch shapes of the persistent batched step: one cell per thread at 4, 3
// or 2 resident blocks of 256 threads per SM (64 / 80 / 128 registers), or
// two cells per thread (both cells' loads in flight before the collision) at 3
// blocks of 256 or 2 of 320 threads (80 / 96 registers). aslb_batch_run times
// them on the batch and keeps the fastest.
constexpr int kBatchShapes = 5;
__host__ __device__ constexpr int batch_shape_blocks(int shape) {
  return shape == 0 ? 4 : (shape == 1 || shape == 3 ? 3 : 2);
}
__host__ __device__ constexpr bool batch_shape_pair(int shape) { return shape >= 3; }
__host__ __device__ constexpr int batch_shape_threads(int shape) { return shape == 4 ? 320 : 256; }

// A domain's fused-link words of a cell (LINKS: see BatchLinks). Where some
// cell has both kinds of links, FP16 steps, bound by their instructions and not
// by their bytes, read the two words (48 channels: 0.263 ms per step, 0.276
// with the walls of the one-word form decoded).
// Single: ms per step of channels, against the general form, in the fastest
// shape: FP32 48 / 160 domains 0.362 / 1.143 (0.364 / 1.141), periodic 0.344 /
// 1.093 (0.359 / 1.109); FP16 0.256 / 0.790 (0.261 / 0.806). It is not built
// where it was slower: FP16 periodic 0.252 (0.243), FP64 0.631 (0.619), nor
// for D3Q27, whose one-word masks never hold both kinds.
template <int Q, class S, bool FLAT>
constexpr bool kBatchSingle = Q != 27 && (sizeof(S) == 4 || (sizeof(S) == 2 && FLAT));
template <int Q, class S, int LINKS>
__device__ __forceinline__ uint2 batch_links(const BatchDom& D, unsigned s) {
  if (LINKS == kLinksSingle) {
    const uint32_t w = D.mask32[s];
    return (w >> 31) ? make_uint2(0u, w & 0x7fffffffu) : make_uint2(w, 0u);
  }
  if (sizeof(S) == 2) return D.mask[s];
  return D.mask32 ? link_words<Q>(D.mask32[s]) : D.mask[s];
}

// Neighbour offsets: FLAT when no domain of the batch is periodic (the three
// displacements per axis are then fixed, and the compiler folds them into one
// add per population instead of carrying nine selected offsets per cell).
template <bool FLAT>
__device__ __forceinline__ void batch_offsets(const GridDesc& g, int x, int y, int z, int (&ox)[3], int (&oy)[3],
                                              int (&oz)[3]) {
  if (FLAT) {
    ox[0] = -(int)g.plane; ox[1] = 0; ox[2] = (int)g.plane;
    oy[0] = -g.pitch; oy[1] = 0; oy[2] = g.pitch;
    oz[0] = -1; oz[1] = 0; oz[2] = 1;
  } else {
    nb_offsets(g, x, y, z, ox, oy, oz);
  }
}

// Collision and stores of one cell whose store offsets are recomputed after
// the collision (y and s are made to depend on its result), so the offsets
// used by the loads die with them instead of living across the collision.
template <int Q, class S, bool ODD, bool MASKED, bool FLAT>
__device__ __forceinline__ void batch_finish(S* __restrict__ F, const GridDesc& g, const StepParams& p,
                                             typename MacroT<S>::T* __restrict__ rho_out,
                                             typename MacroT<S>::T* __restrict__ u_out, int x, int y, int z,
                                             unsigned s, uint32_t elide, typename Store<S>::C (&f)[Q],
                                             typename Store<S>::C om0) {
  cell_collide<Q, S, CL_NONE>(g, p, rho_out, u_out, x, y, z, s, f, om0);
  const int y2 = (int)after((unsigned)y, f[0]);
  int ox[3], oy[3], oz[3];
  batch_offsets<FLAT>(g, x, y2, z, ox, oy, oz);
  cell_store<Q, S, ODD, MASKED>(F, p, (unsigned)g.dstride, after(s, f[0]), ox, oy, oz, elide, f);
}

// The domain holding `tile`, searched from d (tiles ascend in the table).
__device__ __forceinline__ int batch_domain(const BatchDom* __restrict__ doms, int ndom, long long tile, int d) {
  if (d < 0) {
    int lo = 0, hi = ndom - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (doms[mid].tile0 <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
  }
  while (d + 1 < ndom && doms[d + 1].tile0 <= tile) ++d;
  return d;
}

// One cell per thread. The blocks of a group share a run of tiles and take
// every group-th tile of it (block j: tiles j, j + K, ...), so neighbouring
// planes, whose populations each pulls from the other, are streamed at the
// same time by neighbouring blocks; a block's planes of one domain are walked
// as one sequence of cells 256 at a time, so the next cell's link word is
// fetched one step ahead across plane boundaries too and the domain's table
// entry is read once per domain, not once per plane.
template <int Q, class S, bool ODD, int LINKS, bool FLAT, int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS)
    k_batch_step(const BatchDom* __restrict__ doms, int ndom, const long long* __restrict__ starts, int K,
                 const StepParams p) {
  using C = typename Store<S>::C;
  using M = typename MacroT<S>::T;
  const int grp = (int)blockIdx.x / K;
  wait_before();
  let_next();
  long long tile = starts[grp] + (int)blockIdx.x % K;
  const long long tend = starts[grp + 1];
  int d = -1;
  while (tile < tend) {
    d = batch_domain(doms, ndom, tile, d);
    const BatchDom& D = doms[d];
    const GridDesc g = D.g;
    // this block's planes of the domain in the run: xa, xa + K, ... <= xb
    const int xa = (int)(tile - D.tile0) + 1;
    const int xb = (int)(min(tend, D.tile0 + g.nx) - D.tile0);
    tile += (long long)K * ((xb - xa) / K + 1);
    const unsigned plane_cells = (unsigned)(g.ny * g.nz);
    const unsigned nz = (unsigned)g.nz, nz_inv = D.nz_inv;
    S* F = (S*)D.F;
    const C om0 = std::is_same<C, double>::value ? C(D.om0d) : C(D.om0f);
    const bool masked = LINKS && D.mask;
    // storage index of cell l of plane x (y rows of nz cells, z fastest)
    auto cell_index = [&](int x, unsigned l, int& y, int& z) {
      unsigned yq = __umulhi(l + 1u, nz_inv);
      if (yq * nz > l) --yq;  // exact quotient for l < 2^32 / nz - 1
      y = (int)yq + 1;
      z = (int)(l - yq * nz) + 1;
      return (unsigned)sidx(g, x, y, z);
    };
    // (x, l): this thread's cell; advancing by 256 cells may cross planes
    int x = xa;
    unsigned l = threadIdx.x;
    while (l >= plane_cells && x <= xb) {
      l -= plane_cells;
      x += K;
    }
    uint2 mnext = make_uint2(0u, 0u);
    if (masked && x <= xb) {
      int y1, z1;
      mnext = batch_links<Q, S, LINKS>(D, cell_index(x, l, y1, z1));
    }
    while (x <= xb) {
      int y, z;
      const unsigned s = cell_index(x, l, y, z);
      const uint32_t bounce = mnext.x, elide = mnext.y;
      int xn = x;
      unsigned ln = l + 256u;
      while (ln >= plane_cells && xn <= xb) {
        ln -= plane_cells;
        xn += K;
      }
      if (masked && xn <= xb) {
        int y1, z1;
        mnext = batch_links<Q, S, LINKS>(D, cell_index(xn, ln, y1, z1));
      }
      int ox[3], oy[3], oz[3];
      batch_offsets<FLAT>(g, x, y, z, ox, oy, oz);
      C f[Q];
      cell_load<Q, S, ODD, LINKS != 0>(F, (unsigned)g.dstride, s, ox, oy, oz, bounce, f);
      batch_finish<Q, S, ODD, LINKS != 0, FLAT>(F, g, p, (M*)D.rho, (M*)D.u, x, y, z, s, elide, f, om0);
      x = xn;
      l = ln;
    }
  }
}

// Two cells per thread, NT cells apart in the block's sequence of cells,
// collided as a pair in packed FP32 (no periodic domain in the batch). The
// pair too is walked across plane boundaries: the planes of such batches hold
// two to eight times NT cells, and stopping at each plane's end left a third
// of the threads without a second cell.
template <int Q, class S, bool ODD, int LINKS, int BLOCKS, int NT>
__global__ void __launch_bounds__(NT, BLOCKS)
    k_batch_step_pair(const BatchDom* __restrict__ doms, int ndom, const long long* __restrict__ starts, int K,
                      const StepParams p) {
  using M = typename MacroT<S>::T;
  int d = -1;
  const int grp = (int)blockIdx.x / K;
  wait_before();
  let_next();
  long long tile = starts[grp] + (int)blockIdx.x % K;
  const long long tend = starts[grp + 1];
  while (tile < tend) {
    d = batch_domain(doms, ndom, tile, d);
    const BatchDom& D = doms[d];
    const GridDesc g = D.g;
    // this block's planes of the domain in the run, as in k_batch_step
    const int x0 = (int)(tile - D.tile0) + 1;
    const int x1 = (int)(min(tend, D.tile0 + g.nx) - D.tile0);
    tile += (long long)K * ((x1 - x0) / K + 1);
    const unsigned plane_cells = (unsigned)(g.ny * g.nz);
    const unsigned nz = (unsigned)g.nz, nz_inv = D.nz_inv;
    S* F = (S*)D.F;
    const bool masked = LINKS && D.mask;
    const float om0 = D.om0f;
    auto row_of = [&](unsigned l, int& y, int& z) {
      unsigned yq = __umulhi(l + 1u, nz_inv);
      if (yq * nz > l) --yq;  // exact quotient for l < 2^32 / nz - 1
      y = (int)yq + 1;
      z = (int)(l - yq * nz) + 1;
    };
    auto cell_index = [&](int x, unsigned l) {
      int y, z;
      row_of(l, y, z);
      return (unsigned)sidx(g, x, y, z);
    };
    auto advance = [&](int& x, unsigned& l, unsigned by) {
      l += by;
      while (l >= plane_cells && x <= x1) {
        l -= plane_cells;
        x += K;
      }
    };
    int xa = x0, xb;
    unsigned la = threadIdx.x, lb;
    advance(xa, la, 0u);
    xb = xa;
    lb = la;
    advance(xb, lb, (unsigned)NT);
    uint2 na = make_uint2(0u, 0u), nb = make_uint2(0u, 0u);
    if (masked) {
      if (xa <= x1) na = batch_links<Q, S, LINKS>(D, cell_index(xa, la));
      if (xb <= x1) nb = batch_links<Q, S, LINKS>(D, cell_index(xb, lb));
    }
    while (xa <= x1) {
      const bool has_b = xb <= x1;
      const unsigned sa = cell_index(xa, la), sb = has_b ? cell_index(xb, lb) : 0u;
      const uint2 ma = na, mb = nb;
      const int xa0 = xa, xb0 = xb;
      const unsigned la0 = la, lb0 = lb;
      advance(xa, la, 2u * NT);
      advance(xb, lb, 2u * NT);
      if (masked) {
        if (xa <= x1) na = batch_links<Q, S, LINKS>(D, cell_index(xa, la));
        if (xb <= x1) nb = batch_links<Q, S, LINKS>(D, cell_index(xb, lb));
      }
      int ox[3], oy[3], oz[3];
      batch_offsets<true>(g, 0, 0, 0, ox, oy, oz);
      float fa[Q], fb[Q];
      cell_load<Q, S, ODD, LINKS != 0>(F, (unsigned)g.dstride, sa, ox, oy, oz, ma.x, fa);
      if (has_b) cell_load<Q, S, ODD, LINKS != 0>(F, (unsigned)g.dstride, sb, ox, oy, oz, mb.x, fb);
      F2 f[Q], rho, u[3];
#pragma unroll
      for (int i = 0; i < Q; ++i) f[i] = F2(fa[i], has_b ? fb[i] : 0.f);
      collide_cell<Q, F2, CL_NONE, Store<S>::kDev>(f, p, F2(om0), F2(0.f), rho, u);
      if (p.write_macro) {
        int ya, za, yb, zb;
        row_of(la0, ya, za);
        row_of(lb0, yb, zb);
        const long long aa = aidx(g, xa0, ya, za), ab = aidx(g, xb0, yb, zb);
        auto put = [&](M* out, F2 v) {
          out[aa] = v.lo();
          if (has_b) out[ab] = v.hi();
        };
        if (p.write_rho) put((M*)D.rho, rho);
        if (p.write_vel) {
          put((M*)D.u, u[0]);
          put((M*)D.u + g.L, u[1]);
          put((M*)D.u + 2 * g.L, u[2]);
        }
      }
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        fa[i] = f[i].lo();
        fb[i] = f[i].hi();
      }
      // store offsets recomputed after the collision (see batch_finish)
      const unsigned ds2 = after((unsigned)g.dstride, fa[0]);
      cell_store<Q, S, ODD, LINKS != 0>(F, p, ds2, after(sa, fa[0]), ox, oy, oz, ma.y, fa);
      if (has_b) cell_store<Q, S, ODD, LINKS != 0>(F, p, ds2, after(sb, fb[0]), ox, oy, oz, mb.y, fb);
    }
  }
}

template <int Q, class S>
__global__ void __launch_bounds__(256)
    k_batch_links(const BatchBc* __restrict__ bcs, int nbc, long long nlinks, int parity) {
  const long long t = min((long long)blockIdx.x * blockDim.x + threadIdx.x, nlinks);
  int lo = 0, hi = nbc - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (bcs[mid].link0 <= t) lo = mid; else hi = mid - 1;
  }
  const BatchBc& B = bcs[lo];
  link_apply<Q, S>((S*)B.F, B.dstride, B.links, t < nlinks ? INT_MAX : 0, (int)(t - B.link0), B.ls, B.bp, parity);
}

template <int Q, class S, int SHAPE, bool FLAT, int LINKS>
cudaError_t batch_step_links(const BatchDom* doms, int ndom, const BatchWork& w, const StepParams& p, int parity_in,
                             cudaStream_t st) {
  constexpr int BLOCKS = batch_shape_blocks(SHAPE), NT = batch_shape_threads(SHAPE);
  const int grid = w.grid[BLOCKS - 2], K = w.group[BLOCKS - 2];
  const long long* starts = w.starts + w.off[BLOCKS - 2];
  const bool odd = parity_in == 0;
  auto go = [&](auto kern) { return launch_after(kern, grid, NT, 0, st, doms, ndom, starts, K, p); };
  if constexpr (batch_shape_pair(SHAPE))
    return odd ? go(k_batch_step_pair<Q, S, true, LINKS, BLOCKS, NT>) : go(k_batch_step_pair<Q, S, false, LINKS, BLOCKS, NT>);
  else
    return odd ? go(k_batch_step<Q, S, true, LINKS, FLAT, BLOCKS>) : go(k_batch_step<Q, S, false, LINKS, FLAT, BLOCKS>);
}

// Two cells per thread are built for D3Q15 / D3Q19 in 4- and 2-byte storage
// without a periodic domain; other batches take the one-cell shape with the
// same residency (in batches of periodic channels, two cells per thread with
// the offsets wrapped were 6 to 20 % slower than one).
template <int Q, class S, int SHAPE, bool FLAT>
cudaError_t batch_step_shape(const BatchDom* doms, int ndom, const BatchWork& w, int links, const StepParams& p,
                             int parity_in, cudaStream_t st) {
  if constexpr (batch_shape_pair(SHAPE) && (!FLAT || Q == 27 || sizeof(S) == 8)) {
    return batch_step_shape<Q, S, SHAPE == 3 ? 1 : 2, FLAT>(doms, ndom, w, links, p, parity_in, st);
  } else {
    if (links == kLinksNone) return batch_step_links<Q, S, SHAPE, FLAT, kLinksNone>(doms, ndom, w, p, parity_in, st);
    if constexpr (kBatchSingle<Q, S, FLAT>)
      if (links == kLinksSingle)
        return batch_step_links<Q, S, SHAPE, FLAT, kLinksSingle>(doms, ndom, w, p, parity_in, st);
    return batch_step_links<Q, S, SHAPE, FLAT, kLinksBoth>(doms, ndom, w, p, parity_in, st);
  }
}

template <int Q, class S, bool FLAT>
cudaError_t batch_step_flat(const BatchDom* doms, int ndom, const BatchWork& w, int links, const StepParams& p,
                            int parity_in, int shape, cudaStream_t st) {
  switch (shape) {
    case 0: return batch_step_shape<Q, S, 0, FLAT>(doms, ndom, w, links, p, parity_in, st);
    case 1: return batch_step_shape<Q, S, 1, FLAT>(doms, ndom, w, links, p, parity_in, st);
    case 2: return batch_step_shape<Q, S, 2, FLAT>(doms, ndom, w, links, p, parity_in, st);
    case 3: return batch_step_shape<Q, S, 3, FLAT>(doms, ndom, w, links, p, parity_in, st);
    case 4: return batch_step_shape<Q, S, 4, FLAT>(doms, ndom, w, links, p, parity_in, st);
  }
  return cudaErrorInvalidValue;
}

template <int Q, class S>
cudaError_t batch_step_impl(const BatchDom* doms, int ndom, const BatchWork& w, int links, const StepParams& p,
                            int parity_in, int shape, cudaStream_t st) {
  if (w.ntiles <= 0) return cudaSuccess;
  return w.periodic ? batch_step_flat<Q, S, false>(doms, ndom, w, links, p, parity_in, shape, st)
                    : batch_step_flat<Q, S, true>(doms, ndom, w, links, p, parity_in, shape, st);
}

template <int Q, class S>
cudaError_t batch_links_impl(const BatchBc* bcs, int nbc, long long nlinks, int parity, cudaStream_t st) {
  if (nlinks <= 0) return cudaSuccess;
  return launch_after(k_batch_links<Q, S>, (unsigned)((nlinks + 255) / 256), 256, 0, st, bcs, nbc, nlinks, parity);
}

}  // namespace aslb
