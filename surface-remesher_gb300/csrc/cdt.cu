// cdt.cu -- the constrained Delaunay triangulation of the CDT stage on the
// GPU: the reference hands gDel2D (gDel2D/GPU/GpuDelaunay.cu:46) the free
// sites and the constraint points (delaunay.h:46-67) with the constraint
// segments between those points (delaunay.h:69-75), and gDel2D triangulates
// them and then inserts the segments by flips (GpuDelaunay.cu:749,
// splitAndFlip).  Here:
//
//   1. the sites' Delaunay triangulation (delaunay.cu, exact on the lattice);
//   2. adjacency from a hash of directed edges;
//   3. the constraint points inserted in rounds: every point locates itself
//      by a walk, claims the triangles its split changes (atomicMin of a
//      priority, a fixed bijective hash of its index: claims by plain index
//      let only the first of a run of neighbours win each round), and the
//      points that won all their claims split (1 -> 3 inside a triangle,
//      2 -> 4 on an edge, a fan over the visible hull edges outside the
//      hull); after each round, two flip rounds over the changed triangles
//      (four rounds with their flips per read-back);
//   4. each segment made an edge by flipping the edges that cross it
//      (Sloan's method, cdt_core.cuh recover_segment) and marked: segments
//      already edges at once, the others in rounds where each claims the
//      triangles around the vertices of its crossing edges and the winners
//      are recovered side by side, the rare long ones (or ones with a vertex
//      inside) by one thread;
//   5. flip rounds that restore the Delaunay property on every edge that is
//      not a constraint: the result is the constrained Delaunay
//      triangulation;
//   6. the triangles written in a fixed order (by their smallest vertex, then
//      the next one), so the output does not depend on scheduling.
//
// A flip round: every changed triangle tests its edges towards
// higher-numbered neighbours (cdt_core.cuh first_flip); a flip claims its two
// triangles and their four outer neighbours (whose back links it rewrites);
// the flips that won all six claims are applied.  Lawson's flips end (each
// one lowers the lifted surface), so the rounds end; a round limit turns a
// runaway into an error instead of a hang.
//
// Coordinates: sites (x, y) on the pixel lattice scaled by 2^15; a
// constraint point (px, py) maps to ((px - left) / scale, (py - lower) /
// scale) pixels, rounded to the nearest 2^-15 pixel -- the same frame as
// delaunayInput's (x * scale + left, y * scale + lower) for the sites.  All
// predicates are then exact integers (cdt_core.cuh).  Symbolic perturbation
// ranks: a site ranks y n + x (as in the sites' triangulation), constraint
// point j ranks n^2 + j.
#include "gcvt_internal.cuh"
#include "cdt_core.cuh"
#include "../../include/gcvt_gb300.h"

#include <cmath>
#include <utility>

namespace cvtgb {

using cdt::i64;
using cdt::Mesh;

namespace {

constexpr int kWalk = 1 << 20;    // steps of one point location
constexpr int kRotate = 4096;     // triangles around one vertex
constexpr int kChain = 64;        // visible hull edges from one outside point
constexpr int kFlipRounds = 1 << 16;
constexpr int kFlipPoll = 4;      // flip rounds between read-backs
constexpr int kInterimFlips = 2;  // flip rounds after each insertion round
constexpr int kFlipBlocks = 304;  // grid of the grid-stride flip kernels (2 per SM)
constexpr int kInsertRounds = 1 << 12;
constexpr int kInsertPoll = 4;    // insertion rounds between read-backs
constexpr int kSegQueue = 4096;   // crossing edges of one segment
constexpr int kSegStack = 256;    // pieces of one segment split by vertices inside it
constexpr int kCorr = 8;          // crossing edges of a segment recovered in the parallel rounds
constexpr int kClaim = 128;       // triangles one such segment claims
constexpr int kSegWindow = 1 << 15;  // segments per window of parallel rounds
constexpr int kSegRounds = 1 << 12;

enum CdtErr {
  kErrCoord = 1,       // a constraint point beyond the supported coordinate range
  kErrDuplicate = 2,   // a constraint point on a site or another constraint point
  kErrWalk = 4,        // a location, rotation or chain bound ran out
  kErrHash = 8,        // the edge table is inconsistent or full
  kErrSegment = 16,    // a vertex inside a segment, crossing segments, a bad index pair
  kErrSegLimit = 32,   // a segment's recovery ran out of its bounds
  kErrCapacity = 64    // more triangles than the mesh holds
};

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

#define CCK(call)                                   \
  do {                                              \
    if ((call) != cudaSuccess) return GCVT_ERR_CUDA; \
  } while (0)

// ---- coordinates ---------------------------------------------------------

__global__ void k_cdt_coords(const double *__restrict__ sxy, int F, const double *__restrict__ cxy,
                             int C, double scale, double left, double lower, int n, i64 *X,
                             i64 *Y, i64 *R, int *err) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= F + C) return;
  if (v < F) {
    const i64 x = (i64)sxy[2 * (size_t)v], y = (i64)sxy[2 * (size_t)v + 1];
    X[v] = x << 15;
    Y[v] = y << 15;
    R[v] = y * n + x;
    return;
  }
  const int j = v - F;
  const double u = (cxy[2 * j] - left) / scale * 32768.0,
               w = (cxy[2 * j + 1] - lower) / scale * 32768.0;
  const double lim = 536870912.0;  // 2^29
  if (!(fabs(u) < lim) || !(fabs(w) < lim)) {
    atomicOr(err, kErrCoord);
    X[v] = Y[v] = 0;
  } else {
    X[v] = llrint(u);
    Y[v] = llrint(w);
  }
  R[v] = (i64)n * n + j;
}

// ---- adjacency ------------------------------------------------------------

__device__ __forceinline__ unsigned long long ekey(int u, int w) {
  return ((unsigned long long)(unsigned)u << 32) | (unsigned)w;
}
__device__ __forceinline__ unsigned ehash(unsigned long long k, unsigned mask) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  return (unsigned)k & mask;
}

__global__ void k_edge_insert(const int *__restrict__ tri, int T, unsigned long long *hk, int *hv,
                              unsigned mask, int *err) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * T) return;
  const int t = e / 3, i = e % 3;
  const int u = tri[3 * t + cdt::nx3(i)], w = tri[3 * t + cdt::pv3(i)];
  const unsigned long long k = ekey(u, w);
  unsigned h = ehash(k, mask);
  for (unsigned s = 0; s <= mask; ++s, h = (h + 1) & mask) {
    const unsigned long long old = atomicCAS(hk + h, ~0ull, k);
    if (old == ~0ull) {
      hv[h] = cdt::pack_nb(t, i);
      return;
    }
    if (old == k) break;  // a directed edge twice
  }
  atomicOr(err, kErrHash);
}

__global__ void k_edge_link(const int *__restrict__ tri, int T, const unsigned long long *hk,
                            const int *hv, unsigned mask, int *nbr, int *vt, int *err) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * T) return;
  const int t = e / 3, i = e % 3;
  const int u = tri[3 * t + cdt::nx3(i)], w = tri[3 * t + cdt::pv3(i)];
  if (i == 0) vt[tri[3 * t]] = t;
  if (i == 1) vt[tri[3 * t + 1]] = t;
  if (i == 2) vt[tri[3 * t + 2]] = t;
  const unsigned long long k = ekey(w, u);
  unsigned h = ehash(k, mask);
  int nb = cdt::kNone;
  for (unsigned s = 0; s <= mask; ++s, h = (h + 1) & mask) {
    const unsigned long long cur = hk[h];
    if (cur == k) {
      nb = hv[h];
      break;
    }
    if (cur == ~0ull) break;
  }
  nbr[3 * t + i] = nb;
}

// ---- constraint point insertion --------------------------------------------

// Where a pending point lies, and (outside the hull) the hull edges it sees
// in counter-clockwise order with the hull triangles just before and after
// them -- recorded while nothing changes, so the insertion never walks a
// mesh that other points are changing.
// (The edges lie around the middle of edge[], packed like neighbours: those before
// the exit edge are found going backwards.  Only what is used is written: a copy of
// the whole record per point and round was a third of a one-block round.)
struct Loc {
  int kind, t, i;
  int cnt, before, after;
  int first;               // edge[first .. first + cnt)
  int edge[2 * kChain];
};

// Claims hold (rounds left, priority) (cdt_core.cuh prio): the smallest wins, and a
// round's claims are below every earlier round's, so the array is never cleared
// between rounds (a memset of half a megabyte three times a round before).
typedef unsigned long long Claim;
__device__ __forceinline__ Claim claim_of(unsigned round, unsigned id) {
  return ((Claim)(0xffffffffu - round) << 32) | cdt::prio(id);
}
__device__ __forceinline__ void claim(Claim *cl, int t, Claim pr) { atomicMin(cl + t, pr); }
__device__ __forceinline__ void claim_nbrs(const Mesh &m, Claim *cl, int t, Claim pr) {
  claim(cl, t, pr);
  for (int i = 0; i < 3; ++i) {
    const int nb = m.nbr[3 * t + i];
    if (nb >= 0) claim(cl, cdt::nb_tri(nb), pr);
  }
}

// Locate pending point q and claim what its insertion changes.
__device__ void ins_locate(const Mesh &m, const int *pend, int q, int *start, Loc *loc, Claim *cl,
                           unsigned round, int *done, int *err) {
  const int p = pend[q];
  const Claim pr = claim_of(round, (unsigned)p);
  done[q] = 0;
  Loc &L = loc[q];
  int lt, li;
  const int kind = cdt::locate(m, p, start[q], kWalk, &lt, &li);
  L.kind = kind;
  L.t = lt;
  L.i = li;
  L.cnt = 0;
  if (kind == cdt::kLocFail) {
    atomicOr(err, kErrWalk);
  } else if (kind == cdt::kLocVertex) {
    atomicOr(err, kErrDuplicate);
  } else if (kind == cdt::kLocIn) {
    claim_nbrs(m, cl, lt, pr);
  } else if (kind == cdt::kLocEdge) {
    claim_nbrs(m, cl, lt, pr);
    const int nb = m.nbr[3 * lt + li];
    if (nb >= 0) claim_nbrs(m, cl, cdt::nb_tri(nb), pr);
  } else {  // outside: the visible hull edges around the exit edge
    int ft = lt, fi = li, first = kChain, last = kChain, ok = 1, before = -1, after = -1;
    L.edge[first] = cdt::pack_nb(lt, li);
    for (;;) {
      int pt, pi;
      if (!cdt::hull_prev(m, ft, fi, kRotate, &pt, &pi)) {
        ok = 0;
        break;
      }
      if (cdt::orient(m, m.tri[3 * pt + cdt::nx3(pi)], m.tri[3 * pt + cdt::pv3(pi)], p) >= 0) {
        before = pt;
        break;
      }
      if (kChain - first + 1 >= kChain) {
        ok = 0;
        break;
      }
      ft = pt;
      fi = pi;
      L.edge[--first] = cdt::pack_nb(pt, pi);
    }
    for (ft = lt, fi = li; ok;) {
      int nt, ni;
      if (!cdt::hull_next(m, ft, fi, kRotate, &nt, &ni)) {
        ok = 0;
        break;
      }
      if (cdt::orient(m, m.tri[3 * nt + cdt::nx3(ni)], m.tri[3 * nt + cdt::pv3(ni)], p) >= 0) {
        after = nt;
        break;
      }
      if (last - first + 1 >= kChain) {
        ok = 0;
        break;
      }
      ft = nt;
      fi = ni;
      L.edge[++last] = cdt::pack_nb(nt, ni);
    }
    L.before = before;
    L.after = after;
    L.first = first;
    if (!ok) {
      atomicOr(err, kErrWalk);
      L.kind = cdt::kLocFail;
    } else {
      // claim the chain and the hull edges just before and after it, so that
      // two points never extend the hull next to each other in one round
      L.cnt = last - first + 1;
      for (int k = first; k <= last; ++k) claim(cl, cdt::nb_tri(L.edge[k]), pr);
      if (before >= 0) claim(cl, before, pr);
      if (after >= 0) claim(cl, after, pr);
    }
  }
}

__global__ void k_ins_locate(Mesh m, const int *__restrict__ pend, const int *npp, int *start,
                             Loc *loc, Claim *cl, unsigned round, int *done, int *err) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < *npp) ins_locate(m, pend, q, start, loc, cl, round, done, err);
}

__device__ __forceinline__ bool owns(const Mesh &m, const Claim *cl, int t, Claim pr) {
  return cl[t] == pr;
}
// (every claim is read whatever the others say: the loads are in flight together)
__device__ __forceinline__ bool owns_nbrs(const Mesh &m, const Claim *cl, int t, Claim pr) {
  bool ok = owns(m, cl, t, pr);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int nb = m.nbr[3 * t + i];
    ok &= owns(m, cl, nb >= 0 ? cdt::nb_tri(nb) : t, pr);
  }
  return ok;
}

// What to do with a triangle that changed: it and its neighbours are tested by
// the next flip round.  An edge whose opposite vertices changed belongs to a
// changed triangle, so it is tested from whichever of its triangles has the smaller
// index.  Act marks them in a byte each; ActList also lists each once (the four
// marks of a triangle and its neighbours are set before the first answer is needed).
struct Act {
  uint8_t *act;
  __device__ __forceinline__ void add(const int (&t)[4]) const {
#pragma unroll
    for (int k = 0; k < 4; ++k) act[t[k]] = 1;
  }
};
struct ActList {
  uint8_t *act;
  int *list, *count;
  __device__ __forceinline__ void add(const int (&t)[4]) const {
    unsigned was[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      was[k] = atomicOr(reinterpret_cast<unsigned *>(act) + (t[k] >> 2), 1u << (8 * (t[k] & 3)));
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (!((was[k] >> (8 * (t[k] & 3))) & 1u)) list[atomicAdd(count, 1)] = t[k];
  }
};
template <class A>
__device__ __forceinline__ void touch(const Mesh &m, const A &act, int t) {
  int id[4] = {t, t, t, t};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int nb = m.nbr[3 * t + i];
    if (nb >= 0) id[i + 1] = cdt::nb_tri(nb);
  }
  act.add(id);
}

// Insert pending point q if it won every claim; otherwise it stays pending (its
// walk starts next round from the triangle it reached).
template <class A>
__device__ void ins_apply(const Mesh &m, const int *pend, int q, int *start, const Loc *loc,
                          const Claim *cl, unsigned round, int *ntri, int cap, int *done,
                          const A &act, int *err) {
  const int p = pend[q];
  const Claim pr = claim_of(round, (unsigned)p);
  const Loc &L = loc[q];
  if (L.kind == cdt::kLocFail || L.kind == cdt::kLocVertex) return;
  start[q] = L.t;
  if (L.kind == cdt::kLocIn) {
    if (!owns_nbrs(m, cl, L.t, pr)) return;
    const int s = atomicAdd(ntri, 2);
    if (s + 2 > cap) {
      atomicOr(err, kErrCapacity);
      return;
    }
    cdt::split_in(m, L.t, p, s, s + 1);
    touch(m, act, L.t);
    touch(m, act, s);
    touch(m, act, s + 1);
  } else if (L.kind == cdt::kLocEdge) {
    if (!owns_nbrs(m, cl, L.t, pr)) return;
    const int nb = m.nbr[3 * L.t + L.i];
    if (nb >= 0 && !owns_nbrs(m, cl, cdt::nb_tri(nb), pr)) return;
    const int k = nb >= 0 ? 2 : 1;
    const int s = atomicAdd(ntri, k);
    if (s + k > cap) {
      atomicOr(err, kErrCapacity);
      return;
    }
    cdt::split_edge(m, L.t, L.i, p, s, s + 1);
    touch(m, act, L.t);
    touch(m, act, s);
    if (nb >= 0) {
      touch(m, act, cdt::nb_tri(nb));
      touch(m, act, s + 1);
    }
  } else {
    bool won = (L.before < 0 || owns(m, cl, L.before, pr)) && (L.after < 0 || owns(m, cl, L.after, pr));
    for (int k = 0; k < L.cnt && won; ++k) won = owns(m, cl, cdt::nb_tri(L.edge[L.first + k]), pr);
    if (!won) return;
    const int s = atomicAdd(ntri, L.cnt);
    if (s + L.cnt > cap) {
      atomicOr(err, kErrCapacity);
      return;
    }
    cdt::insert_fan(
        m, [&](int k) { return L.edge[L.first + k]; }, L.cnt, p, [=](int k) { return s + k; });
    for (int k = 0; k < L.cnt; ++k) touch(m, act, s + k);
    start[q] = s;
  }
  done[q] = 1;
}

__global__ void k_ins_apply(Mesh m, const int *__restrict__ pend, const int *npp, int *start,
                            const Loc *__restrict__ loc, const Claim *cl, unsigned round,
                            int *ntri, int cap, int *done, uint8_t *act, int *err) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < *npp)
    ins_apply(m, pend, q, start, loc, cl, round, ntri, cap, done, Act{act}, err);
}

// ---- flips ---------------------------------------------------------------

// The edge that triangle t flips this round (first_flip); the flip claims both triangles
// and the four outer neighbours with the priority of 3 t + i.
__device__ __forceinline__ int flip_mark_one(const Mesh &m, int t, Claim *cl, unsigned round) {
  const int c = cdt::first_flip(m, t);
  if (!c) return 0;
  const int i = c - 1;
  const Claim pr = claim_of(round, (unsigned)(3 * t + i));
  int id[8];
  cdt::flip_claims(m, t, i, id);
#pragma unroll
  for (int k = 0; k < 8; ++k) claim(cl, id[k], pr);
  return c;
}

// Triangle t's marked flip, if it won all its claims.
template <class A>
__device__ __forceinline__ bool flip_apply_one(const Mesh &m, int t, int c, const Claim *cl,
                                               unsigned round, const A &act) {
  const int i = c - 1;
  const Claim pr = claim_of(round, (unsigned)(3 * t + i));
  int id[8];
  cdt::flip_claims(m, t, i, id);
  bool own = true;  // (no early exit: the loads are in flight together)
#pragma unroll
  for (int k = 0; k < 8; ++k) own &= owns(m, cl, id[k], pr);
  if (!own) return false;
  cdt::flip(m, t, i);
  touch(m, act, t);
  touch(m, act, id[4]);
  return true;
}

// Each changed triangle (act) of the *ntri in the mesh; one with nothing to flip is
// settled until a change touches it again.  (grid-stride: a round with few changed
// triangles costs few blocks)
__global__ void k_flip_mark(Mesh m, const int *ntri, int *cand, Claim *cl, unsigned round,
                            uint8_t *act, int *found) {
  const int T = *ntri;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
    const int c = act[t] ? flip_mark_one(m, t, cl, round) : 0;
    cand[t] = c;
    if (c) atomicAdd(found, 1);
    else act[t] = 0;
  }
}

__global__ void k_flip_apply(Mesh m, const int *ntri, const int *cand, const Claim *cl,
                             unsigned round, uint8_t *act, int *flips) {
  const int T = *ntri;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x)
    if (cand[t] && flip_apply_one(m, t, cand[t], cl, round, Act{act})) atomicAdd(flips, 1);
}

// Every insertion round with its flip rounds in one block: the rounds are chains of short
// dependent steps (832 boundary points take 28 rounds; as seven launches each 74 us a
// round, 55 in one block of 1024 threads, 85 in one of 256; 36 with short predicates and
// the loads and marks of a triangle's neighbours in flight together), and the changed
// triangles are listed instead of searched for.  Block barriers order the steps.  After the
// last point the flips run until none is left.
//   Up to kOneBlock points it does them all.  Above, points inside the sites go in
// fastest over the grid, nearly all in the first rounds, while of a chain of boundary
// points few win a round and each round's latency counts.  So up to kOneChain the first
// kInsertPoll rounds run over the grid, and the block goes on if they left more than half.  A
// call on 1024 x 1024 / 4369 sites took, block / grid / this: 2000 inside 1.43 / 1.11 /
// 1.43 ms, 3000 inside 1.82 / 1.24 / 1.25, 2000 in a ring outside 3.35 / 4.26 / 3.35, 3000
// 4.76 / 5.19 / 4.57, 4000 5.81 / 5.42 / 5.47.
constexpr int kOneBlock = 2048, kOneChain = 4096;
constexpr int kOneSegs = 4096;  // segments whose rounds one block does
constexpr int kOneThreads = 1024;

__global__ void __launch_bounds__(kOneThreads) k_insert_all(Mesh m, int *pend, int *start,
                                                            int *pend2, int *start2, int np,
                                                            Loc *loc, Claim *cl, unsigned round,
                                                            int rounds, int *ntri, int cap,
                                                            int *done, uint8_t *act, int *list,
                                                            int *list2, int *cand, int *left,
                                                            bool marked, int *err) {
  __shared__ int s_np, s_n, s_n2, s_stop;
  const int tid = threadIdx.x;
  if (tid == 0) s_n = s_stop = 0;
  __syncthreads();
  // the triangles that rounds over the grid left marked
  for (int w = tid, T = marked ? *ntri : 0; 4 * w < T; w += kOneThreads)
    for (unsigned q = reinterpret_cast<const unsigned *>(act)[w] & 0x01010101u; q; q &= q - 1u) {
      const int t = 4 * w + (__ffs((int)q) - 1) / 8;
      if (t < T) list[atomicAdd(&s_n, 1)] = t;
    }
  __syncthreads();
  for (int r = 0; r < rounds && np > 0; ++r) {
    ++round;
    if (tid == 0) s_np = 0;
    for (int q = tid; q < np; q += kOneThreads) ins_locate(m, pend, q, start, loc, cl, round, done, err);
    __syncthreads();
    for (int q = tid; q < np; q += kOneThreads)
      ins_apply(m, pend, q, start, loc, cl, round, ntri, cap, done, ActList{act, list, &s_n}, err);
    __syncthreads();
    for (int q = tid; q < np; q += kOneThreads)
      if (!done[q]) {
        const int p = atomicAdd(&s_np, 1);
        pend2[p] = pend[q];
        start2[p] = start[q];
      }
    // the last points in: flips until none is left
    __syncthreads();
    const int nflips = s_np ? kInterimFlips : kFlipRounds;
    for (int f = 0; f < nflips; ++f) {
      ++round;
      if (tid == 0) s_n2 = 0;
      __syncthreads();
      const int n = s_n;
      if (n == 0) break;
      for (int k = tid; k < n; k += kOneThreads) {
        const int t = list[k], c = flip_mark_one(m, t, cl, round);
        cand[k] = c;
        if (!c)  // settled
          atomicAnd(reinterpret_cast<unsigned *>(act) + (t >> 2), ~(1u << (8 * (t & 3))));
      }
      __syncthreads();
      const ActList next{act, list2, &s_n2};
      for (int k = tid; k < n; k += kOneThreads) {
        if (!cand[k]) continue;
        const int t = list[k];
        list2[atomicAdd(&s_n2, 1)] = t;  // (still marked)
        flip_apply_one(m, t, cand[k], cl, round, next);
      }
      __syncthreads();
      if (tid == 0) s_n = s_n2;
      int *u = list;
      list = list2;
      list2 = u;
    }
    if (tid == 0) s_stop = *reinterpret_cast<volatile int *>(err);
    __syncthreads();
    np = s_np;
    int *u = pend;
    pend = pend2;
    pend2 = u;
    u = start;
    start = start2;
    start2 = u;
    if (s_stop) break;
    __syncthreads();
  }
  if (tid == 0) *left = np;
}

// ---- segments --------------------------------------------------------------

enum SegState { kSegPending = 0, kSegDone = 1, kSegSerial = 2 };

// Segments that are already edges are marked at once (atomic bit sets, the
// mesh is otherwise read-only here); the others wait for the rounds.  Bad
// index pairs set err.
__global__ void k_seg_mark(Mesh m, const int *__restrict__ segs, int S, int V, int *state,
                           int *err) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= S) return;
  const int a = segs[2 * k], b = segs[2 * k + 1];
  if (a < 0 || b < 0 || a >= V || b >= V || a == b) {
    atomicOr(err, kErrSegment);
    state[k] = kSegDone;
    return;
  }
  state[k] = cdt::mark_constraint(m, a, b, kRotate) ? kSegDone : kSegPending;
}

// A pending segment of the window [base, base + W) claims, with its priority,
// the triangles around its ends and around every end of the edges crossing
// it: all that its recovery reads or writes (Sloan's flips stay inside the
// triangles the segment crosses, whose vertices are those ends, and rewrite
// the back links of their neighbours, which lie around the same vertices).
// The claimed triangles are listed for the apply pass.  A segment that meets
// a vertex or a constraint, or crosses more than kCorr edges, goes to the
// one-thread pass.
__device__ void seg_locate(const Mesh &m, const int *segs, int base, int w, int *state, int *list,
                           int *lcnt, Claim *cl, unsigned round) {
  const int k = base + w;
  if (state[k] != kSegPending) return;
  const int a = segs[2 * k], b = segs[2 * k + 1];
  int q[2 * kCorr], on = -1, cnt = 0;
  if (cdt::collect_crossings(m, a, b, q, kCorr, kWalk, &on, &cnt) != cdt::kSegOk) {
    state[k] = kSegSerial;
    return;
  }
  int *L = list + (size_t)w * kClaim;
  int n = 0;
  for (int e = -2; e < 2 * cnt; ++e) {
    const int v = e == -2 ? a : (e == -1 ? b : q[e]);
    bool seen = false;
    for (int f = -2; f < e && !seen; ++f) seen = (f == -2 ? a : (f == -1 ? b : q[f])) == v;
    if (seen) continue;
    const int c = cdt::fan(m, v, kRotate, L + n, kClaim - n);
    if (c < 0) {
      state[k] = kSegSerial;
      return;
    }
    n += c;
  }
  const Claim pr = claim_of(round, (unsigned)k);
  for (int i = 0; i < n; ++i) claim(cl, L[i], pr);
  lcnt[w] = n;
}
__global__ void k_seg_locate(Mesh m, const int *__restrict__ segs, int base, int W, int *state,
                             int *list, int *lcnt, Claim *cl, unsigned round) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < W) seg_locate(m, segs, base, w, state, list, lcnt, cl, round);
}

// The segments that won every claim are recovered (cdt_core.cuh
// recover_segment); the others count themselves pending for the next round.
__device__ void seg_apply(const Mesh &m, const int *segs, int base, int w, int *state,
                          const int *list, const int *lcnt, const Claim *cl, unsigned round,
                          int *pending, int *err) {
  const int k = base + w;
  if (state[k] != kSegPending) return;
  const int *L = list + (size_t)w * kClaim;
  const Claim pr = claim_of(round, (unsigned)k);
  bool own = true;  // (no early exit: the loads are in flight together)
#pragma unroll 8
  for (int i = 0, n = lcnt[w]; i < n; ++i) own &= cl[L[i]] == pr;
  if (!own) {
    atomicAdd(pending, 1);
    return;
  }
  int q[2 * kCorr], on = -1;
  const int r = cdt::recover_segment(m, segs[2 * k], segs[2 * k + 1], q, kCorr, kWalk, &on);
  if (r == cdt::kSegCrosses) atomicOr(err, kErrSegment);
  else if (r != cdt::kSegOk) atomicOr(err, kErrSegLimit);
  state[k] = kSegDone;
}
__global__ void k_seg_apply(Mesh m, const int *__restrict__ segs, int base, int W, int *state,
                            const int *__restrict__ list, const int *__restrict__ lcnt,
                            const Claim *cl, unsigned round, int *pending, int *err) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < W) seg_apply(m, segs, base, w, state, list, lcnt, cl, round, pending, err);
}

// Every segment round in one block, for up to kOneSegs segments (7 rounds of two
// launches and a read-back: 0.42 ms for 832, 0.19 this way).
__global__ void __launch_bounds__(kOneThreads) k_seg_all(Mesh m, const int *__restrict__ segs,
                                                         int S, int *state, int *list, int *lcnt,
                                                         Claim *cl, unsigned round, int rounds,
                                                         int *err) {
  __shared__ int s_pending;
  for (int r = 0; r < rounds; ++r) {
    ++round;
    if (threadIdx.x == 0) s_pending = 0;
    for (int w = threadIdx.x; w < S; w += kOneThreads)
      seg_locate(m, segs, 0, w, state, list, lcnt, cl, round);
    __syncthreads();
    for (int w = threadIdx.x; w < S; w += kOneThreads)
      seg_apply(m, segs, 0, w, state, list, lcnt, cl, round, &s_pending, err);
    __syncthreads();
    if (s_pending == 0) break;
    __syncthreads();
  }
}

// The segments left to one thread, one after the other (they may share
// crossing edges): long ones, and those with vertices inside them, which
// become the chain of edges between those vertices (as constrained Delaunay
// triangulations split such segments).  Crossing segments set err.
constexpr int kSegThreads = 1024;
__global__ void __launch_bounds__(kSegThreads) k_segments(Mesh m, const int *__restrict__ segs,
                                                          int S, const int *state, int *queue,
                                                          int *stack, int *err) {
  // (usually few or none: the block finds them; one thread walking the list took 50 us
  // more of 832 segments)
  __shared__ unsigned s_left[32];
  for (int base = 0; base < S; base += blockDim.x) {
    const int j = base + threadIdx.x;
    const unsigned left = __ballot_sync(0xffffffffu, j < S && state[j] != kSegDone);
    if ((threadIdx.x & 31) == 0) s_left[threadIdx.x >> 5] = left;
    if (!__syncthreads_or(left != 0)) continue;
    if (threadIdx.x == 0)
      for (int g = 0; g < (int)blockDim.x / 32; ++g)
        for (unsigned q = s_left[g]; q; q &= q - 1u) {
          const int k = base + 32 * g + __ffs((int)q) - 1;
          const int a = segs[2 * k], b = segs[2 * k + 1];
          const int r = cdt::recover_chain(m, a, b, queue, kSegQueue, stack, kSegStack, kWalk);
          if (r == cdt::kSegCrosses) atomicOr(err, kErrSegment);
          else if (r != cdt::kSegOk) atomicOr(err, kErrSegLimit);
        }
    __syncthreads();
  }
}

// ---- output ----------------------------------------------------------------

__global__ void k_emit_count(Mesh m, int T, int *cnt) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  int a, b, c;
  cdt::canon(m.tri + 3 * t, a, b, c);
  atomicAdd(cnt + a, 1);
}

// Triangle t at its owner's offset plus its rank among the owner's
// triangles (cdt_core.cuh owner_rank).
__global__ void k_emit(Mesh m, int T, const int *__restrict__ off, int *out, int cap, int *err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  int a, b, c;
  cdt::canon(m.tri + 3 * t, a, b, c);
  const int rank = cdt::owner_rank(m, t, kRotate);
  if (rank < 0) {
    atomicOr(err, kErrWalk);
    return;
  }
  const int pos = off[a] + rank;
  if (pos < cap) {
    out[3 * (size_t)pos] = a;
    out[3 * (size_t)pos + 1] = b;
    out[3 * (size_t)pos + 2] = c;
  }
}

// Start triangles of the constraint points: a site near each (the first found
// in growing squares around its pixel in the site index grid), or any triangle.
// A warp per point, its lanes side by side along a square (a thread per point
// took 70 us for 832 points).
__global__ void k_ins_start(const i64 *__restrict__ X, const i64 *__restrict__ Y, int F, int C,
                            const int *__restrict__ site_at, int n, const int *vt, int *start) {
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (j >= C) return;  // the whole warp
  const int px = (int)(X[F + j] >> 15), py = (int)(Y[F + j] >> 15);
  int found = -1;
  for (int r = 0; r < 64 && found < 0; ++r) {
    // the ring at Chebyshev distance r: its 8 r cells (1 for r = 0)
    const int cells = r ? 8 * r : 1;
    for (int k0 = 0; k0 < cells && found < 0; k0 += 32) {
      const int k = k0 + lane;
      int dx, dy;
      if (r == 0) dx = dy = 0;
      else if (k < 2 * r) dx = -r + k, dy = -r;          // top, left to right
      else if (k < 4 * r) dx = r, dy = -r + (k - 2 * r);  // right, top to bottom
      else if (k < 6 * r) dx = r - (k - 4 * r), dy = r;   // bottom, right to left
      else dx = -r, dy = r - (k - 6 * r);                 // left, bottom to top
      const int x = px + dx, y = py + dy;
      const int v = k < cells && x >= 0 && y >= 0 && x < n && y < n
                        ? site_at[(size_t)y * n + x] : -1;
      const unsigned hit = __ballot_sync(0xffffffffu, v >= 0);
      if (hit) found = __shfl_sync(0xffffffffu, v, __ffs(hit) - 1);
    }
  }
  if (lane == 0) start[j] = found >= 0 ? vt[found] : 0;
}

__global__ void k_site_at(const i64 *__restrict__ X, const i64 *__restrict__ Y, int F, int n,
                          int *site_at) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= F) return;
  site_at[(size_t)(Y[v] >> 15) * n + (X[v] >> 15)] = v;
}

__global__ void k_iota(int *a, int count, int base) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) a[i] = base + i;
}

// Drop the inserted points from the pending list (order kept).
__global__ void k_compact(const int *__restrict__ pend, const int *__restrict__ start,
                          const int *__restrict__ done, const int *npp, int *pend2, int *start2,
                          int *count) {
  if (blockIdx.x != 0) return;
  const int np = *npp;
  // one block: a running offset over chunks of blockDim.x
  __shared__ int base;
  __shared__ int wsum[32];
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  for (int c0 = 0; c0 < np; c0 += blockDim.x) {
    const int q = c0 + threadIdx.x;
    const int keep = q < np && !done[q];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) wsum[wid] = __popc(bal);
    __syncthreads();
    int pre = 0, tot = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      if (w < wid) pre += wsum[w];
      tot += wsum[w];
    }
    if (keep) {
      const int pos = base + pre + __popc(bal & ((1u << lane) - 1u));
      pend2[pos] = pend[q];
      start2[pos] = start[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) base += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = base;
}

}  // namespace

// The constrained Delaunay triangulation of the free sites of `bits` (point
// indices in gcvt_ctx_extract_points' order) and C constraint points
// (device, 2 C doubles; indices F .. F + C - 1) with S segments (device
// index pairs).  Writes up to cap triangles (3 ints) to out (device) and the
// count to *ntris.
int cdt_compute(const uint64_t *bits, const uint64_t *fixed, int n, unsigned *colcnt,
                const double *cxy, int C, const int *segs, int S, double scale, double left,
                double lower, int *out, unsigned cap, unsigned *ntris, int *detail,
                cudaStream_t s) {
  *ntris = 0;
  if (detail) *detail = 0;
  if (n <= 0 || C < 0 || S < 0 || !(scale > 0)) return GCVT_ERR_ARGUMENT;
  Scratch sc(s);
  // 1. the sites and their Delaunay triangulation
  unsigned F = 0;
  CCK(launch_extract(bits, fixed, n, colcnt, 1.0, 0.0, 0.0, nullptr, 0, colcnt + n, s));
  CCK(cudaMemcpyAsync(&F, colcnt + n, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  CCK(cudaStreamSynchronize(s));
  const long long V = (long long)F + C;
  if (V < 3) return GCVT_OK;
  if (V > (1ll << 28)) return GCVT_ERR_SIZE;
  const int cap_t = (int)(2 * V + 16);
  double *sxy = sc.take<double>(2 * (size_t)F + 2);
  i64 *X = sc.take<i64>((size_t)V), *Y = sc.take<i64>((size_t)V), *R = sc.take<i64>((size_t)V);
  int *tri = sc.take<int>(3 * (size_t)cap_t), *nbr = sc.take<int>(3 * (size_t)cap_t);
  unsigned *cons = sc.take<unsigned>((size_t)cap_t);
  int *vt = sc.take<int>((size_t)V);
  Claim *cl = sc.take<Claim>((size_t)cap_t);
  unsigned round = 0;  // of claims
  int *cand = sc.take<int>((size_t)cap_t);
  uint8_t *act = sc.take<uint8_t>((size_t)cap_t);
  // [0] error bits, [1] triangles, [2] flips wanted, [3] flips made, [4] and
  // [6] points pending (the two lists), [5] segments pending
  int *ctr = sc.take<int>(8);
  if (!sxy || !X || !Y || !R || !tri || !nbr || !cons || !vt || !cl || !cand || !act || !ctr)
    return GCVT_ERR_ALLOC;
  CCK(launch_extract(bits, fixed, n, colcnt, 1.0, 0.0, 0.0, sxy, F, colcnt + n, s));
  CCK(cudaMemsetAsync(ctr, 0, 8 * sizeof(int), s));
  CCK(cudaMemsetAsync(cons, 0, (size_t)cap_t * sizeof(unsigned), s));
  CCK(cudaMemsetAsync(cl, 0xff, (size_t)cap_t * sizeof(Claim), s));
  k_cdt_coords<<<nblk(V, 256), 256, 0, s>>>(sxy, (int)F, cxy, C, scale, left, lower, n, X, Y, R,
                                            ctr);
  CCK(cudaGetLastError());
  unsigned T0 = 0;
  int rc = delaunay_sites_in(bits, fixed, n, tri, (unsigned)cap_t, &T0, s, sc);
  if (rc) return rc;
  if (T0 == 0 && C > 0) return GCVT_ERR_INPUT;  // constraint points need triangulated sites
  Mesh m{tri, nbr, cons, vt, X, Y, R};
  // 2. adjacency
  {
    unsigned hsize = 1;
    while (hsize < 6u * T0 + 64u) hsize <<= 1;
    unsigned long long *hk = sc.take<unsigned long long>(hsize);
    int *hv = sc.take<int>(hsize);
    if (!hk || !hv) return GCVT_ERR_ALLOC;
    CCK(cudaMemsetAsync(hk, 0xff, (size_t)hsize * sizeof(unsigned long long), s));
    CCK(cudaMemsetAsync(vt, 0, (size_t)V * sizeof(int), s));  // a vertex in no triangle: 0
    CCK(cudaMemsetAsync(act, 0, (size_t)cap_t, s));           // the sites' triangulation is Delaunay
    k_edge_insert<<<nblk(3ll * T0, 256), 256, 0, s>>>(tri, (int)T0, hk, hv, hsize - 1, ctr);
    k_edge_link<<<nblk(3ll * T0, 256), 256, 0, s>>>(tri, (int)T0, hk, hv, hsize - 1, nbr, vt,
                                                    ctr);
    CCK(cudaGetLastError());
  }
  int T = (int)T0;
  CCK(cudaMemcpyAsync(ctr + 1, &T, sizeof(int), cudaMemcpyHostToDevice, s));
  int h[8] = {};
  auto pull = [&]() -> int {
    CCK(cudaMemcpyAsync(h, ctr, 8 * sizeof(int), cudaMemcpyDeviceToHost, s));
    CCK(cudaStreamSynchronize(s));
    return GCVT_OK;
  };
  // Delaunay flip rounds over the changed triangles (their count read on the
  // device: insertions of the same batch add triangles)
  const int fgrid = nblk(cap_t, 256) < kFlipBlocks ? nblk(cap_t, 256) : kFlipBlocks;
  auto flip_rounds = [&](int rounds) -> int {
    for (int i = 0; i < rounds; ++i) {
      ++round;
      k_flip_mark<<<fgrid, 256, 0, s>>>(m, ctr + 1, cand, cl, round, act, ctr + 2);
      k_flip_apply<<<fgrid, 256, 0, s>>>(m, ctr + 1, cand, cl, round, act, ctr + 3);
    }
    CCK(cudaGetLastError());
    return GCVT_OK;
  };
  // flip rounds over every triangle until none is left, read back every
  // kFlipPoll rounds (a round that finds nothing to flip changes nothing)
  auto flips = [&]() -> int {
    CCK(cudaMemsetAsync(act, 1, (size_t)cap_t, s));
    for (int r = 0; r < kFlipRounds; r += kFlipPoll) {
      if ((rc = flip_rounds(kFlipPoll - 1))) return rc;
      CCK(cudaMemsetAsync(ctr + 2, 0, 2 * sizeof(int), s));  // the last round's counts
      if ((rc = flip_rounds(1)) || (rc = pull())) return rc;
      if (h[0] || h[2] == 0) return GCVT_OK;
    }
    h[0] |= kErrWalk;
    return GCVT_OK;
  };
  // 3. constraint points
  if (C > 0) {
    int *site_at = sc.take<int>((size_t)n * n);
    int *pend = sc.take<int>(C), *pend2 = sc.take<int>(C);
    int *start = sc.take<int>(C), *start2 = sc.take<int>(C), *done = sc.take<int>(C);
    Loc *loc = sc.take<Loc>(C);
    if (!site_at || !pend || !pend2 || !start || !start2 || !done || !loc) return GCVT_ERR_ALLOC;
    CCK(cudaMemsetAsync(site_at, 0xff, (size_t)n * n * sizeof(int), s));
    k_site_at<<<nblk(F, 256), 256, 0, s>>>(X, Y, (int)F, n, site_at);
    k_ins_start<<<nblk(32ll * C, 128), 128, 0, s>>>(X, Y, (int)F, C, site_at, n, vt, start);
    k_iota<<<nblk(C, 256), 256, 0, s>>>(pend, C, (int)F);  // point indices F + j
    CCK(cudaGetLastError());
    // one round: the points of list a (count *na) locate, claim and insert;
    // those left go to list b (count *nb); then kInterimFlips flip rounds.  Every
    // count is read on the device, so rounds queue without the host.
    auto ins_round = [&](int *pa, int *sa, int *pb, int *sb, int *na, int *nb) -> int {
      ++round;
      k_ins_locate<<<nblk(C, 32), 32, 0, s>>>(m, pa, na, sa, loc, cl, round, done, ctr);
      k_ins_apply<<<nblk(C, 32), 32, 0, s>>>(m, pa, na, sa, loc, cl, round, ctr + 1, cap_t, done,
                                               act, ctr);
      k_compact<<<1, 1024, 0, s>>>(pa, sa, done, na, pb, sb, nb);
      CCK(cudaGetLastError());
      return flip_rounds(kInterimFlips);
    };
    int np = C;
    bool block = C <= kOneBlock;
    if (!block) CCK(cudaMemcpyAsync(ctr + 4, &C, sizeof(int), cudaMemcpyHostToDevice, s));
    // kInsertPoll rounds (lists 1 -> 2 -> 1 ...) per read-back
    for (int r = 0; !block && r < kInsertRounds && np > 0; r += kInsertPoll) {
      for (int k = 0; k < kInsertPoll && rc == GCVT_OK; k += 2) {
        rc = ins_round(pend, start, pend2, start2, ctr + 4, ctr + 6);
        if (rc == GCVT_OK) rc = ins_round(pend2, start2, pend, start, ctr + 6, ctr + 4);
      }
      if (rc == GCVT_OK) rc = pull();
      if (rc != GCVT_OK) return rc;
      if (h[0]) break;
      np = h[4];
      block = r == 0 && C <= kOneChain && 2 * np > C;
    }
    if (block) {
      int *la = sc.take<int>((size_t)cap_t), *lb = sc.take<int>((size_t)cap_t);
      if (!la || !lb) return GCVT_ERR_ALLOC;
      k_insert_all<<<1, kOneThreads, 0, s>>>(m, pend, start, pend2, start2, np, loc, cl, round,
                                             kInsertRounds, ctr + 1, cap_t, done, act, la, lb, cand,
                                             ctr + 4, C > kOneBlock, ctr);
      CCK(cudaGetLastError());
      round += (1 + kInterimFlips) * kInsertRounds + kFlipRounds;
      if ((rc = pull())) return rc;
      np = h[0] ? 0 : h[4];
    }
    if (rc != GCVT_OK) return rc;
    if (!h[0] && np > 0) h[0] |= kErrWalk;
  }
  if ((rc = pull())) return rc;
  T = h[1];
  // 4. segments: those already edges marked at once, the others recovered
  // in parallel rounds of claims (window by window), what is left by one
  // thread; 5. flips that keep them
  if (!h[0] && S > 0) {
    const int Wmax = S < kSegWindow ? S : kSegWindow;
    int *state = sc.take<int>((size_t)S), *lcnt = sc.take<int>((size_t)Wmax);
    int *list = sc.take<int>((size_t)Wmax * kClaim);
    int *queue = sc.take<int>(2 * (size_t)kSegQueue), *stack = sc.take<int>(2 * (size_t)kSegStack);
    if (!state || !lcnt || !list || !queue || !stack) return GCVT_ERR_ALLOC;
    k_seg_mark<<<nblk(S, 256), 256, 0, s>>>(m, segs, S, (int)V, state, ctr);
    CCK(cudaGetLastError());
    if (S <= kOneSegs) {
      k_seg_all<<<1, kOneThreads, 0, s>>>(m, segs, S, state, list, lcnt, cl, round, kSegRounds,
                                          ctr);
      CCK(cudaGetLastError());
      round += kSegRounds;
    }
    for (int base = 0; S > kOneSegs && base < S; base += kSegWindow) {
      const int W = S - base < kSegWindow ? S - base : kSegWindow;
      for (int r = 0; r < kSegRounds; ++r) {
        ++round;
        CCK(cudaMemsetAsync(ctr + 5, 0, sizeof(int), s));
        k_seg_locate<<<nblk(W, 32), 32, 0, s>>>(m, segs, base, W, state, list, lcnt, cl, round);
        k_seg_apply<<<nblk(W, 32), 32, 0, s>>>(m, segs, base, W, state, list, lcnt, cl, round,
                                               ctr + 5, ctr);
        CCK(cudaGetLastError());
        if ((rc = pull())) return rc;
        if (h[5] == 0) break;
      }
    }
    k_segments<<<1, kSegThreads, 0, s>>>(m, segs, S, state, queue, stack, ctr);
    CCK(cudaGetLastError());
    if ((rc = pull())) return rc;
  }
  if (!h[0] && (rc = flips())) return rc;
  if (h[0]) {
    if (detail) *detail = h[0];
    return (h[0] & (kErrCoord | kErrDuplicate | kErrSegment)) ? GCVT_ERR_INPUT : GCVT_ERR_CUDA;
  }
  // 6. output in a fixed order
  int *cnt = sc.take<int>((size_t)V + 1), *off = sc.take<int>((size_t)V + 1);
  if (!cnt || !off) return GCVT_ERR_ALLOC;
  CCK(cudaMemsetAsync(cnt, 0, ((size_t)V + 1) * sizeof(int), s));
  k_emit_count<<<nblk(T, 256), 256, 0, s>>>(m, T, cnt);
  CCK(cudaGetLastError());
  if ((rc = scan_counts(cnt, (int)V, off, nullptr, sc, s))) return rc;
  if (out && cap) {
    k_emit<<<nblk(T, 256), 256, 0, s>>>(m, T, off, out, (int)cap, ctr);
    CCK(cudaGetLastError());
  }
  if ((rc = pull())) return rc;
  if (h[0]) {
    if (detail) *detail = h[0];
    return GCVT_ERR_CUDA;
  }
  *ntris = (unsigned)T;
  return GCVT_OK;
}

}  // namespace cvtgb
