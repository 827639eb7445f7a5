// delaunay.cu -- the Delaunay triangulation of a context's free sites on the
// GPU, in the point order of delaunayInput (delaunay.h:46-57), so that its
// triangles index gcvt_ctx_extract_points' list and feed gcvt_lift.  This is
// the Delaunay part of the reference's CDT stage (gDel2D,
// gDel2D/GPU/GpuDelaunay.cu:46) for the CVT sites; constraint points and
// segments are not inserted.
//
// Sites lie on the integer pixel lattice, so every predicate is exact in
// 64-bit / 128-bit integers.  Co-circular sites (common on a lattice) are
// resolved by symbolic perturbation of the lifting map (simulation of
// simplicity): z(q) = |q|^2 + delta(q), with delta(q) > 0 infinitesimal and
// infinitely larger for a larger rank h(q) = y n + x.  The perturbed lifted
// points are in general position, so their lower hull is one Delaunay
// triangulation of the sites, and every site that evaluates a predicate
// gets the same sign, so all stars agree.
//
// Each site's Delaunay star (its neighbours in angular order) is wrapped from
// the sites in a window around it (quad_stars: four sites of a warp in step,
// eight lanes each; wwrap: a site by the whole warp, where the first does not
// settle it).  What does not fit is inserted one by one into the star, a sorted
// cyclic list in the warp's registers: inverted about the site, the star is the
// part of the candidates' convex hull facing away from the site (a candidate
// inside the current hull never becomes a neighbour later; an inserted one
// removes the neighbours it covers).  What bounds the star kernel is issue
// slots, and at the end the few sites on the hull whose flat triangles take
// many searches, one after the other in their warp.  4096^2, 262,144 CVT sites: 1.43 ms with one warp per site
// inserting every candidate (3,913 instructions a site), 0.29 ms now.
// Certificate, exact: a triangle of the star is final when no site
// outside the window lies in its circumcircle, an open angular gap (>= pi)
// when no site lies strictly inside its cone (then the site is on the
// sites' convex hull); both are searched through a pyramid of tile
// occupancy, and a site found is inserted and the star checked again.  After
// the second window only a star of fewer than two neighbours, or on one line,
// widens it (a window covering the grid is exact).  Warps take the sites in tile order; a triangle is
// written by its vertex that comes first in delaunayInput's order (x, then
// y), counter-clockwise, so the output does not depend on the scheduling.
#include "gcvt_internal.cuh"
#include "../../include/gcvt_gb300.h"

#include <climits>

namespace cvtgb {

namespace {

constexpr int kStar = 64;  // Delaunay neighbours a site can hold

// (dx, dy) packed in one int: dx in the low 16 bits, dy in the high 16
__device__ __forceinline__ int pk(int dx, int dy) {
  return (int)((unsigned)(dx & 0xffff) | ((unsigned)dy << 16));
}
__device__ __forceinline__ int pdx(int v) { return (int)(int16_t)(v & 0xffff); }
__device__ __forceinline__ int pdy(int v) { return v >> 16; }

__device__ __forceinline__ long long cross(int ax, int ay, int bx, int by) {
  return (long long)ax * by - (long long)ay * bx;
}

// angular order around the site: half 0 = [0, pi), half 1 = [pi, 2 pi)
__device__ __forceinline__ int half_of(int x, int y) {
  return (y > 0 || (y == 0 && x > 0)) ? 0 : 1;
}

// the CCW angle from a to b is >= pi (b not strictly left of a, and not the
// same ray)
__device__ __forceinline__ bool open_gap(int ax, int ay, int bx, int by) {
  const long long c = cross(ax, ay, bx, by);
  if (c > 0) return false;
  if (c < 0) return true;
  return (long long)ax * bx + (long long)ay * by < 0;  // opposite rays: exactly pi
}

// Perturbed incircle: is d strictly inside the circle through the site
// (origin), a and b (counter-clockwise)?  Coordinates relative to the site;
// hp, ha, hb, hd the ranks h(q) = y n + x.  With n <= 8192 every
// coordinate difference is below 2^14, each cofactor and lifted term below
// 2^29 and the determinant below 2^61: exact in 64-bit integers.
__device__ __forceinline__ bool in_circle(int ax, int ay, int bx, int by, int dx, int dy,
                                          long long hp, long long ha, long long hb,
                                          long long hd) {
  // rows: p - d, a - d, b - d (p = origin)
  const int r0x = -dx, r0y = -dy, r1x = ax - dx, r1y = ay - dy, r2x = bx - dx, r2y = by - dy;
  const long long m0 = (long long)r1x * r2y - (long long)r1y * r2x;  // cofactor of row 0
  const long long m1 = (long long)r0x * r2y - (long long)r0y * r2x;
  const long long m2 = (long long)r0x * r1y - (long long)r0y * r1x;
  const long long z0 = (long long)r0x * r0x + (long long)r0y * r0y,
                  z1 = (long long)r1x * r1x + (long long)r1y * r1y,
                  z2 = (long long)r2x * r2x + (long long)r2y * r2y;
  const long long d0 = z0 * m0 - z1 * m1 + z2 * m2;
  if (d0 != 0) return d0 > 0;
  // co-circular: z(q) += delta(q), delta growing (infinitesimally) with
  // h(q); the determinant is linear in the z column, so the sign is that of
  // the top-ranked point's cofactor (none is zero: no three of four
  // co-circular points are collinear)
  if (hp > ha && hp > hb && hp > hd) return m0 > 0;
  if (ha > hb && ha > hd) return m1 < 0;
  if (hb > hd) return m2 > 0;
  return m0 - m1 + m2 < 0;
}

__device__ __forceinline__ long long hkey(int n, int x, int y) { return (long long)y * n + x; }

// Tiles are visited in bricks of 4 x 4 (64 x 64 pixels), so that the sites
// a warp handles lie close together and their windows overlap.
constexpr int kBrick = 4;
__device__ __forceinline__ int brick_of(int tx, int ty, int nt0) {
  return ((ty / kBrick) * (nt0 / kBrick) + tx / kBrick) * (kBrick * kBrick) +
         (ty % kBrick) * kBrick + tx % kBrick;
}

// Is every grid point in the closed circumdisc of (site, u, w) inside the
// window?  Relative to the site: centre (Nx, Ny) / D (D > 0), radius^2
// (Nx^2 + Ny^2) / D^2 (the circle passes through the site).  The grid
// outside the window [x0, x1] x [y0, y1] is up to four strips; the disc
// must stay strictly clear of each (exact in 128-bit integers).
__device__ __forceinline__ __int128 axis_gap(long long N, long long D, int lo, int hi) {
  const __int128 a = (__int128)lo * D - N, b = (__int128)N - (__int128)hi * D;
  return a > 0 ? a : (b > 0 ? b : (__int128)0);
}
__device__ bool clear_of(long long Nx, long long Ny, long long D, int lx, int hx, int ly,
                         int hy) {
  if (lx > hx || ly > hy) return true;  // empty strip
  const __int128 gx = axis_gap(Nx, D, lx, hx), gy = axis_gap(Ny, D, ly, hy);
  return gx * gx + gy * gy > (__int128)Nx * Nx + (__int128)Ny * Ny;
}
__device__ bool disc_in_window(int ux, int uy, int wx, int wy, int sx, int sy, int x0, int x1,
                               int y0, int y1, int n) {
  const long long u2 = (long long)ux * ux + (long long)uy * uy,
                  w2 = (long long)wx * wx + (long long)wy * wy;
  const long long D = 2 * cross(ux, uy, wx, wy);
  const long long Nx = wy * u2 - uy * w2, Ny = ux * w2 - wx * u2;
  const int gx0 = -sx, gx1 = n - 1 - sx, gy0 = -sy, gy1 = n - 1 - sy;  // the grid
  const int wx0 = x0 - sx, wx1 = x1 - sx, wy0 = y0 - sy, wy1 = y1 - sy;  // the window
  return clear_of(Nx, Ny, D, gx0, wx0 - 1, gy0, gy1) &&
         clear_of(Nx, Ny, D, wx1 + 1, gx1, gy0, gy1) &&
         clear_of(Nx, Ny, D, wx0, wx1, gy0, wy0 - 1) &&
         clear_of(Nx, Ny, D, wx0, wx1, wy1 + 1, gy1);
}

// disc_in_window decided in floats where that is safe (false: not decided).
// The centre's error is below e (its products' roundings over |D|), the
// radius's below twice that; a grid point outside the window is at least a
// pixel past its edge.
__device__ __forceinline__ bool disc_surely_in(int ux, int uy, int wx, int wy, int sx, int sy,
                                               int x0, int x1, int y0, int y1, int n) {
  const float fux = (float)ux, fuy = (float)uy, fwx = (float)wx, fwy = (float)wy;
  const float u2 = fux * fux + fuy * fuy, w2 = fwx * fwx + fwy * fwy;
  const float iD = 0.5f / (float)(ux * wy - uy * wx);
  const float cx = (fwy * u2 - fuy * w2) * iD, cy = (fux * w2 - fwx * u2) * iD;
  const float e = (fabsf(fwy) + fabsf(fwx)) * u2 + (fabsf(fuy) + fabsf(fux)) * w2;
  const float r = sqrtf(cx * cx + cy * cy) + 4.f * e * iD * 0x1p-21f + 0.01f;
  return (x1 == n - 1 || cx + r < (float)(x1 + 1 - sx)) && (x0 == 0 || cx - r > (float)(x0 - 1 - sx)) &&
         (y1 == n - 1 || cy + r < (float)(y1 + 1 - sy)) && (y0 == 0 || cy - r > (float)(y0 - 1 - sy));
}

// Site occupancy of 16 x 16 pixel tiles and its pyramid (level l: tiles of
// 16 << l pixels, a byte each, nonzero when the tile holds a site).
constexpr int kTile = 16;  // 1 << 4
constexpr int kLevels = 16;
struct Pyr {
  const uint8_t *occ;
  int off[kLevels], nt[kLevels];
  int top;  // the one-node level
};

// The sites in tile order (k_dt_order): tile i's (brick order) are order[p ..
// p + count[i]), p = off[cls[i] ntiles + i].
struct TileSites {
  const int *order;
  const unsigned *off, *count;
  const uint8_t *cls;
};
__device__ __forceinline__ unsigned tile_start(const TileSites &ts, int nt0, int i) {
  return __ldg(ts.off + (size_t)ts.cls[i] * nt0 * nt0 + i);
}

// Free sites: bits & ~fixed.
__device__ __forceinline__ uint64_t free_word(const uint64_t *bits, const uint64_t *fixed,
                                              size_t i) {
  return fixed ? bits[i] & ~fixed[i] : bits[i];
}

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// The star of one site, held by a warp: neighbour k (packed (dx, dy),
// angular order) in lane k % 32 of `a` (k < 32) or of `b`; m and overflow
// are the same in every lane.  Every function below is called by all 32
// lanes with the same arguments and takes the same branches in each.
struct WStar {
  int a, b;
  int m;
  bool overflow;
};

__device__ __forceinline__ int wget(const WStar &s, int k) {
  return __shfl_sync(kFull, k < 32 ? s.a : s.b, k & 31);
}

__device__ __forceinline__ void wset(WStar &s, int k, int v) {
  if (lane_id() == (k & 31)) {
    if (k < 32) s.a = v;
    else s.b = v;
  }
}

// v becomes neighbour pos; neighbours pos.. move up one
__device__ __forceinline__ void wins(WStar &s, int pos, int v) {
  const int l = lane_id();
  const int aup = __shfl_up_sync(kFull, s.a, 1), bup = __shfl_up_sync(kFull, s.b, 1);
  const int a31 = __shfl_sync(kFull, s.a, 31);
  const int na = l < pos ? s.a : (l == pos ? v : aup);
  const int nb = l + 32 < pos ? s.b : (l + 32 == pos ? v : (l == 0 ? a31 : bup));
  s.a = na;
  s.b = nb;
  ++s.m;
}

// neighbour k leaves; neighbours k+1.. move down one
__device__ __forceinline__ void wdel(WStar &s, int k) {
  const int l = lane_id();
  const int adn = __shfl_down_sync(kFull, s.a, 1), bdn = __shfl_down_sync(kFull, s.b, 1);
  const int b0 = __shfl_sync(kFull, s.b, 0);
  const int na = l < k ? s.a : (l == 31 ? b0 : adn);
  const int nb = l + 32 < k ? s.b : bdn;
  s.a = na;
  s.b = nb;
  --s.m;
}

// Insert candidate q (relative (qx, qy)) into the star of site (sx, sy).
// The star is sorted by angle from the +x axis; inverted about the site, its
// neighbours are the hull vertices facing away from the site, and a
// candidate inside that hull never becomes one later (the hull only grows).
__device__ void winsert(WStar &st, int n, int sx, int sy, int qx, int qy) {
  const long long hp = hkey(n, sx, sy), hq = hkey(n, sx + qx, sy + qy);
  const int qv = pk(qx, qy), l = lane_id();
  int m = st.m;
  // q's position (the neighbours before it in angle form a prefix) and a
  // neighbour on the same ray, each lane for its two entries
  const int hqh = half_of(qx, qy);
  bool ba = false, sa = false, bb = false, sb = false;
  if (l < m) {
    const int ux = pdx(st.a), uy = pdy(st.a), hu = half_of(ux, uy);
    const long long c = cross(ux, uy, qx, qy);
    ba = hu < hqh || (hu == hqh && c > 0);
    sa = c == 0 && hu == hqh;
  }
  if (l + 32 < m) {
    const int ux = pdx(st.b), uy = pdy(st.b), hu = half_of(ux, uy);
    const long long c = cross(ux, uy, qx, qy);
    bb = hu < hqh || (hu == hqh && c > 0);
    sb = c == 0 && hu == hqh;
  }
  const unsigned mba = __ballot_sync(kFull, ba), mbb = __ballot_sync(kFull, bb);
  const unsigned msa = __ballot_sync(kFull, sa), msb = __ballot_sync(kFull, sb);
  const int pos = __popc(mba) + __popc(mbb);
  const int same = msa ? __ffs(msa) - 1 : (msb ? 31 + __ffs(msb) : -1);
  int iq;
  if (same >= 0) {
    // the nearer site on a ray wins (the farther one is strictly inside
    // every circle through the site and the nearer one); a nearer q lies
    // outside the hull, so it takes the neighbour's place
    const int u = wget(st, same), ux = pdx(u), uy = pdy(u);
    if ((long long)qx * qx + (long long)qy * qy >= (long long)ux * ux + (long long)uy * uy) return;
    wset(st, same, qv);
    iq = same;
  } else {
    if (m >= 2) {
      const int u = wget(st, (pos + m - 1) % m), w = wget(st, pos % m);
      const int ux = pdx(u), uy = pdy(u), wx = pdx(w), wy = pdy(w);
      if (!open_gap(ux, uy, wx, wy) &&
          !in_circle(ux, uy, wx, wy, qx, qy, hp, hkey(n, sx + ux, sy + uy),
                     hkey(n, sx + wx, sy + wy), hq))
        return;  // inside the hull: never a neighbour
    }
    if (m >= kStar) {
      st.overflow = true;
      return;
    }
    wins(st, pos, qv);
    m = st.m;
    iq = pos;
  }
  // neighbours q now covers: clockwise of q, then counter-clockwise
  while (m >= 3) {
    const int iu = iq ? iq - 1 : m - 1, iuu = iu ? iu - 1 : m - 1;
    const int u = wget(st, iu), uu = wget(st, iuu);
    const int ax = pdx(uu), ay = pdy(uu), vx = pdx(u), vy = pdy(u);
    if (open_gap(ax, ay, qx, qy) ||
        in_circle(ax, ay, qx, qy, vx, vy, hp, hkey(n, sx + ax, sy + ay), hq,
                  hkey(n, sx + vx, sy + vy)))
      break;
    wdel(st, iu);
    m = st.m;
    if (iu < iq) --iq;
  }
  while (m >= 3) {
    const int iw = iq + 1 < m ? iq + 1 : 0, iww = iw + 1 < m ? iw + 1 : 0;
    const int w = wget(st, iw), ww = wget(st, iww);
    const int bx = pdx(ww), by = pdy(ww), vx = pdx(w), vy = pdy(w);
    if (open_gap(qx, qy, bx, by) ||
        in_circle(qx, qy, bx, by, vx, vy, hp, hq, hkey(n, sx + bx, sy + by),
                  hkey(n, sx + vx, sy + vy)))
      break;
    wdel(st, iw);
    m = st.m;
    if (iw < iq) --iq;
  }
}

// Rows [lo, hi] of band b as a bit mask.
__device__ __forceinline__ uint64_t band_rows(int b, int lo, int hi) {
  lo = max(lo - b * kBand, 0);
  hi = min(hi - b * kBand, kBand - 1);
  if (lo > hi) return 0ull;
  const uint64_t up = hi >= 63 ? ~0ull : ((2ull << hi) - 1ull);
  return up & ~((1ull << lo) - 1ull);
}

// The star of site (sx, sy) among the free sites of the window [x0, x1] x
// [y0, y1] by gift wrapping, when they are at most 64 (else false, st unchanged).  The
// candidates lie two per lane; from the nearest one (always a neighbour), the
// next neighbour counter-clockwise of u is the candidate left of u that sees
// (site, u) under the largest angle: a float cotangent (exact integer
// numerator and denominator, one division) and one warp minimum decide, and
// candidates within its error of the minimum -- co-circular ones above all -- are
// compared with the exact perturbed predicate.  An open gap (no candidate to
// the left) ends the walk; the rest is walked clockwise.  Inserting the same
// candidates one by one (winsert) gives the same star in about ten times the
// instructions: every insertion is a chain of decisions the lanes cannot share.
__device__ bool wwrap(WStar &st, const uint64_t *bits, const uint64_t *fixed, int n, int sx, int sy,
                      int x0, int x1, int y0, int y1, int *buf) {
  const int lane = lane_id();
  int cnt = 0;
  for (int cx = x0; cx <= x1; cx += 32) {
    const int x = cx + lane;
    for (int b = y0 / kBand; b <= y1 / kBand; ++b) {
      uint64_t w = 0;
      if (x <= x1) w = free_word(bits, fixed, (size_t)b * n + x) & band_rows(b, y0, y1);
      if (x == sx && sy / kBand == b) w &= ~(1ull << (sy % kBand));
      const int mine = __popcll(w);
      int incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(kFull, incl, 31);
      if (cnt + total > 64) return false;
      int pos = cnt + incl - mine;
      while (w) {
        const int i = __ffsll((long long)w) - 1;
        w &= w - 1ull;
        buf[pos++] = pk(x - sx, b * kBand + i - sy);
      }
      cnt += total;
    }
  }
  __syncwarp();
  const bool two = cnt > 32;
  const int qa = lane < cnt ? buf[lane] : 0, qb = lane + 32 < cnt ? buf[lane + 32] : 0;
  const int ax = pdx(qa), ay = pdy(qa), bx = pdx(qb), by = pdy(qb);
  const int a2 = ax * ax + ay * ay, b2 = bx * bx + by * by;
  __syncwarp();
  st.a = st.b = 0;
  st.m = 0;
  if (cnt == 0) return true;
  const long long hp = hkey(n, sx, sy);
  // the neighbour after u in direction dir (1 counter-clockwise), 0: none
  auto next = [&](int u, int dir) -> int {
    const int ux = pdx(u), uy = pdy(u);
    auto key = [&](int q, int qx, int qy, int q2) -> int {
      const int c = dir * (ux * qy - uy * qx);
      const float k = __fdividef((float)(q2 - ux * qx - uy * qy), (float)c);
      const int i = __float_as_int(k);
      return q != 0 && c > 0 ? i ^ ((i >> 31) & 0x7fffffff) : INT_MAX;
    };
    const int ka = key(qa, ax, ay, a2), kb = two ? key(qb, bx, by, b2) : INT_MAX;
    const int k = __reduce_min_sync(kFull, min(ka, kb));
    if (k == INT_MAX) return 0;
    // integers below 2^28 to float and the division: 2^-20 relative in all
    const float f = __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
    const float t = f + fabsf(f) * 0x1p-17f;
    const int ti = __float_as_int(t), tk = ti ^ ((ti >> 31) & 0x7fffffff);
    unsigned ma = __ballot_sync(kFull, ka <= tk), mb = two ? __ballot_sync(kFull, kb <= tk) : 0u;
    int best = 0;
    while (ma | mb) {
      int c;
      if (ma) {
        c = __shfl_sync(kFull, qa, __ffs(ma) - 1);
        ma &= ma - 1u;
      } else {
        c = __shfl_sync(kFull, qb, __ffs(mb) - 1);
        mb &= mb - 1u;
      }
      if (best) {
        const int px = pdx(best), py = pdy(best), cx = pdx(c), cy = pdy(c);
        const long long hu = hkey(n, sx + ux, sy + uy), hb = hkey(n, sx + px, sy + py),
                        hc = hkey(n, sx + cx, sy + cy);
        const bool inside = dir > 0 ? in_circle(ux, uy, px, py, cx, cy, hp, hu, hb, hc)
                                    : in_circle(px, py, ux, uy, cx, cy, hp, hb, hu, hc);
        if (!inside) continue;
      }
      best = c;
    }
    return best;
  };
  // the nearest candidate
  const unsigned da = lane < cnt ? (unsigned)a2 : 0xffffffffu,
                 db = lane + 32 < cnt ? (unsigned)b2 : 0xffffffffu;
  const unsigned dm = __reduce_min_sync(kFull, min(da, db));
  const unsigned na = __ballot_sync(kFull, da == dm), nb = __ballot_sync(kFull, db == dm);
  const int u0 = na ? __shfl_sync(kFull, qa, __ffs(na) - 1) : __shfl_sync(kFull, qb, __ffs(nb) - 1);
  int m = 1, u = u0;
  wset(st, 0, u0);
  bool open = false;
  for (;;) {
    u = next(u, 1);
    if (u == u0) break;
    if (u == 0) {
      open = true;
      break;
    }
    if (m >= kStar) {  // (cannot happen with at most 64 candidates)
      st.overflow = true;
      return true;
    }
    wset(st, m++, u);
  }
  st.m = m;
  if (open) {
    for (u = u0;;) {
      u = next(u, -1);
      if (u == 0) break;
      if (st.m >= kStar) {
        st.overflow = true;
        return true;
      }
      wins(st, 0, u);
    }
    if (st.m == 1) {
      // nothing on either side: every candidate lies on one line through the site,
      // and the nearest one beyond the site is its other neighbour
      const int ux = pdx(u0), uy = pdy(u0);
      const unsigned oa = ax * ux + ay * uy < 0 ? (unsigned)a2 : 0xffffffffu,
                     ob = bx * ux + by * uy < 0 ? (unsigned)b2 : 0xffffffffu;
      const unsigned o = __reduce_min_sync(kFull, min(oa, ob));
      const unsigned ma = __ballot_sync(kFull, oa == o), mb = __ballot_sync(kFull, ob == o);
      if (o != 0xffffffffu) {
        wset(st, 1, ma ? __shfl_sync(kFull, qa, __ffs(ma) - 1) : __shfl_sync(kFull, qb, __ffs(mb) - 1));
        st.m = 2;
      }
    }
  }
  // the list starts with the smallest angle from the +x axis
  m = st.m;
  auto before = [](int p, int q) {
    const int px = pdx(p), py = pdy(p), qx = pdx(q), qy = pdy(q);
    const int hp_ = half_of(px, py), hq_ = half_of(qx, qy);
    return hp_ < hq_ || (hp_ == hq_ && px * qy - py * qx > 0);
  };
  const int last = wget(st, m - 1);
  int pa = __shfl_up_sync(kFull, st.a, 1), pb = __shfl_up_sync(kFull, st.b, 1);
  const int a31 = __shfl_sync(kFull, st.a, 31);
  if (lane == 0) {
    pa = last;
    pb = a31;
  }
  const unsigned ra = __ballot_sync(kFull, lane < m && before(st.a, pa));
  const unsigned rb = __ballot_sync(kFull, lane + 32 < m && before(st.b, pb));
  const int rot = ra ? __ffs(ra) - 1 : (rb ? 31 + __ffs(rb) : 0);
  auto at = [&](int k) {  // entry (k + rot) mod m
    k += rot;
    if (k >= m) k -= m;
    const int va = __shfl_sync(kFull, st.a, k & 31), vb = __shfl_sync(kFull, st.b, k & 31);
    return k < 32 ? va : vb;
  };
  const int ea = at(lane), eb = at(lane + 32);
  st.a = ea;
  st.b = eb;
  return true;
}

// Insert the free sites of the window [nx0, nx1] x [ny0, ny1] that are not
// in the window [x0, x1] x [y0, y1] inserted before; the lanes take 32
// columns at a time, then insert the sites they found one by one.  A tall window
// (few sites, or one at the end of a row, whose windows grow to the grid) looks at
// the occupancy of 64 x 64 pixels first, a lane per band: a load and a vote per 32
// columns of every band of an empty 8192 x 8192 took one warp 10 ms.
__device__ void wwindow(WStar &st, const uint64_t *bits, const uint64_t *fixed, int n, int sx,
                        int sy, const Pyr &py, int nx0, int nx1, int ny0, int ny1, int x0, int x1,
                        int y0, int y1) {
  const int l = lane_id(), b1 = ny1 / kBand;
  const bool tall = b1 - ny0 / kBand >= 4;
  const uint8_t *occ = py.occ + py.off[2];  // (tiles of 64 pixels)
  for (int cx = nx0; cx <= nx1; cx += 32) {
    const int x = cx + l;
    unsigned used = 0;
    for (int b = ny0 / kBand; b <= b1; ++b) {
      if (tall) {
        const int i = (b - ny0 / kBand) & 31;
        if (i == 0) {
          const uint8_t *o = occ + (size_t)min(b + l, n / kBand - 1) * py.nt[2];
          used = __ballot_sync(kFull, o[cx / kBand] | o[min(cx + 31, n - 1) / kBand]);
        }
        if (!((used >> i) & 1u)) {  // on to the next occupied band
          b += ((used >> i) ? __ffs((int)(used >> i)) - 1 : 32 - i) - 1;
          continue;
        }
      }
      uint64_t w = 0;
      if (x <= nx1) {
        w = free_word(bits, fixed, (size_t)b * n + x) & band_rows(b, ny0, ny1);
        if (x >= x0 && x <= x1) w &= ~band_rows(b, y0, y1);
      }
      unsigned pend = __ballot_sync(kFull, w != 0);
      while (pend) {
        const int L = __ffs(pend) - 1;
        pend &= pend - 1u;
        uint64_t wl = __shfl_sync(kFull, (unsigned long long)w, L);
        while (wl) {
          const int i = __ffsll((long long)wl) - 1;
          wl &= wl - 1ull;
          const int qx = cx + L - sx, qy = b * kBand + i - sy;
          if (qx != 0 || qy != 0) winsert(st, n, sx, sy, qx, qy);
        }
      }
    }
  }
}

// The bounding box of the closed disc with centre (Nx, Ny) / D relative to
// the site (radius = |centre|): FP64 with one pixel of slack, clipped to
// the grid, so it holds every grid point of the disc.
__device__ __forceinline__ void disc_box(long long Nx, long long Ny, long long D, int sx, int sy,
                                         int n, int &bx0, int &bx1, int &by0, int &by1) {
  const double cx = (double)Nx / (double)D, cy = (double)Ny / (double)D;
  const double r = sqrt(cx * cx + cy * cy) + 1.0;
  bx0 = (int)fmax(0.0, floor(sx + cx - r));
  bx1 = (int)fmin(n - 1.0, ceil(sx + cx + r));
  by0 = (int)fmax(0.0, floor(sy + cy - r));
  by1 = (int)fmin(n - 1.0, ceil(sy + cy + r));
}

// The sites of the box [bx0, bx1] x [by0, by1] outside the window that lie
// in the circumcircle of the star's triangle (site, u, w), a lane per
// column, are inserted; true when there were any (the triangle is gone).
__device__ bool wbox_scan(WStar &st, const uint64_t *bits, const uint64_t *fixed, int n, int sx,
                          int sy, int ux, int uy, int wx, int wy, int x0, int x1, int y0, int y1,
                          int bx0, int bx1, int by0, int by1) {
  const long long hp = hkey(n, sx, sy), hu = hkey(n, sx + ux, sy + uy),
                  hw = hkey(n, sx + wx, sy + wy);
  const int lane = lane_id();
  bool found = false;
  for (int cx = bx0; cx <= bx1; cx += 32) {
    const int x = cx + lane;
    for (int b = by0 / kBand; b <= by1 / kBand; ++b) {
      uint64_t w = 0;
      if (x <= bx1) {
        w = free_word(bits, fixed, (size_t)b * n + x) & band_rows(b, by0, by1);
        if (x >= x0 && x <= x1) w &= ~band_rows(b, y0, y1);
      }
      uint64_t hit = 0;
      while (w) {
        const int i = __ffsll((long long)w) - 1;
        w &= w - 1ull;
        const int qx = x - sx, qy = b * kBand + i - sy;
        if ((qx == ux && qy == uy) || (qx == wx && qy == wy)) continue;
        if (in_circle(ux, uy, wx, wy, qx, qy, hp, hu, hw, hkey(n, sx + qx, sy + qy)))
          hit |= 1ull << i;
      }
      unsigned pend = __ballot_sync(kFull, hit != 0);
      while (pend) {
        const int L = __ffs(pend) - 1;
        pend &= pend - 1u;
        uint64_t hl = __shfl_sync(kFull, (unsigned long long)hit, L);
        while (hl) {
          const int i = __ffsll((long long)hl) - 1;
          hl &= hl - 1ull;
          winsert(st, n, sx, sy, cx + L - sx, b * kBand + i - sy);
          found = true;
        }
      }
    }
  }
  return found;
}

// What a search of the occupancy pyramid looks for: the sites in the
// closed circumdisc of the star's triangle (site, u, w) -- centre (Nx, Ny) /
// D relative to the site -- or, for an open angular gap from u to w
// (counter-clockwise, >= pi), the sites strictly inside its cone
// {q : u x q > 0 or q x w > 0}.
struct Probe {
  bool cone;
  int ux, uy, wx, wy;
  long long Nx, Ny, D, hp, hu, hw;
  float cx, cy, r, slack;  // the disc in floats, and the error of a distance to it
};

// Can the tile [px0, px1] x [qy0, qy1] hold a site the probe looks for?
__device__ __forceinline__ bool probe_node(const Probe &pr, int sx, int sy, int px0, int px1,
                                           int qy0, int qy1) {
  if (!pr.cone) {
    // the tile's distance from the centre against the radius, in floats where
    // their difference is above the error, else exactly
    const float dx = fmaxf(fmaxf((float)(px0 - sx) - pr.cx, pr.cx - (float)(px1 - sx)), 0.f);
    const float dy = fmaxf(fmaxf((float)(qy0 - sy) - pr.cy, pr.cy - (float)(qy1 - sy)), 0.f);
    const float d = sqrtf(dx * dx + dy * dy) - pr.r;
    if (d > pr.slack) return false;
    if (d < -pr.slack) return true;
    return !clear_of(pr.Nx, pr.Ny, pr.D, px0 - sx, px1 - sx, qy0 - sy, qy1 - sy);
  }
  // the cross products are linear: their largest value is at a corner
  long long cu = LLONG_MIN, cw = LLONG_MIN;
  for (int c = 0; c < 4; ++c) {
    const int qx = ((c & 1) ? px1 : px0) - sx, qy = ((c >> 1) ? qy1 : qy0) - sy;
    cu = max(cu, cross(pr.ux, pr.uy, qx, qy));
    cw = max(cw, cross(qx, qy, pr.wx, pr.wy));
  }
  return cu > 0 || cw > 0;
}

// Is site q (relative to the site) one the probe looks for?
__device__ __forceinline__ bool probe_site(const Probe &pr, int n, int sx, int sy, int qx,
                                           int qy) {
  if (pr.cone) return cross(pr.ux, pr.uy, qx, qy) > 0 || cross(qx, qy, pr.wx, pr.wy) > 0;
  // decided by the float distance where that is safe (probe_node's bound)
  const float dx = (float)qx - pr.cx, dy = (float)qy - pr.cy;
  const float d = sqrtf(dx * dx + dy * dy) - pr.r;
  if (d > pr.slack) return false;
  if (d < -pr.slack) return true;
  if ((qx == pr.ux && qy == pr.uy) || (qx == pr.wx && qy == pr.wy)) return false;
  return in_circle(pr.ux, pr.uy, pr.wx, pr.wy, qx, qy, pr.hp, pr.hu, pr.hw,
                   hkey(n, sx + qx, sy + qy));
}

constexpr int kWarpsPerBlock = 4;  // k_dt_star's blocks: 128 threads
constexpr int kFrontier = 1536;    // pyramid nodes one warp's search holds
enum { kFinal = 0, kInserted = 1, kGaveUp = 2 };

// Warp-parallel search of the occupancy pyramid for the probe's sites
// outside the window.  The nodes still to test form a stack in the warp's
// shared memory (stk, sp of them already there); each step the lanes take up
// to 32 nodes from its top, and an occupied node not wholly inside the
// window that the probe can reach either puts its children on the stack or,
// as a 16 x 16 tile, has its sites tested by its lane.  As soon as a step
// finds sites, the tile nearest the site among those with any decides: for a
// disc every site of it inside the circle is inserted, for a cone the first
// one found (kInserted).  kFinal when no site is found; kGaveUp when the stack
// would overflow (the caller then widens the window instead).  Each step
// pops at least one node and pushes only lower levels, so the search ends;
// a descent adds at most 3 x 32 nodes per level, so 14 levels stay below
// kFrontier.
__device__ int wsearch(WStar &st, const Pyr &py, const TileSites &ts, int n, int sx, int sy,
                       const Probe &pr, int x0, int x1, int y0, int y1, unsigned *stk, int sp) {
  const int lane = lane_id(), nt0 = py.nt[0];
  while (sp > 0) {
    const int k = min(sp, 32);
    unsigned v = 0;
    if (lane < k) v = stk[sp - k + lane];
    __syncwarp();
    sp -= k;
    unsigned ch[4];
    int nch = 0, hq = 0;
    unsigned key = 0xffffffffu;  // (distance to the site, lane) of a tile with sites found
    if (lane < k) {
      const int l = (int)(v >> 28), tx = (int)((v >> 14) & 0x3fff), ty = (int)(v & 0x3fff);
      const int S = kTile << l;
      const int px0 = tx * S, px1 = min(px0 + S, n) - 1, qy0 = ty * S, qy1 = min(qy0 + S, n) - 1;
      if (py.occ[py.off[l] + ty * py.nt[l] + tx] &&
          !(px0 >= x0 && px1 <= x1 && qy0 >= y0 && qy1 <= y1) &&
          probe_node(pr, sx, sy, px0, px1, qy0, qy1)) {
        if (l > 0) {
          const int cn = py.nt[l - 1];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int cx = 2 * tx + (c & 1), cy = 2 * ty + (c >> 1);
            if (cx < cn && cy < cn)
              ch[nch++] = ((unsigned)(l - 1) << 28) | ((unsigned)cx << 14) | (unsigned)cy;
          }
        } else {  // a tile: its sites until one is found
          const int i = brick_of(tx, ty, nt0);
          const unsigned p = tile_start(ts, nt0, i);
          for (unsigned j = 0, cnt = ts.count[i]; j < cnt; ++j) {
            const int q = __ldg(ts.order + p + j), qx = (q & 0xffff) - sx, qy = pdy(q) - sy;
            if (!probe_site(pr, n, sx, sy, qx, qy)) continue;
            hq = pk(qx, qy);
            const long long dx = px0 + kTile / 2 - sx, dy = qy0 + kTile / 2 - sy;
            key = (unsigned)min((dx * dx + dy * dy) >> 4, (long long)(1 << 26)) << 5 | lane;
            break;
          }
        }
      }
    }
    const unsigned best = __reduce_min_sync(kFull, key);
    if (best != 0xffffffffu) {
      const int L = (int)(best & 31u);
      const unsigned vL = __shfl_sync(kFull, v, L);
      const int qL = __shfl_sync(kFull, hq, L);
      if (pr.cone) {
        winsert(st, n, sx, sy, pdx(qL), pdy(qL));
        return kInserted;
      }
      // the disc: every site of that tile inside the circle, a lane per site
      const int i = brick_of((int)((vL >> 14) & 0x3fff), (int)(vL & 0x3fff), nt0);
      const unsigned p = tile_start(ts, nt0, i), cnt = ts.count[i];
      for (unsigned j0 = 0; j0 < cnt; j0 += 32) {
        int q = 0;
        bool hit = false;
        if (j0 + lane < cnt) {
          const int e = __ldg(ts.order + p + j0 + lane);
          q = pk((e & 0xffff) - sx, pdy(e) - sy);
          hit = probe_site(pr, n, sx, sy, pdx(q), pdy(q));
        }
        for (unsigned pend = __ballot_sync(kFull, hit); pend; pend &= pend - 1u) {
          const int c = __shfl_sync(kFull, q, __ffs(pend) - 1);
          winsert(st, n, sx, sy, pdx(c), pdy(c));
        }
      }
      return kInserted;
    }
    // the children onto the stack
    int off = nch;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, off, o);
      if (lane >= o) off += y;
    }
    const int total = __shfl_sync(kFull, off, 31);
    off -= nch;
    if (sp + total > kFrontier) return kGaveUp;
    for (int c = 0; c < nch; ++c) stk[sp + off + c] = ch[c];
    __syncwarp();
    sp += total;
  }
  return kFinal;
}

// Search for the sites in the circumcircle of (site, u, w) outside the
// window, starting at the pyramid level where the disc's bounding box spans
// at most 2 x 2 nodes.
__device__ int wdisc_search(WStar &st, const Pyr &py, const TileSites &ts, int n, int sx, int sy, int ux, int uy, int wx, int wy, int x0, int x1,
                            int y0, int y1, unsigned *stk) {
  Probe pr;
  pr.cone = false;
  pr.ux = ux, pr.uy = uy, pr.wx = wx, pr.wy = wy;
  const long long u2 = (long long)ux * ux + (long long)uy * uy,
                  w2 = (long long)wx * wx + (long long)wy * wy;
  pr.D = 2 * cross(ux, uy, wx, wy);
  pr.Nx = wy * u2 - uy * w2;
  pr.Ny = ux * w2 - wx * u2;
  pr.hp = hkey(n, sx, sy), pr.hu = hkey(n, sx + ux, sy + uy), pr.hw = hkey(n, sx + wx, sy + wy);
  {
    const double cx = (double)pr.Nx / (double)pr.D, cy = (double)pr.Ny / (double)pr.D;
    pr.cx = (float)cx, pr.cy = (float)cy;
    pr.r = (float)sqrt(cx * cx + cy * cy);
    // centre, radius, squares, root and difference: a few roundings of at most
    // |c| + r + n each
    pr.slack = (2.f * pr.r + 16384.f) * 0x1p-20f;
  }
  int bx0, bx1, by0, by1;
  disc_box(pr.Nx, pr.Ny, pr.D, sx, sy, n, bx0, bx1, by0, by1);
  int l0 = 0;
  while (l0 < py.top && (((bx1 >> (4 + l0)) - (bx0 >> (4 + l0))) > 1 ||
                         ((by1 >> (4 + l0)) - (by0 >> (4 + l0))) > 1))
    ++l0;
  const int tx0 = bx0 >> (4 + l0), ty0 = by0 >> (4 + l0);
  const int ntx = (bx1 >> (4 + l0)) - tx0 + 1, nty = (by1 >> (4 + l0)) - ty0 + 1;  // <= 2 each
  const int lane = lane_id();
  if (lane < ntx * nty)
    stk[lane] = ((unsigned)l0 << 28) | ((unsigned)(tx0 + lane % ntx) << 14) |
                (unsigned)(ty0 + lane / ntx);
  __syncwarp();
  return wsearch(st, py, ts, n, sx, sy, pr, x0, x1, y0, y1, stk, ntx * nty);
}

// Search for the sites strictly inside the open gap's cone, from the root.
__device__ int wcone_search(WStar &st, const Pyr &py, const TileSites &ts, int n, int sx, int sy, int ux, int uy, int wx, int wy, int x0, int x1,
                            int y0, int y1, unsigned *stk) {
  Probe pr;
  pr.cone = true;
  pr.ux = ux, pr.uy = uy, pr.wx = wx, pr.wy = wy;
  pr.Nx = pr.Ny = pr.D = pr.hp = pr.hu = pr.hw = 0;
  pr.cx = pr.cy = pr.r = pr.slack = 0.f;
  if (lane_id() == 0) stk[0] = (unsigned)py.top << 28;
  __syncwarp();
  return wsearch(st, py, ts, n, sx, sy, pr, x0, x1, y0, y1, stk, 1);
}

// Neighbour (k + 1) % m for the lane's entry k (lane l: k = l or l + 32).
__device__ __forceinline__ int wnext(const WStar &s, int k) {
  const int e = k + 1 < s.m ? k + 1 : 0;
  const int va = __shfl_sync(kFull, s.a, e & 31), vb = __shfl_sync(kFull, s.b, e & 31);
  return e < 32 ? va : vb;
}

// The Delaunay star of site (sx, sy), computed by a warp.  The first window
// is sized from the local site density (the 3 x 3 tiles around the site:
// half-width kWindow site spacings, which holds a regular site's neighbours
// and triangles' circles).  When kWiden or more of its triangles reach past
// it (as around irregular sites), the window grows once before any search
// (wrapping again costs less than searching); then the certificate settles the
// triangles exactly, and only a star of fewer than two neighbours doubles the
// window again.  More than 64 candidates (a crowded or uneven neighbourhood) take windows
// of kRing spacings, doubled, wrapped if that leaves few enough, else inserted ring by
// ring: what is inserted one by one counts there.  (kWindow 1.6 to 2.3 and kGrow 1.5 to 2 measure within 5 %, kWiden 3 or
// never 8 % slower on irregular sites.)  A star whose sites all lie on one line
// widens up to kLine first: the next row of a lattice is nearer than what a search of
// the gap's half plane finds.  Returns false when the star
// overflowed, which depends on the order of the insertions too: `rings` inserts the
// windows of 1.4, 2.8, 5.6 ... spacings ring by ring, nearer sites first.
constexpr float kWindow = 2.0f, kGrow = 1.7f, kRing = 1.4f;
constexpr int kWiden = 1;
constexpr int kLine = 128;
constexpr int kBoxCols = 96, kBoxBands = 3;  // largest disc box scanned directly
template <bool rings>
__device__ bool wsite_star(WStar &st, const uint64_t *bits, const uint64_t *fixed, int n, int sx,
                           int sy, const Pyr &py, const TileSites &ts, unsigned *stk) {
  st.a = st.b = 0;
  st.m = 0;
  st.overflow = false;
  const int tx = sx / kTile, ty = sy / kTile, nt0 = py.nt[0], lane = lane_id();
  // (a lane per tile)
  const int ti = tx - 1 + lane % 3, tj = ty - 1 + lane / 3;
  const bool tile = lane < 9 && ti >= 0 && ti < nt0 && tj >= 0 && tj < nt0;
  const unsigned cnt = __reduce_add_sync(kFull, tile ? ts.count[brick_of(ti, tj, nt0)] : 0u);
  const int tiles = __popc(__ballot_sync(kFull, tile));
  int W = (int)ceilf((rings ? kRing : kWindow) *
                     sqrtf((float)(tiles * kTile * kTile) / (float)max(cnt, 1u)));
  W = min(max(W, 4), 2 * n);
  int x0 = sx, x1 = sx, y0 = sy, y1 = sy;  // the window so far: the site
  bool first = true, wrap = !rings, small = rings;
  for (;;) {
    const int nx0 = max(0, sx - W), nx1 = min(n - 1, sx + W);
    const int ny0 = max(0, sy - W), ny1 = min(n - 1, sy + W);
    // wrapped in the first two windows while the candidates are few, then ring by ring
    // (the star so far is the one of every site of the window before)
    const bool few = wrap && wwrap(st, bits, fixed, n, sx, sy, nx0, nx1, ny0, ny1,
                                   reinterpret_cast<int *>(stk));
    if (wrap && !few && !small) {  // crowded: the smaller windows
      small = true;
      W = max(4, (int)ceilf(kRing / kWindow * W));
      continue;
    }
    wrap = few;
    if (!wrap) wwindow(st, bits, fixed, n, sx, sy, py, nx0, nx1, ny0, ny1, x0, x1, y0, y1);
    x0 = nx0;
    x1 = nx1;
    y0 = ny0;
    y1 = ny1;
    if (st.overflow) return false;
    if (x0 == 0 && y0 == 0 && x1 == n - 1 && y1 == n - 1) return true;  // every site seen
    // certificate, exact: the sites inside a triangle's circumcircle or an
    // open gap's cone are inserted until there are none.  A triangle (or gap)
    // a search found final stays final while it is in the star (its circle
    // and the window do not change), so its key (u, w) is kept, one per lane,
    // and not searched again after another triangle changed the star.
    long long vkey = 0;
    int nver = 0;
    bool ok, changed;
    int rounds = 0;
    do {
      if (++rounds > (1 << 16)) {  // more insertions than any star needs: give up
        st.overflow = true;
        return false;
      }
      changed = false;
      const int m = st.m;
      ok = m >= 2;  // fewer than two neighbours: a wider window
      if (m == 2 && !rings && W < kLine) {
        const int u = wget(st, 0), w = wget(st, 1);
        ok = cross(pdx(u), pdy(u), pdx(w), pdy(w)) != 0;
      }
      if (!ok) break;
      // each lane checks its two triangles against the window; the ones
      // that the window does not settle are searched one by one
      bool need_a = false, need_b = false;
      {
        const int wa = wnext(st, lane), wb = wnext(st, lane + 32);
        if (lane < m) {
          const int ux = pdx(st.a), uy = pdy(st.a), wx = pdx(wa), wy = pdy(wa);
          need_a = open_gap(ux, uy, wx, wy) ||
                   (!disc_surely_in(ux, uy, wx, wy, sx, sy, x0, x1, y0, y1, n) &&
                    !disc_in_window(ux, uy, wx, wy, sx, sy, x0, x1, y0, y1, n));
        }
        if (lane + 32 < m) {
          const int ux = pdx(st.b), uy = pdy(st.b), wx = pdx(wb), wy = pdy(wb);
          need_b = open_gap(ux, uy, wx, wy) ||
                   (!disc_surely_in(ux, uy, wx, wy, sx, sy, x0, x1, y0, y1, n) &&
                    !disc_in_window(ux, uy, wx, wy, sx, sy, x0, x1, y0, y1, n));
        }
      }
      unsigned pa = __ballot_sync(kFull, need_a), pb = __ballot_sync(kFull, need_b);
      if (first && rounds == 1 && __popc(pa) + __popc(pb) >= kWiden) {
        ok = false;  // an irregular neighbourhood: a wider window before searching
        break;
      }
      while (pa || pb) {
        int k;
        if (pa) {
          k = __ffs(pa) - 1;
          pa &= pa - 1u;
        } else {
          k = 31 + __ffs(pb);
          pb &= pb - 1u;
        }
        const int u = wget(st, k), w = wget(st, k + 1 < m ? k + 1 : 0);
        const int ux = pdx(u), uy = pdy(u), wx = pdx(w), wy = pdy(w);
        const long long key = ((long long)(unsigned)u << 32) | (unsigned)w;
        if (__ballot_sync(kFull, lane < nver && vkey == key)) continue;  // known final
        int res;
        if (open_gap(ux, uy, wx, wy)) {
          res = wcone_search(st, py, ts, n, sx, sy, ux, uy, wx, wy, x0, x1, y0, y1, stk);
        } else {
          // a small disc: its bounding box outside the window, column by
          // column; a large one through the occupancy pyramid
          const long long u2 = (long long)ux * ux + (long long)uy * uy,
                          w2 = (long long)wx * wx + (long long)wy * wy;
          const long long D = 2 * cross(ux, uy, wx, wy);
          int bx0, bx1, by0, by1;
          disc_box(wy * u2 - uy * w2, ux * w2 - wx * u2, D, sx, sy, n, bx0, bx1, by0, by1);
          res = bx1 - bx0 < kBoxCols && by1 / kBand - by0 / kBand < kBoxBands
                    ? (wbox_scan(st, bits, fixed, n, sx, sy, ux, uy, wx, wy, x0, x1, y0, y1, bx0,
                                 bx1, by0, by1)
                           ? kInserted
                           : kFinal)
                    : wdisc_search(st, py, ts, n, sx, sy, ux, uy, wx, wy, x0, x1, y0, y1,
                                   stk);
        }
        if (res == kGaveUp) {  // the search did not fit: a wider window instead
          ok = false;
          break;
        }
        const bool found = res == kInserted;
        if (st.overflow) return false;
        if (found) {
          changed = true;
          break;
        }
        if (nver < 32) {  // final: remembered
          if (lane == nver) vkey = key;
          ++nver;
        }
      }
    } while (changed);
    if (ok) return true;
    wrap = wrap && first;
    W = first && !small ? min((int)ceilf(kGrow * W), 2 * n) : min(2 * W, 2 * n);
    first = false;
  }
}

// Sites per tile (brick order) and level 0 of the occupancy pyramid: one
// thread per (column, 64-row band).
__global__ void k_dt_tiles(const uint64_t *__restrict__ bits, const uint64_t *__restrict__ fixed,
                           int n, uint8_t *occ0, int nt0, unsigned *tcnt) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int nb = n / kBand;
  if (i >= (long long)nb * n) return;
  const int b = (int)(i / n), x = (int)(i % n);
  const uint64_t w = free_word(bits, fixed, (size_t)b * n + x);
  for (int q = 0; q < kBand / kTile; ++q) {
    const unsigned c = (unsigned)__popcll((w >> (q * kTile)) & 0xffffull);
    if (c) {
      const int ty = b * (kBand / kTile) + q, tx = x / kTile;
      occ0[ty * nt0 + tx] = 1;
      atomicAdd(&tcnt[brick_of(tx, ty, nt0)], c);
    }
  }
}

// Level l from level l - 1.
__global__ void k_dt_up(const uint8_t *__restrict__ lo, int nlo, uint8_t *hi, int nhi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nhi * nhi) return;
  const int x = i % nhi, y = i / nhi;
  uint8_t v = 0;
  for (int c = 0; c < 4; ++c) {
    const int cx = 2 * x + (c & 1), cy = 2 * y + (c >> 1);
    if (cx < nlo && cy < nlo) v |= lo[cy * nlo + cx];
  }
  hi[i] = v;
}

// The four-site form's lists (quad_stars): candidates, neighbours.  In a tile of which
// more than half is sites its smallest window (9 x 9 pixels) holds about 40: that form
// would try and leave its four sites to one warp, one after the other, so they take a
// warp each (a block of 121 x 121 sites 812 -> 691 us).
constexpr int kQuadCand = 32, kQuadStar = 16;
constexpr unsigned kTileCrowd = kTile * kTile / 2;

// Edge tiles first: an occupied tile with an empty tile (or the grid's edge)
// among its eight neighbours holds the sites whose stars reach far (flat
// triangles along the sites' boundary, convex-hull gaps).  Their sites are
// listed before the interior ones so the long stars start first instead of
// finishing last.  ccnt[c * ntiles + i]: the sites of brick-order tile i in
// class c (0 edge, 1 crowded, 2 interior).
__global__ void k_dt_class(const uint8_t *__restrict__ occ0, int nt0,
                           const unsigned *__restrict__ tilecnt, unsigned *ccnt, uint8_t *cls) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt0 * nt0) return;
  const int brick = i / (kBrick * kBrick), in = i % (kBrick * kBrick);
  const int tx = (brick % (nt0 / kBrick)) * kBrick + in % kBrick;
  const int ty = (brick / (nt0 / kBrick)) * kBrick + in / kBrick;
  bool edge = false;
  for (int dy = -1; dy <= 1; ++dy)
    for (int dx = -1; dx <= 1; ++dx) {
      const int x = tx + dx, y = ty + dy;
      edge |= x < 0 || y < 0 || x >= nt0 || y >= nt0 || !occ0[y * nt0 + x];
    }
  const unsigned c = tilecnt[i];
  const int k = edge ? 0 : (c > kTileCrowd ? 1 : 2);
  for (int j = 0; j < 3; ++j) ccnt[(size_t)j * nt0 * nt0 + i] = j == k ? c : 0u;
  cls[i] = (uint8_t)k;
}

// Per column: free sites in the bands before each band, and in the column.
// One warp per 32 columns; the band loop is unrolled so the loads overlap.
__global__ void k_dt_columns(const uint64_t *__restrict__ bits, const uint64_t *__restrict__ fixed,
                             int n, unsigned *colpre, unsigned *colcnt) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n) return;
  unsigned c = 0;
#pragma unroll 8
  for (int b = 0; b < n / kBand; ++b) {
    colpre[(size_t)b * n + x] = c;
    c += __popcll(free_word(bits, fixed, (size_t)b * n + x));
  }
  colcnt[x] = c;
}

// The sites in tile order, edge tiles first: one thread per tile (brick
// order), its sites by column, then row.
__global__ void k_dt_order(const uint64_t *__restrict__ bits, const uint64_t *__restrict__ fixed,
                           int n, int nt0, const unsigned *__restrict__ toff,
                           const uint8_t *__restrict__ cls, int *order) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nt0 * nt0) return;
  const int brick = i / (kBrick * kBrick), in = i % (kBrick * kBrick);
  const int tx = (brick % (nt0 / kBrick)) * kBrick + in % kBrick;
  const int ty = (brick / (nt0 / kBrick)) * kBrick + in / kBrick;
  const int y0 = ty * kTile, b = y0 / kBand, sh = y0 % kBand;
  unsigned pos = toff[(size_t)cls[i] * nt0 * nt0 + i];
  for (int x = tx * kTile; x < tx * kTile + kTile; ++x) {
    uint64_t w = (free_word(bits, fixed, (size_t)b * n + x) >> sh) & 0xffffull;
    while (w) {
      const int k = __ffsll((long long)w) - 1;
      w &= w - 1ull;
      order[pos++] = pk(x, y0 + k);
    }
  }
}

__device__ __forceinline__ int site_index(const uint64_t *bits, const uint64_t *fixed, int n,
                                          const unsigned *coloff, const unsigned *colpre, int x,
                                          int y) {
  const int b = y / kBand, i = y % kBand;
  const uint64_t w = free_word(bits, fixed, (size_t)b * n + x);
  const uint64_t below = i ? (w & ((1ull << i) - 1ull)) : 0ull;
  return (int)(coloff[x] + colpre[(size_t)b * n + x] + (unsigned)__popcll(below));
}

// What a star kernel writes per site (under its index in delaunayInput's
// order): its pixel, its star, the star's size and the triangles it writes --
// the ones it comes first in, in (x, y) order.
struct StarOut {
  const unsigned *coloff, *colpre;
  int *sitepos, *stars, *degree;
  unsigned *tcount;
  int *err;
};

__device__ __forceinline__ bool owns_tri(int sx, int sy, int u, int w) {
  const int ux = sx + pdx(u), uy = sy + pdy(u), wx = sx + pdx(w), wy = sy + pdy(w);
  return (sx < ux || (sx == ux && sy < uy)) && (sx < wx || (sx == wx && sy < wy));
}

// One site by the whole warp, any case.
template <bool rings>
__device__ __noinline__ void full_site(const uint64_t *bits, const uint64_t *fixed, int n, int pos,
                                       const Pyr &py, const TileSites &ts, unsigned *stk,
                                       const StarOut &out) {
  const int lane = lane_id();
  const int sx = pdx(pos) & 0xffff, sy = pdy(pos);
  const int xm = site_index(bits, fixed, n, out.coloff, out.colpre, sx, sy);
  WStar st;
  if (!wsite_star<rings>(st, bits, fixed, n, sx, sy, py, ts, stk)) {
    if (lane == 0) {
      atomicOr(out.err, 1);
      out.sitepos[xm] = pos;
      out.degree[xm] = 0;
      out.tcount[xm] = 0;
    }
    return;
  }
  const int m = st.m;
  int *row = out.stars + (size_t)xm * kStar;
  if (lane < m) row[lane] = st.a;
  if (lane + 32 < m) row[lane + 32] = st.b;
  auto owns = [&](int u, int w) {
    return m >= 2 && !open_gap(pdx(u), pdy(u), pdx(w), pdy(w)) && owns_tri(sx, sy, u, w);
  };
  const int wa = wnext(st, lane), wb = wnext(st, lane + 32);
  const bool oa = lane < m && owns(st.a, wa), ob = lane + 32 < m && owns(st.b, wb);
  const int own = __popc(__ballot_sync(kFull, oa)) + __popc(__ballot_sync(kFull, ob));
  if (lane == 0) {
    out.sitepos[xm] = pos;
    out.degree[xm] = m;
    out.tcount[xm] = own;
  }
}

// Four sites of a warp, eight lanes each, for the common case: at most 32
// candidates in a window of kQuadWindow spacings (radius <= 31 pixels), a closed star
// of at most 16 neighbours, every triangle's circle surely inside the window.
// The same gift wrapping as wwrap; the four walks go in step, so a step's
// instructions serve four sites.  Offsets up to 31 pixels keep every cotangent's
// numerator and denominator exact in floats.  Returns the groups it leaves to
// full_site (none of 258,177 interior sites at 4096^2).  A warp per site by wwrap
// alone took 1,449 instructions a site, this 600.
constexpr float kQuadWindow = 1.8f;
struct QuadScratch {
  int cand[4][kQuadCand];
  int star[4][kQuadStar];
};

__device__ __forceinline__ unsigned quad_stars(const uint64_t *bits, const uint64_t *fixed, int n,
                                               int t0, int nsites, const Pyr &py,
                                               const TileSites &ts, QuadScratch &sc,
                                               const StarOut &out) {
  const int lane = lane_id(), g = lane >> 3, l = lane & 7;
  const bool on = t0 + g < nsites;
  const int epos = ts.order[min(t0 + g, nsites - 1)];
  const int sx = pdx(epos) & 0xffff, sy = pdy(epos);
  // the window from the 3 x 3 tiles' site counts
  const int tx = sx / kTile, ty = sy / kTile, nt0 = py.nt[0];
  unsigned near = 0;
  for (int k = l; k < 9; k += 8) {
    const int i = tx - 1 + k % 3, j = ty - 1 + k / 3;
    if (i >= 0 && i < nt0 && j >= 0 && j < nt0) near += ts.count[brick_of(i, j, nt0)];
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) near += __shfl_xor_sync(kFull, near, o);
  const int tiles = (min(tx + 1, nt0 - 1) - max(tx - 1, 0) + 1) *
                    (min(ty + 1, nt0 - 1) - max(ty - 1, 0) + 1);
  int W = (int)ceilf(kQuadWindow * sqrtf((float)(tiles * kTile * kTile) / (float)max(near, 1u)));
  W = max(W, 4);
  bool ok = on && W <= 31;
  W = min(W, 31);
  const int x0 = max(0, sx - W), x1 = min(n - 1, sx + W);
  const int y0 = max(0, sy - W), y1 = min(n - 1, sy + W), o = sy - y0;
  // candidates: a lane per column, a column's rows as one word from row y0 on
  int cnt = 0;
  {
    const int b0 = y0 / kBand, b1 = y1 / kBand, sh = y0 % kBand;
    const uint64_t rm = (2ull << (y1 - y0)) - 1ull;
    const int ncol = __reduce_max_sync(kFull, x1 - x0 + 1);
    for (int c = 0; c < ncol; c += 8) {
      const int x = x0 + c + l;
      uint64_t w = 0;
      if (ok && x <= x1) {
        w = free_word(bits, fixed, (size_t)b0 * n + x) >> sh;
        if (b1 > b0) w |= free_word(bits, fixed, (size_t)b1 * n + x) << (kBand - sh);
        w &= rm;
        if (x == sx) w &= ~(1ull << o);
      }
      const int mine = __popcll(w);
      int incl = mine;
#pragma unroll
      for (int i = 1; i < 8; i <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, i, 8);
        if (l >= i) incl += v;
      }
      int p = cnt + incl - mine;
      cnt += __shfl_sync(kFull, incl, 7, 8);
      while (w) {
        const int i = __ffsll((long long)w) - 1;
        w &= w - 1ull;
        if (p < kQuadCand) sc.cand[g][p] = pk(x - sx, i - o);
        ++p;
      }
    }
  }
  ok = ok && cnt >= 3 && cnt <= kQuadCand;
  __syncwarp();
  constexpr int kPer = kQuadCand / 8;
  const int nj = (__reduce_max_sync(kFull, ok ? cnt : 0) + 7) / 8;  // candidates per lane used
  float qx[kPer], qy[kPer], q2[kPer];
  unsigned near_q = 0xffffffffu;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int k = l + 8 * j;
    const int q = ok && k < cnt ? sc.cand[g][k] : 0;
    qx[j] = (float)pdx(q), qy[j] = (float)pdy(q);
    q2[j] = qx[j] * qx[j] + qy[j] * qy[j];
    if (q) near_q = min(near_q, ((unsigned)q2[j] << 5) | (unsigned)k);
  }
#pragma unroll
  for (int i = 4; i > 0; i >>= 1) near_q = min(near_q, __shfl_xor_sync(kFull, near_q, i));
  const int u0 = ok ? sc.cand[g][near_q & 31u] : 0;  // the nearest: a neighbour
  int u = u0, m = 1;
  if (l == 0) sc.star[g][0] = u0;
  bool act = ok;
  const long long hp = hkey(n, sx, sy);
  while (__any_sync(kFull, act)) {
    const float ux = (float)pdx(u), uy = (float)pdy(u);
    float k[kPer], kmin = INFINITY;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      k[j] = INFINITY;
      if (j < nj) {
        const float c = ux * qy[j] - uy * qx[j];
        const float d = q2[j] - (ux * qx[j] + uy * qy[j]);
        if (c > 0.f) k[j] = __fdividef(d, c);
        kmin = fminf(kmin, k[j]);
      }
    }
#pragma unroll
    for (int i = 4; i > 0; i >>= 1) kmin = fminf(kmin, __shfl_xor_sync(kFull, kmin, i));
    const float t = kmin + fabsf(kmin) * 0x1p-17f;
    unsigned cand = 0;  // bit 8 j + lane: candidates within the error of the smallest
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (j < nj) cand |= ((__ballot_sync(kFull, k[j] <= t) >> (8 * g)) & 0xffu) << (8 * j);
    if (!(kmin < INFINITY)) {  // an open gap
      if (act) ok = false;
      act = false;
    }
    if (act) {
      const int first = __ffs(cand) - 1;
      cand &= cand - 1u;
      int best = sc.cand[g][first];
      while (cand) {  // co-circular, or nearly
        const int c = sc.cand[g][__ffs(cand) - 1];
        cand &= cand - 1u;
        if (in_circle(pdx(u), pdy(u), pdx(best), pdy(best), pdx(c), pdy(c), hp,
                      hkey(n, sx + pdx(u), sy + pdy(u)), hkey(n, sx + pdx(best), sy + pdy(best)),
                      hkey(n, sx + pdx(c), sy + pdy(c))))
          best = c;
      }
      if (best == u0) {
        act = false;
      } else if (m == kQuadStar) {
        ok = act = false;
      } else {
        if (l == 0) sc.star[g][m] = best;
        ++m;
        u = best;
      }
    }
    __syncwarp();
  }
  // certificate, and where the angular order starts
  const unsigned gm = 0xffu << (8 * g);
  bool bad = false;
  int rot = 0;
#pragma unroll
  for (int h = 0; h < kQuadStar / 8; ++h) {
    const int k = l + 8 * h;
    bool lead = false;
    if (ok && k < m) {
      const int a = sc.star[g][k], p = sc.star[g][k ? k - 1 : m - 1],
                w = sc.star[g][k + 1 < m ? k + 1 : 0];
      bad = bad || !disc_surely_in(pdx(a), pdy(a), pdx(w), pdy(w), sx, sy, x0, x1, y0, y1, n);
      const int ha = half_of(pdx(a), pdy(a)), hq = half_of(pdx(p), pdy(p));
      lead = ha < hq || (ha == hq && pdx(a) * pdy(p) - pdy(a) * pdx(p) > 0);
    }
    const unsigned lm = __ballot_sync(kFull, lead) & gm;
    if (lm) rot = 8 * h + __ffs(lm >> (8 * g)) - 1;
  }
  if (__ballot_sync(kFull, bad) & gm) ok = false;
  int xm = 0;
  if (ok && l == 0) xm = site_index(bits, fixed, n, out.coloff, out.colpre, sx, sy);
  xm = __shfl_sync(kFull, xm, 0, 8);
  int own = 0;
#pragma unroll
  for (int h = 0; h < kQuadStar / 8; ++h) {
    const int k = l + 8 * h;
    bool mine = false;
    if (ok && k < m) {
      int i = k + rot;
      if (i >= m) i -= m;
      const int a = sc.star[g][i], w = sc.star[g][i + 1 < m ? i + 1 : 0];
      out.stars[(size_t)xm * kStar + k] = a;
      mine = owns_tri(sx, sy, a, w);
    }
    own += __popc(__ballot_sync(kFull, mine) & gm);
  }
  if (ok && l == 0) {
    out.sitepos[xm] = epos;
    out.degree[xm] = m;
    out.tcount[xm] = own;
  }
  const unsigned left = __ballot_sync(kFull, on && !ok && l == 0);
  __syncwarp();
  return (left & 1u) | ((left >> 7) & 2u) | ((left >> 14) & 4u) | ((left >> 21) & 8u);
}

// The stars of the sites in tile order: a warp per site for the nedge sites
// of edge tiles (their stars reach far) and crowded ones, four sites per warp for the
// others.
__global__ void __launch_bounds__(32 * kWarpsPerBlock, 5)
    k_dt_star(const uint64_t *__restrict__ bits, const uint64_t *__restrict__ fixed, int n,
              int nsites, int nedge, Pyr py, TileSites ts, StarOut out) {
  __shared__ union {
    unsigned front[kFrontier];
    QuadScratch quad;
  } s_warp[kWarpsPerBlock];
  const int t = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  auto &sw = s_warp[threadIdx.x >> 5];
  if (t < nedge) {
    full_site<false>(bits, fixed, n, ts.order[t], py, ts, sw.front, out);
    return;
  }
  const int t0 = nedge + 4 * (t - nedge);
  if (t0 >= nsites) return;  // the whole warp
  unsigned left = quad_stars(bits, fixed, n, t0, nsites, py, ts, sw.quad, out);
  for (; left; left &= left - 1u)
    full_site<false>(bits, fixed, n, ts.order[t0 + __ffs(left) - 1], py, ts, sw.front, out);
}

// The sites whose star overflowed (no neighbours), ring by ring.  (In k_dt_star this
// path would cost every launch 2 %: registers spilled.)
__global__ void __launch_bounds__(32 * kWarpsPerBlock)
    k_dt_rings(const uint64_t *__restrict__ bits, const uint64_t *__restrict__ fixed, int n,
               int nsites, Pyr py, TileSites ts, StarOut out) {
  __shared__ unsigned s_front[kWarpsPerBlock][kFrontier];
  const int t = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (t >= nsites || out.degree[t]) return;  // the whole warp
  full_site<true>(bits, fixed, n, out.sitepos[t], py, ts, s_front[threadIdx.x >> 5], out);
}

__global__ void k_dt_emit(const uint64_t *__restrict__ bits, const uint64_t *__restrict__ fixed,
                          int n, const int *__restrict__ sitepos, int nsites,
                          const unsigned *__restrict__ coloff, const unsigned *__restrict__ colpre,
                          const int *__restrict__ stars, const int *__restrict__ degree,
                          const unsigned *__restrict__ toff, int *tris, unsigned cap) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nsites) return;
  const int sx = pdx(sitepos[t]) & 0xffff, sy = pdy(sitepos[t]);
  const int m = degree[t];
  unsigned pos = toff[t];
  for (int k = 0; k < m; ++k) {
    const int u = stars[(size_t)t * kStar + k], w = stars[(size_t)t * kStar + (k + 1) % m];
    if (m < 2 || open_gap(pdx(u), pdy(u), pdx(w), pdy(w))) continue;
    const int ux = sx + pdx(u), uy = sy + pdy(u), wx = sx + pdx(w), wy = sy + pdy(w);
    const bool first = (sx < ux || (sx == ux && sy < uy)) && (sx < wx || (sx == wx && sy < wy));
    if (!first) continue;
    if (pos < cap) {
      tris[3 * (size_t)pos] = t;
      tris[3 * (size_t)pos + 1] = site_index(bits, fixed, n, coloff, colpre, ux, uy);
      tris[3 * (size_t)pos + 2] = site_index(bits, fixed, n, coloff, colpre, wx, wy);
    }
    ++pos;
  }
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

#define DCK(call)                                 \
  do {                                            \
    if ((call) != cudaSuccess) return GCVT_ERR_CUDA; \
  } while (0)

int scan(const unsigned *count, int n, unsigned *offset, Scratch &sc, cudaStream_t s) {
  return scan_counts(reinterpret_cast<const int *>(count), n, reinterpret_cast<int *>(offset),
                     nullptr, sc, s);
}

}  // namespace

// The Delaunay triangles of the free sites of `bits` (n x n, n a multiple of
// 64), as indices into delaunayInput's point order; host-synchronous on `s`.
int delaunay_sites(const uint64_t *bits, const uint64_t *fixed, int n, int *tris, unsigned cap,
                   unsigned *ntris, cudaStream_t s) {
  Scratch sc(s);
  return delaunay_sites_in(bits, fixed, n, tris, cap, ntris, s, sc);
}

// The same with the caller's scratch (a caller that holds one already: the
// device's scratch lock is not taken twice).
int delaunay_sites_in(const uint64_t *bits, const uint64_t *fixed, int n, int *tris,
                      unsigned cap, unsigned *ntris, cudaStream_t s, Scratch &sc) {
  *ntris = 0;
  if (n <= 0 || n % kBand) return GCVT_ERR_ARGUMENT;
  const size_t nb = (size_t)(n / kBand) * n;
  const int nt0 = n / kTile, ntiles = nt0 * nt0;
  unsigned *colpre = sc.take<unsigned>(nb), *colcnt = sc.take<unsigned>(n),
           *coloff = sc.take<unsigned>(n + 1),
           *tilecnt = sc.take<unsigned>(ntiles), *ccnt = sc.take<unsigned>(3 * (size_t)ntiles),
           *tileoff = sc.take<unsigned>(3 * (size_t)ntiles + 1);
  uint8_t *cls = sc.take<uint8_t>(ntiles);
  int *err = sc.take<int>(1);
  Pyr py{};
  size_t occ_bytes = 0;
  for (int l = 0, t = nt0;; ++l, t = (t + 1) / 2) {
    if (l >= kLevels) return GCVT_ERR_ARGUMENT;
    py.off[l] = (int)occ_bytes;
    py.nt[l] = t;
    occ_bytes += (size_t)t * t;
    if (t == 1) {
      py.top = l;
      break;
    }
  }
  uint8_t *occ = sc.take<uint8_t>(occ_bytes);
  py.occ = occ;
  if (!colpre || !colcnt || !coloff || !tilecnt || !ccnt || !tileoff || !cls || !err ||
      !occ)
    return GCVT_ERR_ALLOC;
  DCK(cudaMemsetAsync(err, 0, sizeof(int), s));
  DCK(cudaMemsetAsync(occ, 0, occ_bytes, s));
  DCK(cudaMemsetAsync(tilecnt, 0, (size_t)ntiles * sizeof(unsigned), s));
  k_dt_columns<<<nblk(n, 64), 64, 0, s>>>(bits, fixed, n, colpre, colcnt);
  DCK(cudaGetLastError());
  k_dt_tiles<<<nblk((long long)nb, 256), 256, 0, s>>>(bits, fixed, n, occ, nt0, tilecnt);
  DCK(cudaGetLastError());
  for (int l = 1; l <= py.top; ++l) {
    k_dt_up<<<nblk((long long)py.nt[l] * py.nt[l], 256), 256, 0, s>>>(
        occ + py.off[l - 1], py.nt[l - 1], occ + py.off[l], py.nt[l]);
    DCK(cudaGetLastError());
  }
  int rc = scan(colcnt, n, coloff, sc, s);
  if (rc) return rc;
  k_dt_class<<<nblk(ntiles, 256), 256, 0, s>>>(occ, nt0, tilecnt, ccnt, cls);
  DCK(cudaGetLastError());
  if ((rc = scan(ccnt, 3 * ntiles, tileoff, sc, s))) return rc;
  unsigned nsites_u = 0, nedge_u = 0;
  DCK(cudaMemcpyAsync(&nsites_u, coloff + n, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  DCK(cudaMemcpyAsync(&nedge_u, tileoff + 2 * ntiles, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  DCK(cudaStreamSynchronize(s));
  
  const int nsites = (int)nsites_u, nedge = (int)nedge_u;
  if (nsites < 3) return GCVT_OK;
  int *order = sc.take<int>(nsites), *sitepos = sc.take<int>(nsites),
      *stars = sc.take<int>((size_t)nsites * kStar), *degree = sc.take<int>(nsites);
  unsigned *tcnt = sc.take<unsigned>(nsites), *toff = sc.take<unsigned>(nsites + 1);
  if (!order || !sitepos || !stars || !degree || !tcnt || !toff) return GCVT_ERR_ALLOC;
  k_dt_order<<<nblk(ntiles, 128), 128, 0, s>>>(bits, fixed, n, nt0, tileoff, cls, order);
  DCK(cudaGetLastError());
  const TileSites ts{order, tileoff, tilecnt, cls};
  const StarOut out{coloff, colpre, sitepos, stars, degree, tcnt, err};
  const long long warps = nedge + (nsites - nedge + 3ll) / 4;
  k_dt_star<<<nblk(warps, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, s>>>(
      bits, fixed, n, nsites, nedge, py, ts, out);
  DCK(cudaGetLastError());
  unsigned h[2] = {0, 0};
  for (int k = 0; k < 2; ++k) {
    if (k) {
      DCK(cudaMemsetAsync(err, 0, sizeof(int), s));
      k_dt_rings<<<nblk(nsites, kWarpsPerBlock), 32 * kWarpsPerBlock, 0, s>>>(
          bits, fixed, n, nsites, py, ts, out);
      DCK(cudaGetLastError());
    }
    if ((rc = scan(tcnt, nsites, toff, sc, s))) return rc;
    if (tris && cap) {
      k_dt_emit<<<nblk(nsites, 128), 128, 0, s>>>(bits, fixed, n, sitepos, nsites, coloff, colpre,
                                                  stars, degree, toff, tris, cap);
      DCK(cudaGetLastError());
    }
    DCK(cudaMemcpyAsync(&h[0], toff + nsites, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    DCK(cudaMemcpyAsync(&h[1], err, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    DCK(cudaStreamSynchronize(s));
    if (!h[1]) break;  // else the stars that overflowed once more
  }
  if (h[1]) return GCVT_ERR_INPUT;
  *ntris = h[0];
  return GCVT_OK;
}

}  // namespace cvtgb
