// cells.cu -- one Lloyd iteration: k_list lays the current sites out in bitmap
// order, then k_cell (k_cell_warp for fewer sites) lets every site compute its own
// Voronoi cell exactly, sum the density moments over it, and move; up to 8192
// sites both in one launch (k_cell_few).
//
// In a Lloyd iteration the labels themselves are never needed, only each
// site's sums over its cell (gcvt.cu:1008-1023) and the energy
// (gcvt.cu:1059-1083).  The PBA+ labelling (labeller.cu) is a total order per
// pixel -- nearest site, then smaller x, then the 64-row band rule for a mirror
// pair -- so "pixel p belongs to site s" is "s beats every other site t at p".
// In coordinates relative to s (p = s + (u, v), t = s + (A, B)):
//     |p - s|^2 - |p - t|^2 = 2Au + 2Bv - (A^2 + B^2)
//     A > 0 (t right of s, s wins ties):   u <= floor(N / 2A)
//     A < 0 (t left of s, t wins ties):    u >= floor(N / 2A) + 1
//     A = 0 (same column): row v is s's iff B (2v - B) < 0, or = 0 and the
//                          band rule picks s,
// with N = A^2 + B^2 - 2Bv, exact in 32-bit integers.  The cell is the
// intersection, one interval per row.
//
// Candidates t come from the site bitmap in the disc of radius W around s.
// Certificate: if every summed pixel lies within R of s and 2R <= W, no site
// outside the disc can beat s there (|p - t| > W - R >= R); otherwise the
// window grows (W <- min(2R + 1, 2W)) and the cell is redone; a window
// covering the grid is exact by construction.  The starting W of a site is
// the hint at its pixel: 2R + slack of the cell the site that moved there
// had, or, after a load, of its own cell in the level start's label grid
// (k_cover).
//
// Rows are visited outward from s.  A row may hold no pixel of the cell while
// a row further out does (a sliver narrower than a pixel), so the walk ends
// only when lo > hi + 1: then the largest lower cut is at least lo - 1 >= hi + 1,
// above the smallest upper cut (< hi + 1), so the real chord of the convex
// cell is empty, and so is every chord further from s.
//
// Covering bound.  A cell at the domain boundary is open towards the empty
// region, so its row walk alone would cross the whole grid.  Every density
// pixel p lies within `cover` of its owner (DevState::cover), so only pixels
// with |p - s| <= cover can be s's: the walk stays in that disc and the
// window never needs to exceed 2 cover.  The bound carries itself from one
// iteration to the next: if the pixel p was within R of its owner s and s
// moved by d, p is within R + d of the site now at s's new pixel (a merged
// site leaves another at that pixel), so cover' = ceil(sqrt(max R^2)) +
// ceil(sqrt(max d^2)), both maxima taken over this iteration's cells.  The
// first iteration of a level takes it from a label grid (k_cover).
//
// Work split.  k_cell runs one warp per block, as many blocks as fit on the
// GPU; each warp takes the next group of 32 listed sites from a ticket, one
// site per lane.  A lane keeps its site's candidates as two bytes each, bounds
// seven rows per pass over them in floats (cell_float: exact where float_walk
// says so, else cell_general's integer division), lists the rows and sums
// their pixels two rows at a time in packed FP32.  What bounds it: issue slots
// and the latency of L1 misses, not bandwidth (60 MB an iteration).  Against
// integer bounds row pair by row pair and scalar sums: 118 -> 81 us an
// iteration at 4096^2 / 262,144 sites (75.5 -> 45.1 M warp instructions), 0.42
// -> 0.26 ms at 8192^2.  Records of 8 bytes in shared memory (4 KB a warp) took
// 120 us: they leave the density rows too little L1.  The energy is reduced in a fixed order
// whatever warp takes which group: the sites of a group by a butterfly, 64
// groups by the warp finishing the last of them, the 64-group totals by the
// warp finishing the last 64-group; that warp also runs the schedule.  Sites move by atomicOr into the next bitmap;
// the first to set a bit also counts it for the next k_list.
#include "gcvt_internal.cuh"

#include <cstddef>

namespace cvtgb {

constexpr int kMaxCand = 64;  // candidate records per site; more: streamed
constexpr int kGroupsPerSlot = 64;

__device__ __forceinline__ void tsum_c(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  float bp = __fsub_rn(s, a);
  float ap = __fsub_rn(s, bp);
  e = __fadd_rn(__fsub_rn(a, ap), __fsub_rn(b, bp));
}

// (ah, al) += (bh, bl), two-float.  Commutative: the error term of TwoSum is
// exact, so both lanes of a butterfly get the same result.
__device__ __forceinline__ void dfa(float &ah, float &al, float bh, float bl) {
  float s, e;
  tsum_c(ah, bh, s, e);
  e = __fadd_rn(e, __fadd_rn(al, bl));
  ah = __fadd_rn(s, e);
  al = __fsub_rn(e, __fsub_rn(ah, s));
}

// (ah, al) += k * (bh, bl) for a small integer k (exact product via fma).
__device__ __forceinline__ void dfa_scaled(float &ah, float &al, float k, float bh, float bl) {
  const float ph = __fmul_rn(k, bh);
  const float pl = __fmaf_rn(k, bh, -ph) + k * bl;
  dfa(ah, al, ph, pl);
}

// Two floats in one 64-bit register: the packed FP32 instructions of sm_100+
// do both halves in one issue slot, each half rounded as the scalar
// instruction rounds it.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float f2_lo(F2 a) {
  float x;
  asm("mov.b64 {%0, _}, %1;" : "=f"(x) : "l"(a.v));
  return x;
}
__device__ __forceinline__ float f2_hi(F2 a) {
  float y;
  asm("mov.b64 {_, %0}, %1;" : "=f"(y) : "l"(a.v));
  return y;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// a - b: the product b * -1 is exact, so the sum is rounded once
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, f2(-1.f, -1.f), a); }

// dfa on both halves: (ah, al) += (bh, bl).
__device__ __forceinline__ void dfa2(F2 &ah, F2 &al, F2 bh, F2 bl) {
  const F2 s = add2(ah, bh), bp = sub2(s, ah), ap = sub2(s, bp);
  F2 e = add2(sub2(ah, ap), sub2(bh, bp));
  e = add2(e, add2(al, bl));
  ah = add2(s, e);
  al = sub2(e, sub2(ah, s));
}
// the same with bl = 0
__device__ __forceinline__ void dfa2_0(F2 &ah, F2 &al, F2 bh) {
  const F2 s = add2(ah, bh), bp = sub2(s, ah), ap = sub2(s, bp);
  F2 e = add2(sub2(ah, ap), sub2(bh, bp));
  e = add2(e, al);
  ah = add2(s, e);
  al = sub2(e, sub2(ah, s));
}

// floor(sqrt(v)) and ceil(sqrt(v)) for 0 <= v < 2^30, exact.
__device__ __forceinline__ int isqrt_floor(int v) {
  int h = (int)sqrtf((float)v);
  while (h * h > v) --h;
  while ((h + 1) * (h + 1) <= v) ++h;
  return h;
}
__device__ __forceinline__ int isqrt_ceil(int v) {
  const int h = isqrt_floor(v);
  return h * h == v ? h : h + 1;
}

// floor(N / D) for D > 0, exact, by integer division.
__device__ __forceinline__ int floordiv(int N, int D) {
  int q = N / D;
  if ((N % D != 0) && (N < 0)) --q;
  return q;
}

// Row-v bounds from the site t = s + (A, B), A != 0, when the candidates do
// not fit the record list (same-column sites are already row limits).
__device__ __forceinline__ void constrain_rel(int A, int B, int v, int &lo, int &hi) {
  if (A == 0) return;
  const int N = A * A + B * B - 2 * B * v;
  if (A > 0) hi = min(hi, floordiv(N, 2 * A));
  else lo = max(lo, floordiv(-N, -2 * A) + 1);
}

__device__ __forceinline__ uint64_t row_mask(int lo_i, int hi_i) {  // bits lo_i..hi_i
  const uint64_t up = hi_i >= 63 ? ~0ull : ((2ull << hi_i) - 1ull);
  return up & ~((1ull << lo_i) - 1ull);
}

struct CellSums {
  float wh, wl, xh, xl, yh, yl, eh, el;  // W, SX, SY (relative to the site), E
  int r2;                                // max |p - s|^2 over the summed pixels
};

// floor(N / D), D > 0, |N| < 2^23, given r ~ 1/D from rcp.approx (at most 1
// ulp off): the estimate is within 1, one exact correction fixes it.
__device__ __forceinline__ int floordiv_r(int N, int D, float r) {
  int q = __float2int_rd(__fmul_rn((float)N, r));
  const int rem = N - q * D;
  q += (rem >= D) - (rem < 0);
  return q;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Bounds of rows v0 and v0 + dir (relative to s) in one pass over the
// records.  A record {K, S | D << 16} bounds row v by floor((K - S v) / |D|):
// an upper bound when D > 0, a lower one (+1) when D < 0.  When the records
// did not hold every candidate, the candidates are read from the bitmap.
struct RowPair {
  int lo0, hi0, lo1, hi1;
};

__device__ __forceinline__ RowPair row_bounds2(const int2 *rec, int cnt, bool ovf, bool fast,
                                               const uint64_t *__restrict__ bits, int n, int sx,
                                               int sy, int x0, int x1, int b0, int b1, int y0,
                                               int y1, long long Wc, int v0, int dir) {
  RowPair p{-sx, n - 1 - sx, -sx, n - 1 - sx};
  const int v1 = v0 + dir;
  if (!ovf) {
    for (int k = 0; k < cnt; ++k) {
      const int2 r = rec[k];
      const int S = (int)(int16_t)((unsigned)r.y & 0xffffu);
      const int D = (int)(int16_t)((unsigned)r.y >> 16);
      const int aD = abs(D);
      const int N0 = r.x - S * v0, N1 = N0 - S * dir;
      int q0, q1;
      if (fast) {
        const float rr = rcp_approx((float)aD);
        q0 = floordiv_r(N0, aD, rr);
        q1 = floordiv_r(N1, aD, rr);
      } else {
        q0 = floordiv(N0, aD);
        q1 = floordiv(N1, aD);
      }
      if (D > 0) {
        p.hi0 = min(p.hi0, q0);
        p.hi1 = min(p.hi1, q1);
      } else {
        p.lo0 = max(p.lo0, q0 + 1);
        p.lo1 = max(p.lo1, q1 + 1);
      }
    }
    return p;
  }
  for (int x = x0; x <= x1; ++x)
    for (int b = b0; b <= b1; ++b) {
      uint64_t w = __ldg(bits + (size_t)b * n + x) &
                   row_mask(max(y0 - 64 * b, 0), min(y1 - 64 * b, 63));
      while (w) {
        const int i = __ffsll((long long)w) - 1;
        w &= w - 1ull;
        const int A = x - sx, B = 64 * b + i - sy;
        const int K = A * A + B * B;
        if (K == 0 || (long long)K > Wc) continue;
        constrain_rel(A, B, v0, p.lo0, p.hi0);
        constrain_rel(A, B, v1, p.lo1, p.hi1);
      }
    }
  return p;
}

// FP32 sums of one chunk [u0, u1] (at most 16 pixels) of a row: density,
// x-moment and x^2-moment relative to the site.
__device__ __forceinline__ void chunk_sums(const float *__restrict__ row, int u0, int u1,
                                           float &rw, float &rx, float &rq) {
  rw = 0.f, rx = 0.f, rq = 0.f;
  float dx = (float)u0;
#pragma unroll 4
  for (int u = u0; u <= u1; ++u) {
    const float rho = __ldg(row + u);
    const float t = __fmul_rn(dx, rho);
    rw = __fadd_rn(rw, rho);
    rx = __fadd_rn(rx, t);
    rq = __fmaf_rn(t, dx, rq);
    dx = __fadd_rn(dx, 1.0f);
  }
}

// A chunk of row v (fv = v, fv2 = v^2) folded into the two-float cell sums.
__device__ __forceinline__ void fold_chunk(CellSums &c, float rw, float rx, float rq, float fv,
                                           float fv2) {
  dfa(c.wh, c.wl, rw, 0.f);
  dfa(c.xh, c.xl, rx, 0.f);
  dfa_scaled(c.yh, c.yl, fv, rw, 0.f);
  float qh = rq, ql = 0.f;
  dfa_scaled(qh, ql, fv2, rw, 0.f);
  dfa(c.eh, c.el, qh, ql);
}

// Sums of row v = [da, db] (relative columns) into c: FP32 over chunks of at
// most 16 pixels (relative error below 16 ulp of the chunk), chunks folded
// into the two-float cell sums.
__device__ __forceinline__ void row_sums(const float *__restrict__ row, int da, int db, int v,
                                         CellSums &c) {
  const float fv = (float)v, fv2 = (float)(v * v);
  for (int u0 = da; u0 <= db; u0 += 16) {
    float rw, rx, rq;
    chunk_sums(row, u0, min(db, u0 + 15), rw, rx, rq);
    fold_chunk(c, rw, rx, rq, fv, fv2);
  }
}

// The pixels [da, db] of row v the cell with bounds [lo, hi] sums: clipped to
// the density support and the covering disc; false when none.
__device__ __forceinline__ bool row_span(const int2 *__restrict__ support, int sx, int sy, int rb2,
                                         int v, int lo, int hi, int &da, int &db) {
  const int2 s = __ldg(support + sy + v);
  da = max(lo, s.x - sx), db = min(hi, s.y - 1 - sx);
  if (da > db) return false;
  if (max(da * da, db * db) + v * v > rb2) {  // clip to the covering disc
    const int hx = isqrt_floor(rb2 - v * v);
    da = max(da, -hx);
    db = min(db, hx);
    if (da > db) return false;
  }
  return true;
}

// Row v of the cell with bounds [lo, hi]: its span, R2, its sums.
__device__ __forceinline__ void take_row(const float *__restrict__ density,
                                         const int2 *__restrict__ support, int n, int sx, int sy,
                                         int rb2, int v, int lo, int hi, int &R2, CellSums &c) {
  int da, db;
  if (!row_span(support, sx, sy, rb2, v, lo, hi, da, db)) return;
  R2 = max(R2, max(da * da, db * db) + v * v);
  row_sums(density + (size_t)(sy + v) * n + sx, da, db, v, c);
}

// A site in s's own column at row offset B != 0: s keeps the rows strictly on
// its side of the mirror row, and the mirror row (B even) if the band rule
// says so.
__device__ __forceinline__ void same_column_limit(int B, int sy, int &vmin, int &vmax) {
  if (B > 0) {
    int m = (B - 1) >> 1;
    if (!(B & 1) && (((sy + B) >> 6) != ((sy + B / 2) >> 6))) m = B / 2;
    vmax = min(vmax, m);
  } else {
    int m = -((-B - 1) >> 1);
    if (!(B & 1) && ((sy >> 6) == ((sy + B / 2) >> 6))) m = B / 2;
    vmin = max(vmin, m);
  }
}

// The record {K, S | D << 16} of candidate t = s + (A, B), A != 0, K = A^2 + B^2
// (|S|, |D| <= 2 (n - 1) fit 16 bits).
__device__ __forceinline__ int2 make_rec(int A, int B, int K) {
  const int S = A > 0 ? 2 * B : -2 * B;
  return make_int2(A > 0 ? K : -K, (int)(((unsigned)S & 0xffffu) | ((unsigned)(2 * A) << 16)));
}

// The sites of one bitmap word (column offset A, bit i at row offset B0 + i)
// as candidates of s: a record each, or a row limit for a site in s's column.
__device__ __forceinline__ void gather_word(uint64_t w, int A, int B0, int sy, long long Wc,
                                            int2 *rec, int &cnt, bool &ovf, int &vmin,
                                            int &vmax) {
  while (w) {
    const int i = __ffsll((long long)w) - 1;
    w &= w - 1ull;
    const int B = B0 + i;
    const int K = A * A + B * B;
    if (K == 0 || (long long)K > Wc) continue;  // s itself; outside the disc
    if (A == 0) {
      same_column_limit(B, sy, vmin, vmax);
      continue;
    }
    if (cnt >= kMaxCand) {
      ovf = true;
      continue;
    }
    rec[cnt++] = make_rec(A, B, K);
  }
}

// The float accumulators of a cell, packed: (W, SX) and (SY, E), two-float.
struct CellAcc {
  F2 wxh, wxl, yeh, yel;
};

// fold_chunk on the packed accumulators: the same operations in the same
// order, two of the four sums per instruction (34 instructions instead of 56).
__device__ __forceinline__ void fold_chunk2(CellAcc &c, float rw, float rx, float rq, float fv,
                                            float fv2) {
  dfa2_0(c.wxh, c.wxl, f2(rw, rx));
  const F2 rr = f2(rw, rw), k = f2(fv, fv2);
  const F2 nph = mul2(f2(-fv, -fv2), rr);  // -(v rw, v^2 rw)
  const F2 pl = fma2(k, rr, nph);
  const float ph = -f2_hi(nph);
  float s, e;  // (rq, 0) += (ph, pl)
  tsum_c(rq, ph, s, e);
  e = __fadd_rn(e, f2_hi(pl));
  const float qh = __fadd_rn(s, e);
  const float ql = __fsub_rn(e, __fsub_rn(qh, s));
  dfa2(c.yeh, c.yel, f2(-f2_lo(nph), qh), f2(f2_lo(pl), ql));
}

// The pixels of a row span as bits from its first aligned column, and that
// column; an empty span has no bits.
struct RowPix {
  const float *p;  // the density at the first aligned column
  unsigned m;
  float dx;        // that column relative to the site
};

// chunk_sums of two rows at once (at most 16 pixels each): aligned 16-byte
// loads, the first eight columns of both rows in flight together, the two rows
// in the two halves of the packed instructions.  Pixels outside a span add
// +-0, which changes no sum.
__device__ __forceinline__ void pair_sums(const RowPix &a, const RowPix &b, F2 &rw, F2 &rx,
                                          F2 &rq) {
  const F2 one = f2(1.f, 1.f);
  F2 dx = f2(a.dx, b.dx);
  rw = rx = rq = f2(0.f, 0.f);
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 *pa = reinterpret_cast<const float4 *>(a.p);
  const float4 *pb = reinterpret_cast<const float4 *>(b.p);
  unsigned ma = a.m, mb = b.m;
  float4 qa = ma ? __ldg(pa) : z, qb = mb ? __ldg(pb) : z;
  float4 na = ma >> 4 ? __ldg(pa + 1) : z, nb = mb >> 4 ? __ldg(pb + 1) : z;
  for (int k = 2;; ++k) {
    const float va[4] = {qa.x, qa.y, qa.z, qa.w}, vb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const F2 p = f2((ma >> j) & 1u ? va[j] : 0.f, (mb >> j) & 1u ? vb[j] : 0.f);
      const F2 t = mul2(dx, p);
      rw = add2(rw, p);
      rx = add2(rx, t);
      rq = fma2(t, dx, rq);
      dx = add2(dx, one);
    }
    ma >>= 4;
    mb >>= 4;
    if (!(ma | mb)) break;
    qa = na;
    qb = nb;
    na = ma >> 4 ? __ldg(pa + k) : z;
    nb = mb >> 4 ? __ldg(pb + k) : z;
  }
}

// One attempt at the cell with the window radius W, general form: candidates
// as integer records (or straight from the bitmap when they do not fit),
// bounds by exact integer division.  Returns the cell's sums; c.r2 = max
// |p - s|^2.
__device__ __noinline__ CellSums cell_general(const float *__restrict__ density,
                                              const int2 *__restrict__ support,
                                              const uint64_t *__restrict__ bits, int n, int sx,
                                              int sy, int W, int rb, int vmin, int vmax) {
  int2 rec[kMaxCand];  // {K, S | D << 16} of the window's candidates
  const int rb2 = rb * rb;
  const int x0 = max(0, sx - W), x1 = min(n - 1, sx + W);
  const int y0 = max(0, sy - W), y1 = min(n - 1, sy + W);
  const bool whole = x0 == 0 && y0 == 0 && x1 == n - 1 && y1 == n - 1;
  const int b0 = y0 >> 6, b1 = y1 >> 6;
  const long long W2 = (long long)W * W;
  // candidates: the disc of radius W, or every site when the window holds
  // the grid (no certificate needed then)
  const long long Wc = whole ? (1ll << 62) : W2;
  int cnt = 0;
  bool ovf = false;
  for (int x = x0; x <= x1; ++x)
    for (int b = b0; b <= b1; ++b)
      gather_word(__ldg(bits + (size_t)b * n + x) &
                      row_mask(max(y0 - 64 * b, 0), min(y1 - 64 * b, 63)),
                  x - sx, 64 * b - sy, sy, Wc, rec, cnt, ovf, vmin, vmax);
  // |K - S v| <= 2 W^2 + 2 W rb: below 2^23 the reciprocal estimate is safe
  const bool fast = 2 * W2 + 2 * (long long)W * rb < (1ll << 23);
  CellSums c{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0};
  int R2 = 0;
  // rows outward from s, two per pass over the records: up from v = 0, down
  // from v = -1, inside the row limits
  for (int dir = 1; dir >= -1; dir -= 2) {
    const int vend = dir > 0 ? vmax : vmin;
    for (int v = dir > 0 ? max(0, vmin) : min(-1, vmax); dir > 0 ? v <= vend : v >= vend;
         v += 2 * dir) {
      const RowPair p =
          row_bounds2(rec, cnt, ovf, fast, bits, n, sx, sy, x0, x1, b0, b1, y0, y1, Wc, v, dir);
      if (p.lo0 > p.hi0 + 1) break;  // the cell has ended in this direction
      if (p.lo0 <= p.hi0) take_row(density, support, n, sx, sy, rb2, v, p.lo0, p.hi0, R2, c);
      const int v1 = v + dir;
      if ((dir > 0 ? v1 > vend : v1 < vend) || p.lo1 > p.hi1 + 1) break;
      if (p.lo1 <= p.hi1) take_row(density, support, n, sx, sy, rb2, v1, p.lo1, p.hi1, R2, c);
    }
  }
  c.r2 = R2;
  return c;
}

// Where the float walk below is exact: W^2 (W + 2 rb) < 1.25 2^20.  A candidate
// (A, B) bounds row v by floor(t) (+ 1 for a lower bound), t = (K - 2 B v) / 2A,
// computed as k + s v with k = K / 2A and s = -B / A rounded (r ~ 1/A within an
// ulp scales both alike).  Its error, the row steps and the final sum included,
// is below 6 2^-24 (|k| + |s v|) <= 6 2^-24 (W^2 / 2 + W rb) < 1 / 4W there, and t
// is a multiple of 1 / 2|A| >= 1 / 2W, so floor(t) = floor(t~ + 1 / 4W) -- for
// every record alike, so the smallest (largest) t~ of a row gives its bound
// with one floor.  (W <= 109 follows; rb <= 511 lets a row fit one word.)
__device__ __forceinline__ bool float_walk(int W, int rb) {
  return W <= 127 && rb <= 511 && W * W * (W + 2 * rb) < (5 << 18);
}

constexpr int kRowsPass = 7;   // rows bounded per pass over the records (6 and 8: 4 % slower)
constexpr int kRowList = 24;   // rows listed before their pixels are summed

// The float 128 + a byte minus 128 (no conversion instruction).
__device__ __forceinline__ float byte_val(uint32_t w, unsigned sel) {
  return __uint_as_float(__byte_perm(w, 0x4b000000u, sel)) - 8388736.0f;
}

// Record i (0 or 1) of a record word: bound k + s v.
__device__ __forceinline__ void rec_line(uint32_t w, int i, float &k, float &s) {
  const float A = byte_val(w, i ? 0x7442u : 0x7440u), B = byte_val(w, i ? 0x7443u : 0x7441u);
  const float r = rcp_approx(A);
  s = -B * r;
  k = __fmaf_rn(A, A, B * B) * (0.5f * r);
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// A listed row: v, first column da and last column db relative to the site.
__device__ __forceinline__ uint32_t pack_row(int v, int da, int db) {
  return (uint32_t)(v & 0x3ff) | ((uint32_t)(da & 0x7ff) << 10) | ((uint32_t)(db - da) << 21);
}

// One attempt at the cell with the window radius W where float_walk holds.
// False when the candidates do not fit (the caller takes cell_general).
// What lives per lane decides the speed: 32 warps share an SM's L1, which also
// holds the density rows, so a candidate is two bytes (A + 128, B + 128; its line is
// recomputed per pass) and a row one word.
__device__ __forceinline__ bool cell_float(const float *__restrict__ density,
                                           const int2 *__restrict__ support,
                                           const uint64_t *__restrict__ bits, int n, int sx, int sy,
                                           int W, int rb, int vmin, int vmax, CellSums &out) {
  uint32_t rec[kMaxCand / 2];  // two candidates a word: those left of s, then those right of it
  uint32_t rows[kRowList + kRowsPass];
  unsigned short *rec16 = reinterpret_cast<unsigned short *>(rec);
  const int rb2 = rb * rb, W2 = W * W;
  const int x0 = max(0, sx - W), x1 = min(n - 1, sx + W);
  const int y0 = max(0, sy - W), y1 = min(n - 1, sy + W);
  int cnt = 0, nl = 0;
  auto put = [&](int A, int B) {
    if (A * A + B * B > W2) return;
    if (cnt < kMaxCand) rec16[cnt] = (unsigned short)((A + 128) | ((B + 128) << 8));
    ++cnt;
  };
  auto even = [&]() {  // an odd list repeats its last record
    if ((cnt & 1) && cnt < kMaxCand) rec16[cnt] = rec16[cnt - 1];
    cnt += cnt & 1;
  };
  if (W <= 31) {
    // a column's window rows as one word of up to 63 bits, bit i = row y0 + i,
    // from two or three 32-row halves of the bitmap words
    const uint32_t *hw = reinterpret_cast<const uint32_t *>(bits);
    const int h0 = y0 >> 5, sh = y0 & 31, nr = y1 - y0 + 1;
    const int h1 = h0 + (sh + nr > 32), h2 = h1 + (sh + nr > 64);
    const uint32_t *p0 = hw + 2 * (size_t)(h0 >> 1) * n + (h0 & 1);
    const uint32_t *p1 = hw + 2 * (size_t)(h1 >> 1) * n + (h1 & 1);
    const uint32_t *p2 = hw + 2 * (size_t)(h2 >> 1) * n + (h2 & 1);
    const bool tall = nr > 32;
    const uint32_t mlo = nr >= 32 ? ~0u : (1u << nr) - 1u;
    const uint32_t mhi = tall ? (1u << (nr - 32)) - 1u : 0u;
    const int o = sy - y0;  // s's own bit
    uint32_t w0 = __ldg(p0 + 2 * x0), w1 = __ldg(p1 + 2 * x0), w2 = tall ? __ldg(p2 + 2 * x0) : 0u;
    for (int x = x0; x <= x1; ++x) {
      uint32_t lo = __funnelshift_r(w0, w1, sh) & mlo;
      uint32_t hi = tall ? __funnelshift_r(w1, w2, sh) & mhi : 0u;
      if (x < x1) {  // the next column's words in flight
        w0 = __ldg(p0 + 2 * x + 2);
        w1 = __ldg(p1 + 2 * x + 2);
        if (tall) w2 = __ldg(p2 + 2 * x + 2);
      }
      const int A = x - sx;
      if (A == 0) {
        // s's own column: the nearest site on each side limits the rows
        even();
        nl = cnt;
        const uint64_t col = (uint64_t)lo | ((uint64_t)hi << 32);
        const uint64_t up = (col >> o) >> 1, dn = col & ((1ull << o) - 1ull);
        if (up) same_column_limit(__ffsll((long long)up), sy, vmin, vmax);
        if (dn) same_column_limit(63 - __clzll((long long)dn) - o, sy, vmin, vmax);
        continue;
      }
      while (lo) {
        const int i = __ffs(lo) - 1;
        lo &= lo - 1u;
        put(A, i - o);
      }
      while (hi) {
        const int i = __ffs(hi) + 31;
        hi &= hi - 1u;
        put(A, i - o);
      }
    }
  } else {
    const int b0 = y0 >> 6, b1 = y1 >> 6;
    for (int x = x0; x <= x1; ++x) {
      const int A = x - sx;
      if (A == 0) {
        even();
        nl = cnt;
      }
      for (int b = b0; b <= b1; ++b) {
        uint64_t w = __ldg(bits + (size_t)b * n + x) &
                     row_mask(max(y0 - 64 * b, 0), min(y1 - 64 * b, 63));
        while (w) {
          const int i = __ffsll((long long)w) - 1;
          w &= w - 1ull;
          const int B = 64 * b + i - sy;
          if (A) put(A, B);
          else if (B) same_column_limit(B, sy, vmin, vmax);
        }
      }
    }
  }
  even();
  if (cnt > kMaxCand) return false;
  nl >>= 1;
  cnt >>= 1;
  const float eps = 0.25f / (float)W;
  const F2 z = f2(0.f, 0.f);
  CellAcc acc{z, z, z, z};
  int R2 = 0;
  // rows outward from s: up from v = 0, then down from v = -1, inside the row
  // limits, kRowsPass per pass over the records.  One loop for both
  // directions, and the rows are listed before they are summed: a lane whose
  // cell has ended upwards goes on downwards while its neighbours are still
  // going up.
  int dir = 1, v = max(0, vmin);
  bool done = false;
  do {
    int m = 0;
    do {
      if (dir > 0 && v > vmax) {
        dir = -1;
        v = min(-1, vmax);
      }
      if (dir < 0 && v < vmin) {
        done = true;
        break;
      }
      float lo[kRowsPass], hi[kRowsPass];
#pragma unroll
      for (int j = 0; j < kRowsPass; ++j) {
        lo[j] = (float)(-sx - 1);
        hi[j] = (float)(n - 1 - sx);
      }
      const float fv = (float)v, fd = (float)dir;
      for (int k = 0; k < nl; ++k) {
        const uint32_t w = rec[k];
        float k0, s0, k1, s1;
        rec_line(w, 0, k0, s0);
        rec_line(w, 1, k1, s1);
        k0 = __fmaf_rn(s0, fv, k0), k1 = __fmaf_rn(s1, fv, k1);
        s0 *= fd, s1 *= fd;
#pragma unroll
        for (int j = 0; j < kRowsPass; ++j)
          lo[j] = max3(lo[j], __fmaf_rn(s0, (float)j, k0), __fmaf_rn(s1, (float)j, k1));
      }
      for (int k = nl; k < cnt; ++k) {
        const uint32_t w = rec[k];
        float k0, s0, k1, s1;
        rec_line(w, 0, k0, s0);
        rec_line(w, 1, k1, s1);
        k0 = __fmaf_rn(s0, fv, k0), k1 = __fmaf_rn(s1, fv, k1);
        s0 *= fd, s1 *= fd;
#pragma unroll
        for (int j = 0; j < kRowsPass; ++j)
          hi[j] = min3(hi[j], __fmaf_rn(s0, (float)j, k0), __fmaf_rn(s1, (float)j, k1));
      }
      // the rows' spans until the row limit, or until the cell has ended in
      // this direction
      bool ended = false;
#pragma unroll
      for (int j = 0; j < kRowsPass; ++j) {
        const int vv = v + j * dir;
        const int2 sup = __ldg(support + min(max(sy + vv, 0), n - 1));
        const int l = __float2int_rd(lo[j] + eps) + 1, h = __float2int_rd(hi[j] + eps);
        ended = ended || l > h + 1 || (dir > 0 ? vv > vmax : vv < vmin);
        int da = max(l, sup.x - sx), db = min(h, sup.y - 1 - sx);
        if (!ended && da <= db) {
          int d2 = max(da * da, db * db) + vv * vv;
          if (d2 > rb2) {  // clip to the covering disc
            const int hx = isqrt_floor(rb2 - vv * vv);
            da = max(da, -hx);
            db = min(db, hx);
            d2 = max(da * da, db * db) + vv * vv;
          }
          if (da <= db) {
            R2 = max(R2, d2);
            rows[m++] = pack_row(vv, da, db);
          }
        }
      }
      if (ended) {
        done = dir < 0;
        dir = -1;
        v = min(-1, vmax);
      } else {
        v += kRowsPass * dir;
      }
    } while (!done && m <= kRowList);
    // the listed rows' pixels, two rows at a time
    for (int i = 0; i < m; i += 2) {
      const uint32_t wa = rows[i], wb = i + 1 < m ? rows[i + 1] : 0u;
      const int va = (int)(wa << 22) >> 22, vb = (int)(wb << 22) >> 22;
      const int da = sx + ((int)(wa << 11) >> 21), db = sx + ((int)(wb << 11) >> 21);
      const int la = (int)(wa >> 21), lb = (int)(wb >> 21);
      const float *ra = density + (size_t)(sy + va) * n, *rb_ = density + (size_t)(sy + vb) * n;
      const float fa = (float)va, fb = (float)vb;
      if (max(la, lb) < 16) {
        RowPix pa, pb;
        const int qa = da & ~3, qb = db & ~3;
        pa.p = ra + qa;
        pb.p = rb_ + qb;
        pa.dx = (float)(qa - sx);
        pb.dx = (float)(qb - sx);
        pa.m = ((2u << la) - 1u) << (da - qa);
        pb.m = i + 1 < m ? ((2u << lb) - 1u) << (db - qb) : 0u;
        F2 rw, rx, rq;
        pair_sums(pa, pb, rw, rx, rq);
        // (an empty row folds as zeros: the accumulators are normalised)
        fold_chunk2(acc, f2_lo(rw), f2_lo(rx), f2_lo(rq), fa, fa * fa);
        fold_chunk2(acc, f2_hi(rw), f2_hi(rx), f2_hi(rq), fb, fb * fb);
      } else {
#pragma unroll 1
        for (int k = 0; k < 2 && i + k < m; ++k) {
          const int u1 = (k ? db + lb : da + la) - sx;
          for (int u0 = (k ? db : da) - sx; u0 <= u1; u0 += 16) {
            float rw, rx, rq;
            chunk_sums((k ? rb_ : ra) + sx, u0, min(u1, u0 + 15), rw, rx, rq);
            fold_chunk2(acc, rw, rx, rq, k ? fb : fa, k ? fb * fb : fa * fa);
          }
        }
      }
    }
  } while (!done);
  out.wh = f2_lo(acc.wxh), out.wl = f2_lo(acc.wxl);
  out.xh = f2_hi(acc.wxh), out.xl = f2_hi(acc.wxl);
  out.yh = f2_lo(acc.yeh), out.yl = f2_lo(acc.yel);
  out.eh = f2_hi(acc.yeh), out.el = f2_hi(acc.yel);
  out.r2 = R2;
  return true;
}

// Exact cell of site (sx, sy) and its sums.  bits: current site bitmap;
// W: initial window radius; rb: the covering bound.
__device__ CellSums cell_sums(const LevelBufs &a, const uint64_t *__restrict__ bits, int n, int sx,
                              int sy, int W, int rb) {
  const float *density = a.density;
  const int2 *support = a.support;
  const int2 yr = *a.sup_range;  // rows [yr.x, yr.y) hold every nonzero density
  const int vlo = max(yr.x, sy - rb) - sy, vhi = min(yr.y - 1, sy + rb) - sy;
  W = max(1, min(W, 2 * rb));
  CellSums c;
  for (;;) {
    if (!float_walk(W, rb) ||
        !cell_float(density, support, bits, n, sx, sy, W, rb, vlo, vhi, c))
      c = cell_general(density, support, bits, n, sx, sy, W, rb, vlo, vhi);
    const bool whole = W >= sx && W >= sy && W >= n - 1 - sx && W >= n - 1 - sy;
    // R2 <= rb^2, so a window of 2 rb always passes
    if (whole || 4ll * c.r2 <= (long long)W * W) return c;
    W = min(min(2 * isqrt_ceil(c.r2) + 1, 2 * W), 2 * rb);
  }
}

// Centroid coordinate base + (Sh + Sl) / (Wh + Wl), rounded once to float
// (two-float quotient; W = 0 gives NaN as the reference's 0/0 does).
__device__ __forceinline__ float cell_centroid(int base, float Sh, float Sl, float Wh, float Wl) {
  const float q = __fdiv_rn(Sh, Wh);
  const float rr = __fadd_rn(__fmaf_rn(-q, Wh, Sh), __fmaf_rn(-q, Wl, Sl));
  const float q2 = __fdiv_rn(rr, Wh);
  float s, e;
  tsum_c((float)base, q, s, e);
  return __fadd_rn(s, __fadd_rn(e, q2));
}

// Add to *counter after every earlier write of this thread is visible
// (an atomic with release semantics): the writer's half of a counter
// handoff, where whoever brings the counter to its target fences and reads
// the others' results.  Cheaper than a full fence before a plain atomic.
__device__ __forceinline__ unsigned add_release(unsigned *counter, unsigned by = 1u) {
  unsigned prev;
  asm volatile("atom.add.release.gpu.u32 %0, [%1], %2;"
               : "=r"(prev)
               : "l"(counter), "r"(by)
               : "memory");
  return prev;
}

__device__ __forceinline__ uint64_t *bits_at(const LevelBufs &a, int k) {
  return k == 0 ? a.bits[0] : (k == 1 ? a.bits[1] : a.bits[2]);
}
__device__ __forceinline__ unsigned *counts_at(const LevelBufs &a, int k) {
  return k == 0 ? a.counts[0] : (k == 1 ? a.counts[1] : a.counts[2]);
}

// Warp reduction of (energy two-float, max r2, max move2) in a fixed order.
__device__ __forceinline__ void warp_reduce(float &eh, float &el, unsigned &r2, unsigned &mv) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float oh = __shfl_xor_sync(0xffffffffu, eh, o);
    const float ol = __shfl_xor_sync(0xffffffffu, el, o);
    dfa(eh, el, oh, ol);
  }
  r2 = __reduce_max_sync(0xffffffffu, r2);
  mv = __reduce_max_sync(0xffffffffu, mv);
}

// The gCVT schedule after an iteration of energy E (gcvt.cu:1105-1142), the
// next covering bound, and the rotation of the bitmaps.
__device__ void run_schedule(DevState *st, double E, unsigned r2, unsigned mv, int n, int cur) {
  st->energy = E;
  const int i = st->iter;
  if (i % 10 == 0) st->sampled = E;          // gcvt.cu:1116-1117
  st->iter = i + 1;                          // gcvt.cu:1123
  st->level_iters += 1;
  int stop = 0;
  if ((i + 1) % 10 == 0) {                   // gcvt.cu:1125-1140
    const double diff = st->last_energy - st->sampled;
    const double grad = diff / 10.0;
    st->omega = (float)fmin(2.0, 1.0 + diff);
    if (st->use_stop_rule && (st->level ? grad < 3e-1 : grad < 1e-5)) stop = 1;
    else st->last_energy = st->sampled;
  }
  if (st->use_stop_rule ? (st->iter >= st->max_iter) : (st->level_iters >= st->fixed_iters))
    stop = 1;                                // gcvt.cu:1142
  if (st->target_energy > 0.0 && E <= st->target_energy) stop = 1;  // time-to-energy runs
  if (stop) st->stopped = 1;
  st->cover = min(isqrt_ceil((int)r2) + isqrt_ceil((int)mv), 2 * n);
  st->cur = cur == 2 ? 0 : cur + 1;
  st->done_blocks = 0;
  __threadfence();
}

// The end of a pass: MODE 0 and 4 (a plain iteration, MODE 4 also writing
// the learned step's features) run the schedule; MODE 5 (the iteration of
// the jumped sites) also judges the jump: it stands if the jumped sites'
// energy is below the energy of the sites it started from (when no jump was
// proposed, MODE 5 is a plain iteration); MODE 2 (features only, nothing
// moves) just closes the pass.
template <int MODE>
__device__ void pass_done(DevState *st, double E, unsigned r2, unsigned mv, int n, int cur) {
  if (MODE == 5 && st->gate_active) {
    st->gate_e1 = E;
    st->gate_accept = E < st->gate_e0 ? 1 : 0;
  }
  if (MODE == 0 || MODE == 4 || MODE == 5) {
    run_schedule(st, E, r2, mv, n, cur);
  } else {
    st->done_blocks = 0;
    __threadfence();
  }
}

// What one chart's iteration reads at its start.
struct IterView {
  const uint64_t *bits;  // current sites
  uint64_t *nxt;         // where the moved sites go
  unsigned *cnt_nxt;     // their per-list-block counts
  float omega;
  int W0, rb, nsites, cur, nxt_i, slack;
  unsigned ngroups;      // 32-site groups of the list
};

__device__ __forceinline__ IterView iter_view(const LevelBufs &a) {
  const DevState *st = a.st;
  IterView v;
  v.cur = st->snap_cur;
  v.nxt_i = v.cur == 2 ? 0 : v.cur + 1;
  v.bits = bits_at(a, v.cur);
  v.nxt = bits_at(a, v.nxt_i);
  v.cnt_nxt = counts_at(a, v.nxt_i);
  v.omega = st->snap_omega;
  v.W0 = st->snap_window;
  v.rb = st->snap_cover;
  v.nsites = st->snap_count;
  v.slack = st->hint_slack;
  v.ngroups = (unsigned)(v.nsites + 31) / 32;
  return v;
}

// The snapshot k_cell reads (k_list, before the iteration; thread 0 of the
// chart's first list block).  A stopped chart records only that it stopped.
__device__ __forceinline__ void take_snapshot(DevState *st) {
  st->snap_stopped = st->stopped;
  st->snap_cur = st->cur;
  st->snap_omega = st->omega;
  st->snap_window = st->window;
  st->snap_cover = st->cover;
}

// Features of listed site idx at (sx, sy) with cell sums cs, for the learned
// step, all in units of the mean cell radius (DevState::feat_scale): its
// pending Lloyd displacement (the centroid of its cell minus the site, not
// yet rounded to a pixel; 0 for a cell without density), its last three
// applied moves (newest first) and the density gradient over the density at
// the site.
__device__ __forceinline__ void site_features(const LevelBufs &a, const IterView &v, int idx,
                                              int sx, int sy, const CellSums &cs) {
  const int n = a.n;
  const float r = a.st->feat_scale, ir = 1.0f / r;
  const uint64_t h = a.hist[v.cur][(size_t)sy * n + sx];
  float *f = a.feat + (size_t)idx * 10;
  const bool mass = cs.wh > 0.f;
  const float cx = mass ? cell_centroid(sx, cs.xh, cs.xl, cs.wh, cs.wl) - (float)sx : 0.f;
  const float cy = mass ? cell_centroid(sy, cs.yh, cs.yl, cs.wh, cs.wl) - (float)sy : 0.f;
  f[0] = cx * ir;
  f[1] = cy * ir;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f[2 + 2 * k] = (float)(int8_t)(h >> (16 * k)) * ir;
    f[3 + 2 * k] = (float)(int8_t)(h >> (16 * k + 8)) * ir;
  }
  const float *d = a.density;
  const float r0 = d[(size_t)sy * n + sx];
  const int xa = max(sx - 1, 0), xb = min(sx + 1, n - 1), ya = max(sy - 1, 0), yb = min(sy + 1, n - 1);
  const float gx = (d[(size_t)sy * n + xb] - d[(size_t)sy * n + xa]) / (float)(xb - xa);
  const float gy = (d[(size_t)yb * n + sx] - d[(size_t)ya * n + sx]) / (float)(yb - ya);
  f[8] = r0 > 0.f ? gx / r0 * r : 0.f;
  f[9] = r0 > 0.f ? gy / r0 * r : 0.f;
}

// Group g of a chart (32 listed sites, one per lane).  MODE 0: cells, moves,
// and the group's share of the energy reduction; the warp that completes the
// chart's last 64-group runs its schedule.  MODE 1: moments only, written as
// doubles (W, X, Y, E) at each site pixel of out4 (four n*n planes).
// The move of listed site e at (sx, sy) with cell sums cs (gcvt.cu:753-781):
// the over-relaxed centroid rounded to float, then to a pixel; fixed sites
// and zero-density targets stay.  The site goes into the next bitmap (the
// first to set a bit counts it for the next list), leaves its window hint and
// (learned steps) its move history and id at its new pixel.  Returns the
// move's squared length.  With centry, the count is left to the caller: the
// list block to count in goes to *centry (-1: the bit was set already), so
// that a warp adds its group's sites with one atomic per list block instead
// of one per site (many sites land in one list block, and same-address
// atomics serialise).
__device__ __forceinline__ unsigned move_site(const LevelBufs &a, const IterView &v, uint32_t e,
                                              int sx, int sy, const CellSums &cs,
                                              int *centry = nullptr) {
  const int n = a.n;
  const size_t pid = (size_t)sy * n + sx;
  const float cx = cell_centroid(sx, cs.xh, cs.xl, cs.wh, cs.wl);
  const float cy = cell_centroid(sy, cs.yh, cs.yl, cs.wh, cs.wl);
  const float fx = __fadd_rn(__fmaf_rn(__fsub_rn(cx, (float)sx), v.omega, (float)sx), 0.5f);
  const float fy = __fadd_rn(__fmaf_rn(__fsub_rn(cy, (float)sy), v.omega, (float)sy), 0.5f);
  int nx = min(max(__float2int_rz(fx), 0), n - 1);
  int ny = min(max(__float2int_rz(fy), 0), n - 1);
  if ((e & 0x8000u) || a.density[(size_t)ny * n + nx] == 0.0f) { nx = sx; ny = sy; }
  const unsigned mv = (unsigned)((nx - sx) * (nx - sx) + (ny - sy) * (ny - sy));
  const size_t widx = (size_t)(ny / kBand) * n + nx;
  const unsigned long long bit = 1ull << (ny % kBand);
  const unsigned long long old =
      atomicOr(reinterpret_cast<unsigned long long *>(v.nxt + widx), bit);
  const int entry = (old & bit) ? -1 : (int)(widx / kListWords);
  if (centry) *centry = entry;
  else if (entry >= 0) atomicAdd(v.cnt_nxt + entry, 1u);
  const size_t npid = (size_t)ny * n + nx;
  a.hint[npid] = (uint8_t)min(2 * isqrt_ceil(cs.r2) + v.slack, 255);
  if (a.hist[0]) {  // this move becomes the newest of the site's last four
    const int mx = min(max(nx - sx, -127), 127), my = min(max(ny - sy, -127), 127);
    a.hist[v.nxt_i][npid] = (a.hist[v.cur][pid] << 16) | (uint64_t)(uint8_t)mx |
                            ((uint64_t)(uint8_t)my << 8);
  }
  if (a.ids[0]) a.ids[v.nxt_i][npid] = a.ids[v.cur][pid];
  return mv;
}

// The energy reduction after group g (lane i holds site 32 g + i's energy
// two-float, max cell radius^2 and move^2): group total -> slot; the warp
// finishing the last group of a 64-group reduces the 64 slots; the warp
// finishing the last 64-group totals them and closes the pass (pass_done).
template <int MODE>
__device__ __forceinline__ void group_tail(const LevelBufs &a, const IterView &v, unsigned g,
                                           int lane, float eh, float el, unsigned r2,
                                           unsigned mv) {
  DevState *st = a.st;
  warp_reduce(eh, el, r2, mv);
  int last = 0;
  const unsigned sg = g / kGroupsPerSlot;
  const unsigned sbase = sg * kGroupsPerSlot;
  const unsigned starget = min((unsigned)kGroupsPerSlot, v.ngroups - sbase);
  if (lane == 0) {
    a.gslot[g] = make_float4(eh, el, __uint_as_float(r2), __uint_as_float(mv));
    last = add_release(a.scnt + sg) == starget - 1;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
  eh = el = 0.f;
  r2 = mv = 0;
  for (unsigned k = lane; k < starget; k += 32) {
    const float4 q = __ldcg(a.gslot + sbase + k);
    dfa(eh, el, q.x, q.y);
    r2 = max(r2, __float_as_uint(q.z));
    mv = max(mv, __float_as_uint(q.w));
  }
  warp_reduce(eh, el, r2, mv);
  const unsigned nslots = (v.ngroups + kGroupsPerSlot - 1) / kGroupsPerSlot;
  last = 0;
  if (lane == 0) {
    a.sslot[sg] = make_float4(eh, el, __uint_as_float(r2), __uint_as_float(mv));
    a.scnt[sg] = 0u;
    last = add_release(&st->done_blocks) == nslots - 1;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
  eh = el = 0.f;
  r2 = mv = 0;
  for (unsigned k = lane; k < nslots; k += 32) {
    const float4 q = __ldcg(a.sslot + k);
    dfa(eh, el, q.x, q.y);
    r2 = max(r2, __float_as_uint(q.z));
    mv = max(mv, __float_as_uint(q.w));
  }
  warp_reduce(eh, el, r2, mv);
  if (lane == 0) {
    const double E = ((double)eh + (double)el) * st->energy_scale;
    pass_done<MODE>(st, E, r2, mv, a.n, v.cur);
  }
}

// Group g of a chart (32 listed sites, one per lane).  MODE 0: cells, moves,
// and the group's share of the energy reduction.  MODE 1: moments only,
// written as doubles (W, X, Y, E) at each site pixel of out4 (four n*n
// planes).  MODE 2: the learned step's features of the sites (nothing
// moves).  MODE 4: MODE 0 and the features, with each site's window in
// jaux.  MODE 5: MODE 0 for the jumped sites (the pass then judges the jump).
// The next work item of a persistent warp: its first is its block index (no
// atomic), the rest come from the ticket, numbered after that first wave (a
// ticket every warp takes at once is a burst of same-address atomics).
__device__ __forceinline__ unsigned next_item(unsigned *ticket, bool first, int lane) {
  unsigned g = blockIdx.x;
  if (!first) {
    if (lane == 0) g = gridDim.x + atomicAdd(ticket, 1u);
    g = __shfl_sync(0xffffffffu, g, 0);
  }
  return g;
}

template <int MODE>
__device__ void cell_group(const LevelBufs &a, const IterView &v, unsigned g, int lane,
                           double *out4) {
  const int n = a.n;
  float eh = 0.f, el = 0.f;
  unsigned r2 = 0, mv = 0;
  int centry = -1;
  const int idx = (int)g * 32 + lane;
  if (idx < v.nsites) {
    const uint32_t e = a.list[idx];
    const int sx = (int)(e & 0x7fffu), sy = (int)(e >> 16);
    const size_t pid = (size_t)sy * n + sx;
    const int h = a.hint[pid];
    const CellSums cs = cell_sums(a, v.bits, n, sx, sy, h ? h : v.W0, v.rb);
    if (MODE == 1) {
      const size_t nn = (size_t)n * n;
      const double Wd = (double)cs.wh + (double)cs.wl;
      out4[pid] = Wd;
      out4[nn + pid] = (double)sx * Wd + ((double)cs.xh + (double)cs.xl);
      out4[2 * nn + pid] = (double)sy * Wd + ((double)cs.yh + (double)cs.yl);
      out4[3 * nn + pid] = (double)cs.eh + (double)cs.el;
    } else {
      dfa(eh, el, cs.eh, cs.el);
      r2 = (unsigned)cs.r2;
      if (MODE == 2 || MODE == 4) site_features(a, v, idx, sx, sy, cs);
      if (MODE == 4) a.jaux[idx] = (uint32_t)min(2 * isqrt_ceil(cs.r2) + v.slack, 255);
      if (MODE != 2) mv = move_site(a, v, e, sx, sy, cs, &centry);
    }
  }
  __syncwarp();
  // the group's new sites, counted per list block: one atomic per block
  const unsigned want = __ballot_sync(0xffffffffu, centry >= 0);
  if (centry >= 0) {
    const unsigned peers = __match_any_sync(want, centry);
    if (lane == __ffs(peers) - 1) atomicAdd(v.cnt_nxt + centry, (unsigned)__popc(peers));
  }
  if (MODE == 1) return;
  group_tail<MODE>(a, v, g, lane, eh, el, r2, mv);
}

// ---------------------------------------------------------------------------
// One site per warp, for problems with few sites (a lane-per-site group runs
// one site's whole cell serially, and only a few groups exist).  The same cell
// and the same sums, bit for bit: a warp gathers its site's candidates, bounds
// the rows one per lane and sums their 16-pixel chunks one per lane; the chunks
// are then folded into the cell sums in the lane-per-site order.  The energy
// reduction keeps its groups: each site's contribution waits in
// LevelBufs::sitev, and the warp finishing a group's last sites reduces it.
// ---------------------------------------------------------------------------

constexpr int kWarpEnts = 96;  // chunk sums of a site kept in shared memory

constexpr int kWarpRec = 128;  // candidates of a site kept in shared memory
constexpr int kBlockSites = 8;  // sites (warps) per block

struct alignas(16) WarpScratch {  // (ent and, reused, the whole are read as float4)
  int2 rec[kWarpRec];  // left of s first: float lines {k, s}, or make_rec's records
  // per 16-pixel chunk of the rows, in fold order: the terms of (W, SX, SY, E),
  // high then low parts (the padding spreads the block's sites over the banks)
  float ent[kWarpEnts][8];
  float sum[8];   // folded already: (W, SX, SY, E) high, then low
  int m;          // chunks left to fold; -1: sum holds the result
  int r2;
  int pad[26];
};
static_assert(sizeof(WarpScratch) % 128 == 16, "sites 4 banks apart (fold: lane 4 s + q)");
static_assert(offsetof(WarpScratch, ent) % 16 == 0, "float4 entries");

// Sums of the pixels [u0, u1] (at most 16, relative to the site) of a row, all
// its aligned 16-byte loads in flight together.
__device__ __forceinline__ void chunk_quads(const float *__restrict__ row, int u0, int u1, int sx,
                                            float &rw, float &rx, float &rq) {
  const int q0 = (sx + u0) & ~3, last = (sx + u1 - q0) >> 2;
  const float4 *p = reinterpret_cast<const float4 *>(row + q0);
  const unsigned m = ((2u << (u1 - u0)) - 1u) << (sx + u0 - q0);
  float4 q[5];
#pragma unroll
  for (int k = 0; k < 5; ++k)
    q[k] = k <= last ? __ldg(p + k) : make_float4(0.f, 0.f, 0.f, 0.f);
  rw = 0.f, rx = 0.f, rq = 0.f;
  float dx = (float)(q0 - sx);
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    if (k > last) break;
    const float v[4] = {q[k].x, q[k].y, q[k].z, q[k].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float rho = (m >> (4 * k + j)) & 1u ? v[j] : 0.f;
      const float t = __fmul_rn(dx, rho);
      rw = __fadd_rn(rw, rho);
      rx = __fadd_rn(rx, t);
      rq = __fmaf_rn(t, dx, rq);
      dx = __fadd_rn(dx, 1.0f);
    }
  }
}

// Row v's summed pixels [da, db] of a cell from its records; false when the
// cell has ended there (or v is past the row limits).
template <bool FLT>
__device__ __forceinline__ bool warp_row(const int2 *__restrict__ support, const WarpScratch &ws,
                                         int n, int sx, int sy, int rb2, int nl, int cnt, float eps,
                                         bool fast, int v, int vmin, int vmax, int &da, int &db) {
  const int2 sup = __ldg(support + min(max(sy + v, 0), n - 1));
  int l = -sx, h = n - 1 - sx;
  if (FLT) {
    float lo = (float)(-sx - 1), hi = (float)(n - 1 - sx);
    const float fv = (float)v;
    const float2 *rec = reinterpret_cast<const float2 *>(ws.rec);
    for (int k = 0; k < nl; ++k) lo = fmaxf(lo, __fmaf_rn(rec[k].y, fv, rec[k].x));
    for (int k = nl; k < cnt; ++k) hi = fminf(hi, __fmaf_rn(rec[k].y, fv, rec[k].x));
    l = __float2int_rd(lo + eps) + 1, h = __float2int_rd(hi + eps);
  } else {
    for (int k = 0; k < cnt; ++k) {
      const int2 r = ws.rec[k];
      const int S = (int)(int16_t)((unsigned)r.y & 0xffffu);
      const int D = (int)(int16_t)((unsigned)r.y >> 16);
      const int aD = abs(D), N = r.x - S * v;
      const int q = fast ? floordiv_r(N, aD, rcp_approx((float)aD))
                         : floordiv(N, aD);
      if (D > 0) h = min(h, q);
      else l = max(l, q + 1);
    }
  }
  da = max(l, sup.x - sx), db = min(h, sup.y - 1 - sx);
  if (l > h + 1 || v < vmin || v > vmax) return false;
  if (da <= db && max(da * da, db * db) + v * v > rb2) {  // clip to the covering disc
    const int hx = isqrt_floor(rb2 - v * v);
    da = max(da, -hx);
    db = min(db, hx);
  }
  return true;
}

// The candidates of a column as bits from row y0 of the window (W <= 31): the
// rows of the disc of radius W2^(1/2) around the site, its own column and bit
// excepted.
__device__ __forceinline__ uint64_t disc_rows(uint64_t col, int A, int W2, int o) {
  const int h2 = W2 - A * A;
  int h = (int)sqrtf((float)h2);  // floor(sqrt(h2)), at most one off
  h += ((h + 1) * (h + 1) <= h2) - (h * h > h2);
  const int lo = max(o - h, 0), hi = o + h;  // hi <= 62
  return col & (((2ull << hi) - 1ull) & ~((1ull << lo) - 1ull));
}

// The chunks e0 .. e0 + m - 1 of the warp's rows (a lane a row v, its pixels [da, db] in
// nch chunks, incl up to it) into ws.ent, one per lane.
__device__ __forceinline__ void chunk_entries(const float *__restrict__ density, int n, int sx,
                                              int sy, int da, int db, int v, int incl, int nch,
                                              int e0, int m, int lane, WarpScratch &ws) {
  constexpr unsigned kFull = 0xffffffffu;
  for (int k = lane; k - lane < m; k += 32) {
    const int e = e0 + k;
    int r = 0;  // the row of chunk e: the rows whose chunks all come before it
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(kFull, incl, r + o - 1) <= e) r += o;
    const int ra = __shfl_sync(kFull, da, r), rb_ = __shfl_sync(kFull, db, r);
    const int rv = __shfl_sync(kFull, v, r), ri = __shfl_sync(kFull, incl - nch, r);
    if (k < m) {
      const int u0 = ra + 16 * (e - ri);
      float rw, rx, rq;
      chunk_quads(density + (size_t)(sy + rv) * n, u0, min(rb_, u0 + 15), sx, rw, rx, rq);
      // fold_chunk's terms of SY and E
      const float fv = (float)rv, fv2 = (float)(rv * rv);
      const float yh = __fmul_rn(fv, rw), yl = __fmaf_rn(fv, rw, -yh);
      float qh = rq, ql = 0.f;
      dfa_scaled(qh, ql, fv2, rw, 0.f);
      float4 *o = reinterpret_cast<float4 *>(ws.ent[k]);
      o[0] = make_float4(rw, rx, yh, qh);
      o[1] = make_float4(0.f, 0.f, yl, ql);
    }
  }
}

// The cell of a site by a warp with the window radius W (FLT: float_walk
// holds): its rows' chunk sums into ws.ent, or, when they are too many for
// it or the cell is tall, folded into ws.sum.  False when the candidates do not
// fit.  What bounds it is latency and issue slots, so every step is spread
// over the lanes: a lane per window column, per row, per 16-pixel chunk.
template <bool FLT>
__device__ __forceinline__ bool warp_cell(const float *__restrict__ density,
                                          const int2 *__restrict__ support,
                                          const uint64_t *__restrict__ bits, int n, int sx, int sy,
                                          int W, int rb, int vmin, int vmax, int lane,
                                          WarpScratch &ws, int &r2) {
  constexpr unsigned kFull = 0xffffffffu;
  const int rb2 = rb * rb;
  const int x0 = max(0, sx - W), x1 = min(n - 1, sx + W);
  const int y0 = max(0, sy - W), y1 = min(n - 1, sy + W);
  // candidates: a lane per column, compacted into shared memory in column order
  int cnt = 0, nl = 0;
  const int b0 = y0 >> 6, b1 = y1 >> 6;
  if (FLT && W <= 31) {  // at most 63 columns of at most 63 rows: one word a column
    const int sh = y0 & 63, W2 = W * W, o = sy - y0;
    const uint64_t rm = row_mask(0, y1 - y0);
    const uint64_t *p0 = bits + (size_t)b0 * n, *p1 = bits + (size_t)b1 * n;
    uint64_t w[2][2];  // two columns a lane, all words in flight together
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int x = x0 + 32 * k + lane;
      w[k][0] = x <= x1 ? __ldg(p0 + x) : 0ull;
      w[k][1] = x <= x1 && b1 > b0 ? __ldg(p1 + x) : 0ull;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (x0 + 32 * k > x1) break;
      const int x = x0 + 32 * k + lane, A = x - sx;
      uint64_t col = w[k][0] >> sh;
      if (sh) col |= w[k][1] << (64 - sh);
      col &= rm;
      if (A == 0) {  // s's own column: the nearest site on each side limits the rows
        const uint64_t up = (col >> o) >> 1, dn = col & ((1ull << o) - 1ull);
        if (up) same_column_limit(__ffsll((long long)up), sy, vmin, vmax);
        if (dn) same_column_limit(63 - __clzll((long long)dn) - o, sy, vmin, vmax);
        col = 0ull;
      } else if (x <= x1) {
        col = disc_rows(col, A, W2, o);
      }
      const int mine = __popcll(col);
      int incl = mine;
#pragma unroll
      for (int i = 1; i < 32; i <<= 1) {
        const int u = __shfl_up_sync(kFull, incl, i);
        if (lane >= i) incl += u;
      }
      nl += __reduce_add_sync(kFull, A < 0 ? mine : 0);
      int pos = cnt + incl - mine;
      const float r = rcp_approx((float)A);
      while (col) {
        const int B = __ffsll((long long)col) - 1 - o;
        col &= col - 1ull;
        if (pos < kWarpRec)
          ws.rec[pos] = make_int2(__float_as_int(0.5f * (float)(A * A + B * B) * r),
                                  __float_as_int(-(float)B * r));
        ++pos;
      }
      cnt += __shfl_sync(kFull, incl, 31);
    }
  } else {
    const bool whole = x0 == 0 && y0 == 0 && x1 == n - 1 && y1 == n - 1;
    // every site when the window holds the grid (no certificate needed then)
    const int Wc = whole ? 0x7fffffff : (int)min((long long)W * W, 0x7fffffffll);
    for (int c0 = x0; c0 <= x1; c0 += 32) {
      const int x = c0 + lane, A = x - sx;
      int mine = 0;
      auto each = [&](auto &&f) {  // f(B, K) of the column's candidates
        if (x > x1) return;
        for (int b = b0; b <= b1; ++b) {
          uint64_t w = __ldg(bits + (size_t)b * n + x) &
                       row_mask(max(y0 - 64 * b, 0), min(y1 - 64 * b, 63));
          while (w) {
            const int B = 64 * b + __ffsll((long long)w) - 1 - sy;
            w &= w - 1ull;
            const int K = A * A + B * B;
            if (K && K <= Wc) f(B, K);
          }
        }
      };
      each([&](int B, int) {
        if (A == 0) same_column_limit(B, sy, vmin, vmax);
        else ++mine;
      });
      int incl = mine;
#pragma unroll
      for (int i = 1; i < 32; i <<= 1) {
        const int u = __shfl_up_sync(kFull, incl, i);
        if (lane >= i) incl += u;
      }
      nl += __reduce_add_sync(kFull, A < 0 ? mine : 0);
      if (mine) {
        int pos = cnt + incl - mine;
        const float r = rcp_approx((float)A);
        each([&](int B, int K) {
          if (pos < kWarpRec)
            ws.rec[pos] = FLT ? make_int2(__float_as_int(0.5f * (float)K * r),
                                          __float_as_int(-(float)B * r))
                              : make_rec(A, B, K);
          ++pos;
        });
      }
      cnt += __shfl_sync(kFull, incl, 31);
    }
  }
  vmin = __reduce_max_sync(kFull, vmin);
  vmax = __reduce_min_sync(kFull, vmax);
  if (cnt > kWarpRec) return false;
  __syncwarp();
  const float eps = 0.25f / (float)W;
  // |K - S v| <= 2 W^2 + 2 W rb: below 2^23 the reciprocal estimate is safe
  const bool fast = 2ll * W * W + 2ll * W * rb < (1ll << 23);
  int R2 = 0;
  // rows outward from s, one per lane: first sixteen up and sixteen down at
  // once; a cell that has not ended there on both sides is walked again 32
  // rows at a time, up and then down
  float ah = 0.f, al = 0.f;  // folded here: lane q < 4 holds sum q of (W, SX, SY, E)
  int pass = 0, dir = 1, base = 0, left = -1;
  for (;;) {
    const int v = pass == 0 ? (lane < 16 ? lane : 15 - lane) : base + dir * lane;
    int da = 1, db = 0;
    const bool in = warp_row<FLT>(support, ws, n, sx, sy, rb2, nl, cnt, eps, fast, v, vmin, vmax,
                                  da, db);
    // (a row before the limits' near end is skipped, one past their far end
    // ends the walk)
    const bool skip = v >= 0 ? v < vmin : v > vmax;
    const unsigned stop = __ballot_sync(kFull, !in && !skip);
    unsigned live;  // the lanes whose rows are walked
    if (pass == 0) {
      const unsigned su = stop & 0xffffu, sd = stop >> 16;
      if (!su || !sd) {
        pass = 1;
        continue;
      }
      live = ((1u << (__ffs(su) - 1)) - 1u) | (((1u << (__ffs(sd) - 1)) - 1u) << 16);
    } else {
      live = stop ? (1u << (__ffs(stop) - 1)) - 1u : kFull;
    }
    const bool has = ((live >> lane) & 1u) && in && da <= db;
    if (has) R2 = max(R2, max(da * da, db * db) + v * v);
    // the rows' 16-pixel chunks in fold order (row after row), one per lane
    const int nch = has ? (db - da + 16) >> 4 : 0;
    int incl = nch;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    const int total = __shfl_sync(kFull, incl, 31);
    const bool defer = pass == 0 && total <= kWarpEnts;
    for (int e0 = 0; e0 < total; e0 += kWarpEnts) {
      const int m = min(total - e0, kWarpEnts);
      chunk_entries(density, n, sx, sy, da, db, v, incl, nch, e0, m, lane, ws);
      __syncwarp();
      if (defer) continue;
      if (lane < 4) {  // the four sums side by side, chunk after chunk
#pragma unroll 4
        for (int k = 0; k < m; ++k) dfa(ah, al, ws.ent[k][lane], ws.ent[k][4 + lane]);
      }
      __syncwarp();
    }
    if (pass == 0) {
      if (defer) left = total;
      break;
    }
    if (stop) {
      if (dir < 0) break;
      dir = -1;
      base = -1;
    } else {
      base += 32 * dir;
    }
  }
  if (left < 0 && lane < 4) {
    ws.sum[lane] = ah;
    ws.sum[4 + lane] = al;
  }
  if (lane == 0) ws.m = left;
  r2 = __reduce_max_sync(kFull, R2);
  return true;
}

// The same for a window of more than kWarpRec candidates (clusters, sites along a line,
// a region without sites): they pass through shared memory in batches, again for every 32
// rows.  Without it every lane walked the whole cell (cell_general): 1085 sites on a
// circle of 768 x 768 228 ms an iteration, 3.6 now; a cluster of 1122 103 and 2.3.
// Returns max |p - s|^2 over the summed pixels; the sums are in ws.sum.
__device__ __noinline__ int warp_cell_crowded(const float *__restrict__ density,
                                              const int2 *__restrict__ support,
                                              const uint64_t *__restrict__ bits, int n, int sx,
                                              int sy, int W, int rb, int vmin, int vmax, int lane,
                                              WarpScratch &ws) {
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned before = (1u << lane) - 1u;
  const int rb2 = rb * rb;
  const int x0 = max(0, sx - W), x1 = min(n - 1, sx + W);
  const int y0 = max(0, sy - W), y1 = min(n - 1, sy + W);
  const bool whole = x0 == 0 && y0 == 0 && x1 == n - 1 && y1 == n - 1;
  const int Wc = whole ? 0x7fffffff : (int)min((long long)W * W, 0x7fffffffll);
  const int b0 = y0 >> 6, b1 = y1 >> 6;
  auto rows_of = [&](int x, int b) {
    return __ldg(bits + (size_t)b * n + x) & row_mask(max(y0 - 64 * b, 0), min(y1 - 64 * b, 63));
  };
  for (int b = b0 + lane; b <= b1; b += 32)  // s's own column
    for (uint64_t w = rows_of(sx, b); w; w &= w - 1ull) {
      const int B = 64 * b + __ffsll((long long)w) - 1 - sy;
      if (B) same_column_limit(B, sy, vmin, vmax);
    }
  vmin = __reduce_max_sync(kFull, vmin);
  vmax = __reduce_min_sync(kFull, vmax);
  // |K - S v| <= 2 W^2 + 2 W rb: below 2^23 the reciprocal estimate is safe
  const bool fast = 2ll * W * W + 2ll * W * rb < (1ll << 23);
  int R2 = 0;
  float ah = 0.f, al = 0.f;  // lane q < 4 holds sum q of (W, SX, SY, E)
  for (int dir = 1, base = 0;;) {
    const int v = base + dir * lane;
    int l = -sx, h = n - 1 - sx, fill = 0;
    auto bound = [&]() {  // this lane's row by the candidates of the batch
      __syncwarp();
      for (int k = 0; k < fill; ++k) {
        const int2 r = ws.rec[k];
        const int S = (int)(int16_t)((unsigned)r.y & 0xffffu);
        const int D = (int)(int16_t)((unsigned)r.y >> 16);
        const int aD = abs(D), N = r.x - S * v;
        const int q = fast ? floordiv_r(N, aD, rcp_approx((float)aD)) : floordiv(N, aD);
        if (D > 0) h = min(h, q);
        else l = max(l, q + 1);
      }
      __syncwarp();
      fill = 0;
    };
    for (int c0 = x0; c0 <= x1; c0 += 32) {
      const int x = c0 + lane, A = x - sx;
      for (int b = b0; b <= b1; ++b) {
        uint64_t w = x <= x1 && A ? rows_of(x, b) : 0ull;
        for (;;) {  // a candidate a lane until there are none
          int B = 0, K = 0;
          bool has = false;
          while (w && !has) {
            B = 64 * b + __ffsll((long long)w) - 1 - sy;
            w &= w - 1ull;
            K = A * A + B * B;
            has = K <= Wc;
          }
          const unsigned m = __ballot_sync(kFull, has);
          if (!m) break;
          if (has) ws.rec[fill + __popc(m & before)] = make_rec(A, B, K);
          fill += __popc(m);
          if (fill > kWarpRec - 32) bound();
        }
      }
    }
    bound();
    // the row's pixels, and how far the rows are walked (as warp_row and warp_cell)
    const int2 sup = __ldg(support + min(max(sy + v, 0), n - 1));
    int da = max(l, sup.x - sx), db = min(h, sup.y - 1 - sx);
    const bool in = l <= h + 1 && v >= vmin && v <= vmax;
    if (in && da <= db && max(da * da, db * db) + v * v > rb2) {
      const int hx = isqrt_floor(rb2 - v * v);
      da = max(da, -hx);
      db = min(db, hx);
    }
    const bool skip = v >= 0 ? v < vmin : v > vmax;
    const unsigned stop = __ballot_sync(kFull, !in && !skip);
    const unsigned live = stop ? (1u << (__ffs(stop) - 1)) - 1u : kFull;
    const bool has = ((live >> lane) & 1u) && in && da <= db;
    if (has) R2 = max(R2, max(da * da, db * db) + v * v);
    const int nch = has ? (db - da + 16) >> 4 : 0;
    int incl = nch;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    const int total = __shfl_sync(kFull, incl, 31);
    for (int e0 = 0; e0 < total; e0 += kWarpEnts) {
      const int m = min(total - e0, kWarpEnts);
      chunk_entries(density, n, sx, sy, da, db, v, incl, nch, e0, m, lane, ws);
      __syncwarp();
      if (lane < 4) {
#pragma unroll 4
        for (int k = 0; k < m; ++k) dfa(ah, al, ws.ent[k][lane], ws.ent[k][4 + lane]);
      }
      __syncwarp();
    }
    if (!stop) {
      base += 32 * dir;
    } else if (dir > 0) {
      dir = -1;
      base = -1;
    } else {
      break;
    }
  }
  if (lane < 4) {
    ws.sum[lane] = ah;
    ws.sum[4 + lane] = al;
  }
  if (lane == 0) ws.m = -1;
  return __reduce_max_sync(kFull, R2);
}

// The cell of a site by a warp, left in ws (chunks to fold, or the sums).
__device__ void cell_sums_warp(const LevelBufs &a, const uint64_t *__restrict__ bits, int n, int sx,
                               int sy, int W, int rb, int lane, WarpScratch &ws) {
  const float *density = a.density;
  const int2 *support = a.support;
  const int2 yr = *a.sup_range;
  const int vlo = max(yr.x, sy - rb) - sy, vhi = min(yr.y - 1, sy + rb) - sy;
  W = max(1, min(W, 2 * rb));
  int r2 = 0;
  for (;;) {
    const bool fits =
        float_walk(W, rb)
            ? warp_cell<true>(density, support, bits, n, sx, sy, W, rb, vlo, vhi, lane, ws, r2)
            : warp_cell<false>(density, support, bits, n, sx, sy, W, rb, vlo, vhi, lane, ws, r2);
    if (!fits)
      r2 = warp_cell_crowded(density, support, bits, n, sx, sy, W, rb, vlo, vhi, lane, ws);
    const bool whole = W >= sx && W >= sy && W >= n - 1 - sx && W >= n - 1 - sy;
    if (whole || 4ll * r2 <= (long long)W * W) break;
    W = min(min(2 * isqrt_ceil(r2) + 1, 2 * W), 2 * rb);
    __syncwarp();
  }
  if (lane == 0) ws.r2 = r2;
}

// The end of an iteration of few groups, from the groups' totals gt (visible to this
// warp): group_tail's reduction of the slots and of their totals.
template <int MODE>
__device__ __forceinline__ void few_slots(const LevelBufs &a, const IterView &v, const float4 *gt,
                                          int lane) {
  float th = 0.f, tl = 0.f;  // lane k: slot k's total
  unsigned tr2 = 0, tmv = 0;
  for (unsigned sb = 0, k = 0; sb < v.ngroups; sb += kGroupsPerSlot, ++k) {
    float eh = 0.f, el = 0.f;
    unsigned r2 = 0, mv = 0;
    for (unsigned i = lane; i < min((unsigned)kGroupsPerSlot, v.ngroups - sb); i += 32) {
      const float4 q = gt == a.gslot ? __ldcg(gt + sb + i) : gt[sb + i];
      dfa(eh, el, q.x, q.y);
      r2 = max(r2, __float_as_uint(q.z));
      mv = max(mv, __float_as_uint(q.w));
    }
    warp_reduce(eh, el, r2, mv);
    tr2 = max(tr2, r2), tmv = max(tmv, mv);
    if (lane == (int)k) dfa(th, tl, eh, el);
  }
  warp_reduce(th, tl, tr2, tmv);
  if (lane == 0) {
    const double E = ((double)th + (double)tl) * a.st->energy_scale;
    pass_done<MODE>(a.st, E, tr2, tmv, a.n, v.cur);
  }
}

// The energy reduction after group g of the block kernel below: group_tail's
// sums in the same order, but with one counter (the groups are few), so the
// warp finishing the last group reduces every slot.
template <int MODE>
__device__ __forceinline__ void few_groups_tail(const LevelBufs &a, const IterView &v, unsigned g,
                                                int lane, float eh, float el, unsigned r2,
                                                unsigned mv) {
  DevState *st = a.st;
  warp_reduce(eh, el, r2, mv);
  int last = 0;
  if (lane == 0) {
    a.gslot[g] = make_float4(eh, el, __uint_as_float(r2), __uint_as_float(mv));
    last = add_release(&st->done_blocks) == v.ngroups - 1;
  }
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
  few_slots<MODE>(a, v, a.gslot, lane);
}

// The sums of the block's sites, folded by one warp: lane 4 s + q takes sum q of
// site s; lane s (and s + 8 ...) gets site s's.
__device__ __forceinline__ CellSums fold_block(const WarpScratch *scratch, int count, int lane) {
  const int s = lane >> 2, q = lane & 3;
  float ah = 0.f, al = 0.f;
  if (s < count) {
    const WarpScratch &ws = scratch[s];
    const int m = ws.m;
    if (m < 0) ah = ws.sum[q], al = ws.sum[4 + q];
#pragma unroll 4
    for (int k = 0; k < m; ++k) dfa(ah, al, ws.ent[k][q], ws.ent[k][4 + q]);
  }
  CellSums cs;
  const int src = (lane & 7) * 4;
  constexpr unsigned kFull = 0xffffffffu;
  cs.wh = __shfl_sync(kFull, ah, src), cs.wl = __shfl_sync(kFull, al, src);
  cs.xh = __shfl_sync(kFull, ah, src + 1), cs.xl = __shfl_sync(kFull, al, src + 1);
  cs.yh = __shfl_sync(kFull, ah, src + 2), cs.yl = __shfl_sync(kFull, al, src + 2);
  cs.eh = __shfl_sync(kFull, ah, src + 3), cs.el = __shfl_sync(kFull, al, src + 3);
  return cs;
}

__device__ __forceinline__ void site_values(const LevelBufs &a, const IterView &v, unsigned g,
                                            int lane, float &eh, float &el, unsigned &r2,
                                            unsigned &mv) {
  eh = el = 0.f, r2 = mv = 0;
  if (g < v.ngroups && g * 32 + lane < (unsigned)v.nsites) {
    const float4 t = __ldcg(a.sitev + g * 32 + lane);
    eh = t.x, el = t.y, r2 = __float_as_uint(t.z), mv = __float_as_uint(t.w);
  }
}

// After a block wrote `count` of group g's site values: if they were the group's
// last, the group's values, lane l site l's.
__device__ __forceinline__ bool group_done(const LevelBufs &a, const IterView &v, unsigned g,
                                           unsigned count, int lane, float &eh, float &el,
                                           unsigned &r2, unsigned &mv) {
  const unsigned gsize = min(32u, (unsigned)v.nsites - g * 32);
  int last = 0;
  if (lane == 0) last = add_release(a.gcnt + g, count) == gsize - count;
  if (!__shfl_sync(0xffffffffu, last, 0)) return false;
  __threadfence();
  if (lane == 0) a.gcnt[g] = 0u;
  site_values(a, v, g, lane, eh, el, r2, mv);
  return true;
}

// One Lloyd iteration, one listed site per warp, kBlockSites sites per block.
// Each warp leaves its site's chunk sums in shared memory; then one warp folds
// and moves the block's sites, four lanes a site (a fold is one long chain of
// dependent additions, and most of a site's instructions when a warp runs it
// alone).  1024^2 / 4096 sites, list included: 43 -> 19 us an iteration (38.8 -> 25 us
// for the cell kernel with each warp folding its own site).  MODE 0, 4 and 5 as
// in k_cell (MODE 4 also writes the learned step's features, MODE 5 judges a
// jump).
template <int MODE>
__global__ void __launch_bounds__(32 * kBlockSites, 4) k_cell_warp(LevelBufs a) {
  __shared__ WarpScratch scratch[kBlockSites];
  __shared__ unsigned s_item;
  static_assert(kBlockSites == 8 && kWarpSites / 32 <= 32 * kGroupsPerSlot, "lane 4 s + q; slots");
  DevState *st = a.st;
  if (st->snap_stopped) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  IterView v = iter_view(a);
  ++v.slack;  // a retried cell holds up its block: a wider window costs less (1.35 -> 1.30 ms)
  if (v.ngroups == 0) {  // no sites: the schedule still advances
    if (blockIdx.x == 0 && threadIdx.x == 0) pass_done<MODE>(st, 0.0, 0u, 0u, a.n, v.cur);
    return;
  }
  const int n = a.n;
  if (v.nsites > kWarpSites) {  // more sites than LevelBufs::sitev holds: per lane
    unsigned g = blockIdx.x * kBlockSites + warp;
    while (g < v.ngroups) {
      cell_group<MODE>(a, v, g, lane, nullptr);
      if (lane == 0) g = gridDim.x * kBlockSites + atomicAdd(&st->ticket, 1u);
      g = __shfl_sync(0xffffffffu, g, 0);
    }
    return;
  }
  for (unsigned item = blockIdx.x; item * kBlockSites < (unsigned)v.nsites;) {
    const unsigned idx0 = item * kBlockSites, idx = idx0 + warp;
    const int count = min(kBlockSites, v.nsites - (int)idx0);
    if ((int)warp < count) {
      const uint32_t e = a.list[idx];
      const int sx = (int)(e & 0x7fffu), sy = (int)(e >> 16);
      const int h = a.hint[(size_t)sy * n + sx];
      cell_sums_warp(a, v.bits, n, sx, sy, h ? h : v.W0, v.rb, lane, scratch[warp]);
    }
    if (threadIdx.x == 0) s_item = gridDim.x + atomicAdd(&st->ticket, 1u);
    __syncthreads();
    item = s_item;
    if (warp == 0) {
      CellSums cs = fold_block(scratch, count, lane);
      const unsigned g = idx0 / 32;  // the block's sites lie in one group
      if (lane < count) {
        cs.r2 = scratch[lane].r2;
        const uint32_t e = a.list[idx0 + lane];
        const int sx = (int)(e & 0x7fffu), sy = (int)(e >> 16);
        float eh = 0.f, el = 0.f;
        dfa(eh, el, cs.eh, cs.el);
        if (MODE == 4) {
          site_features(a, v, (int)idx0 + lane, sx, sy, cs);
          a.jaux[idx0 + lane] = (uint32_t)min(2 * isqrt_ceil(cs.r2) + v.slack, 255);
        }
        const unsigned mv = move_site(a, v, e, sx, sy, cs);
        a.sitev[idx0 + lane] =
            make_float4(eh, el, __uint_as_float((unsigned)cs.r2), __uint_as_float(mv));
      }
      __syncwarp();
      float eh, el;
      unsigned r2, mv;
      if (group_done(a, v, g, (unsigned)count, lane, eh, el, r2, mv))
        few_groups_tail<MODE>(a, v, g, lane, eh, el, r2, mv);
    }
    __syncthreads();  // the scratch and s_item are free again
  }
}

// The whole iteration of a few sites (up to kFewSites) in one launch, without
// k_list: a block finds its eight sites from the bitmap and the per-block counts
// itself (2 to 3 us, every block the same), and the block that arrives last reduces
// the energy (in the groups' order) and runs the schedule.  Every block arrives
// exactly once, so none still starts when the state changes.  Such an iteration is
// latency from end to end (a launch, the list, one cell per warp, the tail), so the
// launch it saves shows: 50 iterations of 4096 sites of 1024 x 1024 1.31 -> 1.25 ms,
// with a learned step every fourth 2.11 -> 2.00 ms, a whole 256 x 256 run of about 70
// 1.65 -> 1.46 ms.
// Above 8192 sites a block would take several turns at finding its sites; k_list then
// costs less than they do.
__global__ void __launch_bounds__(32 * kBlockSites, 4) k_cell_few(LevelBufs a) {
  __shared__ WarpScratch scratch[kBlockSites];
  __shared__ unsigned s_pre[kFewBlocks + 1], s_w[kBlockSites];
  __shared__ uint32_t s_site[kBlockSites];
  __shared__ bool s_last;
  constexpr int kThreads = 32 * kBlockSites;
  static_assert(kListWords == 2 * kThreads && kFewBlocks == 2 * kThreads, "two per thread");
  static_assert(4 * kBlockSites * sizeof(float4) <= sizeof(scratch), "group totals in scratch");
  DevState *st = a.st;
  if (st->stopped) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = a.n;
  const size_t nwords = (size_t)(n / kBand) * n;
  const int nlb = (int)((nwords + kListWords - 1) / kListWords);
  IterView v;
  v.cur = st->cur;
  v.nxt_i = v.cur == 2 ? 0 : v.cur + 1;
  v.bits = bits_at(a, v.cur);
  v.nxt = bits_at(a, v.nxt_i);
  v.cnt_nxt = counts_at(a, v.nxt_i);
  v.omega = st->omega;
  v.W0 = st->window;
  v.rb = st->cover;
  v.slack = st->hint_slack + 1;  // (as in k_cell_warp)
  if (!st->gate_active) {  // the bitmap and counts the next iteration writes (as k_list)
    const int z = v.cur == 0 ? 2 : v.cur - 1;
    uint64_t *zw = bits_at(a, z);
    unsigned *zc = counts_at(a, z);
    const size_t t0 = (size_t)blockIdx.x * kThreads + tid, step = (size_t)gridDim.x * kThreads;
    for (size_t i = t0; i < nwords; i += step) zw[i] = 0ull;
    for (size_t i = t0; i < (size_t)nlb; i += step) zc[i] = 0u;
  }
  // inclusive scan of two values a thread over the block; returns the sum before them
  auto before = [&](unsigned mine, unsigned &total) {
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    unsigned off = incl - mine;
    total = 0;
    for (int k = 0; k < kBlockSites; ++k) {
      if (k < warp) off += s_w[k];
      total += s_w[k];
    }
    __syncthreads();
    return off;
  };
  {
    const unsigned *counts = counts_at(a, v.cur);
    const unsigned c0 = 2 * tid < nlb ? counts[2 * tid] : 0u,
                   c1 = 2 * tid + 1 < nlb ? counts[2 * tid + 1] : 0u;
    unsigned total;
    const unsigned off = before(c0 + c1, total);
    s_pre[2 * tid] = off;
    s_pre[2 * tid + 1] = off + c0;
    if (tid == 0) s_pre[kFewBlocks] = total;
    __syncthreads();
  }
  v.nsites = min((int)s_pre[kFewBlocks], kFewSites);  // (sites are never added)
  v.ngroups = (unsigned)(v.nsites + 31) / 32;
  // up to 32 groups: the last block reduces them in one go; more: each group by the
  // block that completes it (one block alone took 8 us for 128 groups)
  const bool fold_last = v.ngroups <= 4 * kBlockSites;
  for (unsigned item = blockIdx.x; item * kBlockSites < (unsigned)v.nsites; item += gridDim.x) {
    const unsigned idx0 = item * kBlockSites;
    const int count = min(kBlockSites, v.nsites - (int)idx0);
    int lb = 0, hi = nlb - 1;  // the list block of site idx0
    while (lb < hi) {
      const int mid = (lb + hi + 1) >> 1;
      if (s_pre[mid] <= idx0) lb = mid;
      else hi = mid - 1;
    }
    for (; lb < nlb && s_pre[lb] < idx0 + count; ++lb) {
      if (s_pre[lb + 1] == s_pre[lb]) continue;
      const size_t w0 = (size_t)lb * kListWords + 2 * tid;
      uint64_t w[2] = {0ull, 0ull};
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (w0 + k < nwords) w[k] = __ldg(v.bits + w0 + k);
      unsigned total;
      unsigned idx = s_pre[lb] + before((unsigned)(__popcll(w[0]) + __popcll(w[1])), total) - idx0;
#pragma unroll
      for (int k = 0; k < 2; ++k)
        for (uint64_t q = w[k]; q; q &= q - 1ull, ++idx)
          if (idx < (unsigned)count) {  // (idx wraps below idx0)
            const size_t t = w0 + k;
            const int b = (int)(t / (unsigned)n);
            s_site[idx] = (uint32_t)(t % (unsigned)n) |
                          ((uint32_t)(b * kBand + __ffsll((long long)q) - 1) << 16);
          }
    }
    __syncthreads();
    if (warp < count) {
      const uint32_t e = s_site[warp];
      const int sx = (int)(e & 0x7fffu), sy = (int)(e >> 16);
      const int h = a.hint[(size_t)sy * n + sx];
      cell_sums_warp(a, v.bits, n, sx, sy, h ? h : v.W0, v.rb, lane, scratch[warp]);
    }
    __syncthreads();
    if (warp == 0) {
      CellSums cs = fold_block(scratch, count, lane);
      if (lane < count) {
        cs.r2 = scratch[lane].r2;
        uint32_t e = s_site[lane];
        const int sx = (int)(e & 0x7fffu), sy = (int)(e >> 16);
        e |= (uint32_t)((a.fixed_bits[(size_t)(sy / kBand) * n + sx] >> (sy % kBand)) & 1ull) << 15;
        float eh = 0.f, el = 0.f;
        dfa(eh, el, cs.eh, cs.el);
        const unsigned mv = move_site(a, v, e, sx, sy, cs);
        a.sitev[idx0 + lane] =
            make_float4(eh, el, __uint_as_float((unsigned)cs.r2), __uint_as_float(mv));
      }
      __syncwarp();
      float eh, el;
      unsigned r2, mv;
      const unsigned g = idx0 / 32;
      if (!fold_last && group_done(a, v, g, (unsigned)count, lane, eh, el, r2, mv)) {
        warp_reduce(eh, el, r2, mv);
        if (lane == 0) a.gslot[g] = make_float4(eh, el, __uint_as_float(r2), __uint_as_float(mv));
      }
    }
    __syncthreads();  // the scratch is free again
  }
  if (tid == 0) s_last = add_release(&st->done_blocks) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  float4 *gt = reinterpret_cast<float4 *>(scratch);
  if (fold_last) {  // four groups a warp, their loads in flight together
    float eh[4], el[4];
    unsigned r2[4], mv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      site_values(a, v, warp + k * kBlockSites, lane, eh[k], el[k], r2[k], mv[k]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned g = warp + k * kBlockSites;
      if (g >= v.ngroups) break;
      warp_reduce(eh[k], el[k], r2[k], mv[k]);
      if (lane == 0)
        gt[g] = make_float4(eh[k], el[k], __uint_as_float(r2[k]), __uint_as_float(mv[k]));
    }
    __syncthreads();
  }
  if (warp == 0) {
    if (lane == 0) st->snap_count = st->list_count = v.nsites;
    few_slots<0>(a, v, fold_last ? gt : a.gslot, lane);
  }
}

// One chart.  MODE 0: one Lloyd iteration (sums, move, energy, schedule).
// MODE 1: moments only (gcvt_ctx_moments); the sites do not move.
// MODE 2: the learned step's features of the sites (LevelBufs::feat);
//         nothing moves.
// MODE 4: MODE 0 and the features, for a jump from these sites.
// MODE 5: MODE 0 for the jumped sites, and the gate's decision
//         (DevState::gate_accept); when no jump was proposed
//         (DevState::gate_active 0), exactly MODE 0.
template <int MODE>
__global__ void __launch_bounds__(32, 32) k_cell(LevelBufs a, double *out4) {
  DevState *st = a.st;
  constexpr bool kMoves = MODE == 0 || MODE == 4 || MODE == 5;
  if (kMoves && st->snap_stopped) return;
  const int lane = threadIdx.x;
  const IterView v = iter_view(a);
  if (MODE != 1 && v.ngroups == 0) {  // no sites: the schedule still advances
    if (blockIdx.x == 0 && lane == 0) pass_done<MODE>(st, 0.0, 0u, 0u, a.n, v.cur);
    return;
  }
  for (bool first = true;; first = false) {
    const unsigned g = next_item(&st->ticket, first, lane);
    if (g >= v.ngroups) break;
    cell_group<MODE>(a, v, g, lane, out4);
  }
}

// Many charts, one launch: the groups of all charts that have not stopped form
// one sequence (group offsets per chart from k_list_batch, gofs[c] .. gofs[c+1]),
// handed out by one ticket; each chart keeps its own state, reduction and
// schedule, so a chart's iteration is the same as in k_cell.  MODE 0, 4, 5 as
// in k_cell.  A warp keeps its chart's buffer pointers in shared memory (read
// through the descriptor in global memory, they cost a reload after every store).
template <int MODE>
__global__ void __launch_bounds__(32, 32) k_cell_batch(const LevelBufs *__restrict__ charts,
                                                       int nchart,
                                                       const unsigned *__restrict__ gofs,
                                                       unsigned *ticket) {
  __shared__ LevelBufs a;
  static_assert(sizeof(LevelBufs) % 8 == 0, "copied in 8-byte words");
  const int lane = threadIdx.x;
  if (blockIdx.x == 0) {  // running charts without sites: the schedule still advances
    for (int c = lane; c < nchart; c += 32) {
      DevState *st = charts[c].st;
      if (!st->snap_stopped && st->snap_count == 0)
        pass_done<MODE>(st, 0.0, 0u, 0u, charts[c].n, st->snap_cur);
    }
  }
  const unsigned total = gofs[nchart];
  int chart = -1;
  IterView v{};
  unsigned g0 = 0;
  for (bool first = true;; first = false) {
    const unsigned g = next_item(ticket, first, lane);
    if (g >= total) break;
    int lo = 0, hi = nchart - 1;  // the chart c with gofs[c] <= g < gofs[c + 1]
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(gofs + mid) <= g) lo = mid;
      else hi = mid - 1;
    }
    if (lo != chart) {
      chart = lo;
      __syncwarp();
      for (int k = lane; k < (int)(sizeof(LevelBufs) / 8); k += 32)
        reinterpret_cast<unsigned long long *>(&a)[k] =
            __ldg(reinterpret_cast<const unsigned long long *>(charts + chart) + k);
      __syncwarp();
      v = iter_view(a);
      g0 = __ldg(gofs + chart);
    }
    cell_group<MODE>(a, v, g - g0, lane, nullptr);
  }
}

// Block `blk` of a chart's site list: the sites of bitmap words
// [blk kListWords, (blk+1) kListWords) in bitmap order (word by word, bits in
// row order) with the fixed flag, at the offset the per-block counts give.
// The chart's last block records the list length.  clear: also zero the block's
// words (and count) of the bitmap the next iteration writes -- nobody reads them in
// this one -- unless a jump is being judged (the bitmap then holds the plain step's
// sites until the gate decides).
__device__ void list_block(const LevelBufs &a, unsigned blk, unsigned nblk, bool clear) {
  constexpr int kPer = kListWords / 256;
  __shared__ unsigned wsum[8];
  __shared__ unsigned base_s;
  DevState *st = a.st;
  const int n = a.n;
  const int cur = st->cur;
  const uint64_t *bits = bits_at(a, cur);
  const unsigned *counts = counts_at(a, cur);
  const size_t nwords = (size_t)(n / kBand) * n;
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  if (blk == 0 && tid == 0) {
    st->done_blocks = 0u;
    take_snapshot(st);
  }
  // offset of this block: the counts of the blocks before it
  unsigned pre = 0;
  for (unsigned k = tid; k < blk; k += 256) pre += counts[k];
  pre = __reduce_add_sync(0xffffffffu, pre);
  if (lane == 0) wsum[wib] = pre;
  __syncthreads();
  if (tid == 0) {
    unsigned s = 0;
    for (int k = 0; k < 8; ++k) s += wsum[k];
    base_s = s;
  }
  __syncthreads();
  const unsigned base = base_s;
  // this thread's words and their sites
  const size_t w0 = (size_t)blk * kListWords + (size_t)tid * kPer;
  if (clear && !st->gate_active) {
    const int z = cur == 0 ? 2 : cur - 1;
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (w0 + k < nwords) bits_at(a, z)[w0 + k] = 0ull;
    if (tid == 0) counts_at(a, z)[blk] = 0u;
  }
  uint64_t w[kPer];
  unsigned cnt = 0;
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    w[k] = (w0 + k < nwords) ? bits[w0 + k] : 0ull;
    cnt += __popcll(w[k]);
  }
  // exclusive scan of cnt over the block
  unsigned incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  __syncthreads();  // every thread has read base_s / wsum
  if (lane == 31) wsum[wib] = incl;
  __syncthreads();
  unsigned woff = 0, total = 0;
  for (int k = 0; k < 8; ++k) {
    const unsigned v = wsum[k];
    if (k < wib) woff += v;
    total += v;
  }
  unsigned pos = base + woff + incl - cnt;
  const unsigned cap = (unsigned)n * (unsigned)n;  // list capacity at this size
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    uint64_t word = w[k];
    if (!word) continue;
    const size_t t = w0 + k;
    const int x = (int)(t % (unsigned)n), band = (int)(t / (unsigned)n);
    const uint64_t fw = a.fixed_bits[t];
    while (word) {
      const int i = __ffsll((long long)word) - 1;
      word &= word - 1ull;
      if (pos < cap)
        a.list[pos] = (uint32_t)x | ((uint32_t)(band * kBand + i) << 16) |
                      ((uint32_t)((fw >> i) & 1ull) << 15);
      ++pos;
    }
  }
  if (blk == nblk - 1 && tid == 0) st->list_count = st->snap_count = (int)min(base + total, cap);
  __syncthreads();  // the shared scratch may be reused by the caller
}

// One chart's site list; also rearms the chart's ticket.  respect_stop = 0
// lists a stopped chart too (moments, point extraction) and marks the
// snapshot running.
__global__ void __launch_bounds__(256) k_list(LevelBufs a, int respect_stop) {
  DevState *st = a.st;
  if (respect_stop && st->stopped) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->snap_stopped = 1;
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) st->ticket = 0u;
  list_block(a, blockIdx.x, gridDim.x, respect_stop != 0);
  if (!respect_stop && blockIdx.x == 0 && threadIdx.x == 0) st->snap_stopped = 0;
}

// The site lists of many charts: chart c owns blocks lofs[c] .. lofs[c+1].  The
// blocks after those lay out the group offsets of the charts that run (gofs) for
// k_cell_batch and rearm its ticket, from the charts' block counts alone: a warp per
// chart adds them up, the last of these blocks scans the charts.  (With every list
// block counting itself finished and one thread walking the charts at the end, 64
// charts took 42 us; this way 20.)
constexpr int kChartsPerBlock = 8;

__global__ void __launch_bounds__(256) k_list_batch(const LevelBufs *__restrict__ charts,
                                                    int nchart,
                                                    const unsigned *__restrict__ lofs,
                                                    unsigned *gofs, unsigned *done,
                                                    unsigned *ticket) {
  const unsigned nlist = __ldg(lofs + nchart);
  if (blockIdx.x < nlist) {
    int lo = 0, hi = nchart - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(lofs + mid) <= blockIdx.x) lo = mid;
      else hi = mid - 1;
    }
    const LevelBufs &a = charts[lo];
    const unsigned blk = blockIdx.x - __ldg(lofs + lo);
    if (!a.st->stopped) list_block(a, blk, __ldg(lofs + lo + 1) - __ldg(lofs + lo), true);
    else if (blk == 0 && threadIdx.x == 0) a.st->snap_stopped = 1;
    return;
  }
  __shared__ bool is_last;
  __shared__ unsigned ws[8];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int mc = (int)(blockIdx.x - nlist) * kChartsPerBlock + wib;
  if (mc < nchart) {
    const LevelBufs &a = charts[mc];
    unsigned sum = 0;
    if (!a.st->stopped) {
      const unsigned *counts = counts_at(a, a.st->cur);
      for (unsigned k = lane; k < __ldg(lofs + mc + 1) - __ldg(lofs + mc); k += 32) sum += counts[k];
    }
    sum = min(__reduce_add_sync(0xffffffffu, sum), (unsigned)a.n * (unsigned)a.n);
    if (lane == 0) gofs[mc] = (sum + 31) / 32;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = atomicAdd(done, 1u) == gridDim.x - nlist - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  unsigned acc = 0;
  for (int c0 = 0; c0 < nchart; c0 += 256) {  // 256 charts at a time
    const int c = c0 + threadIdx.x;
    const unsigned mine = c < nchart ? __ldcg(gofs + c) : 0u;
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) ws[wib] = incl;
    __syncthreads();
    unsigned before = acc;
    for (int k = 0; k < 8; ++k) {
      if (k < wib) before += ws[k];
      acc += ws[k];
    }
    if (c < nchart) gofs[c] = before + incl - mine;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    gofs[nchart] = acc;
    *ticket = 0u;
    *done = 0u;
  }
}

// Per-block site counts of the current bitmap (for the first k_list of a
// level; afterwards k_cell counts the sites it places).
__global__ void __launch_bounds__(256) k_count(LevelBufs a) {
  constexpr int kPer = kListWords / 256;
  __shared__ unsigned wsum[8];
  const int n = a.n;
  const int cur = a.st->cur;
  const uint64_t *bits = bits_at(a, cur);
  unsigned *counts = counts_at(a, cur);
  const size_t nwords = (size_t)(n / kBand) * n;
  const size_t w0 = (size_t)blockIdx.x * kListWords + (size_t)threadIdx.x * kPer;
  unsigned cnt = 0;
  for (int k = 0; k < kPer; ++k)
    if (w0 + k < nwords) cnt += __popcll(bits[w0 + k]);
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned s = 0;
    for (int k = 0; k < 8; ++k) s += wsum[k];
    counts[blockIdx.x] = s;
  }
}

// Covering bound from a label grid: cover = ceil(sqrt(max |p - label(p)|^2))
// over the pixels of the density's row support.  One block per row.
// hint[pid] = max(hint[pid], b) on the byte inside its 32-bit word.  Each
// failed compare-and-swap means another byte of the word grew, so the loop is
// short; past the limit the hint just stays lower (a wider first window).
__device__ __forceinline__ void hint_max(uint8_t *hint, size_t pid, unsigned b) {
  unsigned *word = reinterpret_cast<unsigned *>(hint + (pid & ~(size_t)3));
  const int sh = (int)(pid & 3) * 8;
  unsigned old = *reinterpret_cast<volatile unsigned *>(word);
  for (int k = 0; k < 64 && ((old >> sh) & 0xffu) < b; ++k) {
    const unsigned prev = atomicCAS(word, old, (old & ~(0xffu << sh)) | (b << sh));
    if (prev == old) break;
    old = prev;
  }
}

// Covering bound of a label grid (max over density pixels of the squared
// distance to their site), and each site's first window: 2 R + slack with R
// the largest distance from the site to a density pixel of its cell (hint at
// the site pixel, zeroed before), so the first iteration after a load needs
// no window retries.
__global__ void __launch_bounds__(256) k_cover(LevelBufs a) {
  const int n = a.n, y = blockIdx.x;
  const int2 yr = *a.sup_range;
  const unsigned slack = (unsigned)a.st->hint_slack;
  const int lane = threadIdx.x & 31;
  unsigned m = 0;
  if (y >= yr.x && y < yr.y) {
    const int2 s = a.support[y];
    const uint32_t *row = a.labels + (size_t)y * n;
    // 32 consecutive pixels per warp step: the lanes holding one site's label
    // (runs along the row) reduce together, one of them updates the hint
    for (int base = s.x + (int)(threadIdx.x & ~31u); base < s.y; base += blockDim.x) {
      const int x = base + lane;
      const uint32_t v = x < s.y ? row[x] : kMarkerWord;
      const int lx = (int16_t)(v & 0xffffu), ly = (int16_t)(v >> 16);
      const bool site = lx != kMarker;
      const unsigned d2 = site ? (unsigned)((x - lx) * (x - lx) + (y - ly) * (y - ly)) : 0u;
      m = max(m, d2);
      const unsigned grp = __match_any_sync(0xffffffffu, site ? v : kMarkerWord);
      const unsigned g2 = __reduce_max_sync(grp, d2);
      if (site && lane == __ffs(grp) - 1) {
        // ceil(sqrt(g2)) from a float square root, one integer correction up
        unsigned r = (unsigned)sqrtf((float)g2);
        if (r * r < g2) ++r;
        const unsigned b = min(2u * r + slack, 255u);
        const size_t pid = (size_t)ly * n + lx;
        if (a.hint[pid] < b) hint_max(a.hint, pid, b);
      }
    }
  }
  // the block's maximum, then one atomic per block (one per warp onto the
  // single accumulator serialised at the L2)
  __shared__ unsigned wmax[8];
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) wmax[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = max(m, wmax[w]);
    if (m) atomicMax(&a.st->cover_acc, m);
  }
}
__global__ void k_cover_finish(LevelBufs a) {
  DevState *st = a.st;
  st->cover = min(isqrt_ceil((int)st->cover_acc), 2 * a.n);
  st->cover_acc = 0;
}

cudaError_t launch_cover(const LevelBufs &b, cudaStream_t s) {
  k_cover<<<b.n, 256, 0, s>>>(b);
  k_cover_finish<<<1, 1, 0, s>>>(b);
  return cudaGetLastError();
}

size_t list_blocks(int n) {
  const size_t nwords = (size_t)(n / kBand) * n;
  return (nwords + kListWords - 1) / kListWords;
}

size_t cell_groups(int n) { return ((size_t)n * n + 31) / 32; }

cudaError_t launch_list(const LevelBufs &b, int respect_stop, cudaStream_t s) {
  k_list<<<(unsigned)list_blocks(b.n), 256, 0, s>>>(b, respect_stop);
  return cudaGetLastError();
}

cudaError_t launch_count(const LevelBufs &b, cudaStream_t s) {
  k_count<<<(unsigned)list_blocks(b.n), 256, 0, s>>>(b);
  return cudaGetLastError();
}

// Persistent grid of the Lloyd kernel: every warp that fits, per device.
static int g_cell_grid[64] = {};
static int g_warp_grid[64] = {};  // k_cell_warp: its own carveout and occupancy

cudaError_t cells_configure() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (g_cell_grid[dev]) return cudaSuccess;
  int sms = 0, per0 = 0, per1 = 0;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return e;
  // candidates and rows live in local memory: shared memory only for the
  // 1 KB the runtime reserves per block (32 blocks per SM), the rest as L1
  const int carve = 15;
  if ((e = cudaFuncSetAttribute(k_cell<0>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                carve)) != cudaSuccess)
    return e;
  if ((e = cudaFuncSetAttribute(k_cell<1>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                carve)) != cudaSuccess)
    return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per0, k_cell<0>, 32, 0)) != cudaSuccess)
    return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per1, k_cell<1>, 32, 0)) != cudaSuccess)
    return e;
  // every persistent variant shares the grid: the fewest blocks any of them fits
  auto fit = [&](auto fn) -> cudaError_t {
    int per = 0;
    cudaError_t r = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, carve);
    if (r == cudaSuccess) r = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, 32, 0);
    if (r == cudaSuccess) per0 = min(per0, per);
    return r;
  };
  for (auto fn : {k_cell_batch<0>, k_cell_batch<4>, k_cell_batch<5>})
    if ((e = fit(fn)) != cudaSuccess) return e;
  for (auto fn : {k_cell<2>, k_cell<4>, k_cell<5>})
    if ((e = fit(fn)) != cudaSuccess) return e;
  // one site per warp: a block's shared scratch (candidates, chunk sums) is 34 KB
  int perw = 0;
  for (auto fn : {k_cell_warp<0>, k_cell_warp<4>, k_cell_warp<5>}) {
    int per = 0;
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 64)) !=
        cudaSuccess)
      return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, 32 * kBlockSites, 0)) !=
        cudaSuccess)
      return e;
    perw = perw ? min(perw, per) : per;
  }
  {
    int per = 0;
    if ((e = cudaFuncSetAttribute(k_cell_few, cudaFuncAttributePreferredSharedMemoryCarveout, 70)) !=
        cudaSuccess)
      return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cell_few, 32 * kBlockSites, 0)) !=
        cudaSuccess)
      return e;
    perw = min(perw, per);
  }
  g_warp_grid[dev] = sms * max(1, perw);
  g_cell_grid[dev] = sms * max(1, min(per0, per1));
  return cudaSuccess;
}

cudaError_t launch_list_batch(const LevelBufs *charts, int nchart, const unsigned *lofs,
                              unsigned nblocks, unsigned *gofs, unsigned *done, unsigned *ticket,
                              cudaStream_t s) {
  const unsigned extra = (unsigned)((nchart + kChartsPerBlock - 1) / kChartsPerBlock);
  k_list_batch<<<nblocks + extra, 256, 0, s>>>(charts, nchart, lofs, gofs, done, ticket);
  return cudaGetLastError();
}

cudaError_t launch_cells_batch(const LevelBufs *charts, int nchart, const unsigned *gofs,
                               unsigned *ticket, cudaStream_t s, int mode) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !g_cell_grid[dev]) return cudaErrorNotReady;
  const int grid = g_cell_grid[dev];
  switch (mode) {
    case 4: k_cell_batch<4><<<grid, 32, 0, s>>>(charts, nchart, gofs, ticket); break;
    case 5: k_cell_batch<5><<<grid, 32, 0, s>>>(charts, nchart, gofs, ticket); break;
    default: k_cell_batch<0><<<grid, 32, 0, s>>>(charts, nchart, gofs, ticket);
  }
  return cudaGetLastError();
}

int cells_default_grid() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  return g_cell_grid[dev];
}

// One plain Lloyd iteration: the site list and the cells, or, for few sites, one
// launch.
cudaError_t launch_iteration(const LevelBufs &b, cudaStream_t s, int grid) {
  if (b.few && b.sitev) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64 || !g_warp_grid[dev]) return cudaErrorNotReady;
    int wg = min((b.few + kBlockSites - 1) / kBlockSites, g_warp_grid[dev]);
    if (grid > 0) wg = min(wg, grid / kBlockSites);
    k_cell_few<<<max(1, wg), 32 * kBlockSites, 0, s>>>(b);
    return cudaGetLastError();
  }
  const cudaError_t e = launch_list(b, 1, s);
  return e != cudaSuccess ? e : launch_cells(b, 0, nullptr, s, grid);
}

// grid: the persistent grid in blocks (0: every block that fits).
cudaError_t launch_cells(const LevelBufs &b, int moments_only, double *out4, cudaStream_t s,
                         int grid) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !g_cell_grid[dev]) return cudaErrorNotReady;
  if (grid <= 0 || grid > g_cell_grid[dev]) grid = g_cell_grid[dev];
  if ((moments_only == 0 || moments_only == 4 || moments_only == 5) && b.sitev && b.gcnt) {
    // (grid counts warps)
    const int wg = max(1, min(grid / kBlockSites, g_warp_grid[dev])), wt = 32 * kBlockSites;
    if (moments_only == 4) k_cell_warp<4><<<wg, wt, 0, s>>>(b);
    else if (moments_only == 5) k_cell_warp<5><<<wg, wt, 0, s>>>(b);
    else k_cell_warp<0><<<wg, wt, 0, s>>>(b);
    return cudaGetLastError();
  }
  switch (moments_only) {
    case 1: k_cell<1><<<grid, 32, 0, s>>>(b, out4); break;
    case 2: k_cell<2><<<grid, 32, 0, s>>>(b, out4); break;
    case 4: k_cell<4><<<grid, 32, 0, s>>>(b, out4); break;
    case 5: k_cell<5><<<grid, 32, 0, s>>>(b, out4); break;
    default: k_cell<0><<<grid, 32, 0, s>>>(b, out4);
  }
  return cudaGetLastError();
}

}  // namespace cvtgb
