// label_tiles.cu -- the exact labels of a site bitmap tile by tile: per 16 x 16
// pixels the few sites that can own any of them, then every pixel against those.
//
// The labels are labeller.cu's (PBA+'s: nearest site, ties to the smaller x, then
// the 64-row band rule for a mirror pair), as one total order per pixel: squared
// distance, x, and for sites of one column first those in bands up to the pixel's
// own from the lowest one up, then those below the band -- two sites of a column tie
// only as a mirror pair, whose lower site wins exactly when it lies in the pixel's
// band.  Candidates listed in that order carry their position in the low byte of
// the key, so a pixel's owner is one integer minimum.
//
// Which sites: let s* be the site nearest to the tile's centre.  A site t with
// |c - t| > |c - s*| at all four corners c loses to s* everywhere in the tile (the
// difference of the two squared distances is linear).  So the candidates are the
// sites inside or on one of the four circles around the corners through s*.
//
//   * k_label_tiles: a warp per tile.  It reads the bitmap of the tile and the 16
//     pixels around it; if the four circles stay inside that window, the sites
//     there are all there are.
//   * k_label_far: a block per 64 x 64 pixels holding a tile that was not so (far
//     from any site, or crowded).  It finds the nearest site to the block's centre
//     over the occupied 64 x 64 blocks, gathers the sites that can own any of its
//     pixels by the same test, and prunes that list for each of its open tiles.
//   * the row pass (labeller.cu) does grids up to 512 x 512 and crowded ones, and of
//     the others the rows of a band (64 rows) that holds a crowded 64 x 64 block, which
//     the tiles skip, or one that does not fit its lists (by_rows).
//
// What bounds it is issue slots: half of a CVT tile's warp instructions are its 15
// candidates x 256 pixels.  The row pass this replaces spent 330 per row and 32
// columns.  130,000 sites at 3328^2: 161 -> 81 us (tiles 40, blocks 37); a million at
// 8192^2: 1.21 -> 0.39 ms (262, 117).
#include "gcvt_internal.cuh"

namespace cvtgb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kT = 16;              // tile side
constexpr int kMargin = 16;         // window around a tile
constexpr int kWin = kT + 2 * kMargin;
constexpr int kTileWarps = 4;       // tiles per block
constexpr int kGather = 512;        // sites of a window
constexpr int kCand = 128;          // candidates of a tile (below 256: the key's low byte)
constexpr int kFarMacros = 1024;    // 64 x 64 blocks looked at
constexpr int kFarSites = 2048;     // sites gathered for one
constexpr int kCrowdBlock = 380;    // sites of a 64 x 64 block: above it the row pass

// A candidate t relative to a reference site r: |p - t|^2 - |p - r|^2 = c + p.x ax +
// p.y ay for the pixel p of the tile, and t's label.
__device__ __forceinline__ int4 cand_entry(int tx, int ty, int rx, int ry, uint32_t label) {
  return make_int4(-2 * (tx - rx), -2 * (ty - ry), tx * tx + ty * ty - rx * rx - ry * ry,
                   (int)label);
}

// The labels of the tile at (x0, y0) from its m candidates in tie order: lane l
// takes column l % 16 of the rows 8 (l / 16) .. + 7.  The differences stay below 2^22
// (the candidates pass the corner test against the reference), so the key fits.
__device__ __forceinline__ void eval_tile(const int4 *cand, int m, int x0, int y0, int n,
                                          uint32_t *__restrict__ labels) {
  const int lane = threadIdx.x & 31, x = lane & 15, y = (lane >> 4) * 8;
  int best[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) best[j] = 0x7fffffff;
  for (int k = 0; k < m; ++k) {
    const int4 q = cand[k];
    int key = (q.z + x * q.x + y * q.y) * 256 + k;
    const int step = q.y * 256;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      best[j] = min(best[j], key);
      key += step;
    }
  }
  uint32_t *out = labels + (size_t)(y0 + y) * n + x0 + x;
#pragma unroll
  for (int j = 0; j < 8; ++j) out[(size_t)j * n] = (uint32_t)cand[best[j] & 255].w;
}

// Squared distances from the corners (0 or s, 0 or s) to (x, y), and whether one
// is at most r2's.
__device__ __forceinline__ int4 corner_d2(int x, int y, int s) {
  const int ax = x * x, bx = (x - s) * (x - s), ay = y * y, by = (y - s) * (y - s);
  return make_int4(ax + ay, bx + ay, ax + by, bx + by);
}
__device__ __forceinline__ bool corner_in(int x, int y, int s, const int4 &r2) {
  const int4 d = corner_d2(x, y, s);
  return d.x <= r2.x || d.y <= r2.y || d.z <= r2.z || d.w <= r2.w;
}

// Occupied 64 x 64 blocks (a bitmap word per column) as a bit mask per row of
// them, whether one is crowded, no open tiles.  One block per row.
__global__ void __launch_bounds__(1024) k_label_occ(LevelBufs a) {
  __shared__ unsigned mask[4], crowded;
  const int M = a.n / kBand, row = blockIdx.x, lane = threadIdx.x & 31;
  if (threadIdx.x < 4) mask[threadIdx.x] = 0u;
  if (threadIdx.x == 0) crowded = 0u;
  if ((int)threadIdx.x < M) a.open_tiles[row * M + threadIdx.x] = 0u;
  __syncthreads();
  for (int m = threadIdx.x >> 5; m < M; m += 32) {
    const uint64_t *w = cur_bits(a) + (size_t)row * a.n + m * kBand;
    const int sites = __reduce_add_sync(kFull, __popcll(w[lane]) + __popcll(w[lane + 32]));
    if (lane == 0 && sites) atomicOr(mask + (m >> 5), 1u << (m & 31));
    if (lane == 0 && sites > kCrowdBlock) crowded = 1u;
  }
  __syncthreads();
  if (threadIdx.x == 0) a.st->band_rows[row] = (uint8_t)crowded;
  if (threadIdx.x < 4) a.occ[4 * row + threadIdx.x] = mask[threadIdx.x];
}

__global__ void __launch_bounds__(32 * kTileWarps) k_label_tiles(LevelBufs a) {
  __shared__ unsigned short s_site[kTileWarps][kGather];  // (dx + 16) | (dy + 16) << 8
  __shared__ int4 s_cand[kTileWarps][kCand];
  const int n = a.n, lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int x0 = (blockIdx.x * kTileWarps + wib) * kT, y0 = blockIdx.y * kT;
  unsigned short *site = s_site[wib];
  int4 *cand = s_cand[wib];
  const uint64_t *bits = cur_bits(a);
  // the window's sites, column by column, each column in tie order
  const int r0 = y0 - kMargin, bl = r0 >> 6, sh = r0 & 63;  // bl = -1 above the grid
  const int lim = min(kBand * ((y0 >> 6) + 1) - r0, kWin);  // window rows up to the tile's band's end
  const uint64_t upper = (1ull << lim) - 1ull;
  uint64_t col[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = lane + 32 * h, x = x0 - kMargin + c;
    uint64_t w = 0;
    if (c < kWin && x >= 0 && x < n) {
      if (bl >= 0) w = __ldg(bits + (size_t)bl * n + x) >> sh;
      if (sh > 64 - kWin && (bl + 1) * kBand < n)
        w |= __ldg(bits + (size_t)(bl + 1) * n + x) << (64 - sh);
    }
    col[h] = w & ((1ull << kWin) - 1ull);
  }
  if (by_rows(a, y0 / kBand)) return;  // (beside the loads above)
  int cnt = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int mine = __popcll(col[h]);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += u;
    }
    int pos = cnt + incl - mine;
    uint64_t w = col[h] & upper;
    const unsigned dx = (unsigned)(lane + 32 * h);
    while (w) {
      const int i = 63 - __clzll((long long)w);
      w ^= 1ull << i;
      if (pos < kGather) site[pos] = (unsigned short)(dx | (i << 8));
      ++pos;
    }
    w = col[h] & ~upper;
    while (w) {
      const int i = __ffsll((long long)w) - 1;
      w &= w - 1ull;
      if (pos < kGather) site[pos] = (unsigned short)(dx | (i << 8));
      ++pos;
    }
    cnt += __shfl_sync(kFull, incl, 31);
  }
  bool ok = cnt > 0 && cnt <= kGather;
  int m = 0;
  if (ok) {
    __syncwarp();
    // the site nearest to the centre (7.5, 7.5)
    unsigned near = 0xffffffffu;
    for (int k = lane; k < cnt; k += 32) {
      const int v = site[k], dx = (v & 0xff) - kMargin, dy = (v >> 8) - kMargin;
      const int ex = 2 * dx - (kT - 1), ey = 2 * dy - (kT - 1);
      near = min(near, ((unsigned)(ex * ex + ey * ey) << 9) | (unsigned)k);
    }
    near = __reduce_min_sync(kFull, near);
    const int sv = site[near & 511u], sx = (sv & 0xff) - kMargin, sy = (sv >> 8) - kMargin;
    const int4 r2 = corner_d2(sx, sy, kT - 1);
    // a site outside the window is at least kMargin + 1 from every corner
    ok = max(max(r2.x, r2.y), max(r2.z, r2.w)) < (kMargin + 1) * (kMargin + 1);
    if (ok) {
      for (int k0 = 0; k0 < cnt; k0 += 32) {
        const int k = k0 + lane, v = k < cnt ? site[k] : 0;
        const int dx = (v & 0xff) - kMargin, dy = (v >> 8) - kMargin;
        const bool keep = k < cnt && corner_in(dx, dy, kT - 1, r2);
        const unsigned km = __ballot_sync(kFull, keep);
        const int pos = m + __popc(km & ((1u << lane) - 1u));
        if (keep && pos < kCand)
          cand[pos] = cand_entry(dx, dy, sx, sy, pack_xy(x0 + dx, y0 + dy));
        m += __popc(km);
      }
      ok = m <= kCand;
    }
  }
  if (!ok) {  // left to k_label_far
    if (lane == 0) {
      const int M = n / kBand;
      atomicOr(a.open_tiles + (y0 / kBand) * M + x0 / kBand,
               1u << ((y0 % kBand) / kT * 4 + (x0 % kBand) / kT));
    }
    return;
  }
  __syncwarp();
  eval_tile(cand, m, x0, y0, n, a.labels);
}

__device__ __forceinline__ int box_gap(int p, int lo, int hi) { return max(max(lo - p, p - hi), 0); }

template <int kFarThreads>
__global__ void __launch_bounds__(kFarThreads) k_label_far(LevelBufs a) {
  __shared__ uint32_t s_site[kFarSites];      // x | y << 16
  __shared__ unsigned short s_macro[kFarMacros];
  __shared__ int4 s_cand[kFarThreads / 32][kCand];
  __shared__ uint32_t s_key[kFarThreads / 32][kCand], s_pos[kFarThreads / 32][kCand];
  __shared__ unsigned s_min, s_cnt;
  __shared__ unsigned long long s_near;
  const int n = a.n, M = n / kBand, tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
  const int mx = blockIdx.x, my = blockIdx.y;
  const unsigned open = a.open_tiles[my * M + mx];
  // (another block may be flagging the band: one answer for the whole block)
  if (!open || __syncthreads_or(by_rows(a, my))) return;
  const int x0 = mx * kBand, y0 = my * kBand;
  const uint64_t *bits = cur_bits(a);
  if (tid == 0) {
    s_min = 0xffffffffu;
    s_cnt = 0u;
    s_near = ~0ull;
  }
  __syncthreads();
  // an upper bound on the distance from the centre to a site (doubled units: the
  // centre is at (63, 63)): the far corner of the nearest occupied blocks
  const int cx = 2 * x0 + 63, cy = 2 * y0 + 63;
  static_assert(kMaxN / kBand <= kFarThreads, "a thread per row of blocks");
  uint64_t olo = 0, ohi = 0;  // this thread's row of occupied blocks
  if (tid < M) {
    const uint4 q = __ldg(reinterpret_cast<const uint4 *>(a.occ) + tid);
    olo = q.x | ((uint64_t)q.y << 32), ohi = q.z | ((uint64_t)q.w << 32);
  }
  unsigned u = 0xffffffffu;
  if (olo | ohi) {
    // the nearest occupied blocks of the row on either side of column mx
    const uint64_t le_lo = mx >= 63 ? ~0ull : (2ull << mx) - 1ull,
                   le_hi = mx < 64 ? 0ull : (mx == 127 ? ~0ull : (2ull << (mx - 64)) - 1ull);
    const uint64_t ll = olo & le_lo, lh = ohi & le_hi, rl = olo & ~le_lo, rh = ohi & ~le_hi;
    const int kl = lh ? 127 - __clzll((long long)lh) : (ll ? 63 - __clzll((long long)ll) : -1);
    const int kr = rl ? __ffsll((long long)rl) - 1 : (rh ? 63 + __ffsll((long long)rh) : -1);
    auto far2 = [&](int kx) {
      const int bx = 2 * kBand * kx, by = 2 * kBand * tid;
      const int dx = max(abs(cx - bx), abs(bx + 126 - cx)), dy = max(abs(cy - by), abs(by + 126 - cy));
      return (unsigned)(dx * dx + dy * dy);
    };
    if (kl >= 0) u = far2(kl);
    if (kr >= 0) u = min(u, far2(kr));
  }
  u = __reduce_min_sync(kFull, u);
  if (lane == 0) atomicMin(&s_min, u);
  __syncthreads();
  u = s_min;
  if (u == 0xffffffffu) {  // no site anywhere
    for (int t = wib; t < 16; t += kFarThreads / 32) {
      if (!((open >> t) & 1u)) continue;
      uint32_t *out = a.labels + (size_t)(y0 + t / 4 * kT) * n + x0 + t % 4 * kT;
      for (int k = lane; k < kT * kT; k += 32) out[(size_t)(k / kT) * n + k % kT] = kMarkerWord;
    }
    return;
  }
  // the blocks within that distance, and the nearest site in them
  // (reach: blocks farther than that many rows or columns from this one are out)
  auto list_macros = [&](int reach, auto &&want) -> int {
    if (abs(tid - my) <= reach) {
      const int k0 = max(mx - reach, 0), k1 = min(mx + reach, M - 1);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint64_t w = h ? ohi : olo;
        const int f = max(k0 - 64 * h, 0), t = min(k1 - 64 * h, 63);
        w = f > t ? 0ull : w & (t == 63 ? ~0ull : (2ull << t) - 1ull) & ~((1ull << f) - 1ull);
        while (w) {
          const int kx = 64 * h + __ffsll((long long)w) - 1;
          w &= w - 1ull;
          if (!want(kx, tid)) continue;
          const unsigned p = atomicAdd(&s_cnt, 1u);
          if (p < kFarMacros) s_macro[p] = (unsigned short)(tid * M + kx);
        }
      }
    }
    __syncthreads();
    const int c = (int)s_cnt;
    __syncthreads();
    return c;
  };
  auto each_site = [&](int count, auto &&f) {  // f(x, y) of the listed blocks' sites
    for (int q = wib; q < count; q += kFarThreads / 32) {
      const int k = s_macro[q], bx = (k % M) * kBand, by = (k / M) * kBand;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int x = bx + lane + 32 * h;
        uint64_t w = __ldg(bits + (size_t)(k / M) * n + x);
        while (w) {
          const int i = __ffsll((long long)w) - 1;
          w &= w - 1ull;
          f(x, by + i);
        }
      }
    }
  };
  int count = list_macros((int)(sqrtf((float)u) / (2 * kBand)) + 2, [&](int kx, int ky) {
    const int dx = box_gap(cx, 2 * kBand * kx, 2 * kBand * kx + 126),
              dy = box_gap(cy, 2 * kBand * ky, 2 * kBand * ky + 126);
    return (unsigned)(dx * dx + dy * dy) <= u;
  });
  bool ok = count <= kFarMacros;
  if (ok) {
    unsigned long long near = ~0ull;
    each_site(count, [&](int x, int y) {
      const int dx = 2 * x - cx, dy = 2 * y - cy;
      near = min(near, ((unsigned long long)(unsigned)(dx * dx + dy * dy) << 32) |
                           ((unsigned)y << 16) | (unsigned)x);
    });
    atomicMin(&s_near, near);
    if (tid == 0) s_cnt = 0u;
    __syncthreads();
    const int sx = (int)(s_near & 0xffffu) - x0, sy = (int)((s_near >> 16) & 0xffffu) - y0;
    const int4 r2 = corner_d2(sx, sy, kBand - 1);
    // the blocks the circles around the corners reach, and their sites there
    const int rmax = max(max(r2.x, r2.y), max(r2.z, r2.w));
    count = list_macros((int)(sqrtf((float)rmax) / kBand) + 2, [&](int kx, int ky) {
      const int lx = kBand * kx - x0, ly = kBand * ky - y0;
      const int gx0 = box_gap(0, lx, lx + 63), gx1 = box_gap(63, lx, lx + 63);
      const int gy0 = box_gap(0, ly, ly + 63), gy1 = box_gap(63, ly, ly + 63);
      return gx0 * gx0 + gy0 * gy0 <= r2.x || gx1 * gx1 + gy0 * gy0 <= r2.y ||
             gx0 * gx0 + gy1 * gy1 <= r2.z || gx1 * gx1 + gy1 * gy1 <= r2.w;
    });
    ok = count <= kFarMacros;
    if (tid == 0) s_cnt = 0u;
    __syncthreads();
    if (ok) {
      each_site(count, [&](int x, int y) {
        if (!corner_in(x - x0, y - y0, kBand - 1, r2)) return;
        const unsigned p = atomicAdd(&s_cnt, 1u);
        if (p < kFarSites) s_site[p] = (uint32_t)x | ((uint32_t)y << 16);
      });
      __syncthreads();
      ok = s_cnt <= kFarSites;
    }
  }
  if (!ok) {
    if (tid == 0) a.st->band_rows[my] = 1;
    return;
  }
  // the open tiles, a warp each: nearest site to the centre, corner test, tie order
  const int ns = (int)s_cnt;
  for (int t = wib; t < 16; t += kFarThreads / 32) {
    if (!((open >> t) & 1u)) continue;
    const int tx = x0 + t % 4 * kT, ty = y0 + t / 4 * kT;
    unsigned best = 0xffffffffu;
    int bk = 0;
    for (int k = lane; k < ns; k += 32) {
      const int ex = 2 * ((int)(s_site[k] & 0xffffu) - tx) - (kT - 1),
                ey = 2 * ((int)(s_site[k] >> 16) - ty) - (kT - 1);
      const unsigned d = (unsigned)(ex * ex + ey * ey);
      if (d < best) best = d, bk = k;
    }
    const unsigned d0 = __reduce_min_sync(kFull, best);
    bk = __shfl_sync(kFull, bk, __ffs(__ballot_sync(kFull, best == d0)) - 1);
    const int sx = (int)(s_site[bk] & 0xffffu) - tx, sy = (int)(s_site[bk] >> 16) - ty;
    const int4 r2 = corner_d2(sx, sy, kT - 1);
    int m = 0;
    for (int k0 = 0; k0 < ns; k0 += 32) {
      const int k = k0 + lane;
      const uint32_t v = k < ns ? s_site[k] : 0u;
      const int x = (int)(v & 0xffffu), y = (int)(v >> 16);
      const bool keep = k < ns && corner_in(x - tx, y - ty, kT - 1, r2);
      const unsigned km = __ballot_sync(kFull, keep);
      const int pos = m + __popc(km & ((1u << lane) - 1u));
      if (keep && pos < kCand) {
        // tie order: x, then bands up to the tile's from the lowest row up, then the rest
        s_key[wib][pos] = ((uint32_t)x << 16) |
                          (uint32_t)((y >> 6) <= (ty >> 6) ? 0x3fff - y : 0x4000 + y);
        s_pos[wib][pos] = v;
      }
      m += __popc(km);
    }
    if (m > kCand) {
      if (lane == 0) a.st->band_rows[my] = 1;
      continue;
    }
    __syncwarp();
    for (int k = lane; k < m; k += 32) {
      const uint32_t key = s_key[wib][k], v = s_pos[wib][k];
      int rank = 0;
      for (int j = 0; j < m; ++j) rank += s_key[wib][j] < key;
      const int x = (int)(v & 0xffffu), y = (int)(v >> 16);
      s_cand[wib][rank] = cand_entry(x - tx, y - ty, sx, sy, v);
    }
    __syncwarp();
    eval_tile(s_cand[wib], m, tx, ty, n, a.labels);
    __syncwarp();
  }
}

}  // namespace

size_t label_blocks(int n) { return (size_t)(n / kBand) * (n / kBand); }

// Up to 512 x 512 the row pass labels: three launches instead of six (the tiles' three
// and the row pass's, which then look at band_rows), and both are latency there.  A
// labelling call took, rows / tiles: 37 / 51 us at 256 x 256, 50 / 57 at 512 x 512, 92 /
// 75 at 1024 x 1024.  So it does where the sites crowd the tiles' lists, which are too
// short from about 12 pixels a site on, the row pass then following the tiles: 2048 x 2048
// of 16 pixels a site 189 / 106 us, of 13 600 / 95, of 12 595 / 556, of 11 596 / 707; 8192
// x 8192 of 13 8.35 / 3.23 ms, of 12 8.99 / 9.62.  A 64 x 64 block of more than kCrowdBlock
// (10.8 pixels a site) sends its band there before the tiles look at it: the quarter of
// 2048 x 2048 at 4 pixels a site 487 by rows alone, 576 by tiles and all rows, 494 us now;
// a crowded 128 x 128 corner of 8192 x 8192 1.17, 1.39 and 0.55 ms.
constexpr int kRowLabels = 512;
constexpr long long kRowCrowd = 13;

static bool rows_alone(const LevelBufs &b) {
  return b.n <= kRowLabels || kRowCrowd * b.sites >= (long long)b.n * b.n;
}

cudaError_t launch_label_sites(const LevelBufs &b, cudaStream_t s) {
  if (rows_alone(b)) return launch_summary(b, true, s);
  k_label_occ<<<(unsigned)(b.n / kBand), 1024, 0, s>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_label_write(const LevelBufs &b, cudaStream_t s) {
  const unsigned M = (unsigned)(b.n / kBand);
  if (rows_alone(b)) return launch_rows(b, true, s);
  k_label_tiles<<<dim3((unsigned)b.n / (kT * kTileWarps), (unsigned)b.n / kT), 32 * kTileWarps,
                  0, s>>>(b);
  // (wider blocks where a few of them are the kernel's time: 1024 x 1024 with a 64-pixel
  // cluster 50 -> 45 us; 8192 x 8192 with ten sites 205 -> 223)
  if (b.n <= 1536) k_label_far<256><<<dim3(M, M), 256, 0, s>>>(b);
  else k_label_far<128><<<dim3(M, M), 128, 0, s>>>(b);
  // the row pass for its bands
  const cudaError_t e = launch_summary(b, false, s);
  return e == cudaSuccess ? launch_rows(b, false, s) : e;
}

cudaError_t launch_label(const LevelBufs &b, cudaStream_t s) {
  const cudaError_t e = launch_label_sites(b, s);
  return e == cudaSuccess ? launch_label_write(b, s) : e;
}

}  // namespace cvtgb
