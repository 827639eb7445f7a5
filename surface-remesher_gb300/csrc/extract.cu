// extract.cu -- the CDT's input points from the converged sites, on the GPU:
// the loop of delaunayInput (delaunay.h:46-57) that scans the n^2 label grid
// on the host for pixels labelled with themselves and not fixed, and emits
// (x * scale + left, y * scale + lower) in x-major, then y order.  Here the
// site bitmap is compacted column by column: k_col_count counts each
// column's free sites, k_col_write finds each column's offset from those
// counts and writes the points in FP64 (products and sums rounded separately,
// as the host code computes them).
#include "gcvt_internal.cuh"

namespace cvtgb {

// A block takes 32 columns, thread (tx, ty) the bands [ty G, ty G + G) of column
// 32 block + tx, G = ceil(bands / 32): coalesced reads and short chains (a thread
// walking a whole column took 22 us at 2048^2, 3 to 4 now).
struct Bands {
  int b0, b1;
};
__device__ __forceinline__ Bands bands_of(int n) {
  const int nb = n / kBand, G = (nb + 31) / 32, b0 = min(nb, (int)threadIdx.y * G);
  return Bands{b0, min(nb, b0 + G)};
}
__device__ __forceinline__ uint64_t free_bits(const uint64_t *__restrict__ bits,
                                              const uint64_t *__restrict__ fixed, size_t i) {
  return fixed ? bits[i] & ~fixed[i] : bits[i];
}

// Free (not fixed) sites per column of bits (fixed may be null).
__global__ void __launch_bounds__(1024) k_col_count(const uint64_t *__restrict__ bits,
                                                    const uint64_t *__restrict__ fixed, int n,
                                                    unsigned *__restrict__ colcnt) {
  __shared__ unsigned part[32][33];
  const int x = blockIdx.x * 32 + threadIdx.x;
  const Bands r = bands_of(n);
  unsigned c = 0;
  for (int b = r.b0; b < r.b1; ++b) c += __popcll(free_bits(bits, fixed, (size_t)b * n + x));
  part[threadIdx.x][threadIdx.y] = c;  // transposed: warp ty sums column ty
  __syncthreads();
  const unsigned s = __reduce_add_sync(0xffffffffu, part[threadIdx.y][threadIdx.x]);
  if (threadIdx.x == 0) colcnt[blockIdx.x * 32 + threadIdx.y] = s;
}

// Block b writes columns [32 b, 32 b + 32): its offset is the sum of the counts
// before it, then an exclusive scan over its own columns and their bands.
__global__ void __launch_bounds__(1024) k_col_write(const uint64_t *__restrict__ bits,
                                                    const uint64_t *__restrict__ fixed, int n,
                                                    const unsigned *__restrict__ colcnt,
                                                    double scale, double left, double lower,
                                                    double *__restrict__ xy, unsigned capacity,
                                                    unsigned *__restrict__ total) {
  __shared__ unsigned part[32][33], wsum[32], col[32];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx, x0 = blockIdx.x * 32;
  const int x = x0 + tx;
  unsigned pre = 0;
  for (int k = tid; k < x0; k += 1024) pre += colcnt[k];
  pre = __reduce_add_sync(0xffffffffu, pre);
  if (tx == 0) wsum[ty] = pre;
  const Bands r = bands_of(n);
  unsigned c = 0;
  for (int b = r.b0; b < r.b1; ++b) c += __popcll(free_bits(bits, fixed, (size_t)b * n + x));
  part[tx][ty] = c;
  __syncthreads();
  auto scan = [&](unsigned v) {  // inclusive over the warp
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
      if (tx >= o) v += u;
    }
    return v;
  };
  const unsigned mine = part[ty][tx];  // bands tx of column ty
  const unsigned inc = scan(mine);
  if (ty == 0) {  // column offsets
    const unsigned base = __reduce_add_sync(0xffffffffu, wsum[tx]);
    const unsigned cnt = colcnt[x0 + tx], ci = scan(cnt);
    col[tx] = base + ci - cnt;
    if (blockIdx.x == gridDim.x - 1 && tx == 31) *total = base + ci;
  }
  __syncthreads();
  part[ty][tx] = inc - mine;
  __syncthreads();
  unsigned pos = col[tx] + part[tx][ty];
  const double px = __dadd_rn(__dmul_rn((double)x, scale), left);
  for (int b = r.b0; b < r.b1 && pos < capacity; ++b) {
    uint64_t w = free_bits(bits, fixed, (size_t)b * n + x);
    while (w && pos < capacity) {
      const int i = __ffsll((long long)w) - 1;
      w &= w - 1ull;
      xy[2 * (size_t)pos] = px;
      xy[2 * (size_t)pos + 1] = __dadd_rn(__dmul_rn((double)(b * kBand + i), scale), lower);
      ++pos;
    }
  }
}

// (n is a multiple of 32)
cudaError_t launch_extract(const uint64_t *bits, const uint64_t *fixed, int n, unsigned *colcnt,
                           double scale, double left, double lower, double *xy,
                           unsigned capacity, unsigned *total, cudaStream_t s) {
  const dim3 blk(32, 32);
  k_col_count<<<n / 32, blk, 0, s>>>(bits, fixed, n, colcnt);
  k_col_write<<<n / 32, blk, 0, s>>>(bits, fixed, n, colcnt, scale, left, lower, xy, capacity,
                                     total);
  return cudaGetLastError();
}

}  // namespace cvtgb
