// Triangle counting: sum over the entries (i, k) of a lower triangle L of
// |L_i & L_k|, the masked binary product of bmm32_sparse_masked_v5
// (bsrbmm/bsrbmm.cu:1214-1265), which reduces into an int32 (overflows past
// 2^31 triangles, bsrbmm/tc.cu:861-863).  The count is uint64.
//
// Lower triangles (every entry at or below the diagonal) are counted over
// lists of neighbours: tiles of power-law graphs hold one or two bits, so a
// pair of tiles costs two 32-byte sectors and a search for a bit of product.
// A simple graph's triangles do not depend on which end an edge belongs to, so
// once per graph the vertices are ranked by falling degree and every edge goes
// to its end of lower degree, as the other end's rank: a list is at most
// sqrt(2 edges) long, and hubs' lists are short (R-MAT 17: 252 M list entries
// to look at instead of 405 M by vertex number, the longest list 329 instead
// of 5,255).  Per list, a warp per kUnit entries looks up the lists of these
// entries among the list itself: ranks below kBits -- nearly all of a
// power-law graph's -- in an exact bitmap in shared memory, the others behind
// a filter.  Where every row is a few entries long (meshes) the rows are
// counted as they are, a lane each.  Diagonal entries add, per the formula
// above, a term per entry in their column and their row's length.
//
// Bound by the latency of the lists' reads from L2 at 32 warps an SM: kSide
// lists are read side by side (1 / 2 / 4 / 8 of them: 716 / 561 / 491 / 681 us
// at R-MAT 17, ef 16, b = 32; a bitmap of 16,384 ranks: 523; a hash of 1,024
// entries in place of both: 1,171).  Tiles / lists, us, with the lists built:
// R-MAT 17 2,679 / 483, ef 24 shuffled b = 16 5,261 / 921, R-MAT 20
// 75,430 / 7,763, uniform of 100,003 vertices and 24 per vertex b = 8
// 622 / 103, mesh of 10^6 vertices 121 / 42.
//
// Building costs 180 us and more however small the graph, and a program may
// count once.  So a graph's first count goes over lists only where that is no
// slower than over tiles (from kListFirst tiles on, kListFirstLong where block
// rows are long: the tile kernel searches them), and from kListTiles on the
// second count builds them.  First counts, tiles / lists, us (later ones over
// lists 34 to 100): uniform, 24 a vertex, b = 8, 111,000 tiles 120 / 237, 351,000
// 257 / 282, 471,000 317 / 288, 591,000 371 / 313; b = 16, 445,000 497 / 284; b =
// 32, 98,000 273 / 238, 359,000 843 / 305; R-MAT b = 8, 70,000 315 / 319, 122,000
// 438 / 387, 240,000 695 / 475; mesh b = 8, 99,000 106 / 158, 397,000 213 / 201.
// Fewer tiles, tensor-core counts and matrices with an entry above the diagonal
// (looked for before anything is built) keep the tile kernels, as does a call
// under stream capture before the lists are built (nothing can be read back
// there) or one without memory for them.
#include <algorithm>

#include "gather.cuh"

namespace gbo {

namespace {

constexpr int kTPB = 256;

__device__ __forceinline__ int lower_bound_dev(const int* __restrict__ a, int lo, int hi, int key) {
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

constexpr long long kListTiles = 1 << 16;
constexpr long long kListFirst = 1 << 19;
constexpr long long kListFirstLong = 1 << 17;  // where block rows are long:
constexpr int kLongMean = 128;                 // tiles of one on average, or
constexpr int kSkew = 8;                       // the longest against the average
constexpr int kUnit = 64;       // entries of a list that one warp goes through
constexpr int kBits = 32768;    // ranks in a warp's bitmap
constexpr int kPiece = 256;     // entries of a list looked up among at a time
constexpr int kFilterBits = 2048;
constexpr int kSide = 4;        // looked-up lists read side by side
constexpr int kTcWarps = 8;     // warps of a block (5.3 KB of shared memory each)

struct Lists {
  const long long* __restrict__ ptr;
  const int* __restrict__ col;
  int n;
};

__global__ void k_count_cols(const int* __restrict__ col, long long nnz, int* __restrict__ deg) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += (long long)gridDim.x * blockDim.x)
    atomicAdd(deg + col[i], 1);
}

// Ranks by falling degree (row length + column count), by a counting sort over
// bins: exact below 1,024, then 32 an octave (any order is a valid one, so the
// out-degrees that came with a wrapped graph need not be right: they are held
// within the bins).
constexpr int kDegBins = 1024 + 22 * 32;

__device__ __forceinline__ int degree_bin(const GatherList& gl, const int* __restrict__ colcnt, long long i) {
  const long long d = max(gl.ptr[i + 1] - gl.ptr[i] + colcnt[i], 0ll);
  if (d < 1024) return (int)d;
  const int x = (int)min(d, 0x7fffffffll), o = 31 - __clz(x);
  return 1024 + (o - 10) * 32 + ((x >> (o - 5)) & 31);
}

__global__ void __launch_bounds__(1024) k_degree_hist(GatherList gl, const int* __restrict__ colcnt,
                                                      int* __restrict__ hist) {
  __shared__ int h[kDegBins];
  for (int b = (int)threadIdx.x; b < kDegBins; b += 1024) h[b] = 0;
  __syncthreads();
  for (long long i = (long long)blockIdx.x * 1024 + threadIdx.x; i < gl.nrows; i += (long long)gridDim.x * 1024)
    atomicAdd(h + degree_bin(gl, colcnt, i), 1);
  __syncthreads();
  for (int b = (int)threadIdx.x; b < kDegBins; b += 1024)
    if (h[b]) atomicAdd(hist + b, h[b]);
}

// First rank of every bin, the highest degrees first (one block).
__global__ void __launch_bounds__(1024) k_degree_starts(int* __restrict__ hist) {
  __shared__ int warp_sh[32];
  const unsigned lane = threadIdx.x & 31;
  const int wib = (int)(threadIdx.x >> 5);
  int carry = 0;
  for (int b0 = 0; b0 < kDegBins; b0 += 1024) {
    const int b = kDegBins - 1 - (b0 + (int)threadIdx.x);
    const int c = b >= 0 ? hist[b] : 0;
    int x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)lane >= o) x += y;
    }
    if (lane == 31) warp_sh[wib] = x;
    __syncthreads();
    int before = carry, all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < wib) before += warp_sh[w];
      all += warp_sh[w];
    }
    if (b >= 0) hist[b] = before + x - c;
    carry += all;
    __syncthreads();
  }
}

// Ranks: a block counts its vertices per bin, reserves their places and deals
// them out (few atomics reach one bin's counter).
__global__ void __launch_bounds__(1024) k_degree_ranks(GatherList gl, const int* __restrict__ colcnt,
                                                       int* __restrict__ next, int* __restrict__ rank) {
  __shared__ int h[kDegBins], base[kDegBins];
  constexpr int kPer = 4;
  const long long i0 = (long long)blockIdx.x * 1024 * kPer;
  for (int b = (int)threadIdx.x; b < kDegBins; b += 1024) h[b] = 0;
  __syncthreads();
  int bin[kPer], at[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const long long i = i0 + q * 1024 + threadIdx.x;
    bin[q] = i < gl.nrows ? degree_bin(gl, colcnt, i) : -1;
    at[q] = bin[q] >= 0 ? atomicAdd(h + bin[q], 1) : 0;
  }
  __syncthreads();
  for (int b = (int)threadIdx.x; b < kDegBins; b += 1024)
    if (h[b]) base[b] = atomicAdd(next + b, h[b]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kPer; ++q)
    if (bin[q] >= 0) rank[i0 + q * 1024 + threadIdx.x] = base[bin[q]] + at[q];
}

// A warp per row of the lower triangle: count the edges of every owner -- the
// end of higher rank -- (FILL = false), or put the other ends' ranks into the
// owners' lists, in any order.
template <bool FILL>
__global__ void __launch_bounds__(kTPB) k_orient(GatherList gl, const int* __restrict__ rank, int* __restrict__ cnt,
                                                 const long long* __restrict__ optr, int* __restrict__ ocol) {
  constexpr int kPer = 4;  // entries of a lane in flight
  const unsigned lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < gl.nrows; i += nwarps) {
    const int ri = rank[i];
    const long long e = gl.ptr[i + 1];
    for (long long p = gl.ptr[i] + lane; p - lane < e; p += 32 * kPer) {
      int rk[kPer], at[kPer];
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        rk[q] = p + 32 * q < e ? rank[gl.col[p + 32 * q]] : ri;
        if (rk[q] != ri) at[q] = atomicAdd(cnt + max(ri, rk[q]), 1);  // the diagonal is left out
      }
#pragma unroll
      for (int q = 0; q < kPer; ++q)
        if (FILL && rk[q] != ri) ocol[optr[max(ri, rk[q])] + at[q]] = min(ri, rk[q]);
    }
  }
}

// A list of one entry has no pair in it.
__global__ void k_tc_unit_counts(Lists l, int* __restrict__ cnt) {
  for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < l.n; u += (long long)gridDim.x * blockDim.x) {
    const long long a = l.ptr[u + 1] - l.ptr[u];
    cnt[u] = a < 2 ? 0 : (int)((a + kUnit - 1) / kUnit);
  }
}

__global__ void k_tc_units(const int* __restrict__ unit0, int n, int* __restrict__ unit) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    for (int u = unit0[i]; u < unit0[i + 1]; ++u) unit[u] = (int)i;
}

__device__ __forceinline__ void add_count(unsigned long long acc, unsigned long long* count) {
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(count, acc);
}

// Rows of at most kShortRow entries and no diagonal, a lane each.
__global__ void __launch_bounds__(kTPB) k_tc_lanes(GatherList gl, unsigned long long* __restrict__ count) {
  unsigned long long acc = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < gl.nrows;
       i += (long long)gridDim.x * blockDim.x) {
    const long long p = gl.ptr[i];
    const int a = (int)(gl.ptr[i + 1] - p);
    int A[kShortRow];
#pragma unroll
    for (int q = 0; q < kShortRow; ++q) A[q] = q < a ? gl.col[p + q] : -1;
#pragma unroll
    for (int q = 1; q < kShortRow; ++q) {  // entry q's row holds entries before it only
      if (q >= a) continue;
      for (long long b = gl.ptr[A[q]], e = gl.ptr[A[q] + 1]; b < e; ++b) {
        const int x = gl.col[b];
#pragma unroll
        for (int c = 0; c < q; ++c) acc += x == A[c];
      }
    }
  }
  add_count(acc, count);
}

__device__ __forceinline__ unsigned filter_bit(int c) { return ((unsigned)c * 2654435761u) >> 21; }  // of kFilterBits

__global__ void __launch_bounds__(kTcWarps * 32) k_tc_warps(Lists l, const int* __restrict__ unit,
                                                            const int* __restrict__ unit0, int nunits,
                                                            unsigned long long* __restrict__ count) {
  static_assert(kFilterBits == 2048, "filter_bit gives eleven bits");
  __shared__ unsigned bits_sh[kTcWarps][kBits / 32];
  __shared__ unsigned filter_sh[kTcWarps][kFilterBits / 32];
  __shared__ int high_sh[kTcWarps][kPiece];  // the piece's ranks past the bitmap
  const unsigned lane = threadIdx.x & 31;
  const int wib = (int)(threadIdx.x >> 5);
  unsigned *bits = bits_sh[wib], *filter = filter_sh[wib];
  int* high = high_sh[wib];
  for (int w = (int)lane; w < kBits / 32; w += 32) bits[w] = 0u;
  for (int w = (int)lane; w < kFilterBits / 32; w += 32) filter[w] = 0u;
  __syncwarp();
  unsigned long long acc = 0;
  const int nwarps = (int)gridDim.x * kTcWarps;
  for (int q = (int)blockIdx.x * kTcWarps + wib; q < nunits; q += nwarps) {
    const int u = unit[q];
    const long long p = l.ptr[u];
    const int a = (int)(l.ptr[u + 1] - p);
    const int s = (q - unit0[u]) * kUnit, z = min(s + kUnit, a);  // the unit's entries
    for (int h0 = 0; h0 < a; h0 += kPiece) {  // the list, in pieces
      const int h1 = min(h0 + kPiece, a);
      int nh = 0;
      for (int c0 = h0; c0 < h1; c0 += 32) {
        const int x = c0 + (int)lane < h1 ? l.col[p + c0 + lane] : -1;
        const bool far = x >= kBits;
        if (x >= 0 && !far) atomicOr(bits + (x >> 5), 1u << (x & 31));
        if (far) atomicOr(filter + (filter_bit(x) >> 5), 1u << (filter_bit(x) & 31));
        const unsigned m = __ballot_sync(0xffffffffu, far);
        if (far) high[nh + __popc(m & ((1u << lane) - 1u))] = x;
        nh += __popc(m);
      }
      __syncwarp();
      for (int t0 = s; t0 < z; t0 += 32) {
        long long bl = 0;
        int nl = 0;
        if (t0 + (int)lane < z) {
          const int v = l.col[p + t0 + lane];
          bl = l.ptr[v];
          nl = (int)(l.ptr[v + 1] - bl);
        }
        const int m = min(32, z - t0);
        unsigned hits = 0;
        for (int j = 0; j < m; j += kSide) {
          const int* B[kSide];
          int nb[kSide], most = 0;
#pragma unroll
          for (int i = 0; i < kSide; ++i) {  // lanes from m on have nl = 0
            B[i] = l.col + __shfl_sync(0xffffffffu, bl, (j + i) & 31);
            nb[i] = __shfl_sync(0xffffffffu, nl, (j + i) & 31);
            most = max(most, nb[i]);
          }
          for (int b = (int)lane; b < most; b += 32) {
            int x[kSide];
#pragma unroll
            for (int i = 0; i < kSide; ++i) x[i] = b < nb[i] ? B[i][b] : -1;
#pragma unroll
            for (int i = 0; i < kSide; ++i) {
              if ((unsigned)x[i] < (unsigned)kBits) {
                hits += (bits[x[i] >> 5] >> (x[i] & 31)) & 1u;
              } else if (nh > 0 && x[i] >= 0 && ((filter[filter_bit(x[i]) >> 5] >> (filter_bit(x[i]) & 31)) & 1u)) {
                for (int c = 0; c < nh; ++c) hits += high[c] == x[i];
              }
            }
          }
        }
        acc += hits;
      }
      __syncwarp();
      for (int c = h0 + (int)lane; c < h1; c += 32) {  // leave both clear
        const int x = l.col[p + c];
        if (x < kBits) bits[x >> 5] = 0u;
        else filter[filter_bit(x) >> 5] = 0u;
      }
      __syncwarp();
    }
  }
  add_count(acc, count);
}

// The diagonal's share: for every entry (i, k) with i > k and k on the
// diagonal 1 (k is common to rows i and k), for every diagonal (i, i) the
// length of row i.
__global__ void __launch_bounds__(kTPB) k_tc_diagonal(GatherList gl, unsigned long long* __restrict__ count) {
  const unsigned lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  unsigned long long acc = 0;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < gl.nrows; i += nwarps) {
    const long long b = gl.ptr[i], e = gl.ptr[i + 1];
    for (long long p = b + lane; p < e; p += 32) {
      const int k = gl.col[p];
      if (k == i) acc += (unsigned long long)(e - b);
      else acc += gl.ptr[k + 1] > gl.ptr[k] && gl.col[gl.ptr[k + 1] - 1] == k;
    }
  }
  add_count(acc, count);
}

// Whether some entry lies above the diagonal: a thread per block row looks at
// its last tile (block columns ascend).
template <int B>
__global__ void k_above(GView v, unsigned* __restrict__ above) {
  using WT = typename Word<B>::T;
  const int R = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  bool up = false;
  if (R < v.nbr && v.rowptr[R + 1] > v.rowptr[R]) {
    const int t = v.rowptr[R + 1] - 1, C = v.colind[t];
    up = C > R;
    if (C == R) {
      const WT* __restrict__ w = reinterpret_cast<const WT*>(v.val) + (size_t)t * B;
#pragma unroll 8
      for (int r = 0; r < B; ++r) up = up || (w[r] & (WT)(((WT)1 << (B - 1 - r)) - 1));
    }
  }
  if (__any_sync(0xffffffffu, up) && (threadIdx.x & 31) == 0) *above = 1u;
}

// Block row of every tile, from the work items.
__global__ void k_tile_row(GView v, int* __restrict__ tile_row) {
  const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (item >= v.nitems) return;
  const gbo_item it = v.items[item];
  for (int t = it.t0 + (int)(threadIdx.x & 31); t < it.t1; t += 32) tile_row[t] = it.row;
}

// Mask tiles with at most kSparsePairs set bits take the lane-per-hit path:
// the (row, column) bits of the mask go to a per-warp list, and every lane
// with a hit sums popc(A[r] & B[c]) over the list for its own tile pair,
// loading just those rows -- hits of a probe round proceed side by side
// instead of one after another.  Denser masks broadcast the K-tile rows.
constexpr int kSparsePairs = 16;

template <int B>
__global__ void __launch_bounds__(kTPB) k_tc(GView v, long long nblk, const int* __restrict__ tile_row,
                                             int skip_dense, unsigned long long* __restrict__ count) {
  using WT = typename Word<B>::T;
  constexpr int RPL = B > 32 ? 2 : 1;
  __shared__ short pairs_sh[kTPB / 32][kSparsePairs];  // (r << 7) | c
  const unsigned lane = threadIdx.x & 31;
  short* pairs = pairs_sh[threadIdx.x >> 5];
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const WT* __restrict__ val = reinterpret_cast<const WT*>(v.val);
  unsigned long long acc = 0;
  // mask tiles strided over the warps (hub rows spread out)
  for (long long m = warp; m < nblk; m += nwarps) {
    const int I = tile_row[m];
    const int K = v.colind[m];
    // mask rows of tile (I,K)
    WT M0 = 0, M1 = 0;
    if (lane < (unsigned)(B < 32 ? B : 32)) M0 = val[(size_t)m * B + lane];
    if (RPL == 2) M1 = val[(size_t)m * B + 32 + lane];
    // union of the mask columns over the tile's rows
    unsigned long long U = (unsigned long long)M0 | (unsigned long long)M1;
    {
      unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)U);
      unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(U >> 32));
      U = ((unsigned long long)hi << 32) | lo;
    }
    // mask bits as a list when the mask is sparse (lane order = row order)
    int npairs = -1;
    {
      const int c0 = popc_w(M0) + (RPL == 2 ? popc_w(M1) : 0);
      int incl = c0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
      }
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      if (total <= kSparsePairs) {
        int pos = incl - c0;
        for (int h = 0; h < RPL; ++h) {
          const int r = (int)lane + 32 * h;
          unsigned long long w = (unsigned long long)(h ? M1 : M0) << (64 - B);
          while (w) {
            const int c = __clzll(w);
            w &= ~(0x8000000000000000ull >> c);
            pairs[pos++] = (short)((r << 7) | c);
          }
        }
        npairs = total;
      }
      __syncwarp();
    }
    if (npairs < 0 && skip_dense) continue;  // dense masks go to the tensor-core kernel
    // list A: row I, tiles with block column <= K  -> [rowptr[I], m]
    // list B: row K, all tiles (block columns <= K in a lower triangle)
    const int a0 = v.rowptr[I], a1 = (int)m + 1;
    const int b0 = v.rowptr[K], b1 = v.rowptr[K + 1];
    const bool probe_a = (a1 - a0) <= (b1 - b0);
    const int p0 = probe_a ? a0 : b0, p1 = probe_a ? a1 : b1;
    const int s0 = probe_a ? b0 : a0, s1 = probe_a ? b1 : a1;
    if constexpr (B == 32) {
      if (npairs < 0) {
        // dense 32x32 mask: lane r accumulates P[r][c] = sum over hits of
        // popc(A[r] & B[c]) for all 32 columns (B rows broadcast by 32
        // unrolled shuffles, no data-dependent loop), masked once at the end
        unsigned cm[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) cm[c] = 0u;
        for (int base = p0; base < p1; base += 32) {
          const int p = base + (int)lane;
          int hit = -1;
          if (p < p1) {
            const int J = v.colind[p];
            const int q = lower_bound_dev(v.colind, s0, s1, J);
            if (q < s1 && v.colind[q] == J) hit = q;
          }
          unsigned found = __ballot_sync(0xffffffffu, hit >= 0);
          while (found) {
            const int src = __ffs(found) - 1;
            found &= found - 1;
            const int ph = __shfl_sync(0xffffffffu, p, src);
            const int qh = __shfl_sync(0xffffffffu, hit, src);
            const unsigned ar = (unsigned)val[(size_t)(probe_a ? ph : qh) * 32 + lane];
            const unsigned br = (unsigned)val[(size_t)(probe_a ? qh : ph) * 32 + lane];
#pragma unroll
            for (int c = 0; c < 32; ++c) cm[c] += __popc(ar & __shfl_sync(0xffffffffu, br, c));
          }
        }
        const unsigned mr = (unsigned)M0;
#pragma unroll
        for (int c = 0; c < 32; ++c) acc += ((mr >> (31 - c)) & 1u) ? cm[c] : 0u;
        continue;
      }
    }
    for (int base = p0; base < p1; base += 32) {
      const int p = base + (int)lane;
      int hit = -1;
      if (p < p1) {
        const int J = v.colind[p];
        const int q = lower_bound_dev(v.colind, s0, s1, J);
        if (q < s1 && v.colind[q] == J) hit = q;
      }
      unsigned found = __ballot_sync(0xffffffffu, hit >= 0);
      if (npairs >= 0) {  // sparse mask: each lane handles its own hit
        if (hit >= 0) {
          const int ia = probe_a ? p : hit;  // tile (I,J)
          const int ib = probe_a ? hit : p;  // tile (K,J)
          for (int k = 0; k < npairs; ++k) {
            const int pr = pairs[k];
            acc += popc_w((WT)(val[(size_t)ia * B + (pr >> 7)] & val[(size_t)ib * B + (pr & 127)]));
          }
        }
        continue;
      }
      while (found) {
        const int src = __ffs(found) - 1;
        found &= found - 1;
        const int ph = __shfl_sync(0xffffffffu, p, src);
        const int qh = __shfl_sync(0xffffffffu, hit, src);
        const int ia = probe_a ? ph : qh;  // tile (I,J)
        const int ib = probe_a ? qh : ph;  // tile (K,J)
        // only the rows that matter are loaded: A rows with mask bits, B
        // rows of the mask's columns (sparse tiles touch one or two sectors)
        WT A0 = 0, A1 = 0, Bw0 = 0, Bw1 = 0;
        if (lane < (unsigned)(B < 32 ? B : 32)) {
          if (M0) A0 = val[(size_t)ia * B + lane];
          if ((U >> (B - 1 - lane)) & 1ull) Bw0 = val[(size_t)ib * B + lane];
        }
        if (RPL == 2) {
          if (M1) A1 = val[(size_t)ia * B + 32 + lane];
          if ((U >> (31 - lane)) & 1ull) Bw1 = val[(size_t)ib * B + 32 + lane];
        }
        unsigned long long u = U << (64 - B);  // column c at bit 63-c
        while (u) {
          const int c = __clzll(u);
          u &= ~(0x8000000000000000ull >> c);
          WT bc;
          if (RPL == 2)
            bc = c < 32 ? (WT)__shfl_sync(0xffffffffu, (unsigned long long)Bw0, c)
                        : (WT)__shfl_sync(0xffffffffu, (unsigned long long)Bw1, c - 32);
          else
            bc = (WT)__shfl_sync(0xffffffffu, (unsigned)Bw0, c);
          if ((M0 >> (B - 1 - c)) & 1) acc += popc_w((WT)(A0 & bc));
          if (RPL == 2 && ((M1 >> (B - 1 - c)) & 1)) acc += popc_w((WT)(A1 & bc));
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0 && acc) atomicAdd(count, acc);
}

// D += popc(A AND B) over 256-bit rows/columns: the 1-bit tensor-core MMA
// (m16n8k256, A row-major 16x256, B column-major 256x8, s32 accumulators).
// Fragments, with g = lane / 4 and q = lane % 4: a0 = A[g][32q..32q+31],
// a1 = A[g+8][same], a2 = A[g][128+32q..], a3 = A[g+8][128+32q..];
// b0 = B[32q..][g], b1 = B[128+32q..][g]; d0,d1 = D[g][2q, 2q+1],
// d2,d3 = D[g+8][2q, 2q+1].
__device__ __forceinline__ void mma_and_popc(int (&d)[4], unsigned a0, unsigned a1, unsigned a2,
                                             unsigned a3, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k256.row.col.s32.b1.b1.s32.and.popc "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Opt-in (GBO_FLAG_TC_MMA): on the configured graphs this path did not beat
// the CUDA-core one (king mesh b=32: 3.3 vs 3.6 ms but b=16 without it 2.1 ms;
// R-MAT 20 degree-ordered b=32: 25.8 vs 20.5 ms), so it is not the default.
// Dense 32x32 mask tiles (more than kSparsePairs bits) on the tensor cores:
// for a mask tile (I,K) the product P = sum_J A_IJ B_KJ^T over the hits J is
// a 32x32 AND-popc product with the hits' 32-bit rows laid side by side
// along k (8 hits per 256-bit step), then sum_{r,c} M[r][c] P[r][c].
__global__ void __launch_bounds__(kTPB) k_tc32_mma(GView v, long long nblk, const int* __restrict__ tile_row,
                                                   unsigned long long* __restrict__ count) {
  __shared__ int2 hits_sh[kTPB / 32][32];
  __shared__ uint32_t tiles_sh[kTPB / 32][2][8][32];  // A and B tiles of 8 hits
  const unsigned lane = threadIdx.x & 31;
  const int g = (int)(lane >> 2), q4 = (int)(lane & 3);
  int2* hits = hits_sh[threadIdx.x >> 5];
  uint32_t (*sA)[32] = tiles_sh[threadIdx.x >> 5][0];
  uint32_t (*sB)[32] = tiles_sh[threadIdx.x >> 5][1];
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const uint32_t* __restrict__ val = reinterpret_cast<const uint32_t*>(v.val);
  unsigned long long acc = 0;
  for (long long m = warp; m < nblk; m += nwarps) {
    const uint32_t M0 = val[(size_t)m * 32 + lane];
    const int total = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(M0));
    if (total <= kSparsePairs) continue;  // handled by k_tc
    const int I = tile_row[m];
    const int K = v.colind[m];
    const int a0i = v.rowptr[I], a1i = (int)m + 1;
    const int b0i = v.rowptr[K], b1i = v.rowptr[K + 1];
    const bool probe_a = (a1i - a0i) <= (b1i - b0i);
    const int p0 = probe_a ? a0i : b0i, p1 = probe_a ? a1i : b1i;
    const int s0 = probe_a ? b0i : a0i, s1 = probe_a ? b1i : a1i;
    int d[2][4][4];
#pragma unroll
    for (int mb = 0; mb < 2; ++mb)
#pragma unroll
      for (int nb = 0; nb < 4; ++nb)
#pragma unroll
        for (int e = 0; e < 4; ++e) d[mb][nb][e] = 0;
    for (int base = p0; base < p1; base += 32) {
      const int p = base + (int)lane;
      int hit = -1;
      if (p < p1) {
        const int J = v.colind[p];
        const int qq = lower_bound_dev(v.colind, s0, s1, J);
        if (qq < s1 && v.colind[qq] == J) hit = qq;
      }
      const unsigned found = __ballot_sync(0xffffffffu, hit >= 0);
      const int nh = __popc(found);
      if (hit >= 0)
        hits[__popc(found & ((1u << lane) - 1u))] = probe_a ? make_int2(p, hit) : make_int2(hit, p);
      __syncwarp();
      for (int c0 = 0; c0 < nh; c0 += 8) {
        // stage the 8 hits' A tiles (I,J) and B tiles (K,J), one coalesced
        // 128-byte load per tile, then build the fragments from shared memory
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const int2 hh = c0 + h < nh ? hits[c0 + h] : make_int2(-1, -1);
          sA[h][lane] = hh.x >= 0 ? val[(size_t)hh.x * 32 + lane] : 0u;
          sB[h][lane] = hh.y >= 0 ? val[(size_t)hh.y * 32 + lane] : 0u;
        }
        __syncwarp();
        unsigned bq[4][2];
#pragma unroll
        for (int nb = 0; nb < 4; ++nb) {
          bq[nb][0] = sB[q4][8 * nb + g];
          bq[nb][1] = sB[q4 + 4][8 * nb + g];
        }
#pragma unroll
        for (int mb = 0; mb < 2; ++mb) {
          const unsigned a0 = sA[q4][16 * mb + g], a1 = sA[q4][16 * mb + g + 8];
          const unsigned a2 = sA[q4 + 4][16 * mb + g], a3 = sA[q4 + 4][16 * mb + g + 8];
#pragma unroll
          for (int nb = 0; nb < 4; ++nb) mma_and_popc(d[mb][nb], a0, a1, a2, a3, bq[nb][0], bq[nb][1]);
        }
        __syncwarp();
      }
      __syncwarp();
    }
    // sum of P over the mask's bits: row r, column c at bit 31-c of M[r]
#pragma unroll
    for (int mb = 0; mb < 2; ++mb) {
      const uint32_t mr0 = __shfl_sync(0xffffffffu, M0, 16 * mb + g);
      const uint32_t mr1 = __shfl_sync(0xffffffffu, M0, 16 * mb + g + 8);
#pragma unroll
      for (int nb = 0; nb < 4; ++nb) {
        const int col = 8 * nb + 2 * q4;
        if ((mr0 >> (31 - col)) & 1u) acc += (unsigned)d[mb][nb][0];
        if ((mr0 >> (30 - col)) & 1u) acc += (unsigned)d[mb][nb][1];
        if ((mr1 >> (31 - col)) & 1u) acc += (unsigned)d[mb][nb][2];
        if ((mr1 >> (30 - col)) & 1u) acc += (unsigned)d[mb][nb][3];
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0 && acc) atomicAdd(count, acc);
}

}  // namespace

namespace {

// The lists and units of a lower triangle, once per graph.
int build_lists(gbo_graph* g, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g->build_mu);
  if (g->tc_nunits >= 0) return GBO_OK;
  const GatherList gl = gather_of(g);
  const size_t n = (size_t)g->nrows;
  const unsigned grid = std::min(blocks_for(g->nrows, 256), (unsigned)num_sms() * 8u);
  const unsigned gw = std::min(blocks_for_warps(g->nrows, kTPB / 32), (unsigned)num_sms() * 8u);
  char* tmp = nullptr;  // {total, bins, ranks, owners' counts, column counts}
  GBO_CUDA_TRY(pool_malloc_async(&tmp, sizeof(long long) + sizeof(int) * (kDegBins + 3 * n), s));
  const int st = [&]() -> int {
    auto* tot = reinterpret_cast<long long*>(tmp);
    int* bins = reinterpret_cast<int*>(tot + 1);
    int *rank = bins + kDegBins, *own = rank + n;
    const int* colcnt = g->outdeg;
    if (!colcnt) {
      int* c = own + n;
      GBO_CUDA_TRY(cudaMemsetAsync(c, 0, sizeof(int) * n, s));
      if (gl.nnz > 0)
        k_count_cols<<<(unsigned)std::min<long long>((gl.nnz + 255) / 256, num_sms() * 32ll), 256, 0, s>>>(gl.col, gl.nnz, c);
      colcnt = c;
    }
    GBO_TRY(list_alloc(&g->tc_ptr, n + 1, s));
    GBO_TRY(list_alloc(&g->tc_col, (size_t)gl.nnz, s));
    GBO_TRY(list_alloc(&g->tc_unit0, n + 1, s));
    GBO_CUDA_TRY(cudaMemsetAsync(bins, 0, sizeof(int) * kDegBins, s));
    k_degree_hist<<<std::min(blocks_for(g->nrows, 4096), (unsigned)num_sms() * 2u), 1024, 0, s>>>(gl, colcnt, bins);
    k_degree_starts<<<1, 1024, 0, s>>>(bins);
    k_degree_ranks<<<blocks_for(g->nrows, 4096), 1024, 0, s>>>(gl, colcnt, bins, rank);
    GBO_CUDA_TRY(cudaMemsetAsync(own, 0, sizeof(int) * n, s));
    k_orient<false><<<gw, kTPB, 0, s>>>(gl, rank, own, nullptr, nullptr);
    GBO_TRY(exclusive_scan_i32_to_i64(own, g->tc_ptr, g->nrows, tot, s));
    GBO_CUDA_TRY(cudaMemsetAsync(own, 0, sizeof(int) * n, s));
    k_orient<true><<<gw, kTPB, 0, s>>>(gl, rank, own, g->tc_ptr, g->tc_col);
    const Lists l{g->tc_ptr, g->tc_col, g->nrows};
    k_tc_unit_counts<<<grid, 256, 0, s>>>(l, own);
    GBO_TRY(exclusive_scan_i32(own, g->tc_unit0, g->nrows, tot, s));
    long long nu = 0;
    const cudaError_t e = read_back(&nu, tot, sizeof(nu), s);
    if (e != cudaSuccess) return fail_cuda(e, "triangle count units");
    if (nu > 2147483647ll) return fail(GBO_ERR_OVERFLOW, "triangle counting: too many entries");
    GBO_TRY(list_alloc(&g->tc_unit, (size_t)nu, s));
    if (nu > 0) k_tc_units<<<grid, 256, 0, s>>>(g->tc_unit0, g->nrows, g->tc_unit);
    GBO_CUDA_TRY(cudaGetLastError());
    GBO_CUDA_TRY(cudaStreamSynchronize(s));
    g->device_bytes += 12LL * (g->nrows + 1) + 4LL * (gl.nnz + nu);
    g->tc_nunits = (int)nu;
    return GBO_OK;
  }();
  cudaFreeAsync(tmp, s);
  if (st != GBO_OK) {  // nothing half-built stays
    cudaStreamSynchronize(s);
    cudaFree(g->tc_ptr);
    cudaFree(g->tc_col);
    cudaFree(g->tc_unit);
    cudaFree(g->tc_unit0);
    g->tc_ptr = nullptr;
    g->tc_col = g->tc_unit = g->tc_unit0 = nullptr;
  }
  return st;
}

bool counted_by_lane(const gbo_graph* g) { return g->gl_short && !g->gl_diag; }

bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(s, &cap);
  return cap != cudaStreamCaptureStatusNone;
}

// Fills in g->tc_lower.
int find_lower(gbo_graph* g, cudaStream_t s) {
  if (g->tc_lower >= 0) return GBO_OK;
  unsigned *d = nullptr, h = 0;
  GBO_CUDA_TRY(pool_malloc_async(&d, sizeof(unsigned), s));
  const GView v = view_of(g);
  const unsigned grid = blocks_for(g->nbr, 256);
  cudaError_t e = cudaMemsetAsync(d, 0, sizeof(unsigned), s);
  switch (g->b) {
    case 4: k_above<4><<<grid, 256, 0, s>>>(v, d); break;
    case 8: k_above<8><<<grid, 256, 0, s>>>(v, d); break;
    case 16: k_above<16><<<grid, 256, 0, s>>>(v, d); break;
    case 32: k_above<32><<<grid, 256, 0, s>>>(v, d); break;
    default: k_above<64><<<grid, 256, 0, s>>>(v, d); break;
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = read_back(&h, d, sizeof(h), s);
  cudaFreeAsync(d, s);
  if (e != cudaSuccess) return fail_cuda(e, "triangle of a matrix");
  g->tc_lower = h ? 0 : 1;
  return GBO_OK;
}

// Whether the count goes over lists, which are built if need be.
bool lists_ready(gbo_graph* g, cudaStream_t s, bool may_build, int* st) {
  if (g->tc_mma || g->nblk < kListTiles) return false;
  const bool first = !g->tc_counted;
  if (may_build) {
    g->tc_counted = true;
    const bool lng = g->nblk > (long long)kLongMean * g->nbr || (long long)g->longest * g->nbr > kSkew * g->nblk;
    if (first && g->nblk < (lng ? kListFirstLong : kListFirst)) return false;
    *st = find_lower(g, s);
    if (*st == GBO_OK && g->tc_lower) *st = build_gather(g, s);
    if (*st == GBO_OK && g->tc_lower && !counted_by_lane(g)) *st = build_lists(g, s);
    if (*st == GBO_ERR_NOMEM) {
      clear_error();
      *st = GBO_OK;
      return false;
    }
    return *st == GBO_OK && g->tc_lower == 1;
  }
  // under capture: what direct counts have built
  return g->tc_lower == 1 && g->gl_nparts >= 0 && (counted_by_lane(g) || g->tc_nunits >= 0);
}

// The tiles' block rows: made by the first direct count, complete when it goes
// on (any stream may read them then), and kept with the graph.  A count under
// capture before that queues an array of its own (`own`, freed in stream order:
// nodes of the captured graph), since nothing it records has run yet.
int tile_rows(gbo_graph* g, cudaStream_t s, bool may_build, int** rows, bool* own) {
  std::lock_guard<std::mutex> lk(g->build_mu);
  *own = false;
  *rows = g->tile_row;
  if (*rows) return GBO_OK;
  int* t = nullptr;
  GBO_TRY(list_alloc(&t, (size_t)g->nblk, s));
  k_tile_row<<<blocks_for_warps(g->nitems, kTPB / 32), kTPB, 0, s>>>(view_of(g), t);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && may_build) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    cudaFreeAsync(t, s);
    return fail_cuda(e, "tiles' block rows");
  }
  *rows = t;
  *own = !may_build;
  if (may_build) {
    g->tile_row = t;
    g->device_bytes += 4LL * g->nblk;
  }
  return GBO_OK;
}

}  // namespace

int tc_launch(gbo_graph* g, unsigned long long* d_count, cudaStream_t s) {
  GBO_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(unsigned long long), s));
  if (g->nblk == 0) return GBO_OK;
  int st = GBO_OK;
  const bool may_build = !capturing(s);
  if (lists_ready(g, s, may_build, &st)) {
    const unsigned cap = (unsigned)num_sms() * 4u;
    if (counted_by_lane(g)) {
      k_tc_lanes<<<std::min(blocks_for(g->nrows, kTPB), cap * 2), kTPB, 0, s>>>(gather_of(g), d_count);
    } else {
      const Lists l{g->tc_ptr, g->tc_col, g->nrows};
      if (g->tc_nunits > 0)
        k_tc_warps<<<std::min(blocks_for_warps(g->tc_nunits, kTcWarps), cap), kTcWarps * 32, 0, s>>>(
            l, g->tc_unit, g->tc_unit0, g->tc_nunits, d_count);
      if (g->gl_diag)
        k_tc_diagonal<<<std::min(blocks_for_warps(g->nrows, kTPB / 32), cap * 2), kTPB, 0, s>>>(gather_of(g), d_count);
    }
    GBO_CUDA_TRY(cudaGetLastError());
    return GBO_OK;
  }
  GBO_TRY(st);
  GView v = view_of(g);
  int* rows = nullptr;
  bool own = false;
  GBO_TRY(tile_rows(g, s, may_build, &rows, &own));
  long long warps = g->nblk;
  long long cap = (long long)num_sms() * 64;  // 64 resident warps per SM
  if (warps > cap * 8) warps = cap * 8;
  const unsigned grid = blocks_for_warps(warps, kTPB / 32);
  switch (g->b) {
    case 4: k_tc<4><<<grid, kTPB, 0, s>>>(v, g->nblk, rows, 0, d_count); break;
    case 8: k_tc<8><<<grid, kTPB, 0, s>>>(v, g->nblk, rows, 0, d_count); break;
    case 16: k_tc<16><<<grid, kTPB, 0, s>>>(v, g->nblk, rows, 0, d_count); break;
    case 32: if (g->tc_mma) {
      k_tc<32><<<grid, kTPB, 0, s>>>(v, g->nblk, rows, 1, d_count);
      k_tc32_mma<<<grid, kTPB, 0, s>>>(v, g->nblk, rows, d_count);
    } else {
      k_tc<32><<<grid, kTPB, 0, s>>>(v, g->nblk, rows, 0, d_count);
    }; break;
    default: k_tc<64><<<grid, kTPB, 0, s>>>(v, g->nblk, rows, 0, d_count); break;
  }
  const cudaError_t e = cudaGetLastError();
  if (own) cudaFreeAsync(rows, s);
  if (e != cudaSuccess) return fail_cuda(e, "triangle count");
  return GBO_OK;
}

}  // namespace gbo

using namespace gbo;

static int check_tc_graph(const gbo_graph* g) {
  if (!g) return fail(GBO_ERR_INVALID, "graph is NULL");
  if (g->layout != GBO_LAYOUT_ROW) return fail(GBO_ERR_UNSUPPORTED, "TC needs the ROW tile layout");
  if (g->nrows != g->ncols) return fail(GBO_ERR_INVALID, "TC needs a square matrix");
  return GBO_OK;
}

extern "C" int gbo_tc_device(const gbo_graph* lower, unsigned long long* d_count,
                             gbo_stream_t stream) {
  clear_error();
  GBO_TRY(check_tc_graph(lower));
  if (!d_count) return fail(GBO_ERR_INVALID, "count is NULL");
  return tc_launch(const_cast<gbo_graph*>(lower), d_count, as_stream(stream));
}

extern "C" int gbo_tc(const gbo_graph* lower, uint64_t* h_count, gbo_stream_t stream) {
  clear_error();
  GBO_TRY(check_tc_graph(lower));
  if (!h_count) return fail(GBO_ERR_INVALID, "count is NULL");
  cudaStream_t s = as_stream(stream);
  unsigned long long* d = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&d, sizeof(unsigned long long), s));
  int st = tc_launch(const_cast<gbo_graph*>(lower), d, s);
  unsigned long long h = 0;
  if (st == GBO_OK) {
    const cudaError_t e = read_back(&h, d, sizeof(h), s);
    if (e != cudaSuccess) st = fail_cuda(e, "tc readback");
  }
  cudaFreeAsync(d, s);
  if (st == GBO_OK) *h_count = h;
  return st;
}
