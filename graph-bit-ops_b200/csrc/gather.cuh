// Row lists of a ROW-layout graph, and the balanced gather over them for the
// iterations that gather one value per set bit (PageRank and its variants).
// Connected components, triangle counts (tc.cu) and multi-source BFS with wide
// frontier rows (ms_kernels.cuh) walk the same lists in their own ways.
//
// For a value gather the tiles only get in the way: R-MAT graphs hold 1.1 set
// bits per non-empty row word, and walking words dealt a warp's lanes uneven
// work (rows of one to 64 words, then a shuffle search and a segmented scan
// per 32 words).  The row lists are the set columns of every row, 4 bytes
// each, in ascending order (ptr/col, a CSR without the duplicates a packed
// CSR may have had), built from the tiles on first use.
//
// Work split: merge path (Merrill and Garland, "Merge-based parallel sparse
// matrix-vector multiplication", SC 2016).  Row ends and set bits form one
// sequence of nrows + nnz items; part i is its items [i * kPartItems,
// (i + 1) * kPartItems), so every part has the same work whatever the row
// lengths, empty rows included.  A warp takes a part at a time (a block per
// part spent a third of its time at its own barriers).
//
// The gathers: one from L2 moves a 32-byte sector a clock and SM on B200 (290
// G/s over the chip, measured), one that hits L1 three lanes a clock (860
// G/s).  So the shared memory is kept small, and the rest of it is L1.  (A
// table of the 24,576 hottest columns' values in shared memory, 3,250 G/s,
// took L1 from the others: R-MAT 22 15.2 ms for 20 iterations instead of
// 11.7; only graphs with scattered hubs gained, 0.93 for 1.00 ms.)
#pragma once

#include "bmv.cuh"

namespace gbo {

constexpr int kGatherTPB = 1024;  // one block an SM
constexpr int kGatherWarps = kGatherTPB / 32;
// Items per lane; odd, so that lanes' runs in shared memory start on different
// banks.  5 / 7 / 9 / 11 / 13: R-MAT 21 PageRank 4.82 / 4.52 / 4.56 / 4.74 /
// 5.06 ms, a mesh of 640,000 0.60 / 0.55 / 0.56 / 0.54 / 0.53 ms.
constexpr int kGatherItems = 7;
constexpr int kPartItems = 32 * kGatherItems;

// A part: rows [a0, a0 + rows) end in it; row a0 began in an earlier part
// when `open`.
struct __align__(16) GatherPart {
  int a0, rows, open, pad;
};

struct GatherList {
  const long long* __restrict__ ptr = nullptr;  // nrows + 1
  const int* __restrict__ col = nullptr;        // ptr[nrows]
  const GatherPart* __restrict__ part = nullptr;  // nparts
  long long nnz = 0;
  int nrows = 0;
  int nparts = 0;
  // rows of more than kLongRow set bits, for kernels that give a row a warp:
  // chunks of kLongChunk set bits, long row q's from chunk0[q] on
  int nlong = 0;
  int nchunk = 0;
  const int* __restrict__ long_row = nullptr;
  const int* __restrict__ long_chunk0 = nullptr;
};

constexpr int kShortRow = 8;
constexpr int kLongRow = 256;
constexpr int kLongChunk = 256;

// Index among the long rows of the last one whose key (its row, or its first
// chunk) is at most x.
__device__ __forceinline__ int long_index(const int* __restrict__ key, int n, int x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (key[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Build g's row lists if needed (synchronises `s` when it does).
int build_gather(gbo_graph* g, cudaStream_t s);

// The lists' memory: from the library's pool, which has it mapped already when
// a program makes one graph after another (cudaMalloc took 0.1-0.4 ms an
// array).  Freeing waits for the device, as cudaFree does for its own memory.
template <typename T>
int list_alloc(T** p, size_t count, cudaStream_t s) {
  GBO_CUDA_TRY(pool_malloc_async(p, sizeof(T) * (count > 0 ? count : 1), s));
  return GBO_OK;
}
void lists_idle(const void* list);  // before cudaFree of a list
GatherList gather_of(const gbo_graph* g);

// Shared memory of a warp's part: the rows' sums (8 bytes each), the gathered
// values (4) and the row that ends at each of them (2, where the flag bit is
// set); values + rows <= kPartItems.
struct GatherShared {
  double buf[kPartItems];
  unsigned flag[kGatherItems + 1];  // and a word past the end
};

// The set bits of part i: [first, first + count).
__device__ __forceinline__ long long gather_first(const GatherPart& p, int i) {
  return (long long)i * kPartItems - p.a0;
}
__device__ __forceinline__ int gather_count(const GatherList& gl, const GatherPart& p, int i) {
  return (int)min((long long)(kPartItems - p.rows), gl.nnz - gather_first(p, i));
}

// This lane's columns of part i (coalesced; the list is read once a sweep).
__device__ __forceinline__ void gather_columns(const GatherList& gl, const GatherPart& p, int i, unsigned lane,
                                               int (&c)[kGatherItems]) {
  const int k = gather_count(gl, p, i);
  const int* __restrict__ src = gl.col + gather_first(p, i) + lane;
#pragma unroll
  for (int u = 0; u < kGatherItems; ++u) c[u] = (int)lane + 32 * u < k ? __ldcs(src + 32 * u) : 0;
}

// Sums (fp64) of the part's gathered values x (lane l holds values l, l + 32,
// ...) over its rows, by one warp: the sum of row a0 + j in sh.buf[j] for the
// rows that end here (row a0: only this part's share of it when p.open);
// returns, in every lane, the share of row a0 + rows that this part holds.
// Every sum adds its terms in an order that depends on the graph alone.
__device__ __forceinline__ double gather_reduce(const GatherList& gl, const GatherPart& p, int i, GatherShared& sh,
                                                unsigned lane, float (&x)[kGatherItems]) {
  const int k = gather_count(gl, p, i);
  const long long e0 = gather_first(p, i);
  double* sums = sh.buf;
  float* val = reinterpret_cast<float*>(sh.buf + p.rows);
  unsigned short* row = reinterpret_cast<unsigned short*>(val + k);
  if (lane <= kGatherItems) sh.flag[lane] = 0u;
  __syncwarp();
  // row ends: rows without a set bit here have the sum 0
  for (int j = (int)lane; j < p.rows; j += 32) {
    const int b = (int)max(gl.ptr[p.a0 + j] - e0, 0ll), e = (int)(gl.ptr[p.a0 + j + 1] - e0);
    if (e > b) {
      row[e - 1] = (unsigned short)j;
      atomicOr(sh.flag + ((e - 1) >> 5), 1u << ((e - 1) & 31));
    } else {
      sums[j] = 0.0;
    }
  }
#pragma unroll
  for (int u = 0; u < kGatherItems; ++u)
    if ((int)lane + 32 * u < k) val[lane + 32 * u] = x[u];
  __syncwarp();
  // this lane's run of kGatherItems values: the first row that ends in it may
  // have begun before, the others are its own
  const int q0 = (int)lane * kGatherItems;
  const unsigned ends = __funnelshift_r(sh.flag[q0 >> 5], sh.flag[(q0 >> 5) + 1], q0 & 31);
#pragma unroll
  for (int u = 0; u < kGatherItems; ++u) x[u] = q0 + u < k ? val[q0 + u] : 0.f;
  double acc = 0.0, first = 0.0;
  int first_row = -1;
#pragma unroll
  for (int u = 0; u < kGatherItems; ++u) {
    acc += (double)x[u];
    if ((ends >> u) & 1u) {
      const int r = row[q0 + u];
      sums[r] = acc;
      if (first_row < 0) {
        first_row = r;
        first = acc;
      }
      acc = 0.0;
    }
  }
  // carry into each lane: the sums left open by the lanes before it, back to
  // the last one that ended a row (segmented scan)
  bool ended = first_row >= 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double y = __shfl_up_sync(0xffffffffu, acc, o);
    const bool f = __shfl_up_sync(0xffffffffu, ended, o);
    if ((int)lane >= o) {
      if (!ended) acc += y;
      ended = ended || f;
    }
  }
  const double in = __shfl_up_sync(0xffffffffu, acc, 1);
  if (first_row >= 0 && lane > 0) sums[first_row] = in + first;
  __syncwarp();
  return __shfl_sync(0xffffffffu, acc, 31);
}

// The sum of row p.a0 of part i when it began in an earlier part and ends
// here: the shares `tail` of the parts it runs through, in order, then this
// part's `head`.  Called by whole warps, one part a lane (want: this lane has
// such a row); rows over many parts are added up by the warp.
__device__ __forceinline__ double gather_open_sum(const GatherList& gl, const GatherPart& p, int i, bool want,
                                                  const double* __restrict__ head, const double* __restrict__ tail) {
  constexpr int kAlone = 4;
  const unsigned lane = threadIdx.x & 31;
  int s = i;  // the part that holds the row's first set bit
  if (want) s = (int)((p.a0 + gl.ptr[p.a0]) / kPartItems);
  double a = 0.0;
  if (want && i - s <= kAlone)
    for (int q = s; q < i; ++q) a += tail[q];
  for (unsigned m = __ballot_sync(0xffffffffu, want && i - s > kAlone); m; m &= m - 1) {
    const int l = __ffs(m) - 1;
    const int b = __shfl_sync(0xffffffffu, s, l), e = __shfl_sync(0xffffffffu, i, l);
    double v = 0.0;
    for (int q = b + (int)lane; q < e; q += 32) v += tail[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((int)lane == l) a = v;
  }
  return want ? a + head[i] : 0.0;
}

}  // namespace gbo
