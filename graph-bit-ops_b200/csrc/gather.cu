// Row lists (gather.cuh) built from the tiles: set bits of every (unit, row),
// rows' lengths and offsets, then the columns.  A unit is at most kUnitTiles
// tiles of a block row, walked by a lane per row: the lane of a hub's row
// walks few tiles, where a unit per work item let it set the time of the
// launches (R-MAT of 20,001 rows, b = 8, count + fill: 286 -> 33 us).
#include <algorithm>

#include "gather.cuh"
#include "scan.cuh"

namespace gbo {

namespace {

constexpr int kTPB = 256;
constexpr int kUnitTiles = 64;

// Units of every block row.
__global__ void k_unit_counts(GView v, int* __restrict__ units) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i < v.nbr) units[i] = (v.rowptr[i + 1] - v.rowptr[i] + kUnitTiles - 1) / kUnitTiles;
}

__global__ void k_unit_rows(const int* __restrict__ unit0, int nbr, int* __restrict__ unit_row) {
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= nbr) return;
  for (int u = unit0[i]; u < unit0[i + 1]; ++u) unit_row[u] = i;
}

struct Units {
  const int *unit0, *unit_row;
};

// The unit of this group of lanes and its tiles [t0, t1); false: none left.
__device__ __forceinline__ bool unit_of(const GView& v, const Units& un, unsigned lane, int W, int G, long long& u,
                                        int& row, int& t0, int& t1) {
  u = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G + lane / W;
  if (u >= un.unit0[v.nbr]) return false;
  row = un.unit_row[u];
  t0 = v.rowptr[row] + (int)(u - un.unit0[row]) * kUnitTiles;
  t1 = min(t0 + kUnitTiles, v.rowptr[row + 1]);
  return true;
}

// Set bits of row r of every unit's tiles (cnt[unit * B + r]).  b = 4 keeps a
// tile's row in the low bits of a byte.
template <int B>
__global__ void __launch_bounds__(kTPB) k_list_count(GView v, Units un, int* __restrict__ cnt) {
  using WT = typename Word<B>::T;
  using L = Lay<B>;
  const unsigned lane = threadIdx.x & 31;
  long long u;
  int row, t0, t1;
  if (!unit_of(v, un, lane, L::W, L::G, u, row, t0, t1)) return;
  const WT* __restrict__ val = reinterpret_cast<const WT*>(v.val);
#pragma unroll
  for (int h = 0; h < L::RPL; ++h) {
    const int r = (int)lane % L::W + 32 * h;
    int c = 0;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) c += popc_w((WT)(val[(size_t)t * B + r] & (WT)((WT)~(WT)0 >> (sizeof(WT) * 8 - B))));
    cnt[u * B + r] = c;
  }
}

// Every unit's count replaced by the row's count in the units before it; the
// row's length.
__global__ void k_list_starts(const int* __restrict__ unit0, long long rows, int b, int* __restrict__ cnt,
                              int* __restrict__ len) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= rows) return;
  const long long row = gid / b, r = gid % b;
  int s = 0;
  const int u1 = unit0[row + 1];
  for (int u = unit0[row]; u < u1; u += 8) {
    int c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) c[q] = u + q < u1 ? cnt[(long long)(u + q) * b + r] : 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (u + q < u1) cnt[(long long)(u + q) * b + r] = s;
      s += c[q];
    }
  }
  len[gid] = s;
}

template <int B>
__global__ void __launch_bounds__(kTPB) k_list_fill(GView v, Units un, const int* __restrict__ cnt,
                                                    const long long* __restrict__ ptr, int* __restrict__ col) {
  using WT = typename Word<B>::T;
  using L = Lay<B>;
  const unsigned lane = threadIdx.x & 31;
  long long u;
  int brow, first, last;
  if (!unit_of(v, un, lane, L::W, L::G, u, brow, first, last)) return;
  const WT* __restrict__ val = reinterpret_cast<const WT*>(v.val);
#pragma unroll
  for (int h = 0; h < L::RPL; ++h) {
    const int r = (int)lane % L::W + 32 * h;
    const long long row = (long long)brow * B + r;
    if (row >= v.nrows) continue;
    int* out = col + ptr[row] + cnt[u * B + r];
    for (int t0 = first; t0 < last; t0 += 8) {
      WT w[8];
      int c[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        w[q] = t0 + q < last ? val[(size_t)(t0 + q) * B + r] : (WT)0;
        c[q] = t0 + q < last ? v.colind[t0 + q] : 0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        for (unsigned long long a = (unsigned long long)w[q] << (64 - B); a;) {
          const int j = __clzll((long long)a);
          a &= ~(0x8000000000000000ull >> j);
          *out++ = c[q] * B + j;
        }
    }
  }
}

// Merge path: the rows that end in the items [i, i + 1) * kPartItems of (row
// ends, set bits).
__device__ __forceinline__ long long path_row(const long long* __restrict__ ptr, int nrows, long long d) {
  const long long nnz = ptr[nrows];
  d = min(d, nrows + nnz);
  long long lo = max(0ll, d - nnz), hi = min(d, (long long)nrows);
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (ptr[mid + 1] <= d - mid - 1) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

__global__ void k_list_parts(const long long* __restrict__ ptr, int nrows, int nparts, GatherPart* __restrict__ part) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nparts) return;
  const long long a0 = path_row(ptr, nrows, i * kPartItems), a1 = path_row(ptr, nrows, (i + 1) * kPartItems);
  part[i] = GatherPart{(int)a0, (int)(a1 - a0), a0 < nrows && ptr[a0] < i * kPartItems - a0 ? 1 : 0, 0};
}

// Bit 0: a column past its row (the lists ascend: the last one tells); bit 1:
// a column equal to its row, given that none is past it; bit 2: a row of more
// than kShortRow set bits; bit 3: one of more than kLongRow.
__global__ void k_list_shape(const long long* __restrict__ ptr, const int* __restrict__ col, int nrows,
                             unsigned* __restrict__ shape) {
  unsigned s = 0u;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nrows; i += (long long)gridDim.x * blockDim.x) {
    const long long e = ptr[i + 1];
    if (e == ptr[i]) continue;
    const int last = col[e - 1];
    s |= (last > i ? 1u : last == i ? 2u : 0u) | (e - ptr[i] > kShortRow ? 4u : 0u) | (e - ptr[i] > kLongRow ? 8u : 0u);
  }
  s = __reduce_or_sync(0xffffffffu, s);
  if ((threadIdx.x & 31) == 0 && s) atomicOr(shape, s);
}

// Long rows: 1 and the number of chunks where a row is one, else 0.
__global__ void k_long_flags(const int* __restrict__ len, int nrows, int* __restrict__ flag, int* __restrict__ chunks) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrows) return;
  const bool l = len[i] > kLongRow;
  flag[i] = l;
  chunks[i] = l ? (len[i] + kLongChunk - 1) / kLongChunk : 0;
}

__global__ void k_long_fill(const int* __restrict__ len, int nrows, const int* __restrict__ at,
                            const int* __restrict__ chunk_at, int* __restrict__ row, int* __restrict__ chunk0) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrows) return;
  if (len[i] > kLongRow) {
    row[at[i]] = (int)i;
    chunk0[at[i]] = chunk_at[i];
  }
  if (i == 0) chunk0[at[nrows]] = chunk_at[nrows];
}

int build_long(gbo_graph* g, const int* len, cudaStream_t s) {
  const size_t n = (size_t)g->nrows;
  int* tmp = nullptr;  // {flags, chunks, their prefix sums}
  GBO_CUDA_TRY(pool_malloc_async(&tmp, sizeof(int) * (4 * n + 2) + sizeof(long long) * 3, s));
  int *flag = tmp, *chunks = flag + n, *at = chunks + n, *chunk_at = at + n + 1;
  auto* tot = reinterpret_cast<long long*>((reinterpret_cast<uintptr_t>(chunk_at + n + 1) + 7) & ~(uintptr_t)7);
  const int st = [&]() -> int {
    unsigned shape = 0;
    GBO_CUDA_TRY(cudaMemsetAsync(tot, 0, sizeof(shape), s));
    k_list_shape<<<std::min(blocks_for(g->nrows, 256), (unsigned)num_sms() * 8u), 256, 0, s>>>(
        g->gl_ptr, g->gl_col, g->nrows, reinterpret_cast<unsigned*>(tot));
    cudaError_t e = read_back(&shape, tot, sizeof(shape), s);
    if (e != cudaSuccess) return fail_cuda(e, "row lists");
    g->gl_lower = !(shape & 1);
    g->gl_diag = (shape & 2) != 0;
    g->gl_short = !(shape & 4);
    if (!(shape & 8)) {
      GBO_TRY(list_alloc(&g->gl_long_row, 0, s));
      GBO_TRY(list_alloc(&g->gl_long_chunk0, 1, s));
      GBO_CUDA_TRY(cudaMemsetAsync(g->gl_long_chunk0, 0, sizeof(int), s));
      GBO_CUDA_TRY(cudaStreamSynchronize(s));
      return GBO_OK;
    }
    k_long_flags<<<blocks_for(g->nrows, 256), 256, 0, s>>>(len, g->nrows, flag, chunks);
    GBO_TRY(exclusive_scan_i32(flag, at, g->nrows, tot, s));
    GBO_TRY(exclusive_scan_i32(chunks, chunk_at, g->nrows, tot + 1, s));
    long long h[2] = {0, 0};
    e = read_back(h, tot, sizeof(h), s);
    if (e != cudaSuccess) return fail_cuda(e, "long rows");
    if (h[1] > 2147483647ll) return fail(GBO_ERR_OVERFLOW, "row lists: too many entries");
    GBO_TRY(list_alloc(&g->gl_long_row, (size_t)h[0], s));
    GBO_TRY(list_alloc(&g->gl_long_chunk0, (size_t)h[0] + 1, s));
    k_long_fill<<<blocks_for(g->nrows, 256), 256, 0, s>>>(len, g->nrows, at, chunk_at, g->gl_long_row,
                                                          g->gl_long_chunk0);
    GBO_CUDA_TRY(cudaGetLastError());
    GBO_CUDA_TRY(cudaStreamSynchronize(s));  // the lists may be read on any stream from here
    g->gl_nlong = (int)h[0];
    g->gl_nlchunk = (int)h[1];
    g->device_bytes += 4LL * (2 * h[0] + 1);
    return GBO_OK;
  }();
  cudaFreeAsync(tmp, s);
  return st;
}

template <int B>
int build_impl(gbo_graph* g, int* tmp, long long max_units, int* len, long long* tot, cudaStream_t s) {
  const GView v = view_of(g);
  int *unit0 = tmp, *unit_row = unit0 + v.nbr + 1, *cnt = unit_row + max_units;
  k_unit_counts<<<blocks_for(v.nbr, 256), 256, 0, s>>>(v, len);
  GBO_TRY(exclusive_scan_i32(len, unit0, v.nbr, tot, s));
  k_unit_rows<<<blocks_for(v.nbr, 256), 256, 0, s>>>(unit0, v.nbr, unit_row);
  const Units un{unit0, unit_row};
  const unsigned grid = blocks_for_warps((max_units + Lay<B>::G - 1) / Lay<B>::G, kTPB / 32);
  k_list_count<B><<<grid, kTPB, 0, s>>>(v, un, cnt);
  const long long rows = (long long)v.nbr * B;
  k_list_starts<<<blocks_for(rows, 256), 256, 0, s>>>(unit0, rows, B, cnt, len);
  GBO_CUDA_TRY(cudaGetLastError());
  GBO_TRY(exclusive_scan_i32_to_i64(len, g->gl_ptr, v.nrows, tot, s));
  long long nnz = 0;
  const cudaError_t e = read_back(&nnz, tot, sizeof(nnz), s);
  if (e != cudaSuccess) return fail_cuda(e, "row list lengths");
  const long long parts = (v.nrows + nnz + kPartItems - 1) / kPartItems;
  if (parts > 2147483646ll) return fail(GBO_ERR_OVERFLOW, "row lists: too many entries");
  GBO_TRY(list_alloc(&g->gl_col, (size_t)nnz, s));
  GatherPart* part = nullptr;
  GBO_TRY(list_alloc(&part, (size_t)parts, s));
  g->gl_part = part;
  k_list_fill<B><<<grid, kTPB, 0, s>>>(v, un, cnt, g->gl_ptr, g->gl_col);
  k_list_parts<<<blocks_for(parts, 256), 256, 0, s>>>(g->gl_ptr, v.nrows, (int)parts, part);
  GBO_CUDA_TRY(cudaGetLastError());
  GBO_TRY(build_long(g, len, s));
  g->gl_nparts = (int)parts;
  g->gl_nnz = nnz;
  g->device_bytes += 4LL * nnz + 8LL * (v.nrows + 1) + (long long)sizeof(GatherPart) * parts;
  return GBO_OK;
}

}  // namespace

void lists_idle(const void* list) {
  if (!list) return;
  cudaPointerAttributes a;
  int dev = 0;
  if (cudaPointerGetAttributes(&a, list) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) return;
  if (a.device != dev) cudaSetDevice(a.device);
  cudaDeviceSynchronize();
  if (a.device != dev) cudaSetDevice(dev);
}

void free_gather(gbo_graph* g) {
  lists_idle(g->gl_ptr);
  cudaFree(g->gl_ptr);
  cudaFree(g->gl_col);
  cudaFree(g->gl_part);
  cudaFree(g->gl_long_row);
  cudaFree(g->gl_long_chunk0);
  g->gl_long_row = nullptr;
  g->gl_long_chunk0 = nullptr;
  g->gl_nlong = 0;
  g->gl_nlchunk = 0;
  g->gl_ptr = nullptr;
  g->gl_col = nullptr;
  g->gl_part = nullptr;
  g->gl_nparts = -1;
}

int build_gather(gbo_graph* g, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g->build_mu);
  if (g->gl_nparts >= 0) return GBO_OK;
  if (g->layout != GBO_LAYOUT_ROW) return fail(GBO_ERR_UNSUPPORTED, "row lists need the ROW tile layout");
  if (g->nrows <= 0) {
    g->gl_nparts = 0;
    return GBO_OK;
  }
  const size_t rows = (size_t)g->nbr * (size_t)g->b;
  const long long units = g->nbr + g->nblk / kUnitTiles;  // the most there can be
  int* tmp = nullptr;  // {first units, their block rows, counts per (unit, row), lengths}
  long long* tot = nullptr;
  const size_t head = (size_t)g->nbr + 1 + (size_t)units * ((size_t)g->b + 1);
  GBO_CUDA_TRY(pool_malloc_async(&tmp, sizeof(int) * (head + rows), s));
  int st = GBO_OK;
  cudaError_t e = pool_malloc_async(&tot, sizeof(long long), s);
  if (e == cudaSuccess) e = pool_malloc_async(&g->gl_ptr, sizeof(long long) * ((size_t)g->nrows + 1), s);
  if (e != cudaSuccess) st = fail_cuda(e, "row lists");
  int* len = tmp + head;
  if (st == GBO_OK) {
    switch (g->b) {
      case 4: st = build_impl<4>(g, tmp, units, len, tot, s); break;
      case 8: st = build_impl<8>(g, tmp, units, len, tot, s); break;
      case 16: st = build_impl<16>(g, tmp, units, len, tot, s); break;
      case 32: st = build_impl<32>(g, tmp, units, len, tot, s); break;
      default: st = build_impl<64>(g, tmp, units, len, tot, s); break;
    }
  }
  cudaFreeAsync(tmp, s);
  if (tot) cudaFreeAsync(tot, s);
  if (st != GBO_OK) {
    cudaStreamSynchronize(s);
    free_gather(g);
  }
  return st;
}

GatherList gather_of(const gbo_graph* g) {
  GatherList gl;
  gl.ptr = g->gl_ptr;
  gl.col = g->gl_col;
  gl.part = static_cast<const GatherPart*>(g->gl_part);
  gl.nnz = g->gl_nnz;
  gl.nrows = g->nrows;
  gl.nparts = g->gl_nparts;
  gl.nlong = g->gl_nlong;
  gl.nchunk = g->gl_nlchunk;
  gl.long_row = g->gl_long_row;
  gl.long_chunk0 = g->gl_long_chunk0;
  return gl;
}

}  // namespace gbo
