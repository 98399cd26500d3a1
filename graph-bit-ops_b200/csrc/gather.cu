// Row lists (gather.cuh) built from the tiles: set bits of every (work item,
// row), rows' lengths and offsets, then the columns.  Work items bound what
// one warp walks: a hub block row is many items.
#include "gather.cuh"
#include "scan.cuh"

namespace gbo {

namespace {

constexpr int kTPB = 256;

__device__ __forceinline__ long long build_item(unsigned lane, int W, int G) {
  return (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * G + lane / W;
}

// Set bits of row r of every work item's tiles (cnt[item * B + r]); whole
// rows' lengths too where the item is the whole block row.
template <int B>
__global__ void __launch_bounds__(kTPB) k_list_count(GView v, int* __restrict__ cnt, int* __restrict__ len) {
  using WT = typename Word<B>::T;
  using L = Lay<B>;
  const unsigned lane = threadIdx.x & 31;
  const long long item = build_item(lane, L::W, L::G);
  if (item >= v.nitems) return;
  const gbo_item it = v.items[item];
  const WT* __restrict__ val = reinterpret_cast<const WT*>(v.val);
#pragma unroll
  for (int h = 0; h < L::RPL; ++h) {
    const int r = (int)lane % L::W + 32 * h;
    int c = 0;
#pragma unroll 8
    for (int t = it.t0; t < it.t1; ++t) c += popc_w((WT)(val[(size_t)t * B + r] & (WT)((WT)~(WT)0 >> (sizeof(WT) * 8 - B))));
    cnt[item * B + r] = c;
    if (it.slot < 0) len[(long long)it.row * B + r] = c;
  }
}

// Split block rows: each item's count replaced by the row's count in the
// items before it; the row's length.  The items of a block row are adjacent
// and its slots are in their order.
template <int B>
__global__ void k_list_split(GView v, const int* __restrict__ first_item, int* __restrict__ cnt, int* __restrict__ len) {
  const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (long long)v.nsplit * B) return;
  const gbo_split sp = v.splits[gid / B];
  const int r = (int)(gid % B);
  int s = 0;
  for (int q = 0; q < sp.nslots; ++q) {
    int* c = cnt + ((long long)first_item[gid / B] + q) * B + r;
    const int t = *c;
    *c = s;
    s += t;
  }
  len[(long long)sp.row * B + r] = s;
}

// First work item of every split block row.
__global__ void k_list_first(GView v, int* __restrict__ first_item) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.nitems) return;
  const gbo_item it = v.items[i];
  if (it.slot < 0 || it.t0 != v.rowptr[it.row]) return;
  int lo = 0, hi = v.nsplit - 1;  // splits ascend by row
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (v.splits[mid].row < it.row) lo = mid + 1;
    else hi = mid;
  }
  first_item[lo] = (int)i;
}

template <int B>
__global__ void __launch_bounds__(kTPB) k_list_fill(GView v, const int* __restrict__ cnt,
                                                    const long long* __restrict__ ptr, int* __restrict__ col) {
  using WT = typename Word<B>::T;
  using L = Lay<B>;
  const unsigned lane = threadIdx.x & 31;
  const long long item = build_item(lane, L::W, L::G);
  if (item >= v.nitems) return;
  const gbo_item it = v.items[item];
  const WT* __restrict__ val = reinterpret_cast<const WT*>(v.val);
#pragma unroll
  for (int h = 0; h < L::RPL; ++h) {
    const int r = (int)lane % L::W + 32 * h;
    const long long row = (long long)it.row * B + r;
    if (row >= v.nrows) continue;
    int* out = col + ptr[row] + (it.slot >= 0 ? cnt[item * B + r] : 0);
    for (int t0 = it.t0; t0 < it.t1; t0 += 8) {
      WT w[8];
      int c[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        w[u] = t0 + u < it.t1 ? val[(size_t)(t0 + u) * B + r] : (WT)0;
        c[u] = t0 + u < it.t1 ? v.colind[t0 + u] : 0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        for (unsigned long long a = (unsigned long long)w[u] << (64 - B); a;) {
          const int j = __clzll((long long)a);
          a &= ~(0x8000000000000000ull >> j);
          *out++ = c[u] * B + j;
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
    k_long_flags<<<blocks_for(g->nrows, 256), 256, 0, s>>>(len, g->nrows, flag, chunks);
    GBO_TRY(exclusive_scan_i32(flag, at, g->nrows, tot, s));
    GBO_TRY(exclusive_scan_i32(chunks, chunk_at, g->nrows, tot + 1, s));
    long long h[2] = {0, 0};
    const cudaError_t e = read_back(h, tot, sizeof(h), s);
    if (e != cudaSuccess) return fail_cuda(e, "long rows");
    if (h[1] > 2147483647ll) return fail(GBO_ERR_OVERFLOW, "row lists: too many entries");
    GBO_CUDA_TRY(cudaMalloc(&g->gl_long_row, sizeof(int) * (size_t)(h[0] > 0 ? h[0] : 1)));
    GBO_CUDA_TRY(cudaMalloc(&g->gl_long_chunk0, sizeof(int) * (size_t)(h[0] + 1)));
    k_long_fill<<<blocks_for(g->nrows, 256), 256, 0, s>>>(len, g->nrows, at, chunk_at, g->gl_long_row,
                                                          g->gl_long_chunk0);
    GBO_CUDA_TRY(cudaGetLastError());
    g->gl_nlong = (int)h[0];
    g->gl_nlchunk = (int)h[1];
    g->device_bytes += 4LL * (2 * h[0] + 1);
    return GBO_OK;
  }();
  cudaFreeAsync(tmp, s);
  return st;
}

template <int B>
int build_impl(gbo_graph* g, int* cnt, int* len, int* first, long long* tot, cudaStream_t s) {
  const GView v = view_of(g);
  const unsigned grid = blocks_for_warps(((long long)v.nitems + Lay<B>::G - 1) / Lay<B>::G, kTPB / 32);
  k_list_count<B><<<grid, kTPB, 0, s>>>(v, cnt, len);
  if (v.nsplit > 0) {
    k_list_first<<<blocks_for(v.nitems, 256), 256, 0, s>>>(v, first);
    k_list_split<B><<<blocks_for((long long)v.nsplit * B, 256), 256, 0, s>>>(v, first, cnt, len);
  }
  GBO_CUDA_TRY(cudaGetLastError());
  GBO_TRY(exclusive_scan_i32_to_i64(len, g->gl_ptr, v.nrows, tot, s));
  long long nnz = 0;
  const cudaError_t e = read_back(&nnz, tot, sizeof(nnz), s);
  if (e != cudaSuccess) return fail_cuda(e, "row list lengths");
  const long long parts = (v.nrows + nnz + kPartItems - 1) / kPartItems;
  if (parts > 2147483646ll) return fail(GBO_ERR_OVERFLOW, "row lists: too many entries");
  GBO_CUDA_TRY(cudaMalloc(&g->gl_col, sizeof(int) * (size_t)(nnz > 0 ? nnz : 1)));
  GBO_CUDA_TRY(cudaMalloc(&g->gl_part, sizeof(GatherPart) * (size_t)(parts > 0 ? parts : 1)));
  k_list_fill<B><<<grid, kTPB, 0, s>>>(v, cnt, g->gl_ptr, g->gl_col);
  k_list_parts<<<blocks_for(parts, 256), 256, 0, s>>>(g->gl_ptr, v.nrows, (int)parts,
                                                      static_cast<GatherPart*>(g->gl_part));
  GBO_CUDA_TRY(cudaGetLastError());
  GBO_TRY(build_long(g, len, s));
  g->gl_nparts = (int)parts;
  g->gl_nnz = nnz;
  g->device_bytes += 4LL * nnz + 8LL * (v.nrows + 1) + (long long)sizeof(GatherPart) * parts;
  return GBO_OK;
}

}  // namespace

void free_gather(gbo_graph* g) {
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
  if (g->gl_nparts >= 0) return GBO_OK;
  if (g->layout != GBO_LAYOUT_ROW) return fail(GBO_ERR_UNSUPPORTED, "row lists need the ROW tile layout");
  if (g->nrows <= 0) {
    g->gl_nparts = 0;
    return GBO_OK;
  }
  const size_t rows = (size_t)g->nbr * (size_t)g->b, items = (size_t)g->nitems;
  int* tmp = nullptr;  // {counts per (item, row), lengths, first items}
  long long* tot = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&tmp, sizeof(int) * (items * (size_t)g->b + rows + (size_t)g->nsplit + 1), s));
  int st = GBO_OK;
  cudaError_t e = pool_malloc_async(&tot, sizeof(long long), s);
  if (e == cudaSuccess) e = cudaMalloc(&g->gl_ptr, sizeof(long long) * ((size_t)g->nrows + 1));
  if (e != cudaSuccess) st = fail_cuda(e, "row lists");
  int* len = tmp + items * (size_t)g->b;
  int* first = len + rows;
  if (st == GBO_OK) {
    switch (g->b) {
      case 4: st = build_impl<4>(g, tmp, len, first, tot, s); break;
      case 8: st = build_impl<8>(g, tmp, len, first, tot, s); break;
      case 16: st = build_impl<16>(g, tmp, len, first, tot, s); break;
      case 32: st = build_impl<32>(g, tmp, len, first, tot, s); break;
      default: st = build_impl<64>(g, tmp, len, first, tot, s); break;
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
