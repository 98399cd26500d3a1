// B2SR packing on the device (replaces the host-serial csr2bsr_batch_*,
// algorithm/csr2bsr_batch_bsrbmv.cu:9-946, and bsrbmm/csr2bsr_batch.cu).
//
// The reference walks block rows on the host, runs cuSPARSE csr2bsr into a
// dense float b x b buffer per slab and packs it with ToBit*Col.  Here one
// warp lane owns one CSR row of a slab of b rows (b <= 32: 32/b slabs per
// warp; b = 64: each lane owns rows r and r+32).  Because CSR rows are
// sorted, the slab's tiles come out in ascending block-column order by a
// b-way merge: every step takes the smallest head block column m over the
// slab's rows (a segmented shuffle min), each lane ORs the bits of all its
// entries in block column m into its tile row word, and the group emits one
// tile.  A count pass sizes each block row; a scan gives bsrRowPtr; a fill
// pass writes bsrColInd and the tile words (one coalesced store of b words).
// The merge takes one step per tile, with the lanes of rows that miss the
// tile idle, so slabs of more than a few entries go to k_pack_wide instead: a
// block per slab, a thread per entry (see there).
#include <vector>
#include <algorithm>
#include "graph.cuh"

namespace gbo {

namespace {

constexpr int kPackTPB = 256;

template <int B>
struct SlabMap {
  // lanes per slab and slabs per warp
  static constexpr int W = B >= 32 ? 32 : B;
  static constexpr int G = 32 / W;
  static constexpr int RPL = B > 32 ? 2 : 1;  // rows per lane
};

__device__ __forceinline__ int seg_min(int v, int width) {
  for (int o = width >> 1; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Per-lane cursor over one CSR row; head is the column at pos.
struct RowCursor {
  int pos, end, head;
};

__device__ __forceinline__ void init_cursor(RowCursor& c, const int* __restrict__ rowptr, const int* __restrict__ colind,
                                            int row, int nrows, long long nnz, unsigned* derr) {
  c.pos = 0;
  c.end = 0;
  if (row < nrows) {
    const int a = rowptr[row], e = rowptr[row + 1];
    if (a < 0 || e < a || e > nnz) {
      atomicOr(derr, DERR_ROWPTR);
    } else {
      c.pos = a;
      c.end = e;
    }
  }
  c.head = c.pos < c.end ? colind[c.pos] : kINF;
}

template <int B>
__device__ __forceinline__ int head_block(const RowCursor& c) {
  return c.pos < c.end ? c.head / B : kINF;
}

// Consume all entries of block column m from the cursor; OR their bits.  An
// entry below the one before it marks the row unsorted.
template <int B, typename WT>
__device__ __forceinline__ void consume(RowCursor& c, const int* __restrict__ colind, int m,
                                        int ncols, WT& word, unsigned* derr, bool build) {
  while (c.pos < c.end && c.head / B == m) {
    const int col = c.head;
    if (col < 0 || col >= ncols) atomicOr(derr, DERR_COL_BOUNDS);
    if (build) word |= (WT)((WT)1 << (B - 1 - ((unsigned)col % B)));
    if (++c.pos >= c.end) break;
    c.head = colind[c.pos];
    if (c.head < col) atomicOr(derr, DERR_UNSORTED);
  }
}

// Which slabs go to k_pack_wide.  The merge takes a step per tile and, inside
// it, a turn per entry of the longest run, so a slab may be wide when it has
// more than merge_tiles tiles or a row of more than kMergeRow entries.  The
// fill pass knows the tiles; the count pass bounds them by the slab's entries
// (kMergeEntries, which also keeps short slabs of long rows) and by the block
// columns between its first and its last one, and takes the slab only if the
// rows' last entries lie in many of these: a mesh's rows lie side by side, seven
// tiles over any span.  k_pack asks and lists the slab's units.
// Measured (count and fill, us): the merge alone takes 24,700 on R-MAT 19
// (16 edges a vertex, b = 32), where block row 0 alone has 16,384 tiles; wide
// slabs past 48 / 64 / 96 tiles 662 / 660 / 696, and at b = 4 (1,138 / 989 /
// 987, so 80 there).  Meshes (250 entries and 7 tiles a slab at b = 32) merge
// in 92 and would take 185 as wide slabs; a dense 1,100-vertex R-MAT (35
// tiles, rows of hundreds) merges in 231 and takes 144.  kMergeEntries 128 is
// for b = 16 meshes (115; 173 at 64 entries) at the cost of 2 % on R-MAT.
//
// A wide slab costs its entries and a pass over the bitmap of *all* block
// columns, so it also needs enough steps for that (words of the bitmap a step,
// at most: fill_words, count_words) -- or to be a straggler, with more than
// 1 / kStragglers of the graph's work and kAboveMean times a slab's mean, which
// the merge would finish last: no more than kStragglers slabs are, so the pass
// stays linear in the graph -- or to be one of so few slabs that the bitmaps of
// all of them take less than its own merge (kFewSlabs: a block goes through a
// word in 2.3 ns, the merge through a step in 240 and more; 3 rows of 3,000
// entries, 30 M columns, b = 4 2,576 / 238 us, 100 rows of 700, 4 M columns, b = 8
// 954 / 127).  Where the sides meet (uniform graphs, merge / wide, us): fill b = 4,
// 2.7 words a tile 75 / 108; b = 8, 2.7 148 / 148; b = 16, 8 265 / 288; b = 32,
// 10.7 17,525 / 21,143; b = 64, 1.4 15,045 / 15,376; count b = 8, 10.7 words an
// entry 276 / 201, 42.7 869 / 1,216; b = 16, 42.7 6,141 / 5,020.  Stragglers (R-MAT
// 19 / 22, b = 8, fill, us): 16,384 and 4 times the mean 741 / 12,857, 32,768 and 2
// 533 / 17,369, 65,536 and 2 539 / 20,756.
// Without this rule the fill of uniform graphs of 2^23 vertices, 24 a row, took
// 2,574 ms at b = 4 and 736 at b = 8 (merge: 4.3, 4.9), the count of a mesh of
// that size at b = 32 1,299 us (merge: 247).
constexpr int kMergeEntries = 128;
constexpr int kMergeRow = 48;
template <int B>
__host__ __device__ constexpr int merge_tiles() {
  return B == 4 ? 80 : 48;
}
template <int B>
__host__ __device__ constexpr int fill_words() {
  return B == 4 ? 1 : B == 8 ? 3 : B == 16 ? 7 : B == 32 ? 10 : 4;
}
template <int B>
__host__ __device__ constexpr int count_words() {
  return 3 * B;
}
constexpr long long kStragglers = 32768;
constexpr int kAboveMean = 2;
constexpr long long kFewSlabs = 4096;
constexpr int kUnitEntries = 2048;

// Units of a slab with this many entries.
__host__ __device__ __forceinline__ int units_of(long long entries) {
  return entries <= 2 * kUnitEntries ? 1 : (int)((entries + kUnitEntries - 1) / kUnitEntries);
}

struct __align__(16) WideUnit {
  int slab, index, count, first;  // unit `index` of the slab's `count`, which start at unit `first`
};

// The units of the wide slabs, listed by k_pack and taken by k_pack_wide.
struct WideList {
  WideUnit* units = nullptr;          // null: no slab is wide
  unsigned long long* ctr = nullptr;  // {units listed, taken, taken by the hubs' count}, zeroed by the caller
  long long cap = 0;
};

// List a wide slab's units (one lane).  Row pointers that are not monotone
// can ask for more than `cap`: those units get no slab.
__device__ __forceinline__ void list_units(const WideList& wl, int slab, long long entries, long long nnz,
                                           unsigned* derr) {
  const int n = entries > nnz ? 0 : units_of(entries);
  const unsigned long long first = atomicAdd(wl.ctr, (unsigned long long)n);
  const bool fits = n > 0 && first + n <= (unsigned long long)wl.cap;
  if (!fits) atomicOr(derr, DERR_ROWPTR);
  for (int i = 0; i < n && first + i < (unsigned long long)wl.cap; ++i)
    wl.units[first + i] = WideUnit{fits ? slab : -1, i, n, (int)first};
}

template <int B>
__device__ __forceinline__ long long slab_entries(const int* __restrict__ rowptr, long long slab, int nrows) {
  const long long a = slab * B, e = a + B < nrows ? a + B : nrows;
  return (long long)rowptr[e] - (long long)rowptr[a];
}

// COUNT (build=false) and FILL (build=true) share one body.  A wide slab is
// listed for k_pack_wide and left alone (its count starts at zero: its units
// add to it).
template <int B, bool BUILD>
__global__ void __launch_bounds__(kPackTPB) k_pack(const int* __restrict__ rowptr,
                                                   const int* __restrict__ colind, int nrows,
                                                   int ncols, long long nnz, int nbr,
                                                   int* __restrict__ counts,
                                                   const int* __restrict__ bsr_rowptr,
                                                   int* __restrict__ bsr_colind,
                                                   typename Word<B>::T* __restrict__ bsr_val,
                                                   int layout, WideList wl, unsigned* derr) {
  using WT = typename Word<B>::T;
  using M = SlabMap<B>;
  const unsigned lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int g = lane / M::W;          // slab within warp
  const int r = lane % M::W;          // row within slab (first row for B=64)
  const long long slab = warp * M::G + g;
  if (warp * M::G >= nbr) return;     // whole warp idle (uniform)
  bool slab_ok = slab < nbr;

  RowCursor c0, c1;
  const long long row0 = slab * B + r;
  init_cursor(c0, rowptr, colind, slab_ok && row0 < nrows ? (int)row0 : nrows, nrows, nnz, derr);
  if (M::RPL == 2) {
    const long long row1 = slab * B + 32 + r;
    init_cursor(c1, rowptr, colind, slab_ok && row1 < nrows ? (int)row1 : nrows, nrows, nnz, derr);
  }
  if (wl.units) {
    const long long entries = slab_ok ? slab_entries<B>(rowptr, slab, nrows) : 0;
    int longest = c0.end - c0.pos;
    if (M::RPL == 2) longest = max(longest, c1.end - c1.pos);
    longest = -seg_min(-longest, M::W);
    const long long words = (((long long)ncols + B - 1) / B + 31) / 32;  // of the bitmap
    const long long stragglers = min(kStragglers, (long long)nbr / kAboveMean);
    bool w;
    if (BUILD) {
      const int tiles = slab_ok ? bsr_rowptr[slab + 1] - bsr_rowptr[slab] : 0;
      const long long steps = max(tiles, longest);
      w = slab_ok && (tiles > merge_tiles<B>() || longest > kMergeRow) &&
          (steps * fill_words<B>() >= words || steps * stragglers >= bsr_rowptr[nbr] || steps * kFewSlabs >= words * nbr);
    } else {
      const bool straggler = entries * stragglers >= nnz || entries * kFewSlabs >= words * nbr;
      w = slab_ok && entries > kMergeEntries && (entries * count_words<B>() >= words || straggler);
      if (__any_sync(0xffffffffu, w)) {
        int first = c0.head, last = c0.pos < c0.end ? colind[c0.end - 1] : -1;
        const int before = __shfl_up_sync(0xffffffffu, last / B, 1, M::W);
        const unsigned moves = __ballot_sync(0xffffffffu, r > 0 && last >= 0 && last / B != before);
        const int moved = __popc((moves >> (g * M::W)) & (0xffffffffu >> (32 - M::W)));
        if (M::RPL == 2) {
          first = min(first, c1.head);
          last = max(last, c1.pos < c1.end ? colind[c1.end - 1] : -1);
        }
        first = seg_min(first, M::W);
        last = -seg_min(-last, M::W);
        w = w && (longest > kMergeRow || ((straggler || moved > M::W / 4) &&
                                          (long long)last / B - (long long)first / B >= merge_tiles<B>()));
      }
    }
    if (w) {
      if (r == 0) {
        if (!BUILD) counts[slab] = 0;
        list_units(wl, (int)slab, entries, nnz, derr);
      }
      slab_ok = false;
      c0.end = c0.pos;
      if (M::RPL == 2) c1.end = c1.pos;
    }
    if (!__any_sync(0xffffffffu, slab_ok)) return;
  }

  // a slab's tiles stay inside its block row's range of the output
  long long out = 0;
  int room = 0;
  if (BUILD && slab_ok) {
    out = bsr_rowptr[slab];
    room = (int)(bsr_rowptr[slab + 1] - out);
  }
  int ntile = 0;

  while (true) {
    int h = head_block<B>(c0);
    if (M::RPL == 2) h = min(h, head_block<B>(c1));
    const int m = seg_min(h, M::W);
    if (!__any_sync(0xffffffffu, m != kINF)) break;
    WT w0 = 0, w1 = 0;
    if (m != kINF) {
      consume<B, WT>(c0, colind, m, ncols, w0, derr, BUILD);
      if (M::RPL == 2) {
        consume<B, WT>(c1, colind, m, ncols, w1, derr, BUILD);
      }
    }
    if (BUILD) {
      const long long tile = out + ntile;
      const bool put = m != kINF && ntile < room;
      if (layout == GBO_LAYOUT_ROW) {
        if (put) {
          if (r == 0) bsr_colind[tile] = m;
          bsr_val[tile * B + r] = w0;
          if (M::RPL == 2) bsr_val[tile * B + 32 + r] = w1;
        }
      } else {
        // transpose the b x b bit tile with ballots: column word c has row r
        // at bit (b-1-r).
        if (M::RPL == 1) {
          WT mine = 0;
#pragma unroll 4
          for (int cc = 0; cc < B; ++cc) {
            unsigned bal = __ballot_sync(0xffffffffu, (w0 >> (B - 1 - cc)) & 1);
            unsigned seg = (bal >> (g * M::W)) & seg_mask<B>();
            unsigned colw = __brev(seg) >> (32 - (B < 32 ? B : 32));
            if (r == cc) mine = (WT)colw;
          }
          if (put) {
            if (r == 0) bsr_colind[tile] = m;
            bsr_val[tile * B + r] = mine;
          }
        } else {
          unsigned long long lo_w = 0, hi_w = 0;
#pragma unroll 4
          for (int cc = 0; cc < 64; ++cc) {
            unsigned lo = __ballot_sync(0xffffffffu, (unsigned)((w0 >> (63 - cc)) & 1ull));
            unsigned hi = __ballot_sync(0xffffffffu, (unsigned)((w1 >> (63 - cc)) & 1ull));
            unsigned long long colw = __brevll(((unsigned long long)hi << 32) | lo);
            if (cc == (int)r) lo_w = colw;
            if (cc == (int)r + 32) hi_w = colw;
          }
          if (put) {
            if (r == 0) bsr_colind[tile] = m;
            bsr_val[tile * B + r] = (WT)lo_w;
            bsr_val[tile * B + 32 + r] = (WT)hi_w;
          }
        }
      }
    }
    if (m != kINF) ++ntile;
  }
  if (!BUILD && slab_ok && r == 0) counts[slab] = ntile;
}

// Wide slabs.  A block takes a unit: a whole slab or, of a hub slab, the
// block columns between two quantiles of its longest row, about kUnitEntries
// entries.  A thread per row finds the row's entries in the unit (binary
// search); the block walks these with a thread per entry, four in flight,
// and marks their block columns in a shared-memory bitmap, whose set bits are
// the unit's tiles in order.  The count pass adds up the newly set bits.  The
// fill pass ranks the bitmap (per-warp prefix sums of the words' popcounts),
// writes bsrColInd, zeroes the unit's tiles and walks the entries again: in
// the ROW layout the first entry of a run (entries of one row in one block
// column are consecutive) gathers the run's bits and stores the whole row
// word, in the COL layout an entry ORs its bit into its column word.  Block
// columns past the bitmap's `win` are taken in further windows.
//
// What bounds it: the tile writes (a 32x32 tile is 128 bytes for one or two
// row words on power-law graphs); a unit's tiles are zeroed just before their
// words are stored so that both meet in L2.  R-MAT 19, b = 32 (1.4 GB of
// tiles): 357 us for the fill and 107 for the count.  One block of 1,024
// threads per hub slab instead of units: 666 (block row 0 is the tail);
// tiles built in shared memory by a lane per row: 2,000 (serial walks); all
// tiles zeroed by a kernel of their own first: 15 % more.
constexpr int kWideTPB = 128;
constexpr int kWideWarps = kWideTPB / 32;
constexpr int kWideInFlight = 4;
constexpr int kWideBlocksPerSM = 16;
constexpr size_t kWideShared = 224 * 1024;  // dynamic shared memory of a block, at most (227 KB less the static arrays)

// Inclusive sums of the values v[1..B] in place (v[0] = 0), by one warp.
template <int B>
__device__ __forceinline__ void warp_prefix_rows(int* v, unsigned lane) {
  int carry = 0;
#pragma unroll
  for (int h = 0; h < (B + 31) / 32; ++h) {
    const int i = (int)lane + 32 * h;
    int x = i < B ? v[i + 1] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)lane >= o) x += y;
    }
    x += carry;
    if (i < B) v[i + 1] = x;
    carry = __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) v[0] = 0;
}

// `split_only`: the units of hub slabs alone (their counts, ahead of the fill
// pass).  ucnt: tiles of every unit -- written by the count form, summed by
// the fill form into its first tile.
template <int B, bool BUILD>
__global__ void __launch_bounds__(kWideTPB) k_pack_wide(const int* __restrict__ rowptr,
                                                        const int* __restrict__ colind, int nrows, int ncols,
                                                        long long nnz, int nbc, int win,
                                                        WideList wl, bool split_only, int* ucnt, int* __restrict__ counts,
                                                        const int* __restrict__ bsr_rowptr,
                                                        int* __restrict__ bsr_colind,
                                                        typename Word<B>::T* bsr_val, int layout,
                                                        unsigned* derr) {
  using WT = typename Word<B>::T;
  constexpr int F = kWideInFlight;
  extern __shared__ unsigned wide_sh[];
  __shared__ int rp[B + 1], seg_beg[B], seg_pre[B + 1];  // rows' entries: all, the window's first, the window's count before
  __shared__ int longest_sh;
  __shared__ unsigned long long unit_sh;
  __shared__ int wsum[kWideWarps + 1];
  const int nwords = win / 32;
  unsigned* bm = wide_sh;                               // block column w0 + 32 i + k: bit k of word i
  int* pre = reinterpret_cast<int*>(wide_sh + nwords);  // BUILD: tiles before word i within its warp's range
  const int tid = (int)threadIdx.x;
  const unsigned lane = threadIdx.x & 31;
  const int wib = tid >> 5;
  const int shift = nwords <= kWideWarps ? 0 : 32 - __clz((nwords - 1) / kWideWarps);
  const int per_warp = 1 << shift;  // words ranked by one warp
  const unsigned long long nunits = min(wl.ctr[0], (unsigned long long)wl.cap);
  for (;;) {
    __syncthreads();  // the previous unit's readers of the shared arrays
    if (tid == 0) unit_sh = atomicAdd(wl.ctr + (split_only ? 2 : 1), 1ull);
    __syncthreads();
    if (unit_sh >= nunits) return;
    const int ui = (int)unit_sh;
    const WideUnit un = wl.units[ui];
    if (un.slab < 0 || (split_only && un.count == 1)) continue;
    const long long row0 = (long long)un.slab * B;
    const int rows = (int)(row0 + B < nrows ? B : nrows - row0);
    if (tid <= rows) rp[tid] = rowptr[row0 + tid];
    __syncthreads();
    const bool bad = tid < rows && (rp[tid] < 0 || rp[tid + 1] < rp[tid] || rp[tid + 1] > nnz);
    if (__syncthreads_or(bad)) {
      if (tid == 0) {
        atomicOr(derr, DERR_ROWPTR);
        if (!BUILD && ucnt) ucnt[ui] = 0;
      }
      continue;
    }
    long long wa = 0, wz = nbc;  // the unit's block columns
    if (un.count > 1) {
      if (wib == 0) {  // the longest row
        int len = -1, at = 0;
        for (int r = (int)lane; r < rows; r += 32)
          if (rp[r + 1] - rp[r] > len) {
            len = rp[r + 1] - rp[r];
            at = r;
          }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const int l2 = __shfl_xor_sync(0xffffffffu, len, o), a2 = __shfl_xor_sync(0xffffffffu, at, o);
          if (l2 > len || (l2 == len && a2 < at)) {
            len = l2;
            at = a2;
          }
        }
        if (lane == 0) longest_sh = at;
      }
      __syncthreads();
      const int b0 = rp[longest_sh];
      const long long len = rp[longest_sh + 1] - b0;
      if (un.index > 0) wa = min((long long)max(colind[b0 + len * un.index / un.count], 0) / B, (long long)nbc);
      if (un.index + 1 < un.count)
        wz = min((long long)max(colind[b0 + len * (un.index + 1) / un.count], 0) / B, (long long)nbc);
    }
    // The rows' searches below suppose sorted rows and leave out what lies past
    // the last block column: where they are made, this unit's share of the
    // slab's entries is checked one by one (a hub's units before the fill
    // pass, by the count form).
    if (un.count > 1 ? !BUILD : win < nbc) {
      const int e0 = rp[0];
      const long long ne = rp[rows] - e0;
      const long long ez = e0 + ne * (un.index + 1) / un.count;
      for (long long e = e0 + ne * un.index / un.count + tid; e < ez; e += kWideTPB) {
        const int c = colind[e];
        if (c < 0 || c >= ncols) atomicOr(derr, DERR_COL_BOUNDS);
        if (e > e0 && c < colind[e - 1]) {
          bool starts = false;
          for (int r = 0; r < rows; ++r) starts = starts || rp[r] == (int)e;
          if (!starts) atomicOr(derr, DERR_UNSORTED);
        }
      }
    }
    long long t0 = 0, t1 = 0;
    if (BUILD) {
      t0 = bsr_rowptr[un.slab];
      t1 = bsr_rowptr[un.slab + 1];
      if (un.index > 0) {  // behind the tiles of the slab's earlier units
        int v = 0;
        for (int i = tid; i < un.index; i += kWideTPB) v += ucnt[un.first + i];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) wsum[wib] = v;
        __syncthreads();
        for (int q = 0; q < kWideWarps; ++q) t0 += wsum[q];
        __syncthreads();
      }
    }
    int cnt = 0;
    for (long long w0 = wa; w0 < wz; w0 += win) {
      const long long w1 = min(w0 + win, wz);
      const int nw = (int)((w1 - w0 + 31) / 32);  // bitmap words in use
      __syncthreads();
      for (int i = tid; i < nw; i += kWideTPB) bm[i] = 0u;
      if (tid < B) {
        int lo = 0, hi = 0;
        if (tid < rows) {
          lo = rp[tid];
          hi = rp[tid + 1];
          if (w0 > 0 || w1 < nbc) {
            int top = hi;
            while (lo < hi) {  // first entry at or past block column w0
              const int mid = (lo + hi) >> 1;
              if (colind[mid] < w0 * B) lo = mid + 1;
              else hi = mid;
            }
            while (hi < top) {  // first entry at or past block column w1
              const int mid = (hi + top) >> 1;
              if (colind[mid] < w1 * B) hi = mid + 1;
              else top = mid;
            }
          }
        }
        seg_beg[tid] = lo;
        seg_pre[tid + 1] = hi - lo;
      }
      __syncthreads();
      if (wib == 0) warp_prefix_rows<B>(seg_pre, lane);
      __syncthreads();
      const int ne = seg_pre[B];
      // entry q of the window: its row, place, column and the column before it in its row (-1: none)
      auto entry = [&](int q, int& r, int& e, int& c, int& cp) {
        c = cp = -1;
        if (q >= ne) return;
        r = 0;
#pragma unroll
        for (int st = B / 2; st > 0; st >>= 1)
          if (seg_pre[r + st] <= q) r += st;
        e = seg_beg[r] + (q - seg_pre[r]);
        c = colind[e];
        if (e > rp[r]) cp = colind[e - 1];
      };
      for (int qb = tid; qb < ne; qb += kWideTPB * F) {
        int r[F], e[F], c[F], cp[F];
#pragma unroll
        for (int u = 0; u < F; ++u) entry(qb + u * kWideTPB, r[u], e[u], c[u], cp[u]);
#pragma unroll
        for (int u = 0; u < F; ++u) {
          if (qb + u * kWideTPB >= ne) break;
          if (c[u] < 0 || c[u] >= ncols) {
            atomicOr(derr, DERR_COL_BOUNDS);
            continue;
          }
          if (c[u] < cp[u]) atomicOr(derr, DERR_UNSORTED);
          const int C = c[u] / B;
          if (cp[u] >= 0 && cp[u] / B == C) continue;  // marked by the entry before
          const long long k = C - w0;
          if (k < 0 || C >= w1) continue;  // an unsorted row's
          const unsigned bit = 1u << (k & 31);
          if (!(*(volatile unsigned*)(bm + (k >> 5)) & bit) && !(atomicOr(bm + (k >> 5), bit) & bit)) ++cnt;
        }
      }
      if (!BUILD) continue;
      __syncthreads();
      // rank: every warp over its own range of words, then the warps' totals
      const int i0 = wib << shift, i1 = min(i0 + per_warp, nw);
      int run = 0;
      for (int i = i0; i < i1; i += 32) {
        const int p = i + (int)lane < i1 ? __popc(bm[i + lane]) : 0;
        int incl = p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if ((int)lane >= o) incl += y;
        }
        if (i + (int)lane < i1) pre[i + lane] = run + incl - p;
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) wsum[wib + 1] = run;
      __syncthreads();
      if (wib == 0) {
        int v = lane < kWideWarps ? wsum[lane + 1] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, v, o);
          if ((int)lane >= o) v += y;
        }
        if (lane < kWideWarps) wsum[lane + 1] = v;
        if (lane == 0) wsum[0] = 0;
      }
      __syncthreads();
      const long long tz = min(t1, t0 + wsum[kWideWarps]);  // a slab's tiles stay inside its range of the output
      for (int i = i0 + (int)lane; i < i1; i += 32) {
        long long t = t0 + wsum[wib] + pre[i];
        for (unsigned m = bm[i]; m; m &= m - 1, ++t)
          if (t < tz) bsr_colind[t] = (int)(w0 + 32 * i + (__ffs(m) - 1));
      }
      {
        constexpr int kTileWords = B * (int)sizeof(WT) / 4;
        unsigned* z = reinterpret_cast<unsigned*>(bsr_val) + t0 * kTileWords;
        const long long nz = (tz - t0) * kTileWords;
        if (kTileWords % 4 == 0 && reinterpret_cast<uintptr_t>(bsr_val) % 16 == 0)
          for (long long i = tid; i < nz / 4; i += kWideTPB) reinterpret_cast<uint4*>(z)[i] = make_uint4(0u, 0u, 0u, 0u);
        else
          for (long long i = tid; i < nz; i += kWideTPB) z[i] = 0u;
      }
      __syncthreads();
      for (int qb = tid; qb < ne; qb += kWideTPB * F) {
        int r[F], e[F], c[F], cp[F];
#pragma unroll
        for (int u = 0; u < F; ++u) entry(qb + u * kWideTPB, r[u], e[u], c[u], cp[u]);
#pragma unroll
        for (int u = 0; u < F; ++u) {
          if (c[u] < 0 || c[u] >= ncols) continue;  // past the end, or reported above
          const int C = c[u] / B;
          if (C < w0 || C >= w1) continue;
          if (layout == GBO_LAYOUT_ROW && cp[u] >= 0 && cp[u] / B == C) continue;  // inside its run
          const int k = (int)(C - w0);
          const long long t = t0 + wsum[k >> (shift + 5)] + pre[k >> 5] + __popc(bm[k >> 5] & ((1u << (k & 31)) - 1u));
          if (t >= tz) continue;
          if (layout == GBO_LAYOUT_ROW) {
            WT word = (WT)((WT)1 << (B - 1 - c[u] % B));
            for (int f = e[u] + 1; f < rp[r[u] + 1]; ++f) {
              const int cf = colind[f];
              if (cf < 0 || cf / B != C) break;
              word = (WT)(word | ((WT)1 << (B - 1 - cf % B)));
            }
            bsr_val[t * B + r[u]] = word;
          } else {
            const long long wi = t * B + c[u] % B;
            if constexpr (B == 64) {
              atomicOr(reinterpret_cast<unsigned long long*>(bsr_val) + wi, 1ull << (B - 1 - r[u]));
            } else {
              constexpr int kPer = 4 / (int)sizeof(WT);  // words of a 32-bit atomic (little endian)
              atomicOr(reinterpret_cast<unsigned*>(bsr_val) + wi / kPer,
                       (1u << (B - 1 - r[u])) << ((wi % kPer) * 8 * (int)sizeof(WT)));
            }
          }
        }
      }
      t0 = tz;
      __syncthreads();  // wsum is rewritten
    }
    if (!BUILD) {
      for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
      if (lane == 0) wsum[wib] = cnt;
      __syncthreads();
      if (tid == 0) {
        int tot = 0;
        for (int q = 0; q < kWideWarps; ++q) tot += wsum[q];
        if (ucnt) ucnt[ui] = tot;
        if (counts && tot) atomicAdd(counts + un.slab, tot);
      }
    }
  }
}

// ---------------------------------------------------------------- scan
constexpr int kScanTPB = 1024;

__global__ void k_scan_block_sums(const int* __restrict__ in, long long n,
                                  long long* __restrict__ sums) {
  __shared__ long long sh[32];
  long long i = (long long)blockIdx.x * kScanTPB + threadIdx.x;
  long long v = i < n ? in[i] : 0;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    long long s = sh[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = s;
  }
}

// Exclusive scan of up to kScanTPB*kScanTPB block sums by one block (loop).
__global__ void k_scan_sums(long long* __restrict__ sums, long long nb, long long* total) {
  __shared__ long long sh[32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (long long base = 0; base < nb; base += kScanTPB) {
    long long i = base + threadIdx.x;
    long long v = i < nb ? sums[i] : 0;
    // inclusive warp scan
    long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, x, o);
      if ((threadIdx.x & 31) >= (unsigned)o) x += y;
    }
    if ((threadIdx.x & 31) == 31) sh[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
      long long s = sh[threadIdx.x];
      for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, s, o);
        if (threadIdx.x >= (unsigned)o) s += y;
      }
      sh[threadIdx.x] = s;
    }
    __syncthreads();
    long long warp_prefix = (threadIdx.x >> 5) ? sh[(threadIdx.x >> 5) - 1] : 0;
    long long incl = x + warp_prefix + carry;
    if (i < nb) sums[i] = incl - v;
    __syncthreads();
    if (threadIdx.x == kScanTPB - 1) carry = incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// Short inputs (kScanShort): one kernel, every block adding up the counts of
// the blocks before it itself -- at most 15 coalesced loads a thread, where
// the three kernels above cost three launches (16,384 counts: 7 us of kernels, 10 as three).
constexpr long long kScanShort = 16 * kScanTPB;

template <typename OutT>
__global__ void __launch_bounds__(kScanTPB) k_scan_short(const int* __restrict__ in, int n, OutT* __restrict__ out,
                                                         long long* __restrict__ total) {
  __shared__ long long sh[32], base_sh[32];
  const unsigned lane = threadIdx.x & 31;
  const int w = (int)(threadIdx.x >> 5);
  const int i = (int)blockIdx.x * kScanTPB + (int)threadIdx.x;
  long long before = 0;
#pragma unroll 8
  for (int k = (int)threadIdx.x; k < (int)blockIdx.x * kScanTPB; k += kScanTPB) before += in[k];
  const long long v = i < n ? in[i] : 0;
  long long x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, x, o);
    if ((int)lane >= o) x += y;
  }
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 31) sh[w] = x;
  if (lane == 0) base_sh[w] = before;
  __syncthreads();
  long long base = 0;
  for (int q = 0; q < kScanTPB / 32; ++q) base += base_sh[q] + (q < w ? sh[q] : 0);
  const long long excl = base + x - v, most = sizeof(OutT) == 8 ? excl : 2147483647LL;
  if (i < n) out[i] = (OutT)min(excl, most);
  if (i == n - 1) {
    out[n] = (OutT)min(excl + v, sizeof(OutT) == 8 ? excl + v : 2147483647LL);
    *total = excl + v;
  }
}

template <typename OutT>
__global__ void k_scan_apply(const int* __restrict__ in, long long n,
                             const long long* __restrict__ sums, OutT* __restrict__ out,
                             const long long* __restrict__ total) {
  __shared__ long long sh[32];
  long long i = (long long)blockIdx.x * kScanTPB + threadIdx.x;
  long long v = i < n ? in[i] : 0;
  long long x = v;
  for (int o = 1; o < 32; o <<= 1) {
    long long y = __shfl_up_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) >= (unsigned)o) x += y;
  }
  if ((threadIdx.x & 31) == 31) sh[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    long long s = sh[threadIdx.x];
    for (int o = 1; o < 32; o <<= 1) {
      long long y = __shfl_up_sync(0xffffffffu, s, o);
      if (threadIdx.x >= (unsigned)o) s += y;
    }
    sh[threadIdx.x] = s;
  }
  __syncthreads();
  long long warp_prefix = (threadIdx.x >> 5) ? sh[(threadIdx.x >> 5) - 1] : 0;
  long long excl = x - v + warp_prefix + sums[blockIdx.x];
  if (sizeof(OutT) == 8) {
    if (i < n) out[i] = (OutT)excl;
    if (i == 0) out[n] = (OutT)*total;
  } else {
    if (i < n) out[i] = (OutT)(excl > 2147483647LL ? 2147483647LL : excl);
    if (i == 0) out[n] = (OutT)(*total > 2147483647LL ? 2147483647LL : *total);
  }
}

// ------------------------------------------------------- vector packing
template <int B>
__global__ void k_pack_vec(const float* __restrict__ xf, const int32_t* __restrict__ xi, int n,
                           typename Word<B>::T* __restrict__ bits, long long nwords) {
  using WT = typename Word<B>::T;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned lane = threadIdx.x & 31;
  bool v = false;
  if (i < n) v = xf ? (xf[i] > 0.f) : (xi[i] > 0);
  unsigned bal = __brev(__ballot_sync(0xffffffffu, v));  // element (base+k) at bit 31-k
  const long long base = i - lane;                        // first element of this warp
  if (B == 64) {
    // two warps make one 64-bit word: even warp -> high half, odd warp -> low half
    const long long word = base / 64;
    if (lane == 0 && word < nwords) {
      unsigned long long* wp = reinterpret_cast<unsigned long long*>(bits) + word;
      unsigned long long part = ((base / 32) & 1) ? (unsigned long long)bal
                                                  : ((unsigned long long)bal << 32);
      atomicOr(wp, part);
    }
  } else {
    constexpr int S = 32 / B;  // segments per warp chunk
    if ((int)lane < S) {
      const long long word = base / B + lane;
      if (word < nwords) {
        unsigned seg = (bal >> (32 - B * (lane + 1))) & seg_mask<B>();
        bits[word] = (WT)seg;
      }
    }
  }
}

template <int B>
__global__ void k_unpack_vec(const typename Word<B>::T* __restrict__ bits, int n,
                             int32_t* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long w = (unsigned long long)bits[i / B];
  out[i] = (int32_t)((w >> (B - 1 - (i % B))) & 1ull);
}

// ------------------------------------------------------------ out-degree
__global__ void k_col_hist(const int* __restrict__ colind, long long nnz, int ncols,
                           int* __restrict__ deg) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nnz;
       i += (long long)gridDim.x * blockDim.x) {
    int c = colind[i];
    if (c >= 0 && c < ncols) atomicAdd(deg + c, 1);
  }
}
__global__ void k_row_len(const int* __restrict__ rowptr, int nrows, int* __restrict__ deg) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nrows) deg[i] = rowptr[i + 1] - rowptr[i];
}
__global__ void k_inv(const int* __restrict__ deg, int n, float* __restrict__ inv) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) inv[i] = deg[i] > 0 ? 1.0f / (float)deg[i] : 0.0f;
}

// ------------------------------------------------------------- schedule
// Tiles of the longest block row (*longest starts at 0).
__global__ void k_sched_longest(const int* __restrict__ rowptr, int nbr, int* __restrict__ longest) {
  int most = 0;
  for (long long R = (long long)blockIdx.x * blockDim.x + threadIdx.x; R < nbr; R += (long long)gridDim.x * blockDim.x)
    most = max(most, rowptr[R + 1] - rowptr[R]);
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(longest, most);
}

// Tiles per work item.  A graph of many tiles takes `most` (chunk_for).  One
// whose tiles do not give every SM 32 warps of such items, and whose longest
// block row would run far past the others, is cut finer (`fine`): that row's
// item set the time of every product (R-MAT of 20,001 rows, us: fp32 b = 8
// 389 -> 34, b = 32 186 -> 54, Boolean b = 8 61 -> 12; counts at 25,001 rows,
// b = 64, 29 -> 12; min-select at 120,001 rows, b = 16, 287 -> 140).  Without
// such a row the split rows' second launch costs more than it gives (counts,
// uniform of 100,003 rows, b = 8: 6.2 -> 12.3).
struct Chunk {
  int fine, most;
  const int* longest;
  __device__ __forceinline__ int tiles() const { return *longest > 4 * fine ? fine : most; }
};

__global__ void k_sched_counts(const int* __restrict__ rowptr, int nbr, Chunk by,
                               int* __restrict__ nchunk, int* __restrict__ nslot,
                               int* __restrict__ issplit) {
  long long R = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (R >= nbr) return;
  const int chunk = by.tiles();
  int len = rowptr[R + 1] - rowptr[R];
  int k = len <= chunk ? 1 : (len + chunk - 1) / chunk;
  nchunk[R] = k;
  nslot[R] = k > 1 ? k : 0;
  issplit[R] = k > 1 ? 1 : 0;
}

__global__ void k_sched_fill(const int* __restrict__ rowptr, int nbr, Chunk by,
                             const int* __restrict__ item_off, const int* __restrict__ slot_off,
                             const int* __restrict__ split_off, gbo_item* __restrict__ items,
                             gbo_split* __restrict__ splits) {
  long long R = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (R >= nbr) return;
  const int chunk = by.tiles();
  int t0 = rowptr[R], t1 = rowptr[R + 1];
  int len = t1 - t0;
  int k = len <= chunk ? 1 : (len + chunk - 1) / chunk;
  int base = item_off[R];
  if (k == 1) {
    items[base] = gbo_item{(int)R, t0, t1, -1};
  } else {
    int s0 = slot_off[R];
    for (int q = 0; q < k; ++q) {
      int a = t0 + q * chunk;
      int e = min(t1, a + chunk);
      items[base + q] = gbo_item{(int)R, a, e, s0 + q};
    }
    splits[split_off[R]] = gbo_split{(int)R, s0, k, 0};
  }
}

// Block columns of k_pack_wide's bitmap: all of them, as far as their words
// and the words' ranks (8 bytes for 32 block columns) fit a block.
int wide_window(int nbc) {
  const long long all = ((long long)nbc + 1023) / 1024 * 1024;
  return (int)std::max(1024ll, std::min(all, (long long)(kWideShared / 8) / 32 * 1024));
}

template <int B, bool BUILD>
int launch_pack_pass(const int* rowptr, const int* colind, int nrows, int ncols, long long nnz, int nbr, int* counts,
                     const int* bsr_rowptr, int* bsr_colind, typename Word<B>::T* bsr_val, int layout,
                     unsigned* derr, unsigned long long* ctr, cudaStream_t s) {
  using M = SlabMap<B>;
  const long long warps = ((long long)nbr + M::G - 1) / M::G;
  const unsigned grid = blocks_for_warps(warps, kPackTPB / 32);
  // entries of a wide slab, at least (a tile or a row's entry each)
  constexpr int kLeast = merge_tiles<B>() < kMergeRow ? merge_tiles<B>() : kMergeRow;
  // the wide kernel stores the tile array in whole 32-bit words
  const bool wide = nnz > kLeast && (!BUILD || reinterpret_cast<uintptr_t>(bsr_val) % 4 == 0);
  WideList wl;
  int* ucnt = nullptr;
  char* tmp = nullptr;  // the units and (fill pass) their tile counts
  if (wide) {
    const long long slabs = std::min<long long>(nbr, nnz / (kLeast + 1));
    wl.cap = std::max(slabs + nnz / kUnitEntries, 1ll);
    wl.ctr = ctr;
    const size_t unit_bytes = sizeof(WideUnit) * (size_t)wl.cap;
    GBO_CUDA_TRY(pool_malloc_async(&tmp, unit_bytes + (BUILD ? sizeof(int) * (size_t)wl.cap : 0), s));
    wl.units = reinterpret_cast<WideUnit*>(tmp);
    if (BUILD) ucnt = reinterpret_cast<int*>(tmp + unit_bytes);
  }
  k_pack<B, BUILD><<<grid, kPackTPB, 0, s>>>(rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind,
                                             bsr_val, layout, wl, derr);
  int st = GBO_OK;
  if (wide) {
    const int nbc = (ncols + B - 1) / B;
    const int win = wide_window(nbc);
    const unsigned blocks = (unsigned)std::min<long long>(wl.cap, (long long)num_sms() * kWideBlocksPerSM);
    auto launch = [&](auto kern, size_t smem, bool split_only) -> int {
      if (smem > 40 * 1024)
        GBO_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideShared));
      kern<<<blocks, kWideTPB, smem, s>>>(rowptr, colind, nrows, ncols, nnz, nbc, win, wl, split_only, ucnt, counts,
                                          bsr_rowptr, bsr_colind, bsr_val, layout, derr);
      return GBO_OK;
    };
    const size_t bits = (size_t)win / 8;
    // fill: the hub units' tile counts first
    if (!BUILD || nnz > 2 * kUnitEntries) st = launch(k_pack_wide<B, false>, bits, BUILD);
    if (BUILD && st == GBO_OK) st = launch(k_pack_wide<B, true>, 2 * bits, false);
  }
  const cudaError_t e = cudaGetLastError();
  if (tmp) cudaFreeAsync(tmp, s);
  if (e != cudaSuccess) return fail_cuda(e, "pack kernels");
  return st;
}

template <int B>
int launch_pack(bool build, const int* rowptr, const int* colind, int nrows, int ncols,
                long long nnz, int nbr, int* counts, const int* bsr_rowptr, int* bsr_colind,
                void* bsr_val, int layout, unsigned* derr, unsigned long long* ctr, cudaStream_t s) {
  auto* val = reinterpret_cast<typename Word<B>::T*>(bsr_val);
  return build ? launch_pack_pass<B, true>(rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind, val,
                                           layout, derr, ctr, s)
               : launch_pack_pass<B, false>(rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind,
                                            val, layout, derr, ctr, s);
}

int dispatch_pack(int b, bool build, const int* rowptr, const int* colind, int nrows, int ncols,
                  long long nnz, int nbr, int* counts, const int* bsr_rowptr, int* bsr_colind,
                  void* bsr_val, int layout, unsigned* derr, unsigned long long* ctr, cudaStream_t s) {
  switch (b) {
    case 4: return launch_pack<4>(build, rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind, bsr_val, layout, derr, ctr, s);
    case 8: return launch_pack<8>(build, rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind, bsr_val, layout, derr, ctr, s);
    case 16: return launch_pack<16>(build, rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind, bsr_val, layout, derr, ctr, s);
    case 32: return launch_pack<32>(build, rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind, bsr_val, layout, derr, ctr, s);
    case 64: return launch_pack<64>(build, rowptr, colind, nrows, ncols, nnz, nbr, counts, bsr_rowptr, bsr_colind, bsr_val, layout, derr, ctr, s);
  }
  return fail(GBO_ERR_INVALID, "tile_bits must be 4, 8, 16, 32 or 64");
}

int derr_to_status(unsigned e) {
  if (e & DERR_ROWPTR) return fail(GBO_ERR_BOUNDS, "CSR row pointers are not monotone within [0, nnz]");
  if (e & DERR_COL_BOUNDS) return fail(GBO_ERR_BOUNDS, "CSR column index outside [0, ncols)");
  if (e & DERR_UNSORTED) return fail(GBO_ERR_UNSORTED, "CSR column indices are not ascending inside a row");
  return GBO_OK;
}

// A packing pass's device record, zeroed before it: the tile count, the
// counters of the wide units (WideList::ctr) and the error word.
struct PackRecord {
  long long total;
  unsigned long long units[3];
  unsigned derr;
};

}  // namespace

namespace {
template <typename OutT>
int exclusive_scan(const int* d_in, OutT* d_out, long long n, long long* d_total, cudaStream_t s) {
  long long nb = (n + kScanTPB - 1) / kScanTPB;
  if (nb < 1) nb = 1;
  if (n > 0 && n <= kScanShort) {
    k_scan_short<OutT><<<(unsigned)nb, kScanTPB, 0, s>>>(d_in, (int)n, d_out, d_total);
    GBO_CUDA_TRY(cudaGetLastError());
    return GBO_OK;
  }
  long long* sums = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&sums, sizeof(long long) * nb, s));
  k_scan_block_sums<<<(unsigned)nb, kScanTPB, 0, s>>>(d_in, n, sums);
  k_scan_sums<<<1, kScanTPB, 0, s>>>(sums, nb, d_total);
  k_scan_apply<OutT><<<(unsigned)nb, kScanTPB, 0, s>>>(d_in, n, sums, d_out, d_total);
  cudaError_t e = cudaGetLastError();
  cudaFreeAsync(sums, s);
  if (e != cudaSuccess) return fail_cuda(e, "scan kernels");
  return GBO_OK;
}
}  // namespace

int exclusive_scan_i32(const int* d_in, int* d_out, long long n, long long* d_total,
                       cudaStream_t s) {
  return exclusive_scan<int>(d_in, d_out, n, d_total, s);
}

int exclusive_scan_i32_to_i64(const int* d_in, long long* d_out, long long n, long long* d_total,
                              cudaStream_t s) {
  return exclusive_scan<long long>(d_in, d_out, n, d_total, s);
}

// nnzb per block row: counts -> bsr_rowptr (device) and total (host).
static int nnzb_impl(const int* rowptr, const int* colind, int nrows, int ncols, long long nnz,
                     int b, int* bsr_rowptr, long long* h_total, cudaStream_t s) {
  const int nbr = (nrows + b - 1) / b;
  int* counts = nullptr;
  PackRecord* rec = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&counts, sizeof(int) * (size_t)(nbr > 0 ? nbr : 1), s));
  GBO_CUDA_TRY(pool_malloc_async(&rec, sizeof(PackRecord), s));
  GBO_CUDA_TRY(cudaMemsetAsync(rec, 0, sizeof(PackRecord), s));
  int st = GBO_OK;
  if (nbr > 0) {
    st = dispatch_pack(b, false, rowptr, colind, nrows, ncols, nnz, nbr, counts, nullptr, nullptr,
                       nullptr, GBO_LAYOUT_ROW, &rec->derr, rec->units, s);
    if (st == GBO_OK) st = exclusive_scan_i32(counts, bsr_rowptr, nbr, &rec->total, s);
  } else {
    GBO_CUDA_TRY(cudaMemsetAsync(bsr_rowptr, 0, sizeof(int), s));
  }
  PackRecord h = {};
  if (st == GBO_OK) {
    const cudaError_t e = read_back(&h, rec, sizeof(h), s);
    if (e != cudaSuccess) st = fail_cuda(e, "nnzb readback");
  }
  const long long tot = h.total;
  cudaFreeAsync(counts, s);
  cudaFreeAsync(rec, s);
  if (st != GBO_OK) return st;
  GBO_TRY(derr_to_status(h.derr));
  if (tot > 2147483647LL) return fail(GBO_ERR_OVERFLOW, "more than 2^31-1 tiles; use a wider tile");
  *h_total = tot;
  return GBO_OK;
}

// Tile count of the B2SR packing of a device CSR at tile width b (the
// count pass of the packer alone; used by the tile-width tuner).
int count_tiles(const int* d_rowptr, const int* d_colind, int nrows, int ncols, long long nnz, int b,
                long long* nblk, cudaStream_t s) {
  const int nbr = (nrows + b - 1) / b;
  int* tmp = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&tmp, sizeof(int) * ((size_t)nbr + 1), s));
  const int st = nnzb_impl(d_rowptr, d_colind, nrows, ncols, nnz, b, tmp, nblk, s);
  cudaFreeAsync(tmp, s);
  return st;
}

static int fill_impl(const int* rowptr, const int* colind, int nrows, int ncols, long long nnz,
                     int b, int layout, const int* bsr_rowptr, int* bsr_colind, void* bsr_val,
                     cudaStream_t s, bool check) {
  const int nbr = (nrows + b - 1) / b;
  if (nbr == 0) return GBO_OK;
  PackRecord* rec = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&rec, sizeof(PackRecord), s));
  GBO_CUDA_TRY(cudaMemsetAsync(rec, 0, sizeof(PackRecord), s));
  int st = dispatch_pack(b, true, rowptr, colind, nrows, ncols, nnz, nbr, nullptr, bsr_rowptr,
                         bsr_colind, bsr_val, layout, &rec->derr, rec->units, s);
  unsigned herr = 0;
  if (st == GBO_OK && check) {
    const cudaError_t e = read_back(&herr, &rec->derr, sizeof(herr), s);
    if (e != cudaSuccess) st = fail_cuda(e, "pack");
  }
  cudaFreeAsync(rec, s);
  if (st != GBO_OK) return st;
  return derr_to_status(herr);
}

int pack_into(gbo_graph* g, const int* d_rowptr, const int* d_colind, int nrows, int ncols,
              long long nnz, int b, int layout, cudaStream_t s) {
  g->nrows = nrows;
  g->ncols = ncols;
  g->b = b;
  g->layout = layout;
  g->nbr = (nrows + b - 1) / b;
  g->nbc = (ncols + b - 1) / b;
  g->nnz = nnz;
  GBO_CUDA_TRY(cudaMalloc(&g->rowptr, sizeof(int) * (size_t)(g->nbr + 1)));
  long long nblk = 0;
  GBO_TRY(nnzb_impl(d_rowptr, d_colind, nrows, ncols, nnz, b, g->rowptr, &nblk, s));
  g->nblk = nblk;
  size_t vb = (size_t)nblk * (size_t)b * (size_t)word_bytes(b);
  GBO_CUDA_TRY(cudaMalloc(&g->colind, sizeof(int) * (size_t)(nblk > 0 ? nblk : 1)));
  // pad the tile array to 16 bytes so vector loads past the end stay inside
  GBO_CUDA_TRY(cudaMalloc(&g->val, vb + 16));
  g->device_bytes += sizeof(int) * (g->nbr + 1) + sizeof(int) * nblk + vb + 16;
  GBO_TRY(fill_impl(d_rowptr, d_colind, nrows, ncols, nnz, b, layout, g->rowptr, g->colind,
                    g->val, s, false));
  return GBO_OK;
}

int compute_outdeg_from_cols(gbo_graph* g, const int* d_colind, long long nnz, int ncols,
                             cudaStream_t s) {
  GBO_CUDA_TRY(cudaMalloc(&g->outdeg, sizeof(int) * (size_t)(ncols > 0 ? ncols : 1)));
  GBO_CUDA_TRY(cudaMalloc(&g->invdeg, sizeof(float) * (size_t)(ncols > 0 ? ncols : 1)));
  g->device_bytes += 8LL * ncols;
  GBO_CUDA_TRY(cudaMemsetAsync(g->outdeg, 0, sizeof(int) * (size_t)ncols, s));
  if (nnz > 0) {
    unsigned grid = (unsigned)std::min<long long>((nnz + 255) / 256, 148LL * 64);
    k_col_hist<<<grid, 256, 0, s>>>(d_colind, nnz, ncols, g->outdeg);
  }
  if (ncols > 0) k_inv<<<blocks_for(ncols, 256), 256, 0, s>>>(g->outdeg, ncols, g->invdeg);
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

int compute_outdeg_from_rowptr(gbo_graph* g, const int* d_rowptr, int nrows, cudaStream_t s) {
  GBO_CUDA_TRY(cudaMalloc(&g->outdeg, sizeof(int) * (size_t)(nrows > 0 ? nrows : 1)));
  GBO_CUDA_TRY(cudaMalloc(&g->invdeg, sizeof(float) * (size_t)(nrows > 0 ? nrows : 1)));
  g->device_bytes += 8LL * nrows;
  if (nrows > 0) {
    k_row_len<<<blocks_for(nrows, 256), 256, 0, s>>>(d_rowptr, nrows, g->outdeg);
    k_inv<<<blocks_for(nrows, 256), 256, 0, s>>>(g->outdeg, nrows, g->invdeg);
  }
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

void launch_invdeg(const int* d_deg, int n, float* d_inv, cudaStream_t s) {
  if (n > 0) k_inv<<<blocks_for(n, 256), 256, 0, s>>>(d_deg, n, d_inv);
}

int upload_outdeg(gbo_graph* g, const int* h_deg, int n, cudaStream_t s) {
  GBO_CUDA_TRY(cudaMalloc(&g->outdeg, sizeof(int) * (size_t)(n > 0 ? n : 1)));
  GBO_CUDA_TRY(cudaMalloc(&g->invdeg, sizeof(float) * (size_t)(n > 0 ? n : 1)));
  g->device_bytes += 8LL * n;
  if (n > 0) {
    GBO_CUDA_TRY(cudaMemcpyAsync(g->outdeg, h_deg, sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, s));
    launch_invdeg(g->outdeg, n, g->invdeg, s);
  }
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

int build_schedule(gbo_graph* g, cudaStream_t s) {
  const int nbr = g->nbr;
  if (nbr == 0) {
    g->nitems = 0;
    g->nsplit = 0;
    g->nslots = 0;
    return GBO_OK;
  }
  int *nchunk = nullptr, *nslot = nullptr, *issplit = nullptr;
  int *item_off = nullptr, *slot_off = nullptr, *split_off = nullptr;
  long long* tot = nullptr;
  size_t n1 = (size_t)nbr + 1;
  GBO_CUDA_TRY(pool_malloc_async(&nchunk, sizeof(int) * n1 * 6, s));
  nslot = nchunk + n1;
  issplit = nslot + n1;
  item_off = issplit + n1;
  slot_off = item_off + n1;
  split_off = slot_off + n1;
  GBO_CUDA_TRY(pool_malloc_async(&tot, sizeof(long long) * 4, s));
  int* longest = reinterpret_cast<int*>(tot + 3);
  GBO_CUDA_TRY(cudaMemsetAsync(longest, 0, sizeof(long long), s));
  const long long even = g->nblk / ((long long)num_sms() * 32 * groups_per_warp(g->b));
  const int most = chunk_for(g->b);
  const Chunk by{(int)std::min<long long>(most, even / 32 * 32 + 32), most, longest};
  k_sched_longest<<<std::min(blocks_for(nbr, 1024), (unsigned)num_sms()), 1024, 0, s>>>(g->rowptr, nbr, longest);
  k_sched_counts<<<blocks_for(nbr, 256), 256, 0, s>>>(g->rowptr, nbr, by, nchunk, nslot, issplit);
  GBO_TRY(exclusive_scan_i32(nchunk, item_off, nbr, tot + 0, s));
  GBO_TRY(exclusive_scan_i32(nslot, slot_off, nbr, tot + 1, s));
  GBO_TRY(exclusive_scan_i32(issplit, split_off, nbr, tot + 2, s));
  long long h[4];
  GBO_CUDA_TRY(read_back(h, tot, sizeof(h), s));
  g->longest = (int)h[3];
  g->nitems = (int)h[0];
  g->nslots = (int)h[1];
  g->nsplit = (int)h[2];
  GBO_CUDA_TRY(cudaMalloc(&g->items, sizeof(gbo_item) * (size_t)(g->nitems > 0 ? g->nitems : 1)));
  GBO_CUDA_TRY(cudaMalloc(&g->splits, sizeof(gbo_split) * (size_t)(g->nsplit > 0 ? g->nsplit : 1)));
  g->device_bytes += sizeof(gbo_item) * (long long)g->nitems + sizeof(gbo_split) * (long long)g->nsplit;
  k_sched_fill<<<blocks_for(nbr, 256), 256, 0, s>>>(g->rowptr, nbr, by, item_off, slot_off,
                                                    split_off, g->items, g->splits);
  GBO_CUDA_TRY(cudaGetLastError());
  cudaFreeAsync(nchunk, s);
  cudaFreeAsync(tot, s);
  return GBO_OK;
}

// One warp per tile: bit r of the tile's occupancy word is set iff row word
// r is non-zero.  A 32x32 tile spans four 32-byte sectors while R-MAT-like
// graphs hold one or two set bits per tile, so pull kernels that read this
// word first and load only the non-empty row words move about half the
// bytes of a full tile read.
__global__ void k_rowmask32(const unsigned* __restrict__ val, long long nblk,
                            unsigned* __restrict__ mask) {
  const unsigned lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nblk; t += nwarps) {
    const unsigned m = __ballot_sync(0xffffffffu, val[t * 32 + lane] != 0u);
    if (lane == 0) mask[t] = m;
  }
}

// Non-empty row words per work item (items cover the tiles in order).
__global__ void k_item_words(const gbo_item* __restrict__ items, int nitems,
                             const unsigned* __restrict__ mask, int* __restrict__ cnt) {
  const unsigned lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nitems; i += nwarps) {
    const gbo_item it = items[i];
    int c = 0;
    for (int t = it.t0 + (int)lane; t < it.t1; t += 32) c += __popc(mask[t]);
    c = (int)__reduce_add_sync(0xffffffffu, (unsigned)c);
    if (lane == 0) cnt[i] = c;
  }
}

// Copy the non-empty row words of every tile, in tile order and row order
// inside a tile, to `out`; item i's words start at wbase[i].
__global__ void k_pack_rowwords(const gbo_item* __restrict__ items, int nitems,
                                const unsigned* __restrict__ val, const unsigned* __restrict__ mask,
                                const long long* __restrict__ wbase, unsigned* __restrict__ out) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nitems; i += nwarps) {
    const gbo_item it = items[i];
    long long base = wbase[i];
    for (int b0 = it.t0; b0 < it.t1; b0 += 32) {
      const int t = b0 + (int)lane;
      const unsigned m = t < it.t1 ? mask[t] : 0u;
      const int c = __popc(m);
      int incl = c;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
      }
      const int excl = incl - c;
      const int ntile = min(32, it.t1 - b0);
      for (int k0 = 0; k0 < ntile; k0 += 8) {  // eight tiles' words in flight
        unsigned w[8], mk[8];
        int ok[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          mk[u] = __shfl_sync(0xffffffffu, m, (k0 + u) & 31);
          ok[u] = __shfl_sync(0xffffffffu, excl, (k0 + u) & 31);
          if (k0 + u >= ntile) mk[u] = 0u;
          w[u] = (mk[u] >> lane) & 1u ? val[(size_t)(b0 + k0 + u) * 32 + lane] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if ((mk[u] >> lane) & 1u) out[base + ok[u] + __popc(mk[u] & below)] = w[u];
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
}

int build_rowwords(gbo_graph* g, cudaStream_t s) {
  if (!g->rowmask || g->rowword || g->nitems <= 0) return GBO_OK;
  int* cnt = nullptr;
  long long* tot = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&cnt, sizeof(int) * (size_t)g->nitems, s));
  GBO_CUDA_TRY(pool_malloc_async(&tot, sizeof(long long), s));
  GBO_CUDA_TRY(cudaMalloc(&g->item_wbase, sizeof(long long) * ((size_t)g->nitems + 1)));
  g->device_bytes += 8LL * (g->nitems + 1);
  int nsm = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int grid = (int)std::min<long long>(((long long)g->nitems + 7) / 8, 8LL * nsm);
  k_item_words<<<grid, 256, 0, s>>>(g->items, g->nitems, g->rowmask, cnt);
  GBO_TRY(exclusive_scan<long long>(cnt, g->item_wbase, g->nitems, tot, s));
  long long nw = 0;
  GBO_CUDA_TRY(cudaMemcpyAsync(&nw, tot, sizeof(nw), cudaMemcpyDeviceToHost, s));
  GBO_CUDA_TRY(cudaStreamSynchronize(s));
  cudaFreeAsync(cnt, s);
  cudaFreeAsync(tot, s);
  GBO_CUDA_TRY(cudaMalloc(&g->rowword, sizeof(unsigned) * (size_t)(nw > 0 ? nw : 1)));
  g->nrowword = nw;
  g->device_bytes += 4LL * nw;
  k_pack_rowwords<<<grid, 256, 0, s>>>(g->items, g->nitems, static_cast<const unsigned*>(g->val),
                                       g->rowmask, g->item_wbase, g->rowword);
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

// Row-word slices, pass 1: warp per block row; per batch of 32 tiles (lane
// j: tile j's occupancy word) the number of tiles in which row r is
// non-empty is popc of the ballot of bit r, kept by lane r.  Writes the
// tail length max(count - kRwsHead, 0) of every padded row.
__global__ void k_rws_count(const int* __restrict__ rowptr, int nbr, const unsigned* __restrict__ mask,
                            int* __restrict__ tail_len) {
  const unsigned lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long R = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; R < nbr; R += nwarps) {
    const int rs = rowptr[R], re = rowptr[R + 1];
    int c = 0;
    for (int t0 = rs; t0 < re; t0 += 32) {
      const unsigned m = t0 + (int)lane < re ? mask[t0 + lane] : 0u;
#pragma unroll
      for (int r = 0; r < 32; ++r) {
        const unsigned b = __ballot_sync(0xffffffffu, (m >> r) & 1u);
        if ((int)lane == r) c += __popc(b);
      }
    }
    tail_len[R * 32 + lane] = c > kRwsHead ? c - kRwsHead : 0;
  }
}

// Row-word slices, pass 2: warp per block row, lane r walks row r's word of
// every tile in order (one coalesced 128-byte load per tile, four tiles in
// flight) and appends the non-empty ones with their block column: the first
// kRwsHead to the head (entry-major), the rest to the row's tail.  Unused
// head entries get kRwsNone.
__global__ void k_rws_fill(const int* __restrict__ rowptr, const int* __restrict__ colind, int nbr,
                           const unsigned* __restrict__ val, const long long* __restrict__ tail_ptr,
                           uint2* __restrict__ head, uint2* __restrict__ tail) {
  const unsigned lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long R = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; R < nbr; R += nwarps) {
    const int rs = rowptr[R], re = rowptr[R + 1];
    uint2* hp = head + (size_t)R * kRwsHead * 32 + lane;
    uint2* tp = tail + tail_ptr[R * 32 + lane];
    int k = 0;
    for (int t = rs; t < re; t += 4) {
      unsigned w[4];
      int c[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        w[u] = t + u < re ? val[(size_t)(t + u) * 32 + lane] : 0u;
        c[u] = t + u < re ? colind[t + u] : 0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (!w[u]) continue;
        const uint2 e = make_uint2((unsigned)c[u], w[u]);
        if (k < kRwsHead) hp[(size_t)k * 32] = e;
        else tp[k - kRwsHead] = e;
        ++k;
      }
    }
    for (; k < kRwsHead; ++k) hp[(size_t)k * 32] = make_uint2(kRwsNone, 0u);
  }
}

namespace {

// The slices while they are built: they become the graph's when complete.
struct Slices {
  uint2 *head = nullptr, *tail = nullptr;
  long long *tail_ptr = nullptr, *long_chunk0 = nullptr, *chunk_beg = nullptr, *chunk_end = nullptr;
  int *long_row = nullptr, *chunk_row = nullptr;
  unsigned* longbits = nullptr;
  long long ntail = 0, nchunk = 0, bytes = 0;
  int nlong = 0;

  template <typename T>
  int make(T** p, size_t count) {
    const size_t nb = sizeof(T) * (count > 0 ? count : 1);
    GBO_CUDA_TRY(cudaMalloc(p, nb));
    bytes += (long long)nb;
    return GBO_OK;
  }
  template <typename T>
  int upload(T** p, const std::vector<T>& src) {
    GBO_TRY(make(p, src.size()));
    if (!src.empty()) GBO_CUDA_TRY(cudaMemcpy(*p, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice));
    return GBO_OK;
  }
  void release() {
    void* all[] = {head, tail, tail_ptr, long_chunk0, chunk_beg, chunk_end, long_row, chunk_row, longbits};
    for (void* p : all) cudaFree(p);
  }
};

int fill_slices(const gbo_graph* g, Slices& sl, cudaStream_t s) {
  const long long rows = (long long)g->nbr * 32;
  GBO_TRY(sl.make(&sl.tail_ptr, (size_t)rows + 1));
  GBO_TRY(sl.make(&sl.head, (size_t)rows * kRwsHead));
  const int grid = (int)std::min<long long>(((long long)g->nbr + 7) / 8, 16LL * num_sms());
  int* len = nullptr;
  long long* tot = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&len, sizeof(int) * (size_t)rows, s));
  cudaError_t e = pool_malloc_async(&tot, sizeof(long long), s);
  int st = e == cudaSuccess ? GBO_OK : fail_cuda(e, "row-word slices");
  if (st == GBO_OK) {
    k_rws_count<<<grid, 256, 0, s>>>(g->rowptr, g->nbr, g->rowmask, len);
    st = exclusive_scan_i32_to_i64(len, sl.tail_ptr, rows, tot, s);
  }
  if (st == GBO_OK && (e = read_back(&sl.ntail, tot, sizeof(sl.ntail), s)) != cudaSuccess)
    st = fail_cuda(e, "row-word slice lengths");
  cudaFreeAsync(len, s);
  if (tot) cudaFreeAsync(tot, s);
  GBO_TRY(st);
  GBO_TRY(sl.make(&sl.tail, (size_t)sl.ntail));
  k_rws_fill<<<grid, 256, 0, s>>>(g->rowptr, g->colind, g->nbr, static_cast<const unsigned*>(g->val), sl.tail_ptr,
                                  sl.head, sl.tail);
  GBO_CUDA_TRY(cudaGetLastError());
  // long tails cut into chunks (a host pass over the tail offsets, once)
  std::vector<long long> tp((size_t)rows + 1);
  GBO_CUDA_TRY(cudaMemcpyAsync(tp.data(), sl.tail_ptr, sizeof(long long) * tp.size(), cudaMemcpyDeviceToHost, s));
  GBO_CUDA_TRY(cudaStreamSynchronize(s));
  std::vector<int> lrow, crow;
  std::vector<unsigned> lbits((size_t)g->nbr, 0u);
  std::vector<long long> lc0, cbeg, cend;
  for (long long i = 0; i < rows; ++i) {
    const long long n = tp[(size_t)i + 1] - tp[(size_t)i];
    if (n <= kRwsLongTail) continue;
    lrow.push_back((int)i);
    lbits[(size_t)(i / 32)] |= 1u << (31 - i % 32);
    lc0.push_back((long long)cbeg.size());
    for (long long b = tp[(size_t)i]; b < tp[(size_t)i + 1]; b += kRwsChunk) {
      crow.push_back((int)i);
      cbeg.push_back(b);
      cend.push_back(std::min(b + kRwsChunk, tp[(size_t)i + 1]));
    }
  }
  lc0.push_back((long long)cbeg.size());
  sl.nlong = (int)lrow.size();
  sl.nchunk = (long long)cbeg.size();
  GBO_TRY(sl.upload(&sl.long_row, lrow));
  GBO_TRY(sl.upload(&sl.long_chunk0, lc0));
  GBO_TRY(sl.upload(&sl.chunk_row, crow));
  GBO_TRY(sl.upload(&sl.chunk_beg, cbeg));
  GBO_TRY(sl.upload(&sl.chunk_end, cend));
  GBO_TRY(sl.upload(&sl.longbits, lbits));
  return GBO_OK;
}

}  // namespace

// Complete and unchanging once the graph has them: built under the graph's
// lock, all of them or (no memory) none.
int build_rws(gbo_graph* g, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g->build_mu);
  if (g->b != 32 || g->layout != GBO_LAYOUT_ROW || !g->rowmask || g->rws_head || g->nbr <= 0) return GBO_OK;
  Slices sl;
  const int st = fill_slices(g, sl, s);
  if (st != GBO_OK) {
    cudaStreamSynchronize(s);
    sl.release();
    return st;
  }
  g->rws_tail = sl.tail;
  g->rws_ntail = sl.ntail;
  g->rws_tail_ptr = sl.tail_ptr;
  g->rws_long_row = sl.long_row;
  g->rws_long_chunk0 = sl.long_chunk0;
  g->rws_nlong = sl.nlong;
  g->rws_chunk_row = sl.chunk_row;
  g->rws_chunk_beg = sl.chunk_beg;
  g->rws_chunk_end = sl.chunk_end;
  g->rws_nchunk = sl.nchunk;
  g->rws_longbits = sl.longbits;
  g->rws_head = sl.head;
  g->device_bytes += sl.bytes;
  return GBO_OK;
}

int build_rowmask(gbo_graph* g, cudaStream_t s) {
  if (g->b != 32 || g->layout != GBO_LAYOUT_ROW || g->rowmask) return GBO_OK;
  GBO_CUDA_TRY(cudaMalloc(&g->rowmask, sizeof(unsigned) * (size_t)(g->nblk > 0 ? g->nblk : 1)));
  g->device_bytes += 4LL * g->nblk;
  if (g->nblk > 0) {
    int nsm = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long want = (g->nblk + 7) / 8;  // 8 warps per block
    const int grid = (int)std::min<long long>(want, 8LL * nsm);
    k_rowmask32<<<grid, 256, 0, s>>>(static_cast<const unsigned*>(g->val), g->nblk, g->rowmask);
  }
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

int ensure_workspace(gbo_graph* g, size_t bytes, cudaStream_t s) {
  if (g->ws_bytes >= bytes) return GBO_OK;
  if (g->ws) {
    GBO_CUDA_TRY(cudaStreamSynchronize(s));
    GBO_CUDA_TRY(cudaFree(g->ws));
    g->device_bytes -= (long long)g->ws_bytes;
    g->ws = nullptr;
    g->ws_bytes = 0;
  }
  size_t want = bytes + (bytes >> 3) + 256;
  GBO_CUDA_TRY(cudaMalloc(&g->ws, want));
  g->ws_bytes = want;
  g->device_bytes += (long long)want;
  return GBO_OK;
}

}  // namespace gbo

// ------------------------------------------------------------------ C ABI
using namespace gbo;

extern "C" int gbo_b2sr_nnzb(const int* d_csrRowPtr, const int* d_csrColInd, int nrows,
                             int ncols, int nnz, int tile_bits, int* d_bsrRowPtr, int* h_nblocks,
                             gbo_stream_t stream) {
  clear_error();
  if (!valid_tile_bits(tile_bits)) return fail(GBO_ERR_INVALID, "tile_bits must be 4, 8, 16, 32 or 64");
  if (nrows < 0 || ncols < 0 || nnz < 0 || !d_csrRowPtr || !d_bsrRowPtr || !h_nblocks ||
      (nnz > 0 && !d_csrColInd))
    return fail(GBO_ERR_INVALID, "gbo_b2sr_nnzb: bad argument");
  long long tot = 0;
  GBO_TRY(nnzb_impl(d_csrRowPtr, d_csrColInd, nrows, ncols, nnz, tile_bits, d_bsrRowPtr, &tot,
                    as_stream(stream)));
  *h_nblocks = (int)tot;
  return GBO_OK;
}

extern "C" int gbo_b2sr_pack(const int* d_csrRowPtr, const int* d_csrColInd, int nrows,
                             int ncols, int nnz, int tile_bits, int layout,
                             const int* d_bsrRowPtr, int* d_bsrColInd, void* d_bsrVal,
                             gbo_stream_t stream) {
  clear_error();
  if (!valid_tile_bits(tile_bits)) return fail(GBO_ERR_INVALID, "tile_bits must be 4, 8, 16, 32 or 64");
  if (layout != GBO_LAYOUT_ROW && layout != GBO_LAYOUT_COL)
    return fail(GBO_ERR_INVALID, "layout must be GBO_LAYOUT_ROW or GBO_LAYOUT_COL");
  if (nrows < 0 || ncols < 0 || nnz < 0 || !d_csrRowPtr || !d_bsrRowPtr ||
      (nnz > 0 && (!d_csrColInd || !d_bsrColInd || !d_bsrVal)))
    return fail(GBO_ERR_INVALID, "gbo_b2sr_pack: bad argument");
  return fill_impl(d_csrRowPtr, d_csrColInd, nrows, ncols, nnz, tile_bits, layout, d_bsrRowPtr,
                   d_bsrColInd, d_bsrVal, as_stream(stream), true);
}

template <int B>
static int pack_vec_impl(const float* xf, const int32_t* xi, int n, void* bits, cudaStream_t s) {
  long long nw = ((long long)n + B - 1) / B;
  if (B == 64) GBO_CUDA_TRY(cudaMemsetAsync(bits, 0, sizeof(unsigned long long) * nw, s));
  long long threads = ((long long)n + 31) / 32 * 32;
  if (B == 64) threads = nw * 64;  // whole 64-element words
  if (threads == 0) return GBO_OK;
  k_pack_vec<B><<<blocks_for(threads, 256), 256, 0, s>>>(
      xf, xi, n, reinterpret_cast<typename Word<B>::T*>(bits), nw);
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

static int pack_vec_dispatch(const float* xf, const int32_t* xi, int n, int b, void* bits,
                             gbo_stream_t stream) {
  clear_error();
  if (!valid_tile_bits(b)) return fail(GBO_ERR_INVALID, "tile_bits must be 4, 8, 16, 32 or 64");
  if (n < 0 || (n > 0 && (!bits || (!xf && !xi)))) return fail(GBO_ERR_INVALID, "pack_vector: bad argument");
  cudaStream_t s = as_stream(stream);
  switch (b) {
    case 4: return pack_vec_impl<4>(xf, xi, n, bits, s);
    case 8: return pack_vec_impl<8>(xf, xi, n, bits, s);
    case 16: return pack_vec_impl<16>(xf, xi, n, bits, s);
    case 32: return pack_vec_impl<32>(xf, xi, n, bits, s);
    default: return pack_vec_impl<64>(xf, xi, n, bits, s);
  }
}

extern "C" int gbo_pack_vector_f32(const float* d_x, int n, int tile_bits, void* d_bits,
                                   gbo_stream_t stream) {
  return pack_vec_dispatch(d_x, nullptr, n, tile_bits, d_bits, stream);
}
extern "C" int gbo_pack_vector_i32(const int32_t* d_x, int n, int tile_bits, void* d_bits,
                                   gbo_stream_t stream) {
  return pack_vec_dispatch(nullptr, d_x, n, tile_bits, d_bits, stream);
}

extern "C" int gbo_unpack_vector(const void* d_bits, int n, int tile_bits, int32_t* d_out,
                                 gbo_stream_t stream) {
  clear_error();
  if (!valid_tile_bits(tile_bits)) return fail(GBO_ERR_INVALID, "tile_bits must be 4, 8, 16, 32 or 64");
  if (n < 0 || (n > 0 && (!d_bits || !d_out))) return fail(GBO_ERR_INVALID, "unpack_vector: bad argument");
  if (n == 0) return GBO_OK;
  cudaStream_t s = as_stream(stream);
  unsigned grid = blocks_for(n, 256);
  switch (tile_bits) {
    case 4: k_unpack_vec<4><<<grid, 256, 0, s>>>((const uint8_t*)d_bits, n, d_out); break;
    case 8: k_unpack_vec<8><<<grid, 256, 0, s>>>((const uint8_t*)d_bits, n, d_out); break;
    case 16: k_unpack_vec<16><<<grid, 256, 0, s>>>((const uint16_t*)d_bits, n, d_out); break;
    case 32: k_unpack_vec<32><<<grid, 256, 0, s>>>((const uint32_t*)d_bits, n, d_out); break;
    default: k_unpack_vec<64><<<grid, 256, 0, s>>>((const unsigned long long*)d_bits, n, d_out); break;
  }
  GBO_CUDA_TRY(cudaGetLastError());
  return GBO_OK;
}

extern "C" int gbo_invdeg_from_rowptr(const int* d_rowptr, int n, float* d_inv, gbo_stream_t stream) {
  clear_error();
  if (n < 0 || (n > 0 && (!d_rowptr || !d_inv))) return fail(GBO_ERR_INVALID, "invdeg: bad argument");
  if (n == 0) return GBO_OK;
  cudaStream_t s = as_stream(stream);
  int* deg = nullptr;
  GBO_CUDA_TRY(pool_malloc_async(&deg, sizeof(int) * (size_t)n, s));
  k_row_len<<<blocks_for(n, 256), 256, 0, s>>>(d_rowptr, n, deg);
  k_inv<<<blocks_for(n, 256), 256, 0, s>>>(deg, n, d_inv);
  cudaError_t e = cudaGetLastError();
  cudaFreeAsync(deg, s);
  if (e != cudaSuccess) return fail_cuda(e, "invdeg kernels");
  return GBO_OK;
}
