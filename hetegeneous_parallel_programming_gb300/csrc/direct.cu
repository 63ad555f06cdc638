// Direct counting of small graphs and of batches of small graphs.
//
// The general path relabels the graph by degree rank, sorts every row and
// groups edges by target before it counts: 45 to 70 launches and a host read
// in the middle, which is all that a small graph's time consists of.  None of
// it changes a count.  Here the oriented graph keeps the input's ids: whether
// u->v stays is a comparison of (degree, id) pairs, input rows are sorted, so
// the kept entries of a row already are, and kept entries compacted in input
// order are the reference's own edge order (graph.cc:279-290).  Three
// launches and one host read at the end (from 2^20 entries on, and for a batch,
// one more host read before them):
//   direct_rows   row, validity and direction of every entry; each block
//                 compacts its kept entries into its own slice
//   direct_place  slices to their final place, DAG row pointers
//   direct_count  |N+(u) n N+(v)| of every kept edge
// Nothing needs the number of edges on the host: the grid is sized for half
// of the entries (what a symmetric graph keeps) and reads the true number
// from the device.
//
// It needs validated input (sorted, duplicate-free rows).
#include <algorithm>
#include <chrono>

#include "engine.cuh"

namespace tc {

constexpr int DR_THREADS = 256;
constexpr int DR_PER = 4;                             // 32-entry groups per warp
constexpr int DR_TILE = DR_THREADS * DR_PER;          // entries per block
constexpr int DR_GROUPS = DR_TILE / 32;
// Groups per warp in a large batch, whose rows pass is bound by instruction
// issue (73 % of cycles): half as many row searches and fixed costs per entry.  Batches of 1.4 M
// entries 55 -> 57 us up to the counting, 2.5 M 71 -> 69, 8 M 135 -> 121, 98 M
// 1085 -> 885; a small graph wants more warps (ER n = 16384: 2 us a call lost).
constexpr int DR_WIDE_PER = 8;
constexpr int64_t DR_WIDE_MIN_NNZ = int64_t(1) << 21;
constexpr int DR_SMEM_BLOCKS = 4096;                  // block sums every placing block scans for itself
static_assert(DR_GROUPS == 32, "one warp scans a block's group counts");

// Row pointers are int64 below 2^32 in valid input (the validation looks at all
// of their bits); the passes read the low words.
__device__ __forceinline__ uint32_t low_word(const int64_t *__restrict__ rowptr, uint32_t i) {
  return __ldg(reinterpret_cast<const uint32_t *>(rowptr) + 2 * (size_t)i);
}

// Largest r in [0, n) with rowptr[r] <= e, for e of the lane's half warp: 16
// lanes probe 16 pivots at a time, so n = 2^22 takes 6 dependent loads
// instead of 22.  Both halves search at once; all lanes must call it.  Ends
// for any rowptr contents, inside [0, n).
__device__ __forceinline__ uint32_t half_warp_row(const int64_t *__restrict__ rowptr, uint32_t n, uint32_t e,
                                                  int lane) {
  const uint32_t hl = lane & 15, sh = lane & 16;
  uint32_t lo = 0, hi = n;
  while (__any_sync(TC_FULL_MASK, hi - lo > 1)) {
    const uint32_t len = hi - lo, p = lo + (uint32_t)(((unsigned long long)(hl + 1) * len) >> 4) - (hl == 15 ? 1 : 0);
    const bool le = len > 1 && low_word(rowptr, p) <= e;
    const int c = __popc((__ballot_sync(TC_FULL_MASK, le) >> sh) & 0xffffu);
    const uint32_t nlo = __shfl_sync(TC_FULL_MASK, p, sh + max(c - 1, 0));
    const uint32_t nhi = __shfl_sync(TC_FULL_MASK, p, sh + min(c, 15));
    if (len > 1) {
      if (c > 0) lo = nlo;
      if (c < 16) hi = nhi;
    }
  }
  return lo;
}

// Row, row start and row end of a warp's entries [w0, w1), entry w0 + 32 k +
// lane in slot k.  The rows of the first and last entry are searched
// (half_warp_row); where they are at most 32 apart, each lane holds one row's
// end and the entries find theirs by shuffles, else by searches between them.
template <int PER>
__device__ __forceinline__ void entry_rows(const int64_t *__restrict__ rowptr, uint32_t n, uint32_t w0, uint32_t w1,
                                           int lane, uint32_t (&row)[PER], uint32_t (&rb)[PER],
                                           uint32_t (&re)[PER]) {
  const uint32_t r = half_warp_row(rowptr, n, lane < 16 ? w0 : w1 - 1, lane);
  const uint32_t r_lo = __shfl_sync(TC_FULL_MASK, r, 0), r_hi = max(r_lo, __shfl_sync(TC_FULL_MASK, r, 16));
  if (r_hi - r_lo < 32) {
    const uint32_t first = low_word(rowptr, r_lo);
    const uint32_t end = low_word(rowptr, min(r_lo + 1 + lane, n));
    uint32_t i[PER];  // rows from r_lo on that end at or before the entry
#pragma unroll
    for (int k = 0; k < PER; ++k) i[k] = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
      if (PER > DR_PER && step > r_hi - r_lo) continue;  // (a branch costs the few warps of a small graph more)
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const uint32_t x = __shfl_sync(TC_FULL_MASK, end, i[k] + step - 1);
        if (x <= w0 + 32 * k + lane && r_lo + i[k] + step <= r_hi) i[k] += step;
      }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      row[k] = r_lo + i[k];
      re[k] = __shfl_sync(TC_FULL_MASK, end, i[k]);
      const uint32_t before = __shfl_sync(TC_FULL_MASK, end, i[k] > 0 ? i[k] - 1 : 0);
      rb[k] = i[k] > 0 ? before : first;
    }
    return;
  }
  uint32_t hi[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    row[k] = w0 + 32 * k + lane < w1 ? r_lo : r_hi;
    hi[k] = r_hi + 1;
  }
  for (bool more = true; more;) {
    more = false;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      if (hi[k] - row[k] > 1) {
        const uint32_t mid = (row[k] + hi[k]) >> 1;
        if (low_word(rowptr, mid) <= w0 + 32 * k + lane) row[k] = mid;
        else hi[k] = mid;
        more |= hi[k] - row[k] > 1;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    rb[k] = low_word(rowptr, row[k]);
    re[k] = low_word(rowptr, row[k] + 1);
  }
}

// Results of a direct call, all zero at its start.  DX_DONE counts the counting
// kernel's blocks, and the last one hands the words to the host; DX_START,
// DX_COUNT and DX_END are the device's clock (ns) when the passes and the
// counting start and when they end.
enum { DX_TOTAL, DX_M, DX_FLAGS, DX_WORK, DX_ALG, DX_GUESS, DX_MAXN, DX_DONE, DX_START, DX_COUNT, DX_END, DX_WORDS };

__device__ __forceinline__ unsigned long long clock_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Whether the later kernels have nothing to do: invalid input, or lists too
// long.  It is the first thing they read of what the passes before them wrote, by
// an instruction that stays behind begin_pass's wait (a stale "no" would have row
// pointers used that the rows pass has refused), through L1: past it, every warp
// of the grid asked the same line of L2 (ER n = 111 592, 2.2 M entries: 158 -> 166
// us a call).
static_assert(DX_FLAGS % 2 == 0 && DX_WORK == DX_FLAGS + 1, "one 16-byte load");
__device__ __forceinline__ bool direct_off(const unsigned long long *res, unsigned long long max_work) {
  unsigned long long flags, work;
  asm volatile("ld.global.v2.u64 {%0, %1}, [%2];"
               : "=l"(flags), "=l"(work)
               : "l"(__cvta_generic_to_global(res + DX_FLAGS))
               : "memory");
  return (unsigned)flags || work > max_work;
}

// A guess of DX_WORK (see direct_rows_kernel) from DS_WARPS runs of 128 entries
// spread evenly over a large graph.  The host reads it before the passes over
// all entries start (12 us), which costs a graph whose lists are too long 43
// us instead of 170 (R-MAT scale 18).
constexpr int DS_WARPS = 512;
constexpr int64_t DS_MIN_NNZ = int64_t(1) << 20;  // below, the pass itself is as quick

template <bool ORIENT>
__global__ void __launch_bounds__(DR_THREADS) direct_sample_kernel(const int64_t *__restrict__ rowptr,
                                                                  const int32_t *__restrict__ col, int64_t n,
                                                                  int64_t nnz, const int32_t *__restrict__ vgroup,
                                                                  const int64_t *__restrict__ vtx_off,
                                                                  uint32_t row_begin, uint32_t row_end,
                                                                  unsigned long long *__restrict__ res) {
  if ((unsigned)res[DX_FLAGS]) return;
  const int lane = threadIdx.x & 31;
  const uint32_t i = blockIdx.x * (DR_THREADS / 32) + (threadIdx.x >> 5);
  const uint32_t w0 = i * (uint32_t)(nnz / DS_WARPS), w1 = (uint32_t)min(nnz, (int64_t)w0 + 32 * DR_PER);
  uint32_t row[DR_PER], rb[DR_PER], re[DR_PER];
  entry_rows(rowptr, (uint32_t)n, w0, w1, lane, row, rb, re);
  unsigned long long len = 0;
#pragma unroll
  for (int k = 0; k < DR_PER; ++k) {
    const uint32_t e = w0 + 32 * k + lane;
    int64_t v = e < w1 ? col[e] : -1;
    if (vtx_off && v >= 0) v += vtx_off[vgroup[row[k]]];
    if (v < 0 || v >= n || row[k] < row_begin || row[k] >= row_end) continue;
    const uint32_t a = re[k] - rb[k], b = low_word(rowptr, (uint32_t)v + 1) - low_word(rowptr, (uint32_t)v);
    len += ORIENT ? min(a, b) : a + b;  // an undirected edge has two entries
  }
  len = warp_sum(len);
  if (lane == 0) atomicAdd(res + DX_GUESS, len * (unsigned long long)(nnz / (DS_WARPS * 32 * DR_PER)) / (ORIENT ? 2 : 1));
}

// Row, validity and direction of every entry.  A warp finds the rows of its
// first and last entry together (half_warp_row), every lane the rows of its
// own entries between them.  ORIENT: the kept entries (target beats source by
// (degree, id)) are written, compacted, to the block's slice of ku / kv, with
// the bits and counts direct_place needs; else ku receives every entry's row.
// res[DX_WORK] += the lists' lengths, summed over the edges u->v: d+(u) + d+(v) of an
// oriented graph, and where the orientation is made here the degree of u, which
// sums to the same (each vertex's d+ counts once per edge at it).
// Where the graph comes oriented, only the counted rows [row_begin, row_end) have
// work.  With vtx_off the column ids are local to the row's graph (vgroup).  deg: the
// vertices' degrees, or null (from the row pointers).
template <bool ORIENT, int PER>
__global__ void __launch_bounds__(DR_TILE / PER) direct_rows_kernel(
    const int64_t *__restrict__ rowptr, const int32_t *__restrict__ col, int64_t n, int64_t nnz,
    const int32_t *__restrict__ vgroup, const int64_t *__restrict__ vtx_off, const uint32_t *__restrict__ deg,
    uint32_t row_begin, uint32_t row_end, int32_t *__restrict__ ku, int32_t *__restrict__ kv, uint32_t *__restrict__ mask, uint32_t *__restrict__ gpre, uint32_t *__restrict__ bsum,
    unsigned long long *__restrict__ res) {
  __shared__ uint32_t s_cnt[DR_GROUPS];
  __shared__ unsigned long long s_work;
  __shared__ bool s_bad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  begin_pass();
  if (blockIdx.x == 0 && threadIdx.x == 0) res[DX_START] = clock_ns();
  if (threadIdx.x == 0) {
    s_work = 0;
    s_bad = vtx_off && (unsigned)res[DX_FLAGS];  // the graphs' vertex ranges; other blocks may be adding flags
  }
  __syncthreads();
  if (s_bad) return;
  unsigned f = 0;
  unsigned long long len = 0;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= n; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = rowptr[u];
    if (u == 0 && a != 0) f |= VF_ROWPTR_ENDS;
    if (u == n && a != nnz) f |= VF_ROWPTR_ENDS;
    if (u < n && rowptr[u + 1] < a) f |= VF_ROWPTR_ORDER;
    if (a < 0 || a > nnz) f |= VF_ROWPTR_ENDS;
  }
  const int64_t tile = (int64_t)blockIdx.x * DR_TILE;
  const uint32_t w0 = (uint32_t)tile + warp * (32 * PER);  // below 2^32 where it is used
  uint32_t row[PER];
  int32_t vv[PER];
  unsigned bal[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    row[k] = 0;
    vv[k] = 0;
    bal[k] = 0;
  }
  if (tile + warp * (32 * PER) < nnz) {
    const uint32_t w1 = (uint32_t)min(nnz, (int64_t)w0 + 32 * PER);
    uint32_t rb[PER], re[PER], dv[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) vv[k] = w0 + 32 * k + lane < w1 ? __ldg(col + w0 + 32 * k + lane) : -1;
    entry_rows(rowptr, (uint32_t)n, w0, w1, lane, row, rb, re);
    int32_t g_lo = 0, g_hi = 0, base = 0;
    uint32_t size = (uint32_t)n;
    if (vtx_off) {  // one graph for the whole warp, mostly
      g_lo = vgroup[__shfl_sync(TC_FULL_MASK, row[0], 0)];
      g_hi = vgroup[__shfl_sync(TC_FULL_MASK, row[PER - 1], 31)];
      base = (int32_t)vtx_off[g_lo];
      size = (uint32_t)(vtx_off[g_lo + 1] - base);
    }
    int32_t prev_last = w0 > 0 ? __ldg(col + w0 - 1) : -1;  // entry before the warp's
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const uint32_t e = w0 + 32 * k + lane;
      if (g_lo != g_hi) {
        const int32_t gi = vgroup[row[k]];
        base = (int32_t)vtx_off[gi];
        size = (uint32_t)(vtx_off[gi + 1] - base);
      }
      int32_t prev = __shfl_up_sync(TC_FULL_MASK, vv[k], 1);
      if (lane == 0) prev = prev_last;
      prev_last = __shfl_sync(TC_FULL_MASK, vv[k], 31);
      dv[k] = 0;
      if (e < w1) {
        if ((uint32_t)vv[k] >= size) {
          f |= VF_ID_RANGE;
          vv[k] = -1;
        } else {
          if (e > rb[k] && prev >= vv[k]) f |= VF_UNSORTED;
          vv[k] += base;
          if (vv[k] == (int32_t)row[k]) f |= VF_SELF_LOOP;
          dv[k] = deg ? __ldg(deg + vv[k]) : low_word(rowptr, (uint32_t)vv[k] + 1) - low_word(rowptr, (uint32_t)vv[k]);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const uint32_t du = re[k] - rb[k];
      const bool ok = w0 + 32 * k + lane < w1 && vv[k] >= 0;
      if (ORIENT) {
        const bool keep = ok && (du < dv[k] || (du == dv[k] && (int32_t)row[k] < vv[k]));
        bal[k] = __ballot_sync(TC_FULL_MASK, keep);
        if (keep) len += du;
      } else if (w0 + 32 * k + lane < w1) {
        ku[w0 + 32 * k + lane] = (int32_t)row[k];
        if (ok && row[k] >= row_begin && row[k] < row_end) len += (unsigned long long)du + dv[k];
      }
    }
    len = warp_sum(len);
    if (lane == 0 && len) atomicAdd(&s_work, len);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_work) atomicAdd(res + DX_WORK, s_work);
  if (ORIENT) {
    if (lane < PER) {
      unsigned b = bal[0];
#pragma unroll
      for (int k = 1; k < PER; ++k) b = lane == k ? bal[k] : b;
      s_cnt[warp * PER + lane] = __popc(b);
      mask[blockIdx.x * DR_GROUPS + warp * PER + lane] = b;
    }
    __syncthreads();
    const uint32_t c = s_cnt[lane];
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(TC_FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    if (warp == 0) {
      gpre[blockIdx.x * DR_GROUPS + lane] = incl - c;
      if (lane == 31) bsum[blockIdx.x] = incl;
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const uint32_t at = __shfl_sync(TC_FULL_MASK, incl - c, warp * PER + k) + __popc(bal[k] & lt);
      if ((bal[k] >> lane) & 1u) {
        ku[tile + at] = (int32_t)row[k];
        kv[tile + at] = vv[k];
      }
    }
  }
  f = __reduce_or_sync(TC_FULL_MASK, f);
  if (lane == 0 && f) atomicOr(reinterpret_cast<unsigned *>(res + DX_FLAGS), f);
}

// Moves the blocks' slices to their place and derives the DAG row pointers
// from the kept bits.  boff: block offsets (scanned by the caller), or null
// (at most DR_SMEM_BLOCKS blocks), and then every block scans the sums
// itself: 16 KB from L2 cost less than three scan launches.
__global__ void __launch_bounds__(DR_THREADS) direct_place_kernel(
    const int64_t *__restrict__ rowptr, int64_t n, int64_t nnz, int blocks, const uint32_t *__restrict__ bsum,
    const uint32_t *boff, const uint32_t *__restrict__ mask, const uint32_t *__restrict__ gpre,
    const int32_t *__restrict__ ku, const int32_t *__restrict__ kv, int32_t *__restrict__ src,
    int32_t *__restrict__ col, uint32_t *__restrict__ drow, const unsigned long long *res,
    unsigned long long max_work) {
  __shared__ uint32_t s_off[DR_SMEM_BLOCKS + 1];
  __shared__ uint32_t tmp[33];
  begin_pass();
  if (direct_off(res, max_work)) return;
  if (!boff) {
    const int per = ((blocks + DR_THREADS - 1) / DR_THREADS) | 1;  // odd: the threads' slices start in different banks
    const int b0 = min(blocks, (int)threadIdx.x * per), b1 = min(blocks, b0 + per);
    for (int b = threadIdx.x; b < blocks; b += DR_THREADS) s_off[b] = bsum[b];
    __syncthreads();
    uint32_t s = 0, tot;
    for (int b = b0; b < b1; ++b) s += s_off[b];
    uint32_t run = block_exclusive_scan<uint32_t>(s, tmp, &tot);
    for (int b = b0; b < b1; ++b) {
      const uint32_t c = s_off[b];
      s_off[b] = run;
      run += c;
    }
    if (threadIdx.x == 0) s_off[blocks] = tot;
    __syncthreads();
  }
  const uint32_t m = boff ? boff[blocks] : s_off[blocks];
  for (int b = blockIdx.x; b < blocks; b += gridDim.x) {
    const uint32_t at = boff ? boff[b] : s_off[b], c = bsum[b];
    for (uint32_t i = threadIdx.x; i < c; i += DR_THREADS) {
      src[at + i] = ku[(int64_t)b * DR_TILE + i];
      col[at + i] = kv[(int64_t)b * DR_TILE + i];
    }
  }
  for (int64_t u = (int64_t)blockIdx.x * DR_THREADS + threadIdx.x; u <= n; u += (int64_t)gridDim.x * DR_THREADS) {
    const int64_t x = rowptr[u];
    uint32_t p = m;
    if (x < nnz) {
      const int64_t g = x >> 5;
      const int b = (int)(g / DR_GROUPS);
      p = (boff ? boff[b] : s_off[b]) + gpre[g] + __popc(mask[g] & ((1u << (x & 31)) - 1u));
    }
    drow[u] = p;
  }
}

// The counted graph: rows sorted by id.  Row pointers are 32-bit words `1 <<
// shift` apart: those made here, or the low words of the caller's int64.  The
// edges are the entries of rows [row_begin, row_end).
struct DirectDag {
  const uint32_t *rp;
  int shift;
  const int32_t *col;
  const int32_t *src;    // row of every entry
  int64_t n;
  int64_t row_begin, row_end;
  const int32_t *vgroup;               // batch: graph of every vertex
  const int64_t *vtx_off;              // batch: vertex range of every graph
  const uint8_t *label;                // labelled counts
  int want;
  int words, slots;                    // a warp's bitmaps: slots rows, 32 * words ids each (powers of two)
};

constexpr int DC_THREADS = 256;
constexpr int DC_WARPS = DC_THREADS / 32;
constexpr int DC_BLOCKS = 3;        // blocks per SM that the registers allow (and the 64 KB of bitmaps)
constexpr int DC_WORDS = 2048;      // most shared-memory words of a warp: bitmaps of 65536 ids
constexpr int DC_WORDS_MIN = 512;
constexpr int DC_SMEM = DC_WARPS * DC_WORDS * (int)sizeof(uint32_t);
constexpr int DC_SLOTS = 4, DC_SLOTS_HASHED = 2;  // rows at a time
constexpr int DC_U = 4;             // searches in flight per lane
constexpr int DC_GU = 3;            // 16-byte list loads in flight per lane
constexpr int DC_RUNS = 4;          // more rows than this (and bitmaps) in 32 edges: all of them searched
constexpr int DC_SEARCH = 8;        // target list this many times the row's: searched

// A warp takes 32 consecutive edges.  Each of their rows' lists becomes a
// bitmap of ids modulo 32 * words in the warp's 8 KB of shared memory (4
// bitmaps of 16384 ids, 2 or 1 wider ones, or 2 hashed ones in 4 KB), and the targets' lists, read
// in 16-byte groups flattened over the lanes, are tested against their edge's
// bitmap: one shared-memory test per entry instead of a search of log2
// dependent loads.  An edge sets its own target's bit; only the parts of the
// first and last row outside the 32 edges are read for their bits.  A graph of
// at most 32 * words vertices makes the test exact; otherwise a hit is
// confirmed by a search of the row.  Where the edges have more than 4 rows (and
// more than there are bitmaps), or a target's list is much longer than the row's, the shorter
// list's entries are searched in the longer one, flattened over the lanes too.
// Bound by instruction issue at the 24 warps that the bitmaps leave an SM (54 %
// of cycles issue, 3.5 warps wait on L2 for each that does; 256 mixed graphs): the
// per-batch work (sums, bitmaps) is spread over 32 edges whatever their rows,
// which took this kernel from 3.9 ms (a pass per row) to 2.8 ms on 1024 mixed
// small graphs (49 M edges).  Three
// blocks with 3 loads in flight a lane against four with 2 (the bitmaps leave
// room for three): 647 -> 625 us on 256 such graphs; 4 loads 637.
// MODE 0: counts; 1: triangles of every vertex; 2: common neighbours of one
// label.  In MODE 1 the hubs of a skewed graph are in most triangles, and
// additions to one address take turns: the warps spread them over `copies`
// arrays of n counts.
template <int MODE>
__device__ __forceinline__ void direct_count_block(const DirectDag &g, uint32_t *__restrict__ out,
                                                   unsigned long long cap, int chunk,
                                                   unsigned long long *__restrict__ vcount, int copies,
                                                   unsigned long long *__restrict__ totals,
                                                   unsigned long long *res, unsigned long long max_work) {
  extern __shared__ __align__(16) uint32_t s_bm[];
  __shared__ int4 s_rec[DC_WARPS][32];
  __shared__ uint32_t s_hits[DC_WARPS][32];
  __shared__ uint2 s_row[DC_WARPS][32];  // hashed bitmaps: each edge's row, (first entry, length)
  __shared__ unsigned long long s_sum[2];
  if (direct_off(res, max_work)) return;
  const uint32_t first = g.rp[(size_t)g.row_begin << g.shift], last = g.rp[(size_t)g.row_end << g.shift];
  if (blockIdx.x == 0 && threadIdx.x == 0) res[DX_M] = last - first;
  if (out && (unsigned long long)(last - first) > cap) return;  // the host reports it
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  const int wwords = g.words * g.slots, slots = g.slots;
  uint32_t *bm = s_bm + w * wwords, *hits = s_hits[w];
  int4 *rec = s_rec[w];
  if (MODE == 1) vcount += (int64_t)((blockIdx.x * DC_WARPS + w) % copies) * g.n;
  for (int q = lane; q < wwords; q += 32) bm[q] = 0u;
  if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
  __syncthreads();
  const int32_t *__restrict__ col = g.col;
  const uintptr_t col_blk = reinterpret_cast<uintptr_t>(col) >> 4;
  const uint32_t col_off = (uint32_t)(reinterpret_cast<uintptr_t>(col) >> 2) & 3u;  // col[0] in its 16-byte block
  const uint32_t wmask = (uint32_t)g.words - 1u;
  unsigned long long acc = 0, alg = 0;
  int32_t cur = -1;  // batch: the graph acc belongs to
  bool exact = g.n <= 32 * (int64_t)g.words;
  const uint32_t batches = (last - first + 31) / 32, warps = gridDim.x * DC_WARPS;
  for (uint32_t c0 = (blockIdx.x * DC_WARPS + w) * chunk; c0 < batches; c0 += warps * chunk) {
    const uint32_t c1 = min(batches, c0 + chunk);
    for (uint32_t bt = c0; bt < c1; ++bt) {
      const uint32_t f = first + bt * 32, e = f + lane;
      const bool in = e < last;
      const int32_t u = in ? __ldg(g.src + e) : -1, v = in ? __ldg(col + e) : 0;
      uint32_t a0 = 0, b0 = 0, na = 0, nb = 0;
      if (in) {
        const uint32_t *pu = g.rp + ((size_t)(uint32_t)u << g.shift), *pv = g.rp + ((size_t)(uint32_t)v << g.shift);
        a0 = __ldg(pu);
        na = __ldg(pu + (1 << g.shift)) - a0;
        b0 = __ldg(pv);
        nb = __ldg(pv + (1 << g.shift)) - b0;
        alg += na + nb + 1u;
      }
      int32_t gid = -1;
      bool mixed = false;  // batch: the edges belong to several graphs
      if (g.vgroup) {
        gid = in ? __ldg(g.vgroup + u) : -1;
        const int32_t g0 = __shfl_sync(TC_FULL_MASK, gid, 0);
        mixed = __any_sync(TC_FULL_MASK, in && gid != g0);
        if (g0 != cur) {
          if (cur >= 0) {
            acc = warp_sum(acc);
            if (lane == 0 && acc) atomicAdd(totals + cur, acc);
          }
          acc = 0;
          cur = g0;
        }
        // (a bitmap holds ids of one graph, a range of at most its size)
        const int64_t size = in ? g.vtx_off[gid + 1] - g.vtx_off[gid] : 0;
        exact = __all_sync(TC_FULL_MASK, size <= 32 * (int64_t)g.words);
      }
      const bool pe = out != nullptr || MODE == 1 || mixed;  // hits summed per edge
      if (pe) hits[lane] = 0u;
      const int32_t up = __shfl_up_sync(TC_FULL_MASK, u, 1);
      const unsigned hm = __ballot_sync(TC_FULL_MASK, in && (lane == 0 || u != up));  // first edge of each row
      const int run = __popc(hm & ((2u << lane) - 1u)) - 1;                           // the edge's row, from 0
      const int runs = __popc(hm);
      const bool live = in && na > 1 && nb > 0;  // a row of one entry closes nothing
      const bool search = live && (runs > max(slots, DC_RUNS) || nb / DC_SEARCH > na);
      const bool stream = live && !search;

      if (__any_sync(TC_FULL_MASK, search)) {
        const bool a_short = na <= nb;
        const uint32_t ns = search ? (a_short ? na : nb) : 0u;
        uint32_t incl = ns;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(TC_FULL_MASK, incl, o);
          if (lane >= o) incl += y;
        }
        const uint32_t tot = __shfl_sync(TC_FULL_MASK, incl, 31);
        rec[lane] = make_int4((int)incl, (int)((a_short ? a0 : b0) - (incl - ns)), (int)(a_short ? b0 : a0),
                              (int)(a_short ? nb : na));
        __syncwarp();
        int c = 0;
        int4 r = rec[0];
        for (uint32_t i0 = 0; i0 < tot; i0 += 32 * DC_U) {
          int32_t key[DC_U];
          uint32_t lo[DC_U], hi[DC_U], end[DC_U];
          int ce[DC_U], width = 0;
#pragma unroll
          for (int j = 0; j < DC_U; ++j) {
            const uint32_t i = i0 + 32 * j + lane;
            key[j] = 0;
            lo[j] = hi[j] = end[j] = 0;
            if (i < tot) {
              while (i >= (uint32_t)r.x) r = rec[++c];  // ends: rec[31].x == tot > i
              key[j] = __ldg(col + ((uint32_t)r.y + i));
              lo[j] = (uint32_t)r.z;
              hi[j] = end[j] = lo[j] + (uint32_t)r.w;
              width = max(width, r.w);
            }
            ce[j] = c;
          }
          while (width > 0) {
#pragma unroll
            for (int j = 0; j < DC_U; ++j)
              if (lo[j] < hi[j]) {
                const uint32_t mid = lo[j] + ((hi[j] - lo[j]) >> 1);
                if (__ldg(col + mid) < key[j]) lo[j] = mid + 1;
                else hi[j] = mid;
              }
            width >>= 1;
          }
#pragma unroll
          for (int j = 0; j < DC_U; ++j)
            if (lo[j] < end[j] && __ldg(col + lo[j]) == key[j]) {
              if (MODE == 2 && (int)g.label[key[j]] != g.want) continue;
              if (MODE == 1) atomicAdd(vcount + key[j], 1ull);
              if (pe) atomicAdd(hits + ce[j], 1u);
              else ++acc;
            }
        }
        __syncwarp();
      }

      if (!exact) s_row[w][lane] = make_uint2(a0, na);
      // rows r0 .. r0 + slots - 1 at a time
      for (int r0 = 0; r0 < runs && __any_sync(TC_FULL_MASK, stream); r0 += slots) {
        const bool here = in && run >= r0 && run < r0 + slots;
        const unsigned who = __ballot_sync(TC_FULL_MASK, here);
        uint32_t *mine = bm + (here ? run - r0 : 0) * g.words;
        if (here) atomicOr(mine + (((uint32_t)v >> 5) & wmask), 1u << (v & 31));
        // the first row's entries before its edges here, the last row's after
        const int y = __ffs(who) - 1, z = 31 - __clz(who);
        const uint32_t h0 = __shfl_sync(TC_FULL_MASK, a0, y), h1 = f + y, t0 = f + z + 1;
        const uint32_t t1 = __shfl_sync(TC_FULL_MASK, a0 + na, z);
        uint32_t *tail = bm + (__shfl_sync(TC_FULL_MASK, run, z) - r0) * g.words;
        for (uint32_t q = h0 + lane; q < h1; q += 32) {
          const uint32_t x = (uint32_t)__ldg(col + q);
          atomicOr(bm + ((x >> 5) & wmask), 1u << (x & 31));
        }
        for (uint32_t q = t0 + lane; q < t1; q += 32) {
          const uint32_t x = (uint32_t)__ldg(col + q);
          atomicOr(tail + ((x >> 5) & wmask), 1u << (x & 31));
        }
        // the targets' lists in 16-byte groups, each list widened to the
        // aligned blocks that hold it (a block with a valid entry lies in
        // that entry's page).  A record per list that is read: (groups before
        // it, block of group 0, one past its groups, bitmap << 9 | lane << 4 |
        // entries of the last block past the list << 2 | of the first before it)
        const uint32_t B = b0 + col_off, off = B & 3u;
        const uint32_t ng = stream && here ? (off + nb + 3u) >> 2 : 0u;
        uint32_t incl = ng;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(TC_FULL_MASK, incl, o);
          if (lane >= o) incl += t;
        }
        const uint32_t tot = __shfl_sync(TC_FULL_MASK, incl, 31), excl = incl - ng;
        const unsigned full = __ballot_sync(TC_FULL_MASK, ng > 0);
        if (ng > 0)
          rec[__popc(full & lt)] = make_int4((int)excl, (int)((B >> 2) - excl), (int)incl,
                                             (int)((uint32_t)((run - r0) * g.words) << 9 | (uint32_t)lane << 4 |
                                                   ((0u - off - nb) & 3u) << 2 | off));
        __syncwarp();
        int base = -1, hc = 0;  // base: last record that starts before the window of 32 groups
        uint32_t hit_n = 0;
        for (uint32_t i0 = 0; i0 < tot; i0 += 32 * DC_GU) {
          int4 q[DC_GU];
          unsigned valid[DC_GU];  // bit t: entry t of the group belongs to the list
          uint32_t tag[DC_GU];
#pragma unroll
          for (int j = 0; j < DC_GU; ++j) {
            // the lists that start in the window, as bits: a group's list is
            // found by counting them, without walking the records
            const uint32_t s = excl - (i0 + 32 * j), i = i0 + 32 * j + lane;
            const unsigned starts = __reduce_or_sync(TC_FULL_MASK, ng > 0 && s < 32u ? 1u << s : 0u);
            q[j] = make_int4(0, 0, 0, 0);
            valid[j] = 0;
            tag[j] = 0;
            if (i < tot) {
              const int4 r = rec[base + __popc(starts & ((2u << lane) - 1u))];
              q[j] = __ldg(reinterpret_cast<const int4 *>(col_blk << 4) + (uint32_t)((uint32_t)r.y + i));
              const unsigned lo = i == (uint32_t)r.x ? (unsigned)r.w & 3u : 0u;
              const unsigned cut = i + 1 == (uint32_t)r.z ? ((unsigned)r.w >> 2) & 3u : 0u;
              valid[j] = (15u >> cut) & (15u << lo);
              tag[j] = (uint32_t)r.w >> 4;
            }
            base += __popc(starts);
          }
#pragma unroll
          for (int j = 0; j < DC_GU; ++j) {
            const int ce = (int)(tag[j] & 31u);
            if (pe && ce != hc) {
              if (hit_n) atomicAdd(hits + hc, hit_n);
              hc = ce;
              hit_n = 0;
            }
            const uint32_t xs[4] = {(uint32_t)q[j].x, (uint32_t)q[j].y, (uint32_t)q[j].z, (uint32_t)q[j].w};
            const uint32_t *t = bm + (tag[j] >> 5);
            unsigned got = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              got |= (__funnelshift_r(t[(xs[k] >> 5) & wmask], 0u, xs[k]) & 1u) << k;
            got &= valid[j];
            if (MODE == 0 && exact) {
              hit_n += __popc(got);
              continue;
            }
            uint32_t ra = 0, rn = 0;
            if (got && !exact) {
              const uint2 rw = s_row[w][ce];
              ra = rw.x;
              rn = rw.y;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (!((got >> k) & 1u)) continue;
              if (!exact) {
                uint32_t l = 0, h2 = rn;
                while (l < h2) {
                  const uint32_t mid = (l + h2) >> 1;
                  if (__ldg(col + ra + mid) < (int32_t)xs[k]) l = mid + 1;
                  else h2 = mid;
                }
                if (l == rn || __ldg(col + ra + l) != (int32_t)xs[k]) continue;
              }
              if (MODE == 2 && (int)g.label[xs[k]] != g.want) continue;
              if (MODE == 1) atomicAdd(vcount + xs[k], 1ull);
              ++hit_n;
            }
          }
        }
        if (!pe) acc += hit_n;
        else if (hit_n) atomicAdd(hits + hc, hit_n);
        __syncwarp();
        // back to zero
        if ((h1 - h0) + (t1 - t0) > 256) {
          uint4 *b4 = reinterpret_cast<uint4 *>(bm);
          for (int q = lane; q < wwords / 4; q += 32) b4[q] = make_uint4(0u, 0u, 0u, 0u);
        } else {
          if (here) mine[((uint32_t)v >> 5) & wmask] = 0u;
          for (uint32_t q = h0 + lane; q < h1; q += 32) bm[((uint32_t)__ldg(col + q) >> 5) & wmask] = 0u;
          for (uint32_t q = t0 + lane; q < t1; q += 32) tail[((uint32_t)__ldg(col + q) >> 5) & wmask] = 0u;
        }
        __syncwarp();
      }

      if (pe) {
        __syncwarp();
        const uint32_t c = hits[lane];
        if (in) {
          if (out) out[e - first] = c;
          if (MODE == 1 && c) {
            atomicAdd(vcount + u, (unsigned long long)c);
            atomicAdd(vcount + v, (unsigned long long)c);
          }
          if (mixed) {
            if (c) atomicAdd(totals + gid, (unsigned long long)c);
          } else {
            acc += c;
          }
        }
        __syncwarp();
      }
    }
  }
  acc = warp_sum(acc);
  alg = warp_sum(alg);
  if (g.vgroup) {
    if (lane == 0 && acc && cur >= 0) atomicAdd(totals + cur, acc);
    acc = 0;
  }
  if (lane == 0) {
    if (acc) atomicAdd(&s_sum[0], acc);
    if (alg) atomicAdd(&s_sum[1], 4ull * alg);
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_sum[threadIdx.x]) atomicAdd(res + (threadIdx.x ? DX_ALG : DX_TOTAL), s_sum[threadIdx.x]);
}

// The last block to finish writes the results to `host` (mapped page-locked
// memory, or null), so that the host waits for the stream and has them: a copy
// of its own after the kernel took 6 us.
template <int MODE>
__global__ void __launch_bounds__(DC_THREADS, DC_BLOCKS) direct_count_kernel(
    DirectDag g, uint32_t *__restrict__ out, unsigned long long cap, int chunk,
    unsigned long long *__restrict__ vcount, int copies, unsigned long long *__restrict__ totals,
    unsigned long long *res, unsigned long long max_work, volatile unsigned long long *host) {
  __shared__ bool s_last;
  begin_pass();
  if (blockIdx.x == 0 && threadIdx.x == 0) res[DX_COUNT] = clock_ns();
  direct_count_block<MODE>(g, out, cap, chunk, vcount, copies, totals, res, max_work);
  if (!host) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(res + DX_DONE, 1ull) == gridDim.x - 1;
  __syncthreads();
  if (s_last && threadIdx.x < DX_WORDS) {
    __threadfence();
    host[threadIdx.x] = threadIdx.x == DX_END ? clock_ns() : __ldcg(res + threadIdx.x);
    __threadfence_system();
  }
}

// Clears the caller's vertex counts where they are counted in place (one copy),
// once the graph is known to be counted: a refused call leaves them as they were.
__global__ void __launch_bounds__(DC_THREADS) direct_clear_kernel(unsigned long long *__restrict__ out, int64_t n,
                                                                 const unsigned long long *res,
                                                                 unsigned long long max_work) {
  begin_pass();
  if (direct_off(res, max_work)) return;
  for (int64_t u = (int64_t)blockIdx.x * DC_THREADS + threadIdx.x; u < n; u += (int64_t)gridDim.x * DC_THREADS) out[u] = 0;
}

// Sums the copies of the vertex counts.
__global__ void __launch_bounds__(DC_THREADS) direct_vsum_kernel(const unsigned long long *__restrict__ t, int64_t n,
                                                                int copies, unsigned long long *__restrict__ out,
                                                                const unsigned long long *res,
                                                                unsigned long long max_work) {
  begin_pass();
  if (direct_off(res, max_work)) return;
  for (int64_t u = (int64_t)blockIdx.x * DC_THREADS + threadIdx.x; u < n; u += (int64_t)gridDim.x * DC_THREADS) {
    unsigned long long s = 0;
    for (int c = 0; c < copies; ++c) s += t[c * n + u];
    out[u] = s;
  }
}

// ---- host side ---------------------------------------------------------------------

// Which calls count directly: entries and vertices by a bound, and W = summed
// list lengths (see direct_rows_kernel), which skew and density drive and only
// the device knows, by a limit past which the kernels return at once and the
// general path counts, 45 us later than if it had been asked.  Both paths of one
// build, us a call (direct, general asked at once); the lines lie where the direct
// one costs as much as declining, lower where dense parts would lose more:
//   exact bitmaps, count: ER n = 300 40, 290; Chung-Lu n = 60 000 W = 84 M 165,
//     440; R-MAT scale 16 163 M 246, 576, 496 M 487, 670, 990 M 772, 781; scale 14
//     1.4 G 803, 742; clique of 1300 1.1 G 730, 540
//   the same, an oriented input: scale 16 990 M 739, 956; ER of degree 250 0.9 G
//     454, 1888; but clique of 1200 (lists of 1168 on average) 864 M 1000, 660
//   the same, labelled (a byte gathered per hit): scale 16 163 M 356, 575; scale 14
//     349 M 560, 598; scale 15 365 M 620, 586; clique of 900 365 M 1153, 629
//   the same, per vertex (an atomic per triangle): scale 16 51 M 221, 521; 380 M 767,
//     753; scale 13 120 M 469, 536; clique of 450 46 M 548, 599; geometric 102 M 527,
//     484; clique of 640 131 M 1155, 781
//   hashed bitmaps, count: R-MAT scale 17 38 M 237, 398, 102 M 563, 538, 189 M
//     927, 560; Chung-Lu n = 300 000 105 M 417, 469; R-MAT
//     scale 20 of flat skew 116 M 597, 585; geometric n = 130 000 223 M
//     1013, 629; ER n = 130 000 221 M 455, 626; clique of 640 133 M 1262, 632
//   the same, an oriented input: scale 17 102 M 520, 516; scale 18 141 M 752, 646;
//     Chung-Lu 105 M 379, 735, n = 100 000 162 M 616, 1133; scale 17 189 M 932, 601;
//     clique of 640 1236, 1549; geometric 108 M 609, 413
//   the same, labelled: scale 18 56 M 386, 395; Chung-Lu n = 1 M 68 M 298, 458;
//     scale 17 102 M 641, 516; geometric 83 M 528, 472; clique of 500 65 M 804, 553
//   the same, per vertex: scale 19 65 M 435, 433; geometric 83 M 518, 466; scale 17
//     102 M 663, 606; clique of 500 818, 732
constexpr int64_t DIRECT_MAX_NNZ = int64_t(1) << 23;
constexpr int64_t DIRECT_MAX_N = int64_t(1) << 22;

static unsigned long long direct_max_work(int64_t n, int64_t nnz, const DirectReq &rq) {
  const bool exact = n <= 32 * DC_WORDS;
  if (rq.vertex_counts) return exact ? 15ull << 23 : 5ull << 24;
  if (rq.labels) return exact ? 21ull << 24 : 3ull << 25;
  if (!rq.orient) return exact ? std::min(1ull << 30, 1024ull * (unsigned long long)nnz) : 5ull << 25;
  return exact ? 1ull << 30 : 7ull << 24;
}

tc_status direct_init(tc_ctx *ctx) {
  const void *k[] = {(const void *)direct_count_kernel<0>, (const void *)direct_count_kernel<1>,
                     (const void *)direct_count_kernel<2>};
  for (const void *f : k)
    TC_CHECK_CUDA(ctx, cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_SMEM));
  return TC_OK;
}

bool direct_fits(int64_t n, int64_t nnz, const tc_opts &o) {
  return nnz <= DIRECT_MAX_NNZ && n <= DIRECT_MAX_N && o.validate && o.selector == TC_SELECT_FIXED &&
         !o.record_tile_costs;
}

static int rows_blocks(int64_t nnz) { return (int)std::max<int64_t>(1, (nnz + DR_TILE - 1) / DR_TILE); }

// Copies of the vertex counts (MODE 1): up to 32, 2^22 counts in all.
static int vertex_copies(int64_t n) {
  int c = 1;
  while (c < 32 && 2 * c * n <= (int64_t(1) << 22)) c *= 2;
  return c;
}

void direct_sizes(const tc_ctx *ctx, int64_t n, int64_t nnz, const DirectReq &rq, Sizer &sz) {
  const int64_t B = rows_blocks(nnz);
  const int copies = vertex_copies(n);
  sz.take<unsigned long long>(DX_WORDS);
  sz.take<int32_t>(nnz);
  if (rq.vertex_counts && copies > 1) sz.take<unsigned long long>(n * copies);
  if (!rq.orient) return;
  sz.take<int32_t>(nnz);
  sz.take<uint32_t>(B * DR_GROUPS); sz.take<uint32_t>(B * DR_GROUPS);
  sz.take<uint32_t>(B + 1); sz.take<uint32_t>(B + 1);
  sz.take<int32_t>(nnz); sz.take<int32_t>(nnz);
  sz.take<uint32_t>(n + 1);
  sz.take<char>((int64_t)scan_scratch_bytes(ctx, B + 1));
}

// A warp's bitmaps for graphs of up to n vertices.
static void set_bitmaps(DirectDag &g, int64_t n) {
  g.words = DC_WORDS_MIN;
  if (n <= 32 * DC_WORDS)
    while (n > 32 * (int64_t)g.words) g.words *= 2;
  g.slots = n <= 32 * DC_WORDS ? std::min(DC_SLOTS, DC_WORDS / g.words) : DC_SLOTS_HASHED;
}

template <int MODE>
static tc_status launch_count(tc_ctx *ctx, const DirectDag &g, int64_t edges, int chunk, const DirectReq &rq,
                              unsigned long long *vcount, int copies, unsigned long long *totals,
                              unsigned long long *res, unsigned long long max_work, unsigned long long *host) {
  const int64_t batches = std::max<int64_t>(1, (edges + 31) / 32);
  const int smem = DC_WARPS * g.words * g.slots * (int)sizeof(uint32_t);
  const int grid = grid_for(ctx, batches, DC_WARPS, smem > 48 * 1024 ? 3 : 4);
  chunk = (int)std::max<int64_t>(1, std::min<int64_t>(chunk, batches / ((int64_t)grid * DC_WARPS)));
  TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_count_kernel<MODE>, grid, DC_THREADS, smem, g, rq.edge_counts,
                                 (unsigned long long)rq.cap, chunk, vcount, copies, totals, res, max_work, host));
  return TC_OK;
}

tc_status direct_run(tc_ctx *ctx, const DevCSR &d, const DirectReq &rq, Bump &bump, tc_stats *st,
                     bool *declined) {
  const int64_t n = d.n, nnz = d.nnz;
  const int B = rows_blocks(nnz);
  unsigned long long *res = bump.take<unsigned long long>(DX_WORDS);
  int32_t *ku = bump.take<int32_t>(nnz), *kv = nullptr, *src = nullptr, *col = nullptr;
  uint32_t *mask = nullptr, *gpre = nullptr, *bsum = nullptr, *boff = nullptr, *drow = nullptr;
  char *scratch = nullptr;
  const int copies = rq.vertex_counts ? vertex_copies(n) : 1;
  const unsigned long long max_work = direct_max_work(n, nnz, rq);
  if (rq.orient) {
    kv = bump.take<int32_t>(nnz);
    mask = bump.take<uint32_t>((int64_t)B * DR_GROUPS);
    gpre = bump.take<uint32_t>((int64_t)B * DR_GROUPS);
    bsum = bump.take<uint32_t>(B + 1);
    boff = bump.take<uint32_t>(B + 1);
    src = bump.take<int32_t>(nnz);
    col = bump.take<int32_t>(nnz);
    drow = bump.take<uint32_t>(n + 1);
    scratch = bump.take<char>((int64_t)scan_scratch_bytes(ctx, B + 1));
  }
  unsigned long long *vcount = rq.vertex_counts;
  if (copies > 1) vcount = bump.take<unsigned long long>(n * copies);
  if (bump.overflow) return set_error(ctx, TC_ERR_OOM, "arena overflow");
  TC_CHECK_CUDA(ctx, cudaMemsetAsync(res, 0, sizeof(unsigned long long) * DX_WORDS, ctx->stream));
  if (nnz >= DS_MIN_NNZ) {
    constexpr int blocks = DS_WARPS / (DR_THREADS / 32);
    if (rq.orient) direct_sample_kernel<true><<<blocks, DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz, nullptr, nullptr, 0, (uint32_t)n, res);
    else direct_sample_kernel<false><<<blocks, DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz, nullptr, nullptr, (uint32_t)rq.row_begin, (uint32_t)rq.row_end, res);
    TC_CHECK_LAUNCH(ctx);
    TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], res + DX_GUESS, sizeof(unsigned long long),
                                       cudaMemcpyDeviceToHost, ctx->stream));
    TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (ctx->h_pinned[0] > max_work) {
      *declined = true;
      return TC_OK;
    }
  }
  if (copies > 1)
    TC_CHECK_CUDA(ctx, cudaMemsetAsync(vcount, 0, sizeof(unsigned long long) * (size_t)(n * copies), ctx->stream));
  unsigned long long *h = ctx->h_pinned;  // page-locked: the device writes it where it lies
  DirectDag g{nullptr, 0, nullptr, nullptr, n, 0, n, nullptr, nullptr, rq.labels, rq.label, 0, 0};
  set_bitmaps(g, n);
  if (rq.orient) {
    TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_rows_kernel<true, DR_PER>, B, DR_THREADS, 0, d.rowptr, d.col, n, nnz, nullptr,
                                   nullptr, nullptr, 0, (uint32_t)n, ku, kv, mask, gpre, bsum, res));
    if (rq.vertex_counts && copies == 1)
      TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_clear_kernel, grid_for(ctx, n, DC_THREADS, 8), DC_THREADS, 0, vcount, n,
                                     res, max_work));
    const bool scan = B > DR_SMEM_BLOCKS;  // too many block sums for a block to scan
    if (scan) {
      TC_CHECK_CUDA(ctx, cudaMemsetAsync(bsum + B, 0, sizeof(uint32_t), ctx->stream));
      TC_TRY(exclusive_scan_u32(ctx, bsum, boff, B + 1, scratch));
    }
    TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_place_kernel, B, DR_THREADS, 0, d.rowptr, n, nnz, B, bsum,
                                   scan ? boff : nullptr, mask, gpre, ku, kv, src, col, drow, res, max_work));
    g.rp = drow;
    g.col = col;
    g.src = src;
  } else {
    TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_rows_kernel<false, DR_PER>, B, DR_THREADS, 0, d.rowptr, d.col, n, nnz, nullptr,
                                   nullptr, nullptr, (uint32_t)rq.row_begin, (uint32_t)rq.row_end, ku, nullptr, nullptr,
                                   nullptr, nullptr, res));
    g.rp = reinterpret_cast<const uint32_t *>(d.rowptr);
    g.shift = 1;
    g.col = d.col;
    g.src = ku;
    g.row_begin = rq.row_begin;
    g.row_end = rq.row_end;
  }
  const int64_t edges = rq.orient ? nnz / 2 : nnz;
  if (rq.vertex_counts) TC_TRY(launch_count<1>(ctx, g, edges, 1, rq, vcount, copies, nullptr, res, max_work, h));
  else if (rq.labels) TC_TRY(launch_count<2>(ctx, g, edges, 1, rq, nullptr, 1, nullptr, res, max_work, h));
  else TC_TRY(launch_count<0>(ctx, g, edges, 1, rq, nullptr, 1, nullptr, res, max_work, h));
  if (copies > 1)
    TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_vsum_kernel, grid_for(ctx, n, DC_THREADS, 8), DC_THREADS, 0, vcount, n,
                                   copies, rq.vertex_counts, res, max_work));
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[6], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (const unsigned f = (unsigned)h[DX_FLAGS]) return set_error(ctx, TC_ERR_INVALID_GRAPH, "%s", flag_text(f));
  if (h[DX_WORK] > max_work) {
    *declined = true;
    return TC_OK;
  }
  const int64_t m = (int64_t)h[DX_M];
  if (rq.edge_counts && rq.cap < m)
    return set_error(ctx, TC_ERR_INVALID_ARG, "edge_counts holds %lld entries, %lld oriented edges", (long long)rq.cap,
                     (long long)m);
  const auto copies_from = std::chrono::steady_clock::now();
  if (rq.vertex_host)
    TC_CHECK_CUDA(ctx, cudaMemcpy(rq.vertex_host, rq.vertex_counts, sizeof(uint64_t) * (size_t)n, cudaMemcpyDeviceToHost));
  if (rq.edge_host && m > 0)
    TC_CHECK_CUDA(ctx, cudaMemcpy(rq.edge_host, rq.edge_counts, sizeof(uint32_t) * (size_t)m, cudaMemcpyDeviceToHost));
  if (rq.vertex_host || rq.edge_host)
    st->ms_d2h = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - copies_from).count();
  st->m = m;
  st->tiles = (m + TILE_EDGES - 1) / TILE_EDGES;
  st->tiles_per_arm[TC_ARM_FLAT] = st->tiles;  // 32 edges' lists as one flattened run, as that arm
  st->alg_bytes_arm[TC_ARM_FLAT] = st->alg_bytes = h[DX_ALG];
  // events between the passes would keep them apart: the parts are the device
  // clock's, and the copies back, which the host waits for, the host's (events
  // and a wait of their own took 14 of 288 us, Chung-Lu n = 50 000 per vertex)
  const float on_device = elapsed(ctx->ev[0], ctx->ev[6]);
  st->ms_total = on_device + st->ms_d2h;
  if (st->h2d_bytes >= DIRECT_TIMED_H2D) st->ms_h2d = elapsed(ctx->ev[0], ctx->ev[1]);
  else if (st->h2d_bytes) st->ms_h2d = std::max(0.f, on_device - 1e-6f * (float)(h[DX_END] - h[DX_START]));
  st->ms_orient = 1e-6f * (float)(h[DX_COUNT] - h[DX_START]);
  st->ms_arm[TC_ARM_FLAT] = st->ms_count = 1e-6f * (float)(h[DX_END] - h[DX_COUNT]);
  st->d2h_bytes += sizeof(unsigned long long) + (rq.edge_host ? sizeof(uint32_t) * (size_t)m : 0) +
                   (rq.vertex_host ? sizeof(uint64_t) * (size_t)n : 0);
  st->kernel_launches = ctx->launches;
  return TC_OK;
}

// ---- batches -----------------------------------------------------------------------

// Every vertex's graph and degree, and the largest graph's vertices; a vertex range
// outside [0, n) or out of order is flagged.
__global__ void __launch_bounds__(DR_THREADS) direct_group_kernel(const int64_t *__restrict__ vtx_off, int64_t G,
                                                                 int64_t n, const int64_t *__restrict__ rowptr,
                                                                 int32_t *__restrict__ vgroup,
                                                                 uint32_t *__restrict__ deg,
                                                                 unsigned long long *__restrict__ res) {
  for (int64_t g = blockIdx.x; g < G; g += gridDim.x) {
    const int64_t a = vtx_off[g], b = vtx_off[g + 1];
    if (b < a || a < 0 || b > n) {
      if (threadIdx.x == 0) atomicOr(reinterpret_cast<unsigned *>(res + DX_FLAGS), (unsigned)VF_ROWPTR_ORDER);
      continue;
    }
    if (threadIdx.x == 0) atomicMax(res + DX_MAXN, (unsigned long long)(b - a));
    for (int64_t v = a + threadIdx.x; v < b; v += DR_THREADS) {
      vgroup[v] = (int32_t)g;
      deg[v] = (uint32_t)(rowptr[v + 1] - rowptr[v]);
    }
  }
}

// A batch counts directly while its lists are short on average: the summed
// lengths may be BATCH_MAX_LEN per entry.  1024 mixed graphs of 64 to 16384
// vertices (85 M entries, 30 per entry) take 3.6 ms against 7.1 with the
// general path; the streaming tests run at 2.2 T list entries/s, so the
// general path's 0.15 ns an edge is reached at about 300.
// A graph beyond the exact bitmaps has its hits, and the entries that only hash
// alike, confirmed by searches, and pays 4 to 9 ps a list entry.  Per entry of
// the batch, direct against general (us): ER n = 100 000 7.4 712, 813; geometric
// 7.8 887, 839; ER 28 1356, 2016; geometric 29 3033, 2046; R-MAT scale 17 38
// 1698, 1160 and 67 5133, 1846; Chung-Lu n = 2 M 56 8108, 5308; R-MAT scale 18
// 82 6681, 2071.  What such a batch may have in any case is near what one graph
// may (direct_max_work): there the general path's launches cost more.
constexpr int64_t BATCH_MAX_LEN = 128, BATCH_MAX_LEN_HASHED = 8;

static unsigned long long batch_max_work(int64_t max_n, int64_t nnz) {
  if (max_n <= 32 * DC_WORDS) return (unsigned long long)(BATCH_MAX_LEN * std::max<int64_t>(nnz, 1 << 16));
  return (unsigned long long)std::max<int64_t>(BATCH_MAX_LEN_HASHED * nnz, int64_t(3) << 25);
}

bool direct_batch_fits(int64_t nnz, const tc_opts &o) {
  return nnz < (int64_t(1) << 31) && o.validate && o.selector == TC_SELECT_FIXED && !o.record_tile_costs;
}

void direct_batch_sizes(const tc_ctx *ctx, int64_t G, int64_t n, int64_t nnz, Sizer &sz) {
  direct_sizes(ctx, n, nnz, DirectReq(), sz);
  sz.take<int32_t>(n);
  sz.take<uint32_t>(n);
  sz.take<unsigned long long>(G);
}

tc_status direct_batch(tc_ctx *ctx, const DevCSR &d, const int64_t *vtx_off, int64_t G, Bump &bump, uint64_t *totals,
                       tc_stats *st, bool *declined) {
  const int64_t n = d.n, nnz = d.nnz;
  const int B = rows_blocks(nnz);
  unsigned long long *res = bump.take<unsigned long long>(DX_WORDS);
  int32_t *ku = bump.take<int32_t>(nnz), *kv = bump.take<int32_t>(nnz);
  uint32_t *mask = bump.take<uint32_t>((int64_t)B * DR_GROUPS), *gpre = bump.take<uint32_t>((int64_t)B * DR_GROUPS);
  uint32_t *bsum = bump.take<uint32_t>(B + 1), *boff = bump.take<uint32_t>(B + 1);
  int32_t *src = bump.take<int32_t>(nnz), *col = bump.take<int32_t>(nnz);
  uint32_t *drow = bump.take<uint32_t>(n + 1);
  char *scratch = bump.take<char>((int64_t)scan_scratch_bytes(ctx, B + 1));
  int32_t *vgroup = bump.take<int32_t>(n);
  uint32_t *deg = bump.take<uint32_t>(n);
  unsigned long long *tot = bump.take<unsigned long long>(G);
  if (bump.overflow) return set_error(ctx, TC_ERR_OOM, "arena overflow");
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[1], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaMemsetAsync(res, 0, sizeof(unsigned long long) * DX_WORDS, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaMemsetAsync(vgroup, 0, sizeof(int32_t) * (size_t)n, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaMemsetAsync(tot, 0, sizeof(unsigned long long) * (size_t)G, ctx->stream));
  direct_group_kernel<<<(int)std::min<int64_t>(G, 65535), DR_THREADS, 0, ctx->stream>>>(vtx_off, G, n, d.rowptr, vgroup,
                                                                                        deg, res);
  TC_CHECK_LAUNCH(ctx);
  if (nnz >= DS_MIN_NNZ) {
    direct_sample_kernel<true><<<DS_WARPS / (DR_THREADS / 32), DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz,
                                                                                            vgroup, vtx_off, 0, (uint32_t)n, res);
    TC_CHECK_LAUNCH(ctx);
  }
  // the largest graph decides the bitmaps' width, the sampled lists whether to go on
  TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], res, sizeof(unsigned long long) * DX_WORDS,
                                     cudaMemcpyDeviceToHost, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const unsigned long long *h = ctx->h_pinned;
  const int64_t max_n = (int64_t)h[DX_MAXN];
  const unsigned long long max_work = batch_max_work(max_n, nnz);
  if (h[DX_GUESS] > max_work) {
    *declined = true;
    return TC_OK;
  }
  if (nnz >= DR_WIDE_MIN_NNZ)
    TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_rows_kernel<true, DR_WIDE_PER>, B, DR_TILE / DR_WIDE_PER, 0, d.rowptr,
                                   d.col, n, nnz, vgroup, vtx_off, deg, 0, (uint32_t)n, ku, kv, mask, gpre, bsum, res));
  else
    TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_rows_kernel<true, DR_PER>, B, DR_THREADS, 0, d.rowptr, d.col, n, nnz,
                                   vgroup, vtx_off, deg, 0, (uint32_t)n, ku, kv, mask, gpre, bsum, res));
  const bool scan = B > DR_SMEM_BLOCKS;
  if (scan) {
    TC_CHECK_CUDA(ctx, cudaMemsetAsync(bsum + B, 0, sizeof(uint32_t), ctx->stream));
    TC_TRY(exclusive_scan_u32(ctx, bsum, boff, B + 1, scratch));
  }
  TC_CHECK_CUDA(ctx, launch_pass(ctx, direct_place_kernel, std::min(B, ctx->num_sms * 32), DR_THREADS, 0, d.rowptr, n, nnz,
                                 B, bsum, scan ? boff : nullptr, mask, gpre, ku, kv, src, col, drow, res, max_work));
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[5], ctx->stream));
  // runs of 8 batches of 32 edges: a warp rarely leaves a graph inside one
  DirectDag g{drow, 0, col, src, n, 0, n, vgroup, vtx_off, nullptr, 0, 0, 0};
  set_bitmaps(g, max_n);
  TC_TRY(launch_count<0>(ctx, g, nnz / 2, 8, DirectReq(), nullptr, 1, tot, res, max_work, nullptr));
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[6], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], res, sizeof(unsigned long long) * DX_WORDS,
                                     cudaMemcpyDeviceToHost, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (const unsigned f = (unsigned)h[DX_FLAGS]) return set_error(ctx, TC_ERR_INVALID_GRAPH, "%s", flag_text(f));
  if (h[DX_WORK] > max_work) {
    *declined = true;
    return TC_OK;
  }
  TC_CHECK_CUDA(ctx, cudaMemcpyAsync(totals, tot, sizeof(unsigned long long) * G, cudaMemcpyDeviceToHost, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[7], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  st->m = (int64_t)h[DX_M];
  st->tiles = (st->m + TILE_EDGES - 1) / TILE_EDGES;
  st->tiles_per_arm[TC_ARM_FLAT] = st->tiles;
  st->alg_bytes_arm[TC_ARM_FLAT] = st->alg_bytes = h[DX_ALG];
  st->ms_h2d = elapsed(ctx->ev[0], ctx->ev[1]);
  st->ms_orient = elapsed(ctx->ev[1], ctx->ev[5]);
  st->ms_count = elapsed(ctx->ev[5], ctx->ev[6]);
  st->ms_d2h = elapsed(ctx->ev[6], ctx->ev[7]);
  st->ms_total = elapsed(ctx->ev[0], ctx->ev[7]);
  st->d2h_bytes = sizeof(unsigned long long) * G;
  st->kernel_launches = ctx->launches;
  return TC_OK;
}

}  // namespace tc
