// Direct counting of small graphs and of batches of small graphs.
//
// The general path relabels the graph by degree rank, sorts every row and
// groups edges by target before it counts: 45 to 70 launches and a host read
// in the middle, which is all that a small graph's time consists of.  None of
// it changes a count.  Here the oriented graph keeps the input's ids: whether
// u->v stays is a comparison of (degree, id) pairs, input rows are sorted, so
// the kept entries of a row already are, and kept entries compacted in input
// order are the reference's own edge order (graph.cc:279-290).  Three
// launches and one host read at the end:
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

#include "engine.cuh"

namespace tc {

constexpr int DR_THREADS = 256;
constexpr int DR_PER = 4;                             // 32-entry groups per warp
constexpr int DR_TILE = DR_THREADS * DR_PER;          // entries per block
constexpr int DR_GROUPS = DR_TILE / 32;
constexpr int DR_SMEM_BLOCKS = 4096;                  // block sums every placing block scans for itself
static_assert(DR_GROUPS == 32, "one warp scans a block's group counts");

// Largest r in [0, n) with rowptr[r] <= e, for e of the lane's half warp: 16
// lanes probe 16 pivots at a time, so n = 2^22 takes 6 dependent loads
// instead of 22.  Both halves search at once; all lanes must call it.  Ends
// for any rowptr contents, inside [0, n).
__device__ __forceinline__ int64_t half_warp_row(const int64_t *__restrict__ rowptr, int64_t n, int64_t e, int lane) {
  const int hl = lane & 15, sh = lane & 16;
  int64_t lo = 0, hi = n;
  while (__any_sync(TC_FULL_MASK, hi - lo > 1)) {
    const int64_t len = hi - lo, p = lo + ((hl + 1) * len) / 17;
    const bool le = len > 1 && rowptr[p] <= e;
    const int c = __popc((__ballot_sync(TC_FULL_MASK, le) >> sh) & 0xffffu);
    const int64_t nlo = __shfl_sync(TC_FULL_MASK, p, sh + max(c - 1, 0));
    const int64_t nhi = __shfl_sync(TC_FULL_MASK, p, sh + min(c, 15));
    if (len > 1) {
      if (c > 0) lo = nlo;
      if (c < 16) hi = nhi;
    }
  }
  return lo;
}

// Rows of a warp's entries [w0, w1), entry w0 + 32 k + lane in lo[k]: the rows
// of the first and last entry (half_warp_row), then every lane searches its
// own entries' between them, DR_PER searches in flight.
__device__ __forceinline__ void entry_rows(const int64_t *__restrict__ rowptr, int64_t n, int64_t w0, int64_t w1,
                                           int lane, int64_t (&lo)[DR_PER]) {
  const int64_t r = half_warp_row(rowptr, n, lane < 16 ? w0 : w1 - 1, lane);
  const int64_t r_lo = __shfl_sync(TC_FULL_MASK, r, 0), r_hi = __shfl_sync(TC_FULL_MASK, r, 16);
  int64_t hi[DR_PER];
#pragma unroll
  for (int k = 0; k < DR_PER; ++k) {
    lo[k] = r_lo;
    hi[k] = w0 + 32 * k + lane < w1 && r_hi >= r_lo ? r_hi + 1 : r_lo + 1;
  }
  for (bool more = true; more;) {
    more = false;
#pragma unroll
    for (int k = 0; k < DR_PER; ++k) {
      if (hi[k] - lo[k] > 1) {
        const int64_t mid = (lo[k] + hi[k]) >> 1;
        if (rowptr[mid] <= w0 + 32 * k + lane) lo[k] = mid;
        else hi[k] = mid;
        more |= hi[k] - lo[k] > 1;
      }
    }
  }
}

// Results of a direct call, copied to the host in one piece.
enum { DX_TOTAL, DX_M, DX_ALG, DX_FLAGS, DX_WORK, DX_GUESS, DX_WORDS };

// Whether the later kernels have nothing to do: invalid input, or lists too
// long.
__device__ __forceinline__ bool direct_off(const unsigned long long *res, unsigned long long max_work) {
  return (unsigned)res[DX_FLAGS] || res[DX_WORK] > max_work;
}

// A guess of DX_WORK (see direct_rows_kernel) from DS_WARPS runs of 128 entries
// spread evenly over a large graph.  The host reads it before the passes over
// all entries start (12 us), which costs a graph whose lists are too long 25
// us instead of 170 (R-MAT scale 18).
constexpr int DS_WARPS = 512;
constexpr int64_t DS_MIN_NNZ = int64_t(1) << 20;  // below, the pass itself is as quick

template <bool ORIENT>
__global__ void __launch_bounds__(DR_THREADS) direct_sample_kernel(const int64_t *__restrict__ rowptr,
                                                                  const int32_t *__restrict__ col, int64_t n,
                                                                  int64_t nnz, unsigned long long *__restrict__ guess) {
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * (DR_THREADS / 32) + (threadIdx.x >> 5);
  const int64_t w0 = i * (nnz / DS_WARPS), w1 = min(nnz, w0 + 32 * DR_PER);
  int64_t lo[DR_PER];
  entry_rows(rowptr, n, w0, w1, lane, lo);
  unsigned long long len = 0;
#pragma unroll
  for (int k = 0; k < DR_PER; ++k) {
    const int64_t e = w0 + 32 * k + lane;
    const int32_t v = e < w1 ? col[e] : -1;
    if (v < 0 || (int64_t)v >= n) continue;
    const int64_t a = rowptr[lo[k] + 1] - rowptr[lo[k]], b = rowptr[v + 1] - rowptr[v];
    const int64_t l = ORIENT ? min(a, b) : a + b;  // an undirected edge has two entries
    if (l > 0) len += (unsigned long long)l;
  }
  len = warp_sum(len);
  if (lane == 0) atomicAdd(guess, len * (unsigned long long)(nnz / (DS_WARPS * 32 * DR_PER)) / (ORIENT ? 2 : 1));
}

// Row, validity and direction of every entry.  A warp finds the rows of its
// first and last entry together (half_warp_row), every lane the rows of its
// own entries between them.  ORIENT: the kept entries (target beats source by
// (degree, id)) are written, compacted, to the block's slice of ku / kv, with
// the bits and counts direct_place needs; else ku receives every entry's row.
// res[DX_WORK] += the lists' lengths, summed over the edges u->v: d+(u) + d+(v) of an
// oriented graph, and where the orientation is made here the degree of u, which
// sums to the same (each vertex's d+ counts once per edge at it).
// With vtx_off the column ids are local to the row's graph (vgroup).
template <bool ORIENT>
__global__ void __launch_bounds__(DR_THREADS) direct_rows_kernel(
    const int64_t *__restrict__ rowptr, const int32_t *__restrict__ col, int64_t n, int64_t nnz,
    const int32_t *__restrict__ vgroup, const int64_t *__restrict__ vtx_off, int32_t *__restrict__ ku,
    int32_t *__restrict__ kv, uint32_t *__restrict__ mask, uint32_t *__restrict__ gpre, uint32_t *__restrict__ bsum,
    unsigned long long *__restrict__ res) {
  __shared__ uint32_t s_cnt[DR_GROUPS];
  __shared__ unsigned long long s_work;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = lanemask_lt();
  if (threadIdx.x == 0) s_work = 0;
  __syncthreads();
  unsigned f = 0;
  unsigned long long len = 0;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u <= n; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = rowptr[u];
    if (u == 0 && a != 0) f |= VF_ROWPTR_ENDS;
    if (u == n && a != nnz) f |= VF_ROWPTR_ENDS;
    if (u < n && rowptr[u + 1] < a) f |= VF_ROWPTR_ORDER;
    if (a < 0 || a > nnz) f |= VF_ROWPTR_ENDS;
  }
  const int64_t tile = (int64_t)blockIdx.x * DR_TILE, w0 = tile + warp * (32 * DR_PER);
  int32_t uu[DR_PER], vv[DR_PER];
  unsigned bal[DR_PER];
#pragma unroll
  for (int k = 0; k < DR_PER; ++k) {
    uu[k] = vv[k] = 0;
    bal[k] = 0;
  }
  if (w0 < nnz) {
    const int64_t w1 = min(nnz, w0 + 32 * DR_PER);
    int64_t lo[DR_PER];
    entry_rows(rowptr, n, w0, w1, lane, lo);
#pragma unroll
    for (int k = 0; k < DR_PER; ++k) vv[k] = w0 + 32 * k + lane < w1 ? col[w0 + 32 * k + lane] : -1;
    int64_t rb[DR_PER], re[DR_PER], cb[DR_PER], ce[DR_PER];
#pragma unroll
    for (int k = 0; k < DR_PER; ++k) {
      const int64_t e = w0 + 32 * k + lane;
      int64_t size = n;
      int32_t base = 0;
      if (vtx_off && e < w1) {
        const int32_t gi = vgroup[lo[k]];
        base = (int32_t)vtx_off[gi];
        size = vtx_off[gi + 1] - base;
      }
      uu[k] = (int32_t)lo[k];
      if (e < w1) {
        rb[k] = rowptr[lo[k]];
        if ((int64_t)vv[k] >= size || vv[k] < 0) {
          f |= VF_ID_RANGE;
          vv[k] = -1;
        } else {
          if (e > rb[k] && e > 0 && col[e - 1] >= vv[k]) f |= VF_UNSORTED;
          vv[k] += base;
          if (vv[k] == uu[k]) f |= VF_SELF_LOOP;
        }
      }
      if (vv[k] >= 0) {
        re[k] = rowptr[lo[k] + 1];
        cb[k] = rowptr[vv[k]];
        ce[k] = rowptr[vv[k] + 1];
      }
    }
#pragma unroll
    for (int k = 0; k < DR_PER; ++k) {
      if (ORIENT) {
        const bool keep = vv[k] >= 0 && (re[k] - rb[k] < ce[k] - cb[k] ||
                                         (re[k] - rb[k] == ce[k] - cb[k] && uu[k] < vv[k]));
        bal[k] = __ballot_sync(TC_FULL_MASK, keep);
        if (keep) len += (unsigned long long)(re[k] - rb[k]);
      } else if (w0 + 32 * k + lane < w1) {
        ku[w0 + 32 * k + lane] = uu[k];
        if (vv[k] >= 0) len += (unsigned long long)(re[k] - rb[k] + ce[k] - cb[k]);
      }
    }
    len = warp_sum(len);
    if (lane == 0 && len) atomicAdd(&s_work, len);
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_work) atomicAdd(res + DX_WORK, s_work);
  if (ORIENT) {
    if (lane < DR_PER) {
      unsigned b = bal[0];
#pragma unroll
      for (int k = 1; k < DR_PER; ++k) b = lane == k ? bal[k] : b;
      s_cnt[warp * DR_PER + lane] = __popc(b);
      mask[blockIdx.x * DR_GROUPS + warp * DR_PER + lane] = b;
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
    for (int k = 0; k < DR_PER; ++k) {
      const uint32_t at = __shfl_sync(TC_FULL_MASK, incl - c, warp * DR_PER + k) + __popc(bal[k] & lt);
      if ((bal[k] >> lane) & 1u) {
        ku[tile + at] = uu[k];
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
    const uint32_t *__restrict__ boff, const uint32_t *__restrict__ mask, const uint32_t *__restrict__ gpre,
    const int32_t *__restrict__ ku, const int32_t *__restrict__ kv, int32_t *__restrict__ src,
    int32_t *__restrict__ col, uint32_t *__restrict__ drow, unsigned long long *__restrict__ res,
    unsigned long long max_work) {
  __shared__ uint32_t s_off[DR_SMEM_BLOCKS + 1];
  __shared__ uint32_t tmp[33];
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
  if (blockIdx.x == 0 && threadIdx.x == 0) res[DX_M] = m;
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

// The counted graph: rows sorted by id; rp is uint32 (oriented here) or the
// caller's int64.  The edges are entries [first, last) of col.
template <typename RP>
struct DirectDag {
  const RP *rp;
  const int32_t *col;
  const int32_t *src;    // row of every entry
  int64_t n;
  int64_t row_begin, row_end;          // counted rows (int64 row pointers)
  const unsigned long long *m;         // number of entries (rows oriented here)
  const int32_t *vgroup;               // batch: graph of every vertex
  const int64_t *vtx_off;              // batch: vertex range of every graph
  const uint8_t *label;                // labelled counts
  int want;
};

constexpr int DC_THREADS = 256;
constexpr int DC_WARPS = DC_THREADS / 32;
constexpr int DC_WORDS_MIN = 512, DC_WORDS_MAX = 2048;  // per-warp bitmap: 16384 to 65536 ids
constexpr int DC_U = 4;             // searches in flight per lane
constexpr int DC_GU = 2;            // 16-byte list loads in flight per lane
constexpr int DC_RUNS = 4;          // more rows than this in 32 edges: all of them searched
constexpr int DC_SEARCH = 8;        // target list this many times the row's: searched

// A warp takes 32 consecutive edges.  Where they belong to a few rows, the
// row's list becomes a bitmap of ids modulo 32 * WORDS in the warp's shared
// memory and the targets' lists, flattened over the lanes, are read
// (coalesced) and tested against it: one shared-memory test per entry instead
// of a search of log2 dependent loads.  A graph of at most 32 * WORDS vertices
// makes the test exact; otherwise a hit is confirmed by a search of the row.
// Where 32 edges span many short rows, or a target's list is much longer than
// the row's, the shorter list's entries are searched in the longer one,
// flattened over the lanes too.  Bound by L1/L2 latency: 64 warps per SM.
// MODE 0: counts; 1: triangles of every vertex; 2: common neighbours of one
// label.  In MODE 1 the hubs of a skewed graph are in most triangles, and
// additions to one address take turns: the warps spread them over `copies`
// arrays of n counts.
template <int MODE, typename RP, int WORDS>
__global__ void __launch_bounds__(DC_THREADS) direct_count_kernel(DirectDag<RP> g, uint32_t *__restrict__ out,
                                                                 unsigned long long cap, int chunk,
                                                                 unsigned long long *__restrict__ vcount, int copies,
                                                                 unsigned long long *__restrict__ totals,
                                                                 unsigned long long *__restrict__ res,
                                                                 unsigned long long max_work) {
  extern __shared__ __align__(16) uint32_t s_bm[];
  __shared__ int4 s_rec[DC_WARPS][32];
  __shared__ uint32_t s_hits[DC_WARPS][32];
  __shared__ unsigned long long s_sum[2];
  if (direct_off(res, max_work)) return;
  int64_t first = 0, last = 0;
  if (g.m) {
    last = (int64_t)*g.m;
  } else {
    first = (int64_t)g.rp[g.row_begin];
    last = (int64_t)g.rp[g.row_end];
    if (blockIdx.x == 0 && threadIdx.x == 0) res[DX_M] = (unsigned long long)(last - first);
  }
  if (out && (unsigned long long)(last - first) > cap) return;  // the host reports it
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t *bm = s_bm + w * WORDS, *hits = s_hits[w];
  int4 *rec = s_rec[w];
  if (MODE == 1) vcount += (int64_t)(((int64_t)blockIdx.x * DC_WARPS + w) % copies) * g.n;
  for (int q = lane; q < WORDS; q += 32) bm[q] = 0u;
  if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
  __syncthreads();
  const int32_t *__restrict__ col = g.col;
  const uintptr_t col_blk = reinterpret_cast<uintptr_t>(col) >> 4;
  unsigned long long acc = 0, alg = 0;
  int32_t cur = -1;  // batch: the graph acc belongs to
  const int64_t batches = (last - first + 31) / 32, warps = (int64_t)gridDim.x * DC_WARPS;
  for (int64_t c0 = ((int64_t)blockIdx.x * DC_WARPS + w) * chunk; c0 < batches; c0 += warps * chunk) {
    for (int64_t bt = c0; bt < min(batches, c0 + chunk); ++bt) {
      const int64_t e = first + bt * 32 + lane;
      const bool in = e < last;
      const int32_t u = in ? g.src[e] : -1, v = in ? col[e] : 0;
      int64_t a0 = 0, b0 = 0;
      int na = 0, nb = 0;
      if (in) {
        a0 = (int64_t)g.rp[u];
        na = (int)((int64_t)g.rp[u + 1] - a0);
        b0 = (int64_t)g.rp[v];
        nb = (int)((int64_t)g.rp[v + 1] - b0);
        alg += 4ull * (unsigned long long)(na + (int64_t)nb) + 4ull;
      }
      int32_t gid = -1;
      bool mixed = false;  // batch: the edges belong to several graphs
      if (g.vgroup) {
        gid = in ? g.vgroup[u] : -1;
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
      }
      const bool pe = out != nullptr || MODE == 1 || mixed;  // hits summed per edge
      hits[lane] = 0u;
      const int32_t up = __shfl_up_sync(TC_FULL_MASK, u, 1);
      unsigned hm = __ballot_sync(TC_FULL_MASK, in && (lane == 0 || u != up));  // first edge of each row
      const bool live = in && na > 1 && nb > 0;  // a row of one entry closes nothing
      const bool search = live && (__popc(hm) > DC_RUNS || nb / DC_SEARCH > na);
      const bool stream = live && !search;

      if (__any_sync(TC_FULL_MASK, search)) {
        const bool a_short = na <= nb;
        const int ns = search ? (a_short ? na : nb) : 0;
        int incl = ns;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(TC_FULL_MASK, incl, o);
          if (lane >= o) incl += y;
        }
        const int tot = __shfl_sync(TC_FULL_MASK, incl, 31);
        const int64_t ks = (a_short ? a0 : b0) - (incl - ns), ls = a_short ? b0 : a0;
        rec[lane] = make_int4(incl, (int)(uint32_t)ks, (int)(uint32_t)ls, a_short ? nb : na);
        __syncwarp();
        int c = 0;
        int4 r = rec[0];
        for (int i0 = 0; i0 < tot; i0 += 32 * DC_U) {
          int32_t key[DC_U];
          uint32_t lo[DC_U], hi[DC_U], end[DC_U];
          int ce[DC_U], width = 0;
#pragma unroll
          for (int j = 0; j < DC_U; ++j) {
            const int i = i0 + 32 * j + lane;
            key[j] = 0;
            lo[j] = hi[j] = end[j] = 0;
            if (i < tot) {
              while (i >= r.x) r = rec[++c];  // ends: rec[31].x == tot > i
              key[j] = __ldg(col + (uint32_t)((uint32_t)r.y + (uint32_t)i));
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

      if (__any_sync(TC_FULL_MASK, stream)) {
        while (hm) {
          const int h = __ffs(hm) - 1;
          hm &= hm - 1;
          const bool mine = stream && lane >= h && (hm == 0 || lane < __ffs(hm) - 1);
          const unsigned rm = __ballot_sync(TC_FULL_MASK, mine);
          if (!rm) continue;
          const int64_t ra = __shfl_sync(TC_FULL_MASK, a0, h);
          const int rn = __shfl_sync(TC_FULL_MASK, na, h);
          int64_t size = g.n;  // ids of the row's graph span at most this much
          if (g.vgroup) {
            const int32_t rg = __shfl_sync(TC_FULL_MASK, gid, h);
            size = g.vtx_off[rg + 1] - g.vtx_off[rg];
          }
          const bool exact = size <= WORDS * 32;
          for (int q = lane; q < rn; q += 32) {
            const uint32_t x = (uint32_t)__ldg(col + ra + q);
            atomicOr(bm + ((x >> 5) & (WORDS - 1)), 1u << (x & 31));
          }
          // the targets' lists in 16-byte groups, each list widened to the
          // aligned blocks that hold it (a block with a valid entry lies in
          // that entry's page); a record is (groups before and with the edge,
          // first and one past the last valid entry, block of group 0)
          const uintptr_t B = reinterpret_cast<uintptr_t>(col + b0);
          const int off = mine ? (int)((B >> 2) & 3u) : 0, ng = mine ? (off + nb + 3) >> 2 : 0;
          int incl = ng;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(TC_FULL_MASK, incl, o);
            if (lane >= o) incl += y;
          }
          const int tot = __shfl_sync(TC_FULL_MASK, incl, 31), excl = incl - ng;
          rec[lane] = make_int4(incl, 4 * excl + off, 4 * excl + off + nb, (int)((B >> 4) - col_blk) - excl);
          __syncwarp();
          int c = 0, hc = 0;
          uint32_t hit_n = 0;
          int4 r = rec[0];
          for (int i0 = 0; i0 < tot; i0 += 32 * DC_GU) {
            int4 q[DC_GU];
            int lo[DC_GU], hi[DC_GU], ce[DC_GU];
#pragma unroll
            for (int j = 0; j < DC_GU; ++j) {
              const int i = i0 + 32 * j + lane;
              q[j] = make_int4(0, 0, 0, 0);
              lo[j] = hi[j] = 0;
              if (i < tot) {
                while (i >= r.x) r = rec[++c];  // ends: rec[31].x == tot > i
                q[j] = __ldg(reinterpret_cast<const int4 *>((col_blk + (uintptr_t)(r.w + i)) << 4));
                lo[j] = r.y - 4 * i;
                hi[j] = r.z - 4 * i;
              }
              ce[j] = c;
            }
#pragma unroll
            for (int j = 0; j < DC_GU; ++j) {
              if (pe && ce[j] != hc) {
                if (hit_n) atomicAdd(hits + hc, hit_n);
                hc = ce[j];
                hit_n = 0;
              }
              const int32_t xs[4] = {q[j].x, q[j].y, q[j].z, q[j].w};
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                if (t < lo[j] || t >= hi[j]) continue;
                const uint32_t x = (uint32_t)xs[t];
                if (!((bm[(x >> 5) & (WORDS - 1)] >> (x & 31)) & 1u)) continue;
                if (!exact) {
                  int l = 0, h2 = rn;
                  while (l < h2) {
                    const int mid = (l + h2) >> 1;
                    if (__ldg(col + ra + mid) < (int32_t)x) l = mid + 1;
                    else h2 = mid;
                  }
                  if (l == rn || __ldg(col + ra + l) != (int32_t)x) continue;
                }
                if (MODE == 2 && (int)g.label[x] != g.want) continue;
                if (MODE == 1) atomicAdd(vcount + x, 1ull);
                ++hit_n;
              }
            }
          }
          if (!pe) acc += hit_n;
          else if (hit_n) atomicAdd(hits + hc, hit_n);
          __syncwarp();
          if (rn > 128) {
            uint4 *b4 = reinterpret_cast<uint4 *>(bm);
            for (int q = lane; q < WORDS / 4; q += 32) b4[q] = make_uint4(0u, 0u, 0u, 0u);
          } else {
            for (int q = lane; q < rn; q += 32) bm[((uint32_t)__ldg(col + ra + q) >> 5) & (WORDS - 1)] = 0u;
          }
          __syncwarp();
        }
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
    if (alg) atomicAdd(&s_sum[1], alg);
  }
  __syncthreads();
  if (threadIdx.x < 2 && s_sum[threadIdx.x]) atomicAdd(res + (threadIdx.x ? DX_ALG : DX_TOTAL), s_sum[threadIdx.x]);
}

// Sums the copies of the vertex counts.
__global__ void __launch_bounds__(DC_THREADS) direct_vsum_kernel(const unsigned long long *__restrict__ t, int64_t n,
                                                                int copies, unsigned long long *__restrict__ out,
                                                                const unsigned long long *__restrict__ res,
                                                                unsigned long long max_work) {
  if (direct_off(res, max_work)) return;
  for (int64_t u = (int64_t)blockIdx.x * DC_THREADS + threadIdx.x; u < n; u += (int64_t)gridDim.x * DC_THREADS) {
    unsigned long long s = 0;
    for (int c = 0; c < copies; ++c) s += t[c * n + u];
    out[u] = s;
  }
}

// ---- host side ---------------------------------------------------------------------

// Which calls count directly.  Measured against the general path (us, one
// call, whole-GPU clock; W = summed list lengths, see direct_rows_kernel):
//   ER n = 300, 1.5 K entries       297 ->  57    ER n = 16384, degree 16  350 ->  69
//   R-MAT scale 15, 0.9 M entries   940 -> 156    Chung-Lu n = 50000       974 -> 171
//   R-MAT scale 16, degree 64, W = 0.50 G        1865 -> 649
//   complete graph of 1500 vertices, W = 1.7 G    793 -> 835
// Beyond 65536 vertices hits are confirmed by searches and pay less:
//   R-MAT scale 18 of flat skew, W = 0.25 G 2383 -> 826; scale 17, W = 0.42 G 1848 -> 1494;
//   scale 18, W = 1.1 G 2394 -> 3622; ER of 16 M entries 1361 -> 1150.
// So entries are bounded by what the unsorted order costs, and W, which skew
// drives and only the device knows, by a limit: past it the kernels return at
// once and the general path counts.  Per-vertex counts pay
// an atomic per triangle (scale 16, degree 64: 2010 -> 903; complete graph of
// 1500: 3161 -> 4250; a 700-clique among 10^6 vertices, W = 0.17 G, 1245 ->
// 3856) and have the lower limits.
constexpr int64_t DIRECT_MAX_NNZ = int64_t(1) << 23;
constexpr int64_t DIRECT_MAX_N = int64_t(1) << 22;

static unsigned long long direct_max_work(int64_t n, bool per_vertex) {
  const bool exact = n <= 32 * DC_WORDS_MAX;
  if (per_vertex) return exact ? 1ull << 29 : 1ull << 27;
  return exact ? 1ull << 30 : 3ull << 27;
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

template <int MODE, typename RP, int WORDS>
static tc_status launch_count_w(tc_ctx *ctx, const DirectDag<RP> &g, int64_t edges, const DirectReq &rq,
                                unsigned long long *vcount, int copies, unsigned long long *res,
                                unsigned long long max_work) {
  constexpr int smem = DC_WARPS * WORDS * (int)sizeof(uint32_t);
  if (smem > 24 * 1024)  // with the static part above the 48 KB default
    TC_CHECK_CUDA(ctx, cudaFuncSetAttribute(direct_count_kernel<MODE, RP, WORDS>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int64_t batches = std::max<int64_t>(1, (edges + 31) / 32);
  direct_count_kernel<MODE, RP, WORDS><<<grid_for(ctx, batches, DC_WARPS, 8), DC_THREADS, smem, ctx->stream>>>(
      g, rq.edge_counts, (unsigned long long)rq.cap, 1, vcount, copies, nullptr, res, max_work);
  TC_CHECK_LAUNCH(ctx);
  return TC_OK;
}

template <int MODE, typename RP>
static tc_status launch_count(tc_ctx *ctx, const DirectDag<RP> &g, int64_t edges, const DirectReq &rq,
                              unsigned long long *vcount, int copies, unsigned long long *res,
                              unsigned long long max_work) {
  if (g.n <= 32 * DC_WORDS_MIN)
    return launch_count_w<MODE, RP, DC_WORDS_MIN>(ctx, g, edges, rq, vcount, copies, res, max_work);
  if (g.n <= 32 * DC_WORDS_MIN * 2)
    return launch_count_w<MODE, RP, DC_WORDS_MIN * 2>(ctx, g, edges, rq, vcount, copies, res, max_work);
  if (g.n <= 32 * DC_WORDS_MAX) return launch_count_w<MODE, RP, DC_WORDS_MAX>(ctx, g, edges, rq, vcount, copies, res, max_work);
  return launch_count_w<MODE, RP, DC_WORDS_MIN>(ctx, g, edges, rq, vcount, copies, res, max_work);
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
  const unsigned long long max_work = direct_max_work(n, rq.vertex_counts != nullptr);
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
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[1], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaMemsetAsync(res, 0, sizeof(unsigned long long) * DX_WORDS, ctx->stream));
  if (nnz >= DS_MIN_NNZ) {
    constexpr int blocks = DS_WARPS / (DR_THREADS / 32);
    if (rq.orient) direct_sample_kernel<true><<<blocks, DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz, res + DX_GUESS);
    else direct_sample_kernel<false><<<blocks, DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz, res + DX_GUESS);
    TC_CHECK_LAUNCH(ctx);
    TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], res + DX_GUESS, sizeof(unsigned long long),
                                       cudaMemcpyDeviceToHost, ctx->stream));
    TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (ctx->h_pinned[0] > max_work) {
      *declined = true;
      return TC_OK;
    }
  }
  if (rq.vertex_counts)
    TC_CHECK_CUDA(ctx, cudaMemsetAsync(vcount, 0, sizeof(unsigned long long) * (size_t)(n * copies), ctx->stream));
  if (rq.orient) {
    direct_rows_kernel<true><<<B, DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz, nullptr, nullptr, ku, kv, mask,
                                                               gpre, bsum, res);
    TC_CHECK_LAUNCH(ctx);
    if (B > DR_SMEM_BLOCKS) {  // too many block sums for a block to scan
      TC_CHECK_CUDA(ctx, cudaMemsetAsync(bsum + B, 0, sizeof(uint32_t), ctx->stream));
      TC_TRY(exclusive_scan_u32(ctx, bsum, boff, B + 1, scratch));
    }
    direct_place_kernel<<<B, DR_THREADS, 0, ctx->stream>>>(d.rowptr, n, nnz, B, bsum,
                                                           B > DR_SMEM_BLOCKS ? boff : nullptr, mask, gpre, ku, kv, src,
                                                           col, drow, res, max_work);
    TC_CHECK_LAUNCH(ctx);
  } else {
    direct_rows_kernel<false><<<B, DR_THREADS, 0, ctx->stream>>>(d.rowptr, d.col, n, nnz, nullptr, nullptr, ku, nullptr,
                                                                nullptr, nullptr, nullptr, res);
    TC_CHECK_LAUNCH(ctx);
  }
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[5], ctx->stream));
  if (rq.orient) {
    const DirectDag<uint32_t> g{drow, col, src, n, 0, n, res + DX_M, nullptr, nullptr, rq.labels, rq.label};
    if (rq.vertex_counts) TC_TRY((launch_count<1>(ctx, g, nnz / 2, rq, vcount, copies, res, max_work)));
    else if (rq.labels) TC_TRY((launch_count<2>(ctx, g, nnz / 2, rq, nullptr, 1, res, max_work)));
    else TC_TRY((launch_count<0>(ctx, g, nnz / 2, rq, nullptr, 1, res, max_work)));
    if (copies > 1) {
      direct_vsum_kernel<<<grid_for(ctx, n, DC_THREADS, 8), DC_THREADS, 0, ctx->stream>>>(vcount, n, copies,
                                                                                         rq.vertex_counts, res,
                                                                                         max_work);
      TC_CHECK_LAUNCH(ctx);
    }
  } else {
    const DirectDag<int64_t> g{d.rowptr, d.col, ku, n, rq.row_begin, rq.row_end, nullptr, nullptr, nullptr, nullptr, 0};
    TC_TRY((launch_count<0>(ctx, g, nnz, rq, nullptr, 1, res, max_work)));
  }
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[6], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], res, sizeof(unsigned long long) * DX_WORDS,
                                     cudaMemcpyDeviceToHost, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaEventRecord(ctx->ev[7], ctx->stream));
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const unsigned long long *h = ctx->h_pinned;
  if (const unsigned f = (unsigned)h[DX_FLAGS]) return set_error(ctx, TC_ERR_INVALID_GRAPH, "%s", flag_text(f));
  if (h[DX_WORK] > max_work) {
    *declined = true;
    return TC_OK;
  }
  const int64_t m = (int64_t)h[DX_M];
  if (rq.edge_counts && rq.cap < m)
    return set_error(ctx, TC_ERR_INVALID_ARG, "edge_counts holds %lld entries, %lld oriented edges", (long long)rq.cap,
                     (long long)m);
  if (rq.vertex_host)
    TC_CHECK_CUDA(ctx, cudaMemcpy(rq.vertex_host, rq.vertex_counts, sizeof(uint64_t) * (size_t)n, cudaMemcpyDeviceToHost));
  if (rq.edge_host && m > 0)
    TC_CHECK_CUDA(ctx, cudaMemcpy(rq.edge_host, rq.edge_counts, sizeof(uint32_t) * (size_t)m, cudaMemcpyDeviceToHost));
  st->m = m;
  st->tiles = (m + TILE_EDGES - 1) / TILE_EDGES;
  st->tiles_per_arm[TC_ARM_FLAT] = st->tiles;  // 32 edges' lists as one flattened run, as that arm
  st->alg_bytes_arm[TC_ARM_FLAT] = st->alg_bytes = h[DX_ALG];
  st->ms_h2d = elapsed(ctx->ev[0], ctx->ev[1]);
  st->ms_orient = elapsed(ctx->ev[1], ctx->ev[5]);
  st->ms_arm[TC_ARM_FLAT] = st->ms_count = elapsed(ctx->ev[5], ctx->ev[6]);
  st->ms_d2h = elapsed(ctx->ev[6], ctx->ev[7]);
  st->ms_total = elapsed(ctx->ev[0], ctx->ev[7]);
  st->d2h_bytes += sizeof(unsigned long long) + (rq.edge_host ? sizeof(uint32_t) * (size_t)m : 0) +
                   (rq.vertex_host ? sizeof(uint64_t) * (size_t)n : 0);
  st->kernel_launches = ctx->launches;
  return TC_OK;
}

}  // namespace tc
