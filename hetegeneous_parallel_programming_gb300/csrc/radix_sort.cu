// Stable LSD radix sort of uint64 keys (digits of up to 8 bits) and an
// exclusive scan, both "reduce then scan" over a grid of contiguous per-block
// chunks so that no block ever waits on another.
//
// Per digit pass: (1) every block histograms its chunk, (2) one block per
// digit scans the blocks' counts into global offsets, (3) every block re-reads
// its chunk tile by tile, ranks the keys stably inside each warp, exchanges
// them through shared memory into digit order and writes them out, so a
// digit's keys leave as one run.  Stability: a block's chunk precedes the next
// block's chunk, warps own consecutive runs of a tile and lanes own
// consecutive keys of a round.
#include <stdarg.h>

#include <algorithm>

#include "dev_common.cuh"

namespace tc {

tc_status set_error(tc_ctx *ctx, tc_status st, const char *fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (ctx) snprintf(ctx->err, sizeof(ctx->err), "%s", buf);
  set_global_error("%s", buf);
  return st;
}

tc_status arena_reserve(tc_ctx *ctx, size_t bytes, size_t *keep) {
  ctx->arena_used = 0;
  if (bytes <= ctx->arena_cap) return TC_OK;
  size_t cap = align_up(bytes + bytes / 8, size_t(1) << 20);
  char *larger = nullptr;
  if (keep && *keep > 0) {
    if (cudaMalloc((void **)&larger, cap) == cudaSuccess) {
      const cudaError_t e = cudaMemcpyAsync(larger, ctx->arena, *keep, cudaMemcpyDeviceToDevice, ctx->stream);
      if (e != cudaSuccess) cudaFree(larger);
      TC_CHECK_CUDA(ctx, e);
    } else {
      (void)cudaGetLastError();
      larger = nullptr;
      *keep = 0;
    }
  }
  if (ctx->arena) {
    TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    TC_CHECK_CUDA(ctx, cudaFree(ctx->arena));
    ctx->arena = nullptr;
    ctx->arena_cap = 0;
  }
  if (larger) {
    ctx->arena = larger;
    ctx->arena_cap = cap;
    return TC_OK;
  }
  cudaError_t e = cudaMalloc((void **)&ctx->arena, cap);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    ctx->arena = nullptr;
    return set_error(ctx, TC_ERR_OOM, "device arena of %zu bytes: %s", cap, cudaGetErrorString(e));
  }
  ctx->arena_cap = cap;
  return TC_OK;
}

int grid_for(const tc_ctx *ctx, int64_t items, int per_block, int blocks_per_sm) {
  int64_t want = (items + per_block - 1) / per_block;
  int64_t cap = (int64_t)ctx->num_sms * blocks_per_sm;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return (int)want;
}

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_IPL = 10;                        // keys per lane per tile
constexpr int RS_TILE = RS_THREADS * RS_IPL;      // 2560 keys
constexpr int RS_BLOCKS_PER_SM = 4;
constexpr int RS_MAX_PASSES = 8;

struct RsGeom {
  int G;
  int64_t chunk;
};

static RsGeom rs_geom(const tc_ctx *ctx, int64_t N) {
  RsGeom g;
  int64_t tiles = (N + RS_TILE - 1) / RS_TILE;
  int64_t G = (int64_t)ctx->num_sms * RS_BLOCKS_PER_SM;
  if (G > tiles) G = tiles;
  if (G < 1) G = 1;
  int64_t tiles_per = (tiles + G - 1) / G;
  g.chunk = tiles_per * RS_TILE;
  g.G = (int)((N + g.chunk - 1) / g.chunk);
  if (g.G < 1) g.G = 1;
  return g;
}

// Scratch sizes hold for every N up to the one given: a smaller N can take
// more blocks (its chunks are smaller), up to one per tile or the grid's cap.
size_t radix_sort_scratch_bytes(const tc_ctx *ctx, int64_t N) {
  const int64_t G = std::max<int64_t>(
      1, std::min<int64_t>((N + RS_TILE - 1) / RS_TILE, (int64_t)ctx->num_sms * RS_BLOCKS_PER_SM));
  return align_up((size_t)256 * G * sizeof(uint32_t), 256) * 2 + RS_MAX_PASSES * 256 * sizeof(uint32_t);
}

// Digit counts of every block's chunk, [digit][block], and in all (`total`,
// zeroed by the caller).  Warp-private counters; 16-byte loads.
__global__ void __launch_bounds__(RS_THREADS) rs_hist_kernel(const uint64_t *__restrict__ keys, int64_t N, int shift,
                                                            unsigned dmask, int64_t chunk,
                                                            uint32_t *__restrict__ hist,
                                                            uint32_t *__restrict__ total, int G) {
  __shared__ uint32_t cnt[RS_WARPS][256];
  begin_pass();
  const int warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < RS_WARPS * 256; i += RS_THREADS) (&cnt[0][0])[i] = 0;
  __syncthreads();
  const int64_t b = (int64_t)blockIdx.x * chunk, e = min(N, b + chunk);  // b: a multiple of the tile
  const ulonglong2 *k2 = reinterpret_cast<const ulonglong2 *>(keys + b);
  const int64_t pairs = (e - b) / 2;
  constexpr int U = 4;
  for (int64_t i0 = threadIdx.x; i0 < pairs; i0 += U * RS_THREADS) {
    ulonglong2 k[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * RS_THREADS < pairs) k[u] = __ldg(k2 + i0 + u * RS_THREADS);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * RS_THREADS < pairs) {
        atomicAdd(&cnt[warp][(unsigned)(k[u].x >> shift) & dmask], 1u);
        atomicAdd(&cnt[warp][(unsigned)(k[u].y >> shift) & dmask], 1u);
      }
  }
  if (threadIdx.x == 0 && ((e - b) & 1)) atomicAdd(&cnt[0][(unsigned)(keys[e - 1] >> shift) & dmask], 1u);
  __syncthreads();
  for (int d = threadIdx.x; d <= (int)dmask; d += RS_THREADS) {
    uint32_t s = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) s += cnt[w][d];
    hist[(int64_t)d * G + blockIdx.x] = s;
    if (s) atomicAdd(total + d, s);
  }
}

// Digit offsets, block d for digit d: offs[d][b] = (keys with a smaller digit)
// + (keys with digit d in blocks before b).
__global__ void __launch_bounds__(RS_THREADS) rs_scan_kernel(const uint32_t *__restrict__ hist,
                                                            const uint32_t *total,
                                                            uint32_t *__restrict__ offs, int G) {
  __shared__ uint32_t tmp[33];
  begin_pass();
  const int d = blockIdx.x;
  uint32_t run;
  block_exclusive_scan<uint32_t>((int)threadIdx.x < d ? total[threadIdx.x] : 0u, tmp, &run);
  for (int b0 = 0; b0 < G; b0 += RS_THREADS) {
    const int b = b0 + threadIdx.x;
    const uint32_t c = b < G ? hist[(int64_t)d * G + b] : 0u;
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan<uint32_t>(c, tmp, &tot);
    if (b < G) offs[(int64_t)d * G + b] = run + ex;
    run += tot;
  }
}

// Places one digit's keys.  Lanes that hold the same digit find each other by
// one ballot per digit bit (a match instruction took 47 cycles a round); the
// warps' counts give each key its place in the tile, where the keys meet in
// shared memory, and the tile leaves digit by digit, 10 keys (80 bytes) a
// run on average.  16 bytes of memory per key plus 8 for the histogram; bound by
// issue and the barriers between a tile's steps (60 % of cycles issue; 2.5 TB/s
// of DRAM at 16.8 M keys).  33.6 M keys take 163 us, 3.3 TB/s (the direct scatter it
// replaces 460; 16 keys a lane with the ballots of a round after the counters of
// the one before 202), the histogram 46 us, 5.8 TB/s (172).  Keys a lane, by the
// time of a whole R-MAT scale 21 build at four blocks an SM: 10 2562 us, 12 2766,
// 14 at three 2639.  10 spills 8 bytes at that occupancy, 16 spilled 100.
__global__ void __launch_bounds__(RS_THREADS, RS_BLOCKS_PER_SM) rs_scatter_kernel(
    const uint64_t *__restrict__ kin, uint64_t *__restrict__ kout, int64_t N, int shift, int dbits, int64_t chunk,
    const uint32_t *offs, int G) {
  __shared__ uint64_t s_key[RS_TILE];
  __shared__ uint16_t s_cnt[RS_WARPS][256];
  __shared__ uint32_t s_base[256];   // where the tile's digit d goes, minus its start in the tile
  __shared__ uint32_t tmp[33];
  begin_pass();
  static_assert(RS_THREADS == 256, "one thread per digit");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d_own = threadIdx.x;
  const unsigned lt = lanemask_lt(), dmask = (1u << dbits) - 1u;
  uint32_t next = d_own <= (int)dmask ? offs[(int64_t)d_own * G + blockIdx.x] : 0u;  // digit d_own's next slot
  const int64_t b = (int64_t)blockIdx.x * chunk, e = min(N, b + chunk);
  for (int64_t t0 = b; t0 < e; t0 += RS_TILE) {
    const int nt = (int)min((int64_t)RS_TILE, e - t0);
    uint64_t k[RS_IPL];
    uint32_t r[RS_IPL];  // the lanes with the key's digit, then its rank in the warp
    const int base = warp * (32 * RS_IPL) + lane;
#pragma unroll
    for (int it = 0; it < RS_IPL; ++it) k[it] = base + it * 32 < nt ? kin[t0 + base + it * 32] : ~0ull;
    for (int i = threadIdx.x; i < RS_WARPS * 256 / 2; i += RS_THREADS) reinterpret_cast<uint32_t *>(&s_cnt[0][0])[i] = 0u;
    __syncthreads();
    // every round's ballots first: they do not depend on one another
#pragma unroll
    for (int it = 0; it < RS_IPL; ++it) {
      const bool in = base + it * 32 < nt;
      const unsigned d = (unsigned)(k[it] >> shift) & dmask, all = __ballot_sync(TC_FULL_MASK, in);
      r[it] = in ? all : ~all;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q >= dbits) break;
        const bool bit = (d >> q) & 1u;
        const unsigned bal = __ballot_sync(TC_FULL_MASK, bit);
        r[it] &= bit ? bal : ~bal;
      }
    }
#pragma unroll
    for (int it = 0; it < RS_IPL; ++it) {
      const unsigned d = (unsigned)(k[it] >> shift) & dmask, peers = r[it];
      const uint32_t before = s_cnt[warp][d];
      r[it] = before + __popc(peers & lt);
      __syncwarp();
      if (base + it * 32 < nt && (peers >> lane) == 1u)  // the last of them
        s_cnt[warp][d] = (uint16_t)(before + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    uint32_t c = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      const uint32_t x = s_cnt[w][d_own];
      s_cnt[w][d_own] = (uint16_t)c;
      c += x;
    }
    uint32_t tot;
    const uint32_t start = block_exclusive_scan<uint32_t>(c, tmp, &tot);
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) s_cnt[w][d_own] = (uint16_t)(s_cnt[w][d_own] + start);
    s_base[d_own] = next - start;
    next += c;
    __syncthreads();
#pragma unroll
    for (int it = 0; it < RS_IPL; ++it)
      if (base + it * 32 < nt) s_key[s_cnt[warp][(unsigned)(k[it] >> shift) & dmask] + r[it]] = k[it];
    __syncthreads();
    for (int i = threadIdx.x; i < nt; i += RS_THREADS) {
      const uint64_t x = s_key[i];
      kout[s_base[(unsigned)(x >> shift) & dmask] + (uint32_t)i] = x;
    }
    __syncthreads();
  }
}

tc_status radix_sort(tc_ctx *ctx, uint64_t *in, uint64_t *k0, uint64_t *k1, int64_t N, int begin_bit, int end_bit,
                     void *scratch, uint64_t **kres) {
  *kres = in;
  if (N <= 1 || end_bit <= begin_bit) return TC_OK;
  const RsGeom g = rs_geom(ctx, N);
  const size_t table = align_up((size_t)256 * g.G * sizeof(uint32_t), 256);
  uint32_t *hist = (uint32_t *)scratch, *offs = (uint32_t *)((char *)scratch + table);
  uint32_t *total = (uint32_t *)((char *)scratch + 2 * table);
  const int bits = end_bit - begin_bit, passes = (bits + 7) / 8;
  TC_CHECK_CUDA(ctx, cudaMemsetAsync(total, 0, (size_t)passes * 256 * sizeof(uint32_t), ctx->stream));
  uint64_t *ka = in, *kb = k0;
  for (int p = 0, shift = begin_bit; p < passes; ++p) {
    const int dbits = (bits - (shift - begin_bit) + passes - p - 1) / (passes - p);  // even digits: longer runs
    TC_CHECK_CUDA(ctx, launch_pass(ctx, rs_hist_kernel, g.G, RS_THREADS, 0, ka, N, shift, (1u << dbits) - 1u, g.chunk,
                                   hist, total + p * 256, g.G));
    TC_CHECK_CUDA(ctx, launch_pass(ctx, rs_scan_kernel, 1 << dbits, RS_THREADS, 0, hist, total + p * 256, offs,
                                   g.G));
    TC_CHECK_CUDA(ctx, launch_pass(ctx, rs_scatter_kernel, g.G, RS_THREADS, 0, ka, kb, N, shift, dbits, g.chunk,
                                   offs, g.G));
    shift += dbits;
    ka = kb;
    kb = ka == k0 ? k1 : k0;
  }
  *kres = ka;
  return TC_OK;
}

// ---- exclusive scan of int64 ------------------------------------------------------

constexpr int SC_THREADS = 256;
constexpr int SC_IPT = 8;
constexpr int SC_TILE = SC_THREADS * SC_IPT;
constexpr int SC_BLOCKS_PER_SM = 4;

static RsGeom sc_geom(const tc_ctx *ctx, int64_t N) {
  RsGeom g;
  int64_t tiles = (N + SC_TILE - 1) / SC_TILE;
  int64_t G = (int64_t)ctx->num_sms * SC_BLOCKS_PER_SM;
  if (G > tiles) G = tiles;
  if (G < 1) G = 1;
  g.chunk = ((tiles + G - 1) / G) * SC_TILE;
  g.G = (int)((N + g.chunk - 1) / g.chunk);
  if (g.G < 1) g.G = 1;
  return g;
}

size_t scan_scratch_bytes(const tc_ctx *ctx, int64_t N) {
  const int64_t G = std::max<int64_t>(
      1, std::min<int64_t>((N + SC_TILE - 1) / SC_TILE, (int64_t)ctx->num_sms * SC_BLOCKS_PER_SM));
  return align_up((size_t)(G + 1) * sizeof(int64_t), 256);
}

template <typename T>
__global__ void __launch_bounds__(SC_THREADS) sc_reduce_kernel(const T *__restrict__ in, int64_t N,
                                                              int64_t chunk, int64_t *__restrict__ sums) {
  __shared__ long long tmp[33];
  begin_pass();
  const int64_t b = (int64_t)blockIdx.x * chunk, e = min(N, b + chunk);
  long long s = 0;
  for (int64_t i = b + threadIdx.x; i < e; i += SC_THREADS) s += in[i];
  long long tot;
  block_exclusive_scan<long long>(s, tmp, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(1024) sc_top_kernel(int64_t *sums, int G, int64_t *d_total_out) {
  __shared__ long long tmp[33];
  begin_pass();
  // G <= 4 * SMs: at most a few items per thread
  const int per = (G + blockDim.x - 1) / blockDim.x;
  const int b = threadIdx.x * per, e = min(G, b + per);
  long long s = 0;
  for (int i = b; i < e; ++i) s += sums[i];
  long long tot;
  long long run = block_exclusive_scan<long long>(s, tmp, &tot);
  for (int i = b; i < e; ++i) {
    long long t = sums[i];
    sums[i] = run;
    run += t;
  }
  if (threadIdx.x == 0) {
    sums[G] = tot;
    if (d_total_out) *d_total_out = tot;
  }
}

template <typename T>
__global__ void __launch_bounds__(SC_THREADS) sc_down_kernel(const T *in, T *out, int64_t N,
                                                            int64_t chunk, const int64_t *sums) {
  __shared__ long long tmp[33];
  begin_pass();
  const int64_t b = (int64_t)blockIdx.x * chunk, e = min(N, b + chunk);
  long long carry = sums[blockIdx.x];
  for (int64_t t0 = b; t0 < e; t0 += SC_TILE) {
    long long x[SC_IPT];
    long long s = 0;
    const int64_t my = t0 + (int64_t)threadIdx.x * SC_IPT;
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) {
      x[k] = (my + k < e) ? in[my + k] : 0;
      s += x[k];
    }
    long long tot;
    long long run = carry + block_exclusive_scan<long long>(s, tmp, &tot);
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) {
      if (my + k < e) out[my + k] = (T)run;
      run += x[k];
    }
    carry += tot;
  }
}

tc_status exclusive_scan_i64(tc_ctx *ctx, const int64_t *in, int64_t *out, int64_t N, void *scratch,
                             int64_t *d_total_out) {
  if (N <= 0) return TC_OK;
  RsGeom g = sc_geom(ctx, N);
  int64_t *sums = (int64_t *)scratch;
  TC_CHECK_CUDA(ctx, launch_pass(ctx, sc_reduce_kernel<int64_t>, g.G, SC_THREADS, 0, in, N, g.chunk, sums));
  TC_CHECK_CUDA(ctx, launch_pass(ctx, sc_top_kernel, 1, 1024, 0, sums, g.G, d_total_out));
  TC_CHECK_CUDA(ctx, launch_pass(ctx, sc_down_kernel<int64_t>, g.G, SC_THREADS, 0, in, out, N, g.chunk, sums));
  return TC_OK;
}

tc_status exclusive_scan_u32(tc_ctx *ctx, const uint32_t *in, uint32_t *out, int64_t N, void *scratch) {
  if (N <= 0) return TC_OK;
  RsGeom g = sc_geom(ctx, N);
  int64_t *sums = (int64_t *)scratch;
  TC_CHECK_CUDA(ctx, launch_pass(ctx, sc_reduce_kernel<uint32_t>, g.G, SC_THREADS, 0, in, N, g.chunk, sums));
  TC_CHECK_CUDA(ctx, launch_pass(ctx, sc_top_kernel, 1, 1024, 0, sums, g.G, nullptr));
  TC_CHECK_CUDA(ctx, launch_pass(ctx, sc_down_kernel<uint32_t>, g.G, SC_THREADS, 0, in, out, N, g.chunk, sums));
  return TC_OK;
}

}  // namespace tc
