// Device-side graph construction: seeded edge generators (bit-identical to
// the host generators) and the symmetric CSR builder (symmetrise, drop self
// loops, sort, dedup) that turns edge samples into the clean GraphMiner-style
// CSR the counting path expects.
#include <algorithm>
#include <vector>

#include "engine.cuh"
#include "tc_gen_common.h"

using namespace tc;

namespace tc {

__global__ void gen_er_kernel(uint64_t key, uint64_t n, int64_t M, int32_t *src, int32_t *dst) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x)
    tc_er_sample(key, n, (uint64_t)i, &src[i], &dst[i]);
}

__global__ void gen_rmat_kernel(uint64_t key, int scale, uint64_t t1, uint64_t t2, uint64_t t3, int64_t M,
                                int32_t *src, int32_t *dst) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x)
    tc_rmat_sample(key, scale, t1, t2, t3, (uint64_t)i, &src[i], &dst[i]);
}

__global__ void gen_cl_kernel(uint64_t key, const uint64_t *cum, int64_t n, int64_t M, int32_t *src, int32_t *dst) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x)
    tc_cl_sample(key, cum, n, (uint64_t)i, &src[i], &dst[i]);
}

// Two directed keys per undirected sample, or one (min, max) key (HALF);
// self loops and bad ids become the all-ones sentinel, which sorts after
// every real key.
template <bool HALF>
__global__ void edge_keys_kernel(const int32_t *__restrict__ src, const int32_t *__restrict__ dst, int64_t M,
                                 int64_t n, int bits, uint64_t *__restrict__ keys) {
  begin_pass();
  const uint64_t sentinel = (bits >= 32) ? ~0ULL : ((1ULL << (2 * bits)) - 1);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t u = src[i], v = dst[i];
    const bool bad = u == v || u < 0 || v < 0 || (int64_t)u >= n || (int64_t)v >= n;
    if (HALF) {
      keys[i] = bad ? sentinel : ((uint64_t)min(u, v) << bits) | (uint64_t)max(u, v);
    } else {
      keys[2 * i] = bad ? sentinel : ((uint64_t)u << bits) | (uint64_t)v;
      keys[2 * i + 1] = bad ? sentinel : ((uint64_t)v << bits) | (uint64_t)u;
    }
  }
}

// Long lists (half_keys): the edges as (min, max) keys sort and lose their duplicates at
// half the size of the directed list; a second, stable sort by max gives every
// vertex its smaller neighbours in order.  Row w of the CSR is its smaller
// neighbours (from the second order), then its larger ones (from the first):
// both parts are ascending, and an entry's slot is its position plus one row
// offset, so nothing is counted with atomics or scattered at random.
// R-MAT scale 21 (33.6 M samples): 9.35 -> 2.49 ms.  Short lists pay more for the
// launches of the second sort than half of the keys save, and where vertices
// outnumber the samples every vertex's two row starts are searched for, which
// the scan of the degrees beats.  Random lists, us, half keys against directed ones:
// 2^20 samples, n = 2^16 184, 202, 2^19 215, 213, 2^21 281, 249, 2^24 790, 400;
// 2^22 samples, n = 2^20 435, 541, 2^22 573, 620, 2^23 746, 665, 2^27 5458, 1890;
// 2^19 samples, n = 2^15 149, 139; 2^18 samples, n = 2^14 131, 112, 2^27 4089, 1255.
constexpr int64_t HALF_MIN_SAMPLES = int64_t(1) << 20;
static bool half_keys(int64_t n, int64_t M) { return M >= HALF_MIN_SAMPLES && n <= M; }
constexpr int UQ_THREADS = 256;
constexpr int UQ_PER = 8;
constexpr int UQ_TILE = UQ_THREADS * UQ_PER;

// Distinct keys of each tile (WRITE: to their place; off: the tiles' offsets).
// Keys are sorted; the sentinel is not one.
template <bool WRITE>
__global__ void __launch_bounds__(UQ_THREADS) unique_kernel(const uint64_t *keys, int64_t N,
                                                           uint64_t sentinel, uint32_t *__restrict__ cnt,
                                                           const uint32_t *off,
                                                           uint64_t *__restrict__ out) {
  begin_pass();
  __shared__ uint32_t s_w[UQ_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t w0 = (int64_t)blockIdx.x * UQ_TILE + warp * (32 * UQ_PER);
  uint64_t k[UQ_PER];
  unsigned bal[UQ_PER];
  uint32_t c = 0;
#pragma unroll
  for (int j = 0; j < UQ_PER; ++j) k[j] = w0 + 32 * j + lane < N ? keys[w0 + 32 * j + lane] : sentinel;
  uint64_t last = w0 > 0 && w0 < N ? keys[w0 - 1] : sentinel;
#pragma unroll
  for (int j = 0; j < UQ_PER; ++j) {
    uint64_t prev = __shfl_up_sync(TC_FULL_MASK, k[j], 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(TC_FULL_MASK, k[j], 31);
    bal[j] = __ballot_sync(TC_FULL_MASK, k[j] != sentinel && k[j] != prev);
    c += __popc(bal[j]);
  }
  if (lane == 0) s_w[warp] = c;
  __syncthreads();
  uint32_t at = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < UQ_THREADS / 32; ++w) {
    at += w < warp ? s_w[w] : 0u;
    tot += s_w[w];
  }
  if (!WRITE) {
    if (threadIdx.x == 0) cnt[blockIdx.x] = tot;
    return;
  }
  at += off[blockIdx.x];
#pragma unroll
  for (int j = 0; j < UQ_PER; ++j) {
    if ((bal[j] >> lane) & 1u) out[at + __popc(bal[j] & lanemask_lt())] = k[j];
    at += __popc(bal[j]);
  }
}

// start[r] = first of the E keys whose field (key >> shift) & mask is >= r, r in [0, n].
__global__ void field_start_kernel(const uint64_t *__restrict__ keys, int64_t E, int shift, uint64_t mask, int64_t n,
                                   uint32_t *__restrict__ start) {
  begin_pass();
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= n; r += (int64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = (uint32_t)E;
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (((keys[mid] >> shift) & mask) < (uint64_t)r) lo = mid + 1;
      else hi = mid;
    }
    start[r] = lo;
  }
}

// The entries of one order: key i's row is its field at row_shift, its
// neighbour the other field, its slot i + shift_by[row + add].
__global__ void half_rows_kernel(const uint64_t *__restrict__ keys, int64_t E, int bits, int row_shift,
                                 const uint32_t *__restrict__ shift_by, int add, int32_t *__restrict__ col) {
  begin_pass();
  const uint64_t mask = (1ULL << bits) - 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < E; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    const uint32_t row = (uint32_t)((k >> row_shift) & mask);
    col[i + (int64_t)shift_by[row + add]] = (int32_t)((k >> (bits - row_shift)) & mask);
  }
}

__global__ void add_starts_kernel(const uint32_t *__restrict__ a, const uint32_t *__restrict__ b, int64_t n,
                                  int64_t *__restrict__ rowptr) {
  begin_pass();
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= n; r += (int64_t)gridDim.x * blockDim.x)
    rowptr[r] = (int64_t)a[r] + (int64_t)b[r];
}

__global__ void unique_flag_kernel(const uint64_t *__restrict__ keys, int64_t N, uint64_t sentinel,
                                   int64_t *__restrict__ flag) {
  begin_pass();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    flag[i] = (k != sentinel && (i == 0 || keys[i - 1] != k)) ? 1 : 0;
  }
}

__global__ void unique_scatter_kernel(const uint64_t *__restrict__ keys, const int64_t *__restrict__ pos, int64_t N,
                                      uint64_t sentinel, int bits, int32_t *__restrict__ col,
                                      unsigned long long *__restrict__ deg) {
  begin_pass();
  const uint64_t mask = (1ULL << bits) - 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i];
    if (k != sentinel && (i == 0 || keys[i - 1] != k)) {
      col[pos[i]] = (int32_t)(k & mask);
      atomicAdd(&deg[k >> bits], 1ULL);
    }
  }
}

}  // namespace tc

extern "C" {

tc_status tc_gen_edges_device(tc_ctx *ctx, const tc_gen_params *p, int32_t *src, int32_t *dst, int64_t capacity,
                              int64_t *count_out) {
  if (!ctx || !p || !count_out) return set_error(ctx, TC_ERR_INVALID_ARG, "null argument");
  if (p->kind == TC_GEN_RGG) return set_error(ctx, TC_ERR_UNSUPPORTED, "RGG is generated on the host only");
  const int64_t M = tc_gen_num_samples(p);
  if (M < 0) return set_error(ctx, TC_ERR_INVALID_ARG, "%s", global_error());
  *count_out = M;
  if (!src || !dst || M > capacity)
    return set_error(ctx, TC_ERR_INVALID_ARG, "edge buffers hold %lld samples, %lld needed", (long long)capacity,
                     (long long)M);
  TC_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  const int grid = ctx->num_sms * 8;
  if (p->kind == TC_GEN_ER) {
    if (p->n < 1 || p->n > 2147483647LL) return set_error(ctx, TC_ERR_INVALID_ARG, "bad n");
    gen_er_kernel<<<grid, 256, 0, ctx->stream>>>(tc_stream_key(p->seed, TC_SID_ER), (uint64_t)p->n, M, src, dst);
  } else if (p->kind == TC_GEN_RMAT) {
    if (p->scale < 1 || p->scale > 30) return set_error(ctx, TC_ERR_INVALID_ARG, "bad RMAT scale");
    uint64_t t1, t2, t3;
    rmat_thresholds(p->a, p->b, p->c, &t1, &t2, &t3);
    gen_rmat_kernel<<<grid, 256, 0, ctx->stream>>>(tc_stream_key(p->seed, TC_SID_RMAT), p->scale, t1, t2, t3, M, src,
                                                   dst);
  } else if (p->kind == TC_GEN_CHUNG_LU) {
    if (p->n < 1 || p->n > 2147483647LL || !(p->gamma > 1.0)) return set_error(ctx, TC_ERR_INVALID_ARG, "bad CL");
    std::vector<uint64_t> cum((size_t)p->n);
    chung_lu_table(p->n, p->avg_degree, p->gamma, cum.data());
    TC_TRY(arena_reserve(ctx, sizeof(uint64_t) * (size_t)p->n));
    uint64_t *d_cum = (uint64_t *)ctx->arena;
    TC_CHECK_CUDA(ctx, cudaMemcpyAsync(d_cum, cum.data(), sizeof(uint64_t) * (size_t)p->n, cudaMemcpyHostToDevice,
                                       ctx->stream));
    gen_cl_kernel<<<grid, 256, 0, ctx->stream>>>(tc_stream_key(p->seed, TC_SID_CL), d_cum, p->n, M, src, dst);
    TC_CHECK_CUDA(ctx, cudaGetLastError());
    TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // cum is read from pageable memory above
    return TC_OK;
  } else {
    return set_error(ctx, TC_ERR_INVALID_ARG, "unknown generator %d", p->kind);
  }
  TC_CHECK_CUDA(ctx, cudaGetLastError());
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TC_OK;
}

tc_status tc_csr_from_edges(tc_ctx *ctx, int64_t n, int64_t M, const int32_t *src, const int32_t *dst,
                            int32_t on_device, int64_t *rowptr, int32_t *colidx, int64_t capacity, int64_t *nnz_out) {
  if (!ctx || !rowptr || !nnz_out || (M > 0 && (!src || !dst)) || M < 0)
    return set_error(ctx, TC_ERR_INVALID_ARG, "null argument");
  if (n < 1 || n > 2147483647LL) return set_error(ctx, TC_ERR_UNSUPPORTED, "n outside [1, 2^31-1]");
  if (2 * M >= (int64_t(1) << 32)) return set_error(ctx, TC_ERR_UNSUPPORTED, "too many edge samples");
  TC_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  const int bits = bit_width_u64(n > 1 ? (uint64_t)(n - 1) : 1);
  const uint64_t sentinel = (1ULL << (2 * bits)) - 1;
  const bool half = half_keys(n, M);
  const int64_t N = half ? M : 2 * M;  // keys
  const int64_t tiles = (N + UQ_TILE - 1) / UQ_TILE;
  const size_t scratch_bytes =
      std::max(radix_sort_scratch_bytes(ctx, std::max<int64_t>(N, 1)),
               scan_scratch_bytes(ctx, half ? tiles + 1 : std::max<int64_t>(N, n + 1)));
  Sizer sz;
  if (!on_device) { sz.take<int32_t>(M); sz.take<int32_t>(M); }
  sz.take<uint64_t>(N); sz.take<uint64_t>(N);
  if (half) {
    sz.take<uint64_t>(N);
    sz.take<uint32_t>(tiles + 1); sz.take<uint32_t>(n + 1); sz.take<uint32_t>(n + 1);
  } else {
    sz.take<int64_t>(N); sz.take<int64_t>(n + 1);
  }
  sz.take<char>((int64_t)scratch_bytes);
  if (!on_device) { sz.take<int64_t>(n + 1); sz.take<int32_t>(2 * M); }
  TC_TRY(arena_reserve(ctx, sz.used));
  Bump bump{ctx->arena, ctx->arena_cap};
  const int32_t *dsrc = src, *ddst = dst;
  if (!on_device) {
    int32_t *s = bump.take<int32_t>(M), *d = bump.take<int32_t>(M);
    if (M > 0) {
      TC_CHECK_CUDA(ctx, cudaMemcpyAsync(s, src, sizeof(int32_t) * M, cudaMemcpyHostToDevice, ctx->stream));
      TC_CHECK_CUDA(ctx, cudaMemcpyAsync(d, dst, sizeof(int32_t) * M, cudaMemcpyHostToDevice, ctx->stream));
    }
    dsrc = s;
    ddst = d;
  }
  uint64_t *k0 = bump.take<uint64_t>(N), *k1 = bump.take<uint64_t>(N);
  uint64_t *k2 = half ? bump.take<uint64_t>(N) : nullptr;
  uint32_t *tile_cnt = half ? bump.take<uint32_t>(tiles + 1) : nullptr;
  uint32_t *first = half ? bump.take<uint32_t>(n + 1) : nullptr, *second = half ? bump.take<uint32_t>(n + 1) : nullptr;
  int64_t *flag = half ? nullptr : bump.take<int64_t>(N);
  int64_t *deg = half ? nullptr : bump.take<int64_t>(n + 1);
  void *scratch = bump.take<char>((int64_t)scratch_bytes);
  int64_t *drow = on_device ? rowptr : bump.take<int64_t>(n + 1);
  int32_t *dcol_stage = on_device ? nullptr : bump.take<int32_t>(2 * M);
  if (bump.overflow) return set_error(ctx, TC_ERR_OOM, "arena overflow");
  if (!half) TC_CHECK_CUDA(ctx, cudaMemsetAsync(deg, 0, sizeof(int64_t) * (size_t)(n + 1), ctx->stream));
  int64_t nnz = 0;
  if (M > 0) {
    uint64_t *sk = nullptr;
    if (half) {
      TC_CHECK_CUDA(ctx, launch_pass(ctx, edge_keys_kernel<true>, grid_for(ctx, M, 256, 8), 256, 0, dsrc, ddst, M, n,
                                     bits, k0));
      TC_TRY(radix_sort(ctx, k0, k1, k0, N, 0, 2 * bits, scratch, &sk));
      TC_CHECK_CUDA(ctx, launch_pass(ctx, unique_kernel<false>, (unsigned)tiles, UQ_THREADS, 0, sk, N, sentinel,
                                     tile_cnt, nullptr, nullptr));
      TC_CHECK_CUDA(ctx, cudaMemsetAsync(tile_cnt + tiles, 0, sizeof(uint32_t), ctx->stream));
      TC_TRY(exclusive_scan_u32(ctx, tile_cnt, tile_cnt, tiles + 1, scratch));
      ctx->h_pinned[0] = 0;
      TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], tile_cnt + tiles, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                         ctx->stream));
    } else {
      TC_CHECK_CUDA(ctx, launch_pass(ctx, edge_keys_kernel<false>, grid_for(ctx, M, 256, 8), 256, 0, dsrc, ddst, M, n,
                                     bits, k0));
      TC_TRY(radix_sort(ctx, k0, k1, k0, N, 0, 2 * bits, scratch, &sk));
      TC_CHECK_CUDA(ctx, launch_pass(ctx, unique_flag_kernel, grid_for(ctx, N, 256, 8), 256, 0, sk, N, sentinel, flag));
      TC_TRY(exclusive_scan_i64(ctx, flag, flag, N, scratch, (int64_t *)&ctx->d_total[0]));
      TC_CHECK_CUDA(ctx, cudaMemcpyAsync(&ctx->h_pinned[0], ctx->d_total, sizeof(int64_t), cudaMemcpyDeviceToHost,
                                         ctx->stream));
    }
    TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int64_t E = (int64_t)ctx->h_pinned[0];
    nnz = half ? 2 * E : E;
    *nnz_out = nnz;
    if (nnz > capacity || !colidx)
      return set_error(ctx, TC_ERR_INVALID_ARG, "colidx holds %lld entries, %lld needed", (long long)capacity,
                       (long long)nnz);
    int32_t *dcol = on_device ? colidx : dcol_stage;
    if (half) {
      const uint64_t mask = (1ULL << bits) - 1;
      uint64_t *uk = sk == k0 ? k1 : k0, *bk = nullptr;
      TC_CHECK_CUDA(ctx, launch_pass(ctx, unique_kernel<true>, (unsigned)tiles, UQ_THREADS, 0, sk, N, sentinel,
                                     nullptr, tile_cnt, uk));
      TC_CHECK_CUDA(ctx, launch_pass(ctx, field_start_kernel, grid_for(ctx, n + 1, 256, 8), 256, 0, uk, E, bits, mask,
                                     n, first));
      TC_TRY(radix_sort(ctx, uk, sk, k2, E, 0, bits, scratch, &bk));
      TC_CHECK_CUDA(ctx, launch_pass(ctx, field_start_kernel, grid_for(ctx, n + 1, 256, 8), 256, 0, bk, E, 0, mask, n,
                                     second));
      if (E > 0) {
        TC_CHECK_CUDA(ctx, launch_pass(ctx, half_rows_kernel, grid_for(ctx, E, 256, 8), 256, 0, uk, E, bits, bits,
                                       second, 1, dcol));
        TC_CHECK_CUDA(ctx, launch_pass(ctx, half_rows_kernel, grid_for(ctx, E, 256, 8), 256, 0, bk, E, bits, 0, first,
                                       0, dcol));
      }
    } else {
      TC_CHECK_CUDA(ctx, launch_pass(ctx, unique_scatter_kernel, grid_for(ctx, N, 256, 8), 256, 0, sk, flag, N,
                                     sentinel, bits, dcol, (unsigned long long *)deg));
    }
    if (!on_device && nnz > 0)
      TC_CHECK_CUDA(ctx, cudaMemcpyAsync(colidx, dcol_stage, sizeof(int32_t) * nnz, cudaMemcpyDeviceToHost,
                                         ctx->stream));
  } else {
    *nnz_out = 0;
  }
  if (half) {
    TC_CHECK_CUDA(ctx, launch_pass(ctx, add_starts_kernel, grid_for(ctx, n + 1, 256, 8), 256, 0, first, second, n,
                                   drow));
  } else {
    TC_TRY(exclusive_scan_i64(ctx, deg, drow, n + 1, scratch, nullptr));
  }
  if (!on_device)
    TC_CHECK_CUDA(ctx, cudaMemcpyAsync(rowptr, drow, sizeof(int64_t) * (n + 1), cudaMemcpyDeviceToHost, ctx->stream));
  TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TC_OK;
}

}  // extern "C"

extern "C" tc_status tc_count_edges(tc_ctx *ctx, int64_t n, int64_t M, const int32_t *src, const int32_t *dst,
                                    int32_t on_device, const tc_opts *opts, uint64_t *total, tc_stats *stats) {
  if (!ctx || !total) return set_error(ctx, TC_ERR_INVALID_ARG, "null ctx or total");
  if (n < 1 || n > 2147483647LL || M < 0 || (M > 0 && (!src || !dst)))
    return set_error(ctx, TC_ERR_INVALID_ARG, "bad n or edge list");
  if (2 * M >= (int64_t(1) << 32)) return set_error(ctx, TC_ERR_UNSUPPORTED, "too many edge samples");
  TC_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  // the built CSR lives in ctx->aux: at most 2M entries
  const size_t need = align_up(sizeof(int64_t) * (size_t)(n + 1), 256) + align_up(sizeof(int32_t) * (size_t)(2 * M + 1), 256);
  if (need > ctx->aux_cap) {
    TC_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (ctx->aux) TC_CHECK_CUDA(ctx, cudaFree(ctx->aux));
    ctx->aux = nullptr;
    ctx->aux_cap = 0;
    cudaError_t e = cudaMalloc((void **)&ctx->aux, need);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return set_error(ctx, TC_ERR_OOM, "edge-list CSR buffer of %zu bytes: %s", need, cudaGetErrorString(e));
    }
    ctx->aux_cap = need;
  }
  int64_t *rowptr = (int64_t *)ctx->aux;
  int32_t *colidx = (int32_t *)(ctx->aux + align_up(sizeof(int64_t) * (size_t)(n + 1), 256));
  int64_t nnz = 0;
  TC_TRY(tc_csr_from_edges(ctx, n, M, src, dst, on_device, rowptr, colidx, 2 * M, &nnz));
  tc_csr g{n, nnz, rowptr, colidx, 1};
  return tc_count(ctx, &g, opts, total, nullptr, 0, stats);
}
