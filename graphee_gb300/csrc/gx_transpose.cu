// Out-edge CSR (push steps, selective marking) from the CSC: a counting sort
// by source in two passes over buckets of kBucket sources.
//
//  1. A CTA takes a batch of the engine's work units, counts its edges per
//     bucket in shared memory, reserves each bucket's run with one atomic and
//     writes (source within the bucket, destination[, weight]) there.  The
//     buckets' places are known: a bucket's edges are its sources' out-edges.
//  2. A CTA takes a slice of a bucket, counts its sources in shared memory,
//     reserves their places (with an atomic each where the bucket has several
//     slices) and writes the destinations into them; a slice's writes stay
//     within its bucket's part of the CSR, which L2 holds.
// The out-degrees are the caller's: that they count the edges is checked on the
// way (the buckets' next places at the end of the first pass, before its output
// is read, then every source's), and nothing is written outside the CSR.
// The order within a source is unspecified, which min-plus, min-label and
// marking do not observe.  One atomic and one random write per edge
// (transpose_kernel), with R-MAT's hubs drawing thousands of atomics to one
// address, took 65 ms for 263 M weighted edges and 18 for 128 M of a symmetric
// graph without weights; this takes 16 (7 and 9 for the passes) and 3.6.  What
// bounds it now are the second pass's 4-byte writes into L2.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "gx_engine.h"

using namespace gx;

namespace {

constexpr int kBucketBits = 14;                   // sources of a bucket: 64 KB of counters
constexpr int kBucket = 1 << kBucketBits;
constexpr int kMostBuckets = 8192;                // V up to 2^27: 96 KB of a CTA's counters and places
constexpr int kTrThreads = 512;
constexpr int64_t kTrSlice = 128 * 1024;          // edges of a slice
// One pass of transpose_kernel takes less than the two passes' allocations and
// wait (some 0.25 ms) where there are few edges (281 K: a first run of 0.60 ms,
// 1.07 this way), and also with more as long as L2 holds what it scatters and no
// source draws thousands of its atomics, some 16 ns each (uniform, 12 M edges:
// 0.27 ms, 0.54 this way; 18 M of 2 M vertices 1.56 and 0.88; 11 M with a source
// of 100 K out-edges 1.90 and 0.55).
constexpr int64_t kTrLeast = int64_t(4) << 20;
constexpr int64_t kTrBytes = int64_t(64) << 20;  // of destinations, weights and places
constexpr int32_t kTrDegree = 16384;             // of a source

struct TrSlice {
  int64_t begin;   // in the bucketed arrays
  int32_t count;
  int32_t bucket;  // bit 31: the bucket's only slice
};

struct TrArgs {
  const int64_t* off;
  const int32_t* col;
  const uint32_t* w;
  const int2* units;
  const int4* heavy;
  int32_t n_units, batch, chunk, heavy_deg, n_buckets, V;
  int64_t E;
  const int64_t* ooff;
  unsigned long long* bucket_at;  // next place of each bucket
  unsigned long long* source_at;  // next place of each source
  unsigned int* ctr;              // batches claimed; sources with more edges than outdeg says
  uint16_t* src;
  int32_t* dst;
  uint32_t* wt;
  const TrSlice* slices;
  int32_t* ocol;
  uint32_t* ow;
};

// Calls f(edge, vertex) for every edge of unit u, by the warp.
template <class F>
__device__ __forceinline__ void tr_unit_edges(const TrArgs& a, int2 u, int lane, const F& f) {
  if (u.x < 0) {  // a chunk of a heavy vertex
    const int v = a.heavy[-u.x - 1].x;
    const int64_t b = a.off[v] + static_cast<int64_t>(u.y) * a.chunk, e = min(a.off[v + 1], b + a.chunk);
    for (int64_t k = b + lane; k < e; k += 32) f(k, v);
    return;
  }
  int64_t b = 0;
  int len = 0;
  if (lane < u.y - u.x) {
    b = a.off[u.x + lane];
    const int64_t n = a.off[u.x + lane + 1] - b;
    len = n > a.heavy_deg ? 0 : static_cast<int>(n);
  }
  int pre = len;  // entries of the lanes before
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) pre += x;
  }
  const int total = __shfl_sync(0xffffffffu, pre, 31);
  pre -= len;
  for (int k0 = 0; k0 < total; k0 += 32) {
    const int k = k0 + lane;
    int l = 0;  // the last lane whose entries start at or before k (every lane takes part in every shuffle)
#pragma unroll
    for (int sp = 16; sp > 0; sp >>= 1) {
      const int x = __shfl_sync(0xffffffffu, pre, l + sp);
      if (x <= k) l += sp;
    }
    const int lo = __shfl_sync(0xffffffffu, pre, l);
    const int64_t bl = __shfl_sync(0xffffffffu, b, l);
    if (k < total) f(bl + (k - lo), u.x + l);
  }
}

__global__ void __launch_bounds__(kTrThreads) tr_bucket_kernel(const __grid_constant__ TrArgs a) {
  extern __shared__ __align__(16) unsigned char s_mem[];
  unsigned long long* s_at = reinterpret_cast<unsigned long long*>(s_mem);
  unsigned int* s_cnt = reinterpret_cast<unsigned int*>(s_at + a.n_buckets);
  __shared__ int s_batch;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (;;) {
    if (threadIdx.x == 0) s_batch = static_cast<int>(atomicAdd(a.ctr, 1u));
    for (int i = threadIdx.x; i < a.n_buckets; i += kTrThreads) s_cnt[i] = 0;
    __syncthreads();
    const int64_t u0 = static_cast<int64_t>(s_batch) * a.batch;
    if (u0 >= a.n_units) break;
    const int u1 = static_cast<int>(min(u0 + a.batch, static_cast<int64_t>(a.n_units)));
    for (int u = static_cast<int>(u0) + wid; u < u1; u += kTrThreads / 32)
      tr_unit_edges(a, a.units[u], lane, [&](int64_t k, int) { atomicAdd(&s_cnt[a.col[k] >> kBucketBits], 1u); });
    __syncthreads();
    for (int i = threadIdx.x; i < a.n_buckets; i += kTrThreads) {
      const unsigned int n = s_cnt[i];
      if (n) s_at[i] = atomicAdd(a.bucket_at + i, static_cast<unsigned long long>(n));
      s_cnt[i] = 0;
    }
    __syncthreads();
    for (int u = static_cast<int>(u0) + wid; u < u1; u += kTrThreads / 32)
      tr_unit_edges(a, a.units[u], lane, [&](int64_t k, int v) {
        const int32_t s = a.col[k];
        const int b = s >> kBucketBits;
        const unsigned long long p = s_at[b] + atomicAdd(&s_cnt[b], 1u);
        if (p < static_cast<unsigned long long>(a.E)) {  // always, when outdeg counts the edges of col
          a.src[p] = static_cast<uint16_t>(s & (kBucket - 1));
          a.dst[p] = v;
          if (a.w) a.wt[p] = a.w[k];
        }
      });
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kTrThreads) tr_place_kernel(const __grid_constant__ TrArgs a) {
  extern __shared__ __align__(16) unsigned int s_src[];  // counts, then next places from the bucket's start
  const TrSlice sl = a.slices[blockIdx.x];
  const bool only = sl.bucket < 0;
  const int32_t v0 = (sl.bucket & 0x7fffffff) << kBucketBits, nv = min(kBucket, a.V - v0);
  const int64_t start = a.ooff[v0];
  for (int i = threadIdx.x; i < kBucket; i += kTrThreads) s_src[i] = 0;
  __syncthreads();
  if (!only) {
    for (int k = threadIdx.x; k < sl.count; k += kTrThreads) atomicAdd(&s_src[a.src[sl.begin + k] & (kBucket - 1)], 1u);
    __syncthreads();
  }
  for (int i = threadIdx.x; i < nv; i += kTrThreads) {
    if (only) {
      s_src[i] = static_cast<unsigned int>(a.ooff[v0 + i] - start);
    } else if (s_src[i]) {
      const unsigned long long n = s_src[i], p = atomicAdd(a.source_at + v0 + i, n);
      if (p + n > static_cast<unsigned long long>(a.ooff[v0 + i + 1])) a.ctr[1] = 1;
      s_src[i] = static_cast<unsigned int>(p - start);
    }
  }
  __syncthreads();
#pragma unroll 4
  for (int k = threadIdx.x; k < sl.count; k += kTrThreads) {
    const int64_t p = start + atomicAdd(&s_src[a.src[sl.begin + k] & (kBucket - 1)], 1u);
    if (p < a.E) {
      a.ocol[p] = a.dst[sl.begin + k];
      if (a.w) a.ow[p] = a.wt[sl.begin + k];
    }
  }
  if (only) {
    __syncthreads();
    for (int i = threadIdx.x; i < nv; i += kTrThreads)
      if (s_src[i] > static_cast<unsigned int>(a.ooff[v0 + i + 1] - start)) a.ctr[1] = 1;
  }
}

__global__ void tr_bucket_starts_kernel(const int64_t* ooff, int32_t V, int32_t n_buckets, unsigned long long* at) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= n_buckets) at[i] = static_cast<unsigned long long>(ooff[min(static_cast<int64_t>(i) << kBucketBits, static_cast<int64_t>(V))]);
}

}  // namespace

namespace gx {

bool transpose_by_buckets(gx_engine* e, bool weighted, int32_t most, gx_status* status) {
  const int32_t V = e->V;
  const int64_t E = e->E;
  const int64_t nb64 = (static_cast<int64_t>(V) + kBucket - 1) / kBucket;
  if (nb64 > kMostBuckets || E > static_cast<int64_t>(UINT32_MAX) || E < kTrLeast) return false;
  if ((weighted ? 8 : 4) * E + 8 * static_cast<int64_t>(V) < kTrBytes && most < kTrDegree) return false;
  const int32_t nb = static_cast<int32_t>(nb64);
  cudaStream_t s = e->s_comp;
  struct Block {
    unsigned char* p = nullptr;
    ~Block() { dev_free(&p); }
  } block;
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t x = at;
    at += (bytes + 255) & ~size_t(255);
    return x;
  };
  const size_t n = static_cast<size_t>(E);
  const size_t o_src = place(2 * n), o_dst = place(4 * n), o_wt = place(weighted ? 4 * n : 0);
  const size_t o_bucket = place(8 * (static_cast<size_t>(nb) + 1)), o_source = place(8 * static_cast<size_t>(V)),
               o_ctr = place(8);
  const size_t o_slices = place(sizeof(TrSlice) * (n / kTrSlice + static_cast<size_t>(nb)));
  if (dev_alloc(&block.p, at) != GX_OK) return false;  // no room: the caller's one-pass kernel
  auto run = [&]() -> gx_status {
    TrArgs a{};
    a.off = e->d_off;
    a.col = e->d_col;
    a.w = weighted ? e->d_w : nullptr;
    a.units = e->d_units;
    a.heavy = e->d_heavy;
    a.n_units = static_cast<int32_t>(e->units.size());
    a.chunk = e->caps.chunk;
    a.heavy_deg = e->caps.heavy;
    a.n_buckets = nb;
    a.V = V;
    a.E = E;
    a.ooff = e->d_ooff;
    a.bucket_at = reinterpret_cast<unsigned long long*>(block.p + o_bucket);
    a.source_at = reinterpret_cast<unsigned long long*>(block.p + o_source);
    a.ctr = reinterpret_cast<unsigned int*>(block.p + o_ctr);
    a.src = reinterpret_cast<uint16_t*>(block.p + o_src);
    a.dst = reinterpret_cast<int32_t*>(block.p + o_dst);
    a.wt = reinterpret_cast<uint32_t*>(block.p + o_wt);
    a.ocol = e->d_ocol;
    a.ow = e->d_ow;
    std::vector<unsigned long long> start(static_cast<size_t>(nb) + 1), end(static_cast<size_t>(nb));
    tr_bucket_starts_kernel<<<(nb + 256) / 256, 256, 0, s>>>(e->d_ooff, V, nb, a.bucket_at);
    GX_CUDA(cudaMemcpyAsync(start.data(), a.bucket_at, 8 * start.size(), cudaMemcpyDeviceToHost, s));
    GX_CUDA(cudaMemcpyAsync(a.source_at, e->d_ooff, 8 * static_cast<size_t>(V), cudaMemcpyDeviceToDevice, s));
    GX_CUDA(cudaMemsetAsync(a.ctr, 0, 8, s));
    // Batches of about 64 units, fewer where that would leave SMs without.
    const int smem_b = 12 * nb, smem_p = 4 * kBucket;
    GX_CUDA(allow_dynamic_smem(e->dev, reinterpret_cast<const void*>(tr_bucket_kernel)));
    GX_CUDA(allow_dynamic_smem(e->dev, reinterpret_cast<const void*>(tr_place_kernel)));
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tr_bucket_kernel, kTrThreads, smem_b);
    const int grid = std::max(1, per_sm) * e->n_sm;
    a.batch = std::max(1, std::min(64, a.n_units / grid));
    tr_bucket_kernel<<<grid, kTrThreads, smem_b, s>>>(a);
    GX_CUDA(cudaGetLastError());
    GX_CUDA(cudaMemcpyAsync(end.data(), a.bucket_at, 8 * end.size(), cudaMemcpyDeviceToHost, s));
    GX_CUDA(cudaStreamSynchronize(s));  // `start` and `end` have arrived
    for (int32_t b = 0; b < nb; ++b)
      if (end[b] != start[b + 1]) return out_degrees_wrong();
    std::vector<TrSlice> slices;
    for (int32_t b = 0; b < nb; ++b) {
      const int64_t lo = static_cast<int64_t>(start[b]), hi = static_cast<int64_t>(start[b + 1]);
      const bool only = hi - lo <= kTrSlice;
      for (int64_t k = lo; k < hi; k += kTrSlice)
        slices.push_back(TrSlice{k, static_cast<int32_t>(std::min(kTrSlice, hi - k)),
                                 static_cast<int32_t>(static_cast<uint32_t>(b) | (only ? 0x80000000u : 0u))});
    }
    if (slices.empty()) return GX_OK;
    GX_CUDA(cudaMemcpyAsync(block.p + o_slices, slices.data(), slices.size() * sizeof(TrSlice), cudaMemcpyHostToDevice, s));
    a.slices = reinterpret_cast<const TrSlice*>(block.p + o_slices);
    tr_place_kernel<<<static_cast<unsigned>(slices.size()), kTrThreads, smem_p, s>>>(a);
    GX_CUDA(cudaGetLastError());
    // Every bucket has as many edges as its sources' out-degrees say, so a
    // source with fewer has one with more beside it.
    unsigned int over = 0;
    GX_CUDA(cudaMemcpyAsync(&over, a.ctr + 1, 4, cudaMemcpyDeviceToHost, s));
    GX_CUDA(cudaStreamSynchronize(s));
    return over ? out_degrees_wrong() : GX_OK;
  };
  *status = run();
  return true;
}

}  // namespace gx
