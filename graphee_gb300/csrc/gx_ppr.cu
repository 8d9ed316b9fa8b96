// Multi-source personalized PageRank as a sparse-times-dense product over
// the loaded CSC:  R <- restart*S + (1-restart) * A^T D^-1 R,  R0 = S,
// with R a V x k FP32 matrix (k <= 64 sources) and S the one-hot source
// matrix.  No reference counterpart; the per-edge arithmetic is PageRank's
// pull (GraphMP/app/pagerank.cpp:44-48) applied to k rank vectors at once.
//
// HBM layout: rows of W = k rounded up to 8 columns (32..256 bytes).
// Rs[2][V][W] holds R[u,:]/outdeg[u] (double buffer, so an edge costs one
// coalesced row gather of W floats); the final R is written on the last step
// only.
//
// All steps run in ONE persistent cooperative launch, captured in a CUDA
// graph: CTAs sweep a step's work units, meet at a grid barrier (bounded by
// config.wait_limit polls; a timeout raises an abort flag every CTA honours
// and the call returns GX_ERR_TIMEOUT), and go on to the next step.  A row is
// summed by a group of W/2 lanes (a float2 each), so a warp works on 64/W rows
// at once.  What bounds a step is how many row gathers are in flight, and its
// longest unit: units are the engine's edge-capped tiles, whose edges a group
// streams eight at a time across the vertices' boundaries, and chunks of
// kPprChunk in-edges of the vertices above kPprHeavy, a group each.  Chunked
// vertices fold their partial rows in chunk order in the warp group that
// finishes last, so results are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "gx_engine.h"
#include "gx_nvtx.h"

using namespace gx;

namespace {

constexpr int kPprMaxCols = 64;
constexpr int kPprHeavy = 512;    // longest list a group streams inside its tile
constexpr int kPprChunk = 256;    // edges of one chunk of a longer one
constexpr int kPprThreads = 256;
constexpr int kPprWarps = kPprThreads / 32;

struct PprArgs {
  const int64_t* off;
  const int32_t* col;
  const int32_t* outdeg;
  float* rs[2];             // R[u,:]/outdeg[u], double buffer [V][W]
  float* r_out;             // final R [V][W]
  const int2* tiles;        // the engine's units: tile (vb, ve), or x < 0 (not ours)
  const int4* chunks;       // (v, chunk, n_chunks, partial base)
  int32_t n_tiles, n_chunks;
  int32_t iters;
  unsigned int* ctr;        // kQueues work cursors per step
  unsigned int* arrive;     // grid-barrier arrival count per step
  unsigned int* abort;      // set when a grid barrier gives up
  unsigned int wait_limit;  // polls before it does, each a load and a pause of some 64 ns
  float* partial;           // [n_chunks][W]
  unsigned int* ticket;     // per chunked vertex, indexed by partial base
  const int32_t* src;       // [W] source vertex of each column (-1 past k)
  float alpha, restart;
};

// All CTAs of the (co-resident) grid meet after step `it`.  Returns false
// when the wait timed out or another CTA gave up.
__device__ bool ppr_grid_barrier(const PprArgs& a, int it) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(a.arrive + it, 1u);
    int ok = 1;
    volatile unsigned* c = a.arrive + it;
    volatile unsigned* ab = a.abort;
    for (unsigned i = 0; *c < gridDim.x; ++i) {
      if (*ab || i >= a.wait_limit) {
        atomicExch(a.abort, 1u);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    s_ok = ok && !*ab;
  }
  __syncthreads();
  return s_ok != 0;
}

// The chunks of the vertices above kPprHeavy: counted (units null) or written,
// each vertex's side by side from an index that an atomic gives out.
__global__ void ppr_chunks_kernel(const int64_t* off, int32_t V, int4* units, unsigned int* count) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const int64_t d = off[v + 1] - off[v];
    if (d <= kPprHeavy) continue;
    const int n = static_cast<int>((d + kPprChunk - 1) / kPprChunk);
    const int base = static_cast<int>(atomicAdd(count, static_cast<unsigned>(n)));
    if (units)
      for (int c = 0; c < n; ++c) units[base + c] = make_int4(v, c, n, base);
  }
}

// What the lanes of a group hold: its columns and their sources.
template <int W>
struct PprGroup {
  static constexpr int L = W / 2;   // lanes per row, a float2 each
  static constexpr int G = 32 / L;  // groups of a warp
  int gl, grp, s0, s1;
  unsigned mask;

  __device__ __forceinline__ void finish(const PprArgs& a, float* rs_out, bool last, int v, int32_t od,
                                         float2 acc) const {
    float2 r = make_float2(a.alpha * acc.x, a.alpha * acc.y);
    if (s0 == v) r.x += a.restart;
    if (s1 == v) r.y += a.restart;
    const size_t row = static_cast<size_t>(v) * W + 2 * gl;
    if (last) {
      *reinterpret_cast<float2*>(a.r_out + row) = r;
    } else {
      const float inv = 1.0f / static_cast<float>(od > 0 ? od : 1);
      *reinterpret_cast<float2*>(rs_out + row) = make_float2(r.x * inv, r.y * inv);
    }
  }

  // Eight edges p[k .. k + 7] (16-byte aligned), those in [lo, hi) taken, in
  // order; c holds their ids, loaded a step ahead.
  __device__ __forceinline__ void ids(int32_t (&c)[8], const int32_t* p, int k, int hi) const {
    int4 x = make_int4(0, 0, 0, 0), y = x;
    if (k < hi) x = __ldg(reinterpret_cast<const int4*>(p + k));
    if (k + 4 < hi) y = __ldg(reinterpret_cast<const int4*>(p + k + 4));
    c[0] = x.x, c[1] = x.y, c[2] = x.z, c[3] = x.w, c[4] = y.x, c[5] = y.y, c[6] = y.z, c[7] = y.w;
  }
  __device__ __forceinline__ void rows(float2 (&x)[8], const int32_t (&c)[8], const float* rs_in, int k, int lo,
                                       int hi) const {
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      x[t] = make_float2(0.f, 0.f);
      if (k + t >= lo && k + t < hi)
        x[t] = *(reinterpret_cast<const float2*>(rs_in + static_cast<size_t>(c[t]) * W) + gl);
    }
  }
};

template <int W>
__global__ void __launch_bounds__(kPprThreads, 4) ppr_kernel(const __grid_constant__ PprArgs a) {
  typedef PprGroup<W> Group;
  constexpr int L = Group::L, G = Group::G;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  Group q;
  q.gl = lane % L;
  q.grp = lane / L;
  q.mask = L == 32 ? 0xffffffffu : (((1u << L) - 1u) << (q.grp * L));
  q.s0 = a.src[2 * q.gl];
  q.s1 = a.src[2 * q.gl + 1];
  const int first_tile = (a.n_chunks + G - 1) / G, U = first_tile + a.n_tiles;
  const int nq = U / 256 < 1 ? 1 : (U / 256 < kQueues ? U / 256 : kQueues);
  for (int it = 0; it < a.iters; ++it) {
    const float* rs_in = (it & 1) ? a.rs[1] : a.rs[0];
    float* rs_out = (it & 1) ? a.rs[0] : a.rs[1];
    const bool last = it + 1 == a.iters;
    unsigned int* ctr = a.ctr + static_cast<size_t>(kQueues) * kQueueStride * it;
    int qi = (blockIdx.x * kPprWarps + wid) % nq;
    int claim = 0;  // in flight while the last unit is swept
    if (lane == 0) claim = static_cast<int>(atomicAdd(ctr + qi * kQueueStride, 1u));
    for (;;) {
      const int qb = static_cast<int>((static_cast<int64_t>(U) * qi) / nq);
      const int qe = static_cast<int>((static_cast<int64_t>(U) * (qi + 1)) / nq);
      const int u = qb + __shfl_sync(0xffffffffu, claim, 0);
      if (u >= qe) {
        qi = next_queue(ctr, qi, nq, U, lane);
        if (qi < 0) break;
        if (lane == 0) claim = static_cast<int>(atomicAdd(ctr + qi * kQueueStride, 1u));
        continue;
      }
      if (lane == 0) claim = static_cast<int>(atomicAdd(ctr + qi * kQueueStride, 1u));
      if (u < first_tile) {
        // ---- a chunk per group ----
        const int h = u * G + q.grp;
        if (h < a.n_chunks) {
          const int4 un = a.chunks[h];
          const int64_t vb = a.off[un.x], ve = a.off[un.x + 1];
          const int64_t b = vb + static_cast<int64_t>(un.y) * kPprChunk;
          const int lo = static_cast<int>(b & 3), hi = lo + static_cast<int>(ve - b < kPprChunk ? ve - b : kPprChunk);
          const int32_t* p = a.col + (b & ~3ll);
          float2 acc = make_float2(0.f, 0.f);
          int32_t c[8];
          q.ids(c, p, 0, hi);
          for (int k = 0; k < hi; k += 8) {
            float2 x[8];
            q.rows(x, c, rs_in, k, lo, hi);
            q.ids(c, p, k + 8, hi);
#pragma unroll
            for (int t = 0; t < 8; ++t) {  // places outside hold 0
              acc.x += x[t].x;
              acc.y += x[t].y;
            }
          }
          reinterpret_cast<float2*>(a.partial + static_cast<size_t>(un.w + un.y) * W)[q.gl] = acc;
          __threadfence();
          __syncwarp(q.mask);
          unsigned t = 0;
          if (q.gl == 0) t = atomicAdd(a.ticket + un.w, 1u);
          t = __shfl_sync(q.mask, t, 0, L);
          if (t == static_cast<unsigned>(un.z) - 1) {
            __threadfence();
            float2 tot = make_float2(0.f, 0.f);
#pragma unroll 8
            for (int i = 0; i < un.z; ++i) {
              const float2 y =
                  __ldcg(reinterpret_cast<const float2*>(a.partial + static_cast<size_t>(un.w + i) * W) + q.gl);
              tot.x += y.x;
              tot.y += y.y;
            }
            q.finish(a, rs_out, last, un.x, a.outdeg[un.x], tot);
            if (q.gl == 0) a.ticket[un.w] = 0;
          }
        }
        __syncwarp();
        continue;
      }
      // ---- a tile: each group its share of the vertices, one per lane ----
      const int2 tile = a.tiles[u - first_tile];
      if (tile.x < 0) continue;
      const int n = tile.y - tile.x, per = (n + G - 1) / G;
      const int v0 = tile.x + q.grp * per;
      const int cnt = min(per, tile.y - v0);  // may be negative: no vertex left
      int64_t vb = 0, ve = 0;
      int32_t od = 0;
      if (q.gl < cnt) {
        vb = a.off[v0 + q.gl];
        ve = a.off[v0 + q.gl + 1];
        od = a.outdeg[v0 + q.gl];
      }
      const unsigned heavy = __ballot_sync(q.mask, ve - vb > kPprHeavy) >> (q.grp * L);
      for (int j = 0; j < cnt;) {
        if ((heavy >> j) & 1u) {
          ++j;
          continue;
        }
        // A run of vertices up to the next heavy one: its edges are one stream.
        const unsigned rest = heavy >> j;
        const int jn = rest ? j + __ffs(rest) - 1 : cnt;
        const int64_t base = __shfl_sync(q.mask, vb, j, L) & ~3ll;
        const int lo = static_cast<int>(__shfl_sync(q.mask, vb, j, L) - base);
        const int hi = static_cast<int>(__shfl_sync(q.mask, ve, jn - 1, L) - base);
        const int my_end = static_cast<int>(ve - base);  // of the lane's vertex, when it is in the run
        const int32_t* p = a.col + base;
        int end = __shfl_sync(q.mask, my_end, j, L);
        float2 acc = make_float2(0.f, 0.f);
        int32_t c[8];
        q.ids(c, p, 0, hi);
        auto flush = [&]() {
          q.finish(a, rs_out, last, v0 + j, __shfl_sync(q.mask, od, j, L), acc);
          acc = make_float2(0.f, 0.f);
          ++j;
          end = __shfl_sync(q.mask, my_end, j < jn ? j : jn - 1, L);
        };
        for (int k = 0; k < hi; k += 8) {
          float2 x[8];
          q.rows(x, c, rs_in, k, lo, hi);
          q.ids(c, p, k + 8, hi);
#pragma unroll
          for (int t = 0; t < 8; ++t) {
            if (k + t < hi) {
              while (k + t >= end) flush();
              acc.x += x[t].x;
              acc.y += x[t].y;
            }
          }
        }
        while (j < jn) flush();
      }
      __syncwarp();
    }
    if (!ppr_grid_barrier(a, it)) return;
  }
}

// out[v][0, k) = in[perm ? perm[v] : v][0, k) of rows of W columns: the rows
// as the caller numbers them, without the columns past k.
__global__ void ppr_rows_kernel(const float* __restrict__ in, const int32_t* __restrict__ perm, int32_t V, int k, int W,
                                float* __restrict__ out) {
  const int64_t n = static_cast<int64_t>(V) * k, stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t v = static_cast<int32_t>(i / k), j = static_cast<int32_t>(i % k);
    out[i] = in[static_cast<size_t>(perm ? perm[v] : v) * W + j];
  }
}

__global__ void ppr_init_kernel(float* rs, const int32_t* outdeg, const int32_t* src, int k, int W) {
  const int j = threadIdx.x;
  if (j < k) {
    const int v = src[j];
    const int32_t od = outdeg[v];
    rs[static_cast<size_t>(v) * W + j] = 1.0f / static_cast<float>(od > 0 ? od : 1);
  }
}

template <int W>
const void* ppr_kernel_for() {
  return reinterpret_cast<const void*>(ppr_kernel<W>);
}

}  // namespace

extern "C" gx_status gx_ppr(gx_engine* e, int32_t k, const int32_t* sources, int32_t iters, double restart,
                            float* host_out, gx_run_stats* stats) {
  gx::NvtxRange nvtx_range("gx_ppr");
  if (!e || !sources || k < 1 || k > kPprMaxCols || iters < 0 || restart < 0 || restart > 1)
    return fail(GX_ERR_INVALID, "gx_ppr: bad arguments (k must be 1..64)");
  if (!e->loaded) return fail(GX_ERR_STATE, "gx_ppr: no graph loaded");
  if (!e->all_resident) return fail(GX_ERR_STATE, "gx_ppr: needs every shard resident (no shard-cache budget)");
  const int32_t V = e->V;
  for (int j = 0; j < k; ++j)
    if (sources[j] < 0 || sources[j] >= V) return fail(GX_ERR_INVALID, "gx_ppr: source %d outside [0, %d)", sources[j], V);
  GX_CUDA(cudaSetDevice(e->dev));
  BlockBound bound(e->block_bound);
  cudaStream_t s = e->s_comp;
  const int W = k <= 8 ? 8 : k <= 16 ? 16 : k <= 32 ? 32 : 64;
  const size_t rows = static_cast<size_t>(V) * W;
  const size_t steps = static_cast<size_t>(std::max(iters, 1));
  const int32_t n_tiles = static_cast<int32_t>(e->units.size());
  int32_t h_src[kPprMaxCols];
  for (int j = 0; j < kPprMaxCols; ++j) h_src[j] = j < k ? (e->relabeled ? e->h_perm[sources[j]] : sources[j]) : -1;
  // One block for everything of a known size: rows, cursors, flags.
  struct Guard {
    unsigned char *block = nullptr, *chunk_block = nullptr;
    ~Guard() {
      dev_free(&block);
      dev_free(&chunk_block);
    }
  } guard;
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t x = at;
    at += (bytes + 255) & ~size_t(255);
    return x;
  };
  const size_t o_rs0 = place(rows * sizeof(float)), o_rs1 = place(rows * sizeof(float)), o_r = place(rows * sizeof(float));
  const size_t o_src = place(sizeof(h_src));
  const size_t o_zero = at;  // cleared by the graph, in one piece
  const size_t o_ctr = place(sizeof(unsigned int) * kQueues * kQueueStride * steps);
  const size_t o_arrive = place(sizeof(unsigned int) * steps), o_abort = place(sizeof(unsigned int));
  const size_t zero_bytes = at - o_zero;
  const size_t o_count = place(2 * sizeof(unsigned int));
  GX_TRY(dev_alloc(&guard.block, at));
  float* rs0 = reinterpret_cast<float*>(guard.block + o_rs0);
  float* rs1 = reinterpret_cast<float*>(guard.block + o_rs1);
  float* r = reinterpret_cast<float*>(guard.block + o_r);
  int32_t* d_src = reinterpret_cast<int32_t*>(guard.block + o_src);
  unsigned int* abort_flag = reinterpret_cast<unsigned int*>(guard.block + o_abort);
  unsigned int* count = reinterpret_cast<unsigned int*>(guard.block + o_count);
  GX_CUDA(cudaMemcpyAsync(d_src, h_src, sizeof(h_src), cudaMemcpyHostToDevice, s));
  // Chunks of the long lists: counted, then written with their tickets clear.
  GX_CUDA(cudaMemsetAsync(count, 0, 2 * sizeof(unsigned int), s));
  const int plan_grid = std::max(1, std::min(e->n_sm * 4, (V + 255) / 256));
  ppr_chunks_kernel<<<plan_grid, 256, 0, s>>>(e->d_off, V, nullptr, count);
  GX_CUDA(cudaGetLastError());
  unsigned int n_chunks = 0;
  GX_CUDA(cudaMemcpyAsync(&n_chunks, count, sizeof(n_chunks), cudaMemcpyDeviceToHost, s));
  GX_CUDA(cudaStreamSynchronize(s));
  const size_t nc = std::max<size_t>(n_chunks, 1);
  at = 0;
  const size_t o_chunks = place(nc * sizeof(int4)), o_partial = place(nc * W * sizeof(float)),
               o_ticket = place(nc * sizeof(unsigned int));
  GX_TRY(dev_alloc(&guard.chunk_block, at));
  int4* chunks = reinterpret_cast<int4*>(guard.chunk_block + o_chunks);
  unsigned int* ticket = reinterpret_cast<unsigned int*>(guard.chunk_block + o_ticket);
  if (n_chunks) {
    GX_CUDA(cudaMemsetAsync(ticket, 0, nc * sizeof(unsigned int), s));
    ppr_chunks_kernel<<<plan_grid, 256, 0, s>>>(e->d_off, V, chunks, count + 1);
    GX_CUDA(cudaGetLastError());
  }

  PprArgs a{};
  a.off = e->d_off;
  a.col = e->d_col;
  a.outdeg = e->d_outdeg;
  a.rs[0] = rs0;
  a.rs[1] = rs1;
  a.r_out = r;
  a.tiles = e->d_units;
  a.chunks = chunks;
  a.n_tiles = n_tiles;
  a.n_chunks = static_cast<int32_t>(n_chunks);
  a.iters = iters;
  a.ctr = reinterpret_cast<unsigned int*>(guard.block + o_ctr);
  a.arrive = reinterpret_cast<unsigned int*>(guard.block + o_arrive);
  a.abort = abort_flag;
  a.wait_limit = e->cfg.wait_limit;
  a.partial = reinterpret_cast<float*>(guard.chunk_block + o_partial);
  a.ticket = ticket;
  a.src = d_src;
  a.alpha = static_cast<float>(1.0 - restart);
  a.restart = static_cast<float>(restart);
  const void* fn = W == 8 ? ppr_kernel_for<8>() : W == 16 ? ppr_kernel_for<16>() : W == 32 ? ppr_kernel_for<32>()
                                                                                           : ppr_kernel_for<64>();
  int per_sm = 0;
  GX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kPprThreads, 0));
  // Co-resident CTAs only: the grid barrier waits for every one of them.  No
  // more than have a unit per warp: each one more is an arrival every step.
  const int64_t n_units = static_cast<int64_t>(n_tiles) + n_chunks;
  const int grid = static_cast<int>(std::max<int64_t>(
      1, std::min<int64_t>(std::max(1, per_sm) * e->n_sm, (n_units + kPprWarps - 1) / kPprWarps)));
  cudaLaunchConfig_t lc{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  lc.gridDim = dim3(grid);
  lc.blockDim = dim3(kPprThreads);
  lc.dynamicSmemBytes = 0;
  lc.stream = s;
  lc.attrs = attr;
  lc.numAttrs = 1;
  void* kargs[] = {&a};
  // The step's resets, R0 = S and the persistent launch, as one graph.
  auto enqueue = [&]() -> cudaError_t {
    cudaError_t err = cudaMemsetAsync(rs0, 0, rows * sizeof(float), s);
    if (err == cudaSuccess) err = cudaMemsetAsync(guard.block + o_zero, 0, zero_bytes, s);
    if (err != cudaSuccess) return err;
    ppr_init_kernel<<<1, kPprMaxCols, 0, s>>>(rs0, e->d_outdeg, d_src, k, W);
    err = cudaGetLastError();
    if (err == cudaSuccess && iters > 0) err = cudaLaunchKernelExC(&lc, fn, kargs);
    return err;
  };
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::unique_lock<std::shared_mutex> capturing(capture_mutex());
  GX_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  cudaError_t cap_err = enqueue();
  cudaError_t end_err = cudaStreamEndCapture(s, &graph);
  capturing.unlock();
  if (cap_err != cudaSuccess || end_err != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    return fail(GX_ERR_CUDA, "gx_ppr: capture: %s", cudaGetErrorString(cap_err != cudaSuccess ? cap_err : end_err));
  }
  cudaError_t err = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (err != cudaSuccess) return fail(GX_ERR_CUDA, "gx_ppr: graph instantiate: %s", cudaGetErrorString(err));
  cudaEvent_t ev0, ev1;
  GX_CUDA(cudaEventCreate(&ev0));
  GX_CUDA(cudaEventCreate(&ev1));
  GX_CUDA(cudaEventRecord(ev0, s));
  err = cudaGraphLaunch(exec, s);
  if (err == cudaSuccess) err = cudaEventRecord(ev1, s);
  if (err == cudaSuccess) err = cudaEventSynchronize(ev1);
  float ms = 0;
  if (err == cudaSuccess) cudaEventElapsedTime(&ms, ev0, ev1);
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  cudaGraphExecDestroy(exec);
  if (err != cudaSuccess) return fail(GX_ERR_CUDA, "gx_ppr: run failed: %s", cudaGetErrorString(err));
  unsigned int aborted = 0;
  GX_CUDA(cudaMemcpy(&aborted, abort_flag, sizeof(aborted), cudaMemcpyDeviceToHost));
  if (aborted) return fail(GX_ERR_TIMEOUT, "gx_ppr: a grid barrier timed out");
  if (host_out) {
    if (iters == 0) {
      memset(host_out, 0, sizeof(float) * static_cast<size_t>(V) * k);
      for (int j = 0; j < k; ++j) host_out[static_cast<size_t>(sources[j]) * k + j] = 1.f;
    } else {
      // The caller's rows of k columns, put together on the device (rs0 is
      // free by now) and copied in one piece.
      const size_t bytes = sizeof(float) * static_cast<size_t>(V) * k;
      if (e->relabeled || k != W) {
        ppr_rows_kernel<<<e->n_sm * 8, 256, 0, s>>>(r, e->relabeled ? e->d_perm : nullptr, V, k, W, rs0);
        GX_CUDA(cudaGetLastError());
        GX_CUDA(cudaStreamSynchronize(s));
        r = rs0;
      }
      GX_TRY(copy_to_host(e, host_out, r, bytes));
    }
  }
  if (stats) {
    *stats = gx_run_stats{};
    stats->iterations = iters;
    stats->edges_scanned = e->E * static_cast<int64_t>(iters);
    stats->ms_total = ms;
    stats->ms_compute = ms;
    stats->kernel_launches = iters > 0 ? 2 : 1;
    stats->pull_launches = iters > 0 ? 1 : 0;
    stats->ms_pull = ms;
  }
  return GX_OK;
}
