// Triangle counting on the loaded graph, taken as undirected: the CSC of a
// symmetrised, deduplicated edge list (each undirected edge stored in both
// directions, no self-loops).  No reference counterpart: the reference's
// only "tc" (GraphH/list/system/GraphPS.h:15-95) counts reciprocal edges.
//
//  1. orient u -> v iff (deg u, u) < (deg v, v): a DAG, in which every
//     triangle has exactly one edge {u, v} whose ends share its third vertex
//     as out-neighbour;
//  2. write N+(v) in the room its CSC list leaves (no order is needed below,
//     so no count pass or scan comes first), padded to whole 16-byte pieces;
//     where the device has no room for that, the lists are counted first and
//     laid end to end, in half of it;
//  3. count sum over edges {x, y} of |N+(x) n N+(y)|: the end with the longer
//     N+ (x) is staged, the shorter list is scanned (half the probes of
//     scanning N+(v) for every u -> v on R-MAT).  A vertex with much to scan
//     gets a CTA that stages N+(x) as a bitmap over the vertices in shared
//     memory: a probe is one word's load and a shift, exact, and a warp reads
//     128 entries of a scanned list at once.  The others get a warp with a
//     small hash table of N+(x).
// A bitmap holds tc_bits vertices.  A larger graph is renumbered by (degree,
// id), and the bitmap stands for the highest ranks: N+ of a vertex among them
// lies wholly among them, and a vertex below them is left to the warps.
// Counts are exact (64-bit integer sums).  Symmetric R-MAT of scale 20 (4.4 G
// probes of N+(v), 2.0 G of the shorter lists): 18.7 ms with a filter and
// binary searches of N+(u) for every N+(v), 3.0 this way; issue-bound at about
// 15 instructions a probe of a warp's 32; scale 24: 300 -> 86 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <memory>

#include "gx_engine.h"
#include "gx_nvtx.h"

using namespace gx;

namespace {

constexpr int kTcThreads = 256;             // warp kernels
constexpr int kTcWarps = kTcThreads / 32;
// Vertices of a bitmap.  Small bitmaps leave an SM several CTAs, whose waits
// at a vertex's end overlap, large ones leave fewer vertices to the warps:
// symmetric R-MAT of 1 M vertices 3.0 ms with 2^18, 3.6 with 2^19, 4.9 with
// all; 4 M 15.5, 17.7 with 2^19; 16 M 91, 86 with 2^19, 103 with 10^6.
constexpr int64_t kTcBitsLeast = 1 << 18, kTcBitsMost = 1800000;  // 32 and 225 KB
inline int64_t tc_bits(int64_t V) {
  return std::min(V, std::max(kTcBitsLeast, std::min(V / 32, kTcBitsMost)));
}
constexpr int kTcGrab = 4;                  // vertices a warp claims per atomic
// |N+| x degree, a bound of the probes, from which a vertex gets a CTA: 131,072
// vertices 0.37 ms from 2048 to 8192, 0.61 at 16384, 3.1 at 65536 (a warp each
// for hubs); 1 M vertices 3.0 from 2048 to 8192, 3.3 at 1024, 3.7 at 16384.
constexpr int64_t kTcCtaWork = 4096;
constexpr int64_t kTcCtaFirst = 1 << 21;    // ... and from which it is counted before the others
constexpr int kTcPiece = 512;               // entries of a warp's hash table at a time
constexpr int kTcSlots = 2048;
constexpr int32_t kTcNone = -1;             // no vertex: padding, and an empty slot

// What a scan needs of a vertex: its N+.
struct __align__(16) TcInfo {
  int64_t start;  // in dcol, a multiple of 4
  int32_t n;
  int32_t pad;
};

struct TcArgs {
  const int64_t* off;
  const int32_t* col;
  const int2* units;        // the engine's work units and heavy vertices
  const int4* heavy;
  int32_t n_units, chunk, heavy_deg, V;
  const int32_t* deg;
  const int32_t* rank;      // ranked graphs: position by (degree, id), else null
  int32_t* n;               // |N+|
  int32_t* dcol;            // N+ lists (ids, or ranks)
  TcInfo* info;
  int32_t base, bits;       // the bitmap stands for [base, base + bits)
  uint32_t mix, mask;       // unranked: the number dcol holds for an id (tc_mixed)
  int32_t *big, *small;     // vertices for CTAs and for warps; the CTAs' heaviest from big[V] down
  unsigned int* ctr;        // claimed: units; listed: big, small, heaviest; claimed: big, small
  unsigned long long* out;  // triangles, probes
};

__global__ void tc_degree_kernel(const int64_t* off, int32_t V, int32_t* deg, int32_t* n, unsigned long long* keys,
                                 int vb) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
    const int32_t d = static_cast<int32_t>(off[v + 1] - off[v]);
    deg[v] = d;
    n[v] = 0;
    if (keys) keys[v] = static_cast<unsigned long long>(d) << vb | static_cast<unsigned long long>(v);
  }
}

__global__ void tc_rank_kernel(const unsigned long long* sorted, unsigned long long vmask, int32_t V, int32_t* rank) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x)
    rank[sorted[i] & vmask] = i;
}

// The number that stands for vertex y in N+: its rank, or its id mixed within
// [0, V), by an odd factor modulo the next power of two until it lies there.
// (As they are, R-MAT's hot ids, of few set bits, fall into few banks of the
// bitmap: 12.5 wavefronts a load of 32 words, mixed 4.)
__device__ __forceinline__ int32_t tc_mixed(const TcArgs& a, int32_t y) {
  uint32_t x = static_cast<uint32_t>(y);
  do {
    x = (x * a.mix) & a.mask;
  } while (x >= static_cast<uint32_t>(a.V));
  return static_cast<int32_t>(x);
}

// Where N+(v) begins: at least as much room as its list, whole 16-byte pieces.
__device__ __forceinline__ int64_t tc_start(int64_t off, int32_t v) { return (off + 4 * static_cast<int64_t>(v) + 3) & ~3ll; }

// How N+ is laid out: in the room of the CSC's lists, or end to end from
// info[v].start; or only counted, for the latter.
enum : int { kTcSpaced, kTcPacked, kTcCount };
template <int MODE>
__device__ __forceinline__ int64_t tc_place(const TcArgs& a, int32_t v) {
  return MODE == kTcSpaced ? tc_start(a.off[v], v) : MODE == kTcPacked ? a.info[v].start : 0;
}

// The engine's units (tiles of at most 32 vertices, chunks of heavy ones), a
// warp each: the unit's entries 128 at a time, every stage's loads in flight
// together; an entry's vertex is found among the lanes' offsets, and the
// entries kept for one vertex reserve their places with one atomic.
// (A warp per vertex, with R-MAT's hubs, took 0.83 + 0.95 ms to count and fill
// at symmetric scale 20.)
template <int MODE>
__global__ void __launch_bounds__(kTcThreads) tc_fill_kernel(const __grid_constant__ TcArgs a) {
  const int lane = threadIdx.x & 31;
  for (;;) {
    int t = 0;
    if (lane == 0) t = static_cast<int>(atomicAdd(a.ctr, 1u));
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= a.n_units) break;
    const int2 u = a.units[t];
    // The lane's vertex and its entries; a chunk is lane 0's.
    int v = 0;
    int64_t b = 0, e = 0;
    if (u.x < 0) {
      v = a.heavy[-u.x - 1].x;
      b = a.off[v] + static_cast<int64_t>(u.y) * a.chunk;
      e = min(a.off[v + 1], b + a.chunk);
      if (lane > 0) b = e;
    } else if (lane < u.y - u.x) {
      v = u.x + lane;
      b = a.off[v];
      e = a.off[v + 1];
      if (e - b > a.heavy_deg) e = b;  // its chunks' entries
    }
    const int len = static_cast<int>(e - b);
    int pre = len;  // entries of the lanes before
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += x;
    }
    const int total = __shfl_sync(0xffffffffu, pre, 31);
    pre -= len;
    const int32_t dv = len > 0 ? (a.rank ? a.rank[v] : a.deg[v]) : 0;
    const int64_t to = tc_place<MODE>(a, v);
    for (int k0 = 0; k0 < total; k0 += 128) {
      int l[4], lo[4];
      int32_t y[4], dy[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = k0 + 32 * j + lane;
        l[j] = 0;  // the last lane whose entries start at or before k (every lane takes part in every shuffle)
#pragma unroll
        for (int sp = 16; sp > 0; sp >>= 1) {
          const int x = __shfl_sync(0xffffffffu, pre, l[j] + sp);
          if (x <= k) l[j] += sp;
        }
        lo[j] = __shfl_sync(0xffffffffu, pre, l[j]);
        const int64_t bl = __shfl_sync(0xffffffffu, b, l[j]);
        y[j] = k < total ? __ldcs(a.col + bl + (k - lo[j])) : 0;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) dy[j] = a.rank ? a.rank[y[j]] : a.deg[y[j]];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = k0 + 32 * j + lane;
        const int32_t x = __shfl_sync(0xffffffffu, v, l[j]), dx = __shfl_sync(0xffffffffu, dv, l[j]);
        const int64_t tx = __shfl_sync(0xffffffffu, to, l[j]);
        const int hi = lo[j] + __shfl_sync(0xffffffffu, len, l[j]);
        const bool keep = k < total && (dx < dy[j] || (dx == dy[j] && x < y[j]));  // (ranks differ)
        // Lanes first .. last - 1 hold this vertex's entries of the window.
        const int w = k0 + 32 * j, first = max(lo[j] - w, 0), last = max(min(hi - w, 32), 0);
        const unsigned mine = (last >= 32 ? 0xffffffffu : (1u << last) - 1u) & ~((1u << first) - 1u);
        const unsigned m = __ballot_sync(0xffffffffu, keep) & mine;
        int at = 0;
        if (k < total && lane == first && m) at = atomicAdd(a.n + x, __popc(m));
        if (MODE == kTcCount) continue;
        at = __shfl_sync(0xffffffffu, at, first < 32 ? first : 0);
        if (keep) a.dcol[tx + at + __popc(m & ((1u << lane) - 1u))] = a.rank ? dy[j] : tc_mixed(a, y[j]);
      }
    }
  }
}

// Packed lists: their lengths in whole 16-byte pieces, and where they begin.
__global__ void tc_pieces_kernel(const __grid_constant__ TcArgs a, uint32_t* pieces) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < a.V; v += gridDim.x * blockDim.x)
    pieces[v] = (static_cast<uint32_t>(a.n[v]) + 3u) >> 2;
}
__global__ void tc_starts_kernel(const __grid_constant__ TcArgs a, const unsigned long long* at) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < a.V; v += gridDim.x * blockDim.x) {
    a.info[v].start = 4 * static_cast<int64_t>(at[v]);
    a.n[v] = 0;  // counted again as the lists are written
  }
}

// Padding, scan descriptors and the vertices to count from.
template <int MODE>
__global__ void tc_list_kernel(const __grid_constant__ TcArgs a) {
  const int lane = threadIdx.x & 31;
  for (int v0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); v0 < a.V; v0 += gridDim.x * blockDim.x) {
    const int v = v0 + lane;
    bool big = false, small = false;
    if (v < a.V) {
      TcInfo x{tc_place<MODE>(a, v), a.n[v], 0};
      a.info[v] = x;
      for (int k = x.n; k & 3; ++k) a.dcol[x.start + k] = kTcNone;
      const bool in = !a.rank || a.rank[v] >= a.base;
      big = in && static_cast<int64_t>(x.n) * a.deg[v] >= kTcCtaWork;
      small = !big && x.n > 0;
      if (big && static_cast<int64_t>(x.n) * a.deg[v] >= kTcCtaFirst) {
        a.big[a.V - 1 - static_cast<int>(atomicAdd(a.ctr + 3, 1u))] = v;
        big = false;
      }
    }
    const unsigned mb = __ballot_sync(0xffffffffu, big), ms = __ballot_sync(0xffffffffu, small);
    unsigned nb = 0, ns = 0;
    if (lane == 0 && mb) nb = atomicAdd(a.ctr + 1, static_cast<unsigned>(__popc(mb)));
    if (lane == 0 && ms) ns = atomicAdd(a.ctr + 2, static_cast<unsigned>(__popc(ms)));
    nb = __shfl_sync(0xffffffffu, nb, 0);
    ns = __shfl_sync(0xffffffffu, ns, 0);
    const unsigned below = (1u << lane) - 1u;
    if (big) a.big[nb + __popc(mb & below)] = v;
    if (small) a.small[ns + __popc(ms & below)] = v;
  }
}

// Whether the edge {x, y} is counted with x staged: y's list is the shorter.
__device__ __forceinline__ bool tc_scans(int32_t nx, int32_t x, int32_t ny, int32_t y) {
  return ny > 0 && (ny < nx || (ny == nx && y < x));
}

template <int NT>
__device__ __forceinline__ void tc_flush(unsigned long long cnt, unsigned long long work, unsigned long long* out) {
  __shared__ unsigned long long s_red[2][NT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    work += __shfl_xor_sync(0xffffffffu, work, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_red[0][threadIdx.x >> 5] = cnt;
    s_red[1][threadIdx.x >> 5] = work;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long t = 0;
    for (int w = 0; w < NT / 32; ++w) t += s_red[threadIdx.x][w];
    if (t) atomicAdd(out + threadIdx.x, t);
  }
}

// CTA per vertex of a.big: N+(x) as a bitmap; its warps claim 32 of x's
// neighbours at a time, and each half of a warp reads kTcAhead of their lists
// at once, 64 entries of each.
constexpr int kTcAhead = 4;
template <int NT>
__global__ void __launch_bounds__(NT, 2048 / NT / 2) tc_cta_kernel(const __grid_constant__ TcArgs a) {
  extern __shared__ __align__(16) uint32_t s_bits[];
  __shared__ int s_i, s_next;
  const int lane = threadIdx.x & 31;
  const int n_first = static_cast<int>(a.ctr[3]), n_big = n_first + static_cast<int>(a.ctr[1]);
  for (int i = threadIdx.x; i <= a.bits / 32; i += NT) s_bits[i] = 0u;
  unsigned long long cnt = 0, work = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      s_i = static_cast<int>(atomicAdd(a.ctr + 4, 1u));
      s_next = 0;
    }
    __syncthreads();
    if (s_i >= n_big) break;
    const int32_t x = a.big[s_i < n_first ? a.V - 1 - s_i : s_i - n_first];
    const TcInfo ix = a.info[x];
    for (int k = threadIdx.x; k < ix.n; k += NT) {
      const uint32_t r = static_cast<uint32_t>(a.dcol[ix.start + k] - a.base);
      atomicOr(&s_bits[r >> 5], 1u << (r & 31));
    }
    const int64_t b = a.off[x];
    const int deg = static_cast<int>(a.off[x + 1] - b);
    // Neighbours a warp claims at once: at least two claims for every warp.
    const int grab = max(1, min(32, deg / (2 * (NT / 32))));
    __syncthreads();
    unsigned found = 0;
    for (;;) {
      int g = 0;
      if (lane == 0) g = atomicAdd(&s_next, grab);
      g = __shfl_sync(0xffffffffu, g, 0);
      if (g >= deg) break;
      TcInfo iy{0, 0, 0};
      bool take = false;
      if (lane < grab && g + lane < deg) {
        const int32_t y = a.col[b + g + lane];
        iy = a.info[y];
        take = tc_scans(ix.n, x, iy.n, y);
        if (take) work += static_cast<unsigned>(iy.n);
      }
      // Places outside the bitmap (padding, lower ranks) read its last bit,
      // which is never set.
      auto probe = [&](const int4& w) {
        const int32_t id[4] = {w.x, w.y, w.z, w.w};
        uint32_t r[4], x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          r[j] = min(static_cast<uint32_t>(id[j] - a.base), static_cast<uint32_t>(a.bits));
          x[j] = s_bits[r[j] >> 5];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) found += __funnelshift_r(x[j], 0u, r[j]) & 1u;
      };
      // Each half of the warp has the lists of its 16 lanes, 64 entries at a
      // time: half of R-MAT's scanned lists are shorter than that.
      const int half = lane & 16, hl = lane & 15;
      unsigned m = (__ballot_sync(0xffffffffu, take) >> half) & 0xffffu;
      while (__any_sync(0xffffffffu, m != 0)) {
        const int4* p[kTcAhead];
        int n[kTcAhead];
        int4 w[kTcAhead];
#pragma unroll
        for (int j = 0; j < kTcAhead; ++j, m &= m - 1) {
          const int l = half + (m ? __ffs(m) - 1 : 0);
          const int64_t start = __shfl_sync(0xffffffffu, iy.start, l);
          const int ny = __shfl_sync(0xffffffffu, iy.n, l);
          n[j] = m ? ny : 0;
          p[j] = reinterpret_cast<const int4*>(a.dcol + start) + hl;
          if (4 * hl < n[j]) w[j] = __ldg(p[j]);
        }
#pragma unroll
        for (int j = 0; j < kTcAhead; ++j) {
          if (4 * hl < n[j]) probe(w[j]);
          for (int q = 64 + 4 * hl; q < n[j]; q += 64) {
            p[j] += 16;
            probe(__ldg(p[j]));
          }
        }
      }
    }
    cnt += found;
    __syncthreads();
    for (int k = threadIdx.x; k < ix.n; k += NT)
      s_bits[static_cast<uint32_t>(a.dcol[ix.start + k] - a.base) >> 5] = 0u;
  }
  tc_flush<NT>(cnt, work, a.out);
}

// Warp per vertex of a.small: N+(x) in a hash table (linear probing, at most a
// quarter full, kTcPiece entries at a time), the scanned lists of 32
// neighbours as one stream.
__global__ void __launch_bounds__(kTcThreads) tc_warp_kernel(const __grid_constant__ TcArgs a) {
  extern __shared__ __align__(16) int32_t s_tab[];
  const int lane = threadIdx.x & 31;
  int32_t* tab = s_tab + kTcSlots * (threadIdx.x >> 5);
  const int n_small = static_cast<int>(a.ctr[2]);
  unsigned long long cnt = 0, work = 0;
  for (;;) {
    int i0 = 0;
    if (lane == 0) i0 = static_cast<int>(atomicAdd(a.ctr + 5, static_cast<unsigned>(kTcGrab)));
    i0 = __shfl_sync(0xffffffffu, i0, 0);
    if (i0 >= n_small) break;
    for (int i = i0; i < min(i0 + kTcGrab, n_small); ++i) {
      const int32_t x = a.small[i];
      const TcInfo ix = a.info[x];
      const int64_t b = a.off[x];
      const int deg = static_cast<int>(a.off[x + 1] - b);
      for (int p0 = 0; p0 < ix.n; p0 += kTcPiece) {
        const int np = min(kTcPiece, ix.n - p0);
        const int bits = 32 - __clz(max(4 * np - 1, 31));  // 32 slots or more, at most kTcSlots
        for (int k = lane; k < (1 << bits); k += 32) tab[k] = kTcNone;
        __syncwarp();
        const auto slot = [&](int32_t w) { return static_cast<int>((static_cast<uint32_t>(w) * 2654435761u) >> (32 - bits)); };
        const int mask = (1 << bits) - 1;
        for (int k = lane; k < np; k += 32) {
          const int32_t w = a.dcol[ix.start + p0 + k];
          for (int h = slot(w); atomicCAS(tab + h, kTcNone, w) != kTcNone; h = (h + 1) & mask) {
          }
        }
        __syncwarp();
        for (int g = 0; g < deg; g += 32) {
          TcInfo iy{0, 0, 0};
          int len = 0;
          if (g + lane < deg) {
            const int32_t y = a.col[b + g + lane];
            iy = a.info[y];
            if (tc_scans(ix.n, x, iy.n, y)) len = iy.n;
          }
          int pre = len;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += t;
          }
          const int total = __shfl_sync(0xffffffffu, pre, 31);
          pre -= len;
          work += static_cast<unsigned>(len);
          for (int k0 = 0; k0 < total; k0 += 64) {
            int32_t w[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int k = k0 + 32 * j + lane;
              int l = 0;  // (every lane takes part in every shuffle)
#pragma unroll
              for (int sp = 16; sp > 0; sp >>= 1) {
                const int t = __shfl_sync(0xffffffffu, pre, l + sp);
                if (t <= k) l += sp;
              }
              const int lo = __shfl_sync(0xffffffffu, pre, l);
              const int64_t start = __shfl_sync(0xffffffffu, iy.start, l);
              w[j] = k < total ? __ldg(a.dcol + start + (k - lo)) : kTcNone;
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              if (w[j] != kTcNone) {
                for (int h = slot(w[j]);; h = (h + 1) & mask) {
                  const int32_t t = tab[h];
                  if (t == w[j]) ++cnt;
                  if (t == w[j] || t == kTcNone) break;
                }
              }
            }
          }
          __syncwarp();
        }
        __syncwarp();
      }
    }
  }
  tc_flush<kTcThreads>(cnt, work, a.out);
}

struct TcBlock {
  unsigned char* p = nullptr;
  ~TcBlock() { dev_free(&p); }
};

}  // namespace

extern "C" gx_status gx_triangle_count(gx_engine* e, uint64_t* total, gx_run_stats* stats) {
  gx::NvtxRange nvtx_range("gx_triangle_count");
  if (!e || !total) return fail(GX_ERR_INVALID, "gx_triangle_count: bad arguments");
  if (!e->loaded) return fail(GX_ERR_STATE, "gx_triangle_count: no graph loaded");
  if (!e->all_resident)
    return fail(GX_ERR_STATE, "gx_triangle_count: needs every shard resident (no shard-cache budget)");
  GX_CUDA(cudaSetDevice(e->dev));
  BlockBound bound(e->block_bound);
  const int32_t V = e->V;
  cudaStream_t s = e->s_comp;
  cudaEvent_t ev0, ev1, listed, big_done;
  GX_CUDA(cudaEventCreate(&ev0));
  std::unique_ptr<CUevent_st, cudaError_t (*)(cudaEvent_t)> g0(ev0, cudaEventDestroy);
  GX_CUDA(cudaEventCreate(&ev1));
  std::unique_ptr<CUevent_st, cudaError_t (*)(cudaEvent_t)> g1(ev1, cudaEventDestroy);
  GX_CUDA(cudaEventCreateWithFlags(&listed, cudaEventDisableTiming));
  std::unique_ptr<CUevent_st, cudaError_t (*)(cudaEvent_t)> g2(listed, cudaEventDestroy);
  GX_CUDA(cudaEventCreateWithFlags(&big_done, cudaEventDisableTiming));
  std::unique_ptr<CUevent_st, cudaError_t (*)(cudaEvent_t)> g3(big_done, cudaEventDestroy);
  GX_CUDA(cudaEventRecord(ev0, s));
  const bool ranked = V > tc_bits(V);
  int vb = 1;
  while (vb < 31 && (int64_t(1) << vb) < V) ++vb;
  // One block for all arrays; or, without room for it, one for those of a
  // vertex, one that the sort gives back, and the packed lists' own.
  TcBlock block, sort_block, list_block;
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t x = at;
    at += (bytes + 255) & ~size_t(255);
    return x;
  };
  const size_t nv = static_cast<size_t>(V);
  int64_t hist_n = 0, part_n = 0;
  radix_scratch_sizes(V, &hist_n, &part_n);
  const size_t o_deg = place(4 * nv), o_n = place(4 * nv), o_info = place(sizeof(TcInfo) * nv);
  const size_t o_big = place(4 * nv), o_small = place(4 * nv), o_ctr = place(8 * sizeof(unsigned int)),
               o_out = place(2 * sizeof(unsigned long long));
  const size_t o_rank = place(ranked ? 4 * nv : 0), o_sort = at;
  const size_t o_keys = place(ranked ? 16 * nv : 0), o_hist = place(ranked ? 4 * static_cast<size_t>(hist_n) : 0),
               o_offs = place(ranked ? 8 * static_cast<size_t>(hist_n) : 0),
               o_part = place(ranked ? 8 * static_cast<size_t>(part_n) : 0), o_dcol = at;
  place(sizeof(int32_t) * (static_cast<size_t>(e->E) + 4 * nv + 8));
  gx_status room = dev_alloc(&block.p, at);
  const bool packed = room == GX_ERR_OOM;
  unsigned char* sort_at = block.p + o_sort;
  if (packed) {
    room = dev_alloc(&block.p, o_sort);
    if (room == GX_OK && ranked) room = dev_alloc(&sort_block.p, o_dcol - o_sort);
    sort_at = sort_block.p;
  }
  if (room != GX_OK) return room;
  TcArgs a{};
  a.off = e->d_off;
  a.col = e->d_col;
  a.units = e->d_units;
  a.heavy = e->d_heavy;
  a.n_units = static_cast<int32_t>(e->units.size());
  a.chunk = e->caps.chunk;
  a.heavy_deg = e->caps.heavy;
  a.V = V;
  int32_t* deg = reinterpret_cast<int32_t*>(block.p + o_deg);
  a.deg = deg;
  a.n = reinterpret_cast<int32_t*>(block.p + o_n);
  a.info = reinterpret_cast<TcInfo*>(block.p + o_info);
  a.big = reinterpret_cast<int32_t*>(block.p + o_big);
  a.small = reinterpret_cast<int32_t*>(block.p + o_small);
  a.ctr = reinterpret_cast<unsigned int*>(block.p + o_ctr);
  a.out = reinterpret_cast<unsigned long long*>(block.p + o_out);
  a.dcol = packed ? nullptr : reinterpret_cast<int32_t*>(block.p + o_dcol);
  a.bits = static_cast<int32_t>(tc_bits(V));
  a.base = V - a.bits;
  a.mask = vb >= 32 ? 0xffffffffu : (1u << vb) - 1u;
  a.mix = 2654435761u;
  GX_CUDA(cudaMemsetAsync(a.ctr, 0, 8 * sizeof(unsigned int), s));
  GX_CUDA(cudaMemsetAsync(a.out, 0, 2 * sizeof(unsigned long long), s));
  const int grid_v = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(e->n_sm * 8, (V + 255) / 256)));
  unsigned long long* keys = reinterpret_cast<unsigned long long*>(sort_at);
  tc_degree_kernel<<<grid_v, 256, 0, s>>>(e->d_off, V, deg, a.n, ranked ? keys : nullptr, vb);
  if (ranked) {
    unsigned long long* sorted = nullptr;
    GX_TRY(radix_sort_bits(keys, keys + nv, V, vb, 2 * vb, reinterpret_cast<uint32_t*>(sort_at + (o_hist - o_keys)),
                           reinterpret_cast<unsigned long long*>(sort_at + (o_offs - o_keys)),
                           reinterpret_cast<unsigned long long*>(sort_at + (o_part - o_keys)), s, &sorted));
    int32_t* rank = reinterpret_cast<int32_t*>(block.p + o_rank);
    tc_rank_kernel<<<grid_v, 256, 0, s>>>(sorted, (1ull << vb) - 1, V, rank);
    a.rank = rank;
  }
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tc_fill_kernel<kTcSpaced>, kTcThreads, 0);
  const int64_t grid_u = (static_cast<int64_t>(a.n_units) + kTcWarps - 1) / kTcWarps;
  const int grid_fill = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(std::max(1, per_sm) * e->n_sm, grid_u)));
  if (packed) {
    dev_free(&sort_block.p);
    tc_fill_kernel<kTcCount><<<grid_fill, kTcThreads, 0, s>>>(a);
    // The lists' pieces end to end, in a block that the lists' then replaces.
    uint32_t* pieces = reinterpret_cast<uint32_t*>(a.small);
    GX_TRY(dev_alloc(&sort_block.p, 8 * (nv + static_cast<size_t>(part_n))));
    unsigned long long* starts = reinterpret_cast<unsigned long long*>(sort_block.p);
    tc_pieces_kernel<<<grid_v, 256, 0, s>>>(a, pieces);
    GX_TRY(scan_u32(pieces, V, starts, starts + nv, s));
    unsigned long long last = 0;
    uint32_t last_n = 0;
    GX_CUDA(cudaMemcpyAsync(&last, starts + nv - 1, sizeof(last), cudaMemcpyDeviceToHost, s));
    GX_CUDA(cudaMemcpyAsync(&last_n, pieces + nv - 1, sizeof(last_n), cudaMemcpyDeviceToHost, s));
    tc_starts_kernel<<<grid_v, 256, 0, s>>>(a, starts);
    GX_CUDA(cudaMemsetAsync(a.ctr, 0, sizeof(unsigned int), s));  // the units' cursor
    GX_CUDA(cudaStreamSynchronize(s));
    dev_free(&sort_block.p);
    GX_TRY(dev_alloc(&list_block.p, 16 * static_cast<size_t>(last + last_n)));
    a.dcol = reinterpret_cast<int32_t*>(list_block.p);
    tc_fill_kernel<kTcPacked><<<grid_fill, kTcThreads, 0, s>>>(a);
    tc_list_kernel<kTcPacked><<<grid_v, 256, 0, s>>>(a);
  } else {
    tc_fill_kernel<kTcSpaced><<<grid_fill, kTcThreads, 0, s>>>(a);
    tc_list_kernel<kTcSpaced><<<grid_v, 256, 0, s>>>(a);
  }
  GX_CUDA(cudaGetLastError());
  // The CTAs' vertices on the copy stream, the warps' beside them.
  GX_CUDA(cudaEventRecord(listed, s));
  GX_CUDA(cudaStreamWaitEvent(e->s_copy, listed, 0));
  const int smem_cta = (a.bits / 32 + 1) * 4, smem_warp = kTcSlots * kTcWarps * 4;
  // As many CTAs as bitmaps fit an SM, their threads filling it: the fewer
  // threads a vertex has, the fewer wait at its end.
  const int fit = std::max(1, (220 * 1024) / (smem_cta + 2048));
  void (*cta)(TcArgs) = fit >= 6 ? tc_cta_kernel<256> : fit >= 2 ? tc_cta_kernel<512> : tc_cta_kernel<1024>;
  const int cta_threads = fit >= 6 ? 256 : fit >= 2 ? 512 : 1024;
  GX_CUDA(allow_dynamic_smem(e->dev, reinterpret_cast<const void*>(cta)));
  GX_CUDA(allow_dynamic_smem(e->dev, reinterpret_cast<const void*>(tc_warp_kernel)));
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cta, cta_threads, smem_cta);
  cta<<<std::max(1, per_sm) * e->n_sm, cta_threads, smem_cta, e->s_copy>>>(a);
  GX_CUDA(cudaGetLastError());
  GX_CUDA(cudaEventRecord(big_done, e->s_copy));
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tc_warp_kernel, kTcThreads, smem_warp);
  tc_warp_kernel<<<std::max(1, per_sm) * e->n_sm, kTcThreads, smem_warp, s>>>(a);
  GX_CUDA(cudaGetLastError());
  GX_CUDA(cudaStreamWaitEvent(s, big_done, 0));
  unsigned long long res[2] = {0, 0};
  GX_CUDA(cudaMemcpyAsync(res, a.out, sizeof(res), cudaMemcpyDeviceToHost, s));
  GX_CUDA(cudaEventRecord(ev1, s));
  GX_CUDA(cudaEventSynchronize(ev1));
  float ms = 0;
  cudaEventElapsedTime(&ms, ev0, ev1);
  *total = res[0];
  if (stats) {
    *stats = gx_run_stats{};
    stats->iterations = 1;
    stats->edges_scanned = static_cast<int64_t>(res[1]);
    stats->ms_total = ms;
    stats->ms_compute = ms;
    stats->kernel_launches = (ranked ? 6 : 5) + (packed ? 3 : 0);  // the sort's and scan's passes not counted
  }
  return GX_OK;
}
