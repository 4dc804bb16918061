// ROI extraction: bidirectional level-synchronous BFS, as
// ROIExtractor.extract_roi_bfs (UPF:1636-1734).
//
// Marks live in one byte per node (0 unseen, 1 src wave, 2 dst wave, 3 both)
// and are updated with a 32-bit atomicOr on the containing word: OR-ing the
// wave's mark reproduces the reference's three cases exactly (unseen -> mark;
// other wave or both -> 3, which ends the expansion; own mark -> unchanged),
// and the set of marked nodes after each step does not depend on the order in
// which the frontier is processed.  The ROI is then the marked nodes in
// ascending id order (np.where), produced by an order-preserving compaction.
#include <algorithm>
#include <climits>
#include <mutex>
#include <string>

#include "common.cuh"

namespace {

constexpr int BFS_THREADS = 1024;

__device__ __forceinline__ unsigned or_mark(uint8_t *seen, int v, unsigned mark) {
  unsigned *word = (unsigned *)(seen + (v & ~3));
  const int sh = (v & 3) * 8;
  const unsigned old = atomicOr(word, mark << sh);
  return (old >> sh) & 0xffu;
}

struct BfsCtl {
  int total;   // marked nodes
  int depth;
  int met;
  int err;
};

// One CTA runs the whole expansion (depth <= 150 in the reference).
__global__ void __launch_bounds__(BFS_THREADS) roi_bfs_kernel(
    const int32_t *__restrict__ indptr, const int32_t *__restrict__ indices, int32_t N,
    int32_t src, int32_t dst, int32_t max_depth, int32_t max_nodes, uint8_t *seen,
    int32_t *qs0, int32_t *qs1, int32_t *qd0, int32_t *qd1, BfsCtl *ctl) {
  __shared__ int s_next;
  __shared__ int s_met;
  __shared__ int s_err;
  int n_src = 1, n_dst = 1;
  int32_t *qs = qs0, *qs_next = qs1, *qd = qd0, *qd_next = qd1;
  int total;
  if (threadIdx.x == 0) {
    seen[src] = 1;
    seen[dst] = 2;  // src == dst leaves mark 2, as the reference does
    qs[0] = src;
    qd[0] = dst;
    s_met = 0;
    s_err = 0;
  }
  total = (src == dst) ? 1 : 2;
  __syncthreads();
  int depth = 0;
  bool met = false;
  const double limit = (double)max_nodes * 1.5;
  while (depth < max_depth && (n_src > 0 || n_dst > 0) && !met) {
    for (int wave = 0; wave < 2; ++wave) {
      if (wave == 1 && met) break;
      const unsigned mark = wave == 0 ? 1u : 2u;
      const int n = wave == 0 ? n_src : n_dst;
      const int32_t *q = wave == 0 ? qs : qd;
      int32_t *qn = wave == 0 ? qs_next : qd_next;
      if (threadIdx.x == 0) s_next = 0;
      __syncthreads();
      bool met_local = false;
      for (int base = 0; base < n; base += BFS_THREADS) {
        const int i = base + threadIdx.x;
        int beg = 0, end = 0;
        if (i < n) {
          const int u = q[i];
          beg = indptr[u];
          end = indptr[u + 1];
        }
        const int deg = end - beg;
        const int maxdeg = __reduce_max_sync(ORSP_FULL_MASK, deg);
        for (int k = 0; k < maxdeg; ++k) {
          bool push = false;
          int v = 0;
          if (k < deg) {
            v = indices[beg + k];
            const unsigned old = or_mark(seen, v, mark);
            if (old == 0) push = true;
            else if (old != mark) met_local = true;
          }
          const unsigned m = __ballot_sync(ORSP_FULL_MASK, push);
          if (m) {
            const int lane = threadIdx.x & 31;
            const int leader = __ffs(m) - 1;
            int basei = 0;
            if (lane == leader) basei = atomicAdd(&s_next, __popc(m));
            basei = __shfl_sync(ORSP_FULL_MASK, basei, leader);
            if (push) {
              const int idx = basei + __popc(m & lanemask_lt());
              if (idx < N) qn[idx] = v; else s_err = 1;
            }
          }
        }
      }
      if (met_local) s_met = 1;
      __syncthreads();
      const int nn = s_next;
      total += nn;
      met = s_met != 0;
      if (wave == 0) {
        n_src = nn;
        int32_t *t = qs; qs = qs_next; qs_next = t;
      } else {
        n_dst = nn;
        int32_t *t = qd; qd = qd_next; qd_next = t;
      }
      __syncthreads();  // s_next is reset by the next wave
    }
    ++depth;
    if ((double)total > limit) break;
  }
  if (threadIdx.x == 0) {
    ctl->total = total;
    ctl->depth = depth;
    ctl->met = met ? 1 : 0;
    ctl->err = s_err;
  }
}

constexpr int CMP_THREADS = 512;
constexpr int CMP_ITEMS = 16;  // nodes per thread per tile
constexpr int CMP_TILE = CMP_THREADS * CMP_ITEMS;

__device__ __forceinline__ int block_excl_scan(int v, int *smem_warp, int *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(ORSP_FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem_warp[w] = x;
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    int s = lane < nw ? smem_warp[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(ORSP_FULL_MASK, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) smem_warp[lane] = s;
  }
  __syncthreads();
  const int warp_off = w > 0 ? smem_warp[w - 1] : 0;
  *total = smem_warp[(blockDim.x >> 5) - 1];
  const int r = warp_off + x - v;
  __syncthreads();
  return r;
}

// Pass 1: marked-node count per tile.
__global__ void __launch_bounds__(CMP_THREADS) count_tiles_kernel(const uint8_t *seen, int32_t N,
                                                                  int32_t *tile_cnt) {
  __shared__ int sw[32];
  const int64_t t0 = (int64_t)blockIdx.x * CMP_TILE;
  int c = 0;
  for (int j = 0; j < CMP_ITEMS; ++j) {
    const int64_t v = t0 + (int64_t)j * CMP_THREADS + threadIdx.x;
    if (v < N && seen[v]) ++c;
  }
  int tot;
  block_excl_scan(c, sw, &tot);
  if (threadIdx.x == 0) tile_cnt[blockIdx.x] = tot;
}

// Pass 2: exclusive scan of tile counts (one block, serial over chunks).
__global__ void __launch_bounds__(1024) scan_tiles_kernel(int32_t *tile_cnt, int32_t ntiles,
                                                          int32_t *total_out) {
  __shared__ int sw[32];
  int carry = 0;
  for (int base = 0; base < ntiles; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < ntiles ? tile_cnt[i] : 0;
    int tot;
    const int ex = block_excl_scan(v, sw, &tot);
    if (i < ntiles) tile_cnt[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) *total_out = carry;
}

// Pass 3: write marked ids in ascending order.  Within a tile, node
// t0 + j*THREADS + tid is visited in (j, tid) order, which is ascending.
__global__ void __launch_bounds__(CMP_THREADS) write_tiles_kernel(const uint8_t *seen, int32_t N,
                                                                  const int32_t *tile_off,
                                                                  int32_t *out) {
  __shared__ int sw[32];
  const int64_t t0 = (int64_t)blockIdx.x * CMP_TILE;
  int base = tile_off[blockIdx.x];
  for (int j = 0; j < CMP_ITEMS; ++j) {
    const int64_t v = t0 + (int64_t)j * CMP_THREADS + threadIdx.x;
    const int f = (v < N && seen[v]) ? 1 : 0;
    int tot;
    const int ex = block_excl_scan(f, sw, &tot);
    if (f) out[base + ex] = (int32_t)v;
    base += tot;
  }
}

// Truncation to max_nodes with the reference's must-keep list, as
// extract_roi_bfs does it (UPF:1700-1731): must_keep = [src, dst] followed by
// the keep nodes not already in it (list order); the ones missing from the
// ROI are appended after the ascending part in that order; then, if the list
// is longer than max_nodes, the k-th must-keep position (ascending) at or
// past max_nodes is swapped with position k (UPF:1705-1722) and the list is
// cut to max_nodes.  Called by a whole block after the list is written: one
// thread per must-keep node drops repeats and searches the ascending part, so
// the block pays one binary search (about 10 us of dependent loads) instead
// of one thread's scan of the list (617 us for 75 K nodes).  MAX_KEEP bounds
// the list (checked on the host).  Returns the length on thread 0.
constexpr int MAX_KEEP = 256;
__device__ int truncate_block(int32_t *roi, int32_t n0, int32_t max_nodes, int32_t src, int32_t dst,
                              const int32_t *keep, int32_t nkeep) {
  __shared__ int32_t s_mk[MAX_KEEP + 2], s_pos[MAX_KEEP + 2];
  if (nkeep == 0 && n0 <= max_nodes) return n0;  // (source and target are marked, so nothing is appended)
  const int nc = nkeep + 2;
  for (int j = threadIdx.x; j < nc; j += blockDim.x) s_mk[j] = j == 0 ? src : j == 1 ? dst : keep[j - 2];
  __syncthreads();
  for (int j = threadIdx.x; j < nc; j += blockDim.x) {
    const int32_t v = s_mk[j];
    bool dup = false;
    for (int i = 0; i < j; ++i) dup |= s_mk[i] == v;
    int lo = 0, hi = dup ? 0 : n0;  // first position with roi[p] >= v
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (__ldcg(&roi[mid]) < v) lo = mid + 1;
      else hi = mid;
    }
    s_pos[j] = dup ? -2 : (lo < n0 && __ldcg(&roi[lo]) == v) ? lo : -1;
  }
  __syncthreads();
  if (threadIdx.x != 0) return 0;
  int n = n0, nmk = 0;
  for (int j = 0; j < nc; ++j) {
    int p = s_pos[j];
    if (p == -2) continue;
    if (p == -1) {
      roi[n] = s_mk[j];
      p = n++;
    }
    s_pos[nmk++] = p;
  }
  if (n <= max_nodes) return n;
  // positions in ascending order (insertion sort of a short list)
  for (int a = 1; a < nmk; ++a) {
    const int32_t t = s_pos[a];
    int b = a - 1;
    while (b >= 0 && s_pos[b] > t) {
      s_pos[b + 1] = s_pos[b];
      --b;
    }
    s_pos[b + 1] = t;
  }
  for (int k = 0; k < nmk; ++k) {
    const int p = s_pos[k];
    if (p >= max_nodes) {
      const int32_t t = roi[p];
      roi[p] = roi[k];
      roi[k] = t;
    }
  }
  return max_nodes;
}

__global__ void truncate_kernel(int32_t *roi, const int32_t *count_in, int32_t max_nodes, int32_t src, int32_t dst,
                                const int32_t *keep, int32_t nkeep, int32_t *count_out) {
  const int cnt = truncate_block(roi, *count_in, max_nodes, src, dst, keep, nkeep);
  if (threadIdx.x == 0) *count_out = cnt;
}

// The expansion on a uniform lattice (Graph::lat_uniform), one CTA.
//
// A level of the wave front is a chain of dependent accesses, about 100 to
// 300 levels per ROI, so the kernel is bound by the latency of one level, not
// by bandwidth.  roi_bfs_kernel above pays four round trips to L2 per level
// (queue, row pointer, neighbour list, mark), the last one once per neighbour:
// about 11 us.  Here the neighbours follow from the node's coordinates, the
// queues hold packed coordinates in shared memory, and the marks (2 bits per
// node) are in shared memory too when the lattice fits (SM), so a level makes
// no trip to L2 and the marked nodes are compacted from shared memory by the
// same launch.  Larger lattices keep their marks in global memory, up to
// eight neighbours' marks in flight per node.  A queue that runs full sets
// err; the host then runs the general kernel.  Semantics of the marks and of
// the two waves as in roi_bfs_kernel.  (200 x 200 x 6 column-via
// lattice, 75 K marked nodes: 1 295 us with roi_bfs_kernel, 324 us here.)
struct LatBfs {
  int32_t nx, ny, nz, N;
  int32_t src, dst;      // node ids
  int32_t psrc, pdst;    // packed coordinates x | y << 12 | z << 24
  int32_t max_depth, max_nodes;
  int32_t qcap;
  const int32_t *keep;
  int32_t nkeep;
  uint8_t *seen;         // marks in global memory (!SM), zero on entry
  int32_t *roi, *count;  // SM: the list and its length
  BfsCtl *ctl;
  int8_t axis[64];
  uint64_t via_to[64];
};

template <bool SM>
__global__ void __launch_bounds__(BFS_THREADS, 1) roi_bfs_lattice_kernel(const __grid_constant__ LatBfs p) {
  extern __shared__ __align__(16) uint32_t s_dyn[];
  __shared__ int s_next, s_met, s_err;
  __shared__ int s_warp[32];
  int32_t *qb[3];  // the two waves' fronts and the one being built
  for (int i = 0; i < 3; ++i) qb[i] = (int32_t *)s_dyn + (int64_t)i * p.qcap;
  uint32_t *marks = s_dyn + (int64_t)3 * p.qcap;
  const int nwords = (p.N + 15) >> 4;
  if (SM)
    for (int i = threadIdx.x; i < nwords; i += BFS_THREADS) marks[i] = 0;
  __syncthreads();
  auto mark_node = [&](int32_t v, unsigned m) -> unsigned {
    if (SM) {
      const int sh = (v & 15) * 2;
      return (atomicOr(&marks[v >> 4], m << sh) >> sh) & 3u;
    }
    return or_mark(p.seen, v, m);
  };
  int cnt[2] = {1, 1};
  int32_t *front[2] = {qb[0], qb[1]}, *spare = qb[2];
  if (threadIdx.x == 0) {
    if (p.src != p.dst) mark_node(p.src, 1u);
    mark_node(p.dst, 2u);  // src == dst leaves mark 2, as the reference does
    front[0][0] = p.psrc;
    front[1][0] = p.pdst;
    s_met = 0;
    s_err = 0;
  }
  int total = (p.src == p.dst) ? 1 : 2;
  int depth = 0;
  bool met = false;
  const double limit = (double)p.max_nodes * 1.5;
  const int32_t plane = p.nx * p.ny;
  while (depth < p.max_depth && (cnt[0] > 0 || cnt[1] > 0) && !met) {
#pragma unroll
    for (int wave = 0; wave < 2; ++wave) {
      if (wave == 1 && met) break;
      const unsigned mark = wave == 0 ? 1u : 2u;
      if (threadIdx.x == 0) s_next = 0;
      __syncthreads();
      bool met_local = false;
      const int n = cnt[wave];
      for (int i = threadIdx.x; i < n; i += BFS_THREADS) {
        const int32_t pk = front[wave][i];
        const int32_t x = pk & 4095, y = (pk >> 12) & 4095, z = pk >> 24;
        const int32_t id = (z * p.ny + y) * p.nx + x;
        const int ax = p.axis[z];
        const int32_t c = ax == 1 ? x : y, cmax = ax == 1 ? p.nx - 1 : p.ny - 1;
        const int32_t step = ax == 1 ? 1 : p.nx, pstep = ax == 1 ? 1 : 4096;
        uint64_t vm = p.via_to[z];
        bool planar = ax != 0;
        while (planar || vm) {
          int32_t nid[8], npk[8];
          bool has[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            has[k] = false;
            nid[k] = npk[k] = 0;
            if (k < 2 && planar) {
              has[k] = k == 0 ? c > 0 : c < cmax;
              nid[k] = k == 0 ? id - step : id + step;
              npk[k] = k == 0 ? pk - pstep : pk + pstep;
            } else if (vm) {
              const int t = __ffsll((long long)vm) - 1;
              vm &= vm - 1;
              has[k] = true;
              nid[k] = id + (t - z) * plane;
              npk[k] = (pk & 0xffffff) | (t << 24);
            }
          }
          planar = false;
          unsigned old[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) old[k] = has[k] ? mark_node(nid[k], mark) : mark;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (old[k] == 0) {
              const int idx = atomicAdd(&s_next, 1);
              if (idx < p.qcap) spare[idx] = npk[k];
              else s_err = 1;
            } else if (old[k] != mark) {
              met_local = true;
            }
          }
        }
      }
      if (met_local) s_met = 1;
      __syncthreads();
      const int nn = s_next;
      met = s_met != 0;
      const bool full = s_err != 0;
      __syncthreads();  // s_next is reset by the next wave
      total += nn;
      cnt[wave] = nn;
      int32_t *t = front[wave];
      front[wave] = spare;
      spare = t;
      if (full) {
        if (threadIdx.x == 0) {
          p.ctl->err = 1;
          if (SM) *p.count = 0;  // no list: nothing goes to global_to_roi
        }
        return;
      }
    }
    ++depth;
    if ((double)total > limit) break;
  }
  if (threadIdx.x == 0) {
    p.ctl->total = total;
    p.ctl->depth = depth;
    p.ctl->met = met ? 1 : 0;
    p.ctl->err = 0;
  }
  if (!SM) return;
  // the marked nodes in ascending order: each warp takes a contiguous range
  // of mark words, lane after lane
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per = (((nwords + 31) / 32) + 31) & ~31;
  const int w0 = w * per, w1 = min(nwords, w0 + per);
  int mine = 0;
  for (int i = w0 + lane; i < w1; i += 32) mine += __popc((marks[i] | (marks[i] >> 1)) & 0x55555555u);
  mine = __reduce_add_sync(ORSP_FULL_MASK, mine);
  if (lane == 0) s_warp[w] = mine;
  __syncthreads();
  if (w == 0) {
    const int v = s_warp[lane];
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(ORSP_FULL_MASK, x, o);
      if (lane >= o) x += y;
    }
    s_warp[lane] = x - v;
    if (lane == 31) s_next = x;
  }
  __syncthreads();
  int pos = s_warp[w];
  for (int b = w0; b < w1; b += 32) {
    uint32_t m = 0;
    if (b + lane < w1) m = (marks[b + lane] | (marks[b + lane] >> 1)) & 0x55555555u;
    const int c = __popc(m);
    int x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(ORSP_FULL_MASK, x, o);
      if (lane >= o) x += y;
    }
    int at = pos + x - c;
    while (m) {
      const int j = __ffs(m) - 1;
      m &= m - 1;
      __stcg(&p.roi[at++], (b + lane) * 16 + (j >> 1));
    }
    pos += __shfl_sync(ORSP_FULL_MASK, x, 31);
  }
  __syncthreads();
  const int n = truncate_block(p.roi, s_next, p.max_nodes, p.src, p.dst, p.keep, p.nkeep);
  if (threadIdx.x == 0) *p.count = n;
}

// The same expansion on bit sets, where six of them fit in shared memory: of
// each wave the marks, the front and the one being built, a bit per node, rows
// of whole words.
//
// The queues above take a node's neighbours one by one, an atomic on shared
// memory each, and a level of a few hundred nodes two to three microseconds.
// Here a thread takes 32 nodes of a row and ORs what can step into them: the
// word shifted by one either way (x-layers) or the rows above and below
// (y-layers), and the layers whose vias end here.  A thread takes whole rows and
// stays with one layer, so that what depends on the layer is in registers and all
// loads of a word go out together (a thread per column of layers, with one OR for
// the vias of all: 335 us; words dealt out one by one: 264, and 238 with the
// layer fixed).  Only one thread writes a word, so there are no atomics, and one
// barrier per wave and level.  Each wave works on the box that its front can
// have reached; the box only grows, so every level overwrites what the buffer
// held two levels before.  Sets of marks as in roi_bfs_kernel: an unseen node
// joins the front, a node of the other wave ends the expansion.
// (200 x 200 x 6 column-via lattice, 75 K marked nodes, 80 levels: queues 335 us,
// bit sets 215 us, 1 us per wave and level at first and 1.8 where the box is 120
// wide.)
__global__ void __launch_bounds__(BFS_THREADS, 1) roi_bfs_bits_kernel(const __grid_constant__ LatBfs p, int32_t wpr) {
  extern __shared__ __align__(16) uint32_t s_dyn[];
  __shared__ uint32_t s_cnt[2][32];  // per warp: marked nodes, and met from bit 24, of this level and the last
  __shared__ int s_warp[32];
  __shared__ int s_total;
  // rows lie an odd number of words apart: neighbouring threads take
  // neighbouring rows, from distinct banks
  const int32_t pitch = wpr | 1, lw = p.ny * pitch, nwords = p.nz * lw;  // words of a layer, of a set
  uint32_t *const seen[2] = {s_dyn, s_dyn + nwords};
  uint32_t *front[2] = {s_dyn + 2 * nwords, s_dyn + 4 * nwords}, *next[2] = {s_dyn + 3 * nwords, s_dyn + 5 * nwords};
  for (int i = threadIdx.x; i < 6 * nwords; i += BFS_THREADS) s_dyn[i] = 0;
  // this thread's layer, whole warps per layer where they suffice, and its
  // first row
  const int per_z = p.nz <= 32 ? BFS_THREADS / p.nz & ~31 : BFS_THREADS / p.nz;
  const int z = min((int)threadIdx.x / per_z, p.nz - 1);
  int32_t first = (int)threadIdx.x < per_z * p.nz ? (int)threadIdx.x - z * per_z : INT_MAX >> 1;
  const int ax = p.axis[z];
  uint64_t from = 0;  // layers whose vias lead to it
  for (int t = 0; t < p.nz; ++t) from |= (uint64_t)((p.via_to[t] >> z) & 1) << t;
  if (!ax && !from) first = INT_MAX >> 1;  // nothing enters this layer
  __syncthreads();
  int32_t lo_x[2], hi_x[2], lo_y[2], hi_y[2];  // cells that each wave's front can hold
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const int32_t pk = w == 0 ? p.psrc : p.pdst;
    lo_x[w] = hi_x[w] = pk & 4095;
    lo_y[w] = hi_y[w] = (pk >> 12) & 4095;
    if (threadIdx.x == 0) {
      const int32_t i = (pk >> 24) * lw + lo_y[w] * pitch + (lo_x[w] >> 5);
      const uint32_t bit = 1u << (lo_x[w] & 31);
      front[w][i] = bit;
      if (w == 1 || p.src != p.dst) seen[w][i] = bit;  // src == dst leaves mark 2, as the reference does
    }
  }
  __syncthreads();
  int cnt[2] = {1, 1}, total = (p.src == p.dst) ? 1 : 2, depth = 0, slot = 0;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  bool met = false;
  const double limit = (double)p.max_nodes * 1.5;
  const uint32_t tail = p.nx & 31 ? (1u << (p.nx & 31)) - 1u : ~0u;  // nodes of a row's last word
  while (depth < p.max_depth && (cnt[0] > 0 || cnt[1] > 0) && !met) {
#pragma unroll
    for (int wave = 0; wave < 2; ++wave) {
      if (wave == 1 && met) break;
      lo_x[wave] = max(lo_x[wave] - 1, 0), hi_x[wave] = min(hi_x[wave] + 1, p.nx - 1);
      lo_y[wave] = max(lo_y[wave] - 1, 0), hi_y[wave] = min(hi_y[wave] + 1, p.ny - 1);
      const int32_t w0 = lo_x[wave] >> 5, nw = (hi_x[wave] >> 5) - w0 + 1, y0 = lo_y[wave], nr = hi_y[wave] - y0 + 1;
      const uint32_t *const f = front[wave] + z * lw;
      uint32_t *const to = next[wave] + z * lw, *const own = seen[wave] + z * lw, *const other = seen[wave ^ 1] + z * lw;
      uint32_t sum = 0, hit = 0;
      for (int32_t y = y0 + first; y < y0 + nr; y += per_z) {
        int32_t at = y * pitch + w0;
        uint32_t l = w0 > 0 ? f[at - 1] : 0u, c = f[at];
        for (int32_t w = w0; w < w0 + nw; ++w, ++at) {
          // all loads together
          const uint32_t r = w + 1 < wpr ? f[at + 1] : 0u, mine = own[at], theirs = other[at];
          uint32_t u = 0, d = 0;
          if (ax == 2) {
            if (y > 0) u = f[at - pitch];
            if (y + 1 < p.ny) d = f[at + pitch];
          }
          uint32_t in = 0;
          for (int t = 0; t < p.nz; t += 8) {
            const uint32_t m = (uint32_t)(from >> t);
            uint32_t q[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) q[k] = (m >> k) & 1u ? f[at + (t + k - z) * lw] : 0u;
#pragma unroll
            for (int k = 0; k < 8; ++k) in |= q[k];
          }
          in |= u | d;
          if (ax == 1) in |= (c << 1) | (l >> 31) | (c >> 1) | (r << 31);
          if (w == wpr - 1) in &= tail;
          const uint32_t fresh = in & ~mine & ~theirs;
          own[at] = mine | in;
          to[at] = fresh;
          sum += __popc(fresh);
          hit |= in & theirs;
          l = c;
          c = r;
        }
      }
      // (a slot per warp: with 32 atomics on one word 225 us, now 215)
      sum = __reduce_add_sync(ORSP_FULL_MASK, sum + (hit ? 1u << 24 : 0u));
      if (lane == 0) s_cnt[slot][wp] = sum;
      __syncthreads();
      const uint32_t got = s_cnt[slot][lane];
      slot ^= 1;
      cnt[wave] = (int)__reduce_add_sync(ORSP_FULL_MASK, got & 0xffffffu);
      met = __any_sync(ORSP_FULL_MASK, got >> 24);
      total += cnt[wave];
      uint32_t *const t = front[wave];
      front[wave] = next[wave];
      next[wave] = t;
    }
    ++depth;
    if ((double)total > limit) break;
  }
  if (threadIdx.x == 0) {
    p.ctl->total = total;
    p.ctl->depth = depth;
    p.ctl->met = met ? 1 : 0;
    p.ctl->err = 0;
  }
  // the marked nodes in ascending order: each warp takes a range of words, 32
  // at a time, and writes a word's nodes side by side
  const int per = (((nwords + 31) / 32) + 31) & ~31;
  const int b0 = wp * per, b1 = min(nwords, b0 + per);
  int mine = 0;
  for (int i = b0 + lane; i < b1; i += 32) mine += __popc(seen[0][i] | seen[1][i]);
  mine = __reduce_add_sync(ORSP_FULL_MASK, mine);
  if (lane == 0) s_warp[wp] = mine;
  __syncthreads();
  if (wp == 0) {
    const int v = s_warp[lane];
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(ORSP_FULL_MASK, x, o);
      if (lane >= o) x += y;
    }
    s_warp[lane] = x - v;
    if (lane == 31) s_total = x;
  }
  __syncthreads();
  int pos = s_warp[wp];
  for (int b = b0; b < b1; b += 32) {
    const int i = b + lane, row = i / pitch;
    const uint32_t m = i < b1 ? seen[0][i] | seen[1][i] : 0u;
    const int32_t id = row * p.nx + (i - row * pitch) * 32;
    for (uint32_t left = __ballot_sync(ORSP_FULL_MASK, m != 0); left; left &= left - 1) {
      const int k = __ffs(left) - 1;
      const uint32_t mk = __shfl_sync(ORSP_FULL_MASK, m, k);
      const int32_t idk = __shfl_sync(ORSP_FULL_MASK, id, k);
      if ((mk >> lane) & 1u) __stcg(&p.roi[pos + __popc(mk & lanemask_lt())], idk + lane);
      pos += __popc(mk);
    }
  }
  __syncthreads();
  const int n = truncate_block(p.roi, s_total, p.max_nodes, p.src, p.dst, p.keep, p.nkeep);
  if (threadIdx.x == 0) *p.count = n;
}

__global__ void fill_i32_kernel(int32_t *p, int64_t n, int32_t v) {
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += s) p[i] = v;
}

__global__ void scatter_g2r_kernel(const int32_t *roi, const int32_t *count, int32_t *g2r) {
  const int n = *count;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    g2r[roi[i]] = i;
}

// global_to_roi for an inclusive box: -1 everywhere, local id inside
// (local ids ascend with global ids, so ROI rank = global order).
__global__ void box_map_kernel(int32_t *g2r, int64_t N, int32_t nx, int32_t ny, int32_t x0,
                               int32_t x1, int32_t y0, int32_t y1, int32_t z0, int32_t z1) {
  const int64_t plane = (int64_t)nx * ny;
  const int32_t W = x1 - x0 + 1, H = y1 - y0 + 1;
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < N; v += s) {
    const int32_t z = (int32_t)(v / plane);
    const int64_t r = v - (int64_t)z * plane;
    const int32_t y = (int32_t)(r / nx), x = (int32_t)(r - (int64_t)y * nx);
    int32_t id = -1;
    if (x >= x0 && x <= x1 && y >= y0 && y <= y1 && z >= z0 && z <= z1)
      id = ((z - z0) * H + (y - y0)) * W + (x - x0);
    g2r[v] = id;
  }
}

}  // namespace

using namespace orsp;

extern "C" int orsp_roi_box_map(orsp_graph *g, const int32_t *box_h, int32_t *g2r_d,
                                uintptr_t stream) {
  if (!g || !box_h || !g2r_d) { set_error("roi_box_map: NULL argument"); return ORSP_ERR_ARG; }
  if (g->nx <= 0) { set_error("roi_box_map: graph has no lattice dims"); return ORSP_ERR_ARG; }
  const int32_t *b = box_h;
  if (b[0] < 0 || b[2] < 0 || b[4] < 0 || b[1] >= g->nx || b[3] >= g->ny || b[5] >= g->nz ||
      b[1] < b[0] || b[3] < b[2] || b[5] < b[4]) {
    set_error("roi_box_map: box outside the lattice or empty");
    return ORSP_ERR_ARG;
  }
  ORSP_CUDA(cudaSetDevice(g->device));
  const int64_t N = g->N;
  box_map_kernel<<<(int)std::min<int64_t>((N + 255) / 256, 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      g2r_d, N, g->nx, g->ny, b[0], b[1], b[2], b[3], b[4], b[5]);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

static int roi_bfs_impl(orsp_graph *g, int32_t src, int32_t dst, int32_t max_depth, int32_t max_nodes,
                        const int32_t *keep_d, int32_t nkeep, int32_t *roi_nodes_d, int32_t *g2r_d,
                        int32_t *roi_count_h, uintptr_t stream);

extern "C" int orsp_roi_bfs(orsp_graph *g, int32_t src, int32_t dst, int32_t max_depth,
                            int32_t max_nodes, int32_t *roi_nodes_d, int32_t *g2r_d,
                            int32_t *roi_count_h, uintptr_t stream) {
  return roi_bfs_impl(g, src, dst, max_depth, max_nodes, nullptr, 0, roi_nodes_d, g2r_d, roi_count_h, stream);
}

extern "C" int orsp_roi_bfs_keep(orsp_graph *g, int32_t src, int32_t dst, int32_t max_depth,
                                 int32_t max_nodes, const int32_t *keep_d, int32_t nkeep,
                                 int32_t *roi_nodes_d, int32_t *g2r_d, int32_t *roi_count_h,
                                 uintptr_t stream) {
  if (nkeep < 0 || nkeep > MAX_KEEP || (nkeep > 0 && !keep_d)) {
    set_error("roi_bfs_keep: nkeep must be 0.." + std::to_string(MAX_KEEP) + " with a keep list");
    return ORSP_ERR_ARG;
  }
  return roi_bfs_impl(g, src, dst, max_depth, max_nodes, keep_d, nkeep, roi_nodes_d, g2r_d, roi_count_h, stream);
}

// Compaction of the marks into the ascending list, and its truncation.
static int compact_and_truncate(const uint8_t *seen, int32_t N, int32_t *tiles, int32_t *misc, int32_t max_nodes,
                                int32_t src, int32_t dst, const int32_t *keep_d, int32_t nkeep, int32_t *roi_nodes_d,
                                cudaStream_t st) {
  const int ntiles = (int)(((int64_t)N + CMP_TILE - 1) / CMP_TILE);
  count_tiles_kernel<<<ntiles, CMP_THREADS, 0, st>>>(seen, N, tiles);
  ORSP_CUDA(cudaGetLastError());
  scan_tiles_kernel<<<1, 1024, 0, st>>>(tiles, ntiles, misc + 4);
  ORSP_CUDA(cudaGetLastError());
  write_tiles_kernel<<<ntiles, CMP_THREADS, 0, st>>>(seen, N, tiles, roi_nodes_d);
  ORSP_CUDA(cudaGetLastError());
  truncate_kernel<<<1, 128, 0, st>>>(roi_nodes_d, misc + 4, max_nodes, src, dst, keep_d, nkeep, misc + 5);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

static int write_g2r(const int32_t *roi_nodes_d, const int32_t *count_d, int64_t N, int32_t *g2r_d, cudaStream_t st) {
  fill_i32_kernel<<<std::min<int64_t>((N + 255) / 256, 4096), 256, 0, st>>>(g2r_d, N, -1);
  ORSP_CUDA(cudaGetLastError());
  scatter_g2r_kernel<<<std::min<int64_t>((N + 255) / 256, 1024), 256, 0, st>>>(roi_nodes_d, count_d, g2r_d);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

// Shared memory of the lattice expansion: a front on a lattice of moderate
// depth holds up to a few thousand nodes; with the marks in shared memory too
// the queues get 3 584 entries each, which leaves room for the marks of
// 745 000 nodes, otherwise as many as fit.
static constexpr int32_t kBfsSmem = 224 * 1024;
static constexpr int32_t kBfsQueue = 3584;

static int roi_bfs_impl(orsp_graph *g, int32_t src, int32_t dst, int32_t max_depth, int32_t max_nodes,
                        const int32_t *keep_d, int32_t nkeep, int32_t *roi_nodes_d, int32_t *g2r_d,
                        int32_t *roi_count_h, uintptr_t stream) {
  if (!g || !roi_nodes_d || !roi_count_h) { set_error("roi_bfs: NULL argument"); return ORSP_ERR_ARG; }
  if (src < 0 || src >= g->N || dst < 0 || dst >= g->N) { set_error("roi_bfs: src/dst out of range"); return ORSP_ERR_ARG; }
  if (max_nodes <= 0) { set_error("roi_bfs: max_nodes must be > 0"); return ORSP_ERR_ARG; }
  ORSP_CUDA(cudaSetDevice(g->device));
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t N = g->N;
  const int ntiles = (int)((N + CMP_TILE - 1) / CMP_TILE);
  // scratch: seen (N bytes, rounded to 16) | 4 queues of N | tiles | ctl
  const size_t seen_b = ((size_t)N + 15) & ~(size_t)15;
  const size_t q_b = (size_t)N * 4;
  const size_t tiles_b = ((size_t)ntiles * 4 + 15) & ~(size_t)15;
  const size_t total_b = seen_b + 4 * q_b + tiles_b + 64;
  int rc = ensure_scratch(g, total_b);
  if (rc) return rc;
  char *base = (char *)g->scratch;
  uint8_t *seen = (uint8_t *)base;
  int32_t *q[4];
  for (int i = 0; i < 4; ++i) q[i] = (int32_t *)(base + seen_b + i * q_b);
  int32_t *tiles = (int32_t *)(base + seen_b + 4 * q_b);
  int32_t *misc = (int32_t *)(base + seen_b + 4 * q_b + tiles_b);  // [0..3] BfsCtl, [4] total, [5] count
  BfsCtl *ctl = (BfsCtl *)misc;
  const int32_t *h = (const int32_t *)g->pinned;

  // uniform lattices (12-bit coordinates in the queues): the lattice
  // expansion, then, if a queue ran full, the general one
  const bool lattice = g->lattice_ok && g->lat_uniform && g->nx <= 4096 && g->ny <= 4096;
  for (int general = lattice ? 0 : 1; general < 2; ++general) {
    if (!general) {
      LatBfs p{};
      p.nx = g->nx;
      p.ny = g->ny;
      p.nz = g->nz;
      p.N = g->N;
      p.src = src;
      p.dst = dst;
      const int32_t plane = g->nx * g->ny;
      auto pack = [&](int32_t v) { return (v % g->nx) | ((v % plane) / g->nx) << 12 | (v / plane) << 24; };
      p.psrc = pack(src);
      p.pdst = pack(dst);
      p.max_depth = max_depth;
      p.max_nodes = max_nodes;
      p.keep = keep_d;
      p.nkeep = nkeep;
      p.seen = seen;
      p.roi = roi_nodes_d;
      p.count = misc + 5;
      p.ctl = ctl;
      for (int z = 0; z < g->nz; ++z) {
        p.axis[z] = g->layer_axis[z];
        p.via_to[z] = g->via_to[z];
      }
      // bit sets where they fit (up to about 300 000 nodes), else queues with the
      // marks in shared memory, then in global memory
      const int32_t wpr = (g->nx + 31) / 32;
      const int64_t bits_b = 6 * (int64_t)(wpr | 1) * g->ny * g->nz * 4;
      const bool bits = bits_b <= kBfsSmem;
      const int64_t marks_b = ((N + 15) >> 4) * 4;
      const bool sm = bits || marks_b + 3 * (int64_t)kBfsQueue * 4 <= kBfsSmem;
      p.qcap = sm ? kBfsQueue : kBfsSmem / 12;
      const int smem = (int)(3 * (int64_t)p.qcap * 4 + (sm ? marks_b : 0));
      if (bits) {
        ORSP_CUDA(cudaFuncSetAttribute(roi_bfs_bits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBfsSmem));
        roi_bfs_bits_kernel<<<1, BFS_THREADS, bits_b, st>>>(p, wpr);
      } else {
        void (*kfn)(LatBfs) = sm ? roi_bfs_lattice_kernel<true> : roi_bfs_lattice_kernel<false>;
        ORSP_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, kBfsSmem));
        if (!sm) ORSP_CUDA(cudaMemsetAsync(seen, 0, seen_b, st));
        kfn<<<1, BFS_THREADS, smem, st>>>(p);
      }
      ORSP_CUDA(cudaGetLastError());
      if (!sm) rc = compact_and_truncate(seen, g->N, tiles, misc, max_nodes, src, dst, keep_d, nkeep, roi_nodes_d, st);
    } else {
      ORSP_CUDA(cudaMemsetAsync(seen, 0, seen_b, st));
      roi_bfs_kernel<<<1, BFS_THREADS, 0, st>>>(g->indptr, g->indices, g->N, src, dst, max_depth,
                                                max_nodes, seen, q[0], q[1], q[2], q[3], ctl);
      ORSP_CUDA(cudaGetLastError());
      rc = compact_and_truncate(seen, g->N, tiles, misc, max_nodes, src, dst, keep_d, nkeep, roi_nodes_d, st);
    }
    if (rc) return rc;
    // the map goes along before the host waits (after an overflow it is written
    // again): a wait of its own made calls on other graphs 20 % slower
    if (g2r_d) {
      rc = write_g2r(roi_nodes_d, misc + 5, N, g2r_d, st);
      if (rc) return rc;
    }
    ORSP_CUDA(cudaMemcpyAsync(g->pinned, misc, 24, cudaMemcpyDeviceToHost, st));
    ORSP_CUDA(cudaStreamSynchronize(st));
    if (!h[3]) break;
    if (general) { set_error("roi_bfs: queue overflow"); return ORSP_ERR_OVERFLOW; }
  }
  *roi_count_h = h[5];
  return ORSP_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free ROI extraction.
//
// orsp_roi_bfs keeps its work buffers (visit marks, the four wave queues and
// the compaction tiles) in device memory that the library allocates with
// cudaMalloc on first use.  Some callers cannot allow that: a host
// application whose own caching allocator has reserved the GPU's memory up
// front and forbids any other cudaMalloc / cudaFree on the routing path
// (a cudaFree there also synchronises the whole device).
// orsp_roi_bfs_noalloc gives them the same extraction with its work buffers
// in one file-scope device array, so the call itself allocates nothing.  The
// array is sized for graphs of at most ORSP_ROI_BFS_NOALLOC_MAX_NODES nodes
// and every GPU that loads the library holds it (about 8.5 MB) until the
// process exits.
namespace {

constexpr size_t kNaSeenBytes = ((size_t)ORSP_ROI_BFS_NOALLOC_MAX_NODES + 15) & ~(size_t)15;
constexpr size_t kNaQueueBytes = (size_t)ORSP_ROI_BFS_NOALLOC_MAX_NODES * 4;
constexpr size_t kNaTileBytes =
    (((size_t)ORSP_ROI_BFS_NOALLOC_MAX_NODES + CMP_TILE - 1) / CMP_TILE * 4 + 15) & ~(size_t)15;
constexpr size_t kNaBytes = kNaSeenBytes + 4 * kNaQueueBytes + kNaTileBytes + 64;

// Shared by every call on a device; see orsp_roi_bfs_noalloc for the rules.
static __device__ __align__(256) unsigned char g_roi_noalloc_scratch[kNaBytes];

constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
void *g_na_ptr[kNaMaxDevices] = {};

// Device address of the array on `device` (which must be current).  Looked up
// once per device, by the first call on it: in host code the symbol is only a
// host-side stand-in, not a device address.  The address is cached by device
// ordinal, so the call assumes the device's primary context (the runtime
// API's default); a caller that switches driver-API contexts on one device
// would get an address from another context.
int noalloc_scratch(int device, unsigned char **out) {
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (device < 0 || device >= kNaMaxDevices) {
    set_error("roi_bfs_noalloc: device ordinal out of range");
    return ORSP_ERR_ARG;
  }
  if (!g_na_ptr[device]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_roi_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_roi_noalloc_scratch)");
    g_na_ptr[device] = p;
  }
  *out = (unsigned char *)g_na_ptr[device];
  return ORSP_OK;
}

}  // namespace

extern "C" int orsp_roi_bfs_noalloc(orsp_graph *g, int32_t src, int32_t dst, int32_t max_depth,
                                    int32_t max_nodes, int32_t *roi_nodes_d, int32_t *g2r_d,
                                    int32_t *roi_count_h, uintptr_t stream) {
  if (!g || !roi_nodes_d || !roi_count_h) { set_error("roi_bfs_noalloc: NULL argument"); return ORSP_ERR_ARG; }
  if (g->N > ORSP_ROI_BFS_NOALLOC_MAX_NODES) {
    set_error("roi_bfs_noalloc: graph has " + std::to_string(g->N) + " nodes, more than the " +
              std::to_string(ORSP_ROI_BFS_NOALLOC_MAX_NODES) +
              " its fixed work array holds; use orsp_roi_bfs");
    return ORSP_ERR_ARG;
  }
  if (src < 0 || src >= g->N || dst < 0 || dst >= g->N) { set_error("roi_bfs_noalloc: src/dst out of range"); return ORSP_ERR_ARG; }
  if (max_nodes <= 0) { set_error("roi_bfs_noalloc: max_nodes must be > 0"); return ORSP_ERR_ARG; }
  ORSP_CUDA(cudaSetDevice(g->device));
  unsigned char *base = nullptr;
  int rc = noalloc_scratch(g->device, &base);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t N = g->N;
  uint8_t *seen = base;
  int32_t *q[4];
  for (int i = 0; i < 4; ++i) q[i] = (int32_t *)(base + kNaSeenBytes + i * kNaQueueBytes);
  int32_t *tiles = (int32_t *)(base + kNaSeenBytes + 4 * kNaQueueBytes);
  int32_t *misc = (int32_t *)(base + kNaSeenBytes + 4 * kNaQueueBytes + kNaTileBytes);
  BfsCtl *ctl = (BfsCtl *)misc;

  // The array keeps the previous call's contents: the visit marks must start
  // at zero; the queues, tile counts and counters are written before read.
  ORSP_CUDA(cudaMemsetAsync(seen, 0, ((size_t)N + 15) & ~(size_t)15, st));
  roi_bfs_kernel<<<1, BFS_THREADS, 0, st>>>(g->indptr, g->indices, g->N, src, dst, max_depth,
                                            max_nodes, seen, q[0], q[1], q[2], q[3], ctl);
  ORSP_CUDA(cudaGetLastError());
  int rc_c = compact_and_truncate(seen, g->N, tiles, misc, max_nodes, src, dst, nullptr, 0, roi_nodes_d, st);
  if (rc_c) return rc_c;
  if (g2r_d) {
    rc_c = write_g2r(roi_nodes_d, misc + 5, N, g2r_d, st);
    if (rc_c) return rc_c;
  }
  // g->pinned was allocated when the graph was created, not here; it is one
  // buffer per graph, so overlapping calls on one graph race on it too.
  ORSP_CUDA(cudaMemcpyAsync(g->pinned, misc, 24, cudaMemcpyDeviceToHost, st));
  ORSP_CUDA(cudaStreamSynchronize(st));
  const int32_t *h = (const int32_t *)g->pinned;
  if (h[3]) { set_error("roi_bfs_noalloc: queue overflow"); return ORSP_ERR_OVERFLOW; }
  *roi_count_h = h[5];
  return ORSP_OK;
}
