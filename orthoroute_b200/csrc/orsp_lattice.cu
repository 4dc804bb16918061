// Lattice search: single-source shortest paths on the H/V routing lattice by
// shared-memory tile sweeps.
//
// The generic grid search (orsp_sssp.cu) needs one grid-wide round per hop of
// the shortest-path tree (about 1 400 rounds on a 1000 x 1000 grid, each a
// dependent memory chain plus a grid barrier).  On the routing lattice every
// node has at most four in-edges - the two neighbours along its layer's
// routing axis (x on H layers, y on V layers) and the vias to the layers above
// and below - so a tile of TX x TY columns (all layers) can be relaxed to a
// local fixpoint in shared memory with directional sweeps:
//   x-runs on H layers, y-runs on V layers, z-runs through each via column,
// each run a forward and a backward pass (so a straight wave crosses the tile
// in one pass).  Tiles exchange only boundary improvements, once per grid
// round, so the number of grid rounds drops by about the tile width.
//
// Every update is the fp32 round-to-nearest relaxation min(d[v], d[u] + w), so
// the result is the unique fixpoint of the generic search, bit for bit, in any
// order; the backtrace (orsp_sssp.cu) is shared.  A tile that has not
// converged after MAX_CYCLES sweep cycles is simply revisited next round.
//
// Tiles in the next round's list: neighbours whose halo value improved (and
// the tile itself if it did not converge).  Each tile is in a round's list at
// most once (stamp[t] = last round it was queued for), so a tile is only ever
// processed by one CTA per round and owns its nodes' distances.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "fastdiv.cuh"
#include "launch_cache.cuh"
#include "lattice_walk.cuh"

namespace {

constexpr int MAX_CYCLES = 64;

// Layer strides (floats) of a tile's shared arrays: distances with their
// halo, (TY + 2) rows of TX + 3, and the interior arrays (weights, loaded
// distances), TY rows of TX + 1, each padded to 8 (mod 16).  A warp's x- or
// y-runs cover two layers of the same kind, which are two layers apart (H
// and V layers alternate), so a layer offset of 2 x stride = 16 (mod 32)
// puts the second layer's rows on the other half of the banks.
__host__ __device__ constexpr int pad_8_mod_16(int v) { return v + ((8 - v % 16) + 16) % 16; }
__host__ __device__ constexpr int tile_ps(int TX, int TY) { return pad_8_mod_16((TY + 2) * (TX + 3)); }
__host__ __device__ constexpr int tile_wps(int TX, int TY) { return pad_8_mod_16(TY * (TX + 1)); }
// Floats of shared memory per layer of a tile (distances, four weight
// arrays, loaded distances).
__host__ __device__ constexpr int tile_floats_per_layer(int TX, int TY) { return tile_ps(TX, TY) + 5 * tile_wps(TX, TY); }

struct LatCtl {
  GridBarrier bar;
  int err;
  unsigned lcnt[3];  // tile-list counts by round % 3
  unsigned work[3];  // per-round work counters by round % 3
  unsigned rounds;
  unsigned visits;
  unsigned long long cycles;
  unsigned head, tail;  // tile queue positions (asynchronous schedule)
  int pending;          // tiles queued or being visited
  int avail;            // visiting owners: queued tiles less the CTAs waiting for one
  unsigned long long ns[4];  // time in load, sweeps, write-back, scheduling (sum over visits)
};

using orsp::LatBox;

struct LatParams {
  int32_t nx, ny, nz;
  int32_t nbox;
  int32_t seed_per_box;                    // seed i starts box i (boxes with their own distances)
  const LatBox *boxes;                     // searched boxes (disjoint unless each has its own distances)
  const float4 *w4;                        // in-edge weights per node
  uint32_t *dist;
  int32_t *list0, *list1;
  unsigned *stamp;
  int32_t *qslot;  // asynchronous schedule: ring of tile ids (-1 = empty)
  int *tstate;     // 0 idle, 1 queued, 2 visiting, 3 visiting and dirty
  unsigned qcap;
  LatCtl *ctl;
  int8_t axis[64];
  unsigned max_rounds;
  unsigned long long wait_ns, budget_ns;
  int selfcont;
  int prefetch;            // warp-specialised schedule: L2 prefetch of the next tile's rows
  const int32_t *roi_map;  // node-set ROI searches: seeds outside it are ignored
  const float *wcol;       // column vias: gathered via weights [N][nzp] (Graph::wcol)
  int32_t nzp;             // nz rounded up to 4
  int64_t N;
  // layers by axis, as bit sets and as ascending lists (run visits)
  uint64_t hmask, vmask;
  int8_t hlist[64], vlist[64];
  const int32_t *tbox;  // box of each tile (asynchronous schedule)
  unsigned *inbox;      // messages to each tile (visiting owners; else NULL)
  const int *wmin;      // boxes with targets: smallest planar and via weight (float bits; else NULL)
};

__global__ void fill_kernel(uint32_t *p, int64_t n, uint32_t v) {
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += s) p[i] = v;
}

// The fill of the boxes' own distance slices [dbase, dbase + volume), box
// blockIdx.y, skipping boxes with active[j] == 0.
__global__ void fill_slices_kernel(uint32_t *p, const LatBox *__restrict__ boxes, const int32_t *__restrict__ active,
                                   uint32_t v) {
  if (active && !active[blockIdx.y]) return;
  const LatBox B = boxes[blockIdx.y];
  const int64_t count = (int64_t)(B.x1 - B.x0 + 1) * (B.y1 - B.y0 + 1) * (B.z1 - B.z0 + 1);
  uint32_t *q = p + B.dbase;
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += s) q[i] = v;
}

// The same fill over the nodes of a box (x fastest).
__global__ void fill_box_kernel(uint32_t *p, int32_t nx, int32_t ny, int32_t x0, int32_t bw, int32_t y0,
                                int32_t bh, int32_t z0, int64_t count, uint32_t v) {
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  const int64_t plane = (int64_t)bw * bh;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += s) {
    const int64_t z = i / plane;
    const int64_t r = i - z * plane;
    const int32_t y = (int32_t)(r / bw), x = (int32_t)(r - (int64_t)y * bw);
    p[((int64_t)(z0 + z) * ny + (y0 + y)) * nx + (x0 + x)] = v;
  }
}

// Cell i of a box (x fastest, then y, then z) as coordinates: multiply-high
// divisions while the box has fewer than 2^32 cells (the common case),
// 64-bit divisions otherwise.
struct BoxIndex {
  FastDiv fw, fp;
  uint32_t w;
  bool fast;
  __device__ __forceinline__ void init(int64_t bw, int64_t bh, int64_t count) {
    fast = count < ((int64_t)1 << 32) && bw * bh < ((int64_t)1 << 31);
    w = (uint32_t)bw;
    if (fast) {
      fw.init((uint32_t)bw);
      fp.init((uint32_t)(bw * bh));
    }
  }
  __device__ __forceinline__ void split(int64_t i, int64_t plane, int32_t &z, int32_t &y, int32_t &x) const {
    if (fast) {
      const uint32_t u = (uint32_t)i, zz = fp.div(u), r = u - zz * (uint32_t)plane, yy = fw.div(r);
      z = (int32_t)zz;
      y = (int32_t)yy;
      x = (int32_t)(r - yy * w);
    } else {
      const int64_t zz = i / plane, r = i - zz * plane, yy = r / w;
      z = (int32_t)zz;
      y = (int32_t)yy;
      x = (int32_t)(r - yy * w);
    }
  }
};

// Smallest planar and via weight, as float bits, of the nodes that a gather
// passes (wmin NULL: not wanted).  Negative weights and -0 come out negative,
// absent edges and NaN do not count.
__device__ __forceinline__ void min_weight(int2 &m, const float4 &w) {
  m.x = min(m.x, min(__float_as_int(w.x), __float_as_int(w.y)));
  m.y = min(m.y, min(__float_as_int(w.z), __float_as_int(w.w)));
}
__device__ __forceinline__ void record_min(int *wmin, int2 m) {
  m.x = __reduce_min_sync(ORSP_FULL_MASK, m.x);
  m.y = __reduce_min_sync(ORSP_FULL_MASK, m.y);
  if ((threadIdx.x & 31) == 0) {  // (the look first: most warps have nothing to add)
    if (m.x < __ldcg(&wmin[0])) atomicMin(&wmin[0], m.x);
    if (m.y < __ldcg(&wmin[1])) atomicMin(&wmin[1], m.y);
  }
}

// In-edge weights of node v as one float4 {from lower axis neighbour, from
// upper axis neighbour, via from below, via from above}; +inf where absent.
// (MIN: a variant of its own, so that the plain loop keeps four nodes in flight:
// with a test in the loop 58 instead of 43 us for 600 x 600 x 12)
template <bool MIN>
__global__ void gather_kernel(const int32_t *__restrict__ slot_eid, const float *__restrict__ cost,
                              float4 *__restrict__ w, int64_t n, int *wmin) {
  const float INF_F = __int_as_float(0x7f800000);
  int2 m = make_int2(INT_MAX, INT_MAX);
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
#pragma unroll 4
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += s) {
    const int32_t e0 = slot_eid[v], e1 = slot_eid[n + v], e2 = slot_eid[2 * n + v], e3 = slot_eid[3 * n + v];
    const float4 o = make_float4(e0 >= 0 ? __ldg(&cost[e0]) : INF_F, e1 >= 0 ? __ldg(&cost[e1]) : INF_F,
                                 e2 >= 0 ? __ldg(&cost[e2]) : INF_F, e3 >= 0 ? __ldg(&cost[e3]) : INF_F);
    w[v] = o;
    if (MIN) min_weight(m, o);
  }
  if (MIN) record_min(wmin, m);
}

// The same gather for the nodes of a box only (x fastest, then y, then z): cells
// i, i + s, ... of it.
__device__ __forceinline__ void gather_cells(const int32_t *__restrict__ slot_eid, const float *__restrict__ cost,
                                             float4 *__restrict__ w, int64_t n, int32_t nx, int32_t ny, int32_t x0,
                                             int64_t bw, int32_t y0, int64_t bh, int32_t z0, int64_t count, int64_t i,
                                             int64_t s) {
  const float INF_F = __int_as_float(0x7f800000);
  const int64_t plane = bw * bh;
  BoxIndex bi;
  bi.init(bw, bh, count);
  for (; i < count; i += s) {
    int32_t z, y, x;
    bi.split(i, plane, z, y, x);
    const int64_t v = ((int64_t)(z0 + z) * ny + (y0 + y)) * nx + (x0 + x);
    const int32_t e0 = slot_eid[v], e1 = slot_eid[n + v], e2 = slot_eid[2 * n + v], e3 = slot_eid[3 * n + v];
    w[v] = make_float4(e0 >= 0 ? __ldg(&cost[e0]) : INF_F, e1 >= 0 ? __ldg(&cost[e1]) : INF_F,
                       e2 >= 0 ? __ldg(&cost[e2]) : INF_F, e3 >= 0 ? __ldg(&cost[e3]) : INF_F);
  }
}

__global__ void gather_box_kernel(const int32_t *__restrict__ slot_eid, const float *__restrict__ cost,
                                  float4 *__restrict__ w, int64_t n, int32_t nx, int32_t ny, int32_t x0,
                                  int32_t bw, int32_t y0, int32_t bh, int32_t z0, int64_t count) {
  gather_cells(slot_eid, cost, w, n, nx, ny, x0, bw, y0, bh, z0, count,
               (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// The same gather for the nodes of several boxes in one launch: blockIdx.y
// is the box (a device LatBox table), blockIdx.x strides over its cells;
// boxes with active[j] == 0 are skipped (active NULL: none).  Cells shared by
// two boxes are written twice with the same value.
template <bool MIN>
__global__ void gather_boxes_kernel(const int32_t *__restrict__ slot_eid, const float *__restrict__ cost,
                                    float4 *__restrict__ w, int64_t n, int32_t nx, int32_t ny,
                                    const LatBox *__restrict__ boxes, const int32_t *__restrict__ active, int *wmin) {
  if (active && !active[blockIdx.y]) return;
  const float INF_F = __int_as_float(0x7f800000);
  int2 m = make_int2(INT_MAX, INT_MAX);
  const LatBox B = boxes[blockIdx.y];
  const int32_t bw = B.x1 - B.x0 + 1, bh = B.y1 - B.y0 + 1;
  const int64_t plane = (int64_t)bw * bh, count = plane * (B.z1 - B.z0 + 1);
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  BoxIndex bi;
  bi.init(bw, bh, count);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += s) {
    int32_t z, y, x;
    bi.split(i, plane, z, y, x);
    const int64_t v = ((int64_t)(B.z0 + z) * ny + (B.y0 + y)) * nx + (B.x0 + x);
    const int32_t e0 = slot_eid[v], e1 = slot_eid[n + v], e2 = slot_eid[2 * n + v], e3 = slot_eid[3 * n + v];
    const float4 o = make_float4(e0 >= 0 ? __ldg(&cost[e0]) : INF_F, e1 >= 0 ? __ldg(&cost[e1]) : INF_F,
                                 e2 >= 0 ? __ldg(&cost[e2]) : INF_F, e3 >= 0 ? __ldg(&cost[e3]) : INF_F);
    w[v] = o;
    if (MIN) min_weight(m, o);
  }
  if (MIN) record_min(wmin, m);
}

// ---------------------------------------------------------------------------
// Node-set ROI searches (global_to_roi maps, as SimpleDijkstra.find_path_roi
// takes them, UPF:1801-1887): the tile sweeps run over the ROI's bounding box,
// on weights in which every edge that leaves or enters the ROI is +inf.

struct RoiGeom {
  int32_t nx, ny, nz;
  int8_t axis[64];
};

// Bounding box of the ROI, as running maxima bb[6] = {-x0, x1, -y0, y1, -z0,
// z1} (bb starts far below any coordinate): over the node list when given,
// else over every node v with roi_map[v] >= 0.
__global__ void roi_bbox_kernel(const int32_t *__restrict__ nodes, int64_t n, const int32_t *__restrict__ roi_map,
                                int32_t nx, int32_t ny, int64_t N, int *bb) {
  int m[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) m[k] = INT_MIN;
  const int64_t plane = (int64_t)nx * ny;
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  // node ids are int32 (N < 2^31): multiply-high divisions
  FastDiv fp, fx;
  fp.init((uint32_t)plane);
  fx.init((uint32_t)nx);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += s) {
    const int64_t v = nodes ? (int64_t)__ldg(&nodes[i]) : i;
    if (v < 0 || v >= N) continue;
    if (!nodes && __ldg(&roi_map[v]) < 0) continue;
    const uint32_t u = (uint32_t)v, zu = fp.div(u), r = u - zu * (uint32_t)plane, yu = fx.div(r);
    const int32_t z = (int32_t)zu, y = (int32_t)yu, x = (int32_t)(r - yu * (uint32_t)nx);
    m[0] = max(m[0], -x);
    m[1] = max(m[1], x);
    m[2] = max(m[2], -y);
    m[3] = max(m[3], y);
    m[4] = max(m[4], -z);
    m[5] = max(m[5], z);
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int w = __reduce_max_sync(ORSP_FULL_MASK, m[k]);
    if ((threadIdx.x & 31) == 0 && w != INT_MIN) atomicMax(&bb[k], w);
  }
}

// The searched box from the running maxima (an empty ROI gives a box with
// no cells and no tiles).
template <int TX, int TY>
__global__ void roi_box_finish_kernel(const int *bb, LatBox *box) {
  LatBox B;
  if (bb[1] < 0) {
    B.x0 = 0; B.x1 = -1; B.y0 = 0; B.y1 = -1; B.z0 = 0; B.z1 = -1;
    B.ntx = 0;
    B.nty = 0;
  } else {
    B.x0 = -bb[0]; B.x1 = bb[1]; B.y0 = -bb[2]; B.y1 = bb[3]; B.z0 = -bb[4]; B.z1 = bb[5];
    B.ntx = (B.x1 - B.x0 + TX) / TX;
    B.nty = (B.y1 - B.y0 + TY) / TY;
  }
  B.tile0 = 0;
  B.pad = 0;
  B.dbase = -1;
  B.gx = B.gy = B.gz = -1;
  B.pad2 = 0;
  *box = B;
}

// In-edge weights of the box's nodes, as gather_kernel, with +inf on every
// edge u -> v where u or v lies outside the ROI (roi_map < 0; NULL: no
// restriction) or u is a sink (sink[u] != 0; NULL: none).  Grid-stride over
// the box read from device memory.
__global__ void gather_roi_kernel(const int32_t *__restrict__ slot_eid, const float *__restrict__ cost,
                                  float4 *__restrict__ w, int64_t n, RoiGeom G, const LatBox *__restrict__ box,
                                  const int32_t *__restrict__ roi_map, const uint8_t *__restrict__ sink) {
  const float INF_F = __int_as_float(0x7f800000);
  const LatBox B = *box;
  const int64_t bw = B.x1 - B.x0 + 1, bh = B.y1 - B.y0 + 1, bd = B.z1 - B.z0 + 1;
  if (bw <= 0 || bh <= 0 || bd <= 0) return;
  const int64_t plane = bw * bh, count = plane * bd;
  const int64_t nxy = (int64_t)G.nx * G.ny;
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  BoxIndex bi;
  bi.init(bw, bh, count);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += s) {
    int32_t zz, yy, xx;
    bi.split(i, plane, zz, yy, xx);
    const int32_t gz = B.z0 + (int32_t)zz;
    const int64_t v = (int64_t)gz * nxy + (int64_t)(B.y0 + yy) * G.nx + (B.x0 + xx);
    const bool vin = !roi_map || __ldg(&roi_map[v]) >= 0;
    const int64_t step = G.axis[gz] == 1 ? 1 : G.nx;
    const int64_t from[4] = {v - step, v + step, v - nxy, v + nxy};
    float o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int32_t e = __ldg(&slot_eid[k * n + v]);
      bool ok = e >= 0 && vin;
      if (ok) {
        const int64_t u = from[k];
        ok = (!roi_map || __ldg(&roi_map[u]) >= 0) && !(sink && __ldg(&sink[u]));
      }
      o[k] = ok ? __ldg(&cost[e]) : INF_F;
    }
    w[v] = make_float4(o[0], o[1], o[2], o[3]);
  }
}

// Column-via weights of the nodes of a box (column vias, Graph::cvia):
// wcol[v * nzp + za] (nzp = nz rounded up to 4) = the smaller cost of the (up to two) parallel vias from
// layer za of v's column into v, for every layer za of the box; +inf where
// there is none, where u or v lies outside the ROI (roi_map < 0; NULL: no
// restriction) or u is a sink (sink[u] != 0; NULL: none).  The box is read
// from device memory (bx) or given by value (bx NULL).
__global__ void gather_col_kernel(const int32_t *__restrict__ vcol_eid, const float *__restrict__ cost,
                                  float *__restrict__ wcol, int64_t n, int32_t nx, int32_t ny, int32_t nz, int32_t nzp,
                                  const LatBox *__restrict__ bx, LatBox bv, const int32_t *__restrict__ roi_map,
                                  const uint8_t *__restrict__ sink) {
  const float INF_F = __int_as_float(0x7f800000);
  const LatBox B = bx ? *bx : bv;
  const int64_t bw = B.x1 - B.x0 + 1, bh = B.y1 - B.y0 + 1, bd = B.z1 - B.z0 + 1;
  if (bw <= 0 || bh <= 0 || bd <= 0) return;
  const int64_t plane = bw * bh, cells = plane * bd, count = cells * bd;
  const int64_t nxy = (int64_t)nx * ny;
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  // cells of the box stacked bd times (one copy per source layer): the
  // "layer" coordinate of this split runs over bd * bd
  BoxIndex bi;
  bi.init(bw, bh, count);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += s) {
    int32_t zq, yy, xx;
    bi.split(i, plane, zq, yy, xx);
    const int64_t za = B.z0 + zq / (int32_t)bd;  // source layer
    const int32_t zz = zq - (int32_t)((za - B.z0) * bd);
    const int64_t col = (int64_t)(B.y0 + yy) * nx + (B.x0 + xx);
    const int64_t v = (int64_t)(B.z0 + zz) * nxy + col;
    const int32_t e0 = __ldg(&vcol_eid[za * n + v]), e1 = __ldg(&vcol_eid[((int64_t)nz + za) * n + v]);
    float w = INF_F;
    if (e0 >= 0) {
      const int64_t u = za * nxy + col;
      bool ok = !roi_map || (__ldg(&roi_map[v]) >= 0 && __ldg(&roi_map[u]) >= 0);
      ok = ok && !(sink && __ldg(&sink[u]));
      if (ok) {
        w = __ldg(&cost[e0]);
        if (e1 >= 0) w = fminf(w, __ldg(&cost[e1]));
      }
    }
    wcol[v * nzp + za] = w;
  }
}

__device__ __forceinline__ LatBox load_box(const LatParams &p, int b) {
  const int32_t *q = (const int32_t *)(p.boxes + b);
  LatBox B;
  B.x0 = __ldg(q + 0);
  B.x1 = __ldg(q + 1);
  B.y0 = __ldg(q + 2);
  B.y1 = __ldg(q + 3);
  B.z0 = __ldg(q + 4);
  B.z1 = __ldg(q + 5);
  B.ntx = __ldg(q + 6);
  B.nty = __ldg(q + 7);
  B.tile0 = __ldg(q + 8);
  B.pad = __ldg(q + 9);
  B.dbase = __ldg((const long long *)(p.boxes + b) + 5);
  B.gx = __ldg(q + 12);
  B.gy = __ldg(q + 13);
  B.gz = __ldg(q + 14);
  B.pad2 = 0;
  return B;
}

// Index of cell (x, y, z) of box B in the distance array: the node id
// (shared distances) or the box's own slice (PRIV, B.dbase >= 0).  The search
// kernels are compiled once per mode, so the shared mode carries no slice
// arithmetic.
template <bool PRIV>
__device__ __forceinline__ int64_t dist_index(const LatParams &p, const LatBox &B, int32_t x, int32_t y, int32_t z) {
  if (!PRIV || B.dbase < 0) return ((int64_t)z * p.ny + y) * p.nx + x;
  const int64_t bw = B.x1 - B.x0 + 1, bh = B.y1 - B.y0 + 1;
  return B.dbase + ((int64_t)(z - B.z0) * bh + (y - B.y0)) * bw + (x - B.x0);
}

// Box of tile t: the last box whose first tile is <= t.
__device__ __forceinline__ int box_of_tile(const LatParams &p, int t) {
  int lo = 0, hi = p.nbox - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&p.boxes[mid].tile0) <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <int TX, int TY>
__device__ __forceinline__ int tile_of(const LatBox &B, int32_t gx, int32_t gy) {
  return B.tile0 + ((gy - B.y0) / TY) * B.ntx + (gx - B.x0) / TX;
}

// Asynchronous schedule: every tile idle, the queue empty, each tile's box
// (and, for visiting owners, no messages and the exchange rows at +inf).
__global__ void lattice_init_kernel(LatParams p, int32_t ntiles, unsigned *got, float4 *rows, int64_t nrows) {
  const int64_t s = (int64_t)gridDim.x * blockDim.x;
  const float INF_F = __int_as_float(0x7f800000);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nrows; i += s)
    rows[i] = make_float4(INF_F, INF_F, INF_F, INF_F);
  const int64_t n = max((int64_t)ntiles, (int64_t)p.qcap);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += s) {
    if (i < ntiles) {
      p.tstate[i] = 0;
      p.stamp[i] = 0;
      if (p.inbox) p.inbox[i] = got[i] = 0;
      p.list0[i] = p.nbox == 1 ? 0 : box_of_tile(p, (int)i);
    }
    if (i < p.qcap) p.qslot[i] = -1;
  }
}

template <int TX, int TY>
__global__ void lattice_seed_kernel(LatParams p, int32_t nseeds, const int32_t *seeds,
                                    const float *seed_cost) {
  LatCtl *c = p.ctl;
  if (threadIdx.x == 0) {
    c->bar.count = 0;
    c->bar.gen = 0;
    c->err = 0;
    for (int i = 0; i < 3; ++i) { c->lcnt[i] = 0; c->work[i] = 0; }
    c->rounds = 0;
    c->visits = 0;
    c->cycles = 0;
    c->head = 0;
    c->tail = 0;
    c->pending = 0;
    c->avail = 0;
    for (int i = 0; i < 4; ++i) c->ns[i] = 0;
  }
  __syncthreads();
  const int32_t plane = p.nx * p.ny;
  for (int i = threadIdx.x; i < nseeds; i += blockDim.x) {
    const int32_t s = seeds[i];
    if (s < 0 || s >= plane * p.nz) continue;
    if (p.roi_map && __ldg(&p.roi_map[s]) < 0) continue;
    const int32_t z = s / plane, r = s - z * plane, y = r / p.nx, x = r - y * p.nx;
    int bi = -1;
    LatBox B;
    if (p.seed_per_box) {
      if (i < p.nbox) {
        B = load_box(p, i);
        if (x >= B.x0 && x <= B.x1 && y >= B.y0 && y <= B.y1 && z >= B.z0 && z <= B.z1) bi = i;
      }
    } else {
      for (int b = 0; b < p.nbox && bi < 0; ++b) {
        B = load_box(p, b);
        if (x >= B.x0 && x <= B.x1 && y >= B.y0 && y <= B.y1 && z >= B.z0 && z <= B.z1) bi = b;
      }
    }
    if (bi < 0) continue;
    const float c0 = seed_cost ? seed_cost[i] : 0.0f;
    if (!(c0 >= 0.0f) || !(c0 < __int_as_float(0x7f800000))) continue;
    atomicMin(&p.dist[p.seed_per_box ? dist_index<true>(p, B, x, y, z) : dist_index<false>(p, B, x, y, z)],
              f_bits(c0));
    // The seed's tile and its neighbours in the box: a tile visit publishes
    // only cells it improved, and a seed is set before any visit, so a seed
    // on a tile edge reaches the next tile through that tile's halo only.
    const int t = tile_of<TX, TY>(B, x, y);
    const int lt = t - B.tile0, tx = lt % B.ntx, ty = lt / B.ntx;
    // its columns start unrelaxed: the first visit takes all of them
    if (p.qslot) p.stamp[t] = 1u;
    const int nb[5] = {t, tx > 0 ? t - 1 : -1, tx < B.ntx - 1 ? t + 1 : -1, ty > 0 ? t - B.ntx : -1,
                       ty < B.nty - 1 ? t + B.ntx : -1};
    for (int j = 0; j < 5; ++j) {
      const int q = nb[j];
      if (q < 0) continue;
      if (p.inbox) {
        // a message for the seed's tile; its neighbours are only taken early
        if (j == 0 && atomicExch(&p.inbox[q], 1u) == 0u) atomicAdd(&c->pending, 1);
        if (atomicCAS(&p.tstate[q], 0, 1) == 0) {
          atomicAdd(&c->avail, 1);
          const unsigned k = atomicAdd(&c->tail, 1u);
          atomicExch(&p.qslot[k % p.qcap], q);
        }
      } else if (p.qslot) {
        if (atomicCAS(&p.tstate[q], 0, 1) == 0) {
          atomicAdd(&c->pending, 1);
          const unsigned k = atomicAdd(&c->tail, 1u);
          atomicExch(&p.qslot[k % p.qcap], q);
        }
      } else if (atomicMax(&p.stamp[q], 1u) < 1u) {
        const unsigned k = atomicAdd(&c->lcnt[0], 1u);
        p.list0[k] = q;
      }
    }
  }
}

// One run of the sweep: cells c[1..n] at stride `ds`, with c[0] and c[n+1]
// the halo values (when `halo`; otherwise the run starts and ends at c[1] and
// c[n]).  Forward: c[i] = min(c[i], c[i-1] + wlo[i]); backward: c[i] =
// min(c[i], c[i+1] + whi[i]); each step a single fp32 round-to-nearest add
// and a min (fminf returns one of its operands; no NaN or -0 occurs here, so
// the result is that of the compare-and-replace form, without a branch).  The
// run is walked in register chunks of 4 (loads first, then the dependent
// chain), and only decreased cells are stored.  Returns whether any cell
// decreased.  Used for runs whose length is known only at run time (tiles cut
// by the box edge, z-runs).
__device__ __forceinline__ bool sweep_run(float *c, int ds, const float *wlo, const float *whi, int ws,
                                          int n, bool halo = true) {
  constexpr int K = 4;
  bool chg = false;
  float prev = halo ? c[0] : __int_as_float(0x7f800000);
  for (int b = 1; b <= n; b += K) {
    float cv[K], wv[K], nv[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (b + k <= n) { cv[k] = c[(b + k) * ds]; wv[k] = wlo[(b + k) * ws]; }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (b + k <= n) { nv[k] = fminf(__fadd_rn(prev, wv[k]), cv[k]); prev = nv[k]; }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (b + k <= n && nv[k] < cv[k]) { c[(b + k) * ds] = nv[k]; chg = true; }
  }
  prev = halo ? c[(n + 1) * ds] : __int_as_float(0x7f800000);
  for (int b = n; b >= 1; b -= K) {
    float cv[K], wv[K], nv[K];
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (b - k >= 1) { cv[k] = c[(b - k) * ds]; wv[k] = whi[(b - k) * ws]; }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (b - k >= 1) { nv[k] = fminf(__fadd_rn(prev, wv[k]), cv[k]); prev = nv[k]; }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (b - k >= 1 && nv[k] < cv[k]) { c[(b - k) * ds] = nv[k]; chg = true; }
  }
  return chg;
}

// The same run for a full tile row or column: length N and strides known at
// compile time, so every shared-memory access is an immediate offset from one
// base, the whole run is in registers and the chain is one add and one min
// per step.
template <int N, int DS, int WS>
__device__ __forceinline__ bool sweep_run_fixed(float *c, const float *wlo, const float *whi) {
  float o[N], v[N];
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = c[(i + 1) * DS];
  float prev = c[0];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    v[i] = fminf(__fadd_rn(prev, wlo[(i + 1) * WS]), o[i]);
    prev = v[i];
  }
  prev = c[(N + 1) * DS];
#pragma unroll
  for (int i = N - 1; i >= 0; --i) {
    v[i] = fminf(__fadd_rn(prev, whi[(i + 1) * WS]), v[i]);
    prev = v[i];
  }
  bool chg = false;
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (v[i] < o[i]) {
      c[(i + 1) * DS] = v[i];
      chg = true;
    }
  return chg;
}

// B consecutive cells of a z-run (stride DS, weights stride WS), forward
// (UP: from below, weights wdn) or backward (from above, weights wup), with
// the chain value carried in `prev`.
template <int B, int DS, int WS, bool UP>
__device__ __forceinline__ bool zrun_block(float *c, const float *w, float &prev) {
  float o[B], v[B];
#pragma unroll
  for (int i = 0; i < B; ++i) o[i] = c[i * DS];
#pragma unroll
  for (int k = 0; k < B; ++k) {
    const int i = UP ? k : B - 1 - k;
    v[i] = fminf(__fadd_rn(prev, w[i * WS]), o[i]);
    prev = v[i];
  }
  bool chg = false;
#pragma unroll
  for (int i = 0; i < B; ++i)
    if (v[i] < o[i]) {
      c[i * DS] = v[i];
      chg = true;
    }
  return chg;
}

// z-run of a column: cells col[z * DS] for z = 0..n-1 (no halo), forward with
// wdn, then backward with wup, in register blocks of 6.
template <int DS, int WS>
__device__ __forceinline__ bool zrun(float *col, const float *wdn, const float *wup, int n) {
  constexpr int B = 6;
  bool chg = false;
  float prev = __int_as_float(0x7f800000);
  int z = 0;
  for (; z + B <= n; z += B) chg |= zrun_block<B, DS, WS, true>(col + z * DS, wdn + z * WS, prev);
  for (; z < n; ++z) chg |= zrun_block<1, DS, WS, true>(col + z * DS, wdn + z * WS, prev);
  prev = __int_as_float(0x7f800000);
  z = n;
  for (; z >= B; z -= B) chg |= zrun_block<B, DS, WS, false>(col + (z - B) * DS, wup + (z - B) * WS, prev);
  for (; z > 0; --z) chg |= zrun_block<1, DS, WS, false>(col + (z - 1) * DS, wup + (z - 1) * WS, prev);
  return chg;
}

// Relaxes one tile (all layers of the box) to a local fixpoint and publishes
// improved values.  Called by all threads of the CTA.  Shared memory:
// distances with a one-cell halo [nzb][TY+2][TX+3], then the interior in-edge
// weights [4][nzb][TY][TX+1] and the interior distances as loaded
// [nzb][TY][TX+1], layers tile_ps / tile_wps floats apart (odd row strides:
// the row walks of the x-sweep and the column walks of the y- and z-sweeps
// are bank-conflict free within a layer; the padded layer strides keep the
// two layers of one warp apart).
// The distances and in-edge weights of one tile column (cells s0 + z * PS /
// w0 + z * WPS in shared memory) in blocks of ZB layers, each block's loads
// all issued before its stores.
template <int ZB, int PS, int WPS>
__device__ __forceinline__ void load_column_blocks_impl(const LatParams &p, int nzb, int64_t d0, int64_t dz,
                                                        int64_t n0, int64_t nxy, float *sd, float *orig, float *wlo,
                                                        float *whi, float *wdn, float *wup, int s0, int w0) {
  for (int zb = 0; zb < nzb; zb += ZB) {
    float dv[ZB];
    float4 wv[ZB];
#pragma unroll
    for (int k = 0; k < ZB; ++k)
      if (zb + k < nzb) {
        dv[k] = bits_f(__ldcg(&p.dist[d0 + (zb + k) * dz]));
        wv[k] = __ldg(&p.w4[n0 + (zb + k) * nxy]);
      }
#pragma unroll
    for (int k = 0; k < ZB; ++k)
      if (zb + k < nzb) {
        const int z = zb + k, wi = z * WPS + w0;
        sd[z * PS + s0] = dv[k];
        orig[wi] = dv[k];
        wlo[wi] = wv[k].x;
        whi[wi] = wv[k].y;
        wdn[wi] = wv[k].z;
        wup[wi] = wv[k].w;
      }
  }
}

// Barrier of the threads that visit tiles: the whole block, or (SPEC) the
// first NW threads only - named barrier 1 - while a scheduler warp runs beside
// them.
template <int NW, bool SPEC>
__device__ __forceinline__ void tile_sync() {
  if (SPEC) asm volatile("bar.sync 1, %0;" ::"r"(NW) : "memory");
  else __syncthreads();
}

// Tensor-memory-accelerator staging of a whole-lattice tile (ORSP_LAT_TMA=1):
// two cp.async.bulk.tensor loads per fresh visit, completing on one mbarrier,
// bring the tile's in-edge weights (box {4, TX, TY, nzb} of the float4 array
// seen as fp32 [nz][ny][nx][4]) and its distances with a halo (box
// {TX + 8, TY + 2, nzb} of the u32 distances [slice][nz][ny][nx], starting at
// x = X0 - 4 so that the start is 16-byte aligned) into a staging area; the
// threads then copy them into the sweep layout (odd row strides), as the
// plain loads do.  Out-of-lattice cells of the box are zero-filled by the
// copy engine and replaced by +inf (halo) or ignored (interior) in the copy.
// The tensor maps cover this GPU's memory only and no load is multicast.
struct TmaCtx {
  const CUtensorMap *tw, *td;  // the kernel's __grid_constant__ tensor maps
  uint32_t mbar;               // shared address of the CTA's mbarrier
  unsigned phase;              // parity of the next completion
  float *sw;                   // staging: weights [nzb][TY][TX] float4
  uint32_t *sdd;               // staging: distances [nzb][TY + 2][TX + 8]
};

__device__ __forceinline__ uint32_t smem_addr(const void *ptr) {
  return (uint32_t)__cvta_generic_to_shared(ptr);
}

// Thread 0 issues the two loads of the tile at (X0, Y0) of distance slice
// `slice`; every thread then waits (bounded) for their completion.
template <int TX, int TY>
__device__ __forceinline__ void tma_stage(const LatParams &p, int32_t X0, int32_t Y0, int32_t z0, int nzb,
                                          int slice, TmaCtx &tc) {
  if (threadIdx.x == 0) {
    const uint32_t bytes = (uint32_t)nzb * (uint32_t)(TY * TX * 16 + (TY + 2) * (TX + 8) * 4);
    // distances other CTAs published (acquired through the tile state) are
    // read by the async proxy; the staging's earlier generic reads come
    // before its async-proxy writes
    asm volatile("fence.proxy.async.global;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc.mbar), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smem_addr(tc.sw)), "l"((uint64_t)tc.tw), "r"(0), "r"(X0), "r"(Y0), "r"(z0), "r"(tc.mbar)
        : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(smem_addr(tc.sdd)), "l"((uint64_t)tc.td), "r"(X0 - 4), "r"(Y0 - 1), "r"(z0), "r"(slice), "r"(tc.mbar)
        : "memory");
  }
  // bounded wait: past wait_ns the search is failed with a timeout, and the
  // wait goes on for one more wait_ns so that the copies are not left in
  // flight into shared memory that the next visit reuses
  const unsigned long long t0 = dev_globaltimer();
  bool timed_out = false;
  for (unsigned spins = 0;; ++spins) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n selp.u32 %0, 1, 0, P;\n}"
        : "=r"(ok)
        : "r"(tc.mbar), "r"(tc.phase)
        : "memory");
    if (ok) break;
    if ((spins & 63u) == 63u) {
      const unsigned long long dt = dev_globaltimer() - t0;
      if (!timed_out && dt > p.wait_ns) {
        atomicCAS(&p.ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
        timed_out = true;
      }
      if (dt > 2 * p.wait_ns) break;
    }
  }
  tc.phase ^= 1u;
}

// Via pass of one column with column vias: for each layer zb of the box in
// turn, d[zb] = min(d[zb], fl(d[za] + w(za -> zb))) over every layer za of the
// box (Gauss-Seidel, so a later layer sees an earlier one's new value), the
// in-weights read as float4 rows wcol[v * nzp ..] (+inf where no via).  col:
// the column's distances in shared memory, layer stride PS; v0: the node of
// the column's layer z0.  Returns the set of layers that decreased.  The
// visit repeats it until nothing changes.
template <int PS>
__device__ __forceinline__ unsigned long long zcol_pass(float *col, const float *__restrict__ wcol, int32_t nzp, int64_t v0,
                                          int64_t nxy, int32_t z0, int32_t nzb) {
  const float INF_F = __int_as_float(0x7f800000);
  unsigned long long chg = 0;
  const int q0 = z0 >> 2, q1 = (z0 + nzb - 1) >> 2;
  for (int zb = 0; zb < nzb; ++zb) {
    const float4 *wr = reinterpret_cast<const float4 *>(wcol + (v0 + (int64_t)zb * nxy) * nzp);
    float best = col[zb * PS];
    for (int q = q0; q <= q1; ++q) {
      const float4 w = __ldg(&wr[q]);
      const float wk[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int za = 4 * q + j - z0;
        if (za >= 0 && za < nzb && wk[j] < INF_F) best = fminf(best, __fadd_rn(col[za * PS], wk[j]));
      }
    }
    if (best < col[zb * PS]) {
      col[zb * PS] = best;
      chg |= 1ull << zb;
    }
  }
  return chg;
}

// Layer lists of the box being visited: H layers (x-runs) and V layers
// (y-runs) as offsets from the box's z0.  Recomputed when a CTA moves to a
// tile of another box.
struct LayerLists {
  int hl[64], vl[64];
  int nh, nv;
  int box;
};

template <int TX, int TY, bool PRIV, bool DEEP = false, bool TMA = false, bool CV = false>
__device__ __forceinline__ void process_tile(const LatParams &p, int t, float *sd, LayerLists &L, int *s_flags,
                                             int *s_act, int *s_nb = nullptr, bool warm = false,
                                             TmaCtx *tma = nullptr) {
  const int bi = box_of_tile(p, t);
  const LatBox B = load_box(p, bi);
  if (threadIdx.x == 0 && L.box != bi) {
    int nh = 0, nv = 0;
    for (int z = B.z0; z <= B.z1; ++z) {
      if (p.axis[z] == 1) L.hl[nh++] = z - B.z0;
      else if (p.axis[z] == 2) L.vl[nv++] = z - B.z0;
    }
    L.nh = nh;
    L.nv = nv;
    L.box = bi;
  }
  __syncthreads();
  const int *s_hl = L.hl, *s_vl = L.vl;
  const int nh = L.nh, nv = L.nv;
  constexpr int SX = TX + 3;
  constexpr int PS = tile_ps(TX, TY);
  constexpr int WSX = TX + 1;
  constexpr int WPS = tile_wps(TX, TY);
  const float INF_F = __int_as_float(0x7f800000);
  const int lt = t - B.tile0;
  const int tx = lt % B.ntx, ty = lt / B.ntx;
  const int32_t X0 = B.x0 + tx * TX, Y0 = B.y0 + ty * TY;
  const int tw = min(TX, B.x1 - X0 + 1), th = min(TY, B.y1 - Y0 + 1);
  const int nzb = B.z1 - B.z0 + 1;
  const int64_t nxy = (int64_t)p.nx * p.ny;
  const int64_t col0 = (int64_t)Y0 * p.nx + X0;  // node of (X0, Y0, z=0)
  float *wlo = sd + nzb * PS;          // slot 0: from the lower axis neighbour
  float *whi = wlo + nzb * WPS;        // slot 1: from the upper axis neighbour
  float *wdn = whi + nzb * WPS;        // slot 2: via from below
  float *wup = wdn + nzb * WPS;        // slot 3: via from above

  float *orig = wup + nzb * WPS;        // interior distances as loaded
  unsigned long long ts0 = 0;
  if (threadIdx.x == 0) ts0 = dev_globaltimer();
  if (threadIdx.x < 5) s_act[threadIdx.x] = 0;
  if (threadIdx.x < 6) s_flags[threadIdx.x] = 0;
  if (s_nb && threadIdx.x < 4) {  // neighbour tiles in the box: left, right, down, up (-1: box edge)
    const int d = threadIdx.x;
    s_nb[d] = d == 0 ? (tx > 0 ? t - 1 : -1)
                     : d == 1 ? (tx < B.ntx - 1 ? t + 1 : -1)
                              : d == 2 ? (ty > 0 ? t - B.ntx : -1) : (ty < B.nty - 1 ? t + B.ntx : -1);
  }
  // ---- load.  Interior cells: distance and the four in-edge weights; halo
  // cells: only those the sweeps read (x-halo of H-layer rows, y-halo of
  // V-layer columns).  Distances are read through L2 (other CTAs write them);
  // weights are read-only.  A thread's first halo cells are loaded before its
  // column (one thread per column (x, y), up to 18 layers in flight at a
  // time), so their round trip overlaps the column's.
  bool staged = false;
  if constexpr (TMA) {
    if (!warm) {
      tma_stage<TX, TY>(p, X0, Y0, B.z0, nzb, PRIV ? B.pad : 0, *tma);
      constexpr int DX = TX + 8, DY = TY + 2;
      const uint32_t *sdd = tma->sdd;
      const float4 *sw4 = (const float4 *)tma->sw;
      const int c = threadIdx.x;
      if (c < th * tw) {
        const int yy = c / tw + 1, xx = c - (yy - 1) * tw + 1;
        const int s0 = yy * SX + xx, w0 = (yy - 1) * WSX + (xx - 1);
        for (int z = 0; z < nzb; ++z) {
          const float dv = __uint_as_float(sdd[(z * DY + yy) * DX + xx + 3]);
          const float4 wv = sw4[(z * TY + yy - 1) * TX + xx - 1];
          const int wi = z * WPS + w0;
          sd[z * PS + s0] = dv;
          orig[wi] = dv;
          wlo[wi] = wv.x;
          whi[wi] = wv.y;
          wdn[wi] = wv.z;
          wup[wi] = wv.w;
        }
      }
      const int nhh = 2 * nh * th, nvh = 2 * nv * tw;
      for (int i = threadIdx.x; i < nhh + nvh; i += (TX * TY)) {
        int z, xx, yy;
        if (i < nhh) {
          const int rowi = i >> 1;
          z = s_hl[rowi / th];
          yy = rowi % th + 1;
          xx = (i & 1) ? tw + 1 : 0;
        } else {
          const int coli = (i - nhh) >> 1;
          z = s_vl[coli / tw];
          xx = coli % tw + 1;
          yy = ((i - nhh) & 1) ? th + 1 : 0;
        }
        const int32_t gx = X0 + xx - 1, gy = Y0 + yy - 1;
        float v = INF_F;
        if (gx >= B.x0 && gx <= B.x1 && gy >= B.y0 && gy <= B.y1) v = __uint_as_float(sdd[(z * DY + yy) * DX + xx + 3]);
        sd[z * PS + yy * SX + xx] = v;
      }
      staged = true;
    }
  }
  if (!staged) {
    const int nhh = 2 * nh * th, nvh = 2 * nv * tw;
    constexpr int HB = 4;  // halo cells per thread in the first batch
    float hv[HB];
    int hs[HB];
#pragma unroll
    for (int k = 0; k < HB; ++k) {
      const int i = threadIdx.x + k * (TX * TY);
      hs[k] = -1;
      hv[k] = INF_F;
      if (i < nhh + nvh) {
        int z, xx, yy;
        if (i < nhh) {
          const int rowi = i >> 1;
          z = s_hl[rowi / th];
          yy = rowi % th + 1;
          xx = (i & 1) ? tw + 1 : 0;
        } else {
          const int coli = (i - nhh) >> 1;
          z = s_vl[coli / tw];
          xx = coli % tw + 1;
          yy = ((i - nhh) & 1) ? th + 1 : 0;
        }
        const int32_t gx = X0 + xx - 1, gy = Y0 + yy - 1;
        hs[k] = z * PS + yy * SX + xx;
        if (gx >= B.x0 && gx <= B.x1 && gy >= B.y0 && gy <= B.y1)
          hv[k] = bits_f(__ldcg(&p.dist[dist_index<PRIV>(p, B, gx, gy, B.z0 + z)]));
      }
    }
    // the thread's column (x, y) of the tile (th * tw <= threads)
    const int c = threadIdx.x;
    if (warm && c < th * tw) {
      // the same tile again: its interior and weights are still in shared
      // memory and equal to what the last visit published
      const int yy = c / tw + 1, xx = c - (yy - 1) * tw + 1;
      const int s0 = yy * SX + xx, w0 = (yy - 1) * WSX + (xx - 1);
      for (int z = 0; z < nzb; ++z) orig[z * WPS + w0] = sd[z * PS + s0];
    } else if (c < th * tw) {
      const int yy = c / tw + 1, xx = c - (yy - 1) * tw + 1;
      const int64_t n0 = (int64_t)B.z0 * nxy + col0 + (int64_t)(yy - 1) * p.nx + (xx - 1);
      const int64_t d0 = dist_index<PRIV>(p, B, X0 + xx - 1, Y0 + yy - 1, B.z0);
      const int64_t dz = (!PRIV || B.dbase < 0) ? nxy : (int64_t)(B.x1 - B.x0 + 1) * (B.y1 - B.y0 + 1);
      const int s0 = yy * SX + xx, w0 = (yy - 1) * WSX + (xx - 1);
      if constexpr (DEEP) {
        // boxes of more than 12 layers: blocks of 18 layers, each fully
        // unrolled and predicated, every load of a block issued before its
        // stores (one round trip for up to 18 layers)
        load_column_blocks_impl<18, PS, WPS>(p, nzb, d0, dz, n0, nxy, sd, orig, wlo, whi, wdn, wup, s0, w0);
      } else {  // twelve layers in flight
#pragma unroll 12
        for (int z = 0; z < nzb; ++z) {
          const float dv = bits_f(__ldcg(&p.dist[d0 + z * dz]));
          const float4 wv = __ldg(&p.w4[n0 + z * nxy]);
          const int wi = z * WPS + w0;
          sd[z * PS + s0] = dv;
          orig[wi] = dv;
          wlo[wi] = wv.x;
          whi[wi] = wv.y;
          wdn[wi] = wv.z;
          wup[wi] = wv.w;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < HB; ++k)
      if (hs[k] >= 0) sd[hs[k]] = hv[k];
    for (int i = threadIdx.x + HB * (TX * TY); i < nhh + nvh; i += (TX * TY)) {
      int z, xx, yy;
      if (i < nhh) {
        const int rowi = i >> 1;
        z = s_hl[rowi / th];
        yy = rowi % th + 1;
        xx = (i & 1) ? tw + 1 : 0;
      } else {
        const int coli = (i - nhh) >> 1;
        z = s_vl[coli / tw];
        xx = coli % tw + 1;
        yy = ((i - nhh) & 1) ? th + 1 : 0;
      }
      const int32_t gx = X0 + xx - 1, gy = Y0 + yy - 1;
      float v = INF_F;
      if (gx >= B.x0 && gx <= B.x1 && gy >= B.y0 && gy <= B.y1)
        v = bits_f(__ldcg(&p.dist[dist_index<PRIV>(p, B, gx, gy, B.z0 + z)]));
      sd[z * PS + yy * SX + xx] = v;
    }
  }
  __syncthreads();
  unsigned long long ts1 = 0;
  if (threadIdx.x == 0) ts1 = dev_globaltimer();

  // ---- sweep cycles.  Each cycle: the planar runs (x-runs on H layers and
  // y-runs on V layers touch disjoint layers, so they run side by side), then
  // the via runs along z.  s_flags[c % 3] records a planar change in cycle c,
  // s_flags[3 + c % 3] a via change.  A pass that changes nothing leaves every
  // constraint it checks satisfied, so once a planar pass changes nothing
  // after a via pass that changed nothing, the tile is at its fixpoint and the
  // cycle's via pass is skipped.
  bool converged = false;
  int cyc = 0;
  const int nplan = nh * th + nv * tw;
  const bool full = tw == TX && th == TY;
  for (; cyc < MAX_CYCLES; ++cyc) {
    if (threadIdx.x == 0) {
      s_flags[(cyc + 1) % 3] = 0;
      s_flags[3 + (cyc + 1) % 3] = 0;
    }
    bool chg = false;
    if (full) {
      for (int rr = threadIdx.x; rr < nplan; rr += (TX * TY)) {
        if (rr < nh * TY) {  // x-run of an H-layer row
          const int z = s_hl[rr / TY], yy = rr % TY + 1;
          const int wo = z * WPS + (yy - 1) * WSX - 1;
          chg |= sweep_run_fixed<TX, 1, 1>(sd + z * PS + yy * SX, wlo + wo, whi + wo);
        } else {  // y-run of a V-layer column
          const int q = rr - nh * TY;
          const int z = s_vl[q / TX], xx = q % TX + 1;
          const int wo = z * WPS + (xx - 1) - WSX;
          chg |= sweep_run_fixed<TY, SX, WSX>(sd + z * PS + xx, wlo + wo, whi + wo);
        }
      }
    } else {
      for (int rr = threadIdx.x; rr < nplan; rr += (TX * TY)) {
        float *cell;
        int wo, ds, ws, n;
        if (rr < nh * th) {  // x-run of an H-layer row
          const int z = s_hl[rr / th], yy = rr % th + 1;
          cell = sd + z * PS + yy * SX;
          wo = z * WPS + (yy - 1) * WSX - 1;
          ds = 1;
          ws = 1;
          n = tw;
        } else {  // y-run of a V-layer column
          const int q = rr - nh * th;
          const int z = s_vl[q / tw], xx = q % tw + 1;
          cell = sd + z * PS + xx;
          wo = z * WPS + (xx - 1) - WSX;
          ds = SX;
          ws = WSX;
          n = th;
        }
        chg |= sweep_run(cell, ds, wlo + wo, whi + wo, ws, n);
      }
    }
    if (chg) s_flags[cyc % 3] = 1;
    __syncthreads();
    if (cyc > 0 && !s_flags[cyc % 3] && !s_flags[3 + (cyc - 1) % 3]) { converged = true; break; }
    chg = false;
    for (int c = threadIdx.x; c < tw * th; c += (TX * TY)) {
      const int xx = c % tw + 1, yy = c / tw + 1;
      if constexpr (CV) {
        const int64_t v0 = (int64_t)B.z0 * nxy + col0 + (int64_t)(yy - 1) * p.nx + (xx - 1);
        chg |= zcol_pass<PS>(sd + yy * SX + xx, p.wcol, p.nzp, v0, nxy, B.z0, nzb) != 0;
      } else {
        const int wo = (yy - 1) * WSX + (xx - 1);
        chg |= zrun<PS, WPS>(sd + yy * SX + xx, wdn + wo, wup + wo, nzb);
      }
    }
    if (chg) s_flags[3 + cyc % 3] = 1;
    __syncthreads();
    if (!s_flags[cyc % 3] && !s_flags[3 + cyc % 3]) { converged = true; break; }
  }
  unsigned long long ts2 = 0;
  if (threadIdx.x == 0) {
    ts2 = dev_globaltimer();
    atomicAdd((unsigned long long *)&p.ctl->cycles, (unsigned long long)(cyc + 1));
  }

  // ---- publish improvements; mark neighbour tiles whose halo changed
  // one thread per column (x, y) of the tile, all its layers: the layer's
  // axis decides which tile edge a changed cell activates
  const int64_t dzs = (!PRIV || B.dbase < 0) ? nxy : (int64_t)(B.x1 - B.x0 + 1) * (B.y1 - B.y0 + 1);
  for (int c = threadIdx.x; c < th * tw; c += (TX * TY)) {
    const int yy = c / tw + 1, xx = c - (yy - 1) * tw + 1;
    const int64_t d0 = dist_index<PRIV>(p, B, X0 + xx - 1, Y0 + yy - 1, B.z0);
    const int s0 = yy * SX + xx, w0 = (yy - 1) * WSX + (xx - 1);
    bool ex = false, ey = false;
    for (int z = 0; z < nzb; ++z) {
      const float v = sd[z * PS + s0];
      if (v < orig[z * WPS + w0]) {
        __stcg(&p.dist[d0 + z * dzs], f_bits(v));
        const int ax = p.axis[B.z0 + z];
        ex |= ax == 1;
        ey |= ax == 2;
      }
    }
    if (ex) {
      if (xx == 1) s_act[0] = 1;
      if (xx == tw) s_act[1] = 1;
    }
    if (ey) {
      if (yy == 1) s_act[2] = 1;
      if (yy == th) s_act[3] = 1;
    }
  }
  if (threadIdx.x == 0 && !converged) s_act[4] = 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long ts3 = dev_globaltimer();
    atomicAdd(&p.ctl->ns[0], ts1 - ts0);
    atomicAdd(&p.ctl->ns[1], ts2 - ts1);
    atomicAdd(&p.ctl->ns[2], ts3 - ts2);
  }
}

// ---------------------------------------------------------------------------
// Run visit: the tile visit of 16 x 16 tiles of up to NZM layers.
//
// The visit above keeps everything in shared memory: each relaxation reads a
// distance and a weight from it, each sweep cycle walks every run forward
// and then backward, and one more cycle that changes nothing ends the visit.
// It is bound by shared-memory accesses and by the length of the dependent
// add-min chains (1.6 us per sweep cycle of a 12-layer tile, 3.2 cycles a
// visit).  Here
//  - a thread owns one planar run (16 cells of a row on an H layer or of a
//    column on a V layer) and one via column for the whole visit, with the
//    weights of both in registers and its run's two halo values too; only
//    the distances are in shared memory, so the planar and the via passes
//    read and write them and nothing else;
//  - the forward and the backward walk of a run start from the same values,
//    run side by side and are combined with a min.  With non-negative weights
//    a shortest path inside a run never turns (the cell where it turned was
//    reached with no more), and the sums along it are those of the one-sided
//    walk, so the result is the run's fixpoint as before, bit for bit, with
//    half the chain;
//  - a pass takes only the runs (columns) in which the other pass changed a
//    cell since they were last taken, by bit sets in shared memory.  A run or
//    column just taken is at its own fixpoint, so when a pass changes
//    nothing that the other one reads, the tile is at its fixpoint and the
//    visit ends, with no confirming cycle.
// Cells outside the box hold +inf with +inf weights, so every run has its
// full length.
// Measured (before -> after, per visit: load / passes / write-back): one
// 18-layer box 2.55 / 6.77 / 1.17 -> 1.65 / 2.66 / 1.78 us; 600 x 600 x 12,
// one source, 795 -> 612 us; 1000 x 1000 x 12, 16 sources, 6.50 -> 4.95 ms;
// 2 048 boxes of up to 400 x 400 x 16, 19.1 -> 9.9 ms (against 32-wide tiles).
//
// Threads: 16 runs per layer, H runs first: 256 threads up to 16 layers, 288
// above.  Shared memory: nzb x 3 x 280 floats (distances, the two planar
// weight arrays as they pass from the column loads to the runs), with ZS
// nzb x 5 x 280 (the via weights too, where two CTAs share an SM's registers).
constexpr int kRunWS = 17;                // row stride (odd: rows and columns hit distinct banks)
constexpr int kRunPS = tile_wps(16, 16);  // layer stride
template <int NZM, bool ZS>
struct RunTile {
  static constexpr int NW = NZM > 16 ? 288 : 256;
  float lo[16], hi[16];    // the run's in-edge weights from its lower / upper neighbours
  float dn[ZS ? 1 : NZM], up[ZS ? 1 : NZM];  // the column's in-edge weights from below / above
  float ha, hb;            // the run's halo values
};

struct RunShared {
  // columns changed by the last planar pass: by row (bits x), by column (bits y)
  unsigned rowx[2][16], coly[2][16];
  // layers changed by the last via pass: by row, by column
  unsigned rowz[2][16], colz[2][16];
  unsigned cells[32 * 16];  // cells changed by the visit's planar passes: [layer][line]
  // thread 0: times in load, passes and write-back and the cycles made,
  // summed over the block's visits and added to the control block at its end
  unsigned long long ns[3], last;
  unsigned cycles;
  __device__ __forceinline__ void clear() {  // the change sets, by the first warp
    const int k = threadIdx.x >> 4, i = threadIdx.x & 15;
    rowx[k][i] = coly[k][i] = rowz[k][i] = colz[k][i] = 0;
  }
  __device__ __forceinline__ void start() { ns[0] = ns[1] = ns[2] = 0, cycles = 0; }
  __device__ __forceinline__ void lap(int i) {
    const unsigned long long t = dev_globaltimer();
    if (i >= 0) ns[i] += t - last;
    last = t;
  }
  __device__ __forceinline__ void flush(LatCtl *c) const {
    atomicAdd(&c->cycles, (unsigned long long)cycles);
    for (int i = 0; i < 3; ++i) atomicAdd(&c->ns[i], ns[i]);
  }
};

__host__ __device__ constexpr int run_smem_floats(int nzb, bool zs) { return nzb * (zs ? 5 : 3) * kRunPS; }

// Asynchronous 8-byte copy from global to shared memory.
__device__ __forceinline__ void copy8_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// OR of `v` over the visiting threads, with their barrier.
template <int NW, bool SPEC>
__device__ __forceinline__ bool tile_sync_or(bool v) {
  if (SPEC) {
    unsigned r;
    asm volatile(
        "{\n .reg .pred P, Q;\n setp.ne.u32 P, %1, 0;\n bar.red.or.pred Q, 1, %2, P;\n selp.u32 %0, 1, 0, Q;\n}"
        : "=r"(r)
        : "r"((unsigned)v), "n"(NW)
        : "memory");
    return r != 0;
  }
  return __syncthreads_or(v) != 0;
}

// Both walks over N cells: LD(i) the cells' values, LO(i) / HI(i) the weights
// from the lower / upper neighbour, a / b the values before the first and
// after the last cell, ST(i, v) stores a decreased cell.  The walks meet in
// the middle; from there on each step completes one cell on either side, so
// at most half of each walk is kept.  Returns the set of decreased cells.
template <int N, class LD, class LO, class HI, class ST>
__device__ __forceinline__ unsigned walk_both(float a, float b, LD ld, LO lo, HI hi, ST st) {
  float o[N], k[N];
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = ld(i);
  unsigned m = 0;
  auto put = [&](int i, float v) {
    if (v < o[i]) {
      st(i, v);
      m |= 1u << i;
    }
  };
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int j = N - 1 - i;
    a = fminf(__fadd_rn(a, lo(i)), o[i]);
    b = fminf(__fadd_rn(b, hi(j)), o[j]);
    if (i < j) {
      k[i] = a;
      k[j] = b;
    } else if (i == j) {
      put(i, fminf(a, b));
    } else {
      put(i, fminf(a, k[i]));
      put(j, fminf(b, k[j]));
    }
  }
  return m;
}

// Where a thread's run and column lie in tile t of box B.
struct RunGeom {
  int32_t X0, Y0, z0;  // the tile's first cell
  int tx, ty, tw, th, nzb;
  unsigned hm, vm;     // the box's H and V layers (bit 0: layer z0)
  bool run, isv, col;
  int rz, rl, rbase;   // the run: layer, line, offset of its first cell
  int xx, yy;          // the column
  int64_t n0;          // its node at z0
};
__device__ __forceinline__ RunGeom run_geom(const LatParams &p, const LatBox &B, int t) {
  RunGeom G;
  const int lt = t - B.tile0;
  G.ty = lt / B.ntx;
  G.tx = lt - G.ty * B.ntx;
  G.X0 = B.x0 + G.tx * 16;
  G.Y0 = B.y0 + G.ty * 16;
  G.z0 = B.z0;
  G.tw = min(16, B.x1 - G.X0 + 1);
  G.th = min(16, B.y1 - G.Y0 + 1);
  G.nzb = B.z1 - B.z0 + 1;
  const uint64_t lay = G.nzb >= 64 ? ~0ull : (1ull << G.nzb) - 1ull, below = (1ull << B.z0) - 1ull;
  G.hm = (unsigned)((p.hmask >> B.z0) & lay);
  G.vm = (unsigned)((p.vmask >> B.z0) & lay);
  const int nh = __popc(G.hm), nv = __popc(G.vm), tid = threadIdx.x;
  G.isv = tid >= nh * 16;
  const int ri = G.isv ? tid - nh * 16 : tid;
  G.rl = ri & 15;
  G.run = ri < 16 * (G.isv ? nv : nh) && G.rl < (G.isv ? G.tw : G.th);
  G.rz = 0;
  if (G.run) G.rz = (G.isv ? p.vlist[__popcll(p.vmask & below) + (ri >> 4)]
                           : p.hlist[__popcll(p.hmask & below) + (ri >> 4)]) - B.z0;
  G.rbase = G.isv ? G.rz * kRunPS + G.rl : G.rz * kRunPS + G.rl * kRunWS;
  G.xx = tid & 15;
  G.yy = tid >> 4;
  G.col = tid < 256 && G.xx < G.tw && G.yy < G.th;
  G.n0 = ((int64_t)B.z0 * p.ny + (G.Y0 + G.yy)) * p.nx + (G.X0 + G.xx);
  return G;
}

// Loads the tile's weights (and, with a column's own distances D0.. in global
// memory, those): the columns' loads, one thread each, then the runs' planar
// weights out of shared memory.  A barrier lies in between, so every thread
// of the visit calls it.
template <int NZM, bool SPEC, bool ZS, bool DIST>
__device__ __forceinline__ void load_tile(const LatParams &p, const RunGeom &G, RunTile<NZM, ZS> &R, float *sd,
                                          float2 *wp, float2 *wz, int64_t d0, int64_t dz) {
  constexpr int NW = RunTile<NZM, ZS>::NW, WS = kRunWS, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  const int64_t nxy = (int64_t)p.nx * p.ny;
  const int nzb = G.nzb;
  if (threadIdx.x < 256) {
    const int w0 = G.yy * WS + G.xx;
    const float4 *src = p.w4 + G.n0;
    if constexpr (ZS) {
      // the weights go to shared memory as they are, 8 bytes per copy, all
      // in flight and without registers to hold them
#pragma unroll
      for (int z = 0; z < NZM; ++z)
        if (z < nzb) {
          if (G.col) {
            copy8_async(&wp[z * PS + w0], src + z * nxy);
            copy8_async(&wz[z * PS + w0], (const float2 *)(src + z * nxy) + 1);
          } else {
            wp[z * PS + w0] = wz[z * PS + w0] = make_float2(INF_F, INF_F);
          }
        }
    }
    float dv[DIST ? NZM : 1];
    float4 wv[ZS ? 1 : NZM];
#pragma unroll
    for (int z = 0; z < NZM; ++z) {
      if (DIST) dv[DIST ? z : 0] = INF_F;
      if (!ZS) wv[ZS ? 0 : z] = make_float4(INF_F, INF_F, INF_F, INF_F);
      if (G.col && z < nzb) {
        if (DIST) dv[DIST ? z : 0] = bits_f(__ldcg(&p.dist[d0 + z * dz]));
        if (!ZS) wv[ZS ? 0 : z] = __ldg(src + z * nxy);
      }
    }
#pragma unroll
    for (int z = 0; z < NZM; ++z) {
      if (z < nzb) {
        if (DIST) sd[z * PS + w0] = dv[DIST ? z : 0];
        if (!ZS) wp[z * PS + w0] = make_float2(wv[ZS ? 0 : z].x, wv[ZS ? 0 : z].y);
      }
      if constexpr (!ZS) {
        R.dn[z] = wv[z].z;
        R.up[z] = wv[z].w;
      }
    }
    if (ZS) asm volatile("cp.async.wait_all;" ::: "memory");
  }
  tile_sync<NW, SPEC>();
  if (G.run) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 w = wp[G.rbase + i * (G.isv ? WS : 1)];
      R.lo[i] = w.x;
      R.hi[i] = w.y;
    }
  }
}

// The passes of a visit, from the runs marked `dirty` (and, with force, every
// column) to the tile's fixpoint, at most max_cycles.  runm / colm collect
// the cells changed in the thread's run and column.  Ends with a barrier
// after the last change; returns whether the fixpoint was reached.
template <int NZM, bool SPEC, bool CV, bool ZS>
__device__ __forceinline__ bool run_passes(const LatParams &p, const RunGeom &G, const RunTile<NZM, ZS> &R,
                                           RunShared &S, float *sd, const float2 *wz, float ha, float hb, bool dirty,
                                           bool force, int max_cycles, unsigned &runm, unsigned &colm) {
  constexpr int NW = RunTile<NZM, ZS>::NW, WS = kRunWS, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  const int nzb = G.nzb;
  float *const cd = sd + G.yy * WS + G.xx;  // the column's distances
  const float2 *const cw = wz + G.yy * WS + G.xx;
  auto run_pass = [&](float *c, auto stride) {
    constexpr int DS = decltype(stride)::value;
    return walk_both<16>(
        ha, hb, [&](int i) { return c[i * DS]; }, [&](int i) { return R.lo[i]; }, [&](int i) { return R.hi[i]; },
        [&](int i, float v) { c[i * DS] = v; });
  };
  bool again = false, converged = false;
  int cyc = 0;
  for (; cyc < max_cycles; ++cyc) {
    const int k = cyc & 1;
    unsigned m = 0;
    if (dirty) {
      if (G.isv) {
        m = run_pass(sd + G.rbase, std::integral_constant<int, WS>());
        if (m) atomicOr(&S.coly[k][G.rl], m);
      } else {
        m = run_pass(sd + G.rbase, std::integral_constant<int, 1>());
        if (m) atomicOr(&S.rowx[k][G.rl], m);
      }
      runm |= m;
    }
    const bool all = force && cyc == 0;
    if (!tile_sync_or<NW, SPEC>(m != 0 || again) && !all) {
      converged = true;
      break;
    }
    unsigned mz = 0;
    if (G.col && (all || again || (((S.rowx[k][G.yy] >> G.xx) | (S.coly[k][G.xx] >> G.yy)) & 1u))) {
      if constexpr (CV) mz = (unsigned)zcol_pass<PS>(cd, p.wcol, p.nzp, G.n0, (int64_t)p.nx * p.ny, G.z0, nzb);
      else
        mz = walk_both<NZM>(
            INF_F, INF_F, [&](int z) { return z < nzb ? cd[z * PS] : INF_F; },
            [&](int z) { return ZS ? (z < nzb ? cw[z * PS].x : INF_F) : R.dn[ZS ? 0 : z]; },
            [&](int z) { return ZS ? (z < nzb ? cw[z * PS].y : INF_F) : R.up[ZS ? 0 : z]; },
            [&](int z, float v) { cd[z * PS] = v; });
      if (mz) {
        if (mz & G.hm) atomicOr(&S.rowz[k][G.yy], mz & G.hm);
        if (mz & G.vm) atomicOr(&S.colz[k][G.xx], mz & G.vm);
        colm |= mz;
      }
    }
    // one Gauss-Seidel pass over a column's layer pairs is not its fixpoint:
    // a column-via column that changed is taken again
    if (CV) again = mz != 0;
    if (threadIdx.x < 16) {
      S.rowx[k ^ 1][threadIdx.x] = S.coly[k ^ 1][threadIdx.x] = 0;
      S.rowz[k ^ 1][threadIdx.x] = S.colz[k ^ 1][threadIdx.x] = 0;
    }
    if (!tile_sync_or<NW, SPEC>(CV ? mz != 0 : (mz & (G.hm | G.vm)) != 0)) {
      converged = true;
      break;
    }
    dirty = G.run && (((G.isv ? S.colz[k][G.rl] : S.rowz[k][G.rl]) >> G.rz) & 1u);
  }
  if (threadIdx.x == 0) S.cycles += cyc + 1;
  return converged;
}

// What a search with a target passes on to the next tile.
//
// U, the target's distance so far, only falls, and a distance x of cell v is
// of use only if x and what is still to go from v do not exceed it.  To go are
// at least |dx| + |dy| planar steps and |dz| vias, each at its smallest weight
// in the launch (goal_weights), so an improvement with x + to go > goal_limit
// activates no tile.  Every cell on a shortest path to the target, those that
// tie among them, passes, so the path is the one of the whole search (cells
// that do not pass keep upper bounds, which the backtrace never takes for a
// parent: rounded sums are monotone).
//
// The margin.  The searched sums are rounded, the bound is not.  With r = U /
// smallest weight below 2^20 each step of a path adds at least 15/16 of its
// weight, so a path has at most r / 0.93 steps, each rounded by at most U
// 2^-24: the sum falls short of the exact one by at most 6.5e-8 r U.  Beyond
// that ratio, and with negative weights, nothing is held back; with zero
// weights x > U decides (no margin: rounded sums never fall).
//
// Half of a box lies nearer than a target drawn from it, and the visits of the
// other half, and corrections that come too late to matter, went into nothing:
// 2 048 boxes of up to 400 x 400 x 16 9.8 -> 6.5 ms, 512 boxes 2.78 -> 1.91 ms.
struct GoalWeights {
  float xy, z;
};
__device__ __forceinline__ GoalWeights goal_weights(const int *wmin) {
  const int mp = __ldg(&wmin[0]), mv = __ldg(&wmin[1]);
  if (min(mp, mv) <= 0) return {0.0f, 0.0f};
  return {__int_as_float(mp) * 0.9999f, __int_as_float(mv) * 0.9999f};
}
__device__ __forceinline__ float goal_limit(float u, const int *wmin) {
  const float INF_F = __int_as_float(0x7f800000);
  const int lo = min(__ldg(&wmin[0]), __ldg(&wmin[1]));
  if (lo < 0) return INF_F;
  if (lo == 0) return u;
  const float r = u / __int_as_float(lo);
  return r < 1048576.0f ? u + u * (r * 1.2e-7f + 1e-6f) : INF_F;
}

// The same visit contract as process_tile.  warm: the tile was visited last
// by this block (its distances are in shared memory, its weights in R), only
// the halo is read again and only the runs whose halo improved are taken
// first.  A tile whose last visit stopped at MAX_CYCLES, or that holds a
// seed, has its stamp set: then every column is taken too.
//
// B: the tile's box, in shared memory.  (Looked up by the visit itself, the
// binary search over the boxes and the box's fields were dependent trips to
// L2 - the streamed weights evict them from L1 - and cost 3 us of an 11 us
// visit with 16 boxes and two CTAs per SM.)
//
// GOAL: the box has a target (SB.gx); s_act[0..3] are then the smallest
// distances passed on at each side, to go included, as float bits.
template <int NZM, bool PRIV, bool SPEC, bool CV, bool ZS, bool GOAL = false>
__device__ __forceinline__ void visit_runs(const LatParams &p, int t, const LatBox &SB, float *sd,
                                           RunTile<NZM, ZS> &R, RunShared &S, int *s_act, int *s_nb, bool warm) {
  constexpr int NW = RunTile<NZM, ZS>::NW, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  const LatBox B = SB;
  const RunGeom G = run_geom(p, B, t);
  const int tid = threadIdx.x;
  if (tid == 0) S.lap(-1);
  if (tid < 5) s_act[tid] = GOAL && tid < 4 ? 0x7f800000 : 0;
  if (s_nb && tid < 4) {  // neighbour tiles in the box: left, right, down, up (-1: box edge)
    s_nb[tid] = tid == 0 ? (G.tx > 0 ? t - 1 : -1)
                         : tid == 1 ? (G.tx < B.ntx - 1 ? t + 1 : -1)
                                    : tid == 2 ? (G.ty > 0 ? t - B.ntx : -1) : (G.ty < B.nty - 1 ? t + B.ntx : -1);
  }
  if (tid < 32) S.clear();
  // ---- load: the run's halo cells (where the box has them), then the column
  float ha = INF_F, hb = INF_F;
  if (G.run) {
    const int32_t gx = G.isv ? G.X0 + G.rl : G.X0, gy = G.isv ? G.Y0 : G.Y0 + G.rl, gz = B.z0 + G.rz;
    if (G.isv) {
      if (G.Y0 > B.y0) ha = bits_f(__ldcg(&p.dist[dist_index<PRIV>(p, B, gx, gy - 1, gz)]));
      if (G.Y0 + 16 <= B.y1) hb = bits_f(__ldcg(&p.dist[dist_index<PRIV>(p, B, gx, gy + 16, gz)]));
    } else {
      if (G.X0 > B.x0) ha = bits_f(__ldcg(&p.dist[dist_index<PRIV>(p, B, gx - 1, gy, gz)]));
      if (G.X0 + 16 <= B.x1) hb = bits_f(__ldcg(&p.dist[dist_index<PRIV>(p, B, gx + 16, gy, gz)]));
    }
  }
  const bool force = __ldcg(&p.stamp[t]) != 0;
  const int64_t dz =
      (!PRIV || B.dbase < 0) ? (int64_t)p.nx * p.ny : (int64_t)(B.x1 - B.x0 + 1) * (B.y1 - B.y0 + 1);
  const int64_t d0 = G.col ? dist_index<PRIV>(p, B, G.X0 + G.xx, G.Y0 + G.yy, B.z0) : 0;
  float2 *const wp = (float2 *)(sd + G.nzb * PS);  // planar weight pairs
  float2 *const wz = wp + G.nzb * PS;              // via weight pairs (ZS)
  bool dirty = G.run;
  if (!warm) {
    load_tile<NZM, SPEC, ZS, true>(p, G, R, sd, wp, wz, d0, dz);
  } else {
    dirty = G.run && (force || ha < R.ha || hb < R.hb);
    tile_sync<NW, SPEC>();
  }
  R.ha = ha;
  R.hb = hb;
  if (tid == 0) S.lap(0);

  unsigned runm = 0, colm = 0;
  const bool converged =
      run_passes<NZM, SPEC, CV, ZS>(p, G, R, S, sd, wz, ha, hb, dirty, force, MAX_CYCLES, runm, colm);
  if (tid == 0) S.lap(1);

  // ---- publish improvements; mark neighbour tiles whose halo changed.  One
  // thread per column: the layers its own passes changed, and its bits of the
  // runs' changed cells.
  if (G.run) S.cells[G.rz * 16 + G.rl] = runm;
  tile_sync<NW, SPEC>();
  if (G.col) {
    const float *const cd = sd + G.yy * kRunWS + G.xx;
#pragma unroll
    for (int z = 0; z < NZM; ++z)
      if (((G.hm | G.vm) >> z) & 1u) {
        const bool h = (G.hm >> z) & 1u;
        if ((S.cells[z * 16 + (h ? G.yy : G.xx)] >> (h ? G.xx : G.yy)) & 1u) colm |= 1u << z;
      }
#pragma unroll
    for (int z = 0; z < NZM; ++z)
      if ((colm >> z) & 1u) __stcg(&p.dist[d0 + z * dz], f_bits(cd[z * PS]));
    if constexpr (GOAL) {
      // per side the smallest x + to go
      const GoalWeights g = goal_weights(p.wmin);
      const float to_go = g.xy * (float)(abs(G.X0 + G.xx - SB.gx) + abs(G.Y0 + G.yy - SB.gy));
      float h = INF_F, v = INF_F;
#pragma unroll
      for (int z = 0; z < NZM; ++z)
        if ((colm >> z) & 1u) {
          const float f = cd[z * PS] + (to_go + g.z * (float)abs(B.z0 + z - SB.gz));
          if ((G.hm >> z) & 1u) h = fminf(h, f);
          else v = fminf(v, f);
        }
      if (h < INF_F) {
        if (G.xx == 0) atomicMin(&s_act[0], __float_as_int(h));
        if (G.xx == G.tw - 1) atomicMin(&s_act[1], __float_as_int(h));
      }
      if (v < INF_F) {
        if (G.yy == 0) atomicMin(&s_act[2], __float_as_int(v));
        if (G.yy == G.th - 1) atomicMin(&s_act[3], __float_as_int(v));
      }
    } else {
      if (colm & G.hm) {
        if (G.xx == 0) s_act[0] = 1;
        if (G.xx == G.tw - 1) s_act[1] = 1;
      }
      if (colm & G.vm) {
        if (G.yy == 0) s_act[2] = 1;
        if (G.yy == G.th - 1) s_act[3] = 1;
      }
    }
  }
  if (tid == 0) {
    if (!converged) s_act[4] = 1;
    if (force == converged) p.stamp[t] = converged ? 0u : 1u;
  }
  tile_sync<NW, SPEC>();
  if (tid == 0) S.lap(2);
}

// ---------------------------------------------------------------------------
// Owner schedule: launches with at most one tile per resident CTA.
//
// One search is bound by the chain of tile visits along its wave front, and a
// visit of the queue schedule spends more on handing the tile over (the
// queue's atomics, loading distances and weights, writing back) than on its
// passes, which in turn start on values that improve while they run.  Here
// tile t belongs to CTA t for the whole search: distances in shared memory,
// weights in registers, loaded once, and the CTAs relax their tiles
// continuously.  Neighbours exchange only the values of boundary cells: each
// tile has an exchange row per side of its runs (exch[tile][side][run]), which
// the neighbour's runs write with plain stores as soon as a pass has improved
// a boundary cell.  A distance is an upper bound at any time and only falls,
// so a halo value needs no flag to go with it: every cycle reads the rows
// anew (coalesced, one value per run and side, the loads overlapping the via
// pass), takes what improved, and an idle tile polls them.  A hop of the wave
// front costs one pass, one store and one load.
//
// Termination.  Publications are also counted as messages (inbox[tile]), by a
// helper warp beside the workers, so that no worker waits for an atomic.  The
// helper reads the inbox count c and asks the workers (s_req); when a whole
// cycle whose halo loads came after that changed nothing, they answer
// (s_ack), and the helper first sends the messages for everything published
// so far (sent count, fence, inbox of the neighbour) and then counts c as
// dealt with.  CTA 0's helper adds up the dealt-with counts and then the sent
// counts; equal sums mean that nothing is under way: both only grow, the
// sent sum was read later, and a tile that works on values whose message has
// not come yet is covered by the sender, which still owes that message.  The
// seeds' tiles start with one message each, sent by the launch.
//
// An owner waits for messages as long as the search runs, so what bounds its
// wait is the launch's time (ORSP_BUDGET_NS), not that of a single wait.
//
// Measured, search kernel, queue schedule with run visits -> owners: 49 tiles
// of 18 layers 193 -> 57 us, 100 x 100 x 4 board 77 (before run visits) -> 19
// us, 91 tiles of a 200 x 200 x 6 column-via lattice 248 -> 133 us.
struct OwnParams {
  LatParams l;
  int32_t tcap, nr;              // tiles (at most), values per exchange row
  int32_t nzb;
  float *exch;                   // [tcap][2][nr]
  unsigned *inbox, *sent, *got;  // [tcap], [tcap + 1], [tcap + 1]
  int *done;
  int32_t *seedt;                // tile of each seed, -1: outside
  int32_t nseeds;
  const int32_t *seeds;
  const float *seed_cost;
  int one;      // a single box, by value
  LatBox box1;
  // weights gathered by the launch's preparation (0: they are there, 1: of the
  // boxes, 2: of the whole lattice)
  int gather;
  const int32_t *slot_eid;
  const float *cost;
  float4 *w;
  uint8_t *par;  // parents recorded instead of distances (NULL: distances), par_bytes per tile
  int par_bytes;
};
constexpr int kOwnSeeds = 4096;

__device__ __forceinline__ LatBox own_box(const OwnParams &o, int b) { return o.one ? o.box1 : load_box(o.l, b); }

// Prepares a launch: block (0, 0) the control words and the seeds' messages, the
// other blocks the exchange rows and the weights of box blockIdx.y: a search is
// short enough for a launch of its own to show.
__global__ void own_init_kernel(const __grid_constant__ OwnParams o) {
  const LatParams &p = o.l;
  const float INF_F = __int_as_float(0x7f800000);
  if (blockIdx.x > 0) {
    const int64_t bx = (int64_t)blockIdx.y * (gridDim.x - 1) + blockIdx.x - 1;
    const int64_t n = (int64_t)o.tcap * 2 * o.nr / 4, s = (int64_t)(gridDim.x - 1) * gridDim.y * blockDim.x;
    for (int64_t i = bx * blockDim.x + threadIdx.x; i < n; i += s)
      ((float4 *)o.exch)[i] = make_float4(INF_F, INF_F, INF_F, INF_F);
    if (o.gather) {
      int32_t x0 = 0, y0 = 0, z0 = 0;
      int64_t bw = p.nx, bh = p.ny, bd = p.nz;
      if (o.gather == 1) {
        const LatBox B = own_box(o, blockIdx.y);
        x0 = B.x0, y0 = B.y0, z0 = B.z0;
        bw = B.x1 - B.x0 + 1, bh = B.y1 - B.y0 + 1, bd = B.z1 - B.z0 + 1;
      }
      gather_cells(o.slot_eid, o.cost, o.w, p.N, p.nx, p.ny, x0, bw, y0, bh, z0, bw * bh * bd,
                   (int64_t)(blockIdx.x - 1) * blockDim.x + threadIdx.x, (int64_t)(gridDim.x - 1) * blockDim.x);
    }
    return;
  }
  if (blockIdx.y > 0) return;
  LatCtl *c = p.ctl;
  if (threadIdx.x == 0) {
    c->err = 0;
    c->rounds = c->visits = 0;
    c->cycles = 0;
    for (int i = 0; i < 4; ++i) c->ns[i] = 0;
    *o.done = 0;
  }
  for (int i = threadIdx.x; i < o.tcap; i += blockDim.x) o.inbox[i] = 0;
  for (int i = threadIdx.x; i <= o.tcap; i += blockDim.x) o.sent[i] = o.got[i] = 0;
  __syncthreads();
  const int32_t plane = p.nx * p.ny;
  for (int i = threadIdx.x; i < o.nseeds; i += blockDim.x) {
    const int32_t s = o.seeds[i];
    int t = -1;
    const float c0 = o.seed_cost ? o.seed_cost[i] : 0.0f;
    if (s >= 0 && s < plane * p.nz && (!p.roi_map || __ldg(&p.roi_map[s]) >= 0) && c0 >= 0.0f && c0 < INF_F) {
      const int32_t z = s / plane, r = s - z * plane, y = r / p.nx, x = r - y * p.nx;
      const int lo = p.seed_per_box ? i : 0, hi = p.seed_per_box ? min(i + 1, p.nbox) : p.nbox;
      for (int b = lo; b < hi && t < 0; ++b) {
        const LatBox B = own_box(o, b);
        if (x >= B.x0 && x <= B.x1 && y >= B.y0 && y <= B.y1 && z >= B.z0 && z <= B.z1) t = tile_of<16, 16>(B, x, y);
      }
    }
    o.seedt[i] = t;
    if (t >= 0 && atomicExch(&o.inbox[t], 1u) == 0u) atomicAdd(&o.sent[o.tcap], 1u);
  }
}

__device__ __forceinline__ float ld_relaxed_f32(const float *p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_f32(float *p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// What the workers and the helper warp of an owner share.
struct OwnShared {
  volatile unsigned req, ack;  // inbox count to deal with, last one dealt with
  int pub[4];                  // sides with publications not yet sent as messages
  volatile int stop, rel;      // the search is over; the tile is given back once it is idle
  volatile int idle, out;      // no work at the last look; the tile's distances are written
  volatile int quit;           // the launch has failed: the workers leave, idle or not
  int tile;
  LatBox box;
};

// The cycles of an owned tile, from the halo values na / nb until it is idle
// and asked to stop, or the launch has failed.  (A tile can stay busy for good:
// costs whose sum around a loop is negative lower its distances until the
// floats saturate.  Every kQuitCycles cycles, under a millisecond, the workers
// look whether to leave all the same.)  pa / pb: the boundary values last
// published; snap: the inbox count read before na and nb.  Returns the number
// of cycles.
constexpr unsigned kQuitCycles = 1024;
template <int NZM, bool CV, bool ZS>
__device__ __forceinline__ unsigned own_cycles(const OwnParams &o, const LatBox &B, const RunGeom &G,
                                               const RunTile<NZM, ZS> &R, RunShared &S, OwnShared &Q, float *sd,
                                               const float2 *wz, float *ex, float na, float nb, float pa, float pb,
                                               bool dirty, bool all, unsigned snap, float &ha, float &hb) {
  constexpr int NW = RunTile<NZM, ZS>::NW, WS = kRunWS, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  const LatParams &p = o.l;
  const int tid = threadIdx.x;
  const bool run = G.run, col = G.col;
  // the neighbours' exchange values that this thread's run writes
  const int step = (G.isv ? B.ntx : 1) * 2 * o.nr;
  const bool lo = run && (G.isv ? G.ty > 0 : G.tx > 0), hi = run && (G.isv ? G.ty < B.nty - 1 : G.tx < B.ntx - 1);
  ha = hb = INF_F;  // halo values taken
  bool again = false, idle = false;
  unsigned cycles = 0;
  float *const cd = sd + G.yy * WS + G.xx;
  const float2 *const cw = wz + G.yy * WS + G.xx;
  for (int k = 0;; k ^= 1) {
    // ---- halo values read since the last look
    unsigned next_snap = 0;
    if (na < ha) ha = na, dirty = true;
    if (nb < hb) hb = nb, dirty = true;
    if (idle) {  // nothing to do at the last look
      const bool stop = Q.stop != 0 || Q.rel != 0;
      if (!tile_sync_or<NW, true>(dirty || stop)) {
        if (tid == 0) {
          Q.ack = snap;
          Q.idle = 1;
          snap = Q.req;
        }
        tile_sync<NW, true>();
        if (run) na = ld_relaxed_f32(ex), nb = ld_relaxed_f32(ex + o.nr);
        continue;
      }
      if (!tile_sync_or<NW, true>(dirty)) break;
      idle = false;
      if (tid == 0) Q.idle = 0;
    }
    // ---- planar pass, boundary improvements published
    unsigned m = 0;
    if (dirty) {
      auto pass = [&](float *c, auto stride) {
        constexpr int DS = decltype(stride)::value;
        m = walk_both<16>(
            ha, hb, [&](int i) { return c[i * DS]; }, [&](int i) { return R.lo[i]; }, [&](int i) { return R.hi[i]; },
            [&](int i, float v) { c[i * DS] = v; });
        const float v0 = c[0], v1 = c[15 * DS];
        if (lo && v0 < pa) {
          pa = v0;
          st_relaxed_f32(ex - step + o.nr, v0);
          __threadfence_block();
          Q.pub[G.isv ? 2 : 0] = 1;
        }
        if (hi && v1 < pb) {
          pb = v1;
          st_relaxed_f32(ex + step, v1);
          __threadfence_block();
          Q.pub[G.isv ? 3 : 1] = 1;
        }
      };
      if (G.isv) {
        pass(sd + G.rbase, std::integral_constant<int, WS>());
        if (m) atomicOr(&S.coly[k][G.rl], m);
      } else {
        pass(sd + G.rbase, std::integral_constant<int, 1>());
        if (m) atomicOr(&S.rowx[k][G.rl], m);
      }
    }
    if (tid == 0) next_snap = Q.req;
    const bool any = tile_sync_or<NW, true>(m != 0 || again);
    // the next cycle's halo values; their round trip overlaps the via pass
    if (run) na = ld_relaxed_f32(ex), nb = ld_relaxed_f32(ex + o.nr);
    // ---- via pass
    unsigned mz = 0;
    if ((any || all) && col && (all || again || (((S.rowx[k][G.yy] >> G.xx) | (S.coly[k][G.xx] >> G.yy)) & 1u))) {
      if constexpr (CV) mz = (unsigned)zcol_pass<PS>(cd, p.wcol, p.nzp, G.n0, (int64_t)p.nx * p.ny, G.z0, G.nzb);
      else
        mz = walk_both<NZM>(
            INF_F, INF_F, [&](int z) { return z < G.nzb ? cd[z * PS] : INF_F; },
            [&](int z) { return ZS ? (z < G.nzb ? cw[z * PS].x : INF_F) : R.dn[ZS ? 0 : z]; },
            [&](int z) { return ZS ? (z < G.nzb ? cw[z * PS].y : INF_F) : R.up[ZS ? 0 : z]; },
            [&](int z, float v) { cd[z * PS] = v; });
      if (mz & G.hm) atomicOr(&S.rowz[k][G.yy], mz & G.hm);
      if (mz & G.vm) atomicOr(&S.colz[k][G.xx], mz & G.vm);
    }
    if (CV) again = mz != 0;
    all = false;
    if (tid < 16) {
      S.rowx[k ^ 1][tid] = S.coly[k ^ 1][tid] = 0;
      S.rowz[k ^ 1][tid] = S.colz[k ^ 1][tid] = 0;
    }
    const bool zany = tile_sync_or<NW, true>(mz != 0);
    dirty = run && (((G.isv ? S.colz[k][G.rl] : S.rowz[k][G.rl]) >> G.rz) & 1u);
    if (++cycles % kQuitCycles == 0 && tile_sync_or<NW, true>(Q.quit != 0)) break;
    idle = !any && !zany;
    if (tid == 0) {
      // a cycle without a change answers the request read before its halo loads
      if (idle) Q.ack = snap;
      snap = next_snap;
    }
  }
  return cycles;
}

// The parents of a column's cells at the fixpoint, by the backtrace's rule (the
// smallest distance d with fl(d + w) = the cell's, then the smallest node id; at
// an equal distance smaller ids only), from the distances, weights and halo
// values on chip.  The walk then reads half a byte per cell from shared memory
// instead of distances and weights through L2, and no distances are written:
// routing 270 nets twice on 100 x 100 x 4 13.3 -> 12.3 ms, one net 87 -> 81 us.
// Only where a box's parents fit the walk's shared memory (kParSmem: 88 tiles of
// 18 layers, 266 of 5, every owner launch of up to 4) and nothing else reads
// distances.
template <int NZM, bool ZS>
__device__ __forceinline__ void record_parents(const RunGeom &G, const RunTile<NZM, ZS> &R, const float *sd,
                                               const float2 *wp, const float2 *wz, uint8_t *par) {
  constexpr int WS = kRunWS, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  const int at = G.yy * WS + G.xx;
  unsigned byte = 0;
#pragma unroll
  for (int z = 0; z < NZM; ++z) {
    if (z >= G.nzb) break;
    const float v = sd[z * PS + at];
    unsigned code = orsp::kParFar;
    if (v < INF_F) {
      code = orsp::kParNone;
      float best = INF_F;
      auto take = [&](unsigned s, float d, float w, bool smaller) {
        if (d < best && __fadd_rn(d, w) == v && (d < v || (d == v && smaller))) {
          best = d;
          code = s;
        }
      };
      // in the order of the ids
      if (z > 0) take(2, sd[(z - 1) * PS + at], ZS ? wz[z * PS + at].x : R.dn[ZS ? 0 : z], true);
      const bool h = (G.hm >> z) & 1u;
      if (h || ((G.vm >> z) & 1u)) {
        const int line = h ? G.yy : G.xx, i = h ? G.xx : G.yy, step = h ? 1 : WS;
        const float2 halo = wp[z * PS + line * WS + 16], w = wp[z * PS + at];
        take(0, i > 0 ? sd[z * PS + at - step] : halo.x, w.x, true);
        take(1, i < 15 ? sd[z * PS + at + step] : halo.y, w.y, false);
      }
      if (z + 1 < G.nzb) take(3, sd[(z + 1) * PS + at], ZS ? wz[z * PS + at].y : R.up[ZS ? 0 : z], false);
    }
    byte |= code << ((z & 1) * 4);
    if ((z & 1) || z + 1 == G.nzb) {
      par[(z >> 1) * 256 + G.yy * 16 + G.xx] = (uint8_t)byte;
      byte = 0;
    }
  }
}

template <int NZM, bool PRIV, bool CV, bool ZS, int MINB>
__global__ void __launch_bounds__(RunTile<NZM, ZS>::NW + 32, MINB)
    lattice_own_kernel(const __grid_constant__ OwnParams o) {
  constexpr int NW = RunTile<NZM, ZS>::NW, WS = kRunWS, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  extern __shared__ __align__(128) float sd[];
  __shared__ RunShared S;
  __shared__ OwnShared Q;
  const LatParams &p = o.l;
  const int t = blockIdx.x, tid = threadIdx.x;
  // the tile's box (a box sized on the device may have fewer tiles than the launch)
  const LatBox B = own_box(o, p.nbox == 1 ? 0 : box_of_tile(p, t));
  const bool mine = t < B.tile0 + B.ntx * B.nty;
  const unsigned long long t_start = dev_globaltimer();
  if (tid < 4) Q.pub[tid] = 0;
  if (tid < 32) S.clear();
  if (tid == 0) {
    Q.req = Q.ack = 0;
    Q.stop = Q.rel = Q.quit = 0;
    S.start();
    S.lap(-1);
  }
  __syncthreads();

  if (tid >= NW) {
    // ------------------------------------------------------------ helper
    const int lane = tid - NW;
    unsigned sent = 0, got = 0, asked = 0;
    // messages to the neighbours on the sides in m, the sent count first.  The
    // lanes that took the sides' flags fence, each behind the boundary values
    // published before its flag, and lane 0 counts the messages after them: a
    // neighbour that sees its count reads those values
    auto send = [&](unsigned m) {
      sent += __popc(m);
      if (lane == 0) __stcg(&o.sent[t], sent);
      __threadfence();
      __syncwarp();
      if (lane == 0) {
        if (m & 1u) atomicAdd(&o.inbox[t - 1], 1u);
        if (m & 2u) atomicAdd(&o.inbox[t + 1], 1u);
        if (m & 4u) atomicAdd(&o.inbox[t - B.ntx], 1u);
        if (m & 8u) atomicAdd(&o.inbox[t + B.ntx], 1u);
      }
    };
    for (unsigned spins = 0;; ++spins) {
      // publications become messages: one lane per side
      const bool pub = lane < 4 && atomicExch(&Q.pub[lane], 0) != 0;
      const unsigned pm = __ballot_sync(ORSP_FULL_MASK, pub);
      const bool acked = asked != got && __shfl_sync(ORSP_FULL_MASK, Q.ack, 0) == asked;
      if (acked) {
        // everything published up to the answer: flags raised since the
        // exchange above are part of it (what lane 0 saw, all lanes follow)
        __syncwarp();
        __threadfence_block();
        const bool more = lane < 4 && atomicExch(&Q.pub[lane], 0) != 0;
        const unsigned both = pm | __ballot_sync(ORSP_FULL_MASK, more);
        if (both) send(both);
        got = asked;
        if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&o.got[t]), "r"(got) : "memory");
      } else if (pm) {
        send(pm);
      }
      unsigned in = 0;
      int stop = 0;
      if (lane == 0) {
        in = ld_acquire_u32(&o.inbox[t]);
        if (ld_acquire_u32((const unsigned *)&p.ctl->err)) stop = Q.quit = 1;
        if (ld_acquire_u32((const unsigned *)o.done)) stop = 1;
      }
      in = __shfl_sync(ORSP_FULL_MASK, in, 0);
      if (asked == got && in != got) {
        asked = in;
        if (lane == 0) Q.req = in;
      }
      if (t == 0 && asked == got) {
        unsigned a = 0, b = 0;
        for (int i = lane; i <= o.tcap; i += 32) a += ld_acquire_u32(&o.got[i]);
        a = __reduce_add_sync(ORSP_FULL_MASK, a);
        __threadfence();
        for (int i = lane; i <= o.tcap; i += 32) b += ld_acquire_u32(&o.sent[i]);
        b = __reduce_add_sync(ORSP_FULL_MASK, b);
        if (a == b) {
          stop = 1;
          if (lane == 0) atomicExch(o.done, 1);
        }
      }
      if (lane == 0 && (spins & 31u) == 31u && dev_globaltimer() - t_start > p.budget_ns) {
        atomicCAS(&p.ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
        stop = Q.quit = 1;
      }
      if (__shfl_sync(ORSP_FULL_MASK, stop, 0)) break;
    }
    if (lane == 0) Q.stop = 1;
    return;
  }

  // -------------------------------------------------------------- workers
  const RunGeom G = run_geom(p, B, t);
  const bool run = mine && G.run, col = mine && G.col;
  RunTile<NZM, ZS> R;
  float2 *const wp = (float2 *)(sd + o.nzb * PS), *const wz = wp + o.nzb * PS;
  float *const ex = o.exch + (int64_t)t * 2 * o.nr + tid;
  bool seeded = false;
  if (mine) {
    for (int i = tid; i < o.nzb * PS; i += NW) sd[i] = INF_F;
    load_tile<NZM, true, ZS, false>(p, G, R, nullptr, wp, wz, 0, 0);  // (with a barrier)
    for (int i = tid; i < o.nseeds; i += NW) {
      if (o.seedt[i] != t) continue;
      seeded = true;
      const int32_t v = o.seeds[i], plane = p.nx * p.ny, z = v / plane, r = v - z * plane, y = r / p.nx, x = r - y * p.nx;
      atomicMin((unsigned *)&sd[(z - B.z0) * PS + (y - G.Y0) * WS + (x - G.X0)],
                f_bits(o.seed_cost ? o.seed_cost[i] : 0.0f));
    }
  }
  seeded = tile_sync_or<NW, true>(seeded);
  if (tid == 0) S.lap(0);
  unsigned cycles = 0;
  float ha = INF_F, hb = INF_F;
  if (mine)
    cycles = own_cycles<NZM, CV, ZS>(o, B, G, R, S, Q, sd, wz, ex, INF_F, INF_F, INF_F, INF_F, run && seeded, seeded,
                                     0u, ha, hb);
  // ---- the box's parents, or its distances.  (The runs' halo values go to the
  // spare column of the planar weights.)
  if (!CV && o.par && run) wp[G.rz * PS + G.rl * WS + 16] = make_float2(ha, hb);
  tile_sync<NW, true>();
  if (!CV && o.par) {
    if (col) record_parents<NZM, ZS>(G, R, sd, wp, wz, o.par + (int64_t)t * o.par_bytes);
  } else if (col) {
    const int64_t dz = (!PRIV || B.dbase < 0) ? (int64_t)p.nx * p.ny : (int64_t)(B.x1 - B.x0 + 1) * (B.y1 - B.y0 + 1);
    const int64_t d0 = dist_index<PRIV>(p, B, G.X0 + G.xx, G.Y0 + G.yy, B.z0);
    const float *const cd = sd + G.yy * kRunWS + G.xx;
    for (int z = 0; z < G.nzb; ++z) p.dist[d0 + z * dz] = f_bits(cd[z * PS]);
  }
  if (tid == 0 && mine) {
    S.lap(1);
    S.cycles = cycles;
    atomicAdd(&p.ctl->visits, 1u);
    S.flush(p.ctl);
  }
}

// Visiting owners: launches with more tiles than resident CTAs and wave fronts
// that do not fill the chip.  Like the owners' bound by the chain of hops along
// the front, but a tile has an owner only while the front is near it: a CTA
// takes a tile from the queue, owns it as above - distances in shared memory,
// weights in registers, boundary values exchanged while it works - until it is
// idle and CTAs are short, writes its distances and takes the next.
//
// tstate: 0 never owned, 1 queued, 2 owned, 4 given back.  `pending` counts
// messages not dealt with: a helper raises it before it sends and lowers it by
// what its workers have dealt with, after it has sent what they published
// meanwhile, so it reaches 0 only at the fixpoint.  A message to a tile that no
// CTA owns queues the tile.  The owner stores its count and leaves state 2
// before it looks at the inbox for the last time, and a sender raises the inbox
// before it looks at the state, so no message is lost between the two.
//
// A CTA without a tile takes a place in the queue (head) and waits for it to be
// filled.  `avail` is the queued tiles less the CTAs that wait; owners of idle
// tiles give them up until kFreeCtas CTAs wait, so a tile that the front
// reaches is taken at once.  (Each takes its place by lowering avail, and puts
// it back where others were first; a compare-and-swap on head let through 0.7
// tiles per us.)  Where CTAs wait, a tile's first message queues its
// neighbours too, before the front reaches them: their weights are on chip when
// it does.  Each tile is taken about once, where the queue schedule visits it
// 4 to 5 times.
//
// Measured, whole search, queue schedule -> visiting owners: 600 x 600 x 12
// 750 -> 540 us (kFreeCtas 0: 760, 16: 570, 64: 540; without the early
// neighbours 560; one CTA per SM 610), 1000 x 1000 x 12 1.62 -> 0.95 ms, 400 x
// 400 x 5 with column vias 620 -> 380 us.
constexpr int kFreeCtas = 32;
template <int NZM, bool PRIV, bool CV>
__global__ void __launch_bounds__(RunTile<NZM, true>::NW + 32, 2)
    lattice_live_kernel(const __grid_constant__ OwnParams o) {
  constexpr bool ZS = true;
  constexpr int NW = RunTile<NZM, ZS>::NW, PS = kRunPS;
  const float INF_F = __int_as_float(0x7f800000);
  extern __shared__ __align__(128) float sd[];
  __shared__ RunShared S;
  __shared__ OwnShared Q;
  const LatParams &p = o.l;
  LatCtl *const ctl = p.ctl;
  const int tid = threadIdx.x;
  auto handover = [&] { asm volatile("bar.sync 2, %0;" ::"n"(NW + 32) : "memory"); };

  if (tid >= NW) {
    // ------------------------------------------------------------ helper
    const unsigned long long t_start = dev_globaltimer();
    const unsigned long long limit = p.budget_ns;
    const int lane = tid - NW;
    int box = -1;
    bool have = false;  // a place in the queue is taken: pos
    unsigned pos = 0, visits = 0;
    // tiles `q` of the lanes with `push`, already in state 1, into the queue
    auto enqueue = [&](bool push, int q) {
      const unsigned m = __ballot_sync(ORSP_FULL_MASK, push);
      if (!m) return;
      __threadfence();
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(&ctl->tail, (unsigned)__popc(m));
      base = __shfl_sync(ORSP_FULL_MASK, base, 0);
      if (lane == 0) atomicAdd(&ctl->avail, __popc(m));
      if (push) atomicExch(&p.qslot[(base + __popc(m & lanemask_lt())) % p.qcap], q);
    };
    for (;;) {
      // ---- the next tile
      if (!have) {
        if (lane == 0) {
          atomicSub(&ctl->avail, 1);
          pos = atomicAdd(&ctl->head, 1u);
        }
        pos = __shfl_sync(ORSP_FULL_MASK, pos, 0);
      }
      have = false;
      const unsigned *slot = (const unsigned *)&p.qslot[pos % p.qcap];
      const unsigned *look = lane == 0 ? slot : lane == 1 ? (const unsigned *)&ctl->pending : (const unsigned *)&ctl->err;
      int t = -1;
      for (unsigned spins = 0;; ++spins) {
        const unsigned v = lane < 3 ? ld_acquire_u32(look) : 0u;
        if (__shfl_sync(ORSP_FULL_MASK, v, 1) == 0u || __shfl_sync(ORSP_FULL_MASK, v, 2) != 0u) break;
        t = (int)__shfl_sync(ORSP_FULL_MASK, v, 0);
        if (t >= 0) break;
        if (lane == 0 && (spins & 31u) == 31u && dev_globaltimer() - t_start > limit)
          atomicCAS(&ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
      }
      unsigned got = 0;
      if (t >= 0) {
        const int bi = p.nbox == 1 ? 0 : __ldg(&p.tbox[t]);
        got = __ldcg(&o.got[t]);
        if (lane == 0) {
          atomicExch((int *)slot, -1);
          atomicExch(&p.tstate[t], 2);
          if (bi != box) Q.box = load_box(p, bi);
          Q.req = Q.ack = got;
          Q.stop = Q.rel = Q.idle = Q.out = Q.quit = 0;
        }
        box = bi;
        if (lane < 4) Q.pub[lane] = 0;
      }
      if (lane == 0) Q.tile = t;
      __syncwarp();
      handover();
      if (t < 0) break;
      ++visits;
      const int ntx = Q.box.ntx, nty = Q.box.nty, lt = t - Q.box.tile0, ty = lt / ntx, tx = lt - ty * ntx;
      const int nb = lane == 0 ? (tx > 0 ? t - 1 : -1)
                               : lane == 1 ? (tx < ntx - 1 ? t + 1 : -1)
                                           : lane == 2 ? (ty > 0 ? t - ntx : -1)
                                                       : lane == 3 ? (ty < nty - 1 ? t + ntx : -1) : -1;
      // messages to the neighbours on the sides in m
      auto send = [&](unsigned m) {
        if (lane == 0) atomicAdd(&ctl->pending, __popc(m));
        __threadfence();
        __syncwarp();
        bool push = false;
        if ((m >> lane) & 1u) {
          atomicAdd(&o.inbox[nb], 1u);
          __threadfence();
          const int st = atomicCAS(&p.tstate[nb], 0, 1);
          push = st == 0 || (st == 4 && atomicCAS(&p.tstate[nb], 4, 1) == 4);
        }
        enqueue(push, nb);
      };
      unsigned asked = got;
      bool reached = false, over = false;
      for (unsigned spins = 0;; ++spins) {
        const bool acked = asked != got && __shfl_sync(ORSP_FULL_MASK, Q.ack, 0) == asked;
        const bool out = __shfl_sync(ORSP_FULL_MASK, Q.out, 0) != 0;
        const bool rest = __shfl_sync(ORSP_FULL_MASK, Q.idle, 0) != 0;
        __syncwarp();  // what lane 0 saw, all lanes follow
        __threadfence_block();
        // everything published up to the answer is sent before the count is
        // dealt with
        const unsigned pm = __ballot_sync(ORSP_FULL_MASK, lane < 4 && atomicExch(&Q.pub[lane & 3], 0) != 0);
        if (pm) send(pm);
        if (acked) {
          if (lane == 0) {
            __threadfence();
            atomicSub(&ctl->pending, (int)(asked - got));
          }
          got = asked;
        }
        if (out) break;
        unsigned v = 0;
        if (lane == 0) v = ld_acquire_u32(&o.inbox[t]);
        if (lane == 1) v = ld_acquire_u32((const unsigned *)&ctl->pending);
        if (lane == 2) v = ld_acquire_u32((const unsigned *)&ctl->err);
        if (lane == 3) v = ld_acquire_u32((const unsigned *)&ctl->avail);
        const unsigned in = __shfl_sync(ORSP_FULL_MASK, v, 0);
        const bool failed = __shfl_sync(ORSP_FULL_MASK, v, 2) != 0u;
        over = failed || __shfl_sync(ORSP_FULL_MASK, v, 1) == 0u;
        const int waiting = (int)__shfl_sync(ORSP_FULL_MASK, v, 3);  // < 0: free CTAs
        if (failed && lane == 0) Q.quit = 1;
        if (over && lane == 0) Q.stop = 1;
        if (asked == got && in != got) {
          asked = in;
          if (lane == 0) Q.req = in;
          if (!reached && waiting < 0) enqueue(nb >= 0 && atomicCAS(&p.tstate[nb], 0, 1) == 0, nb);
          reached = true;
        }
        if (!have && waiting > -kFreeCtas && rest && asked == got && !pm) {
          if (lane == 0) {
            have = atomicSub(&ctl->avail, 1) > -kFreeCtas;
            if (have) pos = atomicAdd(&ctl->head, 1u);
            else atomicAdd(&ctl->avail, 1);
          }
          have = __shfl_sync(ORSP_FULL_MASK, (int)have, 0);
          pos = __shfl_sync(ORSP_FULL_MASK, pos, 0);
          if (have) {
            if (lane == 0) Q.rel = 1;
          }
        }
        if (lane == 0 && (spins & 31u) == 31u && dev_globaltimer() - t_start > limit)
          atomicCAS(&ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
      }
      handover();  // the tile's distances are in memory
      if (over) {
        if (lane == 0) Q.tile = -1;
        __syncwarp();
        handover();
        break;
      }
      // ---- give the tile back
      bool push = false;
      if (lane == 0) {
        __stcg(&o.got[t], got);
        __threadfence();
        atomicExch(&p.tstate[t], 4);
        __threadfence();
        push = ld_acquire_u32(&o.inbox[t]) != got && atomicCAS(&p.tstate[t], 4, 1) == 4;
      }
      enqueue(push, t);
    }
    if (lane == 0) atomicAdd(&ctl->visits, visits);
    return;
  }

  // -------------------------------------------------------------- workers
  RunTile<NZM, ZS> R;
  float2 *const wp = (float2 *)(sd + o.nzb * PS), *const wz = wp + o.nzb * PS;
  if (tid == 0) S.start();
  for (;;) {
    handover();
    const int t = Q.tile;
    if (t < 0) break;
    if (tid == 0) S.lap(-1);
    const LatBox B = Q.box;
    const RunGeom G = run_geom(p, B, t);
    const unsigned snap = Q.ack;
    if (tid < 32) S.clear();
    // the rows' values, what was published to the neighbours, the tile
    float *const ex = o.exch + (int64_t)t * 2 * o.nr + tid;
    const int step = (G.isv ? B.ntx : 1) * 2 * o.nr;
    float na = INF_F, nb = INF_F, pa = INF_F, pb = INF_F;
    if (G.run) {
      na = ld_relaxed_f32(ex);
      nb = ld_relaxed_f32(ex + o.nr);
      if (G.isv ? G.ty > 0 : G.tx > 0) pa = ld_relaxed_f32(ex - step + o.nr);
      if (G.isv ? G.ty < B.nty - 1 : G.tx < B.ntx - 1) pb = ld_relaxed_f32(ex + step);
    }
    const bool force = __ldcg(&p.stamp[t]) != 0;
    const int64_t dz = (!PRIV || B.dbase < 0) ? (int64_t)p.nx * p.ny : (int64_t)(B.x1 - B.x0 + 1) * (B.y1 - B.y0 + 1);
    const int64_t d0 = G.col ? dist_index<PRIV>(p, B, G.X0 + G.xx, G.Y0 + G.yy, B.z0) : 0;
    load_tile<NZM, true, ZS, true>(p, G, R, sd, wp, wz, d0, dz);  // (with a barrier)
    if (tid == 0) {
      S.lap(0);
      if (force) p.stamp[t] = 0;
    }
    float ha, hb;
    const unsigned cycles =
        own_cycles<NZM, CV, ZS>(o, B, G, R, S, Q, sd, wz, ex, na, nb, pa, pb, G.run && force, force, snap, ha, hb);
    if (tid == 0) S.lap(1);
    if (cycles) {
      if (G.col) {
        const float *const cd = sd + G.yy * kRunWS + G.xx;
#pragma unroll
        for (int z = 0; z < NZM; ++z)
          if (z < G.nzb) __stcg(&p.dist[d0 + z * dz], f_bits(cd[z * PS]));
      }
      __threadfence();
    }
    tile_sync<NW, true>();
    if (tid == 0) {
      S.lap(2);
      S.cycles += cycles;
      Q.out = 1;
    }
    handover();
  }
  if (tid == 0) S.flush(ctl);
}

// Tiles to revisit after a visit of tile t: the neighbours whose halo value
// improved (s_act[0..3] = left, right, down, up) and t itself if it did not
// converge (s_act[4]).  Returns the count written to nb[0..4].
__device__ __forceinline__ int revisit_list(const LatParams &p, int t, const int *s_act, int *nb) {
  const LatBox B = load_box(p, box_of_tile(p, t));
  const int lt = t - B.tile0;
  const int tx = lt % B.ntx, ty = lt / B.ntx;
  int k = 0;
  if (s_act[0] && tx > 0) nb[k++] = t - 1;
  if (s_act[1] && tx < B.ntx - 1) nb[k++] = t + 1;
  if (s_act[2] && ty > 0) nb[k++] = t - B.ntx;
  if (s_act[3] && ty < B.nty - 1) nb[k++] = t + B.ntx;
  if (s_act[4]) nb[k++] = t;
  return k;
}

template <int TX, int TY, bool PRIV>
__global__ void __launch_bounds__(TX * TY, 1) lattice_tile_kernel(LatParams p) {
  extern __shared__ float sd[];
  __shared__ LayerLists s_layers;
  __shared__ int s_flags[6];
  __shared__ int s_act[5];
  __shared__ int s_tile;
  LatCtl *ctl = p.ctl;
  const unsigned nblocks = gridDim.x;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  const unsigned long long t_start = dev_globaltimer();
  if (threadIdx.x == 0) s_layers.box = -1;
  __syncthreads();
  unsigned r = 0;
  for (;;) {
    if (ld_acquire_u32((const unsigned *)&ctl->err)) break;
    if (r >= p.max_rounds) {
      if (leader) atomicCAS(&ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
      break;
    }
    const unsigned n_in = ld_acquire_u32(&ctl->lcnt[r % 3]);
    if (n_in == 0) break;  // converged
    const int32_t *inl = (r & 1) ? p.list1 : p.list0;
    int32_t *outl = (r & 1) ? p.list0 : p.list1;
    for (;;) {
      if (threadIdx.x == 0) s_tile = (int)atomicAdd(&ctl->work[r % 3], 1u);
      __syncthreads();
      const int ti = s_tile;
      __syncthreads();
      if (ti >= (int)n_in) break;
      const int t = __ldcg(&inl[ti]);
      process_tile<TX, TY, PRIV>(p, t, sd, s_layers, s_flags, s_act);
      if (threadIdx.x == 0) {
        int nb[5];
        const int k = revisit_list(p, t, s_act, nb);
        for (int j = 0; j < k; ++j) {
          if (atomicMax(&p.stamp[nb[j]], r + 2u) < r + 2u) {
            const unsigned idx = atomicAdd(&ctl->lcnt[(r + 1) % 3], 1u);
            __stcg(&outl[idx], nb[j]);  // idx < ntiles: each tile is queued once per round
          }
        }
        atomicAdd(&ctl->visits, 1u);
      }
    }
    if (leader) {
      ctl->lcnt[(r + 2) % 3] = 0;
      ctl->work[(r + 2) % 3] = 0;
      if (dev_globaltimer() - t_start > p.budget_ns) atomicCAS(&ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
    }
    grid_barrier(&ctl->bar, nblocks, &ctl->err, p.wait_ns);
    ++r;
  }
  if (leader) ctl->rounds = r;
}


// ---------------------------------------------------------------------------
// Asynchronous schedule: no grid barrier.  Tiles wait in a ring queue; each
// CTA repeatedly takes the next tile, visits it and queues the tiles whose
// halo it improved.  A tile is in the queue at most once (state 1) and is
// visited by one CTA at a time (state 2); if its halo improves during a visit
// (state 3) the same CTA visits it again at once (or, with that switched
// off, queues it again).  Only the visiting CTA writes a tile's cells, so
// the copy in its shared memory stays exact between the two visits.  `pending` counts tiles in
// states 1-3; it is raised before a tile is queued and lowered only after the
// visiting CTA has queued everything it activated, so it reaches 0 only when
// no tile can change again - the fixpoint.
__device__ void queue_tile(const LatParams &p, int t) {
  const unsigned k = atomicAdd(&p.ctl->tail, 1u);
  atomicExch(&p.qslot[k % p.qcap], t);
}

// Returns false if the state machine could not be advanced (never expected;
// recorded as an internal error by the caller).
__device__ bool activate_tile(const LatParams &p, int t) {
  for (int tries = 0; tries < 1024; ++tries) {
    const int st = atomicCAS(&p.tstate[t], 0, 1);
    if (st == 0) {
      atomicAdd(&p.ctl->pending, 1);
      queue_tile(p, t);
      return true;
    }
    if (st == 1 || st == 3) return true;
    if (atomicCAS(&p.tstate[t], 2, 3) == 2) return true;  // visiting: mark dirty
  }
  return false;
}

// DEEP: the instantiation for tiles of more than 12 layers (the column load
// in 18-layer blocks); compiled separately so that each layer range gets its
// own register allocation.  MINB: CTAs per SM the registers are sized for
// (2 fits a 16 x 16 tile of up to 12 layers in 128 registers per thread).
//
// TMA: fresh visits stage the tile with tensor loads (TmaCtx); every box is
// the whole lattice (the tensor maps and the staging are sized for p.nz
// layers), distances in slices of N cells (LatBox.pad = slice).  tmw / tmd
// are unused otherwise.
//
// NZM > 0: run visits (visit_runs) of tiles of up to NZM layers.
template <int TX, int TY, bool PRIV, bool DEEP = false, int MINB = 1, bool TMA = false, bool CV = false, int NZM = 0,
          bool ZS = false>
__global__ void __launch_bounds__(NZM > 0 ? RunTile<NZM ? NZM : 1, ZS>::NW : TX *TY, MINB)
    lattice_async_kernel(LatParams p, const __grid_constant__ CUtensorMap tmw, const __grid_constant__ CUtensorMap tmd) {
  extern __shared__ __align__(128) float sd[];
  __shared__ LayerLists s_layers;
  __shared__ int s_flags[6];
  __shared__ int s_act[5];
  __shared__ int s_nb[4];
  __shared__ int s_tile;
  __shared__ __align__(8) unsigned long long s_mbar;
  LatCtl *ctl = p.ctl;
  const unsigned long long t_start = dev_globaltimer();
  TmaCtx tma{};
  if constexpr (TMA) {
    const int64_t off = ((int64_t)p.nz * tile_floats_per_layer(TX, TY) + 31) & ~(int64_t)31;
    tma.tw = &tmw;
    tma.td = &tmd;
    tma.mbar = smem_addr(&s_mbar);
    tma.phase = 0;
    tma.sw = sd + off;
    tma.sdd = (uint32_t *)(sd + off + (int64_t)p.nz * TY * TX * 4);
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tma.mbar) : "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmw) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmd) : "memory");
    }
  }
  __shared__ RunShared s_run;
  if (threadIdx.x == 0) s_layers.box = -1, s_run.start();
  __shared__ LatBox s_box;
  int box = -1;  // thread 0: the box in s_box
  RunTile<NZM ? NZM : 1, ZS> R;
  __syncthreads();
  unsigned visits = 0;
  unsigned long long sched_ns = 0;
  __shared__ int s_cont;
  if (threadIdx.x == 0) s_cont = -1;
  for (;;) {
    if (threadIdx.x == 0 && s_cont < 0) {
      const unsigned long long tq = dev_globaltimer();
      int t = -1;
      if (!ld_acquire_u32((const unsigned *)&ctl->err)) {
        const unsigned pos = atomicAdd(&ctl->head, 1u);
        int *slot = &p.qslot[pos % p.qcap];
        const unsigned long long t0 = dev_globaltimer();
        for (unsigned spins = 0;; ++spins) {
          const int v = (int)ld_acquire_u32((const unsigned *)slot);
          if (v >= 0) {
            atomicExch(slot, -1);
            t = v;
            break;
          }
          if (ld_acquire_u32((const unsigned *)&ctl->pending) == 0) break;  // fixpoint reached
          if (ld_acquire_u32((const unsigned *)&ctl->err)) break;
          if ((spins & 31u) == 31u) {
            const unsigned long long now = dev_globaltimer();
            if (now - t0 > p.wait_ns || now - t_start > p.budget_ns) {
              atomicCAS(&ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
              break;
            }
            __nanosleep(64);
          }
        }
      }
      if (t >= 0) {
        const int bi = NZM > 0 ? __ldg(&p.tbox[t]) : 0;
        atomicExch(&p.tstate[t], 2);
        if (NZM > 0 && bi != box) {
          s_box = load_box(p, bi);
          box = bi;
        }
        __threadfence();
      }
      s_tile = t;
      sched_ns += dev_globaltimer() - tq;
    }
    __syncthreads();
    const bool warm = s_cont >= 0;
    const int t = warm ? s_cont : s_tile;
    __syncthreads();
    if (t < 0) break;
    if constexpr (NZM > 0) visit_runs<NZM, PRIV, false, CV, ZS>(p, t, s_box, sd, R, s_run, s_act, s_nb, warm);
    else process_tile<TX, TY, PRIV, DEEP, TMA, CV>(p, t, sd, s_layers, s_flags, s_act, s_nb, warm, &tma);
    // neighbours are activated by threads 0..3 in parallel, after this
    // tile's distances are visible
    unsigned long long ta = 0;
    if (threadIdx.x == 0) ta = dev_globaltimer();
    if (threadIdx.x < 4) {
      __threadfence();
      const int nb = s_act[threadIdx.x] ? s_nb[threadIdx.x] : -1;
      if (nb >= 0 && !activate_tile(p, nb)) atomicCAS(&ctl->err, DEV_OK, DEV_ERR_INTERNAL);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // leave the visiting state: back to idle, or queued again when dirty
      // (halo changed meanwhile) or not converged
      s_cont = -1;
      if (s_act[4] || atomicCAS(&p.tstate[t], 2, 0) != 2) {
        if (p.selfcont) {
          // visit it again at once: the interior and weights are already in
          // shared memory, so only the halo is read again, and there is no
          // queue handoff.  Visiting again (state 2) is published before the
          // halo is read.
          atomicExch(&p.tstate[t], 2);
          __threadfence();
          s_cont = t;
        } else {
          atomicExch(&p.tstate[t], 1);
          queue_tile(p, t);
        }
      } else {
        atomicSub(&ctl->pending, 1);
      }
      ++visits;
      sched_ns += dev_globaltimer() - ta;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    atomicAdd(&ctl->visits, visits);
    atomicAdd(&ctl->ns[3], sched_ns);
    if (NZM > 0) s_run.flush(ctl);
  }
}

// Scheduler side of a finished visit of tile t with neighbour flags act, by
// one full warp: activate the neighbours whose halo improved (lanes 0..3) and
// leave the visiting state - idle, or queued again when dirty or not
// converged (lane 4).  Everything newly queued takes consecutive queue
// places; `pending` counts it (and drops this visit) before it is visible in
// the queue, so it reaches 0 only at the fixpoint.  Three dependent trips to
// L2 in all; one lane doing the same tile after tile took about 6 us, more
// than the visit it overlaps.
template <bool GOAL>
__device__ void finish_visit(const LatParams &p, int t, const LatBox &B, const int *act, int lane) {
  float lim = 0.0f;
  if (GOAL) {
    lim = __int_as_float(0x7f7fffff);
    if (B.gx >= 0)
      lim = fminf(lim, goal_limit(bits_f(__ldcg(&p.dist[dist_index<true>(p, B, B.gx, B.gy, B.gz)])), p.wmin));
  }
  auto side = [&](int i) { return GOAL ? __int_as_float(act[i]) <= lim : act[i] != 0; };
  __threadfence();
  const int lt = t - B.tile0, ty = lt / B.ntx, tx = lt - ty * B.ntx;
  int q = -1;
  if (lane == 0 && side(0) && tx > 0) q = t - 1;
  if (lane == 1 && side(1) && tx < B.ntx - 1) q = t + 1;
  if (lane == 2 && side(2) && ty > 0) q = t - B.ntx;
  if (lane == 3 && side(3) && ty < B.nty - 1) q = t + B.ntx;
  bool queue = false, bad = q >= 0;
  for (int tries = 0; bad && tries < 1024; ++tries) {
    const int st = atomicCAS(&p.tstate[q], 0, 1);
    queue = st == 0;
    bad = !(st == 0 || st == 1 || st == 3 || atomicCAS(&p.tstate[q], 2, 3) == 2);
  }
  if (lane == 4 && (act[4] || atomicCAS(&p.tstate[t], 2, 0) != 2)) {
    atomicExch(&p.tstate[t], 1);
    q = t;
    queue = true;
  }
  const unsigned m = __ballot_sync(ORSP_FULL_MASK, queue);
  const int n = __popc(m);
  unsigned base = 0;
  if (lane == 0) {
    if (n) base = atomicAdd(&p.ctl->tail, (unsigned)n);
    // (this visit is one of `pending`; the returned value is awaited before
    // the tiles are queued)
    if (n != 1 && atomicAdd(&p.ctl->pending, n - 1) < 1) bad = true;
  }
  base = __shfl_sync(ORSP_FULL_MASK, base, 0);
  if (queue) atomicExch(&p.qslot[(base + __popc(m & lanemask_lt())) % p.qcap], q);
  if (bad) atomicCAS(&p.ctl->err, DEV_OK, DEV_ERR_INTERNAL);
}

// Warp-specialised asynchronous schedule.  The block has NW = TX*TY worker
// threads that visit tiles and one scheduler warp whose lane 0 does all queue
// work, so that the chain of global atomics of a visit (pop, activation of the
// neighbours, the tile's own state transition) overlaps the workers' loads and
// sweeps instead of stalling them.
//
// Handoff protocol.  Handoff k hands tile cur_k (or -1: stop) to the workers
// through s_cur, at named barrier 2, which all NW + 32 threads pass exactly
// once per handoff (the scheduler warp passes it once per loop iteration, the
// workers once before each visit; both stop after the handoff that carries
// -1).  The workers visit cur_k with their own named barrier 1, write the
// visit's neighbour flags into s_act[k & 1] and set s_done = k.  The scheduler finishes visit k (activations, state
// transition) once s_done == k - in its wait loop for the next tile, or just
// after the next handoff - so it never waits for work that only its own
// finished tile would create.  The flags of visit k stay intact until visit
// k + 2 starts, and the scheduler reads them before handoff k + 2.
// Prefetch into L2, by one warp, of the rows a visit of tile t loads: per
// layer of the box, each tile row's in-edge weights (16 B per node) and
// distances, with the x-halo cells and the distance rows just above and
// below the tile where the box has them (the y-halo).  Every address
// prefetched lies inside the weight array or the box's distances.
template <int TX, int TY, bool PRIV>
__device__ __forceinline__ void prefetch_tile_l2(const LatParams &p, int t, const LatBox &SB, int lane) {
  const LatBox B = SB;
  const int lt = t - B.tile0;
  const int tx = lt % B.ntx, ty = lt / B.ntx;
  const int32_t X0 = B.x0 + tx * TX, Y0 = B.y0 + ty * TY;
  const int tw = min(TX, B.x1 - X0 + 1), th = min(TY, B.y1 - Y0 + 1);
  const int nzb = B.z1 - B.z0 + 1;
  const int64_t nxy = (int64_t)p.nx * p.ny;
  const int ya = Y0 > B.y0 ? -1 : 0, yb = Y0 + th - 1 < B.y1 ? th : th - 1;
  const int nrow = yb - ya + 1;
  for (int i = lane; i < nzb * nrow; i += 32) {
    const int zl = i / nrow, yy = ya + i % nrow;
    const int32_t z = B.z0 + zl, y = Y0 + yy;
    const uint32_t *d = &p.dist[dist_index<PRIV>(p, B, X0, y, z)];
    // the row, with its x-halo cells where the box has them
    asm volatile("prefetch.global.L2 [%0];" ::"l"(X0 > B.x0 ? d - 1 : d) : "memory");
    asm volatile("prefetch.global.L2 [%0];" ::"l"(X0 + tw - 1 < B.x1 ? d + tw : d + tw - 1) : "memory");
    if (yy >= 0 && yy < th) {
      const float4 *w = &p.w4[(int64_t)z * nxy + (int64_t)y * p.nx + X0];
      for (int c = 0; c < tw; c += 8) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + c) : "memory");
      asm volatile("prefetch.global.L2 [%0];" ::"l"(w + tw - 1) : "memory");
    }
  }
}

template <int NZM, bool PRIV, int MINB, bool ZS, bool GOAL = false>
__global__ void __launch_bounds__(RunTile<NZM, ZS>::NW + 32, MINB) lattice_spec_kernel(LatParams p) {
  constexpr int NW = RunTile<NZM, ZS>::NW;
  extern __shared__ float sd[];
  __shared__ int s_act[2][5];
  __shared__ volatile int s_cur;
  __shared__ volatile int s_done;
  __shared__ LatBox s_box[2];  // boxes of the handed-over tiles, by parity of the handoff
  LatCtl *ctl = p.ctl;
  __shared__ RunShared s_run;
  if (threadIdx.x == 0) s_run.start();
  if (threadIdx.x == NW) s_done = 0;
  __syncthreads();
  if (threadIdx.x < NW) {
    // ---------------------------------------------------------- workers
    RunTile<NZM, ZS> R;
      unsigned long long idle_ns = 0;
    for (int k = 1;; ++k) {
      unsigned long long tw = 0;
      if (threadIdx.x == 0) tw = dev_globaltimer();
      asm volatile("bar.sync 2, %0;" ::"r"(NW + 32) : "memory");
      if (threadIdx.x == 0) idle_ns += dev_globaltimer() - tw;
      const int t = s_cur;
      if (t < 0) break;
      visit_runs<NZM, PRIV, true, false, ZS, GOAL>(p, t, s_box[k & 1], sd, R, s_run, s_act[k & 1], nullptr, false);
      // the visit ended with barrier 1: every write of it is done, and
      // finish_visit's device fence makes them visible before it activates
      // any tile (the workers do not wait for that fence)
      if (threadIdx.x == 0) {
        __threadfence_block();
        s_done = k;
      }
    }
    if (threadIdx.x == 0) {
      atomicAdd(&ctl->ns[3], idle_ns);
      s_run.flush(ctl);
    }
    return;
  }
  // ------------------------------------------------------------ scheduler
  const int lane = threadIdx.x & 31;
  const unsigned long long t_start = dev_globaltimer();
  int cur = -1;          // tile of the last handoff
  int k = 0;             // index of the last handoff
  bool finished = true;  // visit k finished by the scheduler (or none yet)
  unsigned visits = 0;
  for (;;) {
    int next = -1;
    long long pos = -1;
    const unsigned long long t0 = dev_globaltimer();
    for (unsigned spins = 0;; ++spins) {
      // (one lane reads it: the warp takes the branch as one)
      if (!finished && __shfl_sync(0xffffffffu, s_done, 0) == k) {
        __syncwarp();  // what lane 0 saw, all lanes follow
        finish_visit<GOAL>(p, cur, s_box[k & 1], s_act[k & 1], lane);
        ++visits;
        finished = true;
      }
      int got = 0;  // 1: a tile, 2: stop
      if (lane == 0) {
        if (pos < 0) pos = (long long)atomicAdd(&ctl->head, 1u);
        int *slot = &p.qslot[(unsigned)pos % p.qcap];
        next = (int)ld_acquire_u32((const unsigned *)slot);
        if (next >= 0) {
          atomicExch(slot, -1);
          atomicExch(&p.tstate[next], 2);
          got = 1;
        } else if (ld_acquire_u32((const unsigned *)&ctl->err)) {
          got = 2;
        } else if (finished && ld_acquire_u32((const unsigned *)&ctl->pending) == 0) {
          got = 2;  // fixpoint reached
        } else if ((spins & 31u) == 31u) {
          const unsigned long long now = dev_globaltimer();
          if (now - t0 > p.wait_ns || now - t_start > p.budget_ns) {
            atomicCAS(&ctl->err, DEV_OK, DEV_ERR_TIMEOUT);
            got = 2;
          }
          __nanosleep(64);
        }
      }
      got = __shfl_sync(0xffffffffu, got, 0);
      if (got == 2) next = -1;
      if (got) break;
    }
    next = __shfl_sync(0xffffffffu, next, 0);
    if (lane == 0) {
      s_cur = next;
      __threadfence();  // the tile is marked as visited before its halo is read
    }
    // the workers are still on visit k: hand over the next tile's box and
    // bring its rows into L2
    if (next >= 0) {
      const int32_t *src = (const int32_t *)(p.boxes + __ldg(&p.tbox[next]));
      if (lane < (int)(sizeof(LatBox) / 4)) ((int32_t *)&s_box[(k + 1) & 1])[lane] = __ldg(src + lane);
      __syncwarp();
      if (p.prefetch) prefetch_tile_l2<16, 16, PRIV>(p, next, s_box[(k + 1) & 1], lane);
    }
    __syncwarp();
    asm volatile("bar.sync 2, %0;" ::"r"(NW + 32) : "memory");  // handoff k + 1
    // the workers reached this barrier only after finishing visit k
    if (!finished) {
      finish_visit<GOAL>(p, cur, s_box[k & 1], s_act[k & 1], lane);
      ++visits;
      finished = true;
    }
    if (next < 0) break;
    cur = next;
    ++k;
    finished = false;
  }
  if (lane == 0) atomicAdd(&ctl->visits, visits);
}

unsigned long long env_u64(const char *name, unsigned long long dflt) {
  const char *s = getenv(name);
  if (!s || !*s) return dflt;
  return strtoull(s, nullptr, 10);
}

// Workspace layout for ntiles tiles: 4 tile arrays (lists, stamps, states),
// the ring queue, then the control block.
struct WsLayout {
  size_t list_b, q_b, total;
  unsigned qcap;
};
WsLayout ws_layout(const orsp::Graph *g, int64_t ntiles) {
  WsLayout w;
  w.list_b = (((size_t)ntiles * 4) + 255) & ~(size_t)255;
  w.qcap = (unsigned)(ntiles + 4 * g->num_sms * 4 + 64);
  w.q_b = (((size_t)w.qcap * 4) + 255) & ~(size_t)255;
  w.total = 4 * w.list_b + w.q_b + 256;
  return w;
}

int grow_ws(orsp::Graph *g, size_t need) {
  if (g->lat_ws_bytes < need) {
    cudaFree(g->lat_ws);
    g->lat_ws = nullptr;
    g->lat_ws_bytes = 0;
    ORSP_CUDA(cudaMalloc(&g->lat_ws, need));
    g->lat_ws_bytes = need;
  }
  if (!g->lat_ctl_h) ORSP_CUDA(cudaMallocHost(&g->lat_ctl_h, sizeof(LatCtl)));
  return ORSP_OK;
}

// Column-via weights for the nodes of a box: box_h (host, 6 ints) or box_d
// (device), with the ROI / sink masks of a node-set ROI search.
int gather_col_box(orsp::Graph *g, const float *cost_d, const int32_t *box_h, const LatBox *box_d,
                   const int32_t *roi_map_d, const uint8_t *sink_d, cudaStream_t st) {
  LatBox bv{};
  int64_t count = (int64_t)g->N * g->nz;  // upper bound when the box is on the device
  if (box_h) {
    bv.x0 = box_h[0];
    bv.x1 = box_h[1];
    bv.y0 = box_h[2];
    bv.y1 = box_h[3];
    bv.z0 = box_h[4];
    bv.z1 = box_h[5];
    const int64_t d = box_h[5] - box_h[4] + 1;
    count = (int64_t)(box_h[1] - box_h[0] + 1) * (box_h[3] - box_h[2] + 1) * d * d;
  }
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, (int64_t)g->num_sms * 16));
  gather_col_kernel<<<blocks, 256, 0, st>>>(g->vcol_eid, cost_d, g->wcol, g->N, g->nx, g->ny, g->nz,
                                             (g->nz + 3) & ~3, box_d, bv, roi_map_d, sink_d);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library); nullptr when unavailable.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (!tried) {
    tried = true;
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)f;
    else
      (void)cudaGetLastError();
  }
  return fn;
}

// The two tensor maps of the TMA staging: weights as fp32 [nz][ny][nx][4]
// (box {4, TX, TY, nzb}) and distances as u32 [slices][nz][ny][nx] (box
// {TX + 8, TY + 2, nzb, 1}).  False (plain loads) when a stride or base is
// not 16-byte aligned or the encoder refuses.
bool encode_lattice_maps(const orsp::Graph *g, const LatParams &p, int TX, int TY, int nzb, int64_t slices,
                         CUtensorMap *tmw, CUtensorMap *tmd) {
  const int64_t nx = g->nx, ny = g->ny, nz = g->nz, N = (int64_t)g->N;
  if (nx % 4 != 0 || ((uintptr_t)p.dist & 15) != 0 || ((uintptr_t)p.w4 & 15) != 0) return false;
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint32_t es[4] = {1, 1, 1, 1};
  const cuuint64_t dw[4] = {4, (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
  const cuuint64_t sw[3] = {16, (cuuint64_t)(16 * nx), (cuuint64_t)(16 * nx * ny)};
  const cuuint32_t bw[4] = {4, (cuuint32_t)TX, (cuuint32_t)TY, (cuuint32_t)nzb};
  if (enc(tmw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)p.w4, dw, sw, bw, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  const cuuint64_t dd[4] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz, (cuuint64_t)slices};
  const cuuint64_t sdd[3] = {(cuuint64_t)(4 * nx), (cuuint64_t)(4 * nx * ny), (cuuint64_t)(4 * N)};
  const cuuint32_t bd[4] = {(cuuint32_t)(TX + 8), (cuuint32_t)(TY + 2), (cuuint32_t)nzb, 1};
  if (enc(tmd, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, (void *)p.dist, dd, sdd, bd, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  return true;
}

// Layer bound of the run visit for boxes of up to nzb layers, or 0 where it
// does not apply (more than 18 layers).
int run_visit_layers(int nzb) { return nzb <= 6 ? 6 : nzb <= 12 ? 12 : nzb <= 18 ? 18 : 0; }

// The asynchronous kernels with run visits: column vias (one CTA per SM), the
// warp-specialised schedule, or the plain one; with two CTAs per SM the via
// weights are in shared memory (RunTile ZS: the registers of two CTAs do not
// hold them; 16 sources on 1000 x 1000 x 12: 4.95 ms against 5.64 ms with the
// spills, 2 048 boxes of up to 16 layers: 10.5 against 16.9 ms).
template <int NZM, bool PRIV>
void *run_visit_kernel(bool cv, bool spec, bool two, bool goal) {
  if (PRIV && goal) return (void *)lattice_spec_kernel<NZM, true, 2, true, true>;
  if (cv) return (void *)lattice_async_kernel<16, 16, PRIV, false, 1, false, true, NZM>;
  if (spec)
    return two ? (void *)lattice_spec_kernel<NZM, PRIV, 2, true> : (void *)lattice_spec_kernel<NZM, PRIV, 1, false>;
  return two ? (void *)lattice_async_kernel<16, 16, PRIV, false, 2, false, false, NZM, true>
             : (void *)lattice_async_kernel<16, 16, PRIV, false, 1, false, false, NZM>;
}
template <bool PRIV>
void *run_visit_kernel(int nzm, bool cv, bool spec, bool two, bool goal) {
  return nzm == 6    ? run_visit_kernel<6, PRIV>(cv, spec, two, goal)
         : nzm == 12 ? run_visit_kernel<12, PRIV>(cv, spec, two, goal)
                     : run_visit_kernel<18, PRIV>(cv, spec, two, goal);
}

// Launches a persistent kernel of `want` CTAs per SM where they fit (ctas > 0:
// of that many CTAs), timed when profiling is on.
int launch_persistent(orsp::Graph *g, void *kfn, int threads, size_t smem, int want, int ctas, void **args,
                      cudaStream_t st) {
  // The shared-memory cap is a per-kernel attribute: it is raised to the
  // largest tile once per (kernel, device), never lowered, so a launch with a
  // smaller tile does not invalidate a cached larger one.  The occupancy is
  // cached per (kernel, block, shared memory, device).
  static orsp::LaunchCache caps, occupancies;
  int cap = 0, occ = 0;
  int rc = caps.get(kfn, 0, 0, g->device, &cap, [&](int *bytes) {
    // the opt-in maximum less the kernel's static shared memory
    cudaFuncAttributes fa{};
    ORSP_CUDA(cudaFuncGetAttributes(&fa, kfn));
    ORSP_CUDA(cudaDeviceGetAttribute(bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, g->device));
    *bytes -= (int)fa.sharedSizeBytes;
    ORSP_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, *bytes));
    return ORSP_OK;
  });
  if (rc) return rc;
  rc = occupancies.get(kfn, threads, smem, g->device, &occ, [&](int *blocks) {
    ORSP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, kfn, threads, smem));
    return ORSP_OK;
  });
  if (rc) return rc;
  if (occ < 1) {
    orsp::set_error("lattice search: kernel does not fit on an SM");
    return ORSP_ERR_ARG;
  }
  if (ctas <= 0) ctas = g->num_sms * std::max(1, std::min(occ, want));
  if (orsp::g_timer.on) ORSP_CUDA(cudaEventRecord(orsp::g_timer.a, st));
  // Cooperative launch in both schedules: every CTA is resident, so a CTA
  // waiting for a queue slot never blocks the CTA that will fill it.
  // (launched with the cooperative attribute rather than
  // cudaLaunchCooperativeKernel, so that a stream capture keeps the
  // co-residency guarantee in the graph's kernel node)
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3(ctas);
  lc.blockDim = dim3(threads);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  cudaLaunchAttribute coop[1];
  coop[0].id = cudaLaunchAttributeCooperative;
  coop[0].val.cooperative = 1;
  lc.attrs = coop;
  lc.numAttrs = 1;
  ORSP_CUDA(cudaLaunchKernelExC(&lc, kfn, args));
  if (orsp::g_timer.on) {
    ORSP_CUDA(cudaEventRecord(orsp::g_timer.b, st));
    orsp::g_timer.pending = true;
  }
  return ORSP_OK;
}

// Shape of a launch under the owner schedule.  False when it does not apply:
// more than 18 layers, more tiles than resident CTAs (one per SM, or two with
// the via weights in shared memory), more seeds than it lists.  (Several
// tiles per CTA, weights reloaded at each visit, took more visits than the
// queue makes: 776 against 602 us for 1 444 tiles of 600 x 600 x 12.)
int par_tile_bytes(int nzb) { return 256 * ((nzb + 1) / 2); }
struct OwnShape {
  int per_sm, nzb;
  size_t smem, ws;
};
bool own_shape(const orsp::Graph *g, int64_t ntiles, int nzb, int64_t nseeds, OwnShape *o) {
  if (!run_visit_layers(nzb) || nseeds > kOwnSeeds || ntiles < 1 || ntiles > 2 * (int64_t)g->num_sms) return false;
  o->per_sm = ntiles > g->num_sms ? 2 : 1;
  o->nzb = nzb;
  o->smem = (size_t)run_smem_floats(nzb, o->per_sm == 2) * sizeof(float);
  // exchange rows, seeds' tiles, inbox, sent and dealt-with counts, control
  // and parents
  o->ws = 512 + ((size_t)ntiles * (2 * 16 * nzb + 3) + kOwnSeeds + 2) * 4 + 256 + (size_t)ntiles * par_tile_bytes(nzb);
  return true;
}

int grow_own_ws(orsp::Graph *g, size_t need) {
  if (g->own_ws_bytes >= need) return ORSP_OK;
  cudaFree(g->own_ws);
  g->own_ws = nullptr;
  g->own_ws_bytes = 0;
  ORSP_CUDA(cudaMalloc(&g->own_ws, need));
  g->own_ws_bytes = need;
  return ORSP_OK;
}

template <int NZM, bool PRIV>
void *own_kernel(bool cv, bool two) {
  if (cv)
    return two ? (void *)lattice_own_kernel<NZM, PRIV, true, true, 2> : (void *)lattice_own_kernel<NZM, PRIV, true, false, 1>;
  return two ? (void *)lattice_own_kernel<NZM, PRIV, false, true, 2>
             : (void *)lattice_own_kernel<NZM, PRIV, false, false, 1>;
}
template <bool PRIV>
void *own_kernel(int nzm, bool cv, bool two) {
  return nzm == 6 ? own_kernel<6, PRIV>(cv, two) : nzm == 12 ? own_kernel<12, PRIV>(cv, two) : own_kernel<18, PRIV>(cv, two);
}

constexpr int64_t kLiveTiles = 16384;  // tiles of a launch under visiting owners (38 MB of rows at 18 layers)
size_t live_ws(int64_t ntiles, int nzb) { return ((size_t)ntiles * (2 * 16 * nzb + 2)) * 4 + 256; }

template <bool PRIV, bool CV>
void *live_kernel(int nzm) {
  return nzm == 6 ? (void *)lattice_live_kernel<6, PRIV, CV>
                  : nzm == 12 ? (void *)lattice_live_kernel<12, PRIV, CV> : (void *)lattice_live_kernel<18, PRIV, CV>;
}
template <bool PRIV>
void *live_kernel(int nzm, bool cv) {
  return cv ? live_kernel<PRIV, true>(nzm) : live_kernel<PRIV, false>(nzm);
}

void fill_axes(LatParams &p) {
  p.hmask = p.vmask = 0;
  for (int z = 0, h = 0, v = 0; z < p.nz && z < 64; ++z) {
    if (p.axis[z] == 1) p.hmask |= 1ull << z, p.hlist[h++] = (int8_t)z;
    else if (p.axis[z] == 2) p.vmask |= 1ull << z, p.vlist[v++] = (int8_t)z;
  }
}

// one: the box of a single search (else the device table p.boxes); gather: see
// OwnParams, with up to `blocks` blocks a box.
int launch_own(orsp::Graph *g, LatParams &p, int64_t ntiles, const OwnShape &sh, int32_t nseeds, const int32_t *seeds,
               const float *seed_cost, cudaStream_t st, orsp::LatOptions *opt, const LatBox *one = nullptr,
               int gather = 0, const float *cost = nullptr, int blocks = 0, int64_t par_tiles = 0) {
  int rc = grow_own_ws(g, sh.ws);
  if (rc) return rc;
  if (!g->lat_ctl_h) ORSP_CUDA(cudaMallocHost(&g->lat_ctl_h, sizeof(LatCtl)));
  fill_axes(p);
  OwnParams o{};
  char *b = (char *)g->own_ws;
  p.ctl = (LatCtl *)b;
  o.done = (int *)(b + 256);
  o.nr = 16 * sh.nzb;
  o.exch = (float *)(b + 512);
  o.inbox = (unsigned *)(o.exch + ntiles * 2 * o.nr);
  o.sent = o.inbox + ntiles;
  o.got = o.sent + ntiles + 1;
  o.seedt = (int32_t *)(o.got + ntiles + 1);
  // (par_tiles: tiles of the largest box whose parents are wanted, 0: none)
  o.par_bytes = par_tile_bytes(sh.nzb);
  if (par_tiles > 0 && par_tiles * o.par_bytes <= orsp::kParSmem) {
    o.par = (uint8_t *)(((uintptr_t)(o.seedt + kOwnSeeds) + 255) & ~(uintptr_t)255);
    opt->par_d = o.par;
    opt->par_tile_bytes = o.par_bytes;
    opt->par_smem = (int)(par_tiles * o.par_bytes);
  }
  if (opt) opt->err_d = &p.ctl->err, opt->ctl_d = p.ctl;
  p.wait_ns = env_u64("ORSP_WAIT_NS", 2000000000ull);
  p.budget_ns = env_u64("ORSP_BUDGET_NS", 20000000000ull);
  o.l = p;
  o.one = one != nullptr;
  if (one) o.box1 = *one;
  o.gather = gather;
  o.slot_eid = g->slot_eid;
  o.cost = cost;
  o.w = (float4 *)g->wslot;
  o.tcap = (int32_t)ntiles;
  o.nzb = sh.nzb;
  o.nseeds = nseeds;
  o.seeds = seeds;
  o.seed_cost = seed_cost;
  const int64_t rows = ntiles * 2 * o.nr / 4;
  const unsigned init_y = gather == 1 ? p.nbox : 1;
  const unsigned init_x = 1 + (unsigned)std::max<int64_t>({1, gather ? blocks : 0,
                                                           std::min<int64_t>((rows + 255) / 256, g->num_sms) / init_y});
  own_init_kernel<<<dim3(init_x, init_y), 256, 0, st>>>(o);
  ORSP_CUDA(cudaGetLastError());
  const int nzm = run_visit_layers(sh.nzb);
  const bool cv = p.wcol != nullptr, two = sh.per_sm == 2;
  void *kfn = opt && opt->private_dist ? own_kernel<true>(nzm, cv, two) : own_kernel<false>(nzm, cv, two);
  void *args[] = {&o};
  rc = launch_persistent(g, kfn, (nzm > 16 ? 288 : 256) + 32, sh.smem, sh.per_sm, (int)ntiles, args, st);
  if (rc) return rc;
  if (!opt || opt->copy_ctl)
    ORSP_CUDA(cudaMemcpyAsync(g->lat_ctl_h, p.ctl, sizeof(LatCtl), cudaMemcpyDeviceToHost, st));
  return ORSP_OK;
}

// Whether a launch takes the owner schedule (ORSP_LAT_OWN=0: none does): one
// that fits it, whose boxes are all searched.
bool use_own(const orsp::Graph *g, int64_t ntiles, int nzb, int64_t nseeds, const orsp::LatOptions *opt, OwnShape *sh) {
  if (env_u64("ORSP_LAT_OWN", 1) == 0 || env_u64("ORSP_LAT_ASYNC", 1) == 0 || env_u64("ORSP_LAT_TMA", 0) != 0)
    return false;
  if (env_u64("ORSP_LAT_SPEC", 0) != 0 || env_u64("ORSP_LAT_BLOCKS_PER_SM", 1) > 1) return false;
  if (opt && opt->active) return false;
  return own_shape(g, ntiles, nzb, nseeds, sh) && sh->per_sm <= (int)env_u64("ORSP_OWN_PER_SM", 2);
}

// Whether a launch takes visiting owners (ORSP_LAT_LIVE=0: none does).  `front`
// is the sum of the boxes' sides in tiles, about the tiles that wave fronts
// hold at a time; below one per resident CTA the owners are faster than the
// queue schedules (sources on 1000 x 1000 x 12, 126 tiles each: 2 sources 1.58
// against 2.15 ms, 4 2.86 against 2.57; on 400 x 400 x 6, 50 each: 6 sources
// 0.64 against 0.66 ms, 8 0.79 against 0.67; boxes of 320 x 320 x 4, 40 each: 8
// boxes 0.67 against 0.68 ms, 12 0.88 against 0.71).  Column vias, which have no
// warp-specialised schedule, gain up to twice that (16 sources on 300 x 300 x 8,
// 608 tiles: 1.30 against 1.42 ms).  Launches with activity flags search few of
// their boxes (repair rounds of 32 boxes on 600 x 600 x 18: grouped routing 76
// -> 70 ms).
bool use_live(const orsp::Graph *g, int64_t ntiles, int64_t front, int nzb, const orsp::LatOptions *opt) {
  if (env_u64("ORSP_LAT_LIVE", 1) == 0 || env_u64("ORSP_LAT_ASYNC", 1) == 0 || env_u64("ORSP_LAT_TMA", 0) != 0)
    return false;
  if (env_u64("ORSP_LAT_SPEC", 0) != 0 || env_u64("ORSP_LAT_BLOCKS_PER_SM", 1) > 1) return false;
  if (!run_visit_layers(nzb) || ntiles > kLiveTiles) return false;
  return (opt && opt->active) || front <= (g->cvia ? 4 : 2) * (int64_t)g->num_sms;
}

int launch_lattice(orsp::Graph *g, LatParams &p, int64_t ntiles, int64_t front, int nzb, int32_t nseeds, const int32_t *seeds,
                   const float *seed_cost, cudaStream_t st, orsp::LatOptions *opt) {
  constexpr int TX = 16, TY = 16;
  // (column vias always take the asynchronous schedule)
  const bool async = p.wcol != nullptr || env_u64("ORSP_LAT_ASYNC", 1) != 0;
  const WsLayout L = ws_layout(g, ntiles);
  const size_t list_b = L.list_b, q_b = L.q_b;
  const unsigned qcap = L.qcap;
  int rc0 = grow_ws(g, L.total);
  if (rc0) return rc0;
  char *b = (char *)g->lat_ws;
  p.list0 = (int32_t *)b;
  p.list1 = (int32_t *)(b + list_b);
  p.stamp = (unsigned *)(b + 2 * list_b);
  p.tstate = (int *)(b + 3 * list_b);
  p.qslot = async ? (int32_t *)(b + 4 * list_b) : nullptr;
  p.qcap = qcap;
  p.ctl = (LatCtl *)(b + 4 * list_b + q_b);
  if (opt) opt->err_d = &p.ctl->err, opt->ctl_d = p.ctl;
  p.tbox = async ? p.list0 : nullptr;
  const bool live = use_live(g, ntiles, front, nzb, opt);
  OwnParams o{};
  if (live) {
    rc0 = grow_own_ws(g, live_ws(ntiles, nzb));
    if (rc0) return rc0;
    o.nr = 16 * nzb;
    o.nzb = nzb;
    o.tcap = (int32_t)ntiles;
    o.exch = (float *)g->own_ws;
    o.inbox = (unsigned *)(o.exch + ntiles * 2 * o.nr);
    o.got = o.inbox + ntiles;
    p.inbox = o.inbox;
  }
  if (async) {
    const int64_t rows = live ? ntiles * 2 * o.nr / 4 : 0, n = std::max<int64_t>(std::max<int64_t>(ntiles, qcap), rows);
    lattice_init_kernel<<<(int)std::min<int64_t>((n + 255) / 256, (int64_t)g->num_sms * 8), 256, 0, st>>>(
        p, (int32_t)ntiles, o.got, (float4 *)o.exch, rows);
    ORSP_CUDA(cudaGetLastError());
  } else {
    ORSP_CUDA(cudaMemsetAsync(p.stamp, 0, list_b + (size_t)ntiles * 4, st));  // stamps and states
  }
  lattice_seed_kernel<TX, TY><<<1, 256, 0, st>>>(p, nseeds, seeds, seed_cost);
  ORSP_CUDA(cudaGetLastError());
  fill_axes(p);
  if (live) {
    p.wait_ns = env_u64("ORSP_WAIT_NS", 2000000000ull);
    p.budget_ns = env_u64("ORSP_BUDGET_NS", 20000000000ull);
    o.l = p;
    const int nzl = run_visit_layers(nzb);
    void *kfn = opt && opt->private_dist ? live_kernel<true>(nzl, p.wcol != nullptr)
                                         : live_kernel<false>(nzl, p.wcol != nullptr);
    void *args[] = {&o};
    // ORSP_LIVE_CTAS: that many CTAs instead of two per SM
    int rc = launch_persistent(g, kfn, (nzl > 16 ? 288 : 256) + 32, (size_t)run_smem_floats(nzb, true) * sizeof(float), 2,
                               (int)std::min<unsigned long long>(env_u64("ORSP_LIVE_CTAS", 0), g->num_sms), args, st);
    if (rc) return rc;
    if (!opt || opt->copy_ctl)
      ORSP_CUDA(cudaMemcpyAsync(g->lat_ctl_h, p.ctl, sizeof(LatCtl), cudaMemcpyDeviceToHost, st));
    return ORSP_OK;
  }
  // run visits up to 18 layers; deeper tiles take process_tile
  const int nzm = async ? run_visit_layers(nzb) : 0;
  // ORSP_LAT_BLOCKS_PER_SM: CTAs per SM
  const int want = (int)env_u64("ORSP_LAT_BLOCKS_PER_SM", (opt && opt->blocks_per_sm > 0) ? opt->blocks_per_sm : 1);
  const bool two = nzm && !p.wcol && want >= 2;
  size_t smem = nzm ? (size_t)run_smem_floats(nzb, two) * sizeof(float)
                    : (size_t)nzb * tile_floats_per_layer(TX, TY) * sizeof(float);
  if (smem > 227 * 1024) {
    orsp::set_error("lattice search: too many layers for the shared-memory tile");
    return ORSP_ERR_ARG;
  }
  const bool priv = opt && opt->private_dist;
  // ORSP_LAT_SPEC=1: the warp-specialised asynchronous schedule
  const bool spec = nzm && !p.wcol && env_u64("ORSP_LAT_SPEC", (opt && opt->spec) ? 1 : 0) != 0;
  // ORSP_LAT_TMA=1: tensor-load staging of fresh visits, for whole-lattice
  // boxes (opt->tma_slices: distance slices of N cells, box j in slice j)
  CUtensorMap tmw{}, tmd{};
  bool tma = false;
  if (async && !spec && !p.wcol && want < 2 && nzb <= 12 && nzb == g->nz && opt && opt->tma_slices > 0 &&
      env_u64("ORSP_LAT_TMA", 0) != 0)
    tma = encode_lattice_maps(g, p, TX, TY, nzb, opt->tma_slices, &tmw, &tmd);
  const bool runs = nzm != 0 && !tma;
  if (tma) {
    const size_t base = ((size_t)nzb * tile_floats_per_layer(TX, TY) + 31) & ~(size_t)31;
    smem = (base + (size_t)nzb * TY * TX * 4 + (size_t)nzb * (TY + 2) * (TX + 8)) * sizeof(float);
  }
  void *kfn;
  if (runs) {
    kfn = priv ? run_visit_kernel<true>(nzm, p.wcol != nullptr, spec, two, spec && two && p.wmin)
               : run_visit_kernel<false>(nzm, p.wcol != nullptr, spec, two, false);
  } else if (p.wcol) {
    kfn = priv ? (void *)lattice_async_kernel<16, 16, true, true, 1, false, true>
               : (void *)lattice_async_kernel<16, 16, false, true, 1, false, true>;
  } else if (tma) {
    kfn = priv ? (void *)lattice_async_kernel<16, 16, true, false, 1, true>
               : (void *)lattice_async_kernel<16, 16, false, false, 1, true>;
  } else if (async) {
    kfn = priv ? (void *)lattice_async_kernel<16, 16, true, true> : (void *)lattice_async_kernel<16, 16, false, true>;
  } else {
    kfn = priv ? (void *)lattice_tile_kernel<16, 16, true> : (void *)lattice_tile_kernel<16, 16, false>;
  }
  const int threads = (runs && nzm > 16 ? 288 : TX * TY) + (spec ? 32 : 0);
  p.max_rounds = (unsigned)std::min<unsigned long long>(64ull * (unsigned long long)ntiles + 4096ull, 1ull << 30);
  p.wait_ns = env_u64("ORSP_WAIT_NS", 2000000000ull);
  // ORSP_LAT_SELF=0: a tile to visit again goes back to the queue instead
  p.selfcont = (int)env_u64("ORSP_LAT_SELF", 1);
  // ORSP_LAT_PREFETCH=0: no L2 prefetch of the next tile by the scheduler warp
  p.prefetch = (int)env_u64("ORSP_LAT_PREFETCH", 1);
  p.budget_ns = env_u64("ORSP_BUDGET_NS", 20000000000ull);
  void *args[] = {&p, &tmw, &tmd};  // the tile and spec kernels take p only
  int rc = launch_persistent(g, kfn, threads, smem, want, 0, args, st);
  if (rc) return rc;
  if (!opt || opt->copy_ctl)
    ORSP_CUDA(cudaMemcpyAsync(g->lat_ctl_h, p.ctl, sizeof(LatCtl), cudaMemcpyDeviceToHost, st));
  return ORSP_OK;
}

}  // namespace

namespace orsp {

// Recognises the routing lattice: every planar edge a unit step along its
// layer's single routing axis, no parallel planar edges, and vias either all
// between adjacent layers without parallel edges (slots 2 and 3) or, as in
// the reference's Lattice3D (all-pairs blind/buried vias, duplicated via
// edges, unified_pathfinder.py:1136-1172, 1264-1276), between any two layers
// of a column with at most two parallel edges each (column vias, g->cvia).
int analyze_lattice(Graph *g, const int32_t *indptr_h, const int32_t *indices_h) {
  g->lattice_ok = false;
  g->cvia = false;
  g->lat_uniform = false;
  if (g->nx <= 0 || g->ny <= 0 || g->nz <= 0 || g->nz > 64) return ORSP_OK;
  const int32_t N = g->N, nx = g->nx, ny = g->ny;
  const int64_t nxy = (int64_t)nx * ny;
  std::vector<int8_t> axis(g->nz, -1);
  std::vector<int32_t> slot((size_t)4 * N, -1);
  bool adjacent_vias = true;  // every via spans one layer, no parallel vias
  // edges present: planar ones per layer, columns with a via per layer pair
  std::vector<int64_t> planar_n(g->nz, 0), via_n((size_t)g->nz * g->nz, 0);
  for (int32_t u = 0; u < N; ++u) {
    const int32_t zu = (int32_t)(u / nxy);
    const int32_t ru = (int32_t)(u - zu * nxy);
    const int32_t yu = ru / nx, xu = ru - yu * nx;
    for (int32_t k = indptr_h[u]; k < indptr_h[u + 1]; ++k) {
      const int32_t v = indices_h[k];
      const int32_t zv = (int32_t)(v / nxy);
      const int32_t rv = (int32_t)(v - zv * nxy);
      const int32_t yv = rv / nx, xv = rv - yv * nx;
      const int dz = zv - zu, dx = xv - xu, dy = yv - yu;
      int s = -1;
      if (dz == 0) {
        int ax;
        if (dy == 0 && (dx == 1 || dx == -1)) ax = 1;
        else if (dx == 0 && (dy == 1 || dy == -1)) ax = 2;
        else return ORSP_OK;  // not a unit planar step
        if (axis[zu] == -1) axis[zu] = (int8_t)ax;
        else if (axis[zu] != ax) return ORSP_OK;  // both axes on one layer
        s = (dx + dy > 0) ? 0 : 1;  // entering v from its lower / upper neighbour
      } else if (dx == 0 && dy == 0) {
        if (dz != 1 && dz != -1) {
          adjacent_vias = false;  // a via spanning layers: column vias
          continue;
        }
        s = dz > 0 ? 2 : 3;  // via from below / from above
      } else {
        return ORSP_OK;  // diagonal: not this lattice
      }
      int32_t &slotref = slot[(size_t)s * N + v];
      if (slotref != -1) {
        if (s < 2) return ORSP_OK;  // parallel planar edges
        adjacent_vias = false;      // parallel vias: column vias
        continue;
      }
      slotref = k;
      if (s < 2) ++planar_n[zu];
      else ++via_n[(size_t)zu * g->nz + zv];
    }
  }
  std::vector<int32_t> vcol;
  if (!adjacent_vias) {
    // column vias: every via in-edge of v by source layer, two parallel
    // edges at most (edge ids ascend with u and k, so k = 0 is the smaller)
    vcol.assign((size_t)2 * g->nz * N, -1);
    std::fill(via_n.begin(), via_n.end(), 0);
    for (int32_t u = 0; u < N; ++u) {
      const int32_t zu = (int32_t)(u / nxy);
      const int64_t cu = u - (int64_t)zu * nxy;
      for (int32_t k = indptr_h[u]; k < indptr_h[u + 1]; ++k) {
        const int32_t v = indices_h[k];
        const int32_t zv = (int32_t)(v / nxy);
        if (zv == zu || v - (int64_t)zv * nxy != cu) continue;  // planar (checked above)
        int32_t *e0 = &vcol[((size_t)0 * g->nz + zu) * N + v];
        int32_t *e1 = &vcol[((size_t)1 * g->nz + zu) * N + v];
        if (*e0 < 0) {
          *e0 = k;
          ++via_n[(size_t)zu * g->nz + zv];
        } else if (*e1 < 0) *e1 = k;
        else return ORSP_OK;  // three parallel vias
      }
    }
    for (int32_t v = 0; v < N; ++v) slot[(size_t)2 * N + v] = slot[(size_t)3 * N + v] = -1;
  }
  for (int z = 0; z < g->nz; ++z) g->layer_axis[z] = axis[z] < 0 ? 0 : axis[z];
  g->lat_uniform = true;
  for (int z = 0; z < g->nz; ++z) {
    const int64_t want = axis[z] == 1 ? 2 * (int64_t)(nx - 1) * ny : axis[z] == 2 ? 2 * (int64_t)nx * (ny - 1) : 0;
    if (planar_n[z] != want) g->lat_uniform = false;
    g->via_to[z] = 0;
    for (int t = 0; t < g->nz; ++t) {
      const int64_t n = via_n[(size_t)z * g->nz + t];
      if (n == nxy) g->via_to[z] |= 1ull << t;
      else if (n != 0) g->lat_uniform = false;
    }
  }
  ORSP_CUDA(cudaMalloc(&g->slot_eid, slot.size() * sizeof(int32_t)));
  ORSP_CUDA(cudaMemcpy(g->slot_eid, slot.data(), slot.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
  ORSP_CUDA(cudaMalloc(&g->wslot, slot.size() * sizeof(float)));
  ORSP_CUDA(cudaMalloc(&g->wmin, 2 * sizeof(int)));
  if (!adjacent_vias) {
    ORSP_CUDA(cudaMalloc(&g->vcol_eid, vcol.size() * sizeof(int32_t)));
    ORSP_CUDA(cudaMemcpy(g->vcol_eid, vcol.data(), vcol.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    // weights of every via in-edge of a node by source layer, nz rounded up
    // to 4 so that a node's row is whole float4s; layers without a via hold
    // +inf after each gather of the box, the rest is never read
    ORSP_CUDA(cudaMalloc(&g->wcol, (size_t)((g->nz + 3) & ~3) * N * sizeof(float)));
    g->cvia = true;
  }
  g->lattice_ok = true;
  return ORSP_OK;
}

void free_lattice(Graph *g) {
  cudaFree(g->slot_eid);
  cudaFree(g->wslot);
  cudaFree(g->vcol_eid);
  cudaFree(g->wcol);
  g->vcol_eid = nullptr;
  g->wcol = nullptr;
  g->cvia = false;
  cudaFree(g->lat_ws);
  cudaFree(g->own_ws);
  g->own_ws = nullptr;
  cudaFree(g->wmin);
  g->wmin = nullptr;
  cudaFree(g->lat_box_d);
  if (g->lat_ctl_h) cudaFreeHost(g->lat_ctl_h);
  g->lat_box_d = nullptr;
  g->slot_eid = nullptr;
  g->wslot = nullptr;
  g->lat_ws = nullptr;
  g->lat_ctl_h = nullptr;
}

// (tile_w 32: the depth up to which a batch plan's width-32 bucket takes the
// tile sweeps)
bool lattice_tile_fits(int nzb, int tile_w) {
  const int TX = tile_w ? tile_w : 16, TY = 16;
  const size_t smem = (size_t)nzb * tile_floats_per_layer(TX, TY) * sizeof(float);
  return smem <= 227 * 1024;
}

int reserve_lattice_ws(Graph *g, int64_t ntiles) {
  OwnShape sh;  // launches of up to that many tiles that take the owner schedule
  const int64_t most = 2 * (int64_t)g->num_sms;
  if (own_shape(g, std::min(std::max<int64_t>(ntiles, 1), most), std::min(g->nz, 18), 0, &sh)) {
    int rc = grow_own_ws(g, sh.ws);
    if (rc) return rc;
  }
  if (run_visit_layers(std::min(g->nz, 18))) {  // and visiting owners
    int rc = grow_own_ws(g, live_ws(std::min(ntiles, kLiveTiles), std::min(g->nz, 18)));
    if (rc) return rc;
  }
  return grow_ws(g, ws_layout(g, ntiles).total);
}

int64_t make_lat_boxes(const int32_t *boxes_h, int32_t nbox, LatBox *out) {
  constexpr int TX = 16, TY = 16;
  int64_t t0 = 0;
  for (int32_t i = 0; i < nbox; ++i) {
    const int32_t *b = boxes_h + 6 * (int64_t)i;
    LatBox &B = out[i];
    B.x0 = b[0];
    B.x1 = b[1];
    B.y0 = b[2];
    B.y1 = b[3];
    B.z0 = b[4];
    B.z1 = b[5];
    B.ntx = (b[1] - b[0] + TX) / TX;
    B.nty = (b[3] - b[2] + TY) / TY;
    B.tile0 = (int32_t)t0;
    B.pad = 0;
    B.dbase = -1;
    B.gx = B.gy = B.gz = -1;
    B.pad2 = 0;
    t0 += (int64_t)B.ntx * B.nty;
  }
  return t0;
}

int lat_ctl_words() { return (int)(sizeof(LatCtl) / 4); }

int gather_lattice(Graph *g, const float *cost_d, cudaStream_t st) {
  g->w4_cost = nullptr;  // the caller changes them from here on
  g->w4_gen = 0;
  const int64_t N = g->N;
  gather_kernel<false><<<(int)std::min<int64_t>((N + 255) / 256, 148 * 32), 256, 0, st>>>(g->slot_eid, cost_d,
                                                                                   (float4 *)g->wslot, N, nullptr);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

// Searches pairwise disjoint boxes in one launch.  Distances are reset to
// +inf everywhere (or, with opt->fill_box_only, inside the boxes only - the
// caller's backtrace must then test box membership); only the boxes' weights
// are gathered and only their tiles are visited.  Leaves the distances in
// `dist`; finish_lattice_search reports the status after the stream sync.
int run_lattice_boxes(Graph *g, const float *cost_d, int32_t nseeds, const int32_t *seeds_d,
                      const float *seed_cost_d, int32_t nbox, const int32_t *boxes_h, const LatBox *lboxes_d,
                      uint32_t *dist, cudaStream_t st, LatOptions *opt) {
  const int64_t N = g->N;
  constexpr int TX = 16, TY = 16;
  const bool priv = opt && opt->private_dist;
  int64_t vol_sum = 0;
  int64_t ntiles = 0, front = 0;
  int64_t tmax = 0;  // tiles of the largest box
  int nzb = 1;
  bool whole = false;
  for (int32_t i = 0; i < nbox; ++i) {
    const int32_t *b = boxes_h + 6 * (int64_t)i;
    const int64_t tx = (b[1] - b[0] + TX) / TX, ty = (b[3] - b[2] + TY) / TY;
    ntiles += tx * ty;
    tmax = std::max(tmax, tx * ty);
    front += tx + ty;
    nzb = std::max(nzb, b[5] - b[4] + 1);
    vol_sum += (int64_t)(b[1] - b[0] + 1) * (b[3] - b[2] + 1) * (b[5] - b[4] + 1);
    whole = whole || (b[0] == 0 && b[1] == g->nx - 1 && b[2] == 0 && b[3] == g->ny - 1 && b[4] == 0 &&
                      b[5] == g->nz - 1);
  }
  // overlapping boxes (own distances) may hold more cells than the lattice:
  // then one gather of every node is cheaper than one per box.  A whole
  // gather is skipped when the caller declared, for this search, the same
  // cost array and generation as the last whole gather's.
  const uint64_t decl = g->decl_cost == cost_d ? g->decl_gen : 0;
  g->decl_cost = nullptr;
  g->decl_gen = 0;
  // boxes with their own slices and device activity flags: only the active
  // boxes' weights are gathered and their slices reset (one launch each)
  const bool by_flag = priv && opt->active && !g->cvia && nbox <= 65535;
  int64_t vmax = 1;
  for (int32_t i = 0; i < nbox; ++i) {
    const int32_t *b = boxes_h + 6 * (int64_t)i;
    vmax = std::max<int64_t>(vmax, (int64_t)(b[1] - b[0] + 1) * (b[3] - b[2] + 1) * (b[5] - b[4] + 1));
  }
  const unsigned per_box = (unsigned)std::max<int64_t>(1, std::min<int64_t>((vmax + 255) / 256,
                                                                            148 * 32 / std::max(1, nbox)));
  OwnShape own;
  const bool owned = use_own(g, ntiles, nzb, nseeds, opt, &own);
  // a single box without a device table: the owners take it by value
  LatBox one{};
  if (!lboxes_d) {
    LatBox *hb = owned ? &one : (LatBox *)((char *)g->pinned + 1024);
    make_lat_boxes(boxes_h, 1, hb);
    if (!owned) {
      ORSP_CUDA(cudaMemcpyAsync(g->lat_box_d, hb, sizeof(LatBox), cudaMemcpyHostToDevice, st));
      lboxes_d = (const LatBox *)g->lat_box_d;
    }
  }
  // Boxes with targets, in the warp-specialised schedule only, whose scheduler
  // warp reads the target's distance off the workers' path (in the plain queue
  // schedule, with the boxes of routed nets, whose targets lie at their far
  // ends, 32 of them took 1.2 instead of 1.1 ms).  Not on column vias: a via
  // may cross several layers, and their weights are gathered apart.
  const bool goals = priv && opt->targets && !opt->gathered && opt->spec && !g->cvia && nbox <= 65535 && run_visit_layers(nzb) &&
                     !owned && !use_live(g, ntiles, front, nzb, opt);
  int *const wmin = goals ? g->wmin : nullptr;
  const bool cached = decl != 0 && g->w4_cost == cost_d && g->w4_gen == decl && (!goals || g->w4_min);
  const bool all = !by_flag && (whole || (priv && vol_sum >= N));
  if (goals && !(all && cached)) ORSP_CUDA(cudaMemsetAsync(g->wmin, 0x7f, 2 * sizeof(int), st));
  // the owners' preparation gathers along with the rest it does
  const int own_gather = !owned || g->cvia || (opt && opt->gathered) || (all && cached) ? 0 : all ? 2 : 1;
  if (opt && opt->gathered) {
    // by gather_lattice, kept since
  } else if (own_gather) {
    g->w4_cost = all ? cost_d : nullptr;
    g->w4_gen = all ? decl : 0;
    g->w4_min = false;
  } else if (by_flag) {
    g->w4_cost = nullptr;  // part of wslot is rewritten
    g->w4_gen = 0;
    (goals ? gather_boxes_kernel<true> : gather_boxes_kernel<false>)<<<dim3(per_box, (unsigned)nbox), 256, 0, st>>>(
        g->slot_eid, cost_d, (float4 *)g->wslot, N,
                                                                       g->nx, g->ny, lboxes_d, opt->active, wmin);
    ORSP_CUDA(cudaGetLastError());
  } else if (all) {
    if (!cached) {
      (goals ? gather_kernel<true> : gather_kernel<false>)<<<(int)std::min<int64_t>((N + 255) / 256, 148 * 32), 256, 0,
                                                            st>>>(g->slot_eid, cost_d, (float4 *)g->wslot, N, wmin);
      ORSP_CUDA(cudaGetLastError());
      if (g->cvia) {
        const int32_t full[6] = {0, g->nx - 1, 0, g->ny - 1, 0, g->nz - 1};
        int rc = gather_col_box(g, cost_d, full, nullptr, nullptr, nullptr, st);
        if (rc) return rc;
      }
      g->w4_cost = cost_d;
      g->w4_gen = decl;
      g->w4_min = goals;
    }
  } else {
    g->w4_cost = nullptr;  // part of wslot is rewritten
    g->w4_gen = 0;
    if (!g->cvia && (nbox > 1 || goals) && nbox <= 65535) {
      // one launch for all boxes, as many blocks per box as the largest needs
      // (within a grid of about 32 blocks per SM)
      (goals ? gather_boxes_kernel<true> : gather_boxes_kernel<false>)<<<dim3(per_box, (unsigned)nbox), 256, 0, st>>>(
          g->slot_eid, cost_d, (float4 *)g->wslot,
                                                                         N, g->nx, g->ny, lboxes_d, nullptr, wmin);
      ORSP_CUDA(cudaGetLastError());
    } else {
      for (int32_t i = 0; i < nbox; ++i) {
        const int32_t *b = boxes_h + 6 * (int64_t)i;
        const int32_t bw = b[1] - b[0] + 1, bh = b[3] - b[2] + 1;
        const int64_t count = (int64_t)bw * bh * (b[5] - b[4] + 1);
        gather_box_kernel<<<(int)std::min<int64_t>((count + 255) / 256, 148 * 32), 256, 0, st>>>(
            g->slot_eid, cost_d, (float4 *)g->wslot, N, g->nx, g->ny, b[0], bw, b[2], bh, b[4], count);
        ORSP_CUDA(cudaGetLastError());
        if (g->cvia) {
          int rc = gather_col_box(g, cost_d, b, nullptr, nullptr, nullptr, st);
          if (rc) return rc;
        }
      }
    }
  }
  if (owned && (priv || whole || (opt && opt->fill_box_only))) {
    // the owners write every cell of the boxes
  } else if (by_flag) {
    fill_slices_kernel<<<dim3(per_box, (unsigned)nbox), 256, 0, st>>>(dist, lboxes_d, opt->active, ORSP_INF_BITS);
    ORSP_CUDA(cudaGetLastError());
  } else if (priv) {
    fill_kernel<<<(int)std::min<int64_t>((opt->private_count + 255) / 256, 148 * 32), 256, 0, st>>>(
        dist, opt->private_count, ORSP_INF_BITS);
    ORSP_CUDA(cudaGetLastError());
  } else if (opt && opt->fill_box_only && !whole) {
    for (int32_t i = 0; i < nbox; ++i) {
      const int32_t *b = boxes_h + 6 * (int64_t)i;
      const int32_t bw = b[1] - b[0] + 1, bh = b[3] - b[2] + 1;
      const int64_t count = (int64_t)bw * bh * (b[5] - b[4] + 1);
      fill_box_kernel<<<(int)std::min<int64_t>((count + 255) / 256, 148 * 32), 256, 0, st>>>(
          dist, g->nx, g->ny, b[0], bw, b[2], bh, b[4], count, ORSP_INF_BITS);
      ORSP_CUDA(cudaGetLastError());
    }
  } else {
    fill_kernel<<<(int)std::min<int64_t>((N + 255) / 256, 148 * 32), 256, 0, st>>>(dist, N, ORSP_INF_BITS);
    ORSP_CUDA(cudaGetLastError());
  }
  LatParams p{};
  p.nx = g->nx;
  p.ny = g->ny;
  p.nz = g->nz;
  p.nbox = nbox;
  p.seed_per_box = priv ? 1 : 0;
  p.wmin = wmin;
  p.boxes = lboxes_d;
  p.w4 = (const float4 *)g->wslot;
  p.wcol = g->cvia ? g->wcol : nullptr;
  p.nzp = (g->nz + 3) & ~3;
  p.N = N;
  p.dist = dist;
  for (int z = 0; z < 64; ++z) p.axis[z] = z < g->nz ? g->layer_axis[z] : 0;
  if (owned)
    return launch_own(g, p, ntiles, own, nseeds, seeds_d, seed_cost_d, st, opt, lboxes_d ? nullptr : &one, own_gather,
                      cost_d, (int)std::min<int64_t>(((own_gather == 2 ? N : vmax) + 255) / 256, 148 * 32 / std::max(1, nbox)),
                      opt && opt->parents && !priv && !g->cvia ? tmax : 0);
  return launch_lattice(g, p, ntiles, front, nzb, nseeds, seeds_d, seed_cost_d, st, opt);
}

int run_lattice_search(Graph *g, const float *cost_d, int32_t nseeds, const int32_t *seeds_d,
                       const float *seed_cost_d, const int32_t *box, uint32_t *dist, cudaStream_t st,
                       LatOptions *opt) {
  const int32_t full[6] = {0, g->nx - 1, 0, g->ny - 1, 0, g->nz - 1};
  const int32_t *b = box ? box : full;
  if (!g->lat_box_d) ORSP_CUDA(cudaMalloc(&g->lat_box_d, sizeof(LatBox)));
  return run_lattice_boxes(g, cost_d, nseeds, seeds_d, seed_cost_d, 1, b, nullptr, dist, st, opt);
}

int run_lattice_roi(Graph *g, const float *cost_d, int32_t nseeds, const int32_t *seeds_d,
                    const float *seed_cost_d, const int32_t *roi_map_d, const int32_t *roi_nodes_d,
                    int64_t n_roi, const uint8_t *sink_d, uint32_t *dist, cudaStream_t st, LatOptions *opt) {
  const int64_t N = g->N;
  constexpr int TX = 16, TY = 16;
  if (!g->lat_box_d) ORSP_CUDA(cudaMalloc(&g->lat_box_d, sizeof(LatBox)));
  int rc = ensure_roi_arrays(g);
  if (rc) return rc;
  LatBox *box_d = (LatBox *)g->lat_box_d;
  const int gblocks = g->num_sms * 8;
  if (!roi_map_d && !roi_nodes_d) {
    const int32_t full[6] = {0, g->nx - 1, 0, g->ny - 1, 0, g->nz - 1};
    LatBox *hb = (LatBox *)((char *)g->pinned + 1024);
    make_lat_boxes(full, 1, hb);
    ORSP_CUDA(cudaMemcpyAsync(box_d, hb, sizeof(LatBox), cudaMemcpyHostToDevice, st));
  } else {
    // running maxima start at 0x80808080, below every coordinate
    ORSP_CUDA(cudaMemsetAsync(g->roi_bb, 0x80, 6 * sizeof(int), st));
    const int64_t n = roi_nodes_d ? n_roi : N;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, gblocks));
    roi_bbox_kernel<<<blocks, 256, 0, st>>>(roi_nodes_d, n, roi_map_d, g->nx, g->ny, N, g->roi_bb);
    ORSP_CUDA(cudaGetLastError());
    roi_box_finish_kernel<16, 16><<<1, 1, 0, st>>>(g->roi_bb, box_d);
    ORSP_CUDA(cudaGetLastError());
  }
  RoiGeom G{};
  G.nx = g->nx;
  G.ny = g->ny;
  G.nz = g->nz;
  for (int z = 0; z < 64; ++z) G.axis[z] = z < g->nz ? g->layer_axis[z] : 0;
  gather_roi_kernel<<<(int)std::min<int64_t>((N + 255) / 256, gblocks), 256, 0, st>>>(
      g->slot_eid, cost_d, (float4 *)g->wslot, N, G, box_d, roi_map_d, sink_d);
  ORSP_CUDA(cudaGetLastError());
  if (g->cvia) {
    rc = gather_col_box(g, cost_d, nullptr, box_d, roi_map_d, sink_d, st);
    if (rc) return rc;
  }
  g->w4_cost = nullptr;  // masked weights: not reusable by a whole search
  g->w4_gen = 0;
  g->decl_cost = nullptr;
  g->decl_gen = 0;
  fill_kernel<<<(int)std::min<int64_t>((N + 255) / 256, 148 * 32), 256, 0, st>>>(dist, N, ORSP_INF_BITS);
  ORSP_CUDA(cudaGetLastError());
  LatParams p{};
  p.nx = g->nx;
  p.ny = g->ny;
  p.nz = g->nz;
  p.nbox = 1;
  p.seed_per_box = 0;
  p.boxes = box_d;
  p.w4 = (const float4 *)g->wslot;
  p.wcol = g->cvia ? g->wcol : nullptr;
  p.nzp = (g->nz + 3) & ~3;
  p.N = N;
  p.dist = dist;
  p.roi_map = roi_map_d;
  for (int z = 0; z < 64; ++z) p.axis[z] = z < g->nz ? g->layer_axis[z] : 0;
  // the box is known on the device only: size the tile arrays for the lattice
  const int64_t tx = (g->nx - 1 + TX) / TX, ty = (g->ny - 1 + TY) / TY, ntiles = tx * ty;
  OwnShape own;
  if (use_own(g, ntiles, g->nz, nseeds, opt, &own))
    return launch_own(g, p, ntiles, own, nseeds, seeds_d, seed_cost_d, st, opt);
  return launch_lattice(g, p, ntiles, tx + ty, g->nz, nseeds, seeds_d, seed_cost_d, st, opt);
}

int finish_lattice_search(Graph *g, int32_t *rounds_h) {
  const LatCtl *c = (const LatCtl *)g->lat_ctl_h;
  if (rounds_h) *rounds_h = (int32_t)c->rounds;
  g_counters[0] = c->rounds;
  g_counters[1] = c->visits;
  g_counters[2] = (int64_t)c->cycles;
  for (int i = 0; i < 4; ++i) g_counters[4 + i] = (int64_t)c->ns[i];
  if (c->err) return dev_status_to_orsp(c->err);
  return ORSP_OK;
}

}  // namespace orsp

extern "C" int orsp_graph_cost_generation(orsp_graph *g, const float *cost_d, uint64_t generation) {
  if (!g || !cost_d) {
    orsp::set_error("cost_generation: NULL argument");
    return ORSP_ERR_ARG;
  }
  g->decl_cost = cost_d;
  g->decl_gen = generation;
  return ORSP_OK;
}

extern "C" int orsp_lattice_max_layers(int32_t tile_w, int32_t *out) {
  if (!out || (tile_w != 0 && tile_w != 16 && tile_w != 32)) {
    orsp::set_error("lattice_max_layers: tile width must be 0, 16 or 32");
    return ORSP_ERR_ARG;
  }
  int n = 0;
  while (n < 64 && orsp::lattice_tile_fits(n + 1, tile_w)) ++n;
  *out = n;
  return ORSP_OK;
}
