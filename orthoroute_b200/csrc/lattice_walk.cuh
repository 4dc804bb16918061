// Predecessor walk on the H/V routing lattice.
//
// On the lattice every node v = (x, y, z) has at most four in-neighbours, one
// per slot of the gathered in-edge weights w4[v] (orsp_lattice.cu), or, with
// column vias, its two planar in-neighbours and one via from every other
// layer of its column (LatWalkGeom::wcol):
//   slot 0: the lower neighbour along the layer's axis (x-1 on H layers, y-1 on
//           V layers), slot 1: the upper one (x+1 / y+1),
//   slot 2: the via from below (z-1), slot 3: the via from above (z+1).
// So the parent of v under the settle-order rule of the heap Dijkstra
// (SimpleDijkstra.find_path_roi, unified_pathfinder.py:1846-1887: the
// in-neighbour u with fl32(d[u] + w(u,v)) == d[v] and the smallest
// (d[u], rank u) below (d[v], rank v)) needs one float4 and four distances,
// all independent loads: one memory round trip per step of the walk, where a
// walk over the transposed CSR needs three dependent ones (row pointer, source
// list, distance).  Ranks are node ids by default (box searches rank nodes in
// id order, and a box's own distance slice is laid out in that order too);
// ROI searches pass the ROI index (global_to_roi) as the rank.
#pragma once

#include "common.cuh"

namespace orsp {

struct LatWalkGeom {
  int32_t nx, ny, nz;
  int8_t axis[64];  // 1: x moves (H layer), 2: y moves (V layer), 0: none
  // column vias (the reference's Lattice3D): a node's via in-edges come from
  // every layer of its column, with weights wcol[v * nzp + za] (slots 2 and 3
  // are empty); NULL on a lattice with adjacent vias only
  const float *wcol = nullptr;
  int32_t nzp = 0;
};

// Rank of a node for the tie-break: its id.
struct LatRankId {
  __device__ __forceinline__ int64_t operator()(int64_t v) const { return v; }
};

// Rank of a node inside a node-set ROI: its index in the ROI list
// (global_to_roi[v]); nodes outside the ROI never qualify as parents, since
// their distances stay +inf.
struct LatRankRoi {
  const int32_t *g2r;
  __device__ __forceinline__ int64_t operator()(int64_t v) const { return __ldg(&g2r[v]); }
};

// Coordinates of a node id (ids are below 2^31).
__device__ __forceinline__ void lat_xyz(const LatWalkGeom &G, int64_t v, int32_t &x, int32_t &y, int32_t &z) {
  const uint32_t plane = (uint32_t)G.nx * (uint32_t)G.ny;
  z = (int32_t)((uint32_t)v / plane);
  const uint32_t r = (uint32_t)v - (uint32_t)z * plane;
  y = (int32_t)(r / (uint32_t)G.nx);
  x = (int32_t)(r - (uint32_t)y * (uint32_t)G.nx);
}

// Neighbour of (x, y, z) through slot s, or false if it leaves box B.
__device__ __forceinline__ bool lat_slot_nbr(const LatWalkGeom &G, const LatBox &B, int s, int32_t x, int32_t y,
                                             int32_t z, int32_t &ux, int32_t &uy, int32_t &uz) {
  ux = x;
  uy = y;
  uz = z;
  if (s < 2) {
    const int d = s == 0 ? -1 : 1;
    if (G.axis[z] == 1) ux += d;
    else if (G.axis[z] == 2) uy += d;
    else return false;
  } else {
    uz += s == 2 ? -1 : 1;
  }
  return ux >= B.x0 && ux <= B.x1 && uy >= B.y0 && uy <= B.y1 && uz >= B.z0 && uz <= B.z1;
}

// One step of the walk at v = (x, y, z): its distance bits dv, and the slot of
// its parent with the parent's coordinates and distance bits, or -1 when v is
// not reached or no in-neighbour qualifies.  DIST(x, y, z) gives the distance
// bits of a node inside the box, RANK(node) its rank.  v's own distance, its
// weights and its neighbours' distances are independent loads, issued
// together; ranks are read only where two parents tie or a parent's distance
// equals v's (zero-cost edges).
template <class DIST, class RANK = LatRankId>
__device__ __forceinline__ int lat_parent(const LatWalkGeom &G, const LatBox &B, const float4 *__restrict__ w4,
                                          DIST dist, int32_t x, int32_t y, int32_t z, unsigned &dv,
                                          int32_t &px, int32_t &py, int32_t &pz, unsigned &pdu,
                                          RANK rank = RANK()) {
  constexpr int kCol = 8;  // layers of a column per memory round trip
  const int64_t v = ((int64_t)z * G.ny + y) * G.nx + x;
  const float4 wv = __ldcg(&w4[v]);
  const unsigned dc = dist(x, y, z);
  const float wk[4] = {wv.x, wv.y, wv.z, wv.w};
  unsigned du[4];
  int32_t ux[4], uy[4], uz[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const bool ok = lat_slot_nbr(G, B, s, x, y, z, ux[s], uy[s], uz[s]);
    du[s] = ok ? dist(ux[s], uy[s], uz[s]) : ORSP_INF_BITS;
  }
  dv = dc;
  unsigned bd = ORSP_INF_BITS;
  int bs = -1;
  bool tie = false;
  auto take = [&](int s, unsigned d, float w) {
    if (d == ORSP_INF_BITS || d > dc || f_bits(__fadd_rn(bits_f(d), w)) != dc) return;
    if (d < bd) {
      bd = d;
      bs = s;
      tie = false;
    } else if (d == bd) {
      tie = true;
    }
  };
  if (dc != ORSP_INF_BITS) {
#pragma unroll
    for (int s = 0; s < 4; ++s) take(s, du[s], wk[s]);
  }
  const float *wr = G.wcol ? G.wcol + v * G.nzp : nullptr;
  if (wr) {
    // column vias: a parent in any other layer of the box in this column
    // (slot 4 + its layer)
    for (int32_t zb = B.z0 & ~3; zb <= B.z1; zb += kCol) {
      float w[kCol];
      unsigned d[kCol];
#pragma unroll
      for (int i = 0; i < kCol; i += 4) {
        const float4 q = zb + i < G.nzp ? __ldg((const float4 *)(wr + zb + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
        w[i] = q.x;
        w[i + 1] = q.y;
        w[i + 2] = q.z;
        w[i + 3] = q.w;
      }
#pragma unroll
      for (int i = 0; i < kCol; ++i) {
        const int32_t za = zb + i;
        d[i] = za >= B.z0 && za <= B.z1 && za != z ? dist(x, y, za) : ORSP_INF_BITS;
      }
      if (dc != ORSP_INF_BITS) {
#pragma unroll
        for (int i = 0; i < kCol; ++i) take(4 + zb + i, d[i], w[i]);
      }
    }
  }
  if (bs >= 0 && (tie || bd == dc)) {
    // several parents at distance bd, or a zero-cost step: the smallest rank
    // decides, below v's own where the distances are equal
    const int64_t rv = bd == dc ? rank(v) : 0;
    unsigned br = 0;
    bs = -1;
    auto settle = [&](int s, int64_t u) {
      const int64_t ru = rank(u);
      if (bd == dc && !(ru < rv)) return;
      if (bs < 0 || (unsigned)ru < br) {
        br = (unsigned)ru;
        bs = s;
      }
    };
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (du[s] == bd && f_bits(__fadd_rn(bits_f(bd), wk[s])) == dc)
        settle(s, ((int64_t)uz[s] * G.ny + uy[s]) * G.nx + ux[s]);
    if (wr) {
      for (int32_t za = B.z0; za <= B.z1; ++za)
        if (za != z && dist(x, y, za) == bd && f_bits(__fadd_rn(bits_f(bd), __ldg(&wr[za]))) == dc)
          settle(4 + za, ((int64_t)za * G.ny + y) * G.nx + x);
    }
  }
  if (bs < 0) return -1;
  pdu = bd;
  px = x;
  py = y;
  pz = bs - 4;
#pragma unroll
  for (int s = 0; s < 4; ++s)
    if (bs == s) {
      px = ux[s];
      py = uy[s];
      pz = uz[s];
    }
  return bs;
}

// Cell i steps from (x, y, z) through slot s (the direction a straight run of
// parents takes when every parent sits in slot s of its child), or false if
// it leaves box B.
__device__ __forceinline__ bool lat_run_cell(const LatWalkGeom &G, const LatBox &B, int s, int i, int32_t x,
                                             int32_t y, int32_t z, int32_t &cx, int32_t &cy, int32_t &cz) {
  cx = x;
  cy = y;
  cz = z;
  if (s < 2) {
    const int d = s == 0 ? -i : i;
    if (G.axis[z] == 1) cx += d;
    else if (G.axis[z] == 2) cy += d;
    else if (i) return false;
  } else if (s < 4) {
    cz += s == 2 ? -i : i;
  } else if (i) {
    return false;  // a column via (slot 4 + layer) is a single step
  }
  return cx >= B.x0 && cx <= B.x1 && cy >= B.y0 && cy <= B.y1 && cz >= B.z0 && cz <= B.z1;
}

// The whole walk, by one full warp, from node (x, y, z) until STOP(node, bits)
// holds for the node just appended.  Nodes are appended to out[0..cap) from the
// target back to the start.  Returns the length, 0 (the target is not reached),
// -1 (more than cap nodes) or -2 (a node without a qualifying parent).
//
// Bound by the latency of its dependent rounds, so a round covers as many
// nodes of the path as one memory round trip can.  Paths on the lattice are
// straight runs joined by vias (a layer has one axis, so the direction changes
// only there).  Inside a run the lanes take the cells 0..31 steps ahead of the
// current node; at the first node and behind a via, where the run's direction
// is open, lane 0 takes the current node, 14 lanes the cells ahead in either
// direction and 3 the cells ahead through further vias.  Every lane computes
// its cell's parent with lat_parent; the parent of lane 0's cell says which
// group of lanes holds the path, and the run goes on as long as each cell's
// parent is the next cell of the group.  Each lane's parent is the one the
// sequential walk computes at that node (same distances, same rule), so the
// nodes are those of the one-step walk.
// Against rounds of two dependent loads that predicted only the last direction
// (two rounds per via): the walks of 32 nets on a 600 x 600 x 18 board took
// 36.7 us a launch, now 22.1; of a net on 100 x 100 x 4 12.8 us and 2.1 us for
// its commit, now 10.5 with it; four searches with paths on backplane boards
// 1.51 ms, now 1.01.
constexpr int kWalkSide = 14, kWalkVia = 3;  // 1 + 2 * kWalkSide + kWalkVia lanes

//
// PARENT(x, y, z, bits, px, py, pz): the slot of a cell's parent (-1: none), its
// distance bits and the parent's coordinates.
template <class PARENT, class STOP>
__device__ __forceinline__ int lat_walk_by(const LatWalkGeom &G, const LatBox &B, PARENT parent, STOP stop, int32_t x,
                                           int32_t y, int32_t z, int32_t *out, int32_t cap) {
  static_assert(1 + 2 * kWalkSide + kWalkVia == 32, "one warp");
  const int lane = threadIdx.x & 31;
  int len = 0;
  int s = z > B.z0 ? 2 : 3;  // slot of the last step (at first: a via, direction open)
  for (;;) {
    // this lane's cell: `step` steps from the current node through slot sl
    const bool run = s < 2;
    int sl = s, step = lane, n = 31;
    if (!run && lane) {
      const int g = lane <= kWalkSide ? 0 : lane <= 2 * kWalkSide ? 1 : 2;
      sl = g < 2 ? g : s;
      step = lane - g * kWalkSide;
      n = g < 2 ? kWalkSide : kWalkVia;
    }
    int32_t cx, cy, cz;
    const bool valid = lat_run_cell(G, B, sl, step, x, y, z, cx, cy, cz);
    const int64_t c = ((int64_t)cz * G.ny + cy) * G.nx + cx;
    int ps = -1;
    int32_t px = 0, py = 0, pz = 0;
    unsigned dc = ORSP_INF_BITS;
    if (valid) ps = parent(cx, cy, cz, dc, px, py, pz);
    if (len == 0 && __shfl_sync(ORSP_FULL_MASK, dc, 0) == ORSP_INF_BITS) return 0;
    const bool is_stop = dc != ORSP_INF_BITS && stop(c, dc);
    const unsigned m = __ballot_sync(ORSP_FULL_MASK, lane && !is_stop && ps == sl && step < n);
    // the group that lane 0's parent is in: lanes first+1 .. first+gn
    const int ps0 = __shfl_sync(ORSP_FULL_MASK, ps, 0);
    const bool stop0 = __shfl_sync(ORSP_FULL_MASK, (int)is_stop, 0);
    int first = 0, gn = 0;
    if (!stop0 && ps0 >= 0) {
      if (run) gn = ps0 == s ? 31 : 0;
      else if (ps0 < 2) first = ps0 * kWalkSide, gn = kWalkSide;
      else if (ps0 == s && s < 4) first = 2 * kWalkSide, gn = kWalkVia;
    }
    // its lanes up to the first whose parent is not the next one's cell (the
    // group's last lane never goes on)
    const int last = gn ? __ffs(~(m >> (first + 1))) : 0;
    const int end = last ? first + last : 0;
    if ((lane == 0 || (lane > first && lane <= end)) && len + step < cap) out[len + step] = (int32_t)c;
    len += last + 1;
    if (len > cap) return -1;
    if (__shfl_sync(ORSP_FULL_MASK, (int)is_stop, end)) return len;
    s = __shfl_sync(ORSP_FULL_MASK, ps, end);
    if (s < 0) return -2;
    x = __shfl_sync(ORSP_FULL_MASK, px, end);
    y = __shfl_sync(ORSP_FULL_MASK, py, end);
    z = __shfl_sync(ORSP_FULL_MASK, pz, end);
  }
}

// The walk on distances and weights.
template <class DIST, class STOP, class RANK = LatRankId>
__device__ __forceinline__ int lat_walk_warp(const LatWalkGeom &G, const LatBox &B, const float4 *__restrict__ w4,
                                             DIST dist, STOP stop, int32_t x, int32_t y, int32_t z, int32_t *out,
                                             int32_t cap, RANK rank = RANK()) {
  auto parent = [&](int32_t cx, int32_t cy, int32_t cz, unsigned &dc, int32_t &px, int32_t &py, int32_t &pz) {
    unsigned pdu;
    return lat_parent(G, B, w4, dist, cx, cy, cz, dc, px, py, pz, pdu, rank);
  };
  return lat_walk_by(G, B, parent, stop, x, y, z, out, cap);
}

// Parents recorded by the search (owner schedule, LatOptions::parents): four
// bits per cell - the slot, kParNone, or kParFar where the cell is not reached -
// two layers to a byte, 16 x 16 bytes per pair of layers, tile after tile.
constexpr unsigned kParNone = 4, kParFar = 7;
struct LatParents {
  const uint8_t *par;  // NULL: not recorded
  int32_t tile_bytes;
};

// Brings box B's parents to shared memory, by the whole block; every thread's
// copies have landed when it returns (a barrier is still due).
__device__ __forceinline__ void lat_load_parents(const LatParents &P, const LatBox &B, uint8_t *sm) {
  const int n = B.ntx * B.nty * P.tile_bytes;
  const uint8_t *src = P.par + (int64_t)B.tile0 * P.tile_bytes;
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(sm);
  for (int i = threadIdx.x * 16; i < n; i += blockDim.x * 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + i), "l"(src + i) : "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// The walk on recorded parents, from (x, y, z) to node src, whose distance is 0.
// A round takes a trip to shared memory instead of one to L2.
__device__ __forceinline__ int lat_walk_parents(const LatWalkGeom &G, const LatBox &B, const LatParents &P,
                                                const uint8_t *sm, int64_t src, int32_t x, int32_t y, int32_t z,
                                                int32_t *out, int32_t cap) {
  auto parent = [&](int32_t cx, int32_t cy, int32_t cz, unsigned &dc, int32_t &px, int32_t &py, int32_t &pz) {
    const int lx = cx - B.x0, ly = cy - B.y0, lz = cz - B.z0;
    const int at = ((ly >> 4) * B.ntx + (lx >> 4)) * P.tile_bytes + (lz >> 1) * 256 + (ly & 15) * 16 + (lx & 15);
    const unsigned s = (sm[at] >> ((lz & 1) * 4)) & 15u;
    dc = s == kParFar ? ORSP_INF_BITS : 0u;
    if (s >= kParNone) return -1;
    const bool h = G.axis[cz] == 1;
    const int d = s & 1 ? 1 : -1;
    px = cx + (s < 2 && h ? d : 0);
    py = cy + (s < 2 && !h ? d : 0);
    pz = cz + (s < 2 ? 0 : d);
    return (int)s;
  };
  auto at_src = [src](int64_t v, unsigned) { return v == src; };
  return lat_walk_by(G, B, parent, at_src, x, y, z, out, cap);
}

// Whether the lattice edge u -> v is a via: a planar step changes the id by 1
// or nx, a via by a multiple of a plane (the two coincide only where the layer
// has no planar step of that size).
__device__ __forceinline__ bool lat_is_via(const LatWalkGeom &G, int32_t u, int32_t v) {
  return abs(v - u) >= G.nx * G.ny;
}

// Slot of the in-edge u -> v between lattice neighbours u and v (node ids).
__device__ __forceinline__ int lat_edge_slot(const LatWalkGeom &G, int32_t u, int32_t v) {
  return (lat_is_via(G, u, v) ? 2 : 0) + (u < v ? 0 : 1);
}

// Reverses a walk's nodes (target first) in place, by the whole block.
__device__ __forceinline__ void lat_reverse(int32_t *nodes, int len) {
  for (int i = threadIdx.x; i < len / 2; i += blockDim.x) {
    const int32_t a = nodes[i], b = nodes[len - 1 - i];
    nodes[i] = b;
    nodes[len - 1 - i] = a;
  }
}

// CSR edge of step u -> v: the in-edge of v in the slot that u occupies, or the
// first edge from u's layer where the vias go between any two layers (vcol_eid,
// [2][nz][N] by source layer; the lattice has no other parallel edges).
__device__ __forceinline__ int32_t lat_step_edge(const LatWalkGeom &G, const int32_t *__restrict__ slot_eid,
                                                 const int32_t *__restrict__ vcol_eid, int64_t N, int32_t u,
                                                 int32_t v) {
  if (vcol_eid && lat_is_via(G, u, v)) return __ldg(&vcol_eid[(int64_t)(u / (G.nx * G.ny)) * N + v]);
  return __ldg(&slot_eid[(int64_t)lat_edge_slot(G, u, v) * N + v]);
}

constexpr int kWalkBlock = 128;  // warp 0 walks, the block reverses the path and maps its edges
constexpr int kParBlock = 512;   // the same with recorded parents, which the block loads
constexpr int kParSmem = 200 * 1024;  // parents of a box at most

}  // namespace orsp
