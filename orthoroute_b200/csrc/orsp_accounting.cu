// Edge accounting: cost update, present EMA, history update, overuse count,
// usage commit and path -> edge mapping.
//
// Every floating-point step is written with explicit round-to-nearest
// intrinsics (__fmul_rn / __fadd_rn / __fdiv_rn), so the compiler cannot fuse
// a multiply and an add into an FMA: each kernel reproduces, bit for bit, the
// float32 numpy expression of the reference function it replaces (numpy >= 2
// keeps Python-float scalars "weak", so every operand is rounded to float32).
#include <algorithm>
#include <cstring>
#include <initializer_list>

#include "accounting.cuh"

namespace {

using orsp::apply_usage;
using orsp::live_cost;

inline int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 32));
}

// The whole-array updates read and write each edge once, so they are bound by
// HBM; what keeps them there is bytes in flight.  Four edges per thread in
// 16-byte accesses (4-byte for the uint8 arrays) do that; arrays whose
// addresses are not 16-byte (4-byte) aligned, such as an offset view, and the
// last E mod 4 edges take the same step one edge at a time.  Measured on
// 25.2 M edges, before -> after: history 80 -> 69 us, present EMA 67 -> 47 us
// (6.4 TB/s), overuse 53 -> 42 us, present from usage 33 -> 28 us.
template <int V, typename T>
struct alignas(sizeof(T) * V) Vec {
  T v[V];
};
template <int V, typename T>
__device__ __forceinline__ Vec<V, T> ldv(const T *p, int64_t i) {
  return *reinterpret_cast<const Vec<V, T> *>(p + i * V);
}
// The same from an array that the launch does not write.
template <int V, typename T>
__device__ __forceinline__ Vec<V, T> ldr(const T *p, int64_t i) {
  Vec<V, T> x;
  if constexpr (sizeof(x) == 16) {
    const uint4 u = __ldg(reinterpret_cast<const uint4 *>(p + i * V));
    memcpy(&x, &u, 16);
  } else {
    x = ldv<V>(p, i);
  }
  return x;
}
template <int V, typename T>
__device__ __forceinline__ void stv(T *p, int64_t i, const Vec<V, T> &x) {
  *reinterpret_cast<Vec<V, T> *>(p + i * V) = x;
}

inline bool aligned_to(size_t a, std::initializer_list<const void *> ps) {
  for (const void *p : ps)
    if ((uintptr_t)p % a) return false;
  return true;
}

// EdgeAccountant.update_costs (UPF:973-1043) on one edge.
struct CostParams {
  const float *base, *ema, *cap, *hist;
  const uint8_t *layer, *kind;
  const float *lbias;
  float pres_fac, hist_w, via_mult, base_w;
  int jitter;
  float *out;
};

template <bool BIAS>
__device__ __forceinline__ float cost_of(const CostParams &p, int64_t e, float base, float ema, float cap, float hist,
                                         uint8_t layer, uint8_t kind) {
  // over = xp.maximum(0, present_ema - capacity)
  float over = __fsub_rn(ema, cap);
  over = over > 0.0f ? over : 0.0f;
  float adjusted = __fmul_rn(__fmul_rn(base, p.via_mult), p.base_w);
  float present_term;
  if (BIAS) {
    // per_edge_bias = where(edge_kind == 0, layer_bias[edge_layer], 1.0)
    const bool planar = kind == 0;
    const float peb = planar ? __ldg(&p.lbias[layer]) : 1.0f;
    adjusted = __fmul_rn(adjusted, peb);
    // inverted = where(peb != 0, 1/maximum(peb, 0.5), 1); where(kind==0, inv, 1)
    float inv = 1.0f;
    if (planar && peb != 0.0f) inv = __fdiv_rn(1.0f, peb > 0.5f ? peb : 0.5f);
    present_term = __fmul_rn(__fmul_rn(p.pres_fac, inv), over);
  } else {
    adjusted = __fmul_rn(adjusted, 1.0f);
    present_term = __fmul_rn(p.pres_fac, over);
  }
  float total = __fadd_rn(__fadd_rn(adjusted, present_term), __fmul_rn(p.hist_w, hist));
  if (p.jitter) total = __fadd_rn(total, orsp::index_jitter(e));
  return total;
}

// One whole-array update: op.at<V>(i) is its step on the V edges from V i.  The
// last E mod V edges go along in the same launch, one a thread (a launch of
// their own for each update made small arrays slower than single edges were).
template <int V, class Op>
__global__ void edges_kernel(int64_t E, Op op) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = E / V;
  for (int64_t i = t; i < n; i += stride) op.template at<V>(i);
  if (V > 1 && t < E % V) op.template at<1>(E - 1 - t);
}
template <class Op>
int over_edges(int64_t E, bool vec, const Op &op, cudaStream_t st) {
  if (vec) edges_kernel<4><<<grid_for((E + 3) / 4), 256, 0, st>>>(E, op);
  else edges_kernel<1><<<grid_for(E), 256, 0, st>>>(E, op);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

template <bool BIAS>
struct CostOp {
  CostParams p;
  template <int V>
  __device__ __forceinline__ void at(int64_t i) const {
    const Vec<V, float> b = ldr<V>(p.base, i), m = ldr<V>(p.ema, i), c = ldr<V>(p.cap, i), h = ldr<V>(p.hist, i);
    Vec<V, uint8_t> l{}, k{};
    if (BIAS) {
      l = ldv<V>(p.layer, i);
      k = ldv<V>(p.kind, i);
    }
    Vec<V, float> o;
#pragma unroll
    for (int j = 0; j < V; ++j) o.v[j] = cost_of<BIAS>(p, i * V + j, b.v[j], m.v[j], c.v[j], h.v[j], l.v[j], k.v[j]);
    stv<V>(p.out, i, o);
  }
};

// The live costs of all edges (edges == nullptr, V edges per step).
struct LiveCostOp {
  const float *base;
  const int32_t *usage;
  const float *cap, *hist;
  float pres_fac, hist_w, via_mult, base_w;
  int jitter;
  float *out;
  template <int V>
  __device__ __forceinline__ void at(int64_t i) const {
    const Vec<V, float> b = ldr<V>(base, i), c = ldr<V>(cap, i), h = ldr<V>(hist, i);
    const Vec<V, int32_t> u = ldr<V>(usage, i);
    Vec<V, float> o;
#pragma unroll
    for (int j = 0; j < V; ++j)
      o.v[j] = orsp::live_cost_of(i * V + j, b.v[j], u.v[j], c.v[j], h.v[j], pres_fac, hist_w, via_mult, base_w, jitter);
    stv<V>(out, i, o);
  }
};

__global__ void live_costs_kernel(int64_t n, const int32_t *__restrict__ edges, const float *__restrict__ base,
                                  const int32_t *__restrict__ usage, const float *__restrict__ cap,
                                  const float *__restrict__ hist, float pres_fac, float hist_w,
                                  float via_mult, float base_w, int jitter, float *__restrict__ out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int64_t e = edges[i];
    if (e < 0) continue;
    out[e] = live_cost(e, base, usage, cap, hist, pres_fac, hist_w, via_mult, base_w, jitter);
  }
}

// Same over the paths of a batch (path_len[k]-1 edges of row k).
__global__ void live_costs_paths_kernel(int32_t K, const int32_t *__restrict__ pe,
                                        const int32_t *__restrict__ plen, int32_t cap_row,
                                        const float *__restrict__ base, const int32_t *__restrict__ usage,
                                        const float *__restrict__ cap, const float *__restrict__ hist,
                                        float pres_fac, float hist_w, float via_mult, float base_w,
                                        int jitter, float *__restrict__ out) {
  for (int32_t k = blockIdx.x; k < K; k += gridDim.x) {
    const int32_t len = plen[k];
    if (len < 2) continue;
    const int32_t ne = min(len - 1, cap_row);
    for (int32_t i = threadIdx.x; i < ne; i += blockDim.x) {
      const int32_t e = pe[(int64_t)k * cap_row + i];
      if (e >= 0) out[e] = live_cost(e, base, usage, cap, hist, pres_fac, hist_w, via_mult, base_w, jitter);
    }
  }
}

// EdgeAccountant.update_present_ema (UPF:963-971).
struct EmaOp {
  const float *present;
  float *ema, beta, omb;
  template <int V>
  __device__ __forceinline__ void at(int64_t i) const {
    const Vec<V, float> p = ldr<V>(present, i);
    Vec<V, float> m = ldv<V>(ema, i);
#pragma unroll
    for (int j = 0; j < V; ++j) m.v[j] = __fadd_rn(__fmul_rn(beta, p.v[j]), __fmul_rn(omb, m.v[j]));
    stv<V>(ema, i, m);
  }
};

// EdgeAccountant.update_history (UPF:898-961).
struct HistoryOp {
  float *hist;
  const float *present, *cap, *base;
  float gain, cap_mult, decay;
  template <int V>
  __device__ __forceinline__ void at(int64_t i) const {
    const Vec<V, float> p = ldr<V>(present, i), c = ldr<V>(cap, i);
    Vec<V, float> h = ldv<V>(hist, i), b{};
    if (base) b = ldr<V>(base, i);
#pragma unroll
    for (int j = 0; j < V; ++j) {
      const float kept = __fmul_rn(h.v[j], decay);
      float over = __fsub_rn(p.v[j], c.v[j]);
      over = over > 0.0f ? over : 0.0f;
      float inc = __fmul_rn(gain, over);
      if (base) {
        const float hc = __fmul_rn(cap_mult, b.v[j]);
        inc = inc < hc ? inc : hc;  // xp.minimum (no NaNs here)
      }
      h.v[j] = __fadd_rn(kept, inc);
    }
    stv<V>(hist, i, h);
  }
};

// EdgeAccountant.compute_overuse (UPF:838-876), edge part.  acc: the float64
// sum, the count, and the number of blocks done; the last block writes the
// result (int() truncation of the sum).
struct OveruseAcc {
  double sum;
  unsigned long long cnt;
  unsigned done, pad;
};

template <int V>
__global__ void overuse_kernel(int64_t E, const float *__restrict__ present, const float *__restrict__ cap,
                               OveruseAcc *__restrict__ acc, int64_t *__restrict__ out2) {
  double s = 0.0;
  unsigned long long c = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto add = [&](float p, float k) {
    const float over = __fsub_rn(p, k);
    if (over > 0.0f) {
      s += (double)over;
      ++c;
    }
  };
  for (int64_t i = t; i < E / V; i += stride) {
    const Vec<V, float> p = ldv<V>(present, i), k = ldv<V>(cap, i);
#pragma unroll
    for (int j = 0; j < V; ++j) add(p.v[j], k.v[j]);
  }
  if (V > 1 && t < E % V) add(present[E - 1 - t], cap[E - 1 - t]);
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(ORSP_FULL_MASK, s, o);
    c += __shfl_xor_sync(ORSP_FULL_MASK, c, o);
  }
  __shared__ double ss[32];
  __shared__ unsigned long long sc[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { ss[w] = s; sc[w] = c; }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    s = lane < nw ? ss[lane] : 0.0;
    c = lane < nw ? sc[lane] : 0ull;
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(ORSP_FULL_MASK, s, o);
      c += __shfl_xor_sync(ORSP_FULL_MASK, c, o);
    }
    if (lane == 0) {
      if (c) {
        atomicAdd(&acc->sum, s);
        atomicAdd(&acc->cnt, c);
      }
      __threadfence();
      if (atomicAdd(&acc->done, 1u) == gridDim.x - 1) {
        __threadfence();
        out2[0] = (int64_t)__ldcg(&acc->sum);
        out2[1] = (int64_t)__ldcg(&acc->cnt);
      }
    }
  }
}

struct PresentOp {
  const int32_t *usage;
  float *present;
  template <int V>
  __device__ __forceinline__ void at(int64_t i) const {
    const Vec<V, int32_t> u = ldr<V>(usage, i);
    Vec<V, float> p;
#pragma unroll
    for (int j = 0; j < V; ++j) p.v[j] = (float)u.v[j];
    stv<V>(present, i, p);
  }
};

__global__ void commit_kernel(int64_t n, const int32_t *__restrict__ edges,
                              int32_t *__restrict__ usage, float *__restrict__ present,
                              int32_t sign) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int32_t e = edges[i];
    if (e >= 0) apply_usage(usage, present, e, sign);
  }
}

// Paths of a batched search: path_len[k] nodes give path_len[k]-1 edges.
__global__ void commit_batch_kernel(int32_t K, const int32_t *__restrict__ pe,
                                    const int32_t *__restrict__ plen, int32_t cap,
                                    int32_t *__restrict__ usage, float *__restrict__ present,
                                    int32_t sign) {
  for (int32_t k = blockIdx.x; k < K; k += gridDim.x) {
    const int32_t len = plen[k];
    if (len < 2) continue;
    const int32_t ne = min(len - 1, cap);
    for (int32_t i = threadIdx.x; i < ne; i += blockDim.x) {
      const int32_t e = pe[(int64_t)k * cap + i];
      if (e >= 0) apply_usage(usage, present, e, sign);
    }
  }
}

// _path_to_edges (UPF:5463-5476): first CSR edge u->v per consecutive pair;
// pairs without an edge produce -1 and are compacted away on the host side of
// the call (see orsp_path_to_edges).
__global__ void path_to_edges_kernel(const int32_t *__restrict__ indptr,
                                     const int32_t *__restrict__ indices,
                                     const int32_t *__restrict__ path, int32_t len,
                                     int32_t N, int32_t *__restrict__ out) {
  for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i + 1 < len;
       i += gridDim.x * blockDim.x) {
    const int32_t u = path[i], v = path[i + 1];
    int32_t found = -1;
    if (u >= 0 && u < N) {
      for (int32_t k = indptr[u]; k < indptr[u + 1]; ++k)
        if (indices[k] == v) { found = k; break; }
    }
    out[i] = found;
  }
}

__global__ void compact_edges_kernel(int32_t *edges, int32_t n, int32_t *count) {
  // single warp: stable in-place compaction of the >= 0 entries
  const int lane = threadIdx.x;
  int32_t w = 0;
  for (int32_t b = 0; b < n; b += 32) {
    const int32_t i = b + lane;
    const int32_t v = i < n ? edges[i] : -1;
    const unsigned m = __ballot_sync(ORSP_FULL_MASK, v >= 0);
    __syncwarp();
    if (v >= 0) edges[w + __popc(m & lanemask_lt())] = v;
    w += __popc(m);
    __syncwarp();
  }
  if (lane == 0) *count = w;
}

}  // namespace

using namespace orsp;

extern "C" int orsp_update_costs(int64_t E, const float *base, const float *ema,
                                 const float *cap, const float *hist,
                                 const uint8_t *layer, const uint8_t *kind,
                                 const float *lbias, float pres_fac, float hist_w,
                                 float via_mult, float base_w, int add_jitter,
                                 float *out, uintptr_t stream) {
  if (E < 0 || (E > 0 && (!base || !ema || !cap || !hist || !out))) {
    set_error("update_costs: NULL array");
    return ORSP_ERR_ARG;
  }
  const bool has_bias = lbias || layer || kind;
  if (has_bias && !(lbias && layer && kind)) {
    set_error("update_costs: layer_bias, edge_layer and edge_kind go together");
    return ORSP_ERR_ARG;
  }
  if (E == 0) return ORSP_OK;
  const CostParams p{base, ema, cap, hist, layer, kind, lbias, pres_fac, hist_w, via_mult, base_w, add_jitter, out};
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = aligned_to(16, {base, ema, cap, hist, out}) && aligned_to(4, {layer, kind});
  return lbias ? over_edges(E, vec, CostOp<true>{p}, st) : over_edges(E, vec, CostOp<false>{p}, st);
}

extern "C" int orsp_update_present_ema(int64_t E, const float *present, float *ema,
                                       float beta, float omb, uintptr_t stream) {
  if (E < 0 || (E > 0 && (!present || !ema))) { set_error("ema: NULL array"); return ORSP_ERR_ARG; }
  if (E == 0) return ORSP_OK;
  return over_edges(E, aligned_to(16, {present, ema}), EmaOp{present, ema, beta, omb}, (cudaStream_t)stream);
}

extern "C" int orsp_update_history(int64_t E, float *hist, const float *present,
                                   const float *cap, const float *base, float gain,
                                   float cap_mult, float decay, uintptr_t stream) {
  if (E < 0 || (E > 0 && (!hist || !present || !cap))) { set_error("history: NULL array"); return ORSP_ERR_ARG; }
  if (E == 0) return ORSP_OK;
  return over_edges(E, aligned_to(16, {hist, present, cap, base}),
                    HistoryOp{hist, present, cap, base, gain, cap_mult, decay}, (cudaStream_t)stream);
}

namespace orsp {
// Overuse into a caller-visible device int64[2]; the accumulators live in a
// small per-device buffer owned by this translation unit.
int overuse_into(int64_t E, const float *present, const float *cap, int64_t *out2,
                 void *acc, cudaStream_t st) {
  ORSP_CUDA(cudaMemsetAsync(acc, 0, sizeof(OveruseAcc), st));
  if (aligned_to(16, {present, cap}))
    overuse_kernel<4><<<grid_for((E + 3) / 4), 256, 0, st>>>(E, present, cap, (OveruseAcc *)acc, out2);
  else
    overuse_kernel<1><<<grid_for(E), 256, 0, st>>>(E, present, cap, (OveruseAcc *)acc, out2);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}
}  // namespace orsp

extern "C" int orsp_overuse(int64_t E, const float *present, const float *cap,
                            int64_t *out2_d, int64_t *out2_h, uintptr_t stream) {
  if (E < 0 || !out2_d || (E > 0 && (!present || !cap))) { set_error("overuse: NULL array"); return ORSP_ERR_ARG; }
  static thread_local void *acc = nullptr;
  static thread_local int acc_dev = -1;
  int dev = 0;
  ORSP_CUDA(cudaGetDevice(&dev));
  if (!acc || acc_dev != dev) {
    ORSP_CUDA(cudaMalloc(&acc, sizeof(OveruseAcc)));
    acc_dev = dev;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc = overuse_into(E, present, cap, out2_d, acc, st);
  if (rc) return rc;
  if (out2_h) {
    ORSP_CUDA(cudaMemcpyAsync(out2_h, out2_d, 16, cudaMemcpyDeviceToHost, st));
    ORSP_CUDA(cudaStreamSynchronize(st));
  }
  return ORSP_OK;
}

extern "C" int orsp_present_from_usage(int64_t E, const int32_t *usage, float *present,
                                       uintptr_t stream) {
  if (E < 0 || (E > 0 && (!usage || !present))) { set_error("present_from_usage: NULL array"); return ORSP_ERR_ARG; }
  if (E == 0) return ORSP_OK;
  return over_edges(E, aligned_to(16, {usage, present}), PresentOp{usage, present}, (cudaStream_t)stream);
}

extern "C" int orsp_commit_edges(int64_t n, const int32_t *edges, int32_t *usage,
                                 float *present, int32_t sign, uintptr_t stream) {
  if (n < 0 || (n > 0 && (!edges || !usage))) { set_error("commit: NULL array"); return ORSP_ERR_ARG; }
  if (sign != 1 && sign != -1) { set_error("commit: sign must be +1 or -1"); return ORSP_ERR_ARG; }
  if (n == 0) return ORSP_OK;
  commit_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(n, edges, usage, present, sign);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

extern "C" int orsp_commit_batch(int32_t K, const int32_t *pe, const int32_t *plen,
                                 int32_t cap, int32_t *usage, float *present,
                                 int32_t sign, uintptr_t stream) {
  if (K < 0 || cap <= 0 || (K > 0 && (!pe || !plen || !usage))) { set_error("commit_batch: bad args"); return ORSP_ERR_ARG; }
  if (sign != 1 && sign != -1) { set_error("commit_batch: sign must be +1 or -1"); return ORSP_ERR_ARG; }
  if (K == 0) return ORSP_OK;
  commit_batch_kernel<<<std::min(K, 148 * 8), 128, 0, (cudaStream_t)stream>>>(K, pe, plen, cap,
                                                                               usage, present, sign);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

extern "C" int orsp_path_to_edges(orsp_graph *g, const int32_t *path, int32_t len,
                                  int32_t *edges_out, int32_t *count_h, uintptr_t stream) {
  if (!g || len < 0 || (len > 1 && (!path || !edges_out)) || !count_h) {
    set_error("path_to_edges: bad args");
    return ORSP_ERR_ARG;
  }
  *count_h = 0;
  if (len < 2) return ORSP_OK;
  ORSP_CUDA(cudaSetDevice(g->device));
  cudaStream_t st = (cudaStream_t)stream;
  path_to_edges_kernel<<<(len + 255) / 256, 256, 0, st>>>(g->indptr, g->indices, path, len,
                                                          g->N, edges_out);
  ORSP_CUDA(cudaGetLastError());
  int32_t *cnt_d = nullptr;
  int rc = ensure_scratch(g, 64);
  if (rc) return rc;
  cnt_d = (int32_t *)g->scratch;
  compact_edges_kernel<<<1, 32, 0, st>>>(edges_out, len - 1, cnt_d);
  ORSP_CUDA(cudaGetLastError());
  ORSP_CUDA(cudaMemcpyAsync(g->pinned, cnt_d, 4, cudaMemcpyDeviceToHost, st));
  ORSP_CUDA(cudaStreamSynchronize(st));
  *count_h = *(int32_t *)g->pinned;
  return ORSP_OK;
}

extern "C" int orsp_update_costs_live(int64_t E, const int32_t *edges, int64_t n_edges,
                                      const float *base, const int32_t *usage, const float *cap,
                                      const float *hist, float pres_fac, float hist_w, float via_mult,
                                      float base_w, int add_jitter, float *out, uintptr_t stream) {
  if (E < 0 || !base || !usage || !cap || !hist || !out || (edges && n_edges < 0)) {
    set_error("update_costs_live: NULL array or bad size");
    return ORSP_ERR_ARG;
  }
  const int64_t n = edges ? n_edges : E;
  if (n == 0) return ORSP_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (!edges)
    return over_edges(E, aligned_to(16, {base, usage, cap, hist, out}),
                      LiveCostOp{base, usage, cap, hist, pres_fac, hist_w, via_mult, base_w, add_jitter, out}, st);
  live_costs_kernel<<<grid_for(n), 256, 0, st>>>(n, edges, base, usage, cap, hist, pres_fac, hist_w, via_mult, base_w,
                                                 add_jitter, out);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

extern "C" int orsp_update_costs_live_paths(int32_t K, const int32_t *pe, const int32_t *plen, int32_t cap_row,
                                            const float *base, const int32_t *usage, const float *cap,
                                            const float *hist, float pres_fac, float hist_w, float via_mult,
                                            float base_w, int add_jitter, float *out, uintptr_t stream) {
  if (K < 0 || cap_row <= 0 || (K > 0 && (!pe || !plen || !base || !usage || !cap || !hist || !out))) {
    set_error("update_costs_live_paths: bad args");
    return ORSP_ERR_ARG;
  }
  if (K == 0) return ORSP_OK;
  live_costs_paths_kernel<<<std::min(K, 148 * 8), 128, 0, (cudaStream_t)stream>>>(
      K, pe, plen, cap_row, base, usage, cap, hist, pres_fac, hist_w, via_mult, base_w, add_jitter, out);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}
