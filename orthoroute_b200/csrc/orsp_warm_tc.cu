// The warm-start network's 3x3x3 convolution on the 5th-generation tensor
// cores: tcgen05.mma (kind::f16, bf16 operands, fp32 accumulator in TMEM).
//
// Implicit GEMM, as conv3d_kernel in orsp_warm.cu: M = 128 voxels along x of
// one (z, y) row, N = Cout, K = 27 taps x Cin.  Each CTA is persistent:
//   - it stages every tap's weights once, B[n][k] = Wt[tap][k][n], in shared
//     memory in the K-major canonical UMMA layout without swizzle (core
//     matrices of 8 rows x 16 bytes, rows contiguous; the two 8-element halves
//     of a 16-wide K slice 128 bytes apart, 8-row groups 256 bytes apart);
//   - per tile, nine stages (dz, dy): 256 threads copy one input row once
//     into a stage buffer (cp.async, zero outside the grid; the optional ReLU
//     mask through registers), whose 16-byte rows serve the three (dx) taps
//     A[m][k] = X[z+dz][y+dy][x0+m+dx][k] as descriptors one row apart, and
//     one thread issues the 3 x Cin/16 MMAs (K = 16 each) into the TMEM
//     accumulator and commits them to the buffer's mbarrier, while the copies
//     of the next stages are in flight (a ring of up to six buffers);
//   - the epilogue reads the accumulator with tcgen05.ld (warps w and w + 4
//     share TMEM lanes 32 (w % 4) .., i.e. those voxels, and split the output
//     channels), adds the bias, applies the ReLU and stores bf16 or fp32.
// The weight gradient (wgrad_tc_kernel) is a second tcgen05 GEMM.  Layers of 16
// and 32 channels take the plane kernels (TMA loads) at the end of the file.
// Every mbarrier wait is bounded by the global timer; on expiry the kernel
// records an error, waits once more (bounded) for what is in flight, frees its
// TMEM and returns.  Single-GPU code: no multicast.
#include <cstdlib>
#include <algorithm>
#include <climits>
#include <cstdint>

#include <mutex>
#include <type_traits>

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "orsp_warm.h"

namespace {

constexpr int TC_M = 128;        // voxels per tile: the MMA's M and the accumulator's TMEM lanes
constexpr int TC_THREADS = 128;  // four warps, one per 32-lane quarter of TMEM
constexpr unsigned long long TC_WAIT_NS = 2000000000ull;

// Bound of one wait of a launch (ORSP_WAIT_NS).  What a launch still waits for
// when it has given up, its copies and MMAs in flight, keeps TC_WAIT_NS.
inline unsigned long long tc_wait_ns() {
  const char *s = getenv("ORSP_WAIT_NS");
  return s && *s ? strtoull(s, nullptr, 10) : TC_WAIT_NS;
}

__device__ int g_tc_err = 0;     // set by a kernel whose wait expired (orsp_warm_tc_status)

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor of a K-major operand without swizzle:
// start address, leading byte offset (between the K halves), stride byte
// offset (between 8-row groups), all in 16-byte units; version 1 (sm_100).
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}

// Instruction descriptor: fp32 accumulator, bf16 A and B, both K-major,
// N >> 3 and M >> 4.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}"
      :
      : "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

// One lane of a converged warp.  The MMA warps run their loops with all lanes
// and let one issue: descriptors and counters are then warp-uniform values,
// which the MMA takes from uniform registers as they are (from one lane's
// branch each went through a conversion, and issuing took 51 clocks per MMA).
__device__ __forceinline__ bool elect_lane() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Waits for the phase with the given parity to complete, at most TC_WAIT_NS.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  const unsigned long long t0 = dev_globaltimer();
  for (;;) {
    if (mbar_try(bar, parity)) return true;
    if (dev_globaltimer() - t0 > TC_WAIT_NS) return false;
  }
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared memory of the convolution: all weights (27 taps x Cin/16 K slices
// x Cout rows of 32 bytes), NS stage buffers, NS mbarriers and the TMEM
// address slot.  A stage buffer holds one input row of TC_M + 2 voxels as
// Cin / 8 planes (8 channels each) of 16-byte rows, CV_PLANE bytes apart:
// row r of plane cg at cg * CV_PLANE + r * 16.
constexpr int CV_PLANE = (TC_M + 2) * 16;
__host__ __device__ constexpr size_t cv_weight_bytes(int Cin, int Cout) {
  return static_cast<size_t>(27) * (Cin / 16) * Cout * 32;
}
__host__ __device__ constexpr size_t cv_stage_bytes(int Cin) {
  return (static_cast<size_t>(Cin / 8) * CV_PLANE + 127) & ~static_cast<size_t>(127);
}
__host__ __device__ constexpr size_t cv_smem_bytes(int Cin, int Cout, int ns) {
  return cv_weight_bytes(Cin, Cout) + ns * cv_stage_bytes(Cin) + 8 * ns + 64;
}
// Stage buffers that fit beside the weights in 200 KB (at most 6; 0 when
// fewer than 3 fit).
inline int cv_stages(int Cin, int Cout) {
  const size_t budget = 200 * 1024;
  if (cv_smem_bytes(Cin, Cout, 3) > budget) return 0;
  int ns = 3;
  while (ns < 6 && cv_smem_bytes(Cin, Cout, ns + 1) <= budget) ++ns;
  return ns;
}

// 16-byte global -> shared copy that fills zeros when `bytes` is 0.
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Waits until at most n (0..4) of this thread's copy groups are pending.
__device__ __forceinline__ void cp_async_wait(int n) {
  if (n <= 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
  else if (n == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
  else if (n == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
  else if (n == 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
  else asm volatile("cp.async.wait_group 4;" ::: "memory");
}

constexpr int CV_THREADS = 256;  // eight warps gather; warps w and w + 4 share TMEM lanes 32 (w % 4)..

// Pipelined implicit GEMM.  A stage is one input row (plane z + dz, row
// y + dy) of a tile: the 130 voxels x0 - 1 .. x0 + 128 are copied once, 16
// bytes at a time with cp.async (zero fill outside the grid), into the
// stage's channel planes.  The A operand of tap dx is that buffer itself: in
// the K-major layout without swizzle, a stride of 128 bytes between 8-row
// core-matrix groups puts row m at 16 m bytes, so the descriptor of tap dx
// starts (dx + 1) rows in (row m of tap dx = voxel x0 + m + dx), with the
// planes of a 16-channel K slice CV_PLANE bytes apart.  One copy serves the
// three taps.  Stages run through a ring of NS buffers: while
// the tensor core consumes stages s - 1 and s, the copies of stages
// s + 1 .. s + NS - 2 are in flight.  Buffer b's mbarrier completes when the MMAs of the stage
// last held in b are done (tcgen05.commit), which is what a refill of b waits
// for; the 9th stage of a tile also releases the epilogue.  With the ReLU
// mask the gather goes through registers (plain loads and shared stores).
// CG = Cin / 8 (2, 4 or 8), a template parameter so that the gather's unit
// arithmetic is resolved at compile time.
template <int CG>
__global__ void __launch_bounds__(CV_THREADS, 1) conv3d_tc_kernel(
    const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ Mk, const __nv_bfloat16 *__restrict__ Wt,
    const float *__restrict__ bias, __nv_bfloat16 *__restrict__ Y, float *__restrict__ Yf, int D, int H, int W,
    int Cin, int Cout, int relu, int NS) {
  extern __shared__ __align__(1024) unsigned char sm[];
  const int KC = Cin >> 4;
  const int bblk = Cout * 32;  // bytes of one (tap, 16-wide K slice) weight block
  const size_t SBY = cv_stage_bytes(Cin);
  unsigned char *sB = sm;
  unsigned char *sA = sm + cv_weight_bytes(Cin, Cout);
  unsigned long long *bars = reinterpret_cast<unsigned long long *>(sA + NS * SBY);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bars + NS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ncols = Cout <= 32 ? 32u : 64u;

  // weights: one 16-byte unit = 8 consecutive k of one n
  const int units_per_tap = Cin * Cout / 8;
  for (int i = tid; i < 27 * units_per_tap; i += CV_THREADS) {
    const int tap = i / units_per_tap, r = i - tap * units_per_tap;
    const int kg = r / Cout, n = r - kg * Cout;  // kg: 8-element group of k
    const __nv_bfloat16 *src = Wt + (static_cast<int64_t>(tap) * Cin + kg * 8) * Cout + n;
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t lo = __bfloat16_as_ushort(src[(2 * j) * Cout]);
      const uint32_t hi = __bfloat16_as_ushort(src[(2 * j + 1) * Cout]);
      v[j] = lo | (hi << 16);
    }
    unsigned char *dst = sB + (tap * KC + (kg >> 1)) * bblk + (n >> 3) * 256 + (kg & 1) * 128 + (n & 7) * 16;
    *reinterpret_cast<uint4 *>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
  }
  if (tid == 0) {
    for (int b = 0; b < NS; ++b)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bars + b)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma_idesc_bf16(TC_M, Cout);

  const int ntx = (W + TC_M - 1) / TC_M;
  const int64_t ntiles = static_cast<int64_t>(D) * H * ntx;
  const int64_t my_tiles = ntiles > blockIdx.x ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int64_t nst = my_tiles * 9;

  // copies of stage s into buffer s % NS (nothing past the last stage); one
  // commit group per call on every thread, so the group counts stay uniform
  // This thread's share of a stage is the same for every stage: units
  // u = tid + j * CV_THREADS of (130 voxels) x CG channel groups, channel
  // group fastest, so a warp reads 512 contiguous bytes and the 8 lanes of a
  // 16-byte store phase hit all 32 banks (planes CV_PLANE = 8 banks apart).
  // Per unit: x offset from x0, element offset in the row, destination.
  constexpr int CIN = CG * 8;
  constexpr int UNITS = (TC_M + 2) * CG;
  constexpr int UPT = (UNITS + CV_THREADS - 1) / CV_THREADS;
  int u_x[UPT], u_off[UPT], u_dst[UPT];
#pragma unroll
  for (int j = 0; j < UPT; ++j) {
    const int i = tid + j * CV_THREADS;
    const int vx = i / CG, cg = i % CG;
    const bool unit = i < UNITS;
    u_x[j] = unit ? vx - 1 : INT_MIN / 2;
    u_off[j] = (vx - 1) * CIN + cg * 8;
    u_dst[j] = unit ? cg * CV_PLANE + vx * 16 : -1;
  }

  // Stage cursors advance by one stage at a time (no division per stage):
  // stage index within the tile (dz * 3 + dy), ring buffer and its phase
  // parity, and the tile with its coordinates (divisions once per tile).
  const int ntiles32 = static_cast<int>(ntiles);
  const int nst32 = static_cast<int>(nst);
  struct Cursor {
    int st9, buf, par, t, tx, y, z;
  };
  auto tile_coords = [&](Cursor &c) {
    c.tx = c.t % ntx;
    const int zy = c.t / ntx;
    c.y = zy % H;
    c.z = zy / H;
  };
  auto advance = [&](Cursor &c) {
    if (++c.buf == NS) {
      c.buf = 0;
      c.par ^= 1;
    }
    if (++c.st9 == 9) {
      c.st9 = 0;
      c.t += gridDim.x;
      if (c.t < ntiles32) tile_coords(c);
    }
  };

  // copies of the stage at cursor ci (nothing past the last stage); one
  // commit group per call on every thread, so the group counts stay uniform
  Cursor ci{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};
  tile_coords(ci);
  int si = 0;  // the stage ci points at
  auto issue = [&]() {
    if (si < nst32) {
      const int zz = ci.z + ci.st9 / 3 - 1, yy = ci.y + ci.st9 % 3 - 1, x0 = ci.tx * TC_M;
      const bool rowok = zz >= 0 && zz < D && yy >= 0 && yy < H;
      unsigned char *buf = sA + static_cast<size_t>(ci.buf) * SBY;
      const __nv_bfloat16 *row = X + ((static_cast<int64_t>(rowok ? zz : 0) * H + (rowok ? yy : 0)) * W + x0) * CIN;
#pragma unroll
      for (int j = 0; j < UPT; ++j) {
        const int xx = x0 + u_x[j];
        const bool in = rowok && xx >= 0 && xx < W;
        const __nv_bfloat16 *src = in ? row + u_off[j] : X;
        if (u_dst[j] < 0) continue;
        if (!Mk) {
          cp_async16(buf + u_dst[j], src, in ? 16 : 0);
        } else {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (in) {
            v = *reinterpret_cast<const uint4 *>(src);
            const uint4 mk = *reinterpret_cast<const uint4 *>(Mk + (src - X));
            __nv_bfloat16 *pv = reinterpret_cast<__nv_bfloat16 *>(&v);
            const __nv_bfloat16 *pm = reinterpret_cast<const __nv_bfloat16 *>(&mk);
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (!(__bfloat162float(pm[q]) > 0.0f)) pv[q] = __float2bfloat16(0.0f);
          }
          *reinterpret_cast<uint4 *>(buf + u_dst[j]) = v;
        }
      }
      advance(ci);
    }
    ++si;
    cp_async_commit();
  };

  // the copies run NS - 2 stages ahead; a buffer is refilled two stages
  // after its MMAs were issued, so their completion is not waited for at once
  for (int k = 0; k < NS - 2; ++k) issue();
  bool ok = true;
  Cursor cc{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};  // the stage consumed
  tile_coords(cc);
  Cursor cw{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};  // two stages behind: the buffer refilled next
  int s = 0, issued_buf = -1, issued_par = 0;  // the last stage whose MMAs were committed
  for (; s < nst32; ++s) {
    const int b = cc.buf;
    const int st9 = cc.st9;
    // this thread's copies of stage s have landed; hand them to the async
    // proxy, then every thread's (and a failed wait anywhere ends the loop)
    cp_async_wait(NS - 3);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    ok = __syncthreads_and(ok ? 1 : 0) != 0;
    tc_fence_after();
    if (!ok) break;
    if (tid == 0) {
      const int tapz = (st9 / 3) * 9 + (st9 % 3) * 3;  // (dz, dy) part of the tap index
#pragma unroll 1
      for (int dxi = 0; dxi < 3; ++dxi)
        for (int kc = 0; kc < KC; ++kc) {
          const uint64_t a =
              umma_smem_desc(smem_addr(sA + b * SBY + (2 * kc) * CV_PLANE + dxi * 16), CV_PLANE, 128);
          const uint64_t bd = umma_smem_desc(smem_addr(sB + ((tapz + dxi) * KC + kc) * bblk), 128, 256);
          mma_bf16(tmem, a, bd, idesc, (st9 | dxi | kc) != 0 ? 1u : 0u);
        }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_addr(bars + b))
                   : "memory");
    }
    issued_buf = b;
    issued_par = cc.par;
    // refill the buffer of stage s - 2 with stage s + NS - 2 once its MMAs
    // are done (for s < 2 that buffer has not been used yet)
    if (s >= 2) {
      ok = mbar_wait(smem_addr(bars + cw.buf), static_cast<uint32_t>(cw.par));
      advance(cw);
    }
    issue();
    if (st9 == 8) {
      // last stage of the tile: the accumulator is final once its MMAs are
      ok = __syncthreads_and((ok && mbar_wait(smem_addr(bars + b), static_cast<uint32_t>(cc.par))) ? 1 : 0) != 0;
      if (!ok) break;
      tc_fence_after();
      const int tx = cc.tx, y = cc.y, z = cc.z;
      // warp w: voxels 32 (w % 4) .. + 31 (its TMEM lanes), channel blocks
      // of 16 starting at 16 (w / 4), every second one
      const int m = (warp & 3) * 32 + lane, xx = tx * TC_M + m;
      for (int c0 = (warp >> 2) * 16; c0 < Cout; c0 += 32) {
        uint32_t r[16];
        tmem_ld16(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(c0), r);
        if (xx < W) {
          const int64_t o = ((static_cast<int64_t>(z) * H + y) * W + xx) * Cout + c0;
          float f[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float v = __uint_as_float(r[j]) + (bias ? bias[c0 + j] : 0.0f);
            f[j] = relu ? fmaxf(v, 0.0f) : v;
          }
          if (Yf) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              *reinterpret_cast<float4 *>(Yf + o + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
          } else {
            uint32_t p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
              p[j] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(f[2 * j]))) |
                     (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(f[2 * j + 1]))) << 16);
            *reinterpret_cast<uint4 *>(Y + o) = make_uint4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<uint4 *>(Y + o + 8) = make_uint4(p[4], p[5], p[6], p[7]);
          }
        }
      }
      // the next tile's first MMA overwrites the accumulator: these loads
      // are ordered before it by the next iteration's barrier
      tc_fence_before();
    }
    advance(cc);
  }
  cp_async_wait(0);
  if (!ok) {
    // a wait expired: record it and give the MMAs in flight one more
    // bounded wait (the last stage committed, which completes after all
    // earlier ones) before the accumulator is freed
    if (tid == 0) atomicExch(&g_tc_err, 1);
    if (issued_buf >= 0) mbar_wait(smem_addr(bars + issued_buf), static_cast<uint32_t>(issued_par));
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

// Warp-specialised form of the same convolution (the default;
// ORSP_WARM_TC_WS=0 selects the kernel above).
// Eight producer warps copy the stages and drain the accumulators; one MMA
// warp (lane 0) issues the tensor-core MMAs.  No block barrier separates the
// stages; per-buffer mbarriers hand them over:
//   full[b]   the producers' copies of the stage in b have landed (256
//             arrivals, each after its thread's cp.async group completed and
//             a proxy fence);
//   empty[b]  the MMAs that read b are done (tcgen05.commit);
//   accf[a]   accumulator a holds a finished tile (tcgen05.commit after the
//             tile's last stage);
//   acce[a]   the producers have read accumulator a (256 arrivals).
// Tiles alternate between two TMEM accumulators, so a tile's epilogue runs
// while the MMAs of the next tile proceed.  The producers signal stage s
// after issuing stage s + LAG (LAG = NS - 2, at most 4); a buffer is refilled
// only after its previous stage's MMAs are done, so the copies of LAG stages
// are in flight while the tensor core consumes.  Every wait is bounded; a
// wait that expires sets a shared abort flag that ends every other wait.
constexpr int WS_PROD = 256;
constexpr int WS_THREADS = WS_PROD + 32;

__host__ __device__ constexpr size_t ws_smem_bytes(int Cin, int Cout, int ns) {
  return cv_weight_bytes(Cin, Cout) + ns * cv_stage_bytes(Cin) + 16 * ns + 64;
}

template <int CG>
__global__ void __launch_bounds__(WS_THREADS, 1) conv3d_tc_ws_kernel(
    const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ Mk, const __nv_bfloat16 *__restrict__ Wt,
    const float *__restrict__ bias, __nv_bfloat16 *__restrict__ Y, float *__restrict__ Yf, int D, int H, int W,
    int Cin, int Cout, int relu, int NS, unsigned long long wait_ns) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ volatile int s_abort;
  const int KC = Cin >> 4;
  const int bblk = Cout * 32;
  const size_t SBY = cv_stage_bytes(Cin);
  unsigned char *sB = sm;
  unsigned char *sA = sm + cv_weight_bytes(Cin, Cout);
  unsigned long long *full = reinterpret_cast<unsigned long long *>(sA + NS * SBY);
  unsigned long long *empty = full + NS;
  unsigned long long *accf = empty + NS;
  unsigned long long *acce = accf + 2;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(acce + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ncols1 = Cout <= 32 ? 32u : 64u, ncols = 2 * ncols1;

  const int units_per_tap = Cin * Cout / 8;
  for (int i = tid; i < 27 * units_per_tap; i += WS_THREADS) {
    const int tap = i / units_per_tap, r = i - tap * units_per_tap;
    const int kg = r / Cout, n = r - kg * Cout;
    const __nv_bfloat16 *src = Wt + (static_cast<int64_t>(tap) * Cin + kg * 8) * Cout + n;
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t lo = __bfloat16_as_ushort(src[(2 * j) * Cout]);
      const uint32_t hi = __bfloat16_as_ushort(src[(2 * j + 1) * Cout]);
      v[j] = lo | (hi << 16);
    }
    unsigned char *dst = sB + (tap * KC + (kg >> 1)) * bblk + (n >> 3) * 256 + (kg & 1) * 128 + (n & 7) * 16;
    *reinterpret_cast<uint4 *>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
  }
  if (tid == 0) {
    s_abort = 0;
    for (int b = 0; b < NS; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(full + b)), "r"(WS_PROD) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(empty + b)) : "memory");
    }
    for (int a = 0; a < 2; ++a) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(accf + a)) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(acce + a)), "r"(WS_PROD) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma_idesc_bf16(TC_M, Cout);

  const int ntx = (W + TC_M - 1) / TC_M;
  const int64_t ntiles = static_cast<int64_t>(D) * H * ntx;
  const int64_t my_tiles = ntiles > blockIdx.x ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
  const int ntiles32 = static_cast<int>(ntiles);
  const int nst32 = static_cast<int>(my_tiles * 9);
  const int my32 = static_cast<int>(my_tiles);
  struct Cursor {
    int st9, buf, par, t, tx, y, z;
  };
  auto tile_coords = [&](Cursor &c) {
    c.tx = c.t % ntx;
    const int zy = c.t / ntx;
    c.y = zy % H;
    c.z = zy / H;
  };
  auto advance = [&](Cursor &c) {
    if (++c.buf == NS) {
      c.buf = 0;
      c.par ^= 1;
    }
    if (++c.st9 == 9) {
      c.st9 = 0;
      c.t += gridDim.x;
      if (c.t < ntiles32) tile_coords(c);
    }
  };
  // a bounded wait that also ends when another role has given up
  auto wait = [&](unsigned long long *bar, int parity) -> bool {
    const uint32_t a = smem_addr(bar);
    const unsigned long long t0 = dev_globaltimer();
    for (;;) {
      if (mbar_try(a, static_cast<uint32_t>(parity))) return true;
      if (s_abort) return false;
      if (dev_globaltimer() - t0 > wait_ns) {
        s_abort = 1;
        atomicExch(&g_tc_err, 1);
        return false;
      }
    }
  };
  // the same by a whole warp, whose lanes go on or give up together: one lane
  // may find the phase complete and another the abort flag, and what follows
  // (tcgen05.ld) takes all of them
  auto wait_warp = [&](unsigned long long *bar, int parity) { return __all_sync(0xffffffffu, wait(bar, parity)) != 0; };
  const int LAG = NS - 2 < 4 ? NS - 2 : 4;

  if (warp < 8) {
    // ------------------------------------------------------------ producers
    constexpr int CIN = CG * 8;
    constexpr int UNITS = (TC_M + 2) * CG;
    constexpr int UPT = (UNITS + WS_PROD - 1) / WS_PROD;
    int u_x[UPT], u_off[UPT], u_dst[UPT];
#pragma unroll
    for (int j = 0; j < UPT; ++j) {
      const int i = tid + j * WS_PROD;
      const int vx = i / CG, cg = i % CG;
      const bool unit = i < UNITS;
      u_x[j] = unit ? vx - 1 : INT_MIN / 2;
      u_off[j] = (vx - 1) * CIN + cg * 8;
      u_dst[j] = unit ? cg * CV_PLANE + vx * 16 : -1;
    }
    auto epilogue = [&](int tx, int y, int z, int acc) {
      const int m = (warp & 3) * 32 + lane, xx = tx * TC_M + m;
      for (int c0 = (warp >> 2) * 16; c0 < Cout; c0 += 32) {
        uint32_t r[16];
        tmem_ld16(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + static_cast<uint32_t>(acc) * ncols1 +
                      static_cast<uint32_t>(c0),
                  r);
        if (xx < W) {
          const int64_t o = ((static_cast<int64_t>(z) * H + y) * W + xx) * Cout + c0;
          float f[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float v = __uint_as_float(r[j]) + (bias ? bias[c0 + j] : 0.0f);
            f[j] = relu ? fmaxf(v, 0.0f) : v;
          }
          if (Yf) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              *reinterpret_cast<float4 *>(Yf + o + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
          } else {
            uint32_t p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
              p[j] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(f[2 * j]))) |
                     (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(f[2 * j + 1]))) << 16);
            *reinterpret_cast<uint4 *>(Y + o) = make_uint4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<uint4 *>(Y + o + 8) = make_uint4(p[4], p[5], p[6], p[7]);
          }
        }
      }
    };
    Cursor ci{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};  // the stage issued next
    tile_coords(ci);
    Cursor cs{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};  // the stage signalled next
    Cursor et{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};  // the tile drained next
    tile_coords(et);
    int ep_T = 0;
    bool ok = true;
    // drains tile ep_T (accumulator ep_T & 1) and frees the accumulator
    auto drain = [&]() -> bool {
      if (!wait_warp(accf + (ep_T & 1), (ep_T >> 1) & 1)) return false;
      tc_fence_after();
      epilogue(et.tx, et.y, et.z, ep_T & 1);
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(acce + (ep_T & 1))) : "memory");
      ++ep_T;
      et.t += gridDim.x;
      if (et.t < ntiles32) tile_coords(et);
      return true;
    };
    for (int s = 0; s < nst32 + LAG && ok; ++s) {
      if (s < nst32) {
        // the buffer's previous stage must have been consumed
        if (s >= NS && !wait_warp(empty + ci.buf, ci.par ^ 1)) {
          ok = false;
          break;
        }
        const int zz = ci.z + ci.st9 / 3 - 1, yy = ci.y + ci.st9 % 3 - 1, x0 = ci.tx * TC_M;
        const bool rowok = zz >= 0 && zz < D && yy >= 0 && yy < H;
        unsigned char *buf = sA + static_cast<size_t>(ci.buf) * SBY;
        const __nv_bfloat16 *row = X + ((static_cast<int64_t>(rowok ? zz : 0) * H + (rowok ? yy : 0)) * W + x0) * CIN;
#pragma unroll
        for (int j = 0; j < UPT; ++j) {
          const int xx = x0 + u_x[j];
          const bool in = rowok && xx >= 0 && xx < W;
          const __nv_bfloat16 *src = in ? row + u_off[j] : X;
          if (u_dst[j] < 0) continue;
          if (!Mk) {
            cp_async16(buf + u_dst[j], src, in ? 16 : 0);
          } else {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (in) {
              v = *reinterpret_cast<const uint4 *>(src);
              const uint4 mk = *reinterpret_cast<const uint4 *>(Mk + (src - X));
              __nv_bfloat16 *pv = reinterpret_cast<__nv_bfloat16 *>(&v);
              const __nv_bfloat16 *pm = reinterpret_cast<const __nv_bfloat16 *>(&mk);
#pragma unroll
              for (int q = 0; q < 8; ++q)
                if (!(__bfloat162float(pm[q]) > 0.0f)) pv[q] = __float2bfloat16(0.0f);
            }
            *reinterpret_cast<uint4 *>(buf + u_dst[j]) = v;
          }
        }
        advance(ci);
      }
      cp_async_commit();
      const int sd = s - LAG;
      if (sd >= 0) {
        // this thread's copies of stage sd have landed: hand them to the
        // async proxy and count them in
        cp_async_wait(LAG);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(full + cs.buf)) : "memory");
        advance(cs);
        // two stages of the next tile are handed over: drain the tile before
        if (sd == 9 * ep_T + 10 && !drain()) ok = false;
      }
    }
    while (ok && ep_T < my32) ok = drain();
    cp_async_wait(0);
  } else if (lane == 0) {
    // ------------------------------------------------------------ MMA warp
    Cursor cc{0, 0, 0, static_cast<int>(blockIdx.x), 0, 0, 0};
    int T = 0, last_buf = -1, last_par = 0;
    bool ok = true;
    for (int s = 0; s < nst32; ++s) {
      const int st9 = cc.st9, a = T & 1;
      if (st9 == 0 && T >= 2 && !wait(acce + a, ((T - 2) >> 1) & 1)) { ok = false; break; }
      if (!wait(full + cc.buf, cc.par)) { ok = false; break; }
      tc_fence_after();
      const int tapz = (st9 / 3) * 9 + (st9 % 3) * 3;
#pragma unroll 1
      for (int dxi = 0; dxi < 3; ++dxi)
        for (int kc = 0; kc < KC; ++kc) {
          const uint64_t ad =
              umma_smem_desc(smem_addr(sA + cc.buf * SBY + (2 * kc) * CV_PLANE + dxi * 16), CV_PLANE, 128);
          const uint64_t bd = umma_smem_desc(smem_addr(sB + ((tapz + dxi) * KC + kc) * bblk), 128, 256);
          mma_bf16(tmem + static_cast<uint32_t>(a) * ncols1, ad, bd, idesc, (st9 | dxi | kc) != 0 ? 1u : 0u);
        }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_addr(empty + cc.buf))
                   : "memory");
      if (st9 == 8)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_addr(accf + a))
                     : "memory");
      last_buf = cc.buf;
      last_par = cc.par;
      if (st9 == 8) ++T;
      advance(cc);
    }
    // after a failed wait, the MMAs in flight get one more bounded wait (the
    // last commit completes after all earlier ones) before TMEM is freed
    if (!ok && last_buf >= 0) mbar_wait(smem_addr(empty + last_buf), static_cast<uint32_t>(last_par));
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

// Instruction descriptor with both operands MN-major (bit 15: A, bit 16: B).
__host__ __device__ constexpr uint32_t umma_idesc_bf16_mn(int M, int N) {
  return umma_idesc_bf16(M, N) | (1u << 15) | (1u << 16);
}

constexpr int WG_K = 32;  // voxels per stage of the weight gradient: two K = 16 MMAs

__host__ __device__ constexpr int wg_taps_per_tile(int Cin) { return 128 / Cin; }
__host__ __device__ constexpr int wg_mtiles(int Cin) { return (27 + 128 / Cin - 1) / (128 / Cin); }
__host__ __device__ constexpr size_t wg_smem_bytes(int Cin, int Cout) {
  return static_cast<size_t>(wg_mtiles(Cin)) * 2 * 4096 + static_cast<size_t>(2) * Cout * 32 + 64;
}
__host__ __device__ constexpr uint32_t wg_tmem_cols(int Cin, int Cout) {
  return wg_mtiles(Cin) * Cout <= 32 ? 32u : wg_mtiles(Cin) * Cout <= 64 ? 64u : wg_mtiles(Cin) * Cout <= 128 ? 128u
         : wg_mtiles(Cin) * Cout <= 256 ? 256u : 512u;
}

// Weight gradient dW[tap][ci][co] += sum_v X[v + tap][ci] G[v][co] (G = dY,
// or dY where Yo > 0) on tcgen05: D[m][n] = sum_k A[m][k] B[n][k] with
// m = (tap slot, ci), 128 / Cin taps per 128-row M tile (one TMEM
// accumulator of Cout columns per M tile), n = co, k = voxels, 32 voxels of
// one (z, y) row per stage.  For a fixed voxel both operands are contiguous
// along M or N (channels last), so A and B are MN-major: core matrices of 8
// voxels x 8 channels (16 bytes), K groups 128 bytes apart, 8-channel groups
// 256 bytes apart.  Persistent CTAs each sum a share of the voxels in TMEM
// and add their partial sums to dW with fp32 atomics at the end.
__global__ void __launch_bounds__(TC_THREADS, 1) wgrad_tc_kernel(
    const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ dY, const __nv_bfloat16 *__restrict__ Yo,
    float *__restrict__ dW, int D, int H, int W, int Cin, int Cout) {
  extern __shared__ __align__(1024) unsigned char sm[];
  const int TPM = wg_taps_per_tile(Cin), MT = wg_mtiles(Cin);
  const int bblk = Cout * 32;
  unsigned char *sA = sm;                                  // [MT][2 k-steps] blocks of 4096 bytes
  unsigned char *sB = sm + static_cast<size_t>(MT) * 2 * 4096;  // [2 k-steps] blocks of Cout * 32 bytes
  unsigned long long *bar = reinterpret_cast<unsigned long long *>(sB + 2 * bblk);
  uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ncols = wg_tmem_cols(Cin, Cout);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const uint32_t idesc = umma_idesc_bf16_mn(TC_M, Cout);
  const uint32_t bar_a = smem_addr(bar);
  uint32_t phase = 0;
  bool ok = true, any = false;
  const int nxc = (W + WG_K - 1) / WG_K;
  const int64_t nchunks = static_cast<int64_t>(D) * H * nxc;
  const int cg_in = Cin / 8, cg_out = Cout / 8;
  // 32-bit chunk arithmetic (the host rejects grids with more chunks)
  for (int t = blockIdx.x; t < static_cast<int>(nchunks) && ok; t += gridDim.x) {
    const int xc = t % nxc;
    const int zy = t / nxc;
    const int y = zy % H, z = zy / H;
    const int x0 = xc * WG_K;
    // B: G of the chunk's 32 voxels, 8 output channels per unit
    for (int i = tid; i < WG_K * cg_out; i += TC_THREADS) {
      const int k = i % WG_K, g = i / WG_K;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (x0 + k < W) {
        const int64_t off = ((static_cast<int64_t>(z) * H + y) * W + x0 + k) * Cout + g * 8;
        v = *reinterpret_cast<const uint4 *>(dY + off);
        if (Yo) {
          const uint4 mk = *reinterpret_cast<const uint4 *>(Yo + off);
          __nv_bfloat16 *pv = reinterpret_cast<__nv_bfloat16 *>(&v);
          const __nv_bfloat16 *pm = reinterpret_cast<const __nv_bfloat16 *>(&mk);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (!(__bfloat162float(pm[q]) > 0.0f)) pv[q] = __float2bfloat16(0.0f);
        }
      }
      const int ks = k >> 4, kk = k & 15;
      *reinterpret_cast<uint4 *>(sB + ks * bblk + g * 256 + (kk >> 3) * 128 + (kk & 7) * 16) = v;
    }
    // A: the shifted inputs of the taps of every M tile, 8 input channels per unit
    for (int i = tid; i < MT * TPM * cg_in * WG_K; i += TC_THREADS) {
      const int k = i % WG_K;
      int r = i / WG_K;
      const int cg = r % cg_in;
      r /= cg_in;
      const int slot = r % TPM, mt = r / TPM;
      const int tap = mt * TPM + slot;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (tap < 27 && x0 + k < W) {
        const int zz = z + tap / 9 - 1, yy = y + (tap / 3) % 3 - 1, xx = x0 + k + tap % 3 - 1;
        if (zz >= 0 && zz < D && yy >= 0 && yy < H && xx >= 0 && xx < W)
          v = *reinterpret_cast<const uint4 *>(X + ((static_cast<int64_t>(zz) * H + yy) * W + xx) * Cin + cg * 8);
      }
      const int mg = slot * cg_in + cg;  // 8-row group of m = slot * Cin + 8 cg
      const int ks = k >> 4, kk = k & 15;
      *reinterpret_cast<uint4 *>(sA + (mt * 2 + ks) * 4096 + mg * 256 + (kk >> 3) * 128 + (kk & 7) * 16) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
      for (int mt = 0; mt < MT; ++mt)
        for (int ks = 0; ks < 2; ++ks) {
          const uint64_t a = umma_smem_desc(smem_addr(sA + (mt * 2 + ks) * 4096), 128, 256);
          const uint64_t b = umma_smem_desc(smem_addr(sB + ks * bblk), 128, 256);
          mma_bf16(tmem + static_cast<uint32_t>(mt * Cout), a, b, idesc, (any || ks) ? 1u : 0u);
        }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_a)
                   : "memory");
    }
    ok = __syncthreads_and(mbar_wait(bar_a, phase) ? 1 : 0) != 0;
    phase ^= 1u;
    tc_fence_after();
    any = true;
  }
  if (ok && any) {
    // partial sums: warp w holds rows m = 32w..32w+31 of every M tile
    const int m = warp * 32 + lane, slot = m / Cin, ci = m % Cin;
    for (int mt = 0; mt < MT; ++mt) {
      const int tap = mt * TPM + slot;
      for (int c0 = 0; c0 < Cout; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(mt * Cout + c0), r);
        if (tap < 27) {
          float *dst = dW + (static_cast<int64_t>(tap) * Cin + ci) * Cout + c0;
#pragma unroll
          for (int j = 0; j < 16; ++j) atomicAdd(dst + j, __uint_as_float(r[j]));
        }
      }
    }
  }
  if (!ok) {
    if (tid == 0) atomicExch(&g_tc_err, 1);
    mbar_wait(bar_a, phase ^ 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

// ---------------------------------------------------------------------------
// Plane kernels: convolution and weight gradient of 16- and 32-channel layers
// with up to 32 channels on the other side.
//
// The kernels above copy rows with cp.async into a layout built by hand, run
// MMAs of N = Cout (32) columns, and re-read the 4 KB A operand for every tap:
// 40 clocks of shared memory for 16 of tensor work per MMA, behind a serial
// copy (127 TFLOP/s; the weight gradient, one barrier and one wait per 32
// voxels, 40).  Here
//  - a plane of the tile (32 voxels x 8 rows and its halo) arrives by one TMA
//    load, zero-filled outside the grid, in the swizzled layout that the
//    MMA reads; a CTA marches along z, so a plane is loaded once for the
//    three output planes that use it;
//  - the taps that differ in x share one MMA: N = 3 Cout columns hold their
//    partial products of the same input voxels, and the epilogue adds the
//    three with a shift of one voxel (a TMEM quarter is one row of 32 voxels,
//    so the shift is a shuffle).  27 x Cin / 16 MMAs of 32 columns become
//    9 x Cin / 16 of 96, whose tensor time covers their operand reads;
//  - warps are specialised: TMA, MMA, ReLU-mask (in place in shared memory,
//    only when a mask is given), epilogue on a second accumulator pair.
// Measured, 32 -> 32 channels: 400 x 400 x 18 forward 1 259 -> 177 us (900
// TFLOP/s; 100 us of it are the MMAs, 59 clocks each, the rest the hand-overs
// between the steps and the last, partial round of tiles); 200 x 200 x 18 with
// the ReLU mask: weight gradient 1 982 -> 70 us, input gradient 660 -> 60 us.
// Every wait is bounded; one that expires sets the abort flag that ends the
// others, the TMA thread waits (bounded) for its loads in flight, and TMEM is
// freed.  No load is multicast.
constexpr int PL_X = 32;              // voxels per patch row, one TMEM quarter
constexpr int PL_Y = 8;               // rows of a tile
constexpr int PL_ROWS = PL_Y + 2;     // with the halo rows
constexpr int PL_MASK = 128;          // threads that apply the ReLU mask

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}

// Shared-memory descriptor of a swizzled operand whose rows are C channels of
// bf16 (64-byte swizzle for 32, 32-byte for 16): sbo between groups of eight
// rows, lbo between blocks of C channels (M- or N-major operands only).
template <int C>
__device__ __forceinline__ uint64_t plane_desc(uint32_t addr, uint32_t lbo) {
  constexpr uint64_t layout = C == 32 ? 4 : 6;
  return umma_smem_desc(addr, lbo, 8 * C * 2) | (layout << 61);
}

// The tiles of a launch: nxs x nys columns of tiles, each cut into nzc
// chunks of zc planes; unit u is chunk u / (nxs nys) of column u mod (nxs nys).
struct PlanePlan {
  int nxs, nys, zc, units;
};

struct PlaneUnit {
  int x, y, z0, z1;  // column, planes [z0, z1)
  __device__ __forceinline__ PlaneUnit() {}
  __device__ __forceinline__ PlaneUnit(const PlanePlan &pl, int u, int D) {
    const int cols = pl.nxs * pl.nys, c = u % cols;
    x = c % pl.nxs;
    y = c / pl.nxs;
    z0 = (u / cols) * pl.zc;
    z1 = min(D, z0 + pl.zc);
  }
};

// The weight gradient's tiles: a CTA's share is a range of all columns' planes,
// one column after the other, and shares differ by one plane at most.  Its
// rounding error is that of the longest sums: chunks of one length gave some
// CTAs 24 planes of 200 x 200 x 18 and others 18 (9 and 4 of 72 x 112 x 17).
struct PlaneShare {
  int at, end;
  __device__ __forceinline__ PlaneShare(const PlanePlan &pl, int D) {
    const int64_t n = static_cast<int64_t>(pl.nxs) * pl.nys * D;
    at = static_cast<int>(n * blockIdx.x / gridDim.x);
    end = static_cast<int>(n * (blockIdx.x + 1) / gridDim.x);
  }
  __device__ __forceinline__ bool more() const { return at < end; }
  __device__ __forceinline__ PlaneUnit next(const PlanePlan &pl, int D) {
    PlaneUnit u;
    const int c = at / D;
    u.x = c % pl.nxs;
    u.y = c / pl.nxs;
    u.z0 = at - c * D;
    u.z1 = min(D, u.z0 + end - at);
    at += u.z1 - u.z0;
    return u;
  }
};

// Keeps the elements of NBYTES of bf16 at v where the mask m is positive, by
// PL_MASK threads, a few 16-byte pieces in flight per thread.
template <int NBYTES>
__device__ __forceinline__ void mask_plane(unsigned char *v, const unsigned char *m, int tid) {
  constexpr int STEP = PL_MASK * 16, U = 5;
  static_assert(NBYTES % STEP == 0, "whole steps");
#pragma unroll 1
  for (int i = tid * 16; i < NBYTES; i += STEP * U) {
    uint4 a[U], b[U];
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (i + q * STEP < NBYTES) {
        a[q] = *reinterpret_cast<uint4 *>(v + i + q * STEP);
        b[q] = *reinterpret_cast<const uint4 *>(m + i + q * STEP);
      }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      uint32_t *pa = reinterpret_cast<uint32_t *>(&a[q]);
      const uint32_t *pb = reinterpret_cast<const uint32_t *>(&b[q]);
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        // positive and not NaN: bits 1 .. 0x7f80
        const uint32_t lo = ((pb[w] & 0xffffu) - 1u) < 0x7f80u ? 0xffffu : 0u;
        const uint32_t hi = ((pb[w] >> 16) - 1u) < 0x7f80u ? 0xffff0000u : 0u;
        pa[w] &= lo | hi;
      }
      if (i + q * STEP < NBYTES) *reinterpret_cast<uint4 *>(v + i + q * STEP) = a[q];
    }
  }
}

__device__ __forceinline__ void mbar_init(void *bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(void *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(void *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma_commit(void *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Completes the loads above; the registers pass through so that no use of
// them moves ahead of the wait.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[16], uint32_t (&b)[16], uint32_t (&c)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) asm volatile("" : "+r"(a[k]), "+r"(b[k]), "+r"(c[k]));
}
// 32 bytes as one store where the array is aligned for it.
__device__ __forceinline__ void store32(void *dst, const uint32_t *v, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4 *>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<uint4 *>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
  }
}

constexpr int PL_MAXB = 8;  // plane buffers at most
struct PlaneBars {
  unsigned long long full[PL_MAXB], ready[PL_MAXB], empty[PL_MAXB];  // loaded, masked, consumed
  unsigned long long mfree[2];                                       // mask buffer read
  unsigned long long xfull[2], xempty[2];                            // weight gradient: X planes
  unsigned long long accf[2], acce[2];
  uint32_t tmem;
  volatile int abort;
};

// Waits for `parity` of a barrier, bounded; ends early when another role has
// given up, and makes the others give up when it expires.
__device__ __forceinline__ bool plane_wait(PlaneBars &pb, unsigned long long wait_ns, void *bar, int parity) {
  const uint32_t a = smem_addr(bar);
  if (mbar_try(a, static_cast<uint32_t>(parity))) return true;
  const unsigned long long t0 = dev_globaltimer();
  for (;;) {
    if (mbar_try(a, static_cast<uint32_t>(parity))) return true;
    if (pb.abort) return false;
    if (dev_globaltimer() - t0 > wait_ns) {
      pb.abort = 1;
      atomicExch(&g_tc_err, 1);
      return false;
    }
  }
}

// The same for a whole warp, whose lanes go on or give up together: waiting by
// themselves, one may find the phase complete and another the abort flag, and
// what follows (tcgen05.ld, shuffles) takes all of them.  Lane 0 waits for all
// (a vote on every lane's wait: 181.7 us for 400 x 400 x 18, 32 -> 32, this 177.1).
__device__ __forceinline__ bool plane_wait_warp(PlaneBars &pb, unsigned long long wait_ns, void *bar, int parity) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = plane_wait(pb, wait_ns, bar, parity);
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();  // what lane 0 has waited for is visible to all
  return ok != 0;
}

// TMA, MMA, mask warps, sixteen epilogue warps
template <bool MASK>
__host__ __device__ constexpr int pc_threads() { return 64 + (MASK ? PL_MASK : 0) + 512; }

template <int CIN>
__host__ __device__ constexpr int plane_bytes() { return PL_X * PL_ROWS * CIN * 2; }
template <int CIN>
__host__ __device__ constexpr size_t pc_weight_bytes(int Cout) { return static_cast<size_t>(27) * CIN * Cout * 2; }

// Convolution.  An MMA tile is four rows of 32 voxels (M = 128), a step two of
// them (8 rows) of one output plane; patch columns overlap by two voxels, so a
// row gives 30 outputs.
template <int CIN, bool MASK>
__global__ void __launch_bounds__(pc_threads<MASK>(), 1) conv3d_planes_kernel(
    const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmm,
    const __nv_bfloat16 *__restrict__ Wt, const float *__restrict__ bias, __nv_bfloat16 *__restrict__ Y,
    float *__restrict__ Yf, int D, int H, int W, int Cout, int relu, PlanePlan plan, int NB,
    unsigned long long wait_ns) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ PlaneBars pb;
  constexpr int KC = CIN / 16, PB = plane_bytes<CIN>(), EPI = 2 + (MASK ? PL_MASK / 32 : 0);  // first epilogue warp
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char *const planes = sm;                                    // [NB] planes, 1024-byte aligned
  unsigned char *const masks = planes + static_cast<size_t>(NB) * PB;  // [2] mask planes (MASK)
  unsigned char *const sB = masks + (MASK ? 2 * PB : 0);
  const int N = 3 * Cout, bblk = N * 32;
  // weights: block (dz, dy; 16-wide K slice) of rows n = dx * Cout + co, K-major
  // without swizzle: 8-row groups 256 bytes apart, K halves 128
  for (int i = tid; i < 9 * KC * 2 * N; i += pc_threads<MASK>()) {
    const int n = i % N, r = i / N, kh = r & 1, kc = (r >> 1) % KC, zy = (r >> 1) / KC;
    const int dx = n / Cout, co = n - dx * Cout;
    const __nv_bfloat16 *src = Wt + (static_cast<int64_t>(zy * 3 + dx) * CIN + kc * 16 + kh * 8) * Cout + co;
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = static_cast<uint32_t>(__bfloat16_as_ushort(src[(2 * j) * Cout])) |
             (static_cast<uint32_t>(__bfloat16_as_ushort(src[(2 * j + 1) * Cout])) << 16);
    *reinterpret_cast<uint4 *>(sB + (zy * KC + kc) * bblk + (n >> 3) * 256 + kh * 128 + (n & 7) * 16) =
        make_uint4(v[0], v[1], v[2], v[3]);
  }
  if (tid == 0) {
    pb.abort = 0;
    for (int b = 0; b < NB; ++b) {
      mbar_init(&pb.full[b], 1);
      mbar_init(&pb.ready[b], PL_MASK);
      mbar_init(&pb.empty[b], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&pb.mfree[a], PL_MASK);
      mbar_init(&pb.accf[a], 1);
      mbar_init(&pb.acce[a], 256 * (Cout >> 4));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  const uint32_t ncols = 4 * N <= 256 ? 256u : 512u;  // two steps of two accumulators
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&pb.tmem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = pb.tmem;

  if (warp == 0) {
    if (lane == 0) {
      // -------------------------------------------------------------- TMA
      int n = 0;  // planes issued
      bool ok = true;
      for (int u = blockIdx.x; u < plan.units && ok; u += gridDim.x) {
        const PlaneUnit un(plan, u, D);
        for (int z = max(un.z0 - 1, 0); z <= min(un.z1, D - 1); ++z, ++n) {
          const int b = n % NB;
          if (n >= NB && !plane_wait(pb, wait_ns, &pb.empty[b], (n / NB - 1) & 1)) { ok = false; break; }
          if (MASK && n >= 2 && !plane_wait(pb, wait_ns, &pb.mfree[n & 1], ((n >> 1) - 1) & 1)) { ok = false; break; }
          mbar_expect(&pb.full[b], MASK ? 2 * PB : PB);
          const int x = un.x * (PL_X - 2) - 1, y = un.y * PL_Y - 1;
          tma_load_4d(smem_addr(planes + static_cast<size_t>(b) * PB), &tmx, smem_addr(&pb.full[b]), x, y, z);
          if (MASK) tma_load_4d(smem_addr(masks + (n & 1) * PB), &tmm, smem_addr(&pb.full[b]), x, y, z);
        }
      }
      // the loads in flight land before the block ends, also after a failure
      for (int k = max(0, n - NB); k < n; ++k) mbar_wait(smem_addr(&pb.full[k % NB]), (k / NB) & 1);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA
    const uint32_t idesc = umma_idesc_bf16(TC_M, N);
    const uint64_t bd0 = umma_smem_desc(smem_addr(sB), 128, 256), bstep = static_cast<uint64_t>(bblk >> 4);
    const uint64_t pl0 = plane_desc<CIN>(smem_addr(planes), 16);
    int b = 0, par = 0, step = 0;  // the next plane's buffer and parity; steps made
    bool ok = true;
    for (int u = blockIdx.x; u < plan.units && ok; u += gridDim.x) {
      const PlaneUnit un(plan, u, D);
      // buffers of the planes below, at and above z (-1: outside the grid)
      int bz[3] = {-1, -1, -1};
      auto next = [&]() {  // the next plane of the unit, when it has landed
        ok = ok && plane_wait(pb, wait_ns, MASK ? &pb.ready[b] : &pb.full[b], par);
        const int got = b;
        if (++b == NB) b = 0, par ^= 1;
        return got;
      };
      if (un.z0 > 0) bz[1] = next();
      bz[2] = next();
      for (int z = un.z0; z < un.z1; ++z, ++step) {
        const int a = step & 1;
        bz[0] = bz[1];
        bz[1] = bz[2];
        bz[2] = z + 1 < D ? next() : -1;
        if (ok && step >= 2) ok = plane_wait(pb, wait_ns, &pb.acce[a], ((step >> 1) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (elect_lane()) {
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const uint32_t acc = tmem + static_cast<uint32_t>((a * 2 + j) * N);
            uint32_t add = 0;
#pragma unroll
            for (int dz = 0; dz < 3; ++dz) {
              if (bz[dz] < 0) continue;
              uint64_t bd = bd0 + static_cast<uint64_t>(dz * 3 * KC) * bstep;
              const uint64_t pd = pl0 + static_cast<uint64_t>(bz[dz] * (PB / 16));
#pragma unroll
              for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int kc = 0; kc < KC; ++kc) {
                  // (addresses stay below 2^18: sums of descriptors do not carry)
                  mma_bf16(acc, pd + ((j * 4 + dy) * (PL_X * CIN * 2) + kc * 32) / 16, bd, idesc, add);
                  add = 1;
                  bd += bstep;
                }
            }
          }
          mma_commit(&pb.accf[a]);
          if (bz[0] >= 0) mma_commit(&pb.empty[bz[0]]);
          if (z == un.z1 - 1) {  // the planes still held
            mma_commit(&pb.empty[bz[1]]);
            if (bz[2] >= 0) mma_commit(&pb.empty[bz[2]]);
          }
        }
        __syncwarp();
      }
    }
    // after a failed wait the MMAs in flight get one more bounded wait
    if (!ok && step > 0) mbar_wait(smem_addr(&pb.accf[(step - 1) & 1]), ((step - 1) >> 1) & 1);
    __syncwarp();
  } else if (warp < EPI) {
    // ---------------------------------------------------------------- mask
    if (MASK) {
      int n = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < plan.units && ok; u += gridDim.x) {
        const PlaneUnit un(plan, u, D);
        for (int z = max(un.z0 - 1, 0); z <= min(un.z1, D - 1) && ok; ++z, ++n) {
          const int b = n % NB;
          ok = plane_wait(pb, wait_ns, &pb.full[b], (n / NB) & 1);
          if (!ok) break;
          mask_plane<PB>(planes + static_cast<size_t>(b) * PB, masks + (n & 1) * PB, tid - 64);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          mbar_arrive(&pb.ready[b]);
          mbar_arrive(&pb.mfree[n & 1]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // TMEM quarter warp % 4 (one row of 32 voxels); groups of four warps take
    // MMA tile 0 or 1 and sixteen of the output channels
    const int e = warp - EPI, qd = warp & 3, j = (e >> 2) & 1, c = e >> 3;
    int step = 0;
    bool ok = c * 16 < Cout;
    float bv[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) bv[k] = ok && bias ? __ldg(&bias[c * 16 + k]) : 0.0f;
    const bool wide = ((reinterpret_cast<uintptr_t>(Yf ? static_cast<void *>(Yf) : static_cast<void *>(Y))) & 31) == 0;
    for (int u = blockIdx.x; u < plan.units && ok; u += gridDim.x) {
      const PlaneUnit un(plan, u, D);
      const int y = un.y * PL_Y + j * 4 + qd, x = un.x * (PL_X - 2) - 1 + lane;
      const bool in = lane >= 1 && lane <= 30 && x < W && y < H;
      for (int z = un.z0; z < un.z1; ++z, ++step) {
        const int a = step & 1;
        ok = plane_wait_warp(pb, wait_ns, &pb.accf[a], (step >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
        const uint32_t t0 =
            tmem + (static_cast<uint32_t>(qd * 32) << 16) + static_cast<uint32_t>((a * 2 + j) * N + c * 16);
        uint32_t r0[16], r1[16], r2[16];
        tmem_ld16_async(t0, r0);
        tmem_ld16_async(t0 + Cout, r1);
        tmem_ld16_async(t0 + 2 * Cout, r2);
        tmem_ld_wait(r0, r1, r2);
        tc_fence_before();
        mbar_arrive(&pb.acce[a]);  // the accumulator is read
        float f[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          const float l = __shfl_up_sync(0xffffffffu, __uint_as_float(r0[k]), 1);
          const float r = __shfl_down_sync(0xffffffffu, __uint_as_float(r2[k]), 1);
          const float v = ((l + __uint_as_float(r1[k])) + r) + bv[k];
          f[k] = relu ? fmaxf(v, 0.0f) : v;
        }
        if (!in) continue;
        const int64_t o = ((static_cast<int64_t>(z) * H + y) * W + x) * Cout + c * 16;
        uint32_t p[16];
        if (Yf) {
#pragma unroll
          for (int k = 0; k < 16; ++k) p[k] = __float_as_uint(f[k]);
          store32(Yf + o, p, wide);
          store32(Yf + o + 8, p + 8, wide);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k)
            p[k] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(f[2 * k]))) |
                   (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16(f[2 * k + 1]))) << 16);
          store32(Y + o, p, wide);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

constexpr int PW_THREADS = 64 + PL_MASK + 128;  // TMA, MMA, mask warps, four epilogue warps

// TMEM column of the accumulator of dz for even (0) and odd (1) planes of a
// share: 6 x 48 columns for 16 output channels; 5 x 96 of 512 for 32, the last dz
// has one.
template <int COUT>
__host__ __device__ constexpr int pw_acc(int dz, int odd) {
  return 3 * COUT * (COUT == 16 || dz < 2 ? 2 * dz + odd : 4);
}

template <int CIN>
__host__ __device__ constexpr int pw_x_bytes() { return PL_X * PL_Y * CIN * 2; }  // one shifted X plane
template <int COUT>
__host__ __device__ constexpr int pw_g_bytes() { return PL_X * PL_ROWS * COUT * 2; }

// The CTA's share of dW pair by pair, where its accumulators are not finite:
// the tiles are padded with zeros on both sides, and a zero meets an infinity
// or a NaN of the border there that no pair of the sum holds.  The pairs are X[v
// + tap] and G[v] for v in the grid (X zero outside it), as the zero-padded
// convolution has them; rows and planes of X just outside the grid go with the
// border tiles.  Every warp takes 32 rows (dx, ci) x 16 columns of a (dz, dy).
template <int CIN, int COUT>
__device__ __noinline__ void wgrad_pairs(const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ dY,
                                         const __nv_bfloat16 *__restrict__ Yo, float *__restrict__ dW, int D, int H,
                                         int W, const PlanePlan &plan) {
  constexpr int MT = (3 * CIN + 31) / 32, CT = COUT / 16;
  const int lane = threadIdx.x & 31;
  for (int task = threadIdx.x >> 5; task < MT * CT * 9; task += PW_THREADS / 32) {
    const int m = task % MT * 32 + lane, c0 = task / MT % CT * 16, dz = task / (MT * CT) / 3, dy = task / (MT * CT) % 3;
    const int dx = m / CIN, ci = m % CIN;
    float acc[16] = {};
    for (PlaneShare sh(plan, D); sh.more();) {
      const PlaneUnit un = sh.next(plan, D);
      const int y0 = un.y * PL_Y, ylo = y0 == 0 ? -1 : y0, yhi = y0 + PL_Y >= H ? H : y0 + PL_Y - 1;
      const int zlo = un.z0 == 0 ? -1 : un.z0, zhi = un.z1 == D ? D : un.z1 - 1;
      const int x0 = un.x * PL_X, x1 = min(x0 + PL_X, W);
      for (int zx = max(zlo, dz - 1); zx <= min(zhi, D - 2 + dz); ++zx)
        for (int yx = max(ylo, dy - 1); yx <= min(yhi, H - 2 + dy); ++yx) {
          const bool row = dx < 3 && zx >= 0 && zx < D && yx >= 0 && yx < H;
          const int64_t g0 = (static_cast<int64_t>(zx - dz + 1) * H + (yx - dy + 1)) * W;
          const int64_t r0 = row ? (static_cast<int64_t>(zx) * H + yx) * W : 0;
          for (int x = x0; x < x1; ++x) {
            const int xx = x + dx - 1;
            const float xv =
                row && xx >= 0 && xx < W ? __bfloat162float(X[(r0 + xx) * CIN + ci]) : 0.0f;
            const __nv_bfloat16 *g = dY + (g0 + x) * COUT + c0;
            const __nv_bfloat16 *k = Yo ? Yo + (g0 + x) * COUT + c0 : nullptr;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              const float gv = !k || __bfloat162float(k[q]) > 0.0f ? __bfloat162float(g[q]) : 0.0f;
              acc[q] = fmaf(xv, gv, acc[q]);
            }
          }
        }
    }
    if (dx < 3)
      for (int q = 0; q < 16; ++q)
        atomicAdd(dW + (static_cast<int64_t>(dz * 9 + dy * 3 + dx) * CIN + ci) * COUT + c0 + q, acc[q]);
  }
}

// Weight gradient: for each plane z' of X, row y' and voxel x of a tile,
//   D[dz][(dx, ci)][(dy, co)] += X[z'][y'][x + dx][ci] G[z' - dz][y' - dy][x][co]
// as M = 128 (three dx blocks of CIN channels, the rest of M unused) by N = 3
// COUT (three dy blocks) MMAs over K = 16 voxels; both operands are M- or
// N-major (channels contiguous).  The dx blocks are three TMA loads of the X
// plane, one voxel apart, the dy blocks the G plane one row apart, so one MMA
// serves nine taps.  The accumulators (dz) stay in TMEM over a CTA's share and
// are added to dW once, four values per atomic (adding them twice, in halves of
// the share, took 10 us more).  The rounding error of a sum in TMEM grows with
// its length to the power 1.5, so the planes alternate between two
// accumulators of a dz where TMEM holds them (pw_acc), which are added before
// they leave.
// Error of dW against 64 bits, 200 x 200 x 18, 32 -> 32 channels: 2.34e-6 with
// chunks of one length and one accumulator, 2.34e-6 with even shares, 1.55e-6 with
// both; 144 x 184 x 12, 32 -> 16: 1.18e-6, 8.8e-7, 4.4e-7.
template <int CIN, int COUT, bool MASK>
__global__ void __launch_bounds__(PW_THREADS, 1) wgrad_planes_kernel(
    const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmg,
    const __grid_constant__ CUtensorMap tmm, const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ dY,
    const __nv_bfloat16 *__restrict__ Yo, float *__restrict__ dW, int D, int H, int W, PlanePlan plan,
    unsigned long long wait_ns) {
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ PlaneBars pb;
  __shared__ int s_bad;  // an accumulator is not finite
  constexpr int XB = pw_x_bytes<CIN>(), GB = pw_g_bytes<COUT>(), NG = 4, N = 3 * COUT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char *const xs = sm;               // [2][3] shifted X planes
  unsigned char *const gs = xs + 6 * XB;      // [NG] G planes
  unsigned char *const ms = gs + NG * GB;     // [2] mask planes (MASK)
  if (tid == 0) {
    pb.abort = s_bad = 0;
    for (int b = 0; b < NG; ++b) {
      mbar_init(&pb.full[b], 1);
      mbar_init(&pb.ready[b], PL_MASK);
      mbar_init(&pb.empty[b], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&pb.mfree[a], PL_MASK);
      mbar_init(&pb.xfull[a], 1);
      mbar_init(&pb.xempty[a], 1);
    }
    mbar_init(&pb.accf[0], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  constexpr uint32_t ncols = 512;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&pb.tmem)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = pb.tmem;

  if (warp == 0) {
    if (lane == 0) {
      // -------------------------------------------------------------- TMA
      int n = 0, m = 0;  // G planes, X planes issued
      bool ok = true;
      auto load_g = [&](const PlaneUnit &un, int z) {
        const int b = n % NG;
        if (n >= NG && !plane_wait(pb, wait_ns, &pb.empty[b], (n / NG - 1) & 1)) return false;
        if (MASK && n >= 2 && !plane_wait(pb, wait_ns, &pb.mfree[n & 1], ((n >> 1) - 1) & 1)) return false;
        mbar_expect(&pb.full[b], MASK ? 2 * GB : GB);
        tma_load_4d(smem_addr(gs + b * GB), &tmg, smem_addr(&pb.full[b]), un.x * PL_X, un.y * PL_Y - 1, z);
        if (MASK) tma_load_4d(smem_addr(ms + (n & 1) * GB), &tmm, smem_addr(&pb.full[b]), un.x * PL_X, un.y * PL_Y - 1, z);
        ++n;
        return true;
      };
      for (PlaneShare sh(plan, D); sh.more() && ok;) {
        const PlaneUnit un = sh.next(plan, D);
        const int zhi = min(un.z1, D - 1);
        int zg = max(un.z0 - 1, 0);
        for (int z = un.z0; z < un.z1 && ok; ++z, ++m) {
          while (ok && zg <= min(z + 1, zhi)) ok = load_g(un, zg++);
          const int b = m & 1;
          if (!ok || (m >= 2 && !plane_wait(pb, wait_ns, &pb.xempty[b], ((m >> 1) - 1) & 1))) { ok = false; break; }
          mbar_expect(&pb.xfull[b], 3 * XB);
          for (int dx = 0; dx < 3; ++dx)
            tma_load_4d(smem_addr(xs + (b * 3 + dx) * XB), &tmx, smem_addr(&pb.xfull[b]), un.x * PL_X + dx - 1,
                        un.y * PL_Y, z);
        }
      }
      for (int k = max(0, n - NG); k < n; ++k) mbar_wait(smem_addr(&pb.full[k % NG]), (k / NG) & 1);
      for (int k = max(0, m - 2); k < m; ++k) mbar_wait(smem_addr(&pb.xfull[k & 1]), (k >> 1) & 1);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA
    const uint32_t idesc = umma_idesc_bf16_mn(TC_M, N);
    const uint64_t x0d = plane_desc<CIN>(smem_addr(xs), XB), g0d = plane_desc<COUT>(smem_addr(gs), PL_X * COUT * 2);
    int b = 0, par = 0, m = 0;
    uint32_t used[3][2] = {};
    bool ok = true;
    for (PlaneShare sh(plan, D); sh.more() && ok;) {
      const PlaneUnit un = sh.next(plan, D);
      int bz[3] = {-1, -1, -1};  // G planes below, at and above z
      auto next = [&]() {
        ok = ok && plane_wait(pb, wait_ns, MASK ? &pb.ready[b] : &pb.full[b], par);
        const int got = b;
        if (++b == NG) b = 0, par ^= 1;
        return got;
      };
      if (un.z0 > 0) bz[1] = next();
      bz[2] = next();
      for (int z = un.z0; z < un.z1; ++z, ++m) {
        bz[0] = bz[1];
        bz[1] = bz[2];
        bz[2] = z + 1 < D ? next() : -1;
        if (ok) ok = plane_wait(pb, wait_ns, &pb.xfull[m & 1], (m >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        const bool odd = m & 1;
        if (elect_lane()) {
#pragma unroll
          for (int dz = 0; dz < 3; ++dz) {  // tap dz - 1: the G plane at z - (dz - 1)
            const int g = bz[2 - dz];
            if (g < 0) continue;
            uint64_t ad = x0d + static_cast<uint64_t>((m & 1) * (3 * XB / 16));
            uint64_t bd = g0d + static_cast<uint64_t>(g * (GB / 16));
            const uint32_t acc = tmem + static_cast<uint32_t>(odd ? pw_acc<COUT>(dz, 1) : pw_acc<COUT>(dz, 0));
            uint32_t add = odd ? used[dz][1] : used[dz][0];
#pragma unroll
            for (int k = 0; k < PL_Y * 2; ++k) {
              mma_bf16(acc, ad, bd, idesc, add);
              add = 1;
              ad += 16 * CIN * 2 / 16;
              bd += 16 * COUT * 2 / 16;
            }
          }
          mma_commit(&pb.xempty[m & 1]);
          if (bz[0] >= 0) mma_commit(&pb.empty[bz[0]]);
          if (z == un.z1 - 1) {
            mma_commit(&pb.empty[bz[1]]);
            if (bz[2] >= 0) mma_commit(&pb.empty[bz[2]]);
          }
        }
        __syncwarp();
#pragma unroll
        for (int dz = 0; dz < 3; ++dz)
          if (bz[2 - dz] >= 0) {
            if (!odd || pw_acc<COUT>(dz, 0) == pw_acc<COUT>(dz, 1)) used[dz][0] = 1;
            if (odd || pw_acc<COUT>(dz, 0) == pw_acc<COUT>(dz, 1)) used[dz][1] = 1;
          }
      }
    }
    if (elect_lane()) mma_commit(&pb.accf[0]);  // after every MMA of the CTA, also after a failed wait
    __syncwarp();
    if (!ok) mbar_wait(smem_addr(&pb.accf[0]), 0);
    __syncwarp();
  } else if (warp < 2 + PL_MASK / 32) {
    if (MASK) {
      int n = 0;
      bool ok = true;
      for (PlaneShare sh(plan, D); sh.more() && ok;) {
        const PlaneUnit un = sh.next(plan, D);
        for (int z = max(un.z0 - 1, 0); z <= min(un.z1, D - 1) && ok; ++z, ++n) {
          const int b = n % NG;
          ok = plane_wait(pb, wait_ns, &pb.full[b], (n / NG) & 1);
          if (!ok) break;
          mask_plane<GB>(gs + b * GB, ms + (n & 1) * GB, tid - 64);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          mbar_arrive(&pb.ready[b]);
          mbar_arrive(&pb.mfree[n & 1]);
        }
      }
    }
  }
  // ---------------------------------------------------------------- epilogue
  // Warps 6 to 9, a TMEM quarter each (32 rows of (dx, ci)): they look at the
  // accumulators first and add them to dW when the whole CTA has seen that all
  // are finite.
  const int qd = warp & 3, mrow = qd * 32 + lane, dx = mrow / CIN, ci = mrow % CIN;
  const bool sums = warp >= 2 + PL_MASK / 32 && qd * 32 < 3 * CIN;
  // accumulators that some plane of this CTA wrote: a plane has no G plane
  // above it at the top of the grid, none below at the bottom
  bool used[3][2] = {};
  if (sums) {
    int m = 0;
    for (PlaneShare sh(plan, D); sh.more();) {
      const PlaneUnit un = sh.next(plan, D);
      for (int z = un.z0; z < un.z1; ++z, ++m)
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
          const bool w = dz == 1 || (dz == 0 ? z < D - 1 : z > 0);
          if (pw_acc<COUT>(dz, 0) == pw_acc<COUT>(dz, 1) || !(m & 1)) used[dz][0] = used[dz][0] || w;
          else used[dz][1] = used[dz][1] || w;
        }
    }
  }
  auto accumulators = [&](auto each) {  // each(dz, dy, first channel, 16 values)
    const uint32_t t0 = tmem + (static_cast<uint32_t>(qd * 32) << 16);
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
      if (!used[dz][0] && !used[dz][1]) continue;
      const bool both = used[dz][0] && used[dz][1];
      for (int blk = 0; blk < 3; ++blk) {  // block 0 pairs row y' with G row y' - 1
        // all columns of a block in flight at a time
        const uint32_t t1 = t0 + static_cast<uint32_t>(blk * COUT + pw_acc<COUT>(dz, used[dz][0] ? 0 : 1));
        const uint32_t t2 = both ? t0 + static_cast<uint32_t>(blk * COUT + pw_acc<COUT>(dz, 1)) : t1;
        uint32_t r[COUT / 16][16], o[COUT / 16][16];
#pragma unroll
        for (int c = 0; c < COUT / 16; ++c) {
          tmem_ld16_async(t1 + c * 16, r[c]);
          tmem_ld16_async(t2 + c * 16, o[c]);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < COUT / 16; ++c) {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            asm volatile("" : "+r"(r[c][k]), "+r"(o[c][k]));  // (no use of them before the wait)
            if (both) r[c][k] = __float_as_uint(__uint_as_float(r[c][k]) + __uint_as_float(o[c][k]));
          }
          each(dz, 2 - blk, c * 16, r[c]);
        }
      }
    }
  };
  if (sums && plane_wait_warp(pb, wait_ns, &pb.accf[0], 0)) {
    tc_fence_after();
    bool bad = false;
    accumulators([&](int, int, int, const uint32_t (&r)[16]) {
#pragma unroll
      for (int k = 0; k < 16; ++k) bad = bad || (r[k] & 0x7f800000u) == 0x7f800000u;
    });
    if (bad && dx < 3) s_bad = 1;
    tc_fence_before();
  }
  __syncthreads();
  if (!pb.abort) {
    if (s_bad) {
      wgrad_pairs<CIN, COUT>(X, dY, MASK ? Yo : nullptr, dW, D, H, W, plan);
    } else if (sums) {
      tc_fence_after();
      accumulators([&](int dz, int dy, int c0, const uint32_t (&r)[16]) {
        if (dx >= 3) return;
        float *dst = dW + (static_cast<int64_t>(dz * 9 + dy * 3 + dx) * CIN + ci) * COUT + c0;
        if ((reinterpret_cast<uintptr_t>(dW) & 15) == 0) {
#pragma unroll
          for (int k = 0; k < 16; k += 4)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + k), "f"(__uint_as_float(r[k])),
                         "f"(__uint_as_float(r[k + 1])), "f"(__uint_as_float(r[k + 2])), "f"(__uint_as_float(r[k + 3]))
                         : "memory");
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k) atomicAdd(dst + k, __uint_as_float(r[k]));
        }
      });
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols) : "memory");
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library); nullptr when unavailable.
PFN_cuTensorMapEncodeTiled_v12000 warm_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)f;
    else
      (void)cudaGetLastError();
  });
  return fn;
}

// Map of a [D][H][W][C] bf16 array, box C x 32 voxels x `rows` x 1, swizzled by
// the row of channels; false when the address is not 16-byte aligned or the
// encoder refuses.
bool plane_map(CUtensorMap *m, const void *X, int D, int H, int W, int C, int rows) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = warm_map_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(X) & 15)) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
  const cuuint64_t str[3] = {(cuuint64_t)C * 2, (cuuint64_t)C * 2 * W, (cuuint64_t)C * 2 * W * H};
  const cuuint32_t box[4] = {(cuuint32_t)C, PL_X, (cuuint32_t)rows, 1}, es[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(X), dims, str, box, es,
             CU_TENSOR_MAP_INTERLEAVE_NONE, C == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Cuts D planes of `cols` tile columns into chunks so that the CTA with the
// most work has the fewest planes (a chunk loads about one plane's worth more
// than it computes).
PlanePlan plane_plan(int nxs, int nys, int D, int ctas) {
  PlanePlan best{nxs, nys, D, 0};
  double cost = 1e30;
  const int64_t cols = (int64_t)nxs * nys;
  for (int zc = 1; zc <= D; ++zc) {
    const int64_t units = cols * ((D + zc - 1) / zc);
    if (units > INT32_MAX) continue;
    const double c = (double)((units + ctas - 1) / ctas) * (zc + 0.6);
    if (c < cost) {
      cost = c;
      best.zc = zc;
      best.units = (int)units;
    }
  }
  return best;
}

// db[co] += sum_v G[v][co] (G = dY, or dY where Yo > 0).  Eight channels of a
// voxel (16 bytes) per load, so a thread always sees the same eight channels
// (the grid's stride is a multiple of Cout / 8); sums per block in shared
// memory, one atomic per channel and block.  Bound by reading dY and Yo
// (92 MB for 200 x 200 x 18 x 32 in 23 us).
__global__ void bias_sum_kernel(const uint4 *__restrict__ dY, const uint4 *__restrict__ Yo, float *__restrict__ db,
                                int64_t n, int Cout) {
  extern __shared__ float s_db[];
  for (int c = threadIdx.x; c < Cout; c += blockDim.x) s_db[c] = 0.0f;
  __syncthreads();
  const int64_t first = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  float acc[8] = {};
  constexpr int U = 4;  // loads in flight per thread
  for (int64_t i = first; i < n; i += U * stride) {
    uint4 g[U], m[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      g[q] = make_uint4(0, 0, 0, 0);
      m[q] = make_uint4(0x00010001u, 0x00010001u, 0x00010001u, 0x00010001u);
      if (i + q * stride < n) {
        g[q] = __ldg(&dY[i + q * stride]);
        if (Yo) m[q] = __ldg(&Yo[i + q * stride]);
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const uint32_t gw[4] = {g[q].x, g[q].y, g[q].z, g[q].w}, mw[4] = {m[q].x, m[q].y, m[q].z, m[q].w};
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        if (((mw[w] & 0xffffu) - 1u) < 0x7f80u) acc[2 * w] += __uint_as_float(gw[w] << 16);
        if (((mw[w] >> 16) - 1u) < 0x7f80u) acc[2 * w + 1] += __uint_as_float(gw[w] & 0xffff0000u);
      }
    }
  }
  const int c0 = static_cast<int>(first % (Cout / 8)) * 8;
#pragma unroll
  for (int k = 0; k < 8; ++k) atomicAdd(&s_db[c0 + k], acc[k]);
  __syncthreads();
  for (int c = threadIdx.x; c < Cout; c += blockDim.x) atomicAdd(&db[c], s_db[c]);
}

}  // namespace

using namespace orsp;

// The plane kernel's launch; ORSP_NO_PATH when its loads do not apply (input
// or mask not 16-byte aligned).
static int conv3d_planes(const void *X, const void *mask, const void *Wt, const float *bias, void *Y, float *Yf, int D,
                         int H, int W, int Cin, int Cout, int relu, cudaStream_t st) {
  CUtensorMap tx, tm;
  if (!plane_map(&tx, X, D, H, W, Cin, PL_ROWS)) return ORSP_NO_PATH;
  tm = tx;
  if (mask && !plane_map(&tm, mask, D, H, W, Cin, PL_ROWS)) return ORSP_NO_PATH;
  int dev = 0, sms = 0;
  ORSP_CUDA(cudaGetDevice(&dev));
  ORSP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const PlanePlan plan = plane_plan((W + PL_X - 3) / (PL_X - 2), (H + PL_Y - 1) / PL_Y, D, sms);
  if (plan.units <= 0) return ORSP_NO_PATH;
  const size_t pb = Cin == 32 ? plane_bytes<32>() : plane_bytes<16>();
  const size_t wb = Cin == 32 ? pc_weight_bytes<32>(Cout) : pc_weight_bytes<16>(Cout);
  // (the attribute is the kernel's, for all threads: a size that fits every
  // launch, so that one does not lower it between another's setting and launch)
  constexpr size_t kSmem = 224 * 1024;
  const size_t room = kSmem - wb - (mask ? 2 * pb : 0);
  const int nb = (int)std::min<size_t>(PL_MAXB, room / pb);
  const size_t smem = nb * pb + (mask ? 2 * pb : 0) + wb;
  auto kfn = Cin == 32 ? (mask ? conv3d_planes_kernel<32, true> : conv3d_planes_kernel<32, false>)
                       : (mask ? conv3d_planes_kernel<16, true> : conv3d_planes_kernel<16, false>);
  ORSP_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
  kfn<<<std::min(plan.units, sms), mask ? pc_threads<true>() : pc_threads<false>(), smem, st>>>(tx, tm, (const __nv_bfloat16 *)Wt, bias, (__nv_bfloat16 *)Y,
                                                           Yf, D, H, W, Cout, relu, plan, nb, tc_wait_ns());
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

static int wgrad_planes(const void *X, const void *dY, const void *Yo, float *dW, int D, int H, int W, int Cin,
                        int Cout, cudaStream_t st) {
  CUtensorMap tx, tg, tm;
  if (!plane_map(&tx, X, D, H, W, Cin, PL_Y) || !plane_map(&tg, dY, D, H, W, Cout, PL_ROWS)) return ORSP_NO_PATH;
  tm = tg;
  if (Yo && !plane_map(&tm, Yo, D, H, W, Cout, PL_ROWS)) return ORSP_NO_PATH;
  int dev = 0, sms = 0;
  ORSP_CUDA(cudaGetDevice(&dev));
  ORSP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const PlanePlan plan{(W + PL_X - 1) / PL_X, (H + PL_Y - 1) / PL_Y, 0, 0};
  const int64_t nplanes = (int64_t)plan.nxs * plan.nys * D;
  if (nplanes > INT32_MAX) return ORSP_NO_PATH;
  const size_t xb = Cin == 32 ? pw_x_bytes<32>() : pw_x_bytes<16>(), gb = Cout == 32 ? pw_g_bytes<32>() : pw_g_bytes<16>();
  // (the unused rows of M read past the third X plane, within the allocation)
  const size_t smem = std::max(6 * xb + 4 * gb + (Yo ? 2 * gb : 0), 3 * xb + 128 / Cin * xb);
  auto pick = [&](auto masked) {
    constexpr bool M = decltype(masked)::value;
    return Cin == 32 ? (Cout == 32 ? wgrad_planes_kernel<32, 32, M> : wgrad_planes_kernel<32, 16, M>)
                     : (Cout == 32 ? wgrad_planes_kernel<16, 32, M> : wgrad_planes_kernel<16, 16, M>);
  };
  auto kfn = Yo ? pick(std::true_type()) : pick(std::false_type());
  ORSP_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kfn<<<(int)std::min<int64_t>(nplanes, sms), PW_THREADS, smem, st>>>(
      tx, tg, tm, (const __nv_bfloat16 *)X, (const __nv_bfloat16 *)dY, (const __nv_bfloat16 *)Yo, dW, D, H, W, plan,
      tc_wait_ns());
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

extern "C" int orsp_warm_conv3d_tc(const void *X, const void *mask, const void *Wt, const float *bias, void *Y,
                                   float *Yf, int32_t D, int32_t H, int32_t W, int32_t Cin, int32_t Cout,
                                   int32_t relu, uintptr_t stream) {
  if (!X || !Wt || (!Y && !Yf) || D <= 0 || H <= 0 || W <= 0 || Cin <= 0 || Cin % 16 || Cout <= 0 ||
      Cout % 16 || Cout > 64) {
    set_error("warm_conv3d_tc: bad arguments (Cin, Cout multiples of 16, Cout <= 64)");
    return ORSP_ERR_ARG;
  }
  const char *ws = getenv("ORSP_WARM_TC_WS");
  const bool stage_barrier = ws && ws[0] == '0';
  if (!stage_barrier && (Cin == 16 || Cin == 32) && Cout <= 32) {
    int rc = conv3d_planes(X, mask, Wt, bias, Y, Yf, D, H, W, Cin, Cout, relu, (cudaStream_t)stream);
    if (rc != ORSP_NO_PATH) return rc;
  }
  const int ns = cv_stages(Cin, Cout);
  if (ns < 2) {
    set_error("warm_conv3d_tc: weights of this Cin x Cout and two stages do not fit in shared memory");
    return ORSP_ERR_ARG;
  }
  const size_t smem = cv_smem_bytes(Cin, Cout, ns);
  int dev = 0, sms = 0;
  ORSP_CUDA(cudaGetDevice(&dev));
  ORSP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  void (*kfn)(const __nv_bfloat16 *, const __nv_bfloat16 *, const __nv_bfloat16 *, const float *, __nv_bfloat16 *,
              float *, int, int, int, int, int, int, int) =
      Cin == 16 ? conv3d_tc_kernel<2> : Cin == 32 ? conv3d_tc_kernel<4> : Cin == 64 ? conv3d_tc_kernel<8> : nullptr;
  if (!kfn) {
    set_error("warm_conv3d_tc: Cin must be 16, 32 or 64");
    return ORSP_ERR_ARG;
  }
  ORSP_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t ntiles = static_cast<int64_t>(D) * H * ((W + TC_M - 1) / TC_M);
  if (ntiles * 9 > INT32_MAX) {
    set_error("warm_conv3d_tc: grid too large (the stage counters are 32-bit)");
    return ORSP_ERR_ARG;
  }
  const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(ntiles, sms)));
  // the warp-specialised kernel (producer warps and an MMA warp handing
  // stages over through mbarriers); ORSP_WARM_TC_WS=0: the kernel with one
  // block barrier per stage
  if (!stage_barrier) {
    auto kws = Cin == 16 ? conv3d_tc_ws_kernel<2> : Cin == 32 ? conv3d_tc_ws_kernel<4>
                                                                       : conv3d_tc_ws_kernel<8>;
    const size_t smem_ws = ws_smem_bytes(Cin, Cout, ns);
    ORSP_CUDA(cudaFuncSetAttribute(kws, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_ws));
    kws<<<grid, WS_THREADS, smem_ws, (cudaStream_t)stream>>>((const __nv_bfloat16 *)X, (const __nv_bfloat16 *)mask,
                                                             (const __nv_bfloat16 *)Wt, bias, (__nv_bfloat16 *)Y, Yf,
                                                             D, H, W, Cin, Cout, relu, ns, tc_wait_ns());
    ORSP_CUDA(cudaGetLastError());
    return ORSP_OK;
  }
  kfn<<<grid, CV_THREADS, smem, (cudaStream_t)stream>>>((const __nv_bfloat16 *)X, (const __nv_bfloat16 *)mask,
                                                        (const __nv_bfloat16 *)Wt, bias, (__nv_bfloat16 *)Y, Yf, D, H,
                                                        W, Cin, Cout, relu, ns);
  ORSP_CUDA(cudaGetLastError());
  return ORSP_OK;
}

extern "C" int orsp_warm_tc_status(int32_t *expired) {
  if (!expired) { set_error("warm_tc_status: NULL argument"); return ORSP_ERR_ARG; }
  int v = 0, zero = 0;
  ORSP_CUDA(cudaMemcpyFromSymbol(&v, g_tc_err, sizeof(int)));
  ORSP_CUDA(cudaMemcpyToSymbol(g_tc_err, &zero, sizeof(int)));
  *expired = v;
  return ORSP_OK;
}

extern "C" int orsp_warm_wgrad_tc(const void *X, const void *dY, const void *Yo, float *dW, float *db, int32_t D,
                                  int32_t H, int32_t W, int32_t Cin, int32_t Cout, uintptr_t stream) {
  if (!X || !dY || !dW || D <= 0 || H <= 0 || W <= 0 || Cin <= 0 || Cin % 16 || Cin > 64 || Cout <= 0 ||
      Cout % 16 || Cout > 64 || wg_mtiles(Cin) * Cout > 512) {
    set_error("warm_wgrad_tc: bad arguments (Cin, Cout multiples of 16, at most 64, accumulators within TMEM)");
    return ORSP_ERR_ARG;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0, sms = 0;
  ORSP_CUDA(cudaGetDevice(&dev));
  ORSP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int rc = ORSP_NO_PATH;
  if ((Cin == 16 || Cin == 32) && (Cout == 16 || Cout == 32)) rc = wgrad_planes(X, dY, Yo, dW, D, H, W, Cin, Cout, st);
  if (rc < 0) return rc;
  if (rc == ORSP_NO_PATH) {
    const size_t smem = wg_smem_bytes(Cin, Cout);
    ORSP_CUDA(cudaFuncSetAttribute(wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t nchunks = static_cast<int64_t>(D) * H * ((W + WG_K - 1) / WG_K);
    if (nchunks > INT32_MAX) {
      set_error("warm_wgrad_tc: grid too large (the chunk counter is 32-bit)");
      return ORSP_ERR_ARG;
    }
    const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(nchunks, sms)));
    wgrad_tc_kernel<<<grid, TC_THREADS, smem, st>>>((const __nv_bfloat16 *)X, (const __nv_bfloat16 *)dY,
                                                    (const __nv_bfloat16 *)Yo, dW, D, H, W, Cin, Cout);
    ORSP_CUDA(cudaGetLastError());
  }
  if (db) {
    const int64_t nvox = static_cast<int64_t>(D) * H * W;
    const int per = Cout / 8, threads = 256 / per * per;  // a multiple of the pieces of a voxel
    const int blocks = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((nvox * per + 1023) / 1024, sms * 4)));
    bias_sum_kernel<<<blocks, threads, Cout * sizeof(float), st>>>((const uint4 *)dY, (const uint4 *)Yo, db, nvox * per,
                                                                   Cout);
    ORSP_CUDA(cudaGetLastError());
  }
  return ORSP_OK;
}
