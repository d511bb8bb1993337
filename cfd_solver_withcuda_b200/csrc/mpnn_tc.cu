// Dense layers of the warm-start surrogate on the tensor cores (no reference counterpart).
//
// Every dense block of the network is a two-layer perceptron y = W2 silu(W1 x + b1) + b2 (+ r),
// hidden width 64, whose input row x is up to three row segments side by side, each read from
// its own array, directly or through a row index (the per-edge gathers of the message-passing
// layers are fused into the operand loads).  Operands are rounded to BF16 when they are loaded, the input
// rows into the MMA fragments' registers, weights (and the weight gradients' tiles) into shared memory;
// the products accumulate in FP32 (mma.sync m16n8k16, BF16 inputs, FP32 accumulators); bias, SiLU,
// residual and the SiLU derivative are FP32 epilogues.
//
//   k_mlp_fwd    y and the hidden pre-activation z1 (kept for the backward pass): one warp per 16
//                rows, input rows straight from global memory into the MMA fragments, weights
//                staged once per block.
//   k_mlp_bwd    dz1 = (dy W2) * silu'(z1) and dx = dz1 W1, one warp per 16 rows (k_mlp_bwd_tc: the
//                same on tcgen05).
//   k_wgrad      dW = dz^T x and db = sum of dz over the rows: each block accumulates its 64-row
//                tiles in registers and writes one partial; k_wgrad_reduce sums the partials in
//                block order, so the gradients are the same on every run.
//
// The CPU FP64 restatement these kernels are checked against is oracle/mpnn_ref.py.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "cfd_b200.h"

namespace cfdb {
void set_last_error(const std::string &msg);
}

namespace {

constexpr int TM = 64;    // rows per tile of the weight gradients
constexpr int HID = 64;   // hidden width
constexpr int KMAX = 192; // widest input row
constexpr int LDH = HID + 8;

struct SegDev {
  const float *src;
  const int *idx;
  int width, ld, silu;
};

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float dsilu_f(float z) {
  const float s = 1.0f / (1.0f + expf(-z));
  return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ uint16_t bf(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

// D += A B with A 16x16 (row-major fragment), B 16x8 (column-major fragment), BF16 in, FP32 acc.
__device__ __forceinline__ void mma16816(float d[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t bf2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}
// Four 8x8 BF16 matrices of shared memory (row addresses from lanes 0-7, 8-15, 16-23, 24-31), as
// stored or transposed.
__device__ __forceinline__ void ldsm4(const uint16_t *p, uint32_t r[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}
__device__ __forceinline__ void ldsm4t(const uint16_t *p, uint32_t r[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))));
}
// B fragments of the two column tiles [n, n+16), rows [k, k+16) of B: stored as B^T ([n][k], ld) ...
__device__ __forceinline__ void frag_b2(const uint16_t *s, int ld, int n, int k, int lane, uint32_t b[4]) {
  ldsm4(s + (n + ((lane >> 4) << 3) + (lane & 7)) * ld + k + (((lane >> 3) & 1) << 3), b);
}
// ... and stored as B itself ([k][n], ld).
__device__ __forceinline__ void frag_b2t(const uint16_t *s, int ld, int n, int k, int lane, uint32_t b[4]) {
  ldsm4t(s + (k + (((lane >> 3) & 1) << 3) + (lane & 7)) * ld + n + ((lane >> 4) << 3), b);
}
// A fragment of rows [m, m+16), columns [k, k+16) of A, stored as A^T ([k][m], ld).
__device__ __forceinline__ void frag_at(const uint16_t *s, int ld, int m, int k, int lane, uint32_t a[4]) {
  ldsm4t(s + (k + ((lane >> 4) << 3) + (lane & 7)) * ld + m + (((lane >> 3) & 1) << 3), a);
}
// rows x cols floats ([rows][cols], packed) as BF16 into s ([rp][ld]), zeros outside.  cp: columns
// written (a multiple of 16).
__device__ __forceinline__ void stage_weights(const float *w, int rows, int cols, uint16_t *s, int rp, int cp, int ld) {
  if ((cols & 3) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 && cp == cols) {
    const int c4 = cols >> 2, n = rows * c4;
    const float4 *w4 = reinterpret_cast<const float4 *>(w);
#pragma unroll 8
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
      const int r = e / c4, c = e - r * c4;
      const float4 v = __ldg(w4 + e);
      *reinterpret_cast<uint2 *>(s + r * ld + 4 * c) = make_uint2(bf2(v.x, v.y), bf2(v.z, v.w));
    }
    for (int e = threadIdx.x; e < (rp - rows) * cp; e += blockDim.x) {
      const int r = e / cp, c = e - r * cp;
      s[(rows + r) * ld + c] = 0;
    }
    return;
  }
  for (int e = threadIdx.x; e < rp * cp; e += blockDim.x) {
    const int r = e / cp, c = e - r * cp;
    s[r * ld + c] = (r < rows && c < cols) ? bf(w[r * cols + c]) : 0;
  }
}

// Value of column k of input row `row` (the segments side by side).
__device__ __forceinline__ float seg_value(const SegDev *seg, int nseg, int row, int k) {
  int off = 0;
  for (int s = 0; s < nseg; s++) {
    const int w = seg[s].width;
    if (k < off + w) {
      const int r = seg[s].idx ? seg[s].idx[row] : row;
      const float v = seg[s].src[(size_t)r * seg[s].ld + (k - off)];
      return seg[s].silu ? silu_f(v) : v;
    }
    off += w;
  }
  return 0.0f;
}

struct FwdArgs {
  int M, K, N2, nseg;
  SegDev seg[3];
  const float *w1, *b1, *w2, *b2, *resid;
  int ld_resid;
  float *z1, *y;
  int ld_y;
  int vec_y;  // mma.sync form: y (and the residual) in 8-byte pieces
};

constexpr int kMlpThreads = 256, kMlpWarps = kMlpThreads / 32;

// One warp per 16 input rows.  The A fragments come straight from global memory: the four lanes of
// a fragment row read 8 consecutive floats (one 32-byte sector) per load, a 64-column piece of a
// segment is 16 independent loads per lane, and the hidden layer passes from the accumulators of
// the first product to the A fragments of the second in registers, so that shared memory holds
// only the weights and no barrier separates the tiles.  Bound by the rows' traffic (edge block: 256 B read and
// 512 B written per row, the two gathered rows from L2) and its latency at 16 warps per SM.
// VEC: every segment's width is a multiple of 16, its rows are 8-byte aligned and it has no
// silu(); otherwise the values are fetched one by one.
template <bool VEC>
__global__ void __launch_bounds__(kMlpThreads, 2) k_mlp_fwd(FwdArgs a) {
  extern __shared__ __align__(16) uint16_t sm[];
  const int Kp = (a.K + 15) & ~15, LDX = Kp + 8, N2p = (a.N2 + 15) & ~15;
  uint16_t *sW1 = sm;                // [HID][LDX]   W1 (B operand of GEMM 1, [n][k])
  uint16_t *sW2 = sW1 + HID * LDX;   // [N2p][LDH]   W2 (B operand of GEMM 2)
  stage_weights(a.w1, HID, a.K, sW1, HID, Kp, LDX);
  stage_weights(a.w2, a.N2, HID, sW2, N2p, HID, LDH);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ntiles = (a.M + 15) >> 4;
  for (int tile = blockIdx.x * kMlpWarps + warp; tile < ntiles; tile += gridDim.x * kMlpWarps) {
    const int ra = tile * 16 + g, rb = ra + 8;
    const int la = min(ra, a.M - 1), lb = min(rb, a.M - 1);  // rows past the end repeat the last one, unstored
    float acc[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
    if (VEC) {
      const float *pa[3], *pb[3];
#pragma unroll
      for (int s = 0; s < 3; s++) {
        if (s < a.nseg) {
          const SegDev &q = a.seg[s];
          const int ia = q.idx ? __ldg(q.idx + la) : la, ib = q.idx ? __ldg(q.idx + lb) : lb;
          pa[s] = q.src + (size_t)ia * q.ld + 2 * t;
          pb[s] = q.src + (size_t)ib * q.ld + 2 * t;
        }
      }
      int kb = 0;
#pragma unroll
      for (int s = 0; s < 3; s++) {
        if (s >= a.nseg) break;
        const int w = a.seg[s].width;
        for (int c = 0; c < w; c += 64) {
          float2 x[4][4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (c + 16 * q < w) {
              x[q][0] = *reinterpret_cast<const float2 *>(pa[s] + c + 16 * q);
              x[q][1] = *reinterpret_cast<const float2 *>(pb[s] + c + 16 * q);
              x[q][2] = *reinterpret_cast<const float2 *>(pa[s] + c + 16 * q + 8);
              x[q][3] = *reinterpret_cast<const float2 *>(pb[s] + c + 16 * q + 8);
            }
          }
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (c + 16 * q >= w) break;
            uint32_t af[4];
#pragma unroll
            for (int i = 0; i < 4; i++) af[i] = bf2(x[q][i].x, x[q][i].y);
#pragma unroll
            for (int np = 0; np < 4; np++) {
              uint32_t b4[4];
              frag_b2(sW1, LDX, np * 16, kb + c + 16 * q, lane, b4);
              mma16816(acc[2 * np], af, b4);
              mma16816(acc[2 * np + 1], af, b4 + 2);
            }
          }
        }
        kb += w;
      }
    } else {
      for (int k0 = 0; k0 < Kp; k0 += 16) {
        uint32_t af[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int row = (i & 1) ? lb : la, k = k0 + 2 * t + (i >> 1) * 8;
          const float lo = k < a.K ? seg_value(a.seg, a.nseg, row, k) : 0.0f;
          const float hi = k + 1 < a.K ? seg_value(a.seg, a.nseg, row, k + 1) : 0.0f;
          af[i] = bf2(lo, hi);
        }
#pragma unroll
        for (int np = 0; np < 4; np++) {
          uint32_t b4[4];
          frag_b2(sW1, LDX, np * 16, k0, lane, b4);
          mma16816(acc[2 * np], af, b4);
          mma16816(acc[2 * np + 1], af, b4 + 2);
        }
      }
    }
    // Hidden layer: bias, z1, and silu(z1) packed as the A fragments of the second product (the
    // accumulator layout of column tiles 2j, 2j+1 is the fragment layout of columns [16 j, 16 j + 16)).
    uint32_t hf[4][4];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
      const int col = nt * 8 + 2 * t;
      const float2 b1 = make_float2(__ldg(a.b1 + col), __ldg(a.b1 + col + 1));
      const float z00 = acc[nt][0] + b1.x, z01 = acc[nt][1] + b1.y, z10 = acc[nt][2] + b1.x, z11 = acc[nt][3] + b1.y;
      if (a.z1) {
        if (ra < a.M) *reinterpret_cast<float2 *>(a.z1 + (size_t)ra * HID + col) = make_float2(z00, z01);
        if (rb < a.M) *reinterpret_cast<float2 *>(a.z1 + (size_t)rb * HID + col) = make_float2(z10, z11);
      }
      hf[nt >> 1][(nt & 1) * 2] = bf2(silu_f(z00), silu_f(z01));
      hf[nt >> 1][(nt & 1) * 2 + 1] = bf2(silu_f(z10), silu_f(z11));
    }
#pragma unroll
    for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
      for (int np = 0; np < 4; np++) {
        if (np * 16 < N2p) {
          uint32_t b4[4];
          frag_b2(sW2, LDH, np * 16, j * 16, lane, b4);
          mma16816(acc[2 * np], hf[j], b4);
          mma16816(acc[2 * np + 1], hf[j], b4 + 2);
        }
      }
    }
    if (a.vec_y) {  // 64 columns, even leading dimensions, 8-byte aligned rows
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int row = h ? rb : ra;
        if (row >= a.M) continue;
        float2 r[8];
        if (a.resid) {
#pragma unroll
          for (int nt = 0; nt < 8; nt++)
            r[nt] = *reinterpret_cast<const float2 *>(a.resid + (size_t)row * a.ld_resid + nt * 8 + 2 * t);
        }
#pragma unroll
        for (int nt = 0; nt < 8; nt++) {
          const int col = nt * 8 + 2 * t;
          float v0 = acc[nt][2 * h] + __ldg(a.b2 + col), v1 = acc[nt][2 * h + 1] + __ldg(a.b2 + col + 1);
          if (a.resid) {
            v0 += r[nt].x;
            v1 += r[nt].y;
          }
          *reinterpret_cast<float2 *>(a.y + (size_t)row * a.ld_y + col) = make_float2(v0, v1);
        }
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < 8; nt++) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int row = (q & 2) ? rb : ra, c = nt * 8 + 2 * t + (q & 1);
          if (row >= a.M || c >= a.N2) continue;
          float v = acc[nt][q] + a.b2[c];
          if (a.resid) v += a.resid[(size_t)row * a.ld_resid + c];
          a.y[(size_t)row * a.ld_y + c] = v;
        }
      }
    }
  }
}

// ---- The forward block on the 5th-generation tensor cores (tcgen05) ----
// One CTA of 128 threads per 128-row tile (persistent over tiles): the input rows and the
// weights are staged in shared memory as BF16 in the K-major, no-swizzle canonical layout of the
// tcgen05 matrix descriptors (8-row x 16-byte core matrices, consecutive rows 16 bytes apart,
// row groups SBO = 128 bytes apart, 8-column chunks LBO = rows x 16 bytes apart); one elected
// thread issues the M = 128 MMAs (kind::f16, BF16 operands, FP32 accumulators in tensor memory)
// and commits them to an mbarrier; each warp reads its 32 rows of the accumulator with
// tcgen05.ld, applies bias and SiLU in FP32, writes the hidden layer back to shared memory as the
// A operand of the second MMA, and so on.  The results equal the mma.sync kernel's up to the FP32
// summation order.  Every mbarrier wait is bounded; a wait that runs out records an error in
// g_tc_status (read by cfd_mpnn_status), and the CTA releases its tensor memory and returns.
constexpr int TM_TC = 128;
constexpr long long kTcSpin = 1ll << 22;
__device__ int g_tc_status = 0;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// Byte offset of element (row, k) of a rows x K tile in the canonical K-major layout.
__device__ __forceinline__ uint32_t canon_off(int row, int k, int rows) {
  return (uint32_t)((((k >> 3) * (rows >> 3) + (row >> 3)) << 7) + ((row & 7) << 4) + ((k & 7) << 1));
}
// Shared-memory matrix descriptor: start address, LBO and SBO in 16-byte units, version 1,
// no swizzle.
__device__ __forceinline__ uint64_t make_sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N.
__host__ __device__ constexpr uint32_t make_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  for (long long i = 0; i < kTcSpin; i++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    __nanosleep(64);
  }
  return false;
}
// 16 consecutive FP32 accumulator columns of this thread's row.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__global__ void __launch_bounds__(128) k_mlp_fwd_tc(FwdArgs a) {
  extern __shared__ __align__(1024) uint8_t smb[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  const int Kp = (a.K + 15) & ~15, N2p = a.N2 <= 16 ? 16 : 64;
  uint8_t *sX = smb;                                  // [128 x Kp]  input rows
  uint8_t *sW1 = sX + (size_t)TM_TC * Kp * 2;         // [64 x Kp]   W1
  uint8_t *sS = sW1 + (size_t)HID * Kp * 2;           // [128 x 64]  silu(z1)
  uint8_t *sW2 = sS + (size_t)TM_TC * HID * 2;        // [N2p x 64]  W2
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int e = tid; e < HID * Kp; e += blockDim.x) {
    const int n = e / Kp, k = e - n * Kp;
    *reinterpret_cast<uint16_t *>(sW1 + canon_off(n, k, HID)) = k < a.K ? bf(a.w1[n * a.K + k]) : 0;
  }
  for (int e = tid; e < N2p * HID; e += blockDim.x) {
    const int n = e / HID, k = e - n * HID;
    *reinterpret_cast<uint16_t *>(sW2 + canon_off(n, k, N2p)) = n < a.N2 ? bf(a.w2[n * HID + k]) : 0;
  }
  const uint32_t bar_a = smem_u32(&bar);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(128));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a));
    abort_sh = 0;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_sh;
  const uint32_t d1 = tmem, d2 = tmem + 64;
  const uint32_t lane_base = (uint32_t)(32 * warp) << 16;
  const uint32_t idesc1 = make_idesc(TM_TC, HID), idesc2 = make_idesc(TM_TC, N2p);
  uint32_t parity = 0;
  const int ntiles = (a.M + TM_TC - 1) / TM_TC;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int r0 = tile * TM_TC;
    for (int e = tid; e < TM_TC * Kp; e += blockDim.x) {
      const int r = e / Kp, k = e - r * Kp, row = r0 + r;
      *reinterpret_cast<uint16_t *>(sX + canon_off(r, k, TM_TC)) =
          (row < a.M && k < a.K) ? bf(seg_value(a.seg, a.nseg, row, k)) : 0;
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t xa = smem_u32(sX), wa = smem_u32(sW1);
      for (int k0 = 0; k0 < Kp; k0 += 16) {
        const uint64_t da = make_sdesc(xa + (uint32_t)((k0 >> 3) * (TM_TC >> 3) * 128), TM_TC * 16, 128);
        const uint64_t db = make_sdesc(wa + (uint32_t)((k0 >> 3) * (HID >> 3) * 128), HID * 16, 128);
        tc_mma(d1, da, db, idesc1, k0 > 0 ? 1u : 0u);
      }
      tc_commit(bar_a);
    }
    if (!mbar_wait(bar_a, parity)) {
      if (tid == 0) atomicExch(&g_tc_status, 5 /* CFD_ERR_TIMEOUT */);
      abort_sh = 1;
    }
    parity ^= 1u;
    __syncthreads();
    if (abort_sh) break;
    tc_fence_after();
    const int r = 32 * warp + (tid & 31), row = r0 + r;
#pragma unroll
    for (int c0 = 0; c0 < HID; c0 += 16) {
      float v[16];
      tmem_ld16(d1 + lane_base + c0, v);
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const float z = v[j] + a.b1[c0 + j];
        if (a.z1 && row < a.M) a.z1[(size_t)row * HID + c0 + j] = z;
        *reinterpret_cast<uint16_t *>(sS + canon_off(r, c0 + j, TM_TC)) = bf(silu_f(z));
      }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t sa = smem_u32(sS), wa = smem_u32(sW2);
      for (int k0 = 0; k0 < HID; k0 += 16) {
        const uint64_t da = make_sdesc(sa + (uint32_t)((k0 >> 3) * (TM_TC >> 3) * 128), TM_TC * 16, 128);
        const uint64_t db = make_sdesc(wa + (uint32_t)((k0 >> 3) * (N2p >> 3) * 128), N2p * 16, 128);
        tc_mma(d2, da, db, idesc2, k0 > 0 ? 1u : 0u);
      }
      tc_commit(bar_a);
    }
    if (!mbar_wait(bar_a, parity)) {
      if (tid == 0) atomicExch(&g_tc_status, 5);
      abort_sh = 1;
    }
    parity ^= 1u;
    __syncthreads();
    if (abort_sh) break;
    tc_fence_after();
    for (int c0 = 0; c0 < N2p; c0 += 16) {
      float v[16];
      tmem_ld16(d2 + lane_base + c0, v);
      if (row < a.M) {
#pragma unroll
        for (int j = 0; j < 16; j++) {
          const int c = c0 + j;
          if (c >= a.N2) continue;
          float y = v[j] + a.b2[c];
          if (a.resid) y += a.resid[(size_t)row * a.ld_resid + c];
          a.y[(size_t)row * a.ld_y + c] = y;
        }
      }
    }
    tc_fence_before();
    __syncthreads();
  }
  // After a timed-out wait the MMAs may still be in flight: wait for them (bounded) before the
  // tensor memory is released.
  if (abort_sh) mbar_wait(bar_a, parity);
  tc_fence_after();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128));
}

struct BwdArgs {
  int M, K, N2;
  const float *dy;
  int ld_dy;
  const float *z1, *w1, *w2;
  float *dz1, *dx;
  int ld_dx;
  // mma.sync form only.  ga: rows added to dy through a row map, dy'[r] = dy[r] + ga[gidx[r]].
  // upd: columns [upd_c0, upd_c0 + 64) of dx go to upd[r] = dy'[r] + dx[r][upd_c0 ..] instead of
  // dx (the residual path of a block; upd may be dy itself: a lane reads its elements of dy before
  // it writes the same elements of upd).
  const float *ga;
  int ld_ga;
  const int *gidx;
  float *upd;
  int ld_upd, upd_c0;
  int vec_dx;  // dx in 8-byte pieces
};

// One warp per 16 rows, the structure of k_mlp_fwd: dY rows from global memory into the A fragments,
// dz1 from the accumulators of the first product to the A fragments of the second in registers.
// Both weight matrices are B operands as stored ([k][n]), read with transposing ldmatrix.  VEC: 64
// output columns and 8-byte aligned rows of every array.
template <bool VEC>
__global__ void __launch_bounds__(kMlpThreads, 2) k_mlp_bwd(BwdArgs a) {
  extern __shared__ __align__(16) uint16_t sm[];
  const int Kp = (a.K + 15) & ~15, LDX = Kp + 8, N2p = (a.N2 + 15) & ~15;
  uint16_t *sW1 = sm;               // [HID][LDX]   W1: B operand of dX = dZ1 W1
  uint16_t *sW2 = sW1 + HID * LDX;  // [N2p][LDH]   W2: B operand of dS = dY W2
  stage_weights(a.w1, HID, a.K, sW1, HID, Kp, LDX);
  stage_weights(a.w2, a.N2, HID, sW2, N2p, HID, LDH);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ntiles = (a.M + 15) >> 4;
  for (int tile = blockIdx.x * kMlpWarps + warp; tile < ntiles; tile += gridDim.x * kMlpWarps) {
    const int ra = tile * 16 + g, rb = ra + 8;
    const int la = min(ra, a.M - 1), lb = min(rb, a.M - 1);
    const float *ya = a.dy + (size_t)la * a.ld_dy + 2 * t, *yb = a.dy + (size_t)lb * a.ld_dy + 2 * t;
    const float *ga = nullptr, *gb = nullptr;
    if (VEC && a.ga) {
      ga = a.ga + (size_t)__ldg(a.gidx + la) * a.ld_ga + 2 * t;
      gb = a.ga + (size_t)__ldg(a.gidx + lb) * a.ld_ga + 2 * t;
    }
    uint32_t yf[4][4];
    if (VEC) {
      float2 y[4][4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        y[q][0] = *reinterpret_cast<const float2 *>(ya + 16 * q);
        y[q][1] = *reinterpret_cast<const float2 *>(yb + 16 * q);
        y[q][2] = *reinterpret_cast<const float2 *>(ya + 16 * q + 8);
        y[q][3] = *reinterpret_cast<const float2 *>(yb + 16 * q + 8);
      }
      if (ga) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const float2 v = *reinterpret_cast<const float2 *>(((i & 1) ? gb : ga) + 16 * q + (i >> 1) * 8);
            y[q][i].x += v.x;
            y[q][i].y += v.y;
          }
      }
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 4; i++) yf[q][i] = bf2(y[q][i].x, y[q][i].y);
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float *p = (i & 1) ? yb : ya;
          const int k = 16 * q + (i >> 1) * 8;
          yf[q][i] = bf2(k + 2 * t < a.N2 ? p[k] : 0.0f, k + 2 * t + 1 < a.N2 ? p[k + 1] : 0.0f);
        }
    }
    float2 z[8][2];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
      z[nt][0] = *reinterpret_cast<const float2 *>(a.z1 + (size_t)la * HID + nt * 8 + 2 * t);
      z[nt][1] = *reinterpret_cast<const float2 *>(a.z1 + (size_t)lb * HID + nt * 8 + 2 * t);
    }
    float acc[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (16 * q >= N2p) break;
#pragma unroll
      for (int np = 0; np < 4; np++) {
        uint32_t b4[4];
        frag_b2t(sW2, LDH, np * 16, 16 * q, lane, b4);
        mma16816(acc[2 * np], yf[q], b4);
        mma16816(acc[2 * np + 1], yf[q], b4 + 2);
      }
    }
    uint32_t zf[4][4];
#pragma unroll
    for (int nt = 0; nt < 8; nt++) {
      const int col = nt * 8 + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int row = h ? rb : ra;
        const float d0 = acc[nt][2 * h] * dsilu_f(z[nt][h].x), d1 = acc[nt][2 * h + 1] * dsilu_f(z[nt][h].y);
        if (row < a.M) *reinterpret_cast<float2 *>(a.dz1 + (size_t)row * HID + col) = make_float2(d0, d1);
        zf[nt >> 1][(nt & 1) * 2 + h] = bf2(d0, d1);
      }
    }
    if (!a.dx && !a.upd) continue;
    for (int c0 = 0; c0 < Kp; c0 += 64) {
#pragma unroll
      for (int nt = 0; nt < 8; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
#pragma unroll
      for (int j = 0; j < 4; j++) {
#pragma unroll
        for (int np = 0; np < 4; np++) {
          if (c0 + np * 16 < Kp) {
            uint32_t b4[4];
            frag_b2t(sW1, LDX, c0 + np * 16, j * 16, lane, b4);
            mma16816(acc[2 * np], zf[j], b4);
            mma16816(acc[2 * np + 1], zf[j], b4 + 2);
          }
        }
      }
      if (VEC && a.upd && c0 == a.upd_c0) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int row = h ? rb : ra;
          if (row >= a.M) continue;
          float2 v[8];
#pragma unroll
          for (int nt = 0; nt < 8; nt++) v[nt] = *reinterpret_cast<const float2 *>((h ? yb : ya) + nt * 8);
          if (ga) {
#pragma unroll
            for (int nt = 0; nt < 8; nt++) {
              const float2 w = *reinterpret_cast<const float2 *>((h ? gb : ga) + nt * 8);
              v[nt].x += w.x;
              v[nt].y += w.y;
            }
          }
#pragma unroll
          for (int nt = 0; nt < 8; nt++)
            *reinterpret_cast<float2 *>(a.upd + (size_t)row * a.ld_upd + nt * 8 + 2 * t) =
                make_float2(v[nt].x + acc[nt][2 * h], v[nt].y + acc[nt][2 * h + 1]);
        }
        continue;
      }
#pragma unroll
      for (int nt = 0; nt < 8; nt++) {
        const int col = c0 + nt * 8 + 2 * t;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int row = h ? rb : ra;
          if (row >= a.M) continue;
          float *o = a.dx + (size_t)row * a.ld_dx + col;
          if (a.vec_dx && col + 1 < a.K) {
            *reinterpret_cast<float2 *>(o) = make_float2(acc[nt][2 * h], acc[nt][2 * h + 1]);
          } else {
            if (col < a.K) o[0] = acc[nt][2 * h];
            if (col + 1 < a.K) o[1] = acc[nt][2 * h + 1];
          }
        }
      }
    }
  }
}

// The backward data path on the tensor cores: dS = dY W2 (M = 128 rows, N = 64, K = the block's
// output width rounded up to 16), dz1 = dS * silu'(z1), dX = dz1 W1 (N = the input width rounded up
// to 16, K = 64), the same two-MMA chain as the forward with the transposed weights as the B
// operands: W2^T as (n = 64, k = out) and W1^T as (n = in, k = 64), all BF16 in the canonical
// K-major layout, FP32 accumulators in 64 + in columns of tensor memory.  BF16 rounding of dY, the
// weights and dz1 as in k_mlp_bwd, so the results agree up to the FP32 summation order.
__global__ void __launch_bounds__(128) k_mlp_bwd_tc(BwdArgs a) {
  extern __shared__ __align__(1024) uint8_t smb[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  const int Kp = (a.K + 15) & ~15, N2p = (a.N2 + 15) & ~15;
  uint8_t *sDY = smb;                                 // [128 x N2p]  dY rows
  uint8_t *sW2T = sDY + (size_t)TM_TC * N2p * 2;      // [64 x N2p]   W2^T
  uint8_t *sDZ = sW2T + (size_t)HID * N2p * 2;        // [128 x 64]   dz1
  uint8_t *sW1T = sDZ + (size_t)TM_TC * HID * 2;      // [Kp x 64]    W1^T
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int e = tid; e < HID * N2p; e += blockDim.x) {
    const int n = e / N2p, k = e - n * N2p;  // B(n, k) = W2[k][n]
    *reinterpret_cast<uint16_t *>(sW2T + canon_off(n, k, HID)) = k < a.N2 ? bf(a.w2[k * HID + n]) : 0;
  }
  for (int e = tid; e < Kp * HID; e += blockDim.x) {
    const int n = e / HID, k = e - n * HID;  // B(n, k) = W1[k][n]
    *reinterpret_cast<uint16_t *>(sW1T + canon_off(n, k, Kp)) = n < a.K ? bf(a.w1[k * a.K + n]) : 0;
  }
  const uint32_t bar_a = smem_u32(&bar);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a));
    abort_sh = 0;
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_sh;
  const uint32_t d1 = tmem, d2 = tmem + 64;
  const uint32_t lane_base = (uint32_t)(32 * warp) << 16;
  const uint32_t idesc1 = make_idesc(TM_TC, HID), idesc2 = make_idesc(TM_TC, Kp);
  uint32_t parity = 0;
  const int ntiles = (a.M + TM_TC - 1) / TM_TC;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int r0 = tile * TM_TC;
    for (int e = tid; e < TM_TC * N2p; e += blockDim.x) {
      const int r = e / N2p, k = e - r * N2p, row = r0 + r;
      *reinterpret_cast<uint16_t *>(sDY + canon_off(r, k, TM_TC)) =
          (row < a.M && k < a.N2) ? bf(a.dy[(size_t)row * a.ld_dy + k]) : 0;
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t ya = smem_u32(sDY), wa = smem_u32(sW2T);
      for (int k0 = 0; k0 < N2p; k0 += 16) {
        const uint64_t da = make_sdesc(ya + (uint32_t)((k0 >> 3) * (TM_TC >> 3) * 128), TM_TC * 16, 128);
        const uint64_t db = make_sdesc(wa + (uint32_t)((k0 >> 3) * (HID >> 3) * 128), HID * 16, 128);
        tc_mma(d1, da, db, idesc1, k0 > 0 ? 1u : 0u);
      }
      tc_commit(bar_a);
    }
    if (!mbar_wait(bar_a, parity)) {
      if (tid == 0) atomicExch(&g_tc_status, 5 /* CFD_ERR_TIMEOUT */);
      abort_sh = 1;
    }
    parity ^= 1u;
    __syncthreads();
    if (abort_sh) break;
    tc_fence_after();
    const int r = 32 * warp + (tid & 31), row = r0 + r;
#pragma unroll
    for (int c0 = 0; c0 < HID; c0 += 16) {
      float v[16];
      tmem_ld16(d1 + lane_base + c0, v);
#pragma unroll
      for (int j = 0; j < 16; j++) {
        float d = 0.0f;
        if (row < a.M) {
          d = v[j] * dsilu_f(a.z1[(size_t)row * HID + c0 + j]);
          a.dz1[(size_t)row * HID + c0 + j] = d;
        }
        *reinterpret_cast<uint16_t *>(sDZ + canon_off(r, c0 + j, TM_TC)) = bf(d);
      }
    }
    if (a.dx) {
      fence_async_smem();
      tc_fence_before();
      __syncthreads();
      if (tid == 0) {
        tc_fence_after();
        const uint32_t za = smem_u32(sDZ), wa = smem_u32(sW1T);
        for (int k0 = 0; k0 < HID; k0 += 16) {
          const uint64_t da = make_sdesc(za + (uint32_t)((k0 >> 3) * (TM_TC >> 3) * 128), TM_TC * 16, 128);
          const uint64_t db = make_sdesc(wa + (uint32_t)((k0 >> 3) * (Kp >> 3) * 128), Kp * 16, 128);
          tc_mma(d2, da, db, idesc2, k0 > 0 ? 1u : 0u);
        }
        tc_commit(bar_a);
      }
      if (!mbar_wait(bar_a, parity)) {
        if (tid == 0) atomicExch(&g_tc_status, 5);
        abort_sh = 1;
      }
      parity ^= 1u;
      __syncthreads();
      if (abort_sh) break;
      tc_fence_after();
      for (int c0 = 0; c0 < Kp; c0 += 16) {
        float v[16];
        tmem_ld16(d2 + lane_base + c0, v);
        if (row < a.M) {
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const int c = c0 + j;
            if (c < a.K) a.dx[(size_t)row * a.ld_dx + c] = v[j];
          }
        }
      }
    }
    tc_fence_before();
    __syncthreads();
  }
  // After a timed-out wait the MMAs may still be in flight: wait for them (bounded) before the
  // tensor memory is released.
  if (abort_sh) mbar_wait(bar_a, parity);
  tc_fence_after();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

struct WgArgs {
  int M, N, K, nseg;
  SegDev seg[3];
  const float *dz;
  int ld_dz;
  float *partial;  // [gridDim.x][N*K + N]
  const float *ga;  // optional rows added to dz through a row map (as in BwdArgs)
  int ld_ga;
  const int *gidx;
};

constexpr int kWgThreads = 256;

// dW[n][c] = sum over rows of dz[row][n] x[row][c] as D = A B with A = dz^T (N x TM) and
// B = x (TM x K).  A 64-row tile of dz and x is staged as BF16 rows (16-byte loads, four or eight in
// flight per lane) and read with transposing ldmatrix, so neither operand is transposed by hand;
// db is summed from an FP32 copy of the dz tile, row after row.  MT = number of 16-row tiles of N
// (1 or 4); the eight warps split the N tiles and the pairs of 8-column tiles of K between them.
// Two blocks share an SM, one staging while the other multiplies.  The sums run over the same tiles
// in the same order for every block count in use: tile i belongs to block i mod gridDim.x.
// VEC: every segment's width is a multiple of 16 and its rows (and dz's, N = 64) are 16-byte aligned.
template <int MT, bool VEC>
__global__ void __launch_bounds__(kWgThreads, 2) k_wgrad(WgArgs a) {
  extern __shared__ __align__(16) uint16_t sm[];
  constexpr int Np = MT * 16, LDZ = Np + 8;
  constexpr int WPM = 8 / MT;                        // warps per N tile
  constexpr int NPW = (KMAX / 16 + WPM - 1) / WPM;   // K tile pairs per warp, at most
  const int Kp = (a.K + 15) & ~15, LDX = Kp + 8;
  uint16_t *sZ = sm;                                           // [TM][LDZ]
  uint16_t *sX = sZ + TM * LDZ;                                // [TM][LDX]
  float *sF = reinterpret_cast<float *>(sX + TM * LDX);        // [TM][Np]   dz in FP32 (for db)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int mrow = (warp % MT) * 16, pair0 = warp / MT;
  const int npair = Kp / 16;
  float acc[NPW][2][4];
#pragma unroll
  for (int i = 0; i < NPW; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;
  float bsum = 0.0f;
  const int ntiles = (a.M + TM - 1) / TM;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int r0 = tile * TM;
    __syncthreads();
    if (VEC) {
      // A half warp reads 64 columns of one row; each lane takes rows hw, hw + 16, hw + 32, hw + 48.
      const int hw = threadIdx.x >> 4, c4 = (threadIdx.x & 15) * 4;
      float4 v[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int row = r0 + hw + 16 * i;
        v[i] = row < a.M ? *reinterpret_cast<const float4 *>(a.dz + (size_t)row * a.ld_dz + c4) : make_float4(0, 0, 0, 0);
        if (a.ga)
          w[i] = row < a.M ? *reinterpret_cast<const float4 *>(a.ga + (size_t)__ldg(a.gidx + row) * a.ld_ga + c4)
                           : make_float4(0, 0, 0, 0);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int m = hw + 16 * i;
        if (a.ga) {
          v[i].x += w[i].x;
          v[i].y += w[i].y;
          v[i].z += w[i].z;
          v[i].w += w[i].w;
        }
        *reinterpret_cast<float4 *>(sF + m * Np + c4) = v[i];
        *reinterpret_cast<uint2 *>(sZ + m * LDZ + c4) = make_uint2(bf2(v[i].x, v[i].y), bf2(v[i].z, v[i].w));
      }
      int cb = 0;
#pragma unroll
      for (int s = 0; s < 3; s++) {
        if (s >= a.nseg) break;
        const SegDev &q = a.seg[s];
        int src_row[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int row = r0 + hw + 16 * i;
          src_row[i] = row < a.M ? (q.idx ? __ldg(q.idx + row) : row) : -1;
        }
        for (int c = c4; c < q.width; c += 64) {
#pragma unroll
          for (int i = 0; i < 4; i++)
            v[i] = src_row[i] >= 0 ? *reinterpret_cast<const float4 *>(q.src + (size_t)src_row[i] * q.ld + c)
                                   : make_float4(0, 0, 0, 0);
          if (q.silu) {
#pragma unroll
            for (int i = 0; i < 4; i++)
              v[i] = make_float4(silu_f(v[i].x), silu_f(v[i].y), silu_f(v[i].z), silu_f(v[i].w));
          }
#pragma unroll
          for (int i = 0; i < 4; i++)
            *reinterpret_cast<uint2 *>(sX + (hw + 16 * i) * LDX + cb + c) =
                make_uint2(bf2(v[i].x, v[i].y), bf2(v[i].z, v[i].w));
        }
        cb += q.width;
      }
    } else {
      for (int e = threadIdx.x; e < TM * Np; e += kWgThreads) {
        const int m = e / Np, n = e - m * Np, row = r0 + m;
        const float v = (row < a.M && n < a.N) ? a.dz[(size_t)row * a.ld_dz + n] : 0.0f;
        sF[m * Np + n] = v;
        sZ[m * LDZ + n] = bf(v);
      }
      for (int e = threadIdx.x; e < TM * Kp; e += kWgThreads) {
        const int m = e / Kp, c = e - m * Kp, row = r0 + m;
        sX[m * LDX + c] = (row < a.M && c < a.K) ? bf(seg_value(a.seg, a.nseg, row, c)) : 0;
      }
    }
    __syncthreads();
    if (threadIdx.x < a.N) {
      const int rend = min(TM, a.M - r0);
      if (rend == TM) {
#pragma unroll 16
        for (int m = 0; m < TM; m++) bsum += sF[m * Np + threadIdx.x];
      } else {
        for (int m = 0; m < rend; m++) bsum += sF[m * Np + threadIdx.x];
      }
    }
#pragma unroll
    for (int k0 = 0; k0 < TM; k0 += 16) {
      uint32_t af[4];
      frag_at(sZ, LDZ, mrow, k0, lane, af);
#pragma unroll
      for (int i = 0; i < NPW; i++) {
        const int p = pair0 + i * WPM;
        if (p < npair) {
          uint32_t b4[4];
          frag_b2t(sX, LDX, p * 16, k0, lane, b4);
          mma16816(acc[i][0], af, b4);
          mma16816(acc[i][1], af, b4 + 2);
        }
      }
    }
  }
  float *out = a.partial + (size_t)blockIdx.x * (a.N * a.K + a.N);
#pragma unroll
  for (int i = 0; i < NPW; i++) {
    const int p = pair0 + i * WPM;
    if (p >= npair) continue;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int c = p * 16 + j * 8 + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int n = mrow + g + 8 * h;
        if (n >= a.N) continue;
        if (c < a.K) out[n * a.K + c] = acc[i][j][2 * h];
        if (c + 1 < a.K) out[n * a.K + c + 1] = acc[i][j][2 * h + 1];
      }
    }
  }
  if (threadIdx.x < a.N) out[a.N * a.K + threadIdx.x] = bsum;
}

// dw[j] (j < N*K) and db[j] (j < N) from the per-block partials, summed in block order.  A block
// takes 32 columns: its eight warps bring all partials of those columns into shared memory (up to
// 37 independent loads per lane), then one warp adds them in order, so the serial sum waits on
// shared memory and not on L2.
constexpr int kRedCols = 32;
__global__ void __launch_bounds__(256) k_wgrad_reduce(const float *__restrict__ partial, int nblk, int N, int K,
                                                      float *__restrict__ dw, float *__restrict__ db, int accumulate) {
  __shared__ float sh[CFD_MPNN_WGRAD_BLOCKS][kRedCols];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * kRedCols + lane;
  const int stride = N * K + N;
  const float *p = partial + min(j, stride - 1);
#pragma unroll 16
  for (int b = w; b < nblk; b += 8) sh[b][lane] = __ldg(p + (size_t)b * stride);
  __syncthreads();
  if (w > 0 || j >= stride) return;
  float s = 0.0f;
#pragma unroll 16
  for (int b = 0; b < nblk; b++) s += sh[b][lane];
  float *o = j < N * K ? dw + j : db + (j - N * K);
  *o = accumulate ? *o + s : s;
}

// out[r][j] = a[r][j] + b[r][j] (j < width; leading dimensions given).
__global__ void k_add(float *out, int ldo, const float *a, int lda, const float *b, int ldb, int rows, int width) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)rows * width) return;
  const int r = (int)(e / width), j = (int)(e - (size_t)r * width);
  out[(size_t)r * ldo + j] = a[(size_t)r * lda + j] + b[(size_t)r * ldb + j];
}

// out[r][j] += src[idx[r]][j].
__global__ void k_gather_add(float *out, int ldo, const float *src, int lds, const int *idx, int rows, int width) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)rows * width) return;
  const int r = (int)(e / width), j = (int)(e - (size_t)r * width);
  out[(size_t)r * ldo + j] += src[(size_t)idx[r] * lds + j];
}

// out[r][:] (+)= sum over j in [ptr[r], ptr[r+1]) of x[idx[j]][:], in list order (warp per row).
__global__ void k_segment_sum_acc(const float *__restrict__ x, int ldx, const int *__restrict__ ptr,
                                  const int *__restrict__ idx, int n_rows, int width, float *__restrict__ out, int ldo,
                                  int accumulate) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const int b = ptr[row], e = ptr[row + 1];
  for (int col = lane; col < width; col += 32) {
    float acc = 0.f;
    for (int j = b; j < e; j++) acc += x[(size_t)idx[j] * ldx + col];
    float *o = out + (size_t)row * ldo + col;
    *o = accumulate ? *o + acc : acc;
  }
}

// The same for 64 columns in 8-byte aligned rows: a warp per row, two columns per lane, the list's
// rows loaded four at a time ahead of the additions (which stay in list order).  idx null: the
// list of row r is the rows ptr[r] .. ptr[r+1] themselves.
__device__ __forceinline__ float2 list_sum64(const float *x, int ldx, const int *idx, int b, int e, int lane) {
  float2 acc = make_float2(0.f, 0.f);
  for (int j = b; j < e; j += 4) {
    float2 v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (j + i < e) {
        const int r = idx ? __ldg(idx + j + i) : j + i;
        v[i] = *reinterpret_cast<const float2 *>(x + (size_t)r * ldx + 2 * lane);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (j + i < e) {
        acc.x += v[i].x;
        acc.y += v[i].y;
      }
    }
  }
  return acc;
}

__global__ void __launch_bounds__(256) k_segment_sum64(const float *__restrict__ x, int ldx, const int *__restrict__ ptr,
                                                       const int *__restrict__ idx, int n_rows, float *out, int ldo,
                                                       int accumulate) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  float2 s = list_sum64(x, ldx, idx, __ldg(ptr + row), __ldg(ptr + row + 1), lane);
  float2 *o = reinterpret_cast<float2 *>(out + (size_t)row * ldo + 2 * lane);
  if (accumulate) {
    const float2 v = *o;
    s = make_float2(v.x + s.x, v.y + s.y);
  }
  *o = s;
}

// Backward of the two row gathers of an edge block: out[r] = (out[r] + sum over the edges leaving r of
// dx[.][0, 64)) + sum over the edges entering r (consecutive rows) of dx[.][64, 128).
__global__ void __launch_bounds__(256) k_edge_gather_bwd(const float *__restrict__ dx, int ldx,
                                                         const int *__restrict__ src_ptr,
                                                         const int *__restrict__ src_order,
                                                         const int *__restrict__ dst_ptr, int n_rows, float *out) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const float2 a = list_sum64(dx, ldx, src_order, __ldg(src_ptr + row), __ldg(src_ptr + row + 1), lane);
  const float2 b = list_sum64(dx + HID, ldx, nullptr, __ldg(dst_ptr + row), __ldg(dst_ptr + row + 1), lane);
  float2 *o = reinterpret_cast<float2 *>(out + (size_t)row * HID + 2 * lane);
  const float2 v = *o;
  *o = make_float2((v.x + a.x) + b.x, (v.y + a.y) + b.y);
}

// Mean-squared error: grad = 2 (pred - target) / n and loss = sum (pred - target)^2 / n.  Block 0 sums
// the loss (each thread its stride of values, eight loads ahead of the additions, then a fixed-order
// tree); the other blocks write the gradient.  A gradient written over its inputs (in_place) is block 0's
// too, each value after its thread has read it.
__global__ void __launch_bounds__(1024) k_mse(const float *pred, const float *target, int n, float *grad, float *loss,
                                              bool in_place) {
  const float inv = 1.0f / (float)n;
  if (blockIdx.x > 0) {
    const long long i = (long long)(blockIdx.x - 1) * blockDim.x + threadIdx.x;
    if (i < n) {
      const float d = pred[i] - target[i];
      grad[i] = 2.0f * d * inv;
    }
    return;
  }
  __shared__ float sh[1024];
  float s = 0.0f;
  long long i = threadIdx.x;
  for (; !in_place && i + 7 * 1024 < n; i += 8 * 1024) {
    float d[8];
#pragma unroll
    for (int k = 0; k < 8; k++) d[k] = pred[i + k * 1024] - target[i + k * 1024];
#pragma unroll
    for (int k = 0; k < 8; k++) s += d[k] * d[k];
  }
  for (; i < n; i += 1024) {
    const float d = pred[i] - target[i];
    if (in_place) grad[i] = 2.0f * d * inv;
    s += d * d;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 512; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = sh[0] * inv;
}

cfd_status status_of(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return CFD_OK;
  cfdb::set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
  return CFD_ERR_CUDA;
}

cfd_status bad(const char *what) {
  cfdb::set_last_error(what);
  return CFD_ERR_BAD_ARG;
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

bool copy_segs(int nseg, const cfd_mlp_seg *in, SegDev *out, int &K) {
  if (nseg < 1 || nseg > 3) return false;
  K = 0;
  for (int s = 0; s < nseg; s++) {
    if (!in[s].src || in[s].width < 1 || in[s].ld < in[s].width) return false;
    out[s] = SegDev{in[s].src, in[s].idx, in[s].width, in[s].ld, in[s].silu};
    K += in[s].width;
  }
  for (int s = nseg; s < 3; s++) out[s] = SegDev{nullptr, nullptr, 0, 0, 0};
  return K <= KMAX;
}

size_t mlp_smem(int K, int N2) {  // the two weight matrices of k_mlp_fwd and k_mlp_bwd
  const int Kp = (K + 15) & ~15, N2p = (N2 + 15) & ~15;
  return sizeof(uint16_t) * ((size_t)HID * (Kp + 8) + (size_t)N2p * LDH);
}
size_t tc_smem(int K, int N2) {
  const int Kp = (K + 15) & ~15, N2p = N2 <= 16 ? 16 : 64;
  return 2 * ((size_t)TM_TC * Kp + (size_t)HID * Kp + (size_t)TM_TC * HID + (size_t)N2p * HID);
}
size_t bwd_tc_smem(int K, int N2) {
  const int Kp = (K + 15) & ~15, N2p = (N2 + 15) & ~15;
  return 2 * ((size_t)TM_TC * N2p + (size_t)HID * N2p + (size_t)TM_TC * HID + (size_t)Kp * HID);
}
size_t wg_smem(int K, int MT) {
  const int Kp = (K + 15) & ~15, Np = MT * 16;
  return sizeof(uint16_t) * ((size_t)TM * (Np + 8) + (size_t)TM * (Kp + 8)) + sizeof(float) * (size_t)TM * Np;
}
template <typename F>
void set_smem(F f, size_t bytes) {
  cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

bool aligned(const void *p, size_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; }

// Every segment of width a multiple of 16 in `bytes`-aligned rows (mma.sync kernels' vector forms).
bool segs_vector(const SegDev *seg, int nseg, size_t bytes, bool silu_ok) {
  for (int s = 0; s < nseg; s++)
    if ((seg[s].width & 15) || ((size_t)seg[s].ld * 4) % bytes || !aligned(seg[s].src, bytes) ||
        (seg[s].silu && !silu_ok))
      return false;
  return true;
}

// Two blocks of eight warps per SM, a warp per 16 rows.
int mlp_grid(int rows) {
  const int need = ((rows + 15) / 16 + kMlpWarps - 1) / kMlpWarps, most = 2 * sm_count();
  return need < most ? need : most;
}

void launch_mlp_fwd(FwdArgs &a, cudaStream_t s) {
  a.vec_y = a.N2 == HID && (a.ld_y & 1) == 0 && aligned(a.y, 8) &&
            (!a.resid || ((a.ld_resid & 1) == 0 && aligned(a.resid, 8)));
  const size_t sm = mlp_smem(a.K, a.N2);
  if (segs_vector(a.seg, a.nseg, 8, false)) {
    set_smem(k_mlp_fwd<true>, sm);
    k_mlp_fwd<true><<<mlp_grid(a.M), kMlpThreads, sm, s>>>(a);
  } else {
    set_smem(k_mlp_fwd<false>, sm);
    k_mlp_fwd<false><<<mlp_grid(a.M), kMlpThreads, sm, s>>>(a);
  }
}

bool bwd_vector(const BwdArgs &a) { return a.N2 == HID && (a.ld_dy & 1) == 0 && aligned(a.dy, 8); }

void launch_mlp_bwd(BwdArgs &a, cudaStream_t s) {
  a.vec_dx = a.dx && (a.ld_dx & 1) == 0 && aligned(a.dx, 8);
  const size_t sm = mlp_smem(a.K, a.N2);
  if (bwd_vector(a)) {
    set_smem(k_mlp_bwd<true>, sm);
    k_mlp_bwd<true><<<mlp_grid(a.M), kMlpThreads, sm, s>>>(a);
  } else {
    set_smem(k_mlp_bwd<false>, sm);
    k_mlp_bwd<false><<<mlp_grid(a.M), kMlpThreads, sm, s>>>(a);
  }
}

void launch_wgrad(const WgArgs &a, float *dw, float *db, int accumulate, cudaStream_t s) {
  const int ntiles = (a.M + TM - 1) / TM;
  const int grid = ntiles < 1 ? 1 : (ntiles < CFD_MPNN_WGRAD_BLOCKS ? ntiles : CFD_MPNN_WGRAD_BLOCKS);
  const bool vec = a.N == HID && (a.ld_dz & 3) == 0 && aligned(a.dz, 16) && segs_vector(a.seg, a.nseg, 16, true);
  const size_t sm = wg_smem(a.K, a.N == HID ? 4 : 1);
  auto run = [&](auto k) {
    set_smem(k, sm);
    k<<<grid, kWgThreads, sm, s>>>(a);
  };
  if (a.N != HID) run(k_wgrad<1, false>);
  else if (vec) run(k_wgrad<4, true>);
  else run(k_wgrad<4, false>);
  const int total = a.N * a.K + a.N;
  k_wgrad_reduce<<<(total + kRedCols - 1) / kRedCols, 256, 0, s>>>(a.partial, grid, a.N, a.K, dw, db, accumulate);
}

void launch_segment_sum(const float *x, int ldx, const int *ptr, const int *idx, int n_rows, int width, float *out,
                        int ldo, int accumulate, cudaStream_t s) {
  const int g = (n_rows + 7) / 8;
  if (width == HID && (ldx & 1) == 0 && (ldo & 1) == 0 && aligned(x, 8) && aligned(out, 8))
    k_segment_sum64<<<g, 256, 0, s>>>(x, ldx, ptr, idx, n_rows, out, ldo, accumulate);
  else
    k_segment_sum_acc<<<g, 256, 0, s>>>(x, ldx, ptr, idx, n_rows, width, out, ldo, accumulate);
}

// ---- Whole-network passes (cfd_mpnn_net) ----
struct NetBlock {
  int K, N;
  size_t w1, b1, w2, b2;  // offsets into the parameter and gradient buffers
};

// Layout of the parameters (enc_n, enc_e, edge blocks, node blocks, dec) and of the activations.
struct NetLayout {
  int L;
  NetBlock enc_n, enc_e, dec;
  size_t edge0, node0, edge_sz, node_sz;  // first edge / node block and their strides
  size_t h, e, agg, z_enc_n, z_enc_e, z_edge, z_node, z_dec, dh, de, dagg, dx, dz, total;  // activation floats
  size_t nh, ne;                                                                     // one node / edge activation
  static NetBlock block(size_t &o, int K, int N) {
    NetBlock b{K, N, o, o + (size_t)HID * K, o + (size_t)HID * K + HID, 0};
    b.b2 = b.w2 + (size_t)N * HID;
    o = b.b2 + N;
    return b;
  }
  NetBlock at(size_t first, size_t stride, int l, int K) const {
    size_t o = first + (size_t)l * stride;
    return block(o, K, HID);
  }
  NetBlock edge(int l) const { return at(edge0, edge_sz, l, 3 * HID); }
  NetBlock node(int l) const { return at(node0, node_sz, l, 2 * HID); }
  NetLayout(int layers, int node_in, int edge_in, int out, int N, int E) : L(layers) {
    size_t o = 0;
    enc_n = block(o, node_in, HID);
    enc_e = block(o, edge_in, HID);
    edge0 = o;
    edge_sz = (size_t)HID * 3 * HID + HID + (size_t)HID * HID + HID;
    node0 = edge0 + L * edge_sz;
    node_sz = (size_t)HID * 2 * HID + HID + (size_t)HID * HID + HID;
    o = node0 + L * node_sz;
    dec = block(o, HID, out);
    nh = (size_t)N * HID;
    ne = (size_t)E * HID;
    const size_t most = nh > ne ? nh : ne;
    size_t q = 0;
    auto take = [&](size_t n) {
      const size_t at = q;
      q += n;
      return at;
    };
    h = take((L + 1) * nh);
    e = take((L + 1) * ne);
    agg = take(L * nh);
    z_enc_n = take(nh);
    z_enc_e = take(ne);
    z_edge = take(L * ne);
    z_node = take(L * nh);
    z_dec = take(nh);
    dh = take(nh);
    de = take(ne);
    dagg = take(nh);
    dx = take(3 * most);
    dz = take(most);
    total = q;
  }
};

// Row stride of a network input or gradient (0: packed rows).
int net_ld(int ld, int width) { return ld ? ld : width; }

bool net_ok(const cfd_mpnn_net *n) {
  return n && net_ld(n->ld_xn, n->node_in) >= n->node_in && net_ld(n->ld_xe, n->edge_in) >= n->edge_in &&
         n->layers >= 0 && n->node_in >= 1 && n->node_in <= KMAX && n->edge_in >= 1 && n->edge_in <= KMAX &&
         n->out >= 1 && n->out <= 16 && n->n_nodes >= 0 && n->n_edges >= 0 && n->params && n->act &&
         (n->n_nodes == 0 || (n->xn && n->dst_ptr && n->pred)) && (n->n_edges == 0 || (n->xe && n->src && n->dst)) &&
         aligned(n->params, 16) && aligned(n->act, 16);
}

SegDev seg_of(const float *src, int width, const int *idx = nullptr, int silu = 0) {
  return SegDev{src, idx, width, width, silu};
}

}  // namespace

extern "C" {

int cfd_mpnn_wgrad_blocks(void) { return CFD_MPNN_WGRAD_BLOCKS; }

cfd_status cfd_mpnn_status(int *status, int reset) {
  if (!status) return bad("cfd_mpnn_status: null argument");
  cudaError_t e = cudaMemcpyFromSymbol(status, g_tc_status, sizeof(int));
  if (e == cudaSuccess && reset) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(int));
  }
  if (e != cudaSuccess) {
    cfdb::set_last_error(std::string("cfd_mpnn_status: ") + cudaGetErrorString(e));
    return CFD_ERR_CUDA;
  }
  return CFD_OK;
}

cfd_status cfd_mpnn_mlp_forward(const cfd_mlp_fwd *p, void *stream) {
  if (!p || p->rows < 0 || p->out < 1 || p->out > HID || !p->w1 || !p->b1 || !p->w2 || !p->b2 || !p->y ||
      p->ld_y < p->out || (p->resid && p->ld_resid < p->out))
    return bad("cfd_mpnn_mlp_forward: bad argument");
  FwdArgs a{};
  if (!copy_segs(p->nseg, p->seg, a.seg, a.K)) return bad("cfd_mpnn_mlp_forward: bad input segments (total width <= 192)");
  if (p->rows == 0) return CFD_OK;
  a.M = p->rows;
  a.N2 = p->out;
  a.nseg = p->nseg;
  a.w1 = p->w1;
  a.b1 = p->b1;
  a.w2 = p->w2;
  a.b2 = p->b2;
  a.resid = p->resid;
  a.ld_resid = p->ld_resid;
  a.z1 = p->z1;
  a.y = p->y;
  a.ld_y = p->ld_y;
  if (p->engine == 1) {
    // tcgen05 form: the tiles plus 48 KB, and at least 80 KB, of shared memory per CTA, so that at
    // most two CTAs (2 x 128 tensor-memory columns of the SM's 512) share an SM.
    const size_t need = tc_smem(a.K, a.N2) + 48 * 1024, sm = need > 80 * 1024 ? need : 80 * 1024;
    set_smem(k_mlp_fwd_tc, sm);
    const int ntiles = (a.M + TM_TC - 1) / TM_TC;
    const int grid = ntiles < 2 * sm_count() ? ntiles : 2 * sm_count();
    k_mlp_fwd_tc<<<grid, 128, sm, static_cast<cudaStream_t>(stream)>>>(a);
    return status_of("cfd_mpnn_mlp_forward (tcgen05)");
  }
  launch_mlp_fwd(a, static_cast<cudaStream_t>(stream));
  return status_of("cfd_mpnn_mlp_forward");
}

cfd_status cfd_mpnn_mlp_backward(const cfd_mlp_bwd *p, void *stream) {
  if (!p || p->rows < 0 || p->in_width < 1 || p->in_width > KMAX || p->out < 1 || p->out > HID || !p->dy ||
      p->ld_dy < p->out || !p->z1 || !p->w1 || !p->w2 || !p->dz1 || (p->dx && p->ld_dx < p->in_width))
    return bad("cfd_mpnn_mlp_backward: bad argument");
  if (p->rows == 0) return CFD_OK;
  BwdArgs a{};
  a.M = p->rows;
  a.K = p->in_width;
  a.N2 = p->out;
  a.dy = p->dy;
  a.ld_dy = p->ld_dy;
  a.z1 = p->z1;
  a.w1 = p->w1;
  a.w2 = p->w2;
  a.dz1 = p->dz1;
  a.dx = p->dx;
  a.ld_dx = p->ld_dx;
  if (p->engine == 1) {
    // tcgen05 form: one CTA per SM (at least 120 KB of shared memory each), each holding 256 of
    // the SM's 512 tensor-memory columns.
    const size_t need = bwd_tc_smem(a.K, a.N2) + 16 * 1024, sm = need > 120 * 1024 ? need : 120 * 1024;
    set_smem(k_mlp_bwd_tc, sm);
    const int ntiles = (a.M + TM_TC - 1) / TM_TC;
    const int grid = ntiles < sm_count() ? ntiles : sm_count();
    k_mlp_bwd_tc<<<grid, 128, sm, static_cast<cudaStream_t>(stream)>>>(a);
    return status_of("cfd_mpnn_mlp_backward (tcgen05)");
  }
  launch_mlp_bwd(a, static_cast<cudaStream_t>(stream));
  return status_of("cfd_mpnn_mlp_backward");
}

cfd_status cfd_mpnn_weight_grad(const cfd_mlp_wgrad *p, void *stream) {
  if (!p || p->rows < 0 || !(p->n == HID || (p->n >= 1 && p->n <= 16)) || !p->dz || p->ld_dz < p->n || !p->dw ||
      !p->db || !p->workspace)
    return bad("cfd_mpnn_weight_grad: bad argument (n must be 64 or at most 16)");
  WgArgs a{};
  int K = 0;
  if (!copy_segs(p->nseg, p->seg, a.seg, K)) return bad("cfd_mpnn_weight_grad: bad input segments (total width <= 192)");
  a.M = p->rows;
  a.N = p->n;
  a.K = K;
  a.nseg = p->nseg;
  a.dz = p->dz;
  a.ld_dz = p->ld_dz;
  a.partial = p->workspace;
  launch_wgrad(a, p->dw, p->db, p->accumulate, static_cast<cudaStream_t>(stream));
  return status_of("cfd_mpnn_weight_grad");
}

cfd_status cfd_mpnn_add(float *out, int ldo, const float *a, int lda, const float *b, int ldb, int rows, int width,
                        void *stream) {
  if (rows < 0 || width < 1 || ldo < width || lda < width || ldb < width || (rows > 0 && (!out || !a || !b)))
    return bad("cfd_mpnn_add: bad argument");
  if (rows == 0) return CFD_OK;
  const size_t n = (size_t)rows * width;
  k_add<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(out, ldo, a, lda, b, ldb, rows,
                                                                                    width);
  return status_of("cfd_mpnn_add");
}

cfd_status cfd_mpnn_gather_add(float *out, int ldo, const float *src, int lds, const int *idx, int rows, int width,
                               void *stream) {
  if (rows < 0 || width < 1 || ldo < width || lds < width || (rows > 0 && (!out || !src || !idx)))
    return bad("cfd_mpnn_gather_add: bad argument");
  if (rows == 0) return CFD_OK;
  const size_t n = (size_t)rows * width;
  k_gather_add<<<(unsigned)((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(out, ldo, src, lds, idx,
                                                                                           rows, width);
  return status_of("cfd_mpnn_gather_add");
}

cfd_status cfd_mpnn_segment_sum_acc(const float *x, int ldx, const int *ptr, const int *idx, int n_rows, int width,
                                    float *out, int ldo, int accumulate, void *stream) {
  if (n_rows < 0 || width < 1 || ldx < width || ldo < width || (n_rows > 0 && (!x || !ptr || !idx || !out)))
    return bad("cfd_mpnn_segment_sum_acc: bad argument");
  if (n_rows == 0) return CFD_OK;
  launch_segment_sum(x, ldx, ptr, idx, n_rows, width, out, ldo, accumulate, static_cast<cudaStream_t>(stream));
  return status_of("cfd_mpnn_segment_sum_acc");
}

cfd_status cfd_mpnn_mse(const float *pred, const float *target, int n, float *grad, float *loss, void *stream) {
  if (n < 1 || !pred || !target || !grad || !loss) return bad("cfd_mpnn_mse: bad argument");
  auto overlaps = [&](const float *x) { return x < grad + n && grad < x + n; };
  const bool in_place = overlaps(pred) || overlaps(target);
  k_mse<<<in_place ? 1 : 1 + (n - 1) / 1024 + 1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(pred, target, n, grad, loss,
                                                                                           in_place);
  return status_of("cfd_mpnn_mse");
}

size_t cfd_mpnn_net_floats(int layers, int node_in, int edge_in, int out, int n_nodes, int n_edges) {
  if (layers < 0 || n_nodes < 0 || n_edges < 0) return 0;
  return NetLayout(layers, node_in, edge_in, out, n_nodes, n_edges).total + 4;
}

cfd_status cfd_mpnn_net_forward(const cfd_mpnn_net *n, void *stream) {
  if (!net_ok(n)) return bad("cfd_mpnn_net_forward: bad argument");
  const NetLayout y(n->layers, n->node_in, n->edge_in, n->out, n->n_nodes, n->n_edges);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float *P = n->params;
  float *A = n->act;
  auto run = [&](const NetBlock &b, int rows, int nseg, SegDev s0, SegDev s1, SegDev s2, const float *resid, float *z1,
                 float *out) {
    if (rows == 0) return;
    FwdArgs a{};
    a.M = rows;
    a.K = b.K;
    a.N2 = b.N;
    a.nseg = nseg;
    a.seg[0] = s0;
    a.seg[1] = s1;
    a.seg[2] = s2;
    a.w1 = P + b.w1;
    a.b1 = P + b.b1;
    a.w2 = P + b.w2;
    a.b2 = P + b.b2;
    a.resid = resid;
    a.ld_resid = resid ? HID : 0;
    a.z1 = z1;
    a.y = out;
    a.ld_y = b.N;
    launch_mlp_fwd(a, s);
  };
  const SegDev none{nullptr, nullptr, 0, 0, 0};
  const int N = n->n_nodes, E = n->n_edges;
  run(y.enc_n, N, 1, SegDev{n->xn, nullptr, n->node_in, net_ld(n->ld_xn, n->node_in), 0}, none, none, nullptr, A + y.z_enc_n, A + y.h);
  run(y.enc_e, E, 1, SegDev{n->xe, nullptr, n->edge_in, net_ld(n->ld_xe, n->edge_in), 0}, none, none, nullptr, A + y.z_enc_e, A + y.e);
  for (int l = 0; l < y.L; l++) {
    const float *h = A + y.h + l * y.nh, *e = A + y.e + l * y.ne;
    float *e1 = A + y.e + (l + 1) * y.ne, *agg = A + y.agg + l * y.nh;
    run(y.edge(l), E, 3, seg_of(h, HID, n->src), seg_of(h, HID, n->dst), seg_of(e, HID), e, A + y.z_edge + l * y.ne, e1);
    if (N > 0) launch_segment_sum(e1, HID, n->dst_ptr, nullptr, N, HID, agg, HID, 0, s);
    run(y.node(l), N, 2, seg_of(h, HID), seg_of(agg, HID), none, h, A + y.z_node + l * y.nh, A + y.h + (l + 1) * y.nh);
  }
  run(y.dec, N, 1, seg_of(A + y.h + y.L * y.nh, HID), none, none, nullptr, A + y.z_dec, n->pred);
  return status_of("cfd_mpnn_net_forward");
}

cfd_status cfd_mpnn_net_backward(const cfd_mpnn_net *n, void *stream) {
  if (!net_ok(n) || !n->grads || !n->workspace || net_ld(n->ld_dpred, n->out) < n->out || (n->n_nodes > 0 && (!n->dpred || !n->src_ptr)) ||
      (n->n_edges > 0 && !n->src_order))
    return bad("cfd_mpnn_net_backward: bad argument");
  const NetLayout y(n->layers, n->node_in, n->edge_in, n->out, n->n_nodes, n->n_edges);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float *P = n->params;
  float *A = n->act, *G = n->grads;
  const int N = n->n_nodes, E = n->n_edges;
  float *dh = A + y.dh, *de = A + y.de, *dagg = A + y.dagg, *dx = A + y.dx, *dz = A + y.dz;
  auto wgrad = [&](int rows, int nout, const float *z, int ld_z, int K, int nseg, SegDev s0, SegDev s1, SegDev s2, size_t w,
                   size_t b, const float *ga, int ld_ga, const int *gidx) {
    WgArgs a{};
    a.M = rows;
    a.N = nout;
    a.K = K;
    a.nseg = nseg;
    a.seg[0] = s0;
    a.seg[1] = s1;
    a.seg[2] = s2;
    a.dz = z;
    a.ld_dz = ld_z;
    a.partial = n->workspace;
    a.ga = ga;
    a.ld_ga = ld_ga;
    a.gidx = gidx;
    launch_wgrad(a, G + w, G + b, 0, s);
  };
  const SegDev none{nullptr, nullptr, 0, 0, 0};
  // Gradients of one block from its output gradient dy (+ the rows ga added through gidx): the
  // second layer's weights first (they read dy, which upd may overwrite), then the data path, then
  // the first layer's weights.
  auto block = [&](const NetBlock &b, int rows, const float *dy, int ld_dy, const float *z1, int nseg, SegDev s0, SegDev s1,
                   SegDev s2, float *dxo, int ld_dx, float *upd, int upd_c0, const float *ga, int ld_ga,
                   const int *gidx) {
    wgrad(rows, b.N, dy, ld_dy, HID, 1, seg_of(z1, HID, nullptr, 1), none, none, b.w2, b.b2, ga, ld_ga, gidx);
    if (rows > 0) {
      BwdArgs a{};
      a.M = rows;
      a.K = b.K;
      a.N2 = b.N;
      a.dy = dy;
      a.ld_dy = ld_dy;
      a.z1 = z1;
      a.w1 = P + b.w1;
      a.w2 = P + b.w2;
      a.dz1 = dz;
      a.dx = dxo;
      a.ld_dx = ld_dx;
      a.ga = ga;
      a.ld_ga = ld_ga;
      a.gidx = gidx;
      a.upd = upd;
      a.ld_upd = HID;
      a.upd_c0 = upd_c0;
      launch_mlp_bwd(a, s);
    }
    wgrad(rows, HID, dz, HID, b.K, nseg, s0, s1, s2, b.w1, b.b1, nullptr, 0, nullptr);
  };
  block(y.dec, N, n->dpred, net_ld(n->ld_dpred, n->out), A + y.z_dec, 1, seg_of(A + y.h + y.L * y.nh, HID), none, none, dh, HID, nullptr, 0, nullptr,
        0, nullptr);
  if (E > 0) cudaMemsetAsync(de, 0, y.ne * sizeof(float), s);
  for (int l = y.L - 1; l >= 0; l--) {
    const float *h = A + y.h + l * y.nh, *e = A + y.e + l * y.ne, *agg = A + y.agg + l * y.nh;
    // Node block: dh += its input gradient's columns [0, 64); columns [64, 128) are the gradient of
    // agg, [N][64] rows of their own (the column offset taken off the pointer).
    block(y.node(l), N, dh, HID, A + y.z_node + l * y.nh, 2, seg_of(h, HID), seg_of(agg, HID), none, dagg - HID, HID, dh, 0,
          nullptr, 0, nullptr);
    // Edge block: its output gradient is de + dagg[dst].
    block(y.edge(l), E, de, HID, A + y.z_edge + l * y.ne, 3, seg_of(h, HID, n->src), seg_of(h, HID, n->dst), seg_of(e, HID),
          dx, 3 * HID, de, 2 * HID, dagg, HID, n->dst);
    if (N > 0) k_edge_gather_bwd<<<(N + 7) / 8, 256, 0, s>>>(dx, 3 * HID, n->src_ptr, n->src_order, n->dst_ptr, N, dh);
  }
  block(y.enc_e, E, de, HID, A + y.z_enc_e, 1, SegDev{n->xe, nullptr, n->edge_in, net_ld(n->ld_xe, n->edge_in), 0}, none, none, nullptr, 0, nullptr, 0, nullptr, 0,
        nullptr);
  block(y.enc_n, N, dh, HID, A + y.z_enc_n, 1, SegDev{n->xn, nullptr, n->node_in, net_ld(n->ld_xn, n->node_in), 0}, none, none, nullptr, 0, nullptr, 0, nullptr, 0,
        nullptr);
  return status_of("cfd_mpnn_net_backward");
}

}  // extern "C"
