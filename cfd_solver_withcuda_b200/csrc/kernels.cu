// CUDA kernels of the explicit FV residual/update path (sm_100a, FP64, --fmad=false).
//
// One thread per physical cell gathers its own faces in the reference's face order 0..nF-1,
// so every per-cell sum is formed in the same order as the reference's serial loop and the
// result is deterministic and bit-identical; there are no atomics on data.  Reductions (min dt,
// residual and error norms) use a fixed-shape warp-shuffle tree per block and a fixed-order pass
// over the per-block partials (a last-block pass, or the two-level group pass of the last stage).
#include <algorithm>
#include <climits>
#include <type_traits>

#include "kernels.cuh"
#include "physics.cuh"

namespace cfdb {

namespace {

constexpr int kFluxBlock = 128;
constexpr int kFlux4Block = 128;  // 32 cells x 4 face lanes
constexpr int kBlock = 256;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ bool step_done(const double *ctl) { return ctl[CTL_DONE] != 0.0; }

// Programmatic dependent launch: a kernel launched with programmatic stream serialization may
// start while its predecessor grid drains; it allows its own dependents to launch at entry and
// waits for the predecessor's completion (and memory) before its first global access.  Both are
// no-ops for a normal launch.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches kernel k (smem bytes of dynamic shared memory), with programmatic stream
// serialization when m.pdl is set and the L2 access-policy window of m when it has one.
template <typename... KArgs, typename... Args>
void launch_ks(const DevMesh &m, void (*k)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
               Args... args) {
  if (!m.pdl && !m.l2_bytes) {
    k<<<grid, block, smem, s>>>(args...);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  int na = 0;
  if (m.pdl) {
    at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[na].val.programmaticStreamSerializationAllowed = 1;
    na++;
  }
  if (m.l2_bytes) {
    at[na].id = cudaLaunchAttributeAccessPolicyWindow;
    at[na].val.accessPolicyWindow.base_ptr = m.l2_base;
    at[na].val.accessPolicyWindow.num_bytes = m.l2_bytes;
    at[na].val.accessPolicyWindow.hitRatio = m.l2_hit;
    at[na].val.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    at[na].val.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    na++;
  }
  cfg.attrs = at;
  cfg.numAttrs = na;
  cudaLaunchKernelEx(&cfg, k, args...);
}

template <typename... KArgs, typename... Args>
void launch_k(const DevMesh &m, void (*k)(KArgs...), unsigned grid, unsigned block, cudaStream_t s, Args... args) {
  launch_ks(m, k, grid, block, 0, s, args...);
}

// 32-byte loads and stores of sm_100 (32-byte aligned global addresses).  A warp's rows, records and fluxes
// lie 32 or 64 bytes apart, so as pairs of 16-byte accesses every access touches each of its lines half
// used, and the kernels that gather them were bound by the L1's passes over those lines.  The volatile
// form keeps its place among the thread's stores.
__device__ __forceinline__ double4 ld32(const double4 *p) {
  double4 v;
  asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
// Starts bringing the 16-byte granules inside [off, off + bytes) of a device array into L2.
__device__ __forceinline__ void prefetch_l2(const void *p, size_t off, unsigned int bytes) {
  const size_t a = reinterpret_cast<size_t>(p) + off, lo = (a + 15) & ~(size_t)15;
  const size_t hi = (a + bytes) & ~(size_t)15;
  if (hi > lo) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(lo), "r"((unsigned int)(hi - lo)) : "memory");
}
__device__ __forceinline__ double4 ld32_ordered(const double4 *p) {
  double4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ void st32(double4 *p, const double4 v) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v.x), "d"(v.y), "d"(v.z), "d"(v.w) : "memory");
}
// Eight floats (a cell's FP32 gradients) as two double4.
__device__ __forceinline__ void ld32f(const float4 *p, double4 &a, double4 &b) {
  float v[8];
  asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(p));
  a = make_double4(v[0], v[1], v[2], v[3]);
  b = make_double4(v[4], v[5], v[6], v[7]);
}
// Geometry and cells of one face of the FP32-flux form (DevMesh::frec).
struct FaceRecord {
  float nx, ny, dl, dx, dy;
  int2 on;
};
__device__ __forceinline__ FaceRecord load_face_record(const float4 *rec, size_t i) {
  float v[8];
  asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
      : "l"(rec + 2 * i));
  return FaceRecord{v[0], v[1], v[2], v[3], v[4], make_int2(__float_as_int(v[5]), __float_as_int(v[6]))};
}
__device__ __forceinline__ void st32f(float4 *p, const double g[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(float(g[0])), "f"(float(g[1])),
               "f"(float(g[2])), "f"(float(g[3])), "f"(float(g[4])), "f"(float(g[5])), "f"(float(g[6])), "f"(float(g[7]))
               : "memory");
}

// Item handled by this thread: from the block's work-list range when a list is given (n when the
// thread is past the range's end), else the plain global index.
__device__ __forceinline__ int item_index(const int2 *blk, int n) {
  if (blk) {
    const int2 b = blk[blockIdx.x];
    const int i = b.x + static_cast<int>(threadIdx.x);
    return i < b.y ? i : n;
  }
  return blockIdx.x * blockDim.x + threadIdx.x;
}

__device__ __forceinline__ void flag_bad(int *status, int cell) {
  atomicMin(&status[1], cell);
  atomicCAS(&status[0], 0, 3 /* CFD_ERR_NONPHYSICAL */);
}

__device__ __forceinline__ void store_prim(double *prim, double4 *q4, int NT, int c, const Prim &q) {
  prim[c] = q.rho;
  prim[NT + c] = q.u;
  prim[2 * NT + c] = q.v;
  prim[3 * NT + c] = q.p;
  prim[4 * NT + c] = q.a;
  if (q4) st32(q4 + c, make_double4(q.rho, q.u, q.v, q.p));
}

__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double w = __shfl_xor_sync(kFull, v, o);
    v = w < v ? w : v;
  }
  return v;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Block-wide min; result valid in thread 0.
__device__ __forceinline__ double block_min(double v, double *sh) {
  v = warp_min(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < nw ? sh[lane] : 1e308 * 10.0;
    v = warp_min(v);
  }
  return v;
}

// Block-wide sum (fixed tree); result valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *sh) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < nw ? sh[lane] : 0.0;
    v = warp_sum(v);
  }
  return v;
}

// Warp sums of 8 per-lane values in 9 shuffles: three halving exchanges leave each lane one
// quantity q = 4*bit4 + 2*bit3 + bit2 of its lane id summed over 8 lanes, two more sum the 4
// lanes that share it.  Fixed order, so deterministic.
__device__ __forceinline__ double warp_sums8(const double v[8], int &q) {
  const int lane = threadIdx.x & 31;
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
  double a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double send = h16 ? v[i] : v[i + 4], keep = h16 ? v[i + 4] : v[i];
    a[i] = keep + __shfl_xor_sync(kFull, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const double send = h8 ? a[i] : a[i + 2], keep = h8 ? a[i + 2] : a[i];
    b[i] = keep + __shfl_xor_sync(kFull, send, 8);
  }
  const double send = h4 ? b[0] : b[1], keep = h4 ? b[1] : b[0];
  double c = keep + __shfl_xor_sync(kFull, send, 4);
  c += __shfl_xor_sync(kFull, c, 2);
  c += __shfl_xor_sync(kFull, c, 1);
  q = (h16 ? 4 : 0) + (h8 ? 2 : 0) + (h4 ? 1 : 0);
  return c;
}

// Block sums of 8 per-thread values; the sum of quantity q is returned in thread q (q < 8).
__device__ __forceinline__ double block_sums8(const double v[8], double *sh /* 8 * 32 */) {
  int q;
  const double c = warp_sums8(v, q);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if ((lane & 3) == 0) sh[q * 32 + w] = c;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 8)
    for (int i = 0; i < nw; i++) s += sh[threadIdx.x * 32 + i];
  return s;
}

// Final sums over the per-block partials partial[q * nb + i] (q < NQ), run by the last block: one
// warp per quantity, each lane over a fixed stride of blocks, then a shuffle tree.  The sum of q
// is returned in lane 0 of warp q % (warps per block) for the iteration that handled q.
template <int NQ, typename Store>
__device__ __forceinline__ void sum_partials(const double *partial, int nb, Store store) {
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int q = threadIdx.x >> 5; q < NQ; q += nw) {
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    const double *p = partial + (size_t)q * nb;
    int i = lane;
    for (; i + 96 < nb; i += 128) {
      a0 += __ldcg(p + i);
      a1 += __ldcg(p + i + 32);
      a2 += __ldcg(p + i + 64);
      a3 += __ldcg(p + i + 96);
    }
    for (; i < nb; i += 32) a0 += __ldcg(p + i);
    double a = warp_sum((a0 + a1) + (a2 + a3));
    if (lane == 0) store(q, a);
  }
}

// Reduces nq quantities of n values each, src[q * stride + i] for i < n: the minimum for quantity
// 0 when has_min, sums otherwise.  Warp w takes quantities w, w + nw, ... (at most 3 per warp);
// every lane issues its strided loads of all its quantities before any arithmetic, then a fixed
// shuffle tree, so the result is deterministic.  store(q, v) runs in lane 0 of q's warp.
template <typename Store>
__device__ __forceinline__ void reduce_rows(const double *src, int stride, int n, int nq, bool has_min, Store store) {
  constexpr int kMaxQ = 3, kPer = 4;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double kInf = 1e308 * 10.0;
  int qs[kMaxQ];
  double acc[kMaxQ];
#pragma unroll
  for (int j = 0; j < kMaxQ; j++) {
    qs[j] = w + j * nw;
    acc[j] = (has_min && qs[j] == 0) ? kInf : 0.0;
  }
  for (int base = 0; base < n; base += 32 * kPer) {
    double v[kMaxQ][kPer];
#pragma unroll
    for (int j = 0; j < kMaxQ; j++)
#pragma unroll
      for (int k = 0; k < kPer; k++) {
        const int i = base + k * 32 + lane;
        const bool mn = has_min && qs[j] == 0;
        v[j][k] = (qs[j] < nq && i < n) ? __ldcg(src + (size_t)qs[j] * stride + i) : (mn ? kInf : 0.0);
      }
#pragma unroll
    for (int j = 0; j < kMaxQ; j++)
#pragma unroll
      for (int k = 0; k < kPer; k++) {
        if (has_min && qs[j] == 0) acc[j] = v[j][k] < acc[j] ? v[j][k] : acc[j];
        else acc[j] += v[j][k];
      }
  }
#pragma unroll
  for (int j = 0; j < kMaxQ; j++) {
    if (qs[j] >= nq) continue;  // uniform across the warp
    const double r = (has_min && qs[j] == 0) ? warp_min(acc[j]) : warp_sum(acc[j]);
    if (lane == 0) store(qs[j], r);
  }
}

// Returns true in every thread of the block that finished last among the grid's blocks.  The
// only data the last block reads from other blocks are their partials, which every caller writes
// from threads of warp 0; only that warp fences (a fence in every warp would hold each warp until
// all of its state stores were acknowledged).
__device__ __forceinline__ bool last_block(unsigned int *counter) {
  __shared__ bool is_last;
  if (threadIdx.x < 32) __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = atomicAdd(counter, 1u);
    is_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  return is_last;
}

// Two-level grid reduction of 9 per-block values, written at partial[q * nb + blockIdx.x] by
// threads of warp 0 (q = 0: a minimum, q = 1..8: sums).  Blocks form groups of G consecutive
// blocks; the last block of a group to finish reduces the group's partials in block order into
// partial[9 nb + q * ngroups + group], and the last group to finish reduces those in group order
// into out[9] (shared memory).  Both rounds are a single set of independent loads, and the group
// rounds run while other blocks are still working.  Returns true in the block that wrote out.
__device__ __forceinline__ bool grid_reduce9(const DevState &st, double *out) {
  __shared__ bool flag;
  const int nb = gridDim.x;
  const int G = max(32, (nb + kMaxGroups - 1) / kMaxGroups);
  const int ngroups = (nb + G - 1) / G;
  const int grp = blockIdx.x / G;
  const int gsize = min(G, nb - grp * G);
  if (threadIdx.x < 32) __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) flag = (atomicAdd(&st.gcount[grp], 1u) == (unsigned)(gsize - 1));
  __syncthreads();
  if (!flag) return false;
  double *gp = st.partial + 9 * (size_t)nb;
  reduce_rows(st.partial + (size_t)grp * G, nb, gsize, 9, true,
              [&](int q, double v) { gp[(size_t)q * ngroups + grp] = v; });
  if (threadIdx.x == 0) st.gcount[grp] = 0u;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) flag = (atomicAdd(&st.gcount[kMaxGroups], 1u) == (unsigned)(ngroups - 1));
  __syncthreads();
  if (!flag) return false;
  reduce_rows(gp, ngroups, ngroups, 9, true, [&](int q, double v) { out[q] = v; });
  if (threadIdx.x == 0) st.gcount[kMaxGroups] = 0u;
  __syncthreads();
  return true;
}

// ---------------------------------------------------------------------------------------------
__global__ void k_prim_all(DevMesh m, DevState st) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.NT) return;
  const double *U = st.U;
  Prim q;
  bool ok = eos_prim(U[c], U[m.NT + c], U[2 * m.NT + c], U[3 * m.NT + c], q);
  store_prim(st.prim, st.q4, m.NT, c, q);
  if (!ok) flag_bad(st.status, c);
}

// Apply_Boundary_Conditions (src/Boundary_Conditions.cpp:12-61): one thread per
// (kind, cell, face, ghost) entry writes U and primitives of the ghost row.
//   wall / symmetry  src/Wall_Boundary_Conditions.cpp:8-53, :79-124 (reflect V about the face normal)
//   supersonic inlet src/Inlet_Boundary_Conditions.cpp:41-74 (rho, p prescribed, V extrapolated)
//   subsonic inlet   src/Inlet_Boundary_Conditions.cpp:7-39 (reference energy form)
//   supersonic exit  src/Exit_Boundary_Conditions.cpp:68-94 (copy of U_Cells of the interior cell)
//   subsonic exit    src/Exit_Boundary_Conditions.cpp:83-85 (no-op in the reference)
// Additive forms: total-(p, T) characteristic inflow and static-pressure outflow.
//   far field        CUDA_KERNELS/Boundary_Conditions_Cuda_Kernels.cu:257-325 (inlet kind 4)
//   fixed-p exit     src/Exit_Boundary_Conditions.cpp:8-66 (exit kind 3)
// src_is_S: the supersonic-exit copy reads the stage state (stage-consistent forms) instead of
// U^n; cur_is_S: the state the primitives were last computed from is the stage state.
// Values a boundary state is formed from, read from global memory when a kind needs them.
struct BcGlobal {
  const DevMesh &m;
  const DevState &st;
  int c, f, e, src_is_S, cur_is_S;
  const double4 *bstate;
  const double *bexit;
  __device__ __forceinline__ double nx() const { return m.nx[f * m.NP + c]; }
  __device__ __forceinline__ double ny() const { return m.ny[f * m.NP + c]; }
  __device__ __forceinline__ double a() const { return st.prim[4 * m.NT + c]; }
  __device__ __forceinline__ double cur(int k) const {
    return cur_is_S ? st.S[(size_t)k * m.NP + c] : st.U[(size_t)k * m.NT + c];
  }
  __device__ __forceinline__ double src(int k) const {
    return src_is_S ? st.S[(size_t)k * m.NP + c] : st.U[(size_t)k * m.NT + c];
  }
};

// Conserved ghost state G of an entry of `kind` whose cell has the primitives (rho, u, v, p); false when
// the entry leaves its ghost alone.
template <typename Src>
__device__ __forceinline__ bool bc_values(const Src &s, const BcParams &bp, int kind, double rho, double u, double v,
                                          double p, double G[4]) {
  double G0, G1, G2, G3;
  if (kind == 2 || kind == 3) {
    const double n1 = s.nx(), n2 = s.ny();
    double vdotn = (u * n1 + v * n2);
    double v1g = u - 2.0 * vdotn * n1;
    double v2g = v - 2.0 * vdotn * n2;
    double vmag = 0.5 * (v1g * v1g + v2g * v2g);
    G0 = rho;
    G1 = rho * v1g;
    G2 = rho * v2g;
    G3 = ((p / kGM1) + rho * vmag);
  } else if (kind == 0) {
    if (bp.inlet_bc == 4) {
      const double Ui[4] = {s.cur(0), s.cur(1), s.cur(2), s.cur(3)};
      double Gf[4];
      const double4 fs = s.bstate ? s.bstate[s.e] : make_double4(bp.inlet_rho, bp.inlet_u, bp.inlet_v, bp.inlet_p);
      farfield_state(Ui, s.nx(), s.ny(), fs.x, fs.y, fs.z, fs.w, Gf);
      G0 = Gf[0];
      G1 = Gf[1];
      G2 = Gf[2];
      G3 = Gf[3];
    } else if (bp.inlet_bc == 3) {
      // Fully prescribed inflow (rho, u, v, p), per boundary entry when given (batched solves).
      const double4 q = s.bstate ? s.bstate[s.e] : make_double4(bp.inlet_rho, bp.inlet_u, bp.inlet_v, bp.inlet_p);
      G0 = q.x;
      G1 = q.x * q.y;
      G2 = q.x * q.z;
      G3 = q.w / kGM1 + 0.5 * q.x * (q.y * q.y + q.z * q.z);
    } else if (bp.inlet_bc == 0) {
      double vmag = (u * u + v * v) * 0.5;
      G0 = bp.inlet_rho;
      G1 = bp.inlet_rho * u;
      G2 = bp.inlet_rho * v;
      G3 = (bp.inlet_p / kGM1) + bp.inlet_rho * vmag;
    } else if (bp.inlet_bc == 1) {
      double Vm = 0.5 * (u * u + v * v);
      G0 = bp.inlet_rho;
      G1 = bp.inlet_rho * u;
      G2 = bp.inlet_rho * v;
      G3 = (bp.inlet_p / kGM1) + bp.inlet_rho * Vm * Vm;
    } else {
      // Subsonic inflow with total pressure p0 and total temperature T0 (no reference
      // counterpart: the reference's subsonic inlet is the form above).  n is the outward
      // normal, so inflow has Vn < 0 and the characteristic Vn + a leaves the domain: its
      // invariant R+ = Vn + 2a/(g-1) comes from the interior.  With V = Vn n and
      // H0 = a0^2/(g-1) = a^2/(g-1) + Vn^2/2 this gives
      //   (g+1)/(g-1) a^2 - 2 R+ a + (g-1)/2 R+^2 - a0^2 = 0   (larger root),
      // then Vn = R+ - 2a/(g-1), T = a^2/(g R), p = p0 (T/T0)^(g/(g-1)), rho = p/(R T).
      const double n1 = s.nx(), n2 = s.ny();
      const double a_i = s.a();
      const double vn_i = u * n1 + v * n2;
      const double Rp = vn_i + 2.0 * a_i / kGM1;
      const double p0 = s.bstate ? s.bstate[s.e].x : bp.inlet_p0, t0 = s.bstate ? s.bstate[s.e].y : bp.inlet_t0;
      const double a0sq = kGamma * bp.r_gas * t0;
      const double qa = (kGamma + 1.0) / kGM1, qb = -2.0 * Rp, qc = 0.5 * kGM1 * Rp * Rp - a0sq;
      const double disc = qb * qb - 4.0 * qa * qc;
      const double ab = (-qb + sqrt(disc > 0.0 ? disc : 0.0)) / (2.0 * qa);
      double vn = Rp - 2.0 * ab / kGM1;
      if (vn > 0.0) vn = 0.0;
      const double Tb = ab * ab / (kGamma * bp.r_gas);
      const double pb = p0 * pow(Tb / t0, kGamma / kGM1);
      const double rb = pb / (bp.r_gas * Tb);
      const double ub = vn * n1, vb = vn * n2;
      G0 = rb;
      G1 = rb * ub;
      G2 = rb * vb;
      G3 = pb / kGM1 + 0.5 * rb * (ub * ub + vb * vb);
    }
  } else {  // exit
    if (bp.exit_bc == 1) return false;
    if (bp.exit_bc == 0) {
      G0 = s.src(0);
      G1 = s.src(1);
      G2 = s.src(2);
      G3 = s.src(3);
    } else if (bp.exit_bc == 3) {
      const double rho_Et = s.cur(3);
      double Gf[4];
      fixed_p_exit_state(rho, u, v, p, rho_Et, s.nx(), s.ny(), s.bexit ? s.bexit[s.e] : bp.exit_p, Gf);
      G0 = Gf[0];
      G1 = Gf[1];
      G2 = Gf[2];
      G3 = Gf[3];
    } else {
      // Static-pressure outflow: rho, V extrapolated; p prescribed when the normal Mach
      // number is subsonic, extrapolated otherwise.
      const double n1 = s.nx(), n2 = s.ny();
      const double a_i = s.a();
      const double vn = u * n1 + v * n2;
      const double pb = (vn < a_i) ? (s.bexit ? s.bexit[s.e] : bp.exit_p) : p;
      G0 = rho;
      G1 = rho * u;
      G2 = rho * v;
      G3 = pb / kGM1 + 0.5 * rho * (u * u + v * v);
    }
  }
  G[0] = G0;
  G[1] = G1;
  G[2] = G2;
  G[3] = G3;
  return true;
}

__device__ __forceinline__ void store_ghost(const DevState &st, int NT, int g, const double G[4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) st.U[(size_t)k * NT + g] = G[k];
  Prim q;
  const bool ok = eos_fast(G[0], G[1], G[2], G[3], q);
  store_prim(st.prim, st.q4, NT, g, q);
  if (!ok) flag_bad(st.status, g);
}

__device__ __forceinline__ void bc_entry(const DevMesh &m, const DevState &st, const BcParams &bp, int e, int src_is_S,
                                         int cur_is_S) {
  const int4 b = m.bnd[e];
  const int c = b.y, NT = m.NT;
  const BcGlobal src{m, st, c, b.z, e, src_is_S, cur_is_S, m.bstate, m.bexit};
  double G[4];
  if (bc_values(src, bp, b.x, st.prim[c], st.prim[NT + c], st.prim[2 * NT + c], st.prim[3 * NT + c], G))
    store_ghost(st, NT, b.w, G);
}

// The same from the cell's (rho, u, v, p) row: between pseudo-steps whose primitive planes are not stored
// only the sound speed's plane is current.
__device__ __forceinline__ void bc_entry_row(const DevMesh &m, const DevState &st, const BcParams &bp, int e,
                                             const double4 q) {
  const int4 b = m.bnd[e];
  const BcGlobal src{m, st, b.y, b.z, e, 0, 0, m.bstate, m.bexit};
  double G[4];
  if (bc_values(src, bp, b.x, q.x, q.y, q.z, q.w, G)) store_ghost(st, m.NT, b.w, G);
}

__global__ void k_bc(DevMesh m, DevState st, BcParams bp, int src_is_S, int cur_is_S) {
  pdl_enter();
  const int e = item_index(m.bblk, m.NB);
  if (e >= m.NB || step_done(st.ctl)) return;
  bc_entry(m, st, bp, e, src_is_S, cur_is_S);
}

// Conserved state of cell n for the limiter / LLF: U_Cells (U^n on physical rows, boundary
// values on ghost rows) in the reference's semantics, or the current stage state.
struct USrc {
  const double *U, *S;
  int NT, NP, use_S;
  __device__ __forceinline__ double get(int k, int n) const {
    return (use_S && n < NP) ? S[k * NP + n] : U[k * NT + n];
  }
};

// The state of the cell whose faces are being evaluated.
struct CellState {
  double rc, uc, vc, pc, ac;
  double Uc[4];
  uint8_t degen;
};

template <int DISS, int ORDER>
__device__ __forceinline__ void load_cell(const DevMesh &m, const DevState &st, const USrc &us, int c, CellState &q) {
  const int NT = m.NT;
  const double *prim = st.prim;
  q.rc = prim[c];
  q.uc = prim[NT + c];
  q.vc = prim[2 * NT + c];
  q.pc = prim[3 * NT + c];
  q.ac = prim[4 * NT + c];
  if (DISS == 1 || DISS == 2 || DISS == 5 || DISS == 6 || DISS == 7 || ORDER == 2) {
#pragma unroll
    for (int k = 0; k < 4; k++) q.Uc[k] = us.get(k, c);
  }
  q.degen = m.degen[c];
}

// Geometry of face f of cell c.
struct FaceGeo {
  int N, n2;
  double nx, ny, dl, d1, d2;
};
template <int DISS, int ORDER>
__device__ __forceinline__ FaceGeo load_face(const DevMesh &m, int c, int f) {
  const int idx = f * m.NP + c;
  FaceGeo g;
  g.N = m.nbr[idx];
  g.nx = m.nx[idx];
  g.ny = m.ny[idx];
  g.dl = m.dl[idx];
  if (ORDER == 2 && DISS != 2) {
    g.n2 = m.n2[idx];
    g.d1 = m.d1l[idx];
    g.d2 = m.d2l[idx];
  }
  return g;
}

// Contribution of face f of cell c: X = avg - diss (Calculate_Flux_For_All_Faces,
// src/Net_Flux.cpp:18-43) and the del_t term (|V.n| + a) dl (src/Time_Step.cpp:326-336).
template <int DISS, int ORDER, typename O>
__device__ __forceinline__ void face_contrib(O &o, const DevMesh &m, const DevState &st, const FluxParams &fp,
                                             const USrc &us, const CellState &q, const FaceGeo &g, int f, double X[4],
                                             double &t) {
  const int NP = m.NP, NT = m.NT;
  const double *prim = st.prim;
  const double rc = q.rc, uc = q.uc, vc = q.vc, pc = q.pc, ac = q.ac;
  const int N = g.N;
  const double nx = g.nx, ny = g.ny, dl = g.dl;
  const double rn = prim[N], un = prim[NT + N], vn = prim[2 * NT + N], pn = prim[3 * NT + N], an = prim[4 * NT + N];
  double A[4], D[4];
  if (DISS != 6 && DISS != 7) average_flux<double>(rc, uc, vc, pc, rn, un, vn, pn, nx, ny, dl, A);
  if (DISS == 3 && ORDER == 1) {
    if (N >= NP)
      roe_1o<double>(o, rc, uc, vc, pc, ac, rc, uc, vc, pc, ac, nx, ny, dl, (q.degen >> f) & 1, D);
    else
      roe_1o<double>(o, rc, uc, vc, pc, ac, rn, un, vn, pn, an, nx, ny, dl, (q.degen >> f) & 1, D);
  } else if (DISS == 3 && ORDER == 2) {
    const int n2 = g.n2;
    const double d1 = g.d1, d2 = g.d2;
    double dU[4], phi[4];
    if (!fp.recon_prim) {
      double q1[4], q2[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        q1[k] = us.get(k, N);
        q2[k] = us.get(k, n2);
      }
      limited_slopes<double>(o, fp.limiter, q.Uc, q1, q2, d1, d2, fp.zeta, fp.zeta1, phi);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const double VR = q1[k] + 0.5 * phi[k] * d1;
        const double VL = q.Uc[k] - 0.5 * phi[k] * d1;
        dU[k] = VR - VL;
      }
    } else {
      // MUSCL on (rho, u, v, p) of the stage primitives on the reference stencil; the
      // conserved jump of the two reconstructed face states drives the Roe wave strengths.
      const double qc[4] = {rc, uc, vc, pc};
      const double q1v[4] = {rn, un, vn, pn};
      const double q2v[4] = {prim[n2], prim[NT + n2], prim[2 * NT + n2], prim[3 * NT + n2]};
      double qR[4], qL[4];
      limited_slopes<double>(o, fp.limiter, qc, q1v, q2v, d1, d2, fp.zeta, fp.zeta1, phi);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        qR[k] = q1v[k] + 0.5 * phi[k] * d1;
        qL[k] = qc[k] - 0.5 * phi[k] * d1;
      }
      dU[0] = qR[0] - qL[0];
      dU[1] = qR[0] * qR[1] - qL[0] * qL[1];
      dU[2] = qR[0] * qR[2] - qL[0] * qL[2];
      dU[3] = (o.div_gm1(qR[3]) + 0.5 * qR[0] * (qR[1] * qR[1] + qR[2] * qR[2])) -
              (o.div_gm1(qL[3]) + 0.5 * qL[0] * (qL[1] * qL[1] + qL[2] * qL[2]));
    }
    roe_2o<double>(o, rc, uc, vc, pc, ac, rn, un, vn, pn, an, nx, ny, dl, dU, D);
  } else if (DISS == 2 || DISS == 4 || DISS == 5) {
    // MOVERS, RICCA, MOVERS_NWSC and their second-order forms (src/MOVERS.cpp, src/RICCA.cpp,
    // src/MOVERS_NWSC.cpp); RICCA_2O and MOVERS_NWSC_2O take the limited conserved jump of
    // Second_Order_Limiter (src/Limiters.cpp:97-200), MOVERS_2O does not call it.
    double UR[4], dU2[4] = {0.0, 0.0, 0.0, 0.0};
    if (DISS != 4 || ORDER == 2) {
#pragma unroll
      for (int k = 0; k < 4; k++) UR[k] = us.get(k, N);
    }
    if (ORDER == 2 && DISS != 2) {
      const int n2 = g.n2;
      const double d1 = g.d1, d2 = g.d2;
      double q2[4], phi[4];
#pragma unroll
      for (int k = 0; k < 4; k++) q2[k] = us.get(k, n2);
      limited_slopes<double>(o, fp.limiter, q.Uc, UR, q2, d1, d2, fp.zeta, fp.zeta1, phi);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const double VR = UR[k] + 0.5 * phi[k] * d1;
        const double VL = q.Uc[k] - 0.5 * phi[k] * d1;
        dU2[k] = VR - VL;
      }
    }
    if (DISS == 2)
      movers_diss<double, ORDER>(o, rc, uc, vc, pc, ac, rn, un, vn, pn, an, q.Uc, UR, nx, ny, dl, fp.movers_single,
                                 fp.movers_efix, D);
    else if (DISS == 4)
      ricca_diss<double, ORDER>(o, rc, uc, vc, pc, rn, un, vn, pn, nx, ny, dl, dU2, D);
    else
      nwsc_diss<double, ORDER>(o, rc, uc, vc, pc, rn, un, vn, pn, q.Uc, UR, nx, ny, dl, dU2, D);
  } else if (DISS == 6 || DISS == 7) {
    // Reference forms of AUSM (src/Ausm_Flux.cpp:26-34, from U_Cells) and HLLC
    // (CUDA_KERNELS/HLLC_LLF_Flux_Cuda_Kernels.cu:98-100): faces whose neighbour is a ghost are
    // skipped; the net flux is the sum of the face fluxes.
#pragma unroll
    for (int k = 0; k < 4; k++) A[k] = D[k] = 0.0;
    if (N < NP) {
      double UR[4];
#pragma unroll
      for (int k = 0; k < 4; k++) UR[k] = us.get(k, N);
      if (DISS == 6) {
        ausm_face<double>(o, q.Uc, UR, nx, ny, dl, A);
      } else {
        const double qL[5] = {rc, uc, vc, pc, ac}, qR[5] = {rn, un, vn, pn, an};
        hllc_face<double>(o, qL, q.Uc, qR, UR, nx, ny, dl, A);
      }
    }
  } else {  // LLF 1O
    double UR[4];
#pragma unroll
    for (int k = 0; k < 4; k++) UR[k] = us.get(k, N);
    llf_1o<double>(uc, vc, ac, un, vn, an, q.Uc, UR, nx, ny, dl, D);
  }
#pragma unroll
  for (int k = 0; k < 4; k++) X[k] = A[k] - D[k];
  const double vnf = uc * nx + vc * ny;
  t = (fabs(vnf) + ac) * dl;
}

// del_t = CFL * Area / sum (|V.n| + a) dl, 0 when the sum is not a positive finite number
// (Inviscid_Time_Step, src/Time_Step.cpp:337-358).
__device__ __forceinline__ double cell_dt_a(const FluxParams &fp, double area, double den) {
  if (den <= 0.0 || !isfinite(den)) return 0.0;
  return fp.cfl * area / den;
}
__device__ __forceinline__ double cell_dt(const DevMesh &m, const FluxParams &fp, int c, double den) {
  return cell_dt_a(fp, m.area[c], den);
}

// Block min of del_t to `partial`; the last block writes Min_dt (get_Min_dt,
// src/Numerical_Method.cpp:322-330).
__device__ __forceinline__ void min_dt_epilogue(const DevState &st, double dt, double *sh) {
  double bm = block_min(dt, sh);
  if (threadIdx.x == 0) st.partial[blockIdx.x] = bm;
  if (last_block(st.counter)) {
    double v = 1e308 * 10.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
      double w = __ldcg(&st.partial[i]);
      v = w < v ? w : v;
    }
    v = block_min(v, sh);
    if (threadIdx.x == 0) {
      st.ctl[CTL_DTMIN] = v;
      *st.counter = 0u;
    }
  }
}

// Contribution of one face with the plain operators: for faces whose branch-free evaluation met an
// operand outside its range.
template <int DISS, int ORDER>
__device__ __noinline__ double4 face_contrib_again(const DevMesh &m, const DevState &st, const FluxParams &fp,
                                                   int use_S, int c, int f) {
  const USrc us{st.U, st.S, m.NT, m.NP, use_S};
  Ieee<double> o;
  CellState q;
  load_cell<DISS, ORDER>(m, st, us, c, q);
  double X[4], t;
  face_contrib<DISS, ORDER>(o, m, st, fp, us, q, load_face<DISS, ORDER>(m, c, f), f, X, t);
  return make_double4(X[0], X[1], X[2], X[3]);
}

// Evaluate_Cell_Net_Flux_1O/2O (src/Net_Flux.cpp:46-129) + Evaluate_Time_Step (src/Time_Step.cpp:293-359)
// fused, one thread per cell: faces in order, Net += avg - diss; then del_t; block min + Min_dt.
// MINB: minimum resident blocks per SM the register allocation is made for (6; the second-order forms
// with the directional limiter are also built for 8 and unconstrained, the autotuner picks; the results
// are the same bits).  SRC_S false: the conserved states come from U only (the caller knows no stage
// state is read), which saves the per-load choice between U and the stage state.  The divisions and
// square roots are the branch-free ones (Fast64), whose chains interleave within a face, so the face
// loop is not unrolled: unrolled, the kernels took 124 - 136 registers (12 - 16 warps per SM) and ROE
// 101 us, ROE_2O 117 us on 524,288 cells, against 68 and 103 us in a loop at 80 (B200), although ROE and
// HLLC then spill 144 - 244 bytes per thread and the limited forms 304 - 544, held in L1.  LLF, which
// divides nothing, is unrolled at 80 registers without a spill: 41.8 / 117 / 195 us per pseudo-step at 45,000 /
// 320,000 / 524,288 cells against 43.7 / 123 / 209 in a loop and 45.7 / 137 / 215 unrolled without the bound
// (B200).  A cell with an operand outside their range is evaluated again.
// want (FluxWant bits): del_t is stored, and Min_dt formed, only for evaluations whose value is used.
template <int DISS, int ORDER, int MINB = 6, bool SRC_S = true>
__global__ void __launch_bounds__(kFluxBlock, MINB) k_flux(const __grid_constant__ DevMesh m,
                                                           const __grid_constant__ DevState st,
                                                           const __grid_constant__ FluxParams fp, int src_is_S,
                                                           int want) {
  pdl_enter();
  __shared__ double sh[32];
  const int NP = m.NP, NT = m.NT;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const bool done = step_done(st.ctl);
  double dt = 1e308 * 10.0;
  if (c < NP && !done) {
    const int use_S = SRC_S && fp.consistent && src_is_S;
    const USrc us{st.U, st.S, NT, NP, use_S};
    CellState q;
    load_cell<DISS, ORDER>(m, st, us, c, q);
    const int nf = m.nf[c];
    double N0 = 0.0, N1s = 0.0, N2s = 0.0, N3s = 0.0;
    double den = 0.0;
    Fast64 o;
    auto add_face = [&](int f) {
      double X[4], t;
      face_contrib<DISS, ORDER>(o, m, st, fp, us, q, load_face<DISS, ORDER>(m, c, f), f, X, t);
      N0 += X[0];
      N1s += X[1];
      N2s += X[2];
      N3s += X[3];
      den += t;
    };
    if constexpr (DISS == 1) {  // no divisions
#pragma unroll
      for (int f = 0; f < 4; f++)
        if (f < nf) add_face(f);
    } else {
#pragma unroll 1
      for (int f = 0; f < nf; f++) add_face(f);
    }
    if (o.bad()) {
      N0 = N1s = N2s = N3s = 0.0;
      for (int f = 0; f < nf; f++) {
        const double4 X = face_contrib_again<DISS, ORDER>(m, st, fp, use_S, c, f);
        N0 += X.x;
        N1s += X.y;
        N2s += X.z;
        N3s += X.w;
      }
    }
    st.R[c] = N0;
    st.R[NP + c] = N1s;
    st.R[2 * NP + c] = N2s;
    st.R[3 * NP + c] = N3s;
    if (want) {
      dt = cell_dt(m, fp, c, den);
      st.dtc[c] = dt;
    }
  }
  if (done || !(want & kWantMin)) return;
  min_dt_epilogue(st, dt, sh);
}

// The same evaluation with four lanes per cell (one face each): lane 0 of each quad adds the
// quad's face contributions in face order 0..nF-1 (warp shuffles), so every sum keeps the
// reference's order and value; fewer live registers per thread give the SM more warps to hide
// the gather and FP64 latencies.  R and den are lane 0's.
template <int DISS, int ORDER>
__device__ __forceinline__ void quad_residual(const DevMesh &m, const DevState &st, const FluxParams &fp, int use_S, int c,
                                              int f, int nf, const FaceGeo &g, double R[4], double &den) {
  double X[4] = {0.0, 0.0, 0.0, 0.0}, t = 0.0;
  if (f < nf) {
    const USrc us{st.U, st.S, m.NT, m.NP, use_S};
    CellState q;
    load_cell<DISS, ORDER>(m, st, us, c, q);
    Fast64 o;
    face_contrib<DISS, ORDER>(o, m, st, fp, us, q, g, f, X, t);
    if (o.bad()) {
      const double4 Y = face_contrib_again<DISS, ORDER>(m, st, fp, use_S, c, f);
      X[0] = Y.x;
      X[1] = Y.y;
      X[2] = Y.z;
      X[3] = Y.w;
    }
  }
  double Y[3][4], T[3];
#pragma unroll
  for (int d = 1; d < 4; d++) {
#pragma unroll
    for (int k = 0; k < 4; k++) Y[d - 1][k] = __shfl_down_sync(kFull, X[k], d, 4);
    T[d - 1] = __shfl_down_sync(kFull, t, d, 4);
  }
  R[0] = R[1] = R[2] = R[3] = 0.0;
  den = 0.0;
#pragma unroll
  for (int k = 0; k < 4; k++) R[k] += X[k];
  den += t;
#pragma unroll
  for (int d = 1; d < 4; d++) {
    if (d < nf) {
#pragma unroll
      for (int k = 0; k < 4; k++) R[k] += Y[d - 1][k];
      den += T[d - 1];
    }
  }
}

template <int DISS, int ORDER>
__global__ void __launch_bounds__(kFlux4Block) k_flux4(const __grid_constant__ DevMesh m,
                                                       const __grid_constant__ DevState st,
                                                       const __grid_constant__ FluxParams fp, int src_is_S,
                                                       int want) {
  pdl_enter();
  __shared__ double sh[32];
  const int NP = m.NP;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = gid >> 2, f = gid & 3;
  if (step_done(st.ctl)) return;
  double R[4], den, dt = 1e308 * 10.0;
  const int nf = c < NP ? m.nf[c] : 0;
  const FaceGeo g = load_face<DISS, ORDER>(m, c < NP ? c : 0, f);
  quad_residual<DISS, ORDER>(m, st, fp, fp.consistent && src_is_S, c, f, nf, g, R, den);
  if (c < NP && f == 0) {
#pragma unroll
    for (int k = 0; k < 4; k++) st.R[k * NP + c] = R[k];
    if (want) {
      dt = cell_dt(m, fp, c, den);
      st.dtc[c] = dt;
    }
  }
  if (want & kWantMin) min_dt_epilogue(st, dt, sh);
}

// Evaluate_Cell_Net_Flux_WENO, src/WENO2D.cpp:395-456, one thread per cell.  Quad cells only
// (others get a zero net flux and their del_t, as in the reference).  Stencils walk the neighbour
// slots as the reference does (WENO_Reconstruction_X, :245-393): slot 0 / 1 for the "i" walks and
// 2 / 3 for the "j" walks, a ghost repeated when the walk leaves the domain.  The stencil values
// are the conserved variables the reference rebuilds from the primitives
// (Calculate_Computational_Variables, src/Basic_Functions.cpp:156-163): rho, rho*u, rho*v and the
// energy the primitives were computed from (cur_is_S: the stage state for physical cells).
__device__ __forceinline__ void weno_cons(const DevMesh &m, const DevState &st, int i, int cur_is_S, double U[4]) {
  const int NP = m.NP, NT = m.NT;
  const double rho = st.prim[i];
  U[0] = rho;
  U[1] = rho * st.prim[NT + i];
  U[2] = rho * st.prim[2 * NT + i];
  U[3] = (i < NP && cur_is_S) ? st.S[3 * NP + i] : st.U[3 * NT + i];
}

// Get_Reconstructed_U, src/WENO2D.cpp:216-243.
__device__ __forceinline__ bool weno_recon(const DevMesh &m, const DevState &st, int cur_is_S, bool chr,
                                           const double Lm[16], const double ILm[16], int i1, int i2, int i3, int i4,
                                           int i5, int lr, double U[4]) {
  double s[5][4];
  weno_cons(m, st, i1, cur_is_S, s[0]);
  weno_cons(m, st, i2, cur_is_S, s[1]);
  weno_cons(m, st, i3, cur_is_S, s[2]);
  weno_cons(m, st, i4, cur_is_S, s[3]);
  weno_cons(m, st, i5, cur_is_S, s[4]);
  if (chr) {
    double w[5][4], W[4];
#pragma unroll
    for (int k = 0; k < 5; k++) weno_matvec(Lm, s[k], w[k]);
#pragma unroll
    for (int i = 0; i < 4; i++) W[i] = weno5(w[0][i], w[1][i], w[2][i], w[3][i], w[4][i], lr);
    weno_matvec(ILm, W, U);
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) U[i] = weno5(s[0][i], s[1][i], s[2][i], s[3][i], s[4][i], lr);
  }
  return true;
}

__global__ void __launch_bounds__(kFluxBlock) k_weno(DevMesh m, DevState st, FluxParams fp, int cur_is_S) {
  __shared__ double sh[32];
  const int NP = m.NP, NT = m.NT;
  const int c = item_index(m.cblk, NP);
  const bool done = step_done(st.ctl);
  double dt = 1e308 * 10.0;
  if (c < NP && !done) {
    const int nf = m.nf[c];
    double R[4] = {0.0, 0.0, 0.0, 0.0};
    bool ok = true;
    if (nf == 4) {
      const int im1 = m.nbr[c], ip1 = m.nbr[NP + c], jm1 = m.nbr[2 * NP + c], jp1 = m.nbr[3 * NP + c];
      int im2, im3, ip2, ip3, jm2, jm3, jp2, jp3;
      if (im1 >= NP) {
        im2 = im1;
        im3 = im1;
      } else {
        im2 = m.nbr[im1];
        if (im2 >= NP || im2 < 0) {
          im3 = im2;
        } else {
          im3 = m.nbr[im2];
          if (im3 < 0) im3 = im2;
        }
      }
      if (ip1 >= NP) {
        ip2 = ip1;
        ip3 = ip1;
      } else {
        ip2 = m.nbr[NP + ip1];
        if (ip2 >= NP || ip2 < 0) {
          ip3 = ip2;
        } else {
          ip3 = m.nbr[NP + ip2];
          if (ip3 < 0) ip3 = ip2;
        }
      }
      if (jm1 >= NP) {
        jm2 = jm1;
        jm3 = jm1;
      } else {
        jm2 = m.nbr[2 * NP + jm1];
        jm3 = (jm2 >= NP) ? jm2 : m.nbr[2 * NP + jm2];
      }
      if (jp1 >= NP) {
        jp2 = jp1;
        jp3 = jp1;
      } else {
        jp2 = m.nbr[3 * NP + jp1];
        jp3 = (jp2 >= NP) ? jp2 : m.nbr[3 * NP + jp2];
      }
      // Face stencils (left: shift 0, right: shift 1) of WENO_Reconstruction_X's switch.
      const int st5[4][2][5] = {{{im3, im2, im1, c, ip1}, {im2, im1, c, ip1, ip2}},
                                {{jm3, jm2, jm1, c, jp1}, {jm2, jm1, c, jp1, jp2}},
                                {{im2, im1, c, ip1, ip2}, {im1, c, ip1, ip2, ip3}},
                                {{jm2, jm1, c, jp1, jp2}, {jm1, c, jp1, jp2, jp3}}};
      const int nb[4] = {im1, ip1, jm1, jp1};
#pragma unroll 1
      for (int f = 0; f < 4; f++) {
        const int idx = f * NP + c;
        const double nx = m.nx[idx], ny = m.ny[idx], dl = m.dl[idx];
        double Lm[16], ILm[16];
        if (fp.weno_char) {
          const int N = nb[f];
          ok = weno_lr(st.prim[c], st.prim[NT + c], st.prim[2 * NT + c], st.prim[4 * NT + c], st.prim[N],
                       st.prim[NT + N], st.prim[2 * NT + N], st.prim[4 * NT + N], nx, ny, Lm, ILm) && ok;
        }
        double UL[4], UR[4], F[4];
        const int *a = st5[f][0], *b = st5[f][1];
        weno_recon(m, st, cur_is_S, fp.weno_char, Lm, ILm, a[0], a[1], a[2], a[3], a[4], 0, UL);
        weno_recon(m, st, cur_is_S, fp.weno_char, Lm, ILm, b[0], b[1], b[2], b[3], b[4], 1, UR);
        ok = weno_face_flux(UL, UR, nx, ny, dl, F) && ok;
#pragma unroll
        for (int k = 0; k < 4; k++) R[k] += F[k];
      }
    }
    if (!ok) flag_bad(st.status, c);
    // Evaluate_Time_Step (src/Time_Step.cpp:293-329) from the cell's own state.
    const double uc = st.prim[NT + c], vc = st.prim[2 * NT + c], ac = st.prim[4 * NT + c];
    double den = 0.0;
    for (int f = 0; f < nf; f++) {
      const int idx = f * NP + c;
      const double vnf = uc * m.nx[idx] + vc * m.ny[idx];
      den += (fabs(vnf) + ac) * m.dl[idx];
    }
    dt = cell_dt(m, fp, c, den);
#pragma unroll
    for (int k = 0; k < 4; k++) st.R[k * NP + c] = R[k];
    st.dtc[c] = dt;
  }
  min_dt_epilogue(st, dt, sh);
}

// Face-based evaluation (the Green-Gauss-gradient MUSCL form; no reference counterpart): one
// thread per unique face computes the flux once from its owner's side, in precision T (double,
// or float for the FP32-flux form); the neighbour receives exactly the negated flux, so the
// scheme is conservative to the last bit.  MUSCL on (rho, u, v, p): with d = x_N - x_c and
// D+ = q_N - q_c, the upwind differences are D-_c = 2 grad q_c . d - D+ and
// D-_N = 2 grad q_N . d - D+; q_L = q_c + 0.5 phi(D-_c, D+) D+, q_R = q_N - 0.5 phi(D-_N, D+) D+
// (phi(a, b), r = a/b; the product phi D+ evaluated as muscl_slope).  A ghost neighbour uses the owner's gradient.  A non-positive
// reconstructed density or pressure falls back to the cell-centre state.  Flux: average of the two
// face states plus Roe dissipation between them (with the linear-wave entropy fix when
// fp.eflin > 0).
// Flux of one unique face from the owner's record (c0: rho, u, v, p; c1, c2: gradients) and the
// neighbour's (n0, n1, n2), face normal (nx, ny), length dl and centre-to-centre vector (dx, dy).
// FaceIn: what the flux needs of the two cells: the states, D+ and the two upwind differences per
// variable, and (DISS 103) whether the pressure gradients mark a shock.
template <typename T>
struct FaceIn {
  T qc[4], qn[4], dp[4], dmc[4], dmn[4];
  bool shock;
};
template <typename T, int DISS>
__device__ __forceinline__ void face_in(const double4 c0, const double4 c1, const double4 c2, const double4 n0,
                                        const double4 n1, const double4 n2, const T dx, const T dy, const T shock_fix,
                                        FaceIn<T> &in) {
  const T qc[4] = {T(c0.x), T(c0.y), T(c0.z), T(c0.w)};
  const T qn[4] = {T(n0.x), T(n0.y), T(n0.z), T(n0.w)};
  const T gc[8] = {T(c1.x), T(c1.y), T(c1.z), T(c1.w), T(c2.x), T(c2.y), T(c2.z), T(c2.w)};
  const T gn[8] = {T(n1.x), T(n1.y), T(n1.z), T(n1.w), T(n2.x), T(n2.y), T(n2.z), T(n2.w)};
#pragma unroll
  for (int k = 0; k < 4; k++) {
    in.qc[k] = qc[k];
    in.qn[k] = qn[k];
    in.dp[k] = qn[k] - qc[k];
    in.dmc[k] = T(2.0) * (gc[2 * k] * dx + gc[2 * k + 1] * dy) - in.dp[k];
    in.dmn[k] = T(2.0) * (gn[2 * k] * dx + gn[2 * k + 1] * dy) - in.dp[k];
  }
  in.shock = false;
  if (DISS == 103 && shock_fix > T(0.0)) {
    // Shock sensor of the hybrid: |grad p|^2 |d|^2 > (shock_fix p)^2 in either cell.
    const T d2 = dx * dx + dy * dy;
    const T gpc = gc[6] * gc[6] + gc[7] * gc[7], gpn = gn[6] * gn[6] + gn[7] * gn[7];
    const T tc = shock_fix * qc[3], tn = shock_fix * qn[3];
    in.shock = gpc * d2 > tc * tc || gpn * d2 > tn * tn;
  }
}

template <int KIND>
__device__ __forceinline__ void half_slopes(Fast64 &o, const FaceIn<double> &in, double qL[4], double qR[4]) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    qL[k] = in.qc[k] + muscl_half_slope<KIND>(o, in.dmc[k], in.dp[k]);
    qR[k] = in.qn[k] - muscl_half_slope<KIND>(o, in.dmn[k], in.dp[k]);
  }
}

template <typename T, int DISS, typename O>
__device__ __forceinline__ double4 face_flux_in(O &o, int glim, const FaceIn<T> &in, const T nx, const T ny, const T dl,
                                                const T eflin) {
  T qL[4], qR[4];
  // The slopes.  Fast64: one branch on the limiter for all eight, so that their divisions interleave.
  bool limited = false;
  if constexpr (O::fast) {
    limited = true;
    if (glim == LIM_VANLEER) half_slopes<LIM_VANLEER>(o, in, qL, qR);
    else if (glim == LIM_VANALBADA) half_slopes<LIM_VANALBADA>(o, in, qL, qR);
    else if (glim == LIM_MINMOD) half_slopes<LIM_MINMOD>(o, in, qL, qR);
    else limited = false;
    // Non-positive densities or pressures (an integer test; NaN is flagged by the roots below).
    if (limited) {
      const bool badL = __double2hiint(qL[0]) <= 0 || __double2hiint(qL[3]) <= 0;
      const bool badR = __double2hiint(qR[0]) <= 0 || __double2hiint(qR[3]) <= 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {
        qL[k] = badL ? in.qc[k] : qL[k];
        qR[k] = badR ? in.qn[k] : qR[k];
      }
    }
  }
  if (!limited) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      qL[k] = in.qc[k] + T(0.5) * muscl_slope<T>(glim, in.dmc[k], in.dp[k]);
      qR[k] = in.qn[k] - T(0.5) * muscl_slope<T>(glim, in.dmn[k], in.dp[k]);
    }
    if (!(qL[0] > T(0.0)) || !(qL[3] > T(0.0))) {
#pragma unroll
      for (int k = 0; k < 4; k++) qL[k] = in.qc[k];
    }
    if (!(qR[0] > T(0.0)) || !(qR[3] > T(0.0))) {
#pragma unroll
      for (int k = 0; k < 4; k++) qR[k] = in.qn[k];
    }
  }
  const T aL = o.root(o.div(T(kGamma) * qL[3], qL[0])), aR = o.root(o.div(T(kGamma) * qR[3], qR[0]));
  T A[4], D[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
  // DISS 3: Roe; DISS 103: Roe with the options of the form (linear-wave entropy fix, shock-stable
  // hybrid), a separate instance so that the plain form keeps its register footprint.
  if (DISS == 3 || DISS == 103) {
    average_flux<T>(qL[0], qL[1], qL[2], qL[3], qR[0], qR[1], qR[2], qR[3], nx, ny, dl, A);
    const bool rusanov = DISS == 103 && in.shock;
    if (rusanov) {
      const T vnL = qL[1] * nx + qL[2] * ny, vnR = qR[1] * nx + qR[2] * ny;
      const T sL = fabs(vnL) + aL, sR = fabs(vnR) + aR;
      const T sm = sL > sR ? sL : sR;
      const T UL[4] = {qL[0], qL[0] * qL[1], qL[0] * qL[2],
                       o.div_gm1(qL[3]) + T(0.5) * qL[0] * (qL[1] * qL[1] + qL[2] * qL[2])};
      const T UR[4] = {qR[0], qR[0] * qR[1], qR[0] * qR[2],
                       o.div_gm1(qR[3]) + T(0.5) * qR[0] * (qR[1] * qR[1] + qR[2] * qR[2])};
#pragma unroll
      for (int k = 0; k < 4; k++) D[k] = T(0.5) * sm * (UR[k] - UL[k]) * dl;
    } else {
      roe_1o<T>(o, qL[0], qL[1], qL[2], qL[3], aL, qR[0], qR[1], qR[2], qR[3], aR, nx, ny, dl, false, D,
                DISS == 103 ? eflin : T(0.0));
    }
  } else {
    // Conserved face states for AUSM / HLLC: E = p/(g-1) + rho |V|^2 / 2.
    const T UL[4] = {qL[0], qL[0] * qL[1], qL[0] * qL[2],
                     o.div_gm1(qL[3]) + T(0.5) * qL[0] * (qL[1] * qL[1] + qL[2] * qL[2])};
    const T UR[4] = {qR[0], qR[0] * qR[1], qR[0] * qR[2],
                     o.div_gm1(qR[3]) + T(0.5) * qR[0] * (qR[1] * qR[1] + qR[2] * qR[2])};
    if (DISS == 6) {
      ausm_face<T>(o, UL, UR, nx, ny, dl, A);
    } else if (DISS == 8) {
      ausm_gpu_face<T>(UL, UR, nx, ny, dl, A);
    } else {
      const T q5L[5] = {qL[0], qL[1], qL[2], qL[3], aL}, q5R[5] = {qR[0], qR[1], qR[2], qR[3], aR};
      hllc_face<T>(o, q5L, UL, q5R, UR, nx, ny, dl, A);
    }
  }
  return make_double4(double(A[0] - D[0]), double(A[1] - D[1]), double(A[2] - D[2]), double(A[3] - D[3]));
}

template <typename T, int DISS, typename O>
__device__ __forceinline__ double4 face_flux_rec(O &o, int glim, const double4 c0, const double4 c1, const double4 c2,
                                                 const double4 n0, const double4 n1, const double4 n2, const T nx,
                                                 const T ny, const T dl, const T dx, const T dy, const T eflin,
                                                 const T shock_fix = T(0.0)) {
  FaceIn<T> in;
  face_in<T, DISS>(c0, c1, c2, n0, n1, n2, dx, dy, shock_fix, in);
  return face_flux_in<T, DISS>(o, glim, in, nx, ny, dl, eflin);
}

// Division policy of the face kernels: the branch-free double operations, or plain float ones.
template <typename T>
using FaceOps = typename std::conditional<std::is_same<T, double>::value, Fast64, Ieee<float>>::type;

__device__ __forceinline__ double4 ldcg4(const double4 *p) {
  const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// Flux of face i with the plain operators: for faces whose branch-free evaluation met an operand
// outside its range.  Loads from L2 (the persistent kernel writes rows and records in its launch).
template <int DISS>
__device__ __noinline__ double4 face_flux_again(const DevMesh &m, const DevState &st, const FluxParams &fp, int i) {
  const int2 on = m.fon[i];
  const double4 gq = m.fg4[i];
  const int g = on.y < m.NP ? on.y : on.x;  // a ghost neighbour uses the owner's gradients
  const double4 *rc = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)on.x);
  const double4 *rn = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)g);
  Ieee<double> o;
  return face_flux_rec<double, DISS>(o, fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter, ldcg4(st.q4 + on.x),
                                     ldcg4(rc), ldcg4(rc + 1), ldcg4(st.q4 + on.y), ldcg4(rn), ldcg4(rn + 1), gq.x, gq.y,
                                     gq.z, gq.w, m.fdy[i], fp.eflin, fp.shock_fix);
}

template <typename T, int DISS, int MINB>
__global__ void __launch_bounds__(MINB >= 6 ? 128 : 256, MINB) k_faces(const __grid_constant__ DevMesh m,
                                                                          const __grid_constant__ DevState st,
                                                                          const __grid_constant__ FluxParams fp) {
  pdl_enter();
  const int i = item_index(m.fblk, m.NF);
  if (i >= m.NF || step_done(st.ctl)) return;
  const int NP = m.NP;
  const int glim = fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter;
  int2 on;
  T nx, ny, dl, dx, dy;
  if constexpr (sizeof(T) == sizeof(float)) {
    const FaceRecord r = load_face_record(m.frec, i);
    on = r.on;
    nx = r.nx;
    ny = r.ny;
    dl = r.dl;
    dx = r.dx;
    dy = r.dy;
  } else {
    on = m.fon[i];
    const double4 gq = ld32(m.fg4 + i);
    nx = gq.x;
    ny = gq.y;
    dl = gq.z;
    dx = gq.w;
    dy = m.fdy[i];
  }
  const int c = on.x, N = on.y;
  const double4 c0 = ld32(st.q4 + c), n0 = ld32(st.q4 + N);
  const int G = N < NP ? N : c;  // a ghost neighbour uses the owner's gradients
  double4 c1, c2, n1, n2;
  if (sizeof(T) == sizeof(float)) {
    // FP32-flux form: 32-byte float records (the values face_flux_rec would round to anyway).
    ld32f(st.recf + 2 * (size_t)c, c1, c2);
    ld32f(st.recf + 2 * (size_t)G, n1, n2);
  } else {
    const double4 *rc = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)c);
    const double4 *rn = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)G);
    c1 = ld32(rc);
    c2 = ld32(rc + 1);
    n1 = ld32(rn);
    n2 = ld32(rn + 1);
  }
  FaceOps<T> o;
  double4 F = face_flux_rec<T, DISS>(o, glim, c0, c1, c2, n0, n1, n2, nx, ny, dl, dx, dy, T(fp.eflin), T(fp.shock_fix));
  if constexpr (FaceOps<T>::fast) {
    if (o.bad()) F = face_flux_again<DISS>(m, st, fp, i);
  }
  if constexpr (sizeof(T) == sizeof(float))  // float results: stored as such
    reinterpret_cast<float4 *>(st.F)[i] = make_float4(float(F.x), float(F.y), float(F.z), float(F.w));
  else
    st32(st.F + i, F);
}

// Flux of face id as k_faces left it (FF: the FP32-flux form's floats).
template <bool FF>
__device__ __forceinline__ double4 load_flux(const DevState &st, int id) {
  if (!FF) return ld32(st.F + id);
  const float4 v = reinterpret_cast<const float4 *>(st.F)[id];
  return make_double4(v.x, v.y, v.z, v.w);
}

// Sum of the face fluxes of cell c in face order (+F on the owner side, -F on the neighbour
// side) and the del_t denominator.  The cell's four face-table slots come in one 16-byte load
// without waiting for the face count (an unused slot holds face 0), so the flux loads of every
// face are in flight together; only the sums are predicated on the count.
// CG: the face fluxes were written earlier in the same launch by other thread blocks (the
// persistent stage kernel), so they are loaded from L2 (ld.global.cg), not through L1.
__device__ __forceinline__ int face_id(int e) { return e < 0 ? -e - 1 : e; }

// Sum of a cell's face fluxes in face order, negated on the neighbour side.
__device__ __forceinline__ void sum_faces(int nf, const int4 e4, const double4 F0, const double4 F1, const double4 F2,
                                          const double4 F3, double R[4]) {
  const int e[4] = {e4.x, e4.y, e4.z, e4.w};
  const double4 F[4] = {F0, F1, F2, F3};
  R[0] = R[1] = R[2] = R[3] = 0.0;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    if (f < nf) {
      if (e[f] < 0) {
        R[0] += -F[f].x;
        R[1] += -F[f].y;
        R[2] += -F[f].z;
        R[3] += -F[f].w;
      } else {
        R[0] += F[f].x;
        R[1] += F[f].y;
        R[2] += F[f].z;
        R[3] += F[f].w;
      }
    }
  }
}

template <bool DEN = true, bool CG = false, bool FF = false>
__device__ __forceinline__ void gather_faces(const DevMesh &m, const DevState &st, int c, double R[4], double &den) {
  const int NP = m.NP, NT = m.NT;
  const double uc = DEN ? st.prim[NT + c] : 0.0, vc = DEN ? st.prim[2 * NT + c] : 0.0,
               ac = DEN ? st.prim[4 * NT + c] : 0.0;
  const int nf = m.nf[c];
  const int4 e4 = m.cface4[c];
  const int e[4] = {e4.x, e4.y, e4.z, e4.w};
  double4 F[4];
#pragma unroll
  for (int f = 0; f < 4; f++) {
    const int id = e[f] < 0 ? -e[f] - 1 : e[f];
    F[f] = CG ? ldcg4(st.F + id) : load_flux<FF>(st, id);
  }
  R[0] = R[1] = R[2] = R[3] = 0.0;
  den = 0.0;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    if (f < nf) {
      if (e[f] < 0) {
        R[0] += -F[f].x;
        R[1] += -F[f].y;
        R[2] += -F[f].z;
        R[3] += -F[f].w;
      } else {
        R[0] += F[f].x;
        R[1] += F[f].y;
        R[2] += F[f].z;
        R[3] += F[f].w;
      }
      if (DEN) {
        const int idx = f * NP + c;
        const double vnf = uc * m.nx[idx] + vc * m.ny[idx];
        den += (fabs(vnf) + ac) * m.dl[idx];
      }
    }
  }
}

// Per cell: Net = sum of its face fluxes in face order, del_t from the cell's own state
// (src/Time_Step.cpp:293-329), block min.
template <bool FF>
__global__ void __launch_bounds__(kFluxBlock) k_gather(DevMesh m, DevState st, FluxParams fp) {
  __shared__ double sh[32];
  const int NP = m.NP;
  const int c = item_index(m.cblk, NP);
  const bool done = step_done(st.ctl);
  double dt = 1e308 * 10.0;
  if (c < NP && !done) {
    double R[4], den;
    gather_faces<true, false, FF>(m, st, c, R, den);
    dt = cell_dt(m, fp, c, den);
#pragma unroll
    for (int k = 0; k < 4; k++) st.R[k * NP + c] = R[k];
    st.dtc[c] = dt;
  }
  if (done) return;
  min_dt_epilogue(st, dt, sh);
}

// Estimate_Error (src/Error_Estimate_Update.cpp:10-28) terms of one cell; dU < 1e-9 is the
// reference's signed test.
__device__ __forceinline__ double err_term(double du, double u) {
  double t;
  if (du < 1e-9) t = fabs(du);
  else t = fabs(du) / u;
  return t * t;
}

// Per-block partial sums (4 error terms, 4 residual squares), then the last block reduces the
// partials in block order and applies the step epilogue (Total_Time += Min_dt, iterations++).
__device__ __forceinline__ void reduce_err_and_epilogue(const DevState &st, const double e[8], bool advance_time,
                                                        double dt_for_time) {
  __shared__ double sh[8 * 32];
  double v[8];
#pragma unroll
  for (int q = 0; q < 8; q++) v[q] = e[q];
  const double s = block_sums8(v, sh);
  if (threadIdx.x < 8) st.partial[threadIdx.x * gridDim.x + blockIdx.x] = s;
  if (last_block(st.counter)) {
    double *ctl = st.ctl;
    sum_partials<8>(st.partial, (int)gridDim.x,
                    [ctl](int q, double a) { ctl[(q < 4 ? CTL_ERR + q : CTL_RES + q - 4)] = sqrt(a); });
    __syncthreads();
    if (threadIdx.x == 0) {
      if (advance_time) {
        double t = st.ctl[CTL_TOTAL_TIME] + dt_for_time;
        st.ctl[CTL_TOTAL_TIME] = t;
        st.ctl[CTL_ITER] += 1.0;
        double te = st.ctl[CTL_TEND];
        if (te > 0.0 && t >= te) st.ctl[CTL_DONE] = 1.0;
      }
      *st.counter = 0u;
    }
  }
}

// Stage updates of Runge_Kutta_Method (src/Numerical_Method.cpp:342-457) and Explicit_Method
// (:26-103) for one cell, written with the reference's association order.  kind: 1,2,3 RK3
// stages, 0 explicit, 11..14 classical RK4.  The final kind writes dU and, with fuse_final,
// applies Estimate_Error's terms (e[0..3]), the residual squares (e[4..7]) and Update().
// Stage kinds: 0 explicit; 1-3 the three-stage forms (reference Runge_Kutta_Method or SSP-RK3);
// 11-14 classical RK4; 21-23 the reference GPU TVD-RK3 kernel (21, 22 equal 1, 2); 31-34 the
// reference GPU RK4 kernel.  Kinds 23 and 34 produce U^{n+1} itself, the others dU.
__host__ __device__ __forceinline__ bool first_kind(int kind) {
  return kind == 1 || kind == 11 || kind == 21 || kind == 31;
}
__host__ __device__ __forceinline__ bool final_kind(int kind) {
  return kind == 0 || kind == 3 || kind == 14 || kind == 23 || kind == 34;
}
__host__ __device__ __forceinline__ bool direct_kind(int kind) { return kind == 23 || kind == 34; }

// Inputs of one cell's stage update that do not depend on the residual: U^n, the stage state
// (RK3 stages 2 and 3) and 1/A.  Loaded ahead of the residual gather so that both sets of loads
// are in flight together.
struct StageIn {
  double Un[4], Sk[4], invA;
};

__device__ __forceinline__ void load_stage_in(const DevMesh &m, const DevState &st, int c, int kind, StageIn &in) {
  const int NP = m.NP, NT = m.NT;
  in.invA = m.inv_area[c];
#pragma unroll
  for (int k = 0; k < 4; k++) in.Un[k] = st.U[k * NT + c];
  if (kind == 2 || kind == 3 || kind == 22 || kind == 23) {
#pragma unroll
    for (int k = 0; k < 4; k++) in.Sk[k] = st.S[k * NP + c];
  }
}

// out: the stage state, or (final stages, true returned) dU or U^{n+1} itself.
__device__ __forceinline__ bool stage_values(const DevMesh &m, const DevState &st, int c, int kind, double dt,
                                             const double Rk[4], const double Un[4], const StageIn &in, double out[4]) {
  const int NP = m.NP;
  const double invA = in.invA;
  bool final_stage = false;
  if (kind == 1 || kind == 21) {
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = Un[k] - dt * invA * Rk[k];
  } else if (kind == 2 || kind == 22) {
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = 0.25 * (in.Sk[k] + 3.0 * Un[k] - dt * invA * Rk[k]);
  } else if (kind == 3) {
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = (2.0 / 3.0) * (in.Sk[k] - Un[k] - dt * invA * Rk[k]);
    final_stage = true;
  } else if (kind == 0) {
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = -dt * invA * Rk[k];
    final_stage = true;
  } else if (kind == 23) {
    // tvd_rk3_kernel stage 3 (CUDA_KERNELS/Time_Integration_Cuda_Kernels.cu:125-130):
    // U^{n+1} = (1/3)(U^n + 2 U2 - 2 dt/V R(U2)).
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = (1.0 / 3.0) * (Un[k] + 2.0 * in.Sk[k] - 2.0 * dt * invA * Rk[k]);
    final_stage = true;
  } else if (kind == 31 || kind == 32) {
    // rk4_complete_kernel stages 1-2 (CUDA_KERNELS/Time_Integration_Cuda_Kernels.cu:43-56): the
    // stage state is U^n - dt/(2V) R of the previous stage state (its dissipation terms are zero
    // for the inviscid path).
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = Un[k] - 0.5 * dt * invA * Rk[k];
  } else if (kind == 33) {
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = Un[k] - dt * invA * Rk[k];
  } else if (kind == 34) {
    // Stage 4 (:64-72): U^{n+1} = U^n - dt/(6V) R(U3), the last stage's residual only.
#pragma unroll
    for (int k = 0; k < 4; k++) out[k] = Un[k] - (dt * invA / 6.0) * Rk[k];
    final_stage = true;
  } else if (kind == 11) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      st.Racc[k * NP + c] = Rk[k];
      out[k] = Un[k] - 0.5 * (dt * invA) * Rk[k];
    }
  } else if (kind == 12 || kind == 13) {
    const double w = (kind == 12) ? 0.5 : 1.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      st.Racc[k * NP + c] = st.Racc[k * NP + c] + 2.0 * Rk[k];
      out[k] = Un[k] - w * (dt * invA) * Rk[k];
    }
  } else {  // 14
#pragma unroll
    for (int k = 0; k < 4; k++) {
      double acc = st.Racc[k * NP + c] + Rk[k];
      out[k] = -((dt * invA) * acc) / 6.0;
    }
    final_stage = true;
  }
  return final_stage;
}

__device__ __forceinline__ void cell_update_in(const DevMesh &m, const DevState &st, int c, int kind, double dt,
                                               const double Rk[4], const StageIn &in, int fuse_final, int keep_delu,
                                               double e[8]) {
  const int NP = m.NP, NT = m.NT;
  double Un[4], out[4];
#pragma unroll
  for (int k = 0; k < 4; k++) Un[k] = in.Un[k];
  const bool final_stage = stage_values(m, st, c, kind, dt, Rk, Un, in, out);
  if (!final_stage) {
#pragma unroll
    for (int k = 0; k < 4; k++) st.S[k * NP + c] = out[k];
    Prim q;
    bool ok = eos_prim(out[0], out[1], out[2], out[3], q);
    store_prim(st.prim, st.q4, NT, c, q);
    if (!ok) flag_bad(st.status, c);
  } else {
    // dU and U^{n+1}: the forms that produce U^{n+1} directly keep it exactly (dU = U^{n+1} - U^n
    // is stored for Estimate_Error, and U^{n+1} is parked in the stage state for Update()).
    const bool direct = direct_kind(kind);
    double du[4], nu[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      du[k] = direct ? out[k] - Un[k] : out[k];
      nu[k] = direct ? out[k] : Un[k] + out[k];
    }
    if (keep_delu || !fuse_final) {
#pragma unroll
      for (int k = 0; k < 4; k++) st.dU[k * NP + c] = du[k];
    }
    if (direct && !fuse_final) {
#pragma unroll
      for (int k = 0; k < 4; k++) st.S[k * NP + c] = nu[k];
    }
    if (fuse_final) {
#pragma unroll
      for (int k = 0; k < 4; k++) {
        e[k] += err_term(du[k], Un[k]);  // callers start e at 0 (strided callers sum their cells)
        e[4 + k] += Rk[k] * Rk[k];
        st.U[k * NT + c] = nu[k];
        Un[k] = nu[k];
      }
      Prim q;
      bool ok = eos_prim(Un[0], Un[1], Un[2], Un[3], q);
      store_prim(st.prim, st.q4, NT, c, q);
      if (!ok) flag_bad(st.status, c);
    }
  }
}

__device__ __forceinline__ void cell_update(const DevMesh &m, const DevState &st, int c, int kind, double dt,
                                            const double Rk[4], int fuse_final, int keep_delu, double e[8]) {
  StageIn in;
  load_stage_in(m, st, c, kind, in);
  cell_update_in(m, st, c, kind, dt, Rk, in, fuse_final, keep_delu, e);
}

// lts: 0 Min_dt, 1 Cell::del_t (reference stage 1 only), 2 dt frozen per cell at the first stage,
// 3 Min_dt frozen at the first stage.
// flags (StageFlags): the owner thread writes its ghosts for the next evaluation (GHOSTS), with
// kStageNextStep those of the next pseudo-step's first one; kStageNoNorms leaves the norms out (10 us of the
// last stage's 22 on 524,288 cells).  Bound by its traffic (168 - 232 bytes per cell): 64 registers, 14 us per
// launch on 524,288 cells.  With the boundary kinds (GHOSTS) it takes 94, half the warps per SM and 24 us
// there, but saves the k_bc launches, which pays on small meshes: see stage_ghosts_for.  (As a function that is
// not inlined they leave the kernel at 64 registers; 1.01 - 1.04 x faster on 180,000 cells, 0.95 on 24,000.)
template <bool GHOSTS>
__global__ void __launch_bounds__(kBlock, GHOSTS ? 1 : 4) k_stage(const __grid_constant__ DevMesh m, const __grid_constant__ DevState st,
                                                  const __grid_constant__ BcParams bp, int kind, int lts,
                                                  int fuse_final, int keep_delu, int flags) {
  pdl_enter();
  const int NP = m.NP;
  const int c = item_index(m.cblk, NP);
  const bool done = step_done(st.ctl);
  const bool active = c < NP && !done;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const double dtmin = st.ctl[CTL_DTMIN];
  if (active) {
    const bool first = first_kind(kind);
    if (first) {
      if (lts == 2) st.dtk[c] = st.dtc[c];
    }
    double dt;
    if (lts == 0) dt = dtmin;
    else if (lts == 1) dt = st.dtc[c];
    else if (lts == 2) dt = first ? st.dtc[c] : st.dtk[c];
    else dt = first ? dtmin : st.ctl[CTL_DTSTEP];
    double Rk[4];
#pragma unroll
    for (int k = 0; k < 4; k++) Rk[k] = st.R[k * NP + c];
    cell_update(m, st, c, kind, dt, Rk, fuse_final, keep_delu, e);
  }
  if (first_kind(kind) && blockIdx.x == 0 && threadIdx.x == 0 && !done) st.ctl[CTL_DTSTEP] = dtmin;
  if (fuse_final && final_kind(kind)) {
    if (done) return;
    const double dt_time = (lts >= 2) ? st.ctl[CTL_DTSTEP] : dtmin;
    if (GHOSTS || (flags & kStageNoNorms)) {  // only without t_end
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        st.ctl[CTL_TOTAL_TIME] += dt_time;
        st.ctl[CTL_ITER] += 1.0;
      }
    } else {
      reduce_err_and_epilogue(st, e, true, dt_time);
    }
  }
  if (GHOSTS && active) {
    const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
    const int cur_S = (flags & kStageGhosts) ? 1 : 0;
    for (int i = b0; i < b1; i++) bc_entry(m, st, bp, m.bidx[i], (cur_S && (flags & kStageExitS)) ? 1 : 0, cur_S);
  }
}

// Stage update of cell c from its residual R, shared by the gather and patch forms: stores R,
// takes the stage dt (lts 1: del_t of this evaluation; else del_t frozen at the first stage),
// updates the cell, and with flags bit 1 writes the next stage's ghost states from the owner
// thread (every ghost depends only on its owner cell's new state: Apply_Boundary_Conditions of the
// next stage).  Returns the dt used.
// stage_cell_in: the same with the stage inputs and the frozen dt already loaded (the TMA tile
// form prefetches them into shared memory).
__device__ __forceinline__ double stage_cell_in(const DevMesh &m, const DevState &st, const BcParams &bp, int c,
                                                const double R[4], double dtc, double dt_frozen, const StageIn &in,
                                                int kind, int lts, int fuse_final, int keep_delu, int flags,
                                                double e[8]) {
  const int NP = m.NP;
  const bool first = first_kind(kind);
#pragma unroll
  for (int k = 0; k < 4; k++) st.R[k * NP + c] = R[k];
  double dt;
  if (lts == 1) dt = dtc;
  else {
    if (first) st.dtk[c] = dtc;
    dt = first ? dtc : dt_frozen;
  }
  cell_update_in(m, st, c, kind, dt, R, in, fuse_final, keep_delu, e);
  if ((flags & 2) && !final_kind(kind)) {
    const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
    for (int i = b0; i < b1; i++) bc_entry(m, st, bp, m.bidx[i], (flags & 4) ? 1 : 0, 1);
  }
  return dt;
}
__device__ __forceinline__ double stage_cell(const DevMesh &m, const DevState &st, const BcParams &bp, int c,
                                             const double R[4], double dtc, int kind, int lts, int fuse_final,
                                             int keep_delu, int flags, double e[8]) {
  StageIn in;
  load_stage_in(m, st, c, kind, in);
  const double dt_frozen = (lts != 1 && !first_kind(kind)) ? st.dtk[c] : 0.0;
  return stage_cell_in(m, st, bp, c, R, dtc, dt_frozen, in, kind, lts, fuse_final, keep_delu, flags, e);
}

// Last stage of the fused forms: Estimate_Error's terms, the residual squares and the step's dt
// (the minimum of the per-cell dt frozen at the first stage, i.e. that stage's Min_dt), reduced
// over the grid, then the Total_Time epilogue of the loop body.  Called by every thread.
// stage_final_reduce_sm: the same with its scratch (32 + 8 * 32 + 9 doubles) in caller-provided
// shared memory.
__device__ __forceinline__ void stage_final_reduce_sm(const DevState &st, const double e[8], double dtu, double *scratch) {
  double *sh = scratch, *sh8 = scratch + 32, *red = scratch + 32 + 8 * 32;
  const double sq = block_sums8(e, sh8);
  if (threadIdx.x < 8) st.partial[(1 + threadIdx.x) * gridDim.x + blockIdx.x] = sq;
  const double bm = block_min(dtu, sh);
  if (threadIdx.x == 0) st.partial[blockIdx.x] = bm;
  if (grid_reduce9(st, red) && threadIdx.x == 0) {
    st.ctl[CTL_DTMIN] = red[0];
    st.ctl[CTL_DTSTEP] = red[0];
    for (int q = 0; q < 8; q++) st.ctl[q < 4 ? CTL_ERR + q : CTL_RES + q - 4] = sqrt(red[1 + q]);
    double t = st.ctl[CTL_TOTAL_TIME] + red[0];
    st.ctl[CTL_TOTAL_TIME] = t;
    st.ctl[CTL_ITER] += 1.0;
    double te = st.ctl[CTL_TEND];
    if (te > 0.0 && t >= te) st.ctl[CTL_DONE] = 1.0;
  }
}
__device__ __forceinline__ void stage_final_reduce(const DevState &st, const double e[8], double dtu) {
  __shared__ double scratch[32 + 8 * 32 + 9];
  stage_final_reduce_sm(st, e, dtu, scratch);
}

// Face-based forms with a per-cell time step (lts 1 or 2): the gather of k_gather and the stage
// update of k_stage in one pass, so the residual never leaves registers on its way to the update
// (it is still stored for downloads).  At the final stage the error norms, the step's Min_dt and
// the Total_Time epilogue.
// 80 registers (6 blocks of 128 per SM, 24 warps) without spilling; the unbounded build takes 84
// (5 blocks) and measured 9 % slower on B200.
// STRIDED (the reducing last stage without work lists): a grid of one wave strides over the
// cells, so the per-block fence and arrival count of the grid reduction is paid once per resident
// block instead of once per 128 cells; each thread sums its cells' terms in cell order and the
// grid is fixed per device, so the sums are reproducible.  Its accumulators spill 64 bytes at the
// same 80-register cap, which measured faster than 96 registers at 5 blocks per SM.
template <bool STRIDED, bool FF>
__global__ void __launch_bounds__(kFluxBlock, 6) k_gather_stage(DevMesh m, DevState st, FluxParams fp,
                                                                             BcParams bp, int kind, int lts,
                                                                             int fuse_final, int keep_delu, int flags) {
  pdl_enter();
  const int NP = m.NP;
  if (step_done(st.ctl)) return;
  double dtu = 1e308 * 10.0;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (!STRIDED) {
    const int c = item_index(m.cblk, NP);
    if (c < NP) {
      // The residual gather is issued first; loading the state rows ahead of it (more registers,
      // fewer resident warps) measured slower on B200.
      double R[4], den = 0.0;
      gather_faces<false, false, FF>(m, st, c, R, den);
      const double dtc = (lts == 1 || first_kind(kind)) ? st.dtc[c] : 0.0;  // the only stages that use it
      dtu = stage_cell(m, st, bp, c, R, dtc, kind, lts, fuse_final, keep_delu, flags, e);
    }
  } else {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < NP; c += gridDim.x * blockDim.x) {
      double R[4], den = 0.0;
      gather_faces<false, false, FF>(m, st, c, R, den);
      const double dtc = (lts == 1 || first_kind(kind)) ? st.dtc[c] : 0.0;
      const double dt = stage_cell(m, st, bp, c, R, dtc, kind, lts, fuse_final, keep_delu, flags, e);
      dtu = dt < dtu ? dt : dtu;
    }
  }
  if (fuse_final && final_kind(kind)) stage_final_reduce(st, e, dtu);
}

// Values a boundary state is formed from right after the cell's update: the state in registers.
struct BcRegs {
  const DevMesh &m;
  int c, f, e;
  double av;
  const double *W, *X;  // current state, exit-copy source
  const double4 *bstate;
  const double *bexit;
  __device__ __forceinline__ double nx() const { return m.nx[f * m.NP + c]; }
  __device__ __forceinline__ double ny() const { return m.ny[f * m.NP + c]; }
  __device__ __forceinline__ double a() const { return av; }
  __device__ __forceinline__ double cur(int k) const { return W[k]; }
  __device__ __forceinline__ double src(int k) const { return X[k]; }
};

// k_gather_stage for the stages whose residual, primitive planes and norms nobody can read before they
// are formed again: every stage but the last, and the last stage of every pseudo-step but the last of a
// call without t_end.  It leaves out those stores (R 32 bytes, three or four primitive planes of 8, dU)
// and, in the last stage, all of the reduction but the step's Min_dt; the rows q4, the states, the frozen
// dt, the sound speed (where the next gradient pass forms del_t) and the ghosts stay.  201 - 233 bytes per
// cell, the 64 of its fluxes among them; bound by the latency of the face slots and of the fluxes they name (16 - 18
// long-scoreboard stalls per issue, DRAM 32 % busy): 28 us on 524,288 cells against k_gather_stage's 35.6.
// Six blocks per SM: 53.1 us on 1,038,240 mixed cells, 28.0 on 524,288; seven 54.7 and 27.7, five and
// eight slower.  A persistent loop with the next cell's face slots loaded ahead took 32.0 us, loading the
// stage inputs before the fluxes and the branch-free EOS gained nothing (B200).
// MODE 0: not the last stage; 1: the last stage (one wave of blocks strides over the cells when there are
// no work lists).
template <int MODE, bool FF>
__global__ void __launch_bounds__(kFluxBlock, 6) k_gather_lean(DevMesh m, DevState st, BcParams bp, int kind, int flags,
                                                              int store_a) {
  pdl_enter();
  const int NP = m.NP, NT = m.NT;
  if (step_done(st.ctl)) return;
  double dtu = 1e308 * 10.0;
  const int step = (MODE == 1 && !m.cblk) ? gridDim.x * blockDim.x : NP;
  for (int c = item_index(m.cblk, NP); c < NP; c += step) {
    const int info = m.nfb[c];
    const int4 e4 = m.cface4[c];
    const double4 F0 = load_flux<FF>(st, face_id(e4.x)), F1 = load_flux<FF>(st, face_id(e4.y)),
                  F2 = load_flux<FF>(st, face_id(e4.z)), F3 = load_flux<FF>(st, face_id(e4.w));
    StageIn in;
    load_stage_in(m, st, c, kind, in);
    const bool first = first_kind(kind);
    const double dt = first ? st.dtc[c] : st.dtk[c];
    double R[4], out[4];
    sum_faces(info & 7, e4, F0, F1, F2, F3, R);
    const bool fin = stage_values(m, st, c, kind, dt, R, in.Un, in, out);
    if (first) st.dtk[c] = dt;
    if (MODE == 1 && fin && !direct_kind(kind)) {
#pragma unroll
      for (int k = 0; k < 4; k++) out[k] = in.Un[k] + out[k];
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (MODE == 1) st.U[(size_t)k * NT + c] = out[k];
      else st.S[(size_t)k * NP + c] = out[k];
    }
    Prim q;
    const bool ok = eos_prim(out[0], out[1], out[2], out[3], q);
    st32(st.q4 + c, make_double4(q.rho, q.u, q.v, q.p));
    if (MODE == 1 || store_a) st.prim[4 * (size_t)NT + c] = q.a;
    if (!ok) flag_bad(st.status, c);
    if (MODE == 0 && (info & kHasEntries)) {
      const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
      for (int i = b0; i < b1; i++) {
        const int e = m.bidx[i];
        const int4 b = m.bnd[e];
        const BcRegs src{m, c, b.z, e, q.a, out, (flags & 4) ? out : in.Un, m.bstate, m.bexit};
        double G[4];
        if (bc_values(src, bp, b.x, q.rho, q.u, q.v, q.p, G)) store_ghost(st, NT, b.w, G);
      }
    }
    if (MODE == 1) dtu = dt < dtu ? dt : dtu;
  }
  if (MODE == 1) {
    __shared__ double sh[32];
    const double bm = block_min(dtu, sh);
    if (threadIdx.x == 0) st.partial[blockIdx.x] = bm;
    if (last_block(st.counter)) {
      double v = 1e308 * 10.0;
#pragma unroll 8
      for (int i = threadIdx.x; i < (int)gridDim.x; i += kFluxBlock) {
        const double w = __ldcg(&st.partial[i]);
        v = w < v ? w : v;
      }
      v = block_min(v, sh);
      if (threadIdx.x == 0) {
        st.ctl[CTL_DTMIN] = v;
        st.ctl[CTL_DTSTEP] = v;
        st.ctl[CTL_TOTAL_TIME] += v;
        st.ctl[CTL_ITER] += 1.0;
        *st.counter = 0u;
      }
    }
  }
}

// The FP32-flux form's face records.
__global__ void k_face_records(DevMesh m, float4 *r) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)m.NF) return;
  const double4 g = m.fg4[i];
  const int2 on = m.fon[i];
  r[2 * i] = make_float4(float(g.x), float(g.y), float(g.z), float(g.w));
  r[2 * i + 1] = make_float4(float(m.fdy[i]), __int_as_float(on.x), __int_as_float(on.y), 0.0f);
}

// Weights of the gradient passes: (nx dl, ny dl) of every face slot.
__global__ void k_face_weights(DevMesh m, double2 *gw) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 4 * (size_t)m.NP) gw[i] = make_double2(m.nx[i] * m.dl[i], m.ny[i] * m.dl[i]);
}

// Estimate_Error alone (src/Error_Estimate_Update.cpp:10-28).
__global__ void __launch_bounds__(kBlock) k_error(DevMesh m, DevState st) {
  const int NP = m.NP, NT = m.NT;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c < NP) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      e[k] = err_term(st.dU[k * NP + c], st.U[k * NT + c]);
      double r = st.R[k * NP + c];
      e[4 + k] = r * r;
    }
  }
  reduce_err_and_epilogue(st, e, false, 0.0);
}

// Update() (src/Error_Estimate_Update.cpp:31-43): U += dU, primitives refreshed.
// from_S: the integrator produced U^{n+1} itself (reference GPU forms), parked in the stage state.
__global__ void __launch_bounds__(kBlock) k_update(DevMesh m, DevState st, int from_S) {
  const int NP = m.NP, NT = m.NT;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= NP) return;
  double u[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    u[k] = from_S ? st.S[k * NP + c] : st.U[k * NT + c] + st.dU[k * NP + c];
    st.U[k * NT + c] = u[k];
  }
  Prim q;
  bool ok = eos_prim(u[0], u[1], u[2], u[3], q);
  store_prim(st.prim, st.q4, NT, c, q);
  if (!ok) flag_bad(st.status, c);
}

// Calculate_Gradient_At_Cell_Center (src/Grid_Refine_Functions.cpp:221-246); var indexes the
// device primitive planes (0 rho, 1 u, 2 v, 3 p, 4 a).
__device__ __forceinline__ void gg_gradient(const DevMesh &m, const double *q, int c, double &g0, double &g1) {
  g0 = 0.0;
  g1 = 0.0;
  const int nf = m.nf[c];
  if (nf <= 0 || m.area[c] <= 0.0) return;
  const double pc = q[c];
  for (int f = 0; f < nf; f++) {
    const int idx = f * m.NP + c;
    const int N = m.nbr[idx];
    double pn = pc;
    if (N >= 0 && N < m.NP) pn = q[N];
    const double pf = 0.5 * (pc + pn);
    g0 += pf * m.nx[idx] * m.dl[idx];
    g1 += pf * m.ny[idx] * m.dl[idx];
  }
  g0 *= m.inv_area[c];
  g1 *= m.inv_area[c];
}

// One face's part of a cell's Green-Gauss sums g (its four variables) and, with DT, of the denominator of
// del_t (Inviscid_Time_Step, src/Time_Step.cpp:293-329).
template <bool DT>
__device__ __forceinline__ void gg_face(const double qc[4], double ac, const double qn[4], double nx, double ny,
                                        double dl, double g[8], double &den) {
  const double wx = nx * dl, wy = ny * dl;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double qf = 0.5 * (qc[k] + qn[k]);
    g[2 * k] += qf * wx;
    g[2 * k + 1] += qf * wy;
  }
  if (DT) {
    const double vnf = qc[1] * nx + qc[2] * ny;
    den += (fabs(vnf) + ac) * dl;
  }
}

// Green-Gauss gradients of (rho, u, v, p) of physical cell c from the primitive planes `prim`
// ([5][NT]), multiplied by 1/A (g[2k], g[2k+1]: d/dx, d/dy of variable k), and with DT the
// denominator of del_t (Inviscid_Time_Step, src/Time_Step.cpp:293-329, faces in order).  The
// four neighbour slots come in one 16-byte load without waiting for the face count (an unused
// slot reads the cell itself), so every neighbour's loads are in flight together; the sums run
// over the cell's faces in order.
// q4 is not __restrict__: the first-stage gradient pass writes the ghost rows it then reads.
template <bool DT, bool Q4 = false>
__device__ __forceinline__ void cell_gradients(const DevMesh &m, const double *prim, const double4 *q4, int c,
                                               const double qc[4], double g[8], double &den) {
  const int NP = m.NP, NT = m.NT;
  const int nf = m.nf[c];
  const double ia = m.inv_area[c];
  const double ac = DT ? prim[4 * NT + c] : 0.0;
  const int4 n4 = m.nbr4[c];
  const int nr[4] = {n4.x, n4.y, n4.z, n4.w};
  int nb[4];
#pragma unroll
  for (int f = 0; f < 4; f++) nb[f] = (nr[f] >= 0 && nr[f] < NT) ? nr[f] : c;
  double qn[4][4];
#pragma unroll
  for (int f = 0; f < 4; f++) {
    if (Q4) {
      const double4 v = ld32_ordered(q4 + nb[f]);
      qn[f][0] = v.x;
      qn[f][1] = v.y;
      qn[f][2] = v.z;
      qn[f][3] = v.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) qn[f][k] = prim[k * NT + nb[f]];
    }
  }
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = 0.0;
  den = 0.0;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    if (f >= nf) break;
    const int idx = f * NP + c;
    gg_face<DT>(qc, ac, qn[f], m.nx[idx], m.ny[idx], m.dl[idx], g, den);
  }
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = g[k] * ia;
}

// The gradients alone, from the faces' weights (nx dl, ny dl; the products cell_gradients forms, made once
// with the context): 64 bytes of geometry per cell instead of 96.
__device__ __forceinline__ void cell_gradients_w(const DevMesh &m, const double4 *q4, int c, const double qc[4],
                                                 double g[8]) {
  const int NP = m.NP, NT = m.NT;
  const int nf = m.nfb[c] & 7;
  const int4 n4 = m.nbr4[c];
  const double ia = m.inv_area[c];
  const int nr[4] = {n4.x, n4.y, n4.z, n4.w};
  double4 v[4];
#pragma unroll
  for (int f = 0; f < 4; f++) v[f] = ld32_ordered(q4 + ((nr[f] >= 0 && nr[f] < NT) ? nr[f] : c));
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = 0.0;
#pragma unroll
  for (int f = 0; f < 4; f++) {
    if (f >= nf) break;
    const double2 w = m.gw[(size_t)f * NP + c];
    const double qn[4] = {v[f].x, v[f].y, v[f].z, v[f].w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double qf = 0.5 * (qc[k] + qn[k]);
      g[2 * k] += qf * w.x;
      g[2 * k + 1] += qf * w.y;
    }
  }
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = g[k] * ia;
}

// Gradient records of the face-based forms: the Green-Gauss gradients of (rho, u, v, p) of every
// physical cell, the face value being the mean of the two cell values (a ghost neighbour's value
// carries the boundary state); the states themselves are read from q4.  Work-list entries cover
// record rows NP..NT-1 too (ghost rows), which have nothing to do.
// DT: also del_t of each physical cell (the fused per-cell-dt forms; their Min_dt is formed in
// the last stage's reduction).
// with_bc: first stage of a step; each thread first applies the boundary conditions of its own
// cell's boundary entries (Apply_Boundary_Conditions, as k_bc does), which is exact because a
// ghost row depends only on its owner cell and is read by no other cell's gradient.
// Bound by the latency of its two dependent loads (neighbour slots, then their rows), most of them from
// DRAM: each block first starts bringing what a block one per SM later reads (grad_ahead) into L2, which
// takes a pseudo-step of 524,288 cells from 246.6 to 241 us (FP32-flux 212 to 204.5), 245,000 cells from
// 134 to 131.8 us; at 125,000 cells, in L2 anyway, 75.8 to 76.7, so meshes below two waves leave it out
// (B200).  The same in the face and gather kernels gained nothing: their fluxes and rows are mostly in L2.
template <bool DT>
__global__ void __launch_bounds__(kBlock, 4) k_muscl_gradients(DevMesh m, DevState st, FluxParams fp, BcParams bp,
                                                               int with_bc) {
  pdl_enter();
  const int c = item_index(m.rblk, m.NT);
  const int NP = m.NP;
  if (step_done(st.ctl)) return;
  if (m.grad_ahead > 0 && threadIdx.x < (DT ? 17 : 7)) {
    const int w = blockIdx.x + m.grad_ahead, t = threadIdx.x;
    int c0 = w * kBlock, n = min(kBlock, NP - c0);
    if (m.rblk) {
      const int2 r = w < m.n_rblk ? m.rblk[w] : make_int2(0, 0);
      c0 = r.x;
      n = min(r.y, NP) - r.x;
    }
    if (n > 0) {
      if (t == 0) prefetch_l2(m.nbr4, (size_t)c0 * 16, n * 16);
      else if (t == 1) prefetch_l2(st.q4, (size_t)c0 * 32, n * 32);
      else if (t == 2) prefetch_l2(m.inv_area, (size_t)c0 * 8, n * 8);
      else if (!DT) prefetch_l2(m.gw, ((size_t)(t - 3) * NP + c0) * 16, n * 16);
      else if (t < 7) prefetch_l2(m.nx, ((size_t)(t - 3) * NP + c0) * 8, n * 8);
      else if (t < 11) prefetch_l2(m.ny, ((size_t)(t - 7) * NP + c0) * 8, n * 8);
      else if (t < 15) prefetch_l2(m.dl, ((size_t)(t - 11) * NP + c0) * 8, n * 8);
      else if (t == 15) prefetch_l2(m.area, (size_t)c0 * 8, n * 8);
      else prefetch_l2(st.prim, ((size_t)4 * m.NT + c0) * 8, n * 8);
    }
  }
  if (c < NP) {
    if (with_bc && (m.nfb[c] & kHasEntries)) {
      const double4 q = ld32_ordered(st.q4 + c);
      const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
      for (int i = b0; i < b1; i++) bc_entry_row(m, st, bp, m.bidx[i], q);
    }
    const double4 v = ld32_ordered(st.q4 + c);
    const double qc[4] = {v.x, v.y, v.z, v.w};
    double g[8], den;
    if (DT) cell_gradients<true, true>(m, st.prim, st.q4, c, qc, g, den);
    else cell_gradients_w(m, st.q4, c, qc, g);
    if (st.recf) {
      st32f(st.recf + 2 * (size_t)c, g);
    } else {
      double4 *r = reinterpret_cast<double4 *>(st.rec + 8 * (size_t)c);
      st32(r, make_double4(g[0], g[1], g[2], g[3]));
      st32(r + 1, make_double4(g[4], g[5], g[6], g[7]));
    }
    if (DT) st.dtc[c] = cell_dt(m, fp, c, den);
  }
}

// ---- Persistent form of one stage for batched solves (no reference counterpart) ----
// One cooperative launch per RK stage does the work of k_muscl_gradients, k_faces and
// k_gather_stage: its resident thread blocks walk the (instance, block) work lists of the active
// instances (record rows, faces, cells), phase after phase, with a grid barrier between the
// phases.  Values written in the same launch by other blocks (records, ghost rows, del_t, face
// fluxes) are read from L2.  Every per-cell and per-face operation is the one the three kernels
// do, so the state is bit-identical to theirs; the error norms of the last stage are reduced over
// the persistent blocks (a different summation order than the three-kernel grid).
//
// The barrier waits are bounded: a block that waits longer than kBarrierCycles (about half a
// second) records CFD_ERR_TIMEOUT in the status word and goes on; once the status is set no block
// waits again, so the launch always ends and the host reads the error.  test_arrivals adds
// arrivals that never come (a test of the timeout path; 0 in every run).
constexpr long long kBarrierCycles = 1ll << 30;
constexpr int kPersistBlock = 128;

__device__ __forceinline__ void grid_barrier(unsigned int *count, unsigned int *gen, int *status,
                                             unsigned int test_arrivals) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int *vgen = gen;
    volatile int *vstatus = status;
    const unsigned int g = *vgen;
    __threadfence();
    const unsigned int arrived = atomicAdd(count, 1u) + 1u;
    if (arrived == gridDim.x + test_arrivals) {
      atomicExch(count, 0u);
      __threadfence();
      atomicAdd(gen, 1u);
    } else {
      const long long t0 = clock64();
      while (*vgen == g) {
        if (*vstatus != 0) break;
        if (clock64() - t0 > kBarrierCycles) {
          atomicCAS(status, 0, 5 /* CFD_ERR_TIMEOUT */);
          break;
        }
        __nanosleep(128);
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// MINB: resident blocks per SM the registers are allocated for (4: 116 registers, no spill; 6: 80
// registers and a small spill, 24 warps per SM; 8: 64 registers).  On a batch of 128 ramps on B200
// the FP64 form runs fastest at 6 (25 % faster than at 4) and the FP32-flux form at 8.
template <typename T, int DISS, int MINB>
__global__ void __launch_bounds__(kPersistBlock, MINB) k_persistent_stage(const __grid_constant__ DevMesh m, const __grid_constant__ DevState st,
                                                                       const __grid_constant__ FluxParams fp, BcParams bp, int kind, int lts, int fuse_final,
                                                                       int keep_delu, int flags, int with_dt,
                                                                       int with_bc, unsigned int test_arrivals) {
  const int NP = m.NP;
  if (step_done(st.ctl)) return;  // every block sees the same flag (written by an earlier launch)
  unsigned int *bar_count = st.counter + 4, *bar_gen = st.counter + 5;
  // Phase 1: gradient records (and del_t), the first stage's boundary conditions.
  // Without work lists (a single solve) the phases walk all rows, faces and cells in chunks.
  const int nr = m.rblk ? m.n_rblk : (NP + kWorkItemBlock - 1) / kWorkItemBlock;
  const int nfb = m.fblk ? m.n_fblk : (m.NF + kWorkFaceBlock - 1) / kWorkFaceBlock;
  const int ncb = m.cblk ? m.n_cblk : (NP + kWorkCellBlock - 1) / kWorkCellBlock;
  for (int w = blockIdx.x; w < nr; w += gridDim.x) {
    const int2 b = m.rblk ? m.rblk[w] : make_int2(w * kWorkItemBlock, min((w + 1) * kWorkItemBlock, NP));
    for (int c = b.x + threadIdx.x; c < b.y; c += blockDim.x) {
      if (c >= NP) continue;
      if (with_bc) {
        const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
        for (int i = b0; i < b1; i++) bc_entry(m, st, bp, m.bidx[i], 0, 0);
      }
      const double4 v = st.q4[c];
      const double qc[4] = {v.x, v.y, v.z, v.w};
      double g[8], den;
      if (with_dt) cell_gradients<true, true>(m, st.prim, st.q4, c, qc, g, den);
      else cell_gradients<false, true>(m, st.prim, st.q4, c, qc, g, den);
      if (st.recf) {
        float4 *r = st.recf + 2 * (size_t)c;
        r[0] = make_float4(float(g[0]), float(g[1]), float(g[2]), float(g[3]));
        r[1] = make_float4(float(g[4]), float(g[5]), float(g[6]), float(g[7]));
      } else {
        double4 *r = reinterpret_cast<double4 *>(st.rec + 8 * (size_t)c);
        r[0] = make_double4(g[0], g[1], g[2], g[3]);
        r[1] = make_double4(g[4], g[5], g[6], g[7]);
      }
      if (with_dt) st.dtc[c] = cell_dt(m, fp, c, den);
    }
  }
  grid_barrier(bar_count, bar_gen, st.status, test_arrivals);
  // Phase 2: face fluxes.
  const int glim = fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter;
  for (int w = blockIdx.x; w < nfb; w += gridDim.x) {
    const int2 b = m.fblk ? m.fblk[w] : make_int2(w * kWorkFaceBlock, min((w + 1) * kWorkFaceBlock, m.NF));
    for (int i = b.x + threadIdx.x; i < b.y; i += blockDim.x) {
      const int2 on = m.fon[i];
      const int c = on.x, N = on.y;
      const double4 gq = m.fg4[i];
      const T nx = T(gq.x), ny = T(gq.y), dl = T(gq.z), dx = T(gq.w), dy = T(m.fdy[i]);
      const double4 c0 = ldcg4(st.q4 + c), n0 = ldcg4(st.q4 + N);
      const bool nphys = N < NP;
      double4 c1, c2, n1, n2;
      if (sizeof(T) == sizeof(float)) {
        const float4 a = __ldcg(st.recf + 2 * (size_t)c), bb = __ldcg(st.recf + 2 * (size_t)c + 1);
        c1 = make_double4(a.x, a.y, a.z, a.w);
        c2 = make_double4(bb.x, bb.y, bb.z, bb.w);
        if (nphys) {
          const float4 p = __ldcg(st.recf + 2 * (size_t)N), q = __ldcg(st.recf + 2 * (size_t)N + 1);
          n1 = make_double4(p.x, p.y, p.z, p.w);
          n2 = make_double4(q.x, q.y, q.z, q.w);
        } else {
          n1 = c1;
          n2 = c2;
        }
      } else {
        const double4 *rc = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)c);
        const double4 *rn = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)N);
        c1 = ldcg4(rc);
        c2 = ldcg4(rc + 1);
        n1 = nphys ? ldcg4(rn) : c1;
        n2 = nphys ? ldcg4(rn + 1) : c2;
      }
      FaceOps<T> o;
      double4 F = face_flux_rec<T, DISS>(o, glim, c0, c1, c2, n0, n1, n2, nx, ny, dl, dx, dy, T(fp.eflin),
                                         T(fp.shock_fix));
      if constexpr (FaceOps<T>::fast) {
        if (o.bad()) F = face_flux_again<DISS>(m, st, fp, i);
      }
      st.F[i] = F;
    }
  }
  grid_barrier(bar_count, bar_gen, st.status, test_arrivals);
  // Phase 3: gather of each cell's face fluxes in face order and the stage update.
  double dtu = 1e308 * 10.0;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int w = blockIdx.x; w < ncb; w += gridDim.x) {
    const int2 b = m.cblk ? m.cblk[w] : make_int2(w * kWorkCellBlock, min((w + 1) * kWorkCellBlock, NP));
    for (int c = b.x + threadIdx.x; c < b.y; c += blockDim.x) {
      double R[4], den = 0.0;
      gather_faces<false, true>(m, st, c, R, den);
      const double dtc = (lts == 1 || first_kind(kind)) ? __ldcg(st.dtc + c) : 0.0;
      const double dt = stage_cell(m, st, bp, c, R, dtc, kind, lts, fuse_final, keep_delu, flags, e);
      dtu = dt < dtu ? dt : dtu;
    }
  }
  if (fuse_final && final_kind(kind)) stage_final_reduce(st, e, dtu);
}

// ---- Whole pseudo-steps in one launch (small and mid-size meshes; no reference counterpart) ----
// On a few thousand cells a pseudo-step of the separate kernels is nine launches of a few microseconds,
// nearly all of it launch latency and chains of dependent loads (the index, the geometry it names, the
// count that says how many faces follow ...).  Here one cooperative launch, at most a block per SM, runs
// many pseudo-steps.  Every block keeps a fixed range of one instance's cells and faces whose geometry,
// connectivity, boundary entries and own states stay in shared memory; only what other blocks read goes
// through global memory: the (rho, u, v, p) rows, the gradient records and the face fluxes, one round of
// loads per phase.  A barrier over the instance's blocks separates the phases (gradients; face fluxes;
// gather and update): a single solve is one group of blocks, a batch one per active instance, with blocks
// in proportion to its cells.  Values written in the launch by other blocks are read after the barrier's
// acquire.  The operations are those of the separate kernels in the same order, so states, Min_dt and
// Total_Time are the same bits; the norms are summed over this grid's blocks (another order).  What the
// next step overwrites before anyone can read it (R, del_t's last evaluation, the primitive planes, the
// norms) is formed in the launch's last step alone unless a t_end may end the run at any step.
// (As one thread-block cluster with the hardware's cluster barrier, 2,048 cells took 25 us per
// pseudo-step exchanging through L2 and 30 us through the cluster's shared memory.)
struct StepsArgs {
  int n_steps, n_stages, kind0, keep_delu;
  int cells, faces, entries;  // shared-memory capacity per block
  int reduce;                 // norms, Min_dt and Total_Time (single solves)
  int may_stop;               // a t_end is set
  const StepsBlock *blocks;
  unsigned int *arrivals;     // [groups * kStepsBarrierStride], 0 before the launch, and the give-up flag
  unsigned int *gave_up;
  unsigned int test_arrivals;
};

// Barrier over the n blocks of one group: arrivals count up from 0 and every block polls the count itself,
// so the last arrival reaches the others in one hop.  The waits are bounded like grid_barrier's: a block
// that waits longer than kBarrierCycles records CFD_ERR_TIMEOUT and raises the give-up flag, after which
// no block of this context waits again, so the launch always ends.
__device__ __forceinline__ void steps_barrier(const DevState &st, const StepsArgs &a, unsigned int *count, unsigned int n,
                                              unsigned int &target) {
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned int *gave_up = a.gave_up;
    target += n;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    const long long t0 = clock64();
    for (;;) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      if (v >= target + a.test_arrivals) break;
      if (*gave_up) break;
      if (clock64() - t0 > kBarrierCycles) {
        atomicCAS(st.status, 0, 5 /* CFD_ERR_TIMEOUT */);
        *gave_up = 1u;
        break;
      }
    }
  }
  __syncthreads();
}

constexpr int kStepsThreads = 512;
// Shared memory of a block: per cell 12 geometry values, 1/A, U, the primitives (5), dt; per face 5 geometry
// values; the tables.
__host__ __device__ __forceinline__ size_t steps_smem(int cells, int faces, int entries) {
  return sizeof(double) * (23 * (size_t)cells + 5 * (size_t)faces) + sizeof(int4) * (2 * (size_t)cells + entries) +
         sizeof(int2) * (size_t)faces + sizeof(int) * (2 * (size_t)cells + 1);
}

// Values a boundary state is formed from when the cell's state is in shared memory (the current state is
// both the exit copy's source and the state the primitives came from).
struct BcShared {
  const double *geo, *q, *U;
  size_t ldU;
  int P, l, f, e;
  const double4 *bstate;
  const double *bexit;
  __device__ __forceinline__ double nx() const { return geo[(3 * f) * P + l]; }
  __device__ __forceinline__ double ny() const { return geo[(3 * f + 1) * P + l]; }
  __device__ __forceinline__ double a() const { return q[4 * P + l]; }
  __device__ __forceinline__ double cur(int k) const { return U[k * ldU + l]; }
  __device__ __forceinline__ double src(int k) const { return U[k * ldU + l]; }
};

template <typename T, int DISS>
__global__ void __launch_bounds__(kStepsThreads, 1) k_steps(const __grid_constant__ DevMesh m,
                                                            const __grid_constant__ DevState st,
                                                            const __grid_constant__ FluxParams fp,
                                                            const __grid_constant__ BcParams bp,
                                                            const __grid_constant__ StepsArgs a) {
  extern __shared__ __align__(16) double smd[];
  if (step_done(st.ctl)) return;
  const int NP = m.NP, NT = m.NT, P = a.cells, Q = a.faces;
  const StepsBlock blk = a.blocks[blockIdx.x];
  const int2 cr = make_int2(blk.c0, blk.c1), fr = make_int2(blk.f0, blk.f1);
  unsigned int *const count = a.arrivals + (size_t)blk.group * kStepsBarrierStride;
  const int nc = cr.y - cr.x, nfc = fr.y - fr.x, tid = threadIdx.x;
  double *geo = smd, *ia = geo + 12 * P, *sU = ia + P, *sq = sU + 4 * P, *sdt = sq + 5 * P, *fg = sdt + P;
  int4 *nb4 = reinterpret_cast<int4 *>(fg + 5 * Q);  // neighbour rows (the cell itself in unused slots)
  int4 *cf4 = nb4 + P;                               // face slots
  int4 *be = cf4 + P;                                // boundary entries: kind, face, ghost, id
  int2 *fon = reinterpret_cast<int2 *>(be + a.entries);
  int *bo = reinterpret_cast<int *>(fon + Q), *nf = bo + P + 1;  // first entry of each cell; face counts
  unsigned int arrivals = 0;
  const int e0 = nc > 0 ? m.bptr[cr.x] : 0;
  for (int l = tid; l < nc; l += blockDim.x) {
    const int c = cr.x + l;
#pragma unroll
    for (int f = 0; f < 4; f++) {
      const size_t idx = (size_t)f * NP + c;
      geo[(3 * f) * P + l] = m.nx[idx];
      geo[(3 * f + 1) * P + l] = m.ny[idx];
      geo[(3 * f + 2) * P + l] = m.dl[idx];
    }
    ia[l] = m.inv_area[c];
#pragma unroll
    for (int k = 0; k < 4; k++) sU[k * P + l] = st.U[(size_t)k * NT + c];
    const double4 v = st.q4[c];
    sq[l] = v.x;
    sq[P + l] = v.y;
    sq[2 * P + l] = v.z;
    sq[3 * P + l] = v.w;
    sq[4 * P + l] = st.prim[4 * (size_t)NT + c];
    int4 n = m.nbr4[c];
    n.x = n.x >= 0 && n.x < NT ? n.x : c;
    n.y = n.y >= 0 && n.y < NT ? n.y : c;
    n.z = n.z >= 0 && n.z < NT ? n.z : c;
    n.w = n.w >= 0 && n.w < NT ? n.w : c;
    nb4[l] = n;
    cf4[l] = m.cface4[c];
    nf[l] = m.nf[c];
    const int b0 = m.bptr[c] - e0, b1 = m.bptr[c + 1] - e0;
    bo[l] = b0;
    if (l == nc - 1) bo[nc] = b1;
    for (int i = b0; i < b1; i++) {
      const int e = m.bidx[e0 + i];
      const int4 b = m.bnd[e];
      be[i] = make_int4(b.x, b.z, b.w, e);
    }
  }
  for (int l = tid; l < nfc; l += blockDim.x) {
    const int i = fr.x + l;
    const double4 g = m.fg4[i];
    fg[l] = g.x;
    fg[Q + l] = g.y;
    fg[2 * Q + l] = g.z;
    fg[3 * Q + l] = g.w;
    fg[4 * Q + l] = m.fdy[i];
    fon[l] = m.fon[i];
  }
  __syncthreads();
  // Ghost states of cell l's entries from its current state (Ucur, leading dimension ldU: U or the stage
  // state).
  auto ghosts = [&](int l, const double *Ucur, size_t ldU) {
    for (int i = bo[l]; i < bo[l + 1]; i++) {
      const int4 b = be[i];
      const BcShared src{geo, sq, Ucur, ldU, P, l, b.y, b.w, m.bstate, m.bexit};
      double G[4];
      if (bc_values(src, bp, b.x, sq[l], sq[P + l], sq[2 * P + l], sq[3 * P + l], G)) store_ghost(st, NT, b.z, G);
    }
  };
  const int glim = fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter;
  __shared__ double sh_min[32], fmin_sh[kStepsPerLaunch];
  double *step_min = st.partial + 9 * (size_t)gridDim.x;  // [gridDim.x][n_steps] block minima of the frozen dt
  int step = 0;
  for (; step < a.n_steps; step++) {
    const bool full = step == a.n_steps - 1 || a.may_stop;  // this step's R, norms, ... can be read
    for (int k = 0; k < a.n_stages; k++) {
      const int kind = a.kind0 + k;
      const bool last = k == a.n_stages - 1, with_dt = k == 0 || (last && full);
      for (int l = tid; l < nc; l += blockDim.x) {
        const int c = cr.x + l;
        if (k == 0) ghosts(l, sU, P);
        const int4 n = nb4[l];
        const double4 v[4] = {ld32_ordered(st.q4 + n.x), ld32_ordered(st.q4 + n.y), ld32_ordered(st.q4 + n.z),
                              ld32_ordered(st.q4 + n.w)};
        double qn[4][4], nx[4], ny[4], dl[4];
#pragma unroll
        for (int f = 0; f < 4; f++) {
          qn[f][0] = v[f].x;
          qn[f][1] = v[f].y;
          qn[f][2] = v[f].z;
          qn[f][3] = v[f].w;
          nx[f] = geo[(3 * f) * P + l];
          ny[f] = geo[(3 * f + 1) * P + l];
          dl[f] = geo[(3 * f + 2) * P + l];
        }
        const double qc[4] = {sq[l], sq[P + l], sq[2 * P + l], sq[3 * P + l]};
        double g[8] = {0, 0, 0, 0, 0, 0, 0, 0}, den = 0.0;
        const int cnt = nf[l];
        const double ac = sq[4 * P + l];
#pragma unroll
        for (int f = 0; f < 4; f++)
          if (f < cnt) gg_face<true>(qc, ac, qn[f], nx[f], ny[f], dl[f], g, den);
#pragma unroll
        for (int q = 0; q < 8; q++) g[q] *= ia[l];
        if (sizeof(T) == sizeof(float)) {
          st32f(st.recf + 2 * (size_t)c, g);
        } else {
          double4 *r = reinterpret_cast<double4 *>(st.rec + 8 * (size_t)c);
          st32(r, make_double4(g[0], g[1], g[2], g[3]));
          st32(r + 1, make_double4(g[4], g[5], g[6], g[7]));
        }
        if (with_dt) {
          const double dt = cell_dt_a(fp, m.area[c], den);
          if (k == 0) sdt[l] = dt;
          if (last) st.dtc[c] = dt;
        }
      }
      steps_barrier(st, a, count, blk.blocks, arrivals);
      for (int l = tid; l < nfc; l += blockDim.x) {
        const int2 on = fon[l];
        const int gn = on.y < NP ? on.y : on.x;  // a ghost neighbour uses the owner's gradients
        const double4 c0 = ld32_ordered(st.q4 + on.x), n0 = ld32_ordered(st.q4 + on.y);
        double4 c1, c2, n1, n2;
        if (sizeof(T) == sizeof(float)) {
          const float4 x = st.recf[2 * (size_t)on.x], y = st.recf[2 * (size_t)on.x + 1];
          const float4 z = st.recf[2 * (size_t)gn], w = st.recf[2 * (size_t)gn + 1];
          c1 = make_double4(x.x, x.y, x.z, x.w);
          c2 = make_double4(y.x, y.y, y.z, y.w);
          n1 = make_double4(z.x, z.y, z.z, z.w);
          n2 = make_double4(w.x, w.y, w.z, w.w);
        } else {
          const double4 *rc = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)on.x);
          const double4 *rn = reinterpret_cast<const double4 *>(st.rec + 8 * (size_t)gn);
          c1 = ld32_ordered(rc);
          c2 = ld32_ordered(rc + 1);
          n1 = ld32_ordered(rn);
          n2 = ld32_ordered(rn + 1);
        }
        FaceOps<T> o;
        double4 F = face_flux_rec<T, DISS>(o, glim, c0, c1, c2, n0, n1, n2, T(fg[l]), T(fg[Q + l]), T(fg[2 * Q + l]),
                                           T(fg[3 * Q + l]), T(fg[4 * Q + l]), T(fp.eflin), T(fp.shock_fix));
        if constexpr (FaceOps<T>::fast) {
          if (o.bad()) F = face_flux_again<DISS>(m, st, fp, fr.x + l);
        }
        st32(st.F + fr.x + l, F);
      }
      steps_barrier(st, a, count, blk.blocks, arrivals);
      double dtu = 1e308 * 10.0;
      double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int l = tid; l < nc; l += blockDim.x) {
        const int c = cr.x + l;
        const int4 e4 = cf4[l];
        double R[4];
        sum_faces(nf[l], e4, ld32_ordered(st.F + face_id(e4.x)), ld32_ordered(st.F + face_id(e4.y)),
                  ld32_ordered(st.F + face_id(e4.z)), ld32_ordered(st.F + face_id(e4.w)), R);
        StageIn si;
        si.invA = ia[l];
        double Un[4], out[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          Un[q] = sU[q * P + l];
          si.Sk[q] = st.S[(size_t)q * NP + c];
        }
        const double dt = sdt[l];
        dtu = dt < dtu ? dt : dtu;
        const bool fin = stage_values(m, st, c, kind, dt, R, Un, si, out);
        if (fin) {
          const bool direct = direct_kind(kind);
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const double du = direct ? out[q] - Un[q] : out[q];
            const double nu = direct ? out[q] : Un[q] + out[q];
            if (full) {
              e[q] += err_term(du, Un[q]);
              e[4 + q] += R[q] * R[q];
              st.R[(size_t)q * NP + c] = R[q];
              if (a.keep_delu) st.dU[(size_t)q * NP + c] = du;
              st.U[(size_t)q * NT + c] = nu;
            }
            out[q] = nu;
          }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (fin) sU[q * P + l] = out[q];
          else st.S[(size_t)q * NP + c] = out[q];
        }
        Prim w;
        const bool ok = eos_fast(out[0], out[1], out[2], out[3], w);
        if (!ok) flag_bad(st.status, c);
        sq[l] = w.rho;
        sq[P + l] = w.u;
        sq[2 * P + l] = w.v;
        sq[3 * P + l] = w.p;
        sq[4 * P + l] = w.a;
        if (fin && full) store_prim(st.prim, st.q4, NT, c, w);
        else st32(st.q4 + c, make_double4(w.rho, w.u, w.v, w.p));
        if (!fin) ghosts(l, st.S + cr.x, NP);
        else if (full) st.dtk[c] = dt;
      }
      if (last && a.reduce) {
        if (a.may_stop) {
          stage_final_reduce(st, e, dtu);
        } else if (step < a.n_steps - 1) {
          const double bm = block_min(dtu, sh_min);
          if (tid == 0) step_min[(size_t)blockIdx.x * a.n_steps + step] = bm;
        } else {
          // The earlier steps' Total_Time increments, in step order, before this step's own.
          steps_barrier(st, a, count, blk.blocks, arrivals);
          if (blockIdx.x == 0) {
            for (int s0 = tid; s0 < a.n_steps - 1; s0 += blockDim.x) {
              double v = 1e308 * 10.0;
#pragma unroll 8
              for (int i = 0; i < (int)gridDim.x; i++) {
                const double w = step_min[(size_t)i * a.n_steps + s0];
                v = w < v ? w : v;
              }
              fmin_sh[s0] = v;
            }
            __syncthreads();
            if (tid == 0) {
              double t = st.ctl[CTL_TOTAL_TIME];
              for (int s0 = 0; s0 < a.n_steps - 1; s0++) t += fmin_sh[s0];
              st.ctl[CTL_TOTAL_TIME] = t;
              st.ctl[CTL_ITER] += double(a.n_steps - 1);
            }
          }
          steps_barrier(st, a, count, blk.blocks, arrivals);
          stage_final_reduce(st, e, dtu);
        }
      }
      steps_barrier(st, a, count, blk.blocks, arrivals);
    }
    if (a.may_stop && step_done(st.ctl)) break;  // the same flag in every block
  }
}

// Pseudo-steps of a small per-cell solve in one cooperative launch: four lanes per cell, every cell resident,
// the evaluation of k_flux4 and the update of k_stage one after the other with a grid barrier behind each
// (a stage overwrites the primitives that its neighbours' evaluation reads; Min_dt is complete at the first).
// Min_dt is an atomic minimum of order-preserving keys in three slots used in turn, so that a slot is reset
// two barriers before it is used again.  Same operations on the same operands as the separate kernels: same
// bits.  The residual, del_t and the norms stay out, so a step by the separate kernels follows; a call with a
// t_end, where any step may be the last, runs them throughout.  Bound by
// latency: two barriers, the gathers' L2 rounds (a barrier empties the L1, so what stays the same is kept in
// registers) and one face's dependent FP64 chain per stage.  Per pseudo-step of three stages (separate
// kernels against this, LLF / ROE / ROE_2O / HLLC, B200): 29 / 31 / 33 / 29 us against 17 / 20 / 22 / 19 at
// 1,600 cells, 33 / 38 / 41 / 35 against 24 / 27 / 31 / 27 at 18,944, so every mesh that fits uses it.
struct BcCell {
  double nxv, nyv, av;
  const double *W, *X;  // current state, exit-copy source
  int e;
  const double4 *bstate;
  const double *bexit;
  __device__ __forceinline__ double nx() const { return nxv; }
  __device__ __forceinline__ double ny() const { return nyv; }
  __device__ __forceinline__ double a() const { return av; }
  __device__ __forceinline__ double cur(int k) const { return W[k]; }
  __device__ __forceinline__ double src(int k) const { return X[k]; }
};

struct CellStepsArgs {
  StepsArgs s;
  int lts0, lts1;  // lts argument (see k_stage) of the first stage and of the others
  int src_S;
  unsigned long long *dt_min;  // [3], all ones before the launch
};

__device__ __forceinline__ unsigned long long ordered_key(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : b | (1ull << 63);
}
__device__ __forceinline__ double key_value(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? k & ~(1ull << 63) : ~k));
}

template <int DISS, int ORDER>
__global__ void __launch_bounds__(kFlux4Block, 4) k_cell_steps(const __grid_constant__ DevMesh m,
                                                               const __grid_constant__ DevState st,
                                                               const __grid_constant__ FluxParams fp,
                                                               const __grid_constant__ BcParams bp,
                                                               const __grid_constant__ CellStepsArgs a) {
  __shared__ double sh[32];
  if (step_done(st.ctl)) return;  // the same for every block: nothing in the launch writes the flag
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = gid >> 2, f = gid & 3;
  const int nf = c < m.NP ? m.nf[c] : 0;
  const bool owner = c < m.NP && f == 0, first_thread = gid == 0;
  const int NP = m.NP, NT = m.NT;
  const FaceGeo g = load_face<DISS, ORDER>(m, c < NP ? c : 0, f);
  // The cell's boundary entries; two are kept.
  const int b0 = owner ? m.bptr[c] : 0, ne = owner ? m.bptr[c + 1] - b0 : 0;
  int ent[2];
  int4 bnd[2];
  double2 bn[2];
#pragma unroll
  for (int j = 0; j < 2; j++)
    if (j < ne) {
      ent[j] = m.bidx[b0 + j];
      bnd[j] = m.bnd[ent[j]];
      bn[j] = make_double2(m.nx[bnd[j].z * NP + c], m.ny[bnd[j].z * NP + c]);
    }
  unsigned int arrivals = 0;
  int slot = 0;
  double dtmin = 0.0, dtstep = 0.0, dtk = 0.0, total = first_thread ? st.ctl[CTL_TOTAL_TIME] : 0.0;
  for (int i = 0; i < a.s.n_steps; i++) {
    for (int k = 0; k < a.s.n_stages; k++) {
      const int kind = a.s.kind0 ? a.s.kind0 + k : 0;
      const int lts = k ? a.lts1 : a.lts0;
      const bool last = k == a.s.n_stages - 1;
      const bool want_min = lts == 0 || (k == 0 && lts != 1);
      double R[4], den, dt = 1e308 * 10.0;
      StageIn in;
      if (owner) load_stage_in(m, st, c, kind, in);
      quad_residual<DISS, ORDER>(m, st, fp, fp.consistent && k > 0, c, f, nf, g, R, den);
      if (owner && (want_min || lts == 1)) dt = cell_dt(m, fp, c, den);
      if (want_min) {
        const double bm = block_min(dt, sh);
        if (threadIdx.x == 0) atomicMin(a.dt_min + slot, ordered_key(bm));
      }
      steps_barrier(st, a.s, a.s.arrivals, gridDim.x, arrivals);
      if (want_min) dtmin = key_value(__ldcg(a.dt_min + slot));
      if (first_kind(kind)) {
        dtstep = dtmin;
        dtk = dt;
      }
      if (owner) {
        const double d = lts == 0 ? dtmin : (lts == 1 ? dt : (lts == 2 ? dtk : dtstep));
        double out[4];
        const bool fin = stage_values(m, st, c, kind, d, R, in.Un, in, out);
        if (fin && !direct_kind(kind)) {
#pragma unroll
          for (int j = 0; j < 4; j++) out[j] = in.Un[j] + out[j];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (last) st.U[(size_t)j * NT + c] = out[j];
          else st.S[(size_t)j * NP + c] = out[j];
        }
        Prim q;
        const bool ok = eos_fast(out[0], out[1], out[2], out[3], q);
        store_prim(st.prim, st.q4, NT, c, q);
        if (!ok) flag_bad(st.status, c);
        // The next evaluation's ghosts (after the last stage from U^{n+1}, which `out` is).
        BcCell src{0.0, 0.0, q.a, out, last || a.src_S ? out : in.Un, 0, m.bstate, m.bexit};
        double G[4];
#pragma unroll
        for (int j = 0; j < 2; j++)
          if (j < ne) {
            src.nxv = bn[j].x;
            src.nyv = bn[j].y;
            src.e = ent[j];
            if (bc_values(src, bp, bnd[j].x, q.rho, q.u, q.v, q.p, G)) store_ghost(st, NT, bnd[j].w, G);
          }
        for (int j = 2; j < ne; j++) {
          const int4 b = m.bnd[m.bidx[b0 + j]];
          src.nxv = m.nx[b.z * NP + c];
          src.nyv = m.ny[b.z * NP + c];
          src.e = m.bidx[b0 + j];
          if (bc_values(src, bp, b.x, q.rho, q.u, q.v, q.p, G)) store_ghost(st, NT, b.w, G);
        }
      }
      const int next = slot == 2 ? 0 : slot + 1;
      if (first_thread) {
        if (last) total += lts >= 2 ? dtstep : dtmin;
        a.dt_min[next == 2 ? 0 : next + 1] = ~0ull;
      }
      slot = next;
      steps_barrier(st, a.s, a.s.arrivals, gridDim.x, arrivals);
    }
  }
  if (first_thread) {
    st.ctl[CTL_TOTAL_TIME] = total;
    st.ctl[CTL_ITER] += a.s.n_steps;
    st.ctl[CTL_DTMIN] = dtmin;
    st.ctl[CTL_DTSTEP] = dtstep;
  }
}

// Patch form of one stage of the face-based per-cell-dt forms: one thread block per patch of up
// to kPatchCells cells does the work of k_muscl_gradients, k_faces and k_gather_stage for its
// cells, with the records and face fluxes in shared memory instead of HBM.
//   1. records (rho, u, v, p and gradients) of its own cells and of its halo cells (the cells
//      across its faces), from the stage's primitives `pin`; del_t of its own cells;
//   2. every face of its own cells (a face to a halo cell is evaluated by both patches, from the
//      owner's side, so both get the same bits), +F into the owner's slot and -F into the
//      neighbour's slot when that cell is its own;
//   3. per own cell: the slots summed in face order and the stage update (stage_cell), which
//      writes the new primitives and the next stage's ghosts to st.prim (a different buffer from
//      `pin`: other blocks are still reading their halo primitives from it).
// Every operation on a value is the one the three-kernel form does, in the same order.
template <int DISS>
__global__ void __launch_bounds__(kPatchCells, 5) k_patch_stage(DevMesh m, DevState st, FluxParams fp, BcParams bp,
                                                                int kind, int lts, int fuse_final, int keep_delu,
                                                                int flags, const double *__restrict__ pin) {
  pdl_enter();
  if (step_done(st.ctl)) return;
  extern __shared__ double smem[];
  const int NP = m.NP, NT = m.NT, rows = m.patch_rows;
  const int b = blockIdx.x, tid = threadIdx.x;
  const int2 pr = m.patch[b];
  const int c0 = pr.x, P = min(pr.y, kPatchCells);
  const int h0 = m.phptr[b], H = m.phptr[b + 1] - h0;
  double *srec = smem;             // [12][rows]: rho, u, v, p, then the 8 gradient terms
  double *sF = smem + 12 * rows;   // [4 slots][4][kPatchCells]
  const int glim = fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter;

  // The tables are checked on the host; an entry that would still leave its buffer is skipped and
  // reported as a mesh error instead of being used.
  double dtc = 0.0;
  const int nrow = min(P + H, rows);
  for (int l = tid; l < nrow; l += kPatchCells) {
    const int c = l < P ? c0 + l : m.phcell[h0 + l - P];
    if (c < 0 || c >= NP) {
      atomicCAS(&st.status[0], 0, 7 /* CFD_ERR_MESH */);
      continue;
    }
    double qc[4], g[8], den;
#pragma unroll
    for (int k = 0; k < 4; k++) qc[k] = pin[k * NT + c];
    cell_gradients<true>(m, pin, nullptr, c, qc, g, den);
#pragma unroll
    for (int k = 0; k < 4; k++) srec[k * rows + l] = qc[k];
#pragma unroll
    for (int k = 0; k < 8; k++) srec[(4 + k) * rows + l] = g[k];
    if (l < P) {
      dtc = cell_dt(m, fp, c, den);
      st.dtc[c] = dtc;
    }
  }
  __syncthreads();

  const int f0 = m.pfptr[b], f1 = m.pfptr[b + 1];
  for (int j = f0 + tid; j < f1; j += kPatchCells) {
    const PatchFace fe = m.pface[j];
    const int N = fe.N;
    const int lo = fe.rows & 0xFFFF, ln = (int)((unsigned)fe.rows >> 16);
    const int so = fe.slots & 0xFF, sn = (fe.slots >> 8) & 0xFF;
    const bool bad = lo >= nrow || (ln == 0xFFFF ? (N < NP || N >= NT) : ln >= nrow) ||
                     (so != 0xFF && (so > 3 || lo >= P)) || (sn != 0xFF && (sn > 3 || ln >= P));
    if (bad) {
      atomicCAS(&st.status[0], 0, 7 /* CFD_ERR_MESH */);
      continue;
    }
    const double4 c0r = make_double4(srec[lo], srec[rows + lo], srec[2 * rows + lo], srec[3 * rows + lo]);
    const double4 c1r =
        make_double4(srec[4 * rows + lo], srec[5 * rows + lo], srec[6 * rows + lo], srec[7 * rows + lo]);
    const double4 c2r =
        make_double4(srec[8 * rows + lo], srec[9 * rows + lo], srec[10 * rows + lo], srec[11 * rows + lo]);
    double4 n0r, n1r, n2r;
    if (ln == 0xFFFF) {
      // Ghost neighbour: its state, with the owner's gradient.
      n0r = make_double4(pin[N], pin[NT + N], pin[2 * NT + N], pin[3 * NT + N]);
      n1r = c1r;
      n2r = c2r;
    } else {
      n0r = make_double4(srec[ln], srec[rows + ln], srec[2 * rows + ln], srec[3 * rows + ln]);
      n1r = make_double4(srec[4 * rows + ln], srec[5 * rows + ln], srec[6 * rows + ln], srec[7 * rows + ln]);
      n2r = make_double4(srec[8 * rows + ln], srec[9 * rows + ln], srec[10 * rows + ln], srec[11 * rows + ln]);
    }
    Ieee<double> o;
    const double4 F = face_flux_rec<double, DISS>(o, glim, c0r, c1r, c2r, n0r, n1r, n2r, fe.nx, fe.ny, fe.dl, fe.dx, fe.dy,
                                                    fp.eflin, fp.shock_fix);
    if (so < 4) {
      sF[(so * 4 + 0) * kPatchCells + lo] = F.x;
      sF[(so * 4 + 1) * kPatchCells + lo] = F.y;
      sF[(so * 4 + 2) * kPatchCells + lo] = F.z;
      sF[(so * 4 + 3) * kPatchCells + lo] = F.w;
    }
    if (sn < 4) {
      sF[(sn * 4 + 0) * kPatchCells + ln] = -F.x;
      sF[(sn * 4 + 1) * kPatchCells + ln] = -F.y;
      sF[(sn * 4 + 2) * kPatchCells + ln] = -F.z;
      sF[(sn * 4 + 3) * kPatchCells + ln] = -F.w;
    }
  }
  __syncthreads();

  double dtu = 1e308 * 10.0;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (tid < P && c0 + tid < NP) {
    const int c = c0 + tid;
    const int nf = m.nf[c];
    double R[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int f = 0; f < 4; f++) {
      if (f < nf) {
#pragma unroll
        for (int k = 0; k < 4; k++) R[k] += sF[(f * 4 + k) * kPatchCells + tid];
      }
    }
    // Ghost rows move to the output buffer with their owner (the final stage, and boundary kinds
    // that leave a ghost unchanged, keep its current state); non-final stages overwrite them.
    const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
    for (int q = b0; q < b1; q++) {
      const int g = m.bnd[m.bidx[q]].w;
#pragma unroll
      for (int k = 0; k < 5; k++) st.prim[k * NT + g] = pin[k * NT + g];
      if (st.q4) st.q4[g] = make_double4(pin[g], pin[NT + g], pin[2 * NT + g], pin[3 * NT + g]);
    }
    dtu = stage_cell(m, st, bp, c, R, dtc, kind, lts, fuse_final, keep_delu, flags, e);
  }
  if (fuse_final && final_kind(kind)) stage_final_reduce(st, e, dtu);
}

// ---- Tile form of one stage on a structured block (no reference counterpart) ----
// One thread block per tile of kTileX x kTileY cells does the work of k_muscl_gradients, k_faces
// and k_gather_stage for its cells with everything between them in shared memory:
//   0. the (rho, u, v, p) rows of the tile and of two rings of cells around it (ghost rows
//      beside the block's boundary) from q_in, one coalesced pass per row of the region;
//   1. gradients of the tile's cells and of the halo cells along its four sides (the cells across
//      its boundary faces), del_t of its own cells;
//   2. the flux of every W and S face of its cells, each from its owner's side (a face on the
//      tile boundary is evaluated by both tiles from the same inputs, so both get the same bits);
//   3. per own cell the four fluxes summed in slot order and the stage update (stage_cell), which
//      writes the stage's rows and the next stage's ghost rows to st.q4 (not q_in: other tiles
//      are still reading their halo rows from it).
// Every operation on a value is the one the three-kernel form does, in the same order: the
// gradient terms and the face fluxes are formed per position around the cell and summed in the
// cell's slot order; a slot normal is the owner-side normal negated exactly on the non-owner side
// (checked on the host before the form is offered).
constexpr int kTileX = kTileCellsX;
constexpr int kTileY = kTileCellsY;
constexpr int kTileQW = kTileX + 4, kTileQH = kTileY + 4;  // state region: tile + 2 rings
constexpr int kTileRW = kTileX + 2, kTileRH = kTileY + 2;  // gradient region: tile + 1 ring
constexpr int kTileNW = (kTileX + 1) * kTileY;              // W faces of the tile
constexpr int kTileNS = kTileX * (kTileY + 1);              // S faces of the tile

template <typename T>
struct TileRecT {
  typedef double4 type;
};
template <>
struct TileRecT<float> {
  typedef float4 type;
};

template <typename T>
__host__ __device__ constexpr size_t tile_smem_bytes() {
  return sizeof(double4) * (size_t)(kTileQW * kTileQH + kTileNW + kTileNS) +
         2 * sizeof(typename TileRecT<T>::type) * (size_t)(kTileRW * kTileRH);
}

// acc[k] += t[(R + f) & 3][k] for f = 0..3: position terms summed in the cell's slot order.
template <int R, int K>
__device__ __forceinline__ void rot_sum(const double (&t)[4][K], double (&acc)[K]) {
#pragma unroll
  for (int f = 0; f < 4; f++) {
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] += t[(R + f) & 3][k];
  }
}
template <int K>
__device__ __forceinline__ void slot_order_sum(int r, const double (&t)[4][K], double (&acc)[K]) {
  switch (r) {
    case 0: rot_sum<0, K>(t, acc); break;
    case 1: rot_sum<1, K>(t, acc); break;
    case 2: rot_sum<2, K>(t, acc); break;
    default: rot_sum<3, K>(t, acc); break;
  }
}

// Shared-memory offsets of the four neighbours and the face-table indices of the four faces of
// cell (i, j) at positions E, N, W, S (N and S exchanged when lh).
struct TilePos {
  int dq[4];
  int face[4];  // W-family index (positions 0, 2) or S-family index (1, 3)
};
__device__ __forceinline__ TilePos tile_pos(const TileMesh &tm, int i, int j) {
  TilePos t;
  const int wi = j * (tm.ni + 1) + i, si = j * tm.ni + i;
  t.dq[0] = 1;
  t.dq[2] = -1;
  t.face[0] = wi + 1;
  t.face[2] = wi;
  const int up = tm.lh ? 3 : 1, dn = tm.lh ? 1 : 3;
  t.dq[up] = kTileQW;
  t.dq[dn] = -kTileQW;
  t.face[up] = si + tm.ni;
  t.face[dn] = si;
  return t;
}

// Gradients of physical cell c = (i, j), row qi of the state region, as cell_gradients<DT> forms
// them; with DT also the del_t denominator.
__device__ __forceinline__ void tile_gradients(const DevMesh &m, const DevState &st, const TileMesh &tm,
                                               const double4 *sq, int qi, int c, int i, int j, bool dt, double g[8],
                                               double &den) {
  const unsigned code = tm.code[c];
  const double ia = m.inv_area[c];
  const double ac = dt ? st.prim[4 * m.NT + c] : 0.0;
  const TilePos tp = tile_pos(tm, i, j);
  const double4 qv = sq[qi];
  const double qc[4] = {qv.x, qv.y, qv.z, qv.w};
  double t[4][9];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const double4 fg = (p & 1) ? tm.fs[tp.face[p]] : tm.fw[tp.face[p]];
    const double4 qn = sq[qi + tp.dq[p]];
    const bool own = (code >> (2 + p)) & 1u;
    const double nxf = own ? fg.x : -fg.x, nyf = own ? fg.y : -fg.y, dlf = fg.z;
    const double wx = nxf * dlf, wy = nyf * dlf;
    const double qnv[4] = {qn.x, qn.y, qn.z, qn.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double qf = 0.5 * (qc[k] + qnv[k]);
      t[p][2 * k] = qf * wx;
      t[p][2 * k + 1] = qf * wy;
    }
    const double vnf = qc[1] * nxf + qc[2] * nyf;
    t[p][8] = (fabs(vnf) + ac) * dlf;
  }
  double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  slot_order_sum<9>(code & 3u, t, acc);
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = acc[k] * ia;
  den = acc[8];
}

template <typename T, int DISS>
__global__ void __launch_bounds__(kTileX * kTileY, 2)
    k_tile_stage(DevMesh m, DevState st, FluxParams fp, BcParams bp, TileMesh tm, const double4 *__restrict__ q_in,
                 int kind, int lts, int fuse_final, int keep_delu, int flags, int with_dt) {
  typedef typename TileRecT<T>::type RecV;
  pdl_enter();
  if (step_done(st.ctl)) return;
  extern __shared__ double4 tsm[];
  double4 *sq = tsm;                                           // [QH][QW]
  double4 *sF = sq + kTileQW * kTileQH;                        // W faces [TY][TX + 1], then S faces [TY + 1][TX]
  RecV *srec = reinterpret_cast<RecV *>(sF + kTileNW + kTileNS);  // [RH][RW] x 2
  const int ni = tm.ni, nj = tm.nj, tid = threadIdx.x;
  const int i0 = (blockIdx.x % tm.tiles_i) * kTileX, j0 = (blockIdx.x / tm.tiles_i) * kTileY;
  const int glim = fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter;

  // 0. States of the region (corners of the outer rings beyond the block are never read).
  for (int t = tid; t < kTileQW * kTileQH; t += blockDim.x) {
    const int jj = t / kTileQW, ii = t - jj * kTileQW;
    const int i = i0 + ii - 2, j = j0 + jj - 2;
    const bool in_i = i >= 0 && i < ni, in_j = j >= 0 && j < nj;
    int r = -1;
    if (in_i && in_j) r = j * ni + i;
    else if (in_j && i == -1) r = tm.gW[j];
    else if (in_j && i == ni) r = tm.gE[j];
    else if (in_i && j == -1) r = tm.gS[i];
    else if (in_i && j == nj) r = tm.gN[i];
    sq[t] = r >= 0 ? q_in[r] : make_double4(0.0, 0.0, 0.0, 0.0);
  }
  __syncthreads();

  // 1. Gradients: own cells (thread tid has cell tid), then the halo strips W, E, S, N.
  double dtc = 0.0;
  constexpr int NG = kTileX * kTileY + 2 * kTileY + 2 * kTileX;
  for (int t = tid; t < NG; t += blockDim.x) {
    int gi, gj;
    if (t < kTileX * kTileY) {
      gi = t % kTileX;
      gj = t / kTileX;
    } else {
      const int u = t - kTileX * kTileY;
      if (u < kTileY) {
        gi = -1;
        gj = u;
      } else if (u < 2 * kTileY) {
        gi = kTileX;
        gj = u - kTileY;
      } else if (u < 2 * kTileY + kTileX) {
        gi = u - 2 * kTileY;
        gj = -1;
      } else {
        gi = u - 2 * kTileY - kTileX;
        gj = kTileY;
      }
    }
    const int i = i0 + gi, j = j0 + gj;
    if (i < 0 || i >= ni || j < 0 || j >= nj) continue;
    const int c = j * ni + i;
    const bool own = t < kTileX * kTileY;
    double g[8], den;
    tile_gradients(m, st, tm, sq, (gj + 2) * kTileQW + gi + 2, c, i, j, own && with_dt, g, den);
    RecV *r = srec + 2 * ((gj + 1) * kTileRW + gi + 1);
    if (sizeof(T) == sizeof(float)) {
      r[0] = RecV{T(float(g[0])), T(float(g[1])), T(float(g[2])), T(float(g[3]))};
      r[1] = RecV{T(float(g[4])), T(float(g[5])), T(float(g[6])), T(float(g[7]))};
    } else {
      r[0] = RecV{T(g[0]), T(g[1]), T(g[2]), T(g[3])};
      r[1] = RecV{T(g[4]), T(g[5]), T(g[6]), T(g[7])};
    }
    if (own && with_dt) {
      dtc = cell_dt(m, fp, c, den);
      st.dtc[c] = dtc;
    }
  }
  __syncthreads();

  // 2. Face fluxes: W faces (i0..i0+TX, rows of the tile), then S faces (columns, j0..j0+TY).
  for (int t = tid; t < kTileNW + kTileNS; t += blockDim.x) {
    int fi, fj, lx, ly, hx, hy, gidx;
    bool lo_phys, hi_phys, ohigh;
    double4 gq;
    double gdy;
    if (t < kTileNW) {
      fj = t / (kTileX + 1);
      fi = t - fj * (kTileX + 1);
      const int i = i0 + fi, j = j0 + fj;
      if (i > ni || j >= nj) continue;
      gidx = j * (ni + 1) + i;
      lx = fi - 1;
      ly = fj;
      hx = fi;
      hy = fj;
      lo_phys = i > 0;
      hi_phys = i < ni;
      gq = tm.fw[gidx];
      gdy = tm.fwdy[gidx];
      ohigh = tm.fwo[gidx] != 0;
    } else {
      const int u = t - kTileNW;
      fj = u / kTileX;
      fi = u - fj * kTileX;
      const int i = i0 + fi, j = j0 + fj;
      if (i >= ni || j > nj) continue;
      gidx = j * ni + i;
      lx = fi;
      ly = fj - 1;
      hx = fi;
      hy = fj;
      lo_phys = j > 0;
      hi_phys = j < nj;
      gq = tm.fs[gidx];
      gdy = tm.fsdy[gidx];
      ohigh = tm.fso[gidx] != 0;
    }
    const int ox = ohigh ? hx : lx, oy = ohigh ? hy : ly, nx_ = ohigh ? lx : hx, ny_ = ohigh ? ly : hy;
    const bool nphys = ohigh ? lo_phys : hi_phys;
    const double4 c0 = sq[(oy + 2) * kTileQW + ox + 2], n0 = sq[(ny_ + 2) * kTileQW + nx_ + 2];
    const RecV *ro = srec + 2 * ((oy + 1) * kTileRW + ox + 1);
    const RecV *rn = nphys ? srec + 2 * ((ny_ + 1) * kTileRW + nx_ + 1) : ro;
    const RecV a = ro[0], b = ro[1], p = rn[0], q = rn[1];
    const double4 c1 = make_double4(a.x, a.y, a.z, a.w), c2 = make_double4(b.x, b.y, b.z, b.w);
    const double4 n1 = make_double4(p.x, p.y, p.z, p.w), n2 = make_double4(q.x, q.y, q.z, q.w);
    Ieee<T> o;
    sF[t] = face_flux_rec<T, DISS>(o, glim, c0, c1, c2, n0, n1, n2, T(gq.x), T(gq.y), T(gq.z), T(gq.w), T(gdy),
                                   T(fp.eflin), T(fp.shock_fix));
  }
  __syncthreads();

  // 3. Gather in slot order and stage update of the own cells.
  double dtu = 1e308 * 10.0;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  {
    const int tx = tid % kTileX, ty = tid / kTileX;
    const int i = i0 + tx, j = j0 + ty;
    if (i < ni && j < nj) {
      const int c = j * ni + i;
      const unsigned code = tm.code[c];
      const int wE = ty * (kTileX + 1) + tx + 1, wW = wE - 1;
      const int sS = kTileNW + ty * kTileX + tx, sN = sS + kTileX;
      const int pf[4] = {wE, tm.lh ? sS : sN, wW, tm.lh ? sN : sS};
      double t[4][4];
#pragma unroll
      for (int p = 0; p < 4; p++) {
        const double4 F = sF[pf[p]];
        const bool own = (code >> (2 + p)) & 1u;
        t[p][0] = own ? F.x : -F.x;
        t[p][1] = own ? F.y : -F.y;
        t[p][2] = own ? F.z : -F.z;
        t[p][3] = own ? F.w : -F.w;
      }
      double R[4] = {0.0, 0.0, 0.0, 0.0};
      slot_order_sum<4>(code & 3u, t, R);
      // Ghost rows move to the output buffer with their owner (boundary kinds that leave a ghost
      // unchanged, and the final stage, keep its current state); non-final stages overwrite them.
      const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
      for (int q = b0; q < b1; q++) {
        const int g = m.bnd[m.bidx[q]].w;
        st.q4[g] = q_in[g];
      }
      const double dts = (lts == 1 || first_kind(kind)) ? dtc : 0.0;
      dtu = stage_cell(m, st, bp, c, R, dts, kind, lts, fuse_final, keep_delu, flags, e);
    }
  }
  if (fuse_final && final_kind(kind)) stage_final_reduce(st, e, dtu);
}

// ---- TMA form of the tile stage (no reference counterpart) ----
// The work of k_tile_stage, tile by tile and operation by operation the same (so the same bits),
// with every global load moved to the start of the block and made asynchronous:
//   * one thread issues three cp.async.bulk.tensor loads on one mbarrier: the (rho, u, v, p) rows
//     of the tile and two rings (box 36 x 12 of 32-byte rows; rows beyond the block arrive as
//     zeros), and the 48-byte face records of the W faces (35 x 10) and S faces (34 x 11) that the
//     tile's cells and its one-ring halo cells touch;
//   * every thread issues cp.async copies of its own cell's stage inputs (U^n, the stage state,
//     the frozen dt, sound speed and area for del_t) and of the 1/area of the gradient region,
//     and plain loads of the region's slot codes and of the ghost rows beside the block's rim
//     (which the bulk load fills with zeros; they are written after it lands).
// The gradient, face and update phases then read shared memory only.  A face's flux is written
// over the first 32 bytes of its own record (read only by the thread that computes it).
// The mbarrier wait is bounded (kTmaWaitCycles, about half a second): a block whose wait runs out
// records CFD_ERR_TIMEOUT in the status word and ends.
constexpr int kTmaGW = kTileX + 3, kTmaGH = kTileY + 2;  // W-face records: i0-1 .. i0+TX+1, j0-1 .. j0+TY
constexpr int kTmaSW = kTileX + 2, kTmaSH = kTileY + 3;  // S-face records: i0-1 .. i0+TX, j0-1 .. j0+TY+1
constexpr int kTmaRecD = 6;                              // doubles per face record
constexpr int kTmaSin = 11;  // stage inputs per own cell: U^n [4], stage state [4], frozen dt, a, area
// PRE (true): the stage inputs are prefetched into shared memory at block start (96 KB per block,
// 2 blocks per SM); false: they are loaded where they are used, which leaves room for 3 blocks per
// SM (74 KB each, registers capped at 85).
constexpr unsigned kTmaQBytes = kTileQW * kTileQH * 32u;
constexpr unsigned kTmaGWBytes = kTmaGW * kTmaGH * kTmaRecD * 8u;
constexpr unsigned kTmaGSBytes = kTmaSW * kTmaSH * kTmaRecD * 8u;
constexpr long long kTmaWaitCycles = 1ll << 30;
// Threads of the wide variant: 9 warps for the 256 cells of a tile, so the 552 face fluxes take
// two rounds instead of three (the ninth warp has no own cell; it loads and computes gradients and
// faces).  112 registers x 288 threads still leaves two blocks per SM.
constexpr int kTileThreadsWide = 288;

__host__ __device__ constexpr unsigned tma_round128(unsigned x) { return (x + 127u) & ~127u; }

template <typename T, bool PRE>
struct TileTmaLayout {
  static constexpr unsigned q = 0;
  static constexpr unsigned gw = tma_round128(kTmaQBytes);
  static constexpr unsigned gs = gw + tma_round128(kTmaGWBytes);
  static constexpr unsigned rec = gs + tma_round128(kTmaGSBytes);
  static constexpr unsigned sin =
      rec + tma_round128(2u * (unsigned)sizeof(typename TileRecT<T>::type) * kTileRW * kTileRH);
  static constexpr unsigned ia = sin + (PRE ? kTmaSin * kTileX * kTileY * 8u : 0u);
  static constexpr unsigned code = ia + kTileRW * kTileRH * 8u;
  static constexpr unsigned bar = (code + kTileRW * kTileRH + 7u) & ~7u;
  static constexpr unsigned bytes = bar + 8u + 128u;  // + slack to align the base to 128 bytes
};

__device__ __forceinline__ uint32_t sm_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sm_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap *map, int x, int y, int z) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(x), "r"(y), "r"(z)
               : "memory");
}
// L2 prefetch of the bytes [p, p + n) (widened to 16-byte bounds, as the bulk prefetch needs).
__device__ __forceinline__ void l2_prefetch_range(const void *p, size_t n) {
  if (n == 0) return;
  const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~static_cast<uintptr_t>(15);
  const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + n + 15) & ~static_cast<uintptr_t>(15);
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(static_cast<unsigned>(e - a)) : "memory");
}
__device__ __forceinline__ bool tma_bar_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > kTmaWaitCycles) return false;
  }
}

// Gradients of cell (gi, gj) of the tile's gradient region (row ri = (gj + 1) * kTileRW + gi + 1)
// as tile_gradients forms them, the face values read from the shared records.
__device__ __forceinline__ void tile_gradients_sm(const TileMesh &tm, const double4 *sq, const double *sgw,
                                                  const double *sgs, int qi, int gi, int gj, unsigned code, double ia,
                                                  double ac, double g[8], double &den) {
  const double *fp4[4];
  const int up = tm.lh ? 3 : 1, dn = tm.lh ? 1 : 3;
  fp4[0] = sgw + kTmaRecD * ((gj + 1) * kTmaGW + gi + 2);
  fp4[2] = sgw + kTmaRecD * ((gj + 1) * kTmaGW + gi + 1);
  fp4[up] = sgs + kTmaRecD * ((gj + 2) * kTmaSW + gi + 1);
  fp4[dn] = sgs + kTmaRecD * ((gj + 1) * kTmaSW + gi + 1);
  int dq[4];
  dq[0] = 1;
  dq[2] = -1;
  dq[up] = kTileQW;
  dq[dn] = -kTileQW;
  const double4 qv = sq[qi];
  const double qc[4] = {qv.x, qv.y, qv.z, qv.w};
  double t[4][9];
#pragma unroll
  for (int p = 0; p < 4; p++) {
    const double2 nxy = *reinterpret_cast<const double2 *>(fp4[p]);
    const double dlf = fp4[p][2];
    const double4 qn = sq[qi + dq[p]];
    const bool own = (code >> (2 + p)) & 1u;
    const double nxf = own ? nxy.x : -nxy.x, nyf = own ? nxy.y : -nxy.y;
    const double wx = nxf * dlf, wy = nyf * dlf;
    const double qnv[4] = {qn.x, qn.y, qn.z, qn.w};
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double qf = 0.5 * (qc[k] + qnv[k]);
      t[p][2 * k] = qf * wx;
      t[p][2 * k + 1] = qf * wy;
    }
    const double vnf = qc[1] * nxf + qc[2] * nyf;
    t[p][8] = (fabs(vnf) + ac) * dlf;
  }
  double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  slot_order_sum<9>(code & 3u, t, acc);
#pragma unroll
  for (int k = 0; k < 8; k++) g[k] = acc[k] * ia;
  den = acc[8];
}

template <typename T, int DISS, bool PRE, int NTHR>
__global__ void __launch_bounds__(NTHR, PRE ? 2 : 3)
    k_tile_tma(DevMesh m, DevState st, FluxParams fp, BcParams bp, TileMesh tm, const __grid_constant__ TileMaps maps,
               const double4 *__restrict__ q_in, int kind, int lts, int fuse_final, int keep_delu, int flags,
               int with_dt, int ahead) {
  typedef typename TileRecT<T>::type RecV;
  typedef TileTmaLayout<T, PRE> L;
  pdl_enter();
  if (step_done(st.ctl)) return;
  extern __shared__ unsigned char tma_smem_raw[];
  unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(tma_smem_raw) + 127) &
                                                          ~static_cast<uintptr_t>(127));
  double4 *sq = reinterpret_cast<double4 *>(base + L::q);          // [QH][QW]
  double *sgw = reinterpret_cast<double *>(base + L::gw);          // [GH][GW][6]
  double *sgs = reinterpret_cast<double *>(base + L::gs);          // [SH][SW][6]
  RecV *srec = reinterpret_cast<RecV *>(base + L::rec);            // [RH][RW] x 2
  double *sin = reinterpret_cast<double *>(base + L::sin);         // [kTmaSin][TX * TY]
  double *sia = reinterpret_cast<double *>(base + L::ia);          // [RH][RW]
  unsigned char *scode = base + L::code;                           // [RH][RW]
  const uint32_t bar = sm_u32(base + L::bar);
  const int NP = m.NP, NT = m.NT, ni = tm.ni, nj = tm.nj, tid = threadIdx.x;
  constexpr int NC = kTileX * kTileY;
  static_assert(NTHR >= NC && NTHR % 32 == 0, "one thread per own cell, whole warps");
  static_assert(2 * NTHR >= kTileQW * kTileQH && 2 * NTHR >= kTileRW * kTileRH, "two region rows per thread");
  const int i0 = (blockIdx.x % tm.tiles_i) * kTileX, j0 = (blockIdx.x / tm.tiles_i) * kTileY;
  const int glim = fp.limiter == LIM_REF_MINMOD ? LIM_MINMOD : fp.limiter;
  const bool first = first_kind(kind);
  const bool use_s = kind == 2 || kind == 3 || kind == 22 || kind == 23;

  // 0. Loads.  The mbarrier is initialised, made visible to the async proxy and to the block,
  // then thread 0 posts the byte count and issues the three tensor loads.
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                 "r"(kTmaQBytes + kTmaGWBytes + kTmaGSBytes)
                 : "memory");
    tma_load_3d(sm_u32(sgw), &maps.gw, 0, i0 - 1, j0 - 1, bar);
    tma_load_3d(sm_u32(sgs), &maps.gs, 0, i0 - 1, j0 - 1, bar);
    tma_load_3d(sm_u32(sq), &maps.q, 0, i0 - 2, j0 - 2, bar);
  }
  // Stage inputs of the own cell (thread tid has cell tid of the tile).
  const int tx = tid % kTileX, ty = tid / kTileX;
  const int ci = i0 + tx, cj = j0 + ty;
  const bool own_ok = tid < NC && ci < ni && cj < nj;
  const int c = cj * ni + ci;
  if (PRE && own_ok) {
#pragma unroll
    for (int k = 0; k < 4; k++) cp_async8(sin + k * NC + tid, st.U + (size_t)k * NT + c);
    if (use_s) {
#pragma unroll
      for (int k = 0; k < 4; k++) cp_async8(sin + (4 + k) * NC + tid, st.S + (size_t)k * NP + c);
    }
    if (lts != 1 && !first) cp_async8(sin + 8 * NC + tid, st.dtk + c);
    if (with_dt) {
      cp_async8(sin + 9 * NC + tid, st.prim + 4 * (size_t)NT + c);
      cp_async8(sin + 10 * NC + tid, m.area + c);
    }
  }
  // 1/area and slot codes of the gradient region (tile + one ring, cells inside the block).
  constexpr int NR = kTileRW * kTileRH;
  unsigned char code_r[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int r = tid + h * NTHR;
    if (r < NR) {
      const int gi = r % kTileRW - 1, gj = r / kTileRW - 1;
      const int i = i0 + gi, j = j0 + gj;
      if (i >= 0 && i < ni && j >= 0 && j < nj) {
        cp_async8(sia + r, m.inv_area + (j * ni + i));
        code_r[h] = tm.code[j * ni + i];
      }
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // Ghost rows beside the block's rim in the state region (the tensor load leaves zeros there).
  constexpr int NQ = kTileQW * kTileQH;
  double4 gq[2];
  int gpos[2] = {-1, -1};
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int t = tid + h * NTHR;
    if (t < NQ) {
      const int jj = t / kTileQW, ii = t - jj * kTileQW;
      const int i = i0 + ii - 2, j = j0 + jj - 2;
      const bool in_i = i >= 0 && i < ni, in_j = j >= 0 && j < nj;
      int r = -1;
      if (in_j && i == -1) r = tm.gW[j];
      else if (in_j && i == ni) r = tm.gE[j];
      else if (in_i && j == -1) r = tm.gS[i];
      else if (in_i && j == nj) r = tm.gN[i];
      if (r >= 0) {
        gq[h] = q_in[r];
        gpos[h] = t;
      }
    }
  }
  const bool landed = tma_bar_wait(bar, 0);
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (__syncthreads_or(!landed)) {
    // Record the timeout, then give the copies in flight one more bounded wait before the block
    // (and its shared memory) goes away.
    if (tid == 0) atomicCAS(st.status, 0, 5 /* CFD_ERR_TIMEOUT */);
    tma_bar_wait(bar, 0);
    return;
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (gpos[h] >= 0) sq[gpos[h]] = gq[h];
    const int r = tid + h * NTHR;
    if (r < NR) scode[r] = code_r[h];
  }
  __syncthreads();
  // Every thread has passed its wait: the mbarrier is retired.
  if (tid == 0) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(bar) : "memory");

  // L2 prefetch of the inputs of tile blockIdx.x + ahead (the tile that starts on this SM's slot in
  // the next wave, ahead = resident blocks of the grid), while this tile computes: its three tensor
  // boxes, and the rows of its stage inputs, 1/area and slot codes.  Hints only; the data are final.
  if (ahead > 0 && blockIdx.x + ahead < gridDim.x) {
    const int nbk = blockIdx.x + ahead;
    const int pi0 = (nbk % tm.tiles_i) * kTileX, pj0 = (nbk / tm.tiles_i) * kTileY;
    if (tid == 0) {
      tma_prefetch_3d(&maps.gw, 0, pi0 - 1, pj0 - 1);
      tma_prefetch_3d(&maps.gs, 0, pi0 - 1, pj0 - 1);
      tma_prefetch_3d(&maps.q, 0, pi0 - 2, pj0 - 2);
    } else if (tid >= 32 && tid < 32 + kTileRH) {
      // rows of the gradient region (1/area, slot codes) and of the own cells (stage inputs)
      const int gj = tid - 32 - 1, j = pj0 + gj;
      if (j >= 0 && j < nj) {
        const int ia0 = max(pi0 - 1, 0), ia1 = min(pi0 + kTileX + 1, ni);
        const size_t r0 = (size_t)j * ni;
        l2_prefetch_range(m.inv_area + r0 + ia0, (size_t)(ia1 - ia0) * 8);
        l2_prefetch_range(tm.code + r0 + ia0, (size_t)(ia1 - ia0));
        if (PRE && gj >= 0 && gj < kTileY) {
          const int o1 = min(pi0 + kTileX, ni);
          const size_t nb8 = (size_t)(o1 - pi0) * 8;
#pragma unroll
          for (int k = 0; k < 4; k++) l2_prefetch_range(st.U + (size_t)k * NT + r0 + pi0, nb8);
          if (use_s) {
#pragma unroll
            for (int k = 0; k < 4; k++) l2_prefetch_range(st.S + (size_t)k * NP + r0 + pi0, nb8);
          }
          if (lts != 1 && !first) l2_prefetch_range(st.dtk + r0 + pi0, nb8);
          if (with_dt) {
            l2_prefetch_range(st.prim + 4 * (size_t)NT + r0 + pi0, nb8);
            l2_prefetch_range(m.area + r0 + pi0, nb8);
          }
        }
      }
    }
  }

  // 1. Gradients: own cells (thread tid has cell tid), then the halo strips W, E, S, N.
  double dtc = 0.0;
  constexpr int NG = kTileX * kTileY + 2 * kTileY + 2 * kTileX;
  for (int t = tid; t < NG; t += blockDim.x) {
    int gi, gj;
    if (t < kTileX * kTileY) {
      gi = t % kTileX;
      gj = t / kTileX;
    } else {
      const int u = t - kTileX * kTileY;
      if (u < kTileY) {
        gi = -1;
        gj = u;
      } else if (u < 2 * kTileY) {
        gi = kTileX;
        gj = u - kTileY;
      } else if (u < 2 * kTileY + kTileX) {
        gi = u - 2 * kTileY;
        gj = -1;
      } else {
        gi = u - 2 * kTileY - kTileX;
        gj = kTileY;
      }
    }
    const int i = i0 + gi, j = j0 + gj;
    if (i < 0 || i >= ni || j < 0 || j >= nj) continue;
    const bool own = t < kTileX * kTileY;
    const bool dt = own && with_dt;
    const int ri = (gj + 1) * kTileRW + gi + 1;
    double g[8], den;
    const double ac = dt ? (PRE ? sin[9 * NC + t] : st.prim[4 * (size_t)NT + c]) : 0.0;
    tile_gradients_sm(tm, sq, sgw, sgs, (gj + 2) * kTileQW + gi + 2, gi, gj, scode[ri], sia[ri], ac, g, den);
    RecV *r = srec + 2 * ri;
    if (sizeof(T) == sizeof(float)) {
      r[0] = RecV{T(float(g[0])), T(float(g[1])), T(float(g[2])), T(float(g[3]))};
      r[1] = RecV{T(float(g[4])), T(float(g[5])), T(float(g[6])), T(float(g[7]))};
    } else {
      r[0] = RecV{T(g[0]), T(g[1]), T(g[2]), T(g[3])};
      r[1] = RecV{T(g[4]), T(g[5]), T(g[6]), T(g[7])};
    }
    if (dt) {
      dtc = cell_dt_a(fp, PRE ? sin[10 * NC + t] : m.area[c], den);
      st.dtc[c] = dtc;
    }
  }
  __syncthreads();

  // 2. Face fluxes: W faces (i0..i0+TX, rows of the tile), then S faces (columns, j0..j0+TY);
  // each flux over the first four doubles of its own record.
  for (int t = tid; t < kTileNW + kTileNS; t += blockDim.x) {
    int lx, ly, hx, hy;
    bool lo_phys, hi_phys;
    double *rec;
    if (t < kTileNW) {
      const int fj = t / (kTileX + 1), fi = t - fj * (kTileX + 1);
      const int i = i0 + fi, j = j0 + fj;
      if (i > ni || j >= nj) continue;
      rec = sgw + kTmaRecD * ((fj + 1) * kTmaGW + fi + 1);
      lx = fi - 1;
      ly = fj;
      hx = fi;
      hy = fj;
      lo_phys = i > 0;
      hi_phys = i < ni;
    } else {
      const int u = t - kTileNW;
      const int fj = u / kTileX, fi = u - fj * kTileX;
      const int i = i0 + fi, j = j0 + fj;
      if (i >= ni || j > nj) continue;
      rec = sgs + kTmaRecD * ((fj + 1) * kTmaSW + fi + 1);
      lx = fi;
      ly = fj - 1;
      hx = fi;
      hy = fj;
      lo_phys = j > 0;
      hi_phys = j < nj;
    }
    const double2 g01 = *reinterpret_cast<const double2 *>(rec);
    const double2 g23 = *reinterpret_cast<const double2 *>(rec + 2);
    const double2 g45 = *reinterpret_cast<const double2 *>(rec + 4);
    const bool ohigh = g45.y != 0.0;
    const int ox = ohigh ? hx : lx, oy = ohigh ? hy : ly, nx_ = ohigh ? lx : hx, ny_ = ohigh ? ly : hy;
    const bool nphys = ohigh ? lo_phys : hi_phys;
    const double4 c0 = sq[(oy + 2) * kTileQW + ox + 2], n0 = sq[(ny_ + 2) * kTileQW + nx_ + 2];
    const RecV *ro = srec + 2 * ((oy + 1) * kTileRW + ox + 1);
    const RecV *rn = nphys ? srec + 2 * ((ny_ + 1) * kTileRW + nx_ + 1) : ro;
    const RecV a = ro[0], b = ro[1], p = rn[0], q = rn[1];
    const double4 c1 = make_double4(a.x, a.y, a.z, a.w), c2 = make_double4(b.x, b.y, b.z, b.w);
    const double4 n1 = make_double4(p.x, p.y, p.z, p.w), n2 = make_double4(q.x, q.y, q.z, q.w);
    Ieee<T> o;
    const double4 F = face_flux_rec<T, DISS>(o, glim, c0, c1, c2, n0, n1, n2, T(g01.x), T(g01.y), T(g23.x), T(g23.y),
                                             T(g45.x), T(fp.eflin), T(fp.shock_fix));
    *reinterpret_cast<double2 *>(rec) = make_double2(F.x, F.y);
    *reinterpret_cast<double2 *>(rec + 2) = make_double2(F.z, F.w);
  }
  __syncthreads();

  // 3. Gather in slot order and stage update of the own cells.
  double dtu = 1e308 * 10.0;
  double e[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (own_ok) {
    const unsigned code = scode[(ty + 1) * kTileRW + tx + 1];
    const double *fE = sgw + kTmaRecD * ((ty + 1) * kTmaGW + tx + 2);
    const double *fW = sgw + kTmaRecD * ((ty + 1) * kTmaGW + tx + 1);
    const double *fN = sgs + kTmaRecD * ((ty + 2) * kTmaSW + tx + 1);
    const double *fS = sgs + kTmaRecD * ((ty + 1) * kTmaSW + tx + 1);
    const double *pf[4] = {fE, tm.lh ? fS : fN, fW, tm.lh ? fN : fS};
    double t[4][4];
#pragma unroll
    for (int p = 0; p < 4; p++) {
      const double2 a = *reinterpret_cast<const double2 *>(pf[p]);
      const double2 b = *reinterpret_cast<const double2 *>(pf[p] + 2);
      const bool own = (code >> (2 + p)) & 1u;
      t[p][0] = own ? a.x : -a.x;
      t[p][1] = own ? a.y : -a.y;
      t[p][2] = own ? b.x : -b.x;
      t[p][3] = own ? b.y : -b.y;
    }
    double R[4] = {0.0, 0.0, 0.0, 0.0};
    slot_order_sum<4>(code & 3u, t, R);
    // Ghost rows move to the output buffer with their owner (as in k_tile_stage).
    const int b0 = m.bptr[c], b1 = m.bptr[c + 1];
    for (int q = b0; q < b1; q++) {
      const int g = m.bnd[m.bidx[q]].w;
      st.q4[g] = q_in[g];
    }
    const double dts = (lts == 1 || first) ? dtc : 0.0;
    if (PRE) {
      StageIn in;
      in.invA = sia[(ty + 1) * kTileRW + tx + 1];
#pragma unroll
      for (int k = 0; k < 4; k++) in.Un[k] = sin[k * NC + tid];
      if (use_s) {
#pragma unroll
        for (int k = 0; k < 4; k++) in.Sk[k] = sin[(4 + k) * NC + tid];
      }
      const double dt_frozen = (lts != 1 && !first) ? sin[8 * NC + tid] : 0.0;
      dtu = stage_cell_in(m, st, bp, c, R, dts, dt_frozen, in, kind, lts, fuse_final, keep_delu, flags, e);
    } else {
      dtu = stage_cell(m, st, bp, c, R, dts, kind, lts, fuse_final, keep_delu, flags, e);
    }
  }
  // The state region is no longer read: its first 2.4 KB hold the reduction scratch.
  if (fuse_final && final_kind(kind)) stage_final_reduce_sm(st, e, dtu, reinterpret_cast<double *>(sq));
}

__global__ void k_gradient(DevMesh m, DevState st, int var, double *grad) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.NP) return;
  double g0, g1;
  gg_gradient(m, st.prim + (size_t)var * m.NT, c, g0, g1);
  grad[2 * c] = g0;
  grad[2 * c + 1] = g1;
}

// Compute_Gradient_Refinement_Indicator (src/Grid_Refine_Functions.cpp:8-31).
__global__ void k_amr_indicator(DevMesh m, DevState st, double *ind) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.NP) return;
  double v = 0.0;
  const double h = sqrt(m.area[c]);
  double g0, g1;
  gg_gradient(m, st.prim, c, g0, g1);
  v += sqrt(g0 * g0 + g1 * g1) * h;
  gg_gradient(m, st.prim + 3 * (size_t)m.NT, c, g0, g1);
  const double P = st.prim[3 * m.NT + c];
  if (P > 1e-14) v += (sqrt(g0 * g0 + g1 * g1) / P) * h;
  ind[c] = v;
}

__global__ void k_set_ctl(double *ctl, int idx, double v) { ctl[idx] = v; }

// sum(R_rho^2) over one instance's cell range per block: fixed per-thread strides and a fixed
// block tree, so the value is deterministic.
__global__ void k_instance_residual(const double *R, const int *start, const int *end, double *out) {
  __shared__ double sh[32];
  const int i = blockIdx.x;
  double acc = 0.0;
  for (int c = start[i] + threadIdx.x; c < end[i]; c += blockDim.x) acc += R[c] * R[c];
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) out[i] = acc;
}

// ---- Pointwise evaluation of the face functions (checkers' entry points) ----
// phi(a, b) of the limiter family for n pairs.
__global__ void k_eval_limiter(int limiter, const double *a, const double *b, int n, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = phi_ab<double>(limiter, a[i], b[i]);
}

// Face flux of scheme `scheme` (3 Roe average + dissipation, 6 AUSM, 7 HLLC, 8 reference GPU AUSM)
// for n conserved left/right states [n][4], outward normals [n][2] and lengths [n]; T is the
// arithmetic precision (the states are rounded to T first, as in the FP32-flux form).  Primitive
// variables for Roe and HLLC come from the reference EOS (eos_prim).
template <typename T, typename O>
__device__ __forceinline__ void eval_face(O &o, int scheme, const double *UL, const double *UR, const double *nrm,
                                          const double *len, int i, double *F) {
  const T nx = T(nrm[2 * i]), ny = T(nrm[2 * i + 1]), dl = T(len[i]);
  T A[4], D[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
  const T uL[4] = {T(UL[4 * i]), T(UL[4 * i + 1]), T(UL[4 * i + 2]), T(UL[4 * i + 3])};
  const T uR[4] = {T(UR[4 * i]), T(UR[4 * i + 1]), T(UR[4 * i + 2]), T(UR[4 * i + 3])};
  if (scheme == 6) {
    ausm_face<T>(o, uL, uR, nx, ny, dl, A);
  } else if (scheme == 8) {
    ausm_gpu_face<T>(uL, uR, nx, ny, dl, A);
  } else {
    Prim pl, pr;
    eos_prim(UL[4 * i], UL[4 * i + 1], UL[4 * i + 2], UL[4 * i + 3], pl);
    eos_prim(UR[4 * i], UR[4 * i + 1], UR[4 * i + 2], UR[4 * i + 3], pr);
    const T qL[5] = {T(pl.rho), T(pl.u), T(pl.v), T(pl.p), T(pl.a)};
    const T qR[5] = {T(pr.rho), T(pr.u), T(pr.v), T(pr.p), T(pr.a)};
    if (scheme == 7) {
      hllc_face<T>(o, qL, uL, qR, uR, nx, ny, dl, A);
    } else {
      average_flux<T>(qL[0], qL[1], qL[2], qL[3], qR[0], qR[1], qR[2], qR[3], nx, ny, dl, A);
      roe_1o<T>(o, qL[0], qL[1], qL[2], qL[3], qL[4], qR[0], qR[1], qR[2], qR[3], qR[4], nx, ny, dl, false, D);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; k++) F[4 * i + k] = double(A[k] - D[k]);
}

template <typename T>
__global__ void k_eval_face_flux(int scheme, const double *UL, const double *UR, const double *nrm, const double *len,
                                 int n, double *F) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  FaceOps<T> o;
  eval_face<T>(o, scheme, UL, UR, nrm, len, i, F);
  if (o.bad()) {
    Ieee<T> again;
    eval_face<T>(again, scheme, UL, UR, nrm, len, i, F);
  }
}

// ---- AMR tagging (TagRefinableCells, src/Grid_Refine_Functions.cpp:33-63) on the device ----
// Top-fraction rule: the nRefine largest indicators are found by a radix select over the bit
// patterns of the (non-negative) indicators, 8 bits per pass; ties at the cut are resolved by a
// second radix select over the reference cell ids (lowest ids first).  Counts are integer
// atomics, so the result is deterministic.
struct SelectState {
  unsigned long long prefix;  // key digits fixed so far
  unsigned long long mask;    // bits of prefix that are fixed
  long long remaining;        // rank still to find inside the current prefix
  long long above;            // number of keys strictly beyond the prefix
};

__device__ __forceinline__ unsigned long long amr_key(double v) {
  return v > 0.0 ? static_cast<unsigned long long>(__double_as_longlong(v)) : 0ull;
}

// Histogram of the next 8-bit digit of keys inside the current prefix.  mode 0: keys are the
// indicator bits (descending select); mode 1: keys are reference ids among cells whose indicator
// key equals `match` (ascending select).
__global__ void k_amr_hist(const double *ind, const int *ref, int NP, const SelectState *sel, int shift, int mode,
                           unsigned long long match, unsigned int *hist) {
  __shared__ unsigned int h[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) h[i] = 0u;
  __syncthreads();
  const unsigned long long prefix = sel->prefix, mask = sel->mask;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < NP; c += gridDim.x * blockDim.x) {
    unsigned long long key;
    if (mode == 0) key = amr_key(ind[c]);
    else {
      if (amr_key(ind[c]) != match) continue;
      key = static_cast<unsigned long long>(ref[c]);
    }
    if ((key & mask) == prefix) atomicAdd(&h[(key >> shift) & 255ull], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// Picks the digit holding the wanted rank (from the top for mode 0, from the bottom for mode 1)
// and clears the histogram for the next pass.
__global__ void k_amr_pick(SelectState *sel, int shift, int mode, unsigned int *hist) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  long long rem = sel->remaining;
  long long skipped = 0;
  int digit = 0;
  for (int i = 0; i < 256; i++) {
    const int d = mode == 0 ? 255 - i : i;
    const long long cnt = hist[d];
    if (rem <= cnt) {
      digit = d;
      break;
    }
    rem -= cnt;
    skipped += cnt;
  }
  sel->prefix |= static_cast<unsigned long long>(digit) << shift;
  sel->mask |= 255ull << shift;
  sel->remaining = rem;
  sel->above += skipped;
  for (int i = 0; i < 256; i++) hist[i] = 0u;
}

__global__ void k_amr_tag(const double *ind, const int *ref, int NP, double threshold, int top, const SelectState *sel,
                          const SelectState *sel_ref, uint8_t *tags) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= NP) return;
  const double v = ind[c];
  bool t;
  if (!top) {
    t = v > threshold;
  } else {
    const unsigned long long k = amr_key(v), K = sel->prefix;
    const bool in = k > K || (k == K && static_cast<unsigned long long>(ref[c]) <= sel_ref->prefix);
    t = in && v >= threshold;
  }
  tags[c] = t ? 1 : 0;
}

// Reference-order AoS rows [NT][4] <-> device-order SoA planes [4][NT] (perm: device -> reference).
__global__ void k_import_aos(const double *__restrict__ aos, const int *__restrict__ perm, int NP, int NT, double *U) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NT) return;
  const int r = i < NP ? perm[i] : i;
  const double4 v = reinterpret_cast<const double4 *>(aos)[r];
  U[i] = v.x;
  U[NT + i] = v.y;
  U[2 * NT + i] = v.z;
  U[3 * NT + i] = v.w;
}

__global__ void k_export_aos(const double *__restrict__ U, const int *__restrict__ perm, int NP, int NT, int ld,
                             double *aos) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NT) return;
  const int r = i < NP ? perm[i] : i;
  reinterpret_cast<double4 *>(aos)[r] = make_double4(U[i], U[ld + i], U[2 * ld + i], U[3 * ld + i]);
}

inline int nblk(int n, int b) { return (n + b - 1) / b; }

}  // namespace

// Upper bound on the thread blocks of any flux-kernel variant (sizes the partial-min buffer).
int flux_block_count(int NP) {
  int a = nblk(NP, kFluxBlock), b = nblk(4 * NP, kFlux4Block), c = nblk(NP, kBlock);
  return a > b ? (a > c ? a : c) : (b > c ? b : c);
}

int launch_prim_all(cudaStream_t s, const DevMesh &m, DevState &st) {
  k_prim_all<<<nblk(m.NT, kBlock), kBlock, 0, s>>>(m, st);
  return 1;
}

int launch_bc(cudaStream_t s, const DevMesh &m, DevState &st, const BcParams &bp, int src_is_S, int cur_is_S) {
  if (m.NB == 0) return 0;
  if (m.bblk) {
    if (m.n_bblk == 0) return 0;
    launch_k(m, k_bc, m.n_bblk, kWorkItemBlock, s, m, st, bp, src_is_S, cur_is_S);
  } else {
    launch_k(m, k_bc, nblk(m.NB, kBlock), kBlock, s, m, st, bp, src_is_S, cur_is_S);
  }
  return 1;
}

int launch_instance_residual(cudaStream_t s, const DevState &st, int NP, const int *start, const int *end, int n,
                             double *out) {
  (void)NP;
  if (n <= 0) return 0;
  k_instance_residual<<<n, 256, 0, s>>>(st.R, start, end, out);
  return 1;
}

template <typename T>
void launch_faces_t(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp);

// Lax_Fedrichs (src/Numerical_Method.cpp:459-481): U_c = 0.25 (U_N0 + U_N1 + U_N2 + U_N3) -
// Min_dt A^-1 R_c, in place.  The reference sweeps the cells in its own order, so a cell reads the
// neighbours that come before it with their new values and the others with their old ones.  One
// launch per wavefront level: a cell's level is one more than the highest level of its earlier
// neighbours, so no two cells of a level are neighbours, a level's earlier neighbours are all
// done and its later ones not yet started; every cell then sees what the sequential sweep shows
// it, and the sums are the same bits.
__global__ void __launch_bounds__(kBlock) k_lax_friedrichs(DevMesh m, DevState st, const int *cells, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cells[i];
  const int NP = m.NP, NT = m.NT;
  const int n0 = m.nbr[c], n1 = m.nbr[NP + c], n2 = m.nbr[2 * NP + c], n3 = m.nbr[3 * NP + c];
  const double Dt = st.ctl[CTL_DTMIN];
  const double ia = m.inv_area[c];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double *U = st.U + (size_t)k * NT;
    st.U[(size_t)k * NT + c] = 0.25 * (U[n0] + U[n1] + U[n2] + U[n3]) - Dt * ia * st.R[(size_t)k * NP + c];
  }
}

int launch_lax_friedrichs(cudaStream_t s, const DevMesh &m, DevState &st, const int *cells,
                          const std::vector<int> &level_start) {
  int n = 0;
  for (size_t l = 0; l + 1 < level_start.size(); l++) {
    const int b = level_start[l], e = level_start[l + 1];
    k_lax_friedrichs<<<nblk(e - b, kBlock), kBlock, 0, s>>>(m, st, cells + b, e - b);
    n++;
  }
  return n;
}

// A per-cell form that reads conserved states (limiter, LLF, MOVERS, MOVERS_NWSC, AUSM, HLLC): the
// build that reads them from U alone when no stage state can be asked for (the reference's
// integrators, and the first stage of every form), else the one that picks U or the stage state
// per cell.  Same bits either way.
template <int DISS, int ORDER>
void launch_flux_src(int g, cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, int src_is_S,
                     int want) {
  if (fp.consistent && src_is_S) launch_k(m, k_flux<DISS, ORDER, 6, true>, g, kFluxBlock, s, m, st, fp, src_is_S, want);
  else launch_k(m, k_flux<DISS, ORDER, 6, false>, g, kFluxBlock, s, m, st, fp, src_is_S, want);
}

// The second-order per-cell forms with the directional limiter (ROE_2O, RICCA_2O, MOVERS_NWSC_2O):
// one build per register budget (minimum resident blocks of 128 threads per SM: 1 unconstrained,
// 6 or 8), chosen by fp.flux_minb; every build gives the same bits.
template <int DISS>
void launch_flux_limited(int g, cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, int src_is_S,
                         int want) {
  if (!(fp.consistent && src_is_S)) {
    switch (fp.flux_minb) {
      case 1: launch_k(m, k_flux<DISS, 2, 1, false>, g, kFluxBlock, s, m, st, fp, src_is_S, want); break;
      case 8: launch_k(m, k_flux<DISS, 2, 8, false>, g, kFluxBlock, s, m, st, fp, src_is_S, want); break;
      default: launch_k(m, k_flux<DISS, 2, 6, false>, g, kFluxBlock, s, m, st, fp, src_is_S, want); break;
    }
    return;
  }
  switch (fp.flux_minb) {
    case 1: launch_k(m, k_flux<DISS, 2, 1>, g, kFluxBlock, s, m, st, fp, src_is_S, want); break;
    case 8: launch_k(m, k_flux<DISS, 2, 8>, g, kFluxBlock, s, m, st, fp, src_is_S, want); break;
    default: launch_k(m, k_flux<DISS, 2, 6>, g, kFluxBlock, s, m, st, fp, src_is_S, want); break;
  }
}

int launch_flux(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, int src_is_S, int want) {
  int n = 0;
  if (fp.second_order && fp.muscl) n += launch_muscl_gradients(s, m, st, fp, 0);
  if (fp.second_order && fp.muscl && m.NF > 0) {
    if (fp.precision == 1) launch_faces_t<float>(s, m, st, fp);
    else launch_faces_t<double>(s, m, st, fp);
    (st.recf ? k_gather<true> : k_gather<false>)<<<nblk(m.NP, kFluxBlock), kFluxBlock, 0, s>>>(m, st, fp);
    return n + 2;
  }
  if (fp.weno) {
    k_weno<<<nblk(m.NP, kFluxBlock), kFluxBlock, 0, s>>>(m, st, fp, src_is_S);
    return n + 1;
  }
  if (fp.lanes == 1) {
    const int g = nblk(m.NP, kFluxBlock);
    if (fp.dissipation == 3 && !fp.second_order) launch_k(m, k_flux<3, 1>, g, kFluxBlock, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 2 && !fp.second_order) launch_flux_src<2, 1>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 2) launch_flux_src<2, 2>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 4 && !fp.second_order) launch_k(m, k_flux<4, 1>, g, kFluxBlock, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 5 && !fp.second_order) launch_flux_src<5, 1>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 6) launch_flux_src<6, 1>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 7) launch_flux_src<7, 1>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 3) launch_flux_limited<3>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 4) launch_flux_limited<4>(g, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 5) launch_flux_limited<5>(g, s, m, st, fp, src_is_S, want);
    else launch_flux_src<1, 1>(g, s, m, st, fp, src_is_S, want);
  } else {
    const int g = nblk(4 * m.NP, kFlux4Block);
    if (fp.dissipation == 3 && !fp.second_order) launch_k(m, k_flux4<3, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 2 && !fp.second_order) launch_k(m, k_flux4<2, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 2) launch_k(m, k_flux4<2, 2>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 4 && !fp.second_order) launch_k(m, k_flux4<4, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 4) launch_k(m, k_flux4<4, 2>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 5 && !fp.second_order) launch_k(m, k_flux4<5, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 5) launch_k(m, k_flux4<5, 2>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 6) launch_k(m, k_flux4<6, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 7) launch_k(m, k_flux4<7, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else if (fp.dissipation == 3) launch_k(m, k_flux4<3, 2>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
    else launch_k(m, k_flux4<1, 1>, g, kFlux4Block, s, m, st, fp, src_is_S, want);
  }
  return n + 1;
}

int launch_stage(cudaStream_t s, const DevMesh &m, DevState &st, const BcParams &bp, int kind, int lts, int fuse_final,
                 int keep_delu, int flags) {
  const auto k = (flags & (kStageGhosts | kStageNextStep)) ? k_stage<true> : k_stage<false>;
  if (m.cblk) launch_k(m, k, m.n_cblk, kWorkCellBlock, s, m, st, bp, kind, lts, fuse_final, keep_delu, flags);
  else launch_k(m, k, nblk(m.NP, kBlock), kBlock, s, m, st, bp, kind, lts, fuse_final, keep_delu, flags);
  return 1;
}

int launch_gather(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp) {
  const int g = m.cblk ? m.n_cblk : nblk(m.NP, kFluxBlock);
  (st.recf ? k_gather<true> : k_gather<false>)<<<g, kFluxBlock, 0, s>>>(m, st, fp);
  return 1;
}

// Flux scheme of the face kernels: 3 (Roe) becomes 103 when the Roe options are on.
__host__ __forceinline__ int face_scheme(const FluxParams &fp) {
  return fp.dissipation == 3 && (fp.eflin > 0.0 || fp.shock_fix > 0.0) ? 103 : fp.dissipation;
}

template <typename T, int MINB>
void launch_faces_b(cudaStream_t s, int g, int b, const DevMesh &m, DevState &st, const FluxParams &fp) {
  if (face_scheme(fp) == 103) launch_k(m, k_faces<T, 103, MINB>, g, b, s, m, st, fp);
  else if (fp.dissipation == 6) launch_k(m, k_faces<T, 6, MINB>, g, b, s, m, st, fp);
  else if (fp.dissipation == 7) launch_k(m, k_faces<T, 7, MINB>, g, b, s, m, st, fp);
  else if (fp.dissipation == 8) launch_k(m, k_faces<T, 8, MINB>, g, b, s, m, st, fp);
  else launch_k(m, k_faces<T, 3, MINB>, g, b, s, m, st, fp);
}

// Launch shapes of the face kernel (identical results).  The double kernels take 114 registers
// unbounded: 256-thread blocks then fit 2 per SM (16 warps, shape 0), 256-thread blocks capped
// at 80 registers fit 3 (24 warps, 28 bytes of spill stores; shape 1), 128-thread blocks fit 4 (16
// warps; shape 2), 128-thread blocks capped at 72 or 64 registers fit 7 or 8 (28 or 32 warps,
// 36 or 8 bytes of spill stores held in L1; shapes 3 and 4).  Work lists hold kWorkFaceBlock (128)
// faces per block, so with them every shape runs 128-thread blocks.
template <typename T>
void launch_faces_t(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp) {
  const bool wl = m.fblk != nullptr;
  const int g128 = wl ? m.n_fblk : nblk(m.NF, 128);
  const int g = wl ? m.n_fblk : nblk(m.NF, 256), b = wl ? 128 : 256;
  if (fp.faces_shape == 4) launch_faces_b<T, 8>(s, g128, 128, m, st, fp);
  else if (fp.faces_shape == 3) launch_faces_b<T, 7>(s, g128, 128, m, st, fp);
  else if (fp.faces_shape == 2) launch_faces_b<T, 1>(s, g128, 128, m, st, fp);
  else if (fp.faces_shape == 1) launch_faces_b<T, 3>(s, g, b, m, st, fp);
  else launch_faces_b<T, 1>(s, g, b, m, st, fp);
}

int launch_faces(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp) {
  if (m.fblk && m.n_fblk == 0) return 0;
  if (fp.precision == 1) launch_faces_t<float>(s, m, st, fp);
  else launch_faces_t<double>(s, m, st, fp);
  return 1;
}

int device_sms();

int gather_stage_wave_blocks() {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gather_stage<true, false>, kFluxBlock, 0) != cudaSuccess)
    return 0;
  return sms * per_sm;
}

int launch_gather_stage(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                        int kind, int lts, int fuse_final, int keep_delu, int flags) {
  const int g = m.cblk ? m.n_cblk : nblk(m.NP, kFluxBlock);
  if (!m.cblk && fuse_final && final_kind(kind) && m.wave_blocks > 0 && g > m.wave_blocks)
    launch_k(m, st.recf ? k_gather_stage<true, true> : k_gather_stage<true, false>, m.wave_blocks, kFluxBlock, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu,
             flags);
  else
    launch_k(m, st.recf ? k_gather_stage<false, true> : k_gather_stage<false, false>, g, kFluxBlock, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu, flags);
  return 1;
}

// stage: 0 not the last, 1 the last.
int launch_gather_lean(cudaStream_t s, const DevMesh &m, const DevState &st, const BcParams &bp, int kind, int flags,
                       int store_a) {
  const int g = m.cblk ? m.n_cblk : nblk(m.NP, kFluxBlock);
  if (g == 0) return 0;
  if (final_kind(kind))
    launch_k(m, st.recf ? k_gather_lean<1, true> : k_gather_lean<1, false>, !m.cblk && m.lean_blocks > 0 ? std::min(g, m.lean_blocks) : g, kFluxBlock, s, m, st, bp,
             kind, flags, store_a);
  else launch_k(m, st.recf ? k_gather_lean<0, true> : k_gather_lean<0, false>, g, kFluxBlock, s, m, st, bp, kind, flags, store_a);
  return 1;
}

int gather_lean_wave_blocks() {
  int per_sm = 0;
  const int sms = device_sms();
  if (sms <= 0 || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gather_lean<1, false>, kFluxBlock, 0) != cudaSuccess)
    return 0;
  return sms * per_sm;
}

int launch_face_weights(cudaStream_t s, const DevMesh &m, double2 *gw) {
  k_face_weights<<<(unsigned)((4 * (size_t)m.NP + kBlock - 1) / kBlock), kBlock, 0, s>>>(m, gw);
  return 1;
}

int launch_face_records(cudaStream_t s, const DevMesh &m, float4 *r) {
  k_face_records<<<nblk(m.NF, kBlock), kBlock, 0, s>>>(m, r);
  return 1;
}

template <typename T>
int tile_prepare_t() {
  const int n = static_cast<int>(tile_smem_bytes<T>());
  return cudaFuncSetAttribute(k_tile_stage<T, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_stage<T, 103>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_stage<T, 6>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_stage<T, 7>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_stage<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) == cudaSuccess;
}

int tile_prepare() {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  if (tile_smem_bytes<double>() > (size_t)optin) return 0;
  const int ok = tile_prepare_t<double>() && tile_prepare_t<float>();
  cudaGetLastError();
  return ok;
}

template <typename T>
void launch_tile_t(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                   const TileMesh &tm, const double4 *q_in, int kind, int lts, int fin, int keep_delu, int flags,
                   int with_dt) {
  const unsigned g = static_cast<unsigned>(tm.tiles_i) * static_cast<unsigned>(tm.tiles_j);
  const unsigned b = kTileX * kTileY;
  const size_t sm = tile_smem_bytes<T>();
  const int sch = face_scheme(fp);
  if (sch == 103)
    launch_ks(m, k_tile_stage<T, 103>, g, b, sm, s, m, st, fp, bp, tm, q_in, kind, lts, fin, keep_delu, flags, with_dt);
  else if (sch == 6)
    launch_ks(m, k_tile_stage<T, 6>, g, b, sm, s, m, st, fp, bp, tm, q_in, kind, lts, fin, keep_delu, flags, with_dt);
  else if (sch == 7)
    launch_ks(m, k_tile_stage<T, 7>, g, b, sm, s, m, st, fp, bp, tm, q_in, kind, lts, fin, keep_delu, flags, with_dt);
  else if (sch == 8)
    launch_ks(m, k_tile_stage<T, 8>, g, b, sm, s, m, st, fp, bp, tm, q_in, kind, lts, fin, keep_delu, flags, with_dt);
  else
    launch_ks(m, k_tile_stage<T, 3>, g, b, sm, s, m, st, fp, bp, tm, q_in, kind, lts, fin, keep_delu, flags, with_dt);
}

int launch_tile_stage(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                      const TileMesh &tm, const double4 *q_in, int kind, int lts, int fuse_final, int keep_delu,
                      int flags, int with_dt) {
  if (fp.precision == 1)
    launch_tile_t<float>(s, m, st, fp, bp, tm, q_in, kind, lts, fuse_final, keep_delu, flags, with_dt);
  else
    launch_tile_t<double>(s, m, st, fp, bp, tm, q_in, kind, lts, fuse_final, keep_delu, flags, with_dt);
  return 1;
}

template <typename T, bool PRE, int NTHR>
int tile_tma_prepare_t() {
  const int n = static_cast<int>(TileTmaLayout<T, PRE>::bytes);
  const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  return cudaFuncSetAttribute(k_tile_tma<T, 3, PRE, NTHR>, a, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_tma<T, 103, PRE, NTHR>, a, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_tma<T, 6, PRE, NTHR>, a, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_tma<T, 7, PRE, NTHR>, a, n) == cudaSuccess &&
         cudaFuncSetAttribute(k_tile_tma<T, 8, PRE, NTHR>, a, n) == cudaSuccess;
}

int tile_tma_prepare() {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  if (TileTmaLayout<double, true>::bytes > (unsigned)optin) return 0;
  const int ok = tile_tma_prepare_t<double, true, kTileThreadsWide>() &&
                 tile_tma_prepare_t<float, true, kTileThreadsWide>() &&
                 tile_tma_prepare_t<double, true, kTileX * kTileY>() &&
                 tile_tma_prepare_t<float, true, kTileX * kTileY>() &&
                 tile_tma_prepare_t<double, false, kTileX * kTileY>() &&
                 tile_tma_prepare_t<float, false, kTileX * kTileY>();
  cudaGetLastError();
  return ok;
}

void tile_tma_boxes(int q[3], int gw[3], int gs[3]) {
  q[0] = 4;
  q[1] = kTileQW;
  q[2] = kTileQH;
  gw[0] = kTmaRecD;
  gw[1] = kTmaGW;
  gw[2] = kTmaGH;
  gs[0] = kTmaRecD;
  gs[1] = kTmaSW;
  gs[2] = kTmaSH;
}

template <typename T, bool PRE, int NTHR>
void launch_tile_tma_t(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                       const TileMesh &tm, const TileMaps &maps, const double4 *q_in, int kind, int lts, int fin,
                       int keep_delu, int flags, int with_dt) {
  const unsigned g = static_cast<unsigned>(tm.tiles_i) * static_cast<unsigned>(tm.tiles_j);
  const size_t sm = TileTmaLayout<T, PRE>::bytes;
  const int sch = face_scheme(fp);
  int ahead = 0;
  if (tm.prefetch_ahead) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tile_tma<T, 3, PRE, NTHR>, NTHR, sm) == cudaSuccess)
      ahead = sms * per_sm;
    cudaGetLastError();
  }
  if (sch == 103)
    launch_ks(m, k_tile_tma<T, 103, PRE, NTHR>, g, NTHR, sm, s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin,
              keep_delu, flags, with_dt, ahead);
  else if (sch == 6)
    launch_ks(m, k_tile_tma<T, 6, PRE, NTHR>, g, NTHR, sm, s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu,
              flags, with_dt, ahead);
  else if (sch == 7)
    launch_ks(m, k_tile_tma<T, 7, PRE, NTHR>, g, NTHR, sm, s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu,
              flags, with_dt, ahead);
  else if (sch == 8)
    launch_ks(m, k_tile_tma<T, 8, PRE, NTHR>, g, NTHR, sm, s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu,
              flags, with_dt, ahead);
  else
    launch_ks(m, k_tile_tma<T, 3, PRE, NTHR>, g, NTHR, sm, s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu,
              flags, with_dt, ahead);
}

template <typename T>
void launch_tile_tma_v(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                       const TileMesh &tm, const TileMaps &maps, const double4 *q_in, int kind, int lts, int fin,
                       int keep_delu, int flags, int with_dt, int variant) {
  if (variant == 1)
    launch_tile_tma_t<T, false, kTileX * kTileY>(s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu, flags,
                                                 with_dt);
  else if (variant == 2)
    launch_tile_tma_t<T, true, kTileThreadsWide>(s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu, flags,
                                                 with_dt);
  else
    launch_tile_tma_t<T, true, kTileX * kTileY>(s, m, st, fp, bp, tm, maps, q_in, kind, lts, fin, keep_delu, flags,
                                                with_dt);
}

int launch_tile_tma(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                    const TileMesh &tm, const TileMaps &maps, const double4 *q_in, int kind, int lts, int fuse_final,
                    int keep_delu, int flags, int with_dt, int variant) {
  if (fp.precision == 1)
    launch_tile_tma_v<float>(s, m, st, fp, bp, tm, maps, q_in, kind, lts, fuse_final, keep_delu, flags, with_dt,
                             variant);
  else
    launch_tile_tma_v<double>(s, m, st, fp, bp, tm, maps, q_in, kind, lts, fuse_final, keep_delu, flags, with_dt,
                              variant);
  return 1;
}

size_t patch_smem_bytes(const DevMesh &m) {
  return sizeof(double) * (12 * (size_t)m.patch_rows + 16 * (size_t)kPatchCells);
}

int patch_prepare(const DevMesh &m) {
  const size_t bytes = patch_smem_bytes(m);
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
  if (bytes + 4096 > (size_t)optin) return 0;
  const int n = static_cast<int>(bytes);
  if (cudaFuncSetAttribute(k_patch_stage<103>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) != cudaSuccess ||
      cudaFuncSetAttribute(k_patch_stage<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) != cudaSuccess ||
      cudaFuncSetAttribute(k_patch_stage<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) != cudaSuccess ||
      cudaFuncSetAttribute(k_patch_stage<7>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) != cudaSuccess ||
      cudaFuncSetAttribute(k_patch_stage<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, n) != cudaSuccess)
    return 0;
  return 1;
}

int launch_patch_stage(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, const BcParams &bp,
                       int kind, int lts, int fuse_final, int keep_delu, int flags, const double *prim_in) {
  const size_t sm = patch_smem_bytes(m);
  const int g = m.npatch;
  if (face_scheme(fp) == 103)
    launch_ks(m, k_patch_stage<103>, g, kPatchCells, sm, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu, flags,
              prim_in);
  else if (fp.dissipation == 6)
    launch_ks(m, k_patch_stage<6>, g, kPatchCells, sm, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu, flags,
              prim_in);
  else if (fp.dissipation == 7)
    launch_ks(m, k_patch_stage<7>, g, kPatchCells, sm, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu, flags,
              prim_in);
  else if (fp.dissipation == 8)
    launch_ks(m, k_patch_stage<8>, g, kPatchCells, sm, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu, flags,
              prim_in);
  else
    launch_ks(m, k_patch_stage<3>, g, kPatchCells, sm, s, m, st, fp, bp, kind, lts, fuse_final, keep_delu, flags,
              prim_in);
  return 1;
}

int launch_error(cudaStream_t s, const DevMesh &m, DevState &st) {
  k_error<<<nblk(m.NP, kBlock), kBlock, 0, s>>>(m, st);
  return 1;
}

int launch_eval_limiter(cudaStream_t s, int limiter, const double *a, const double *b, int n, double *out) {
  if (n <= 0) return 0;
  k_eval_limiter<<<nblk(n, kBlock), kBlock, 0, s>>>(limiter, a, b, n, out);
  return 1;
}

int launch_eval_face_flux(cudaStream_t s, int scheme, int precision, const double *UL, const double *UR,
                          const double *nrm, const double *len, int n, double *F) {
  if (n <= 0) return 0;
  if (precision == 1) k_eval_face_flux<float><<<nblk(n, kBlock), kBlock, 0, s>>>(scheme, UL, UR, nrm, len, n, F);
  else k_eval_face_flux<double><<<nblk(n, kBlock), kBlock, 0, s>>>(scheme, UL, UR, nrm, len, n, F);
  return 1;
}

int launch_update(cudaStream_t s, const DevMesh &m, DevState &st, int from_S) {
  k_update<<<nblk(m.NP, kBlock), kBlock, 0, s>>>(m, st, from_S);
  return 1;
}

int launch_gradient(cudaStream_t s, const DevMesh &m, DevState &st, int var, double *grad) {
  k_gradient<<<nblk(m.NP, kBlock), kBlock, 0, s>>>(m, st, var, grad);
  return 1;
}

template <typename T, int DISS>
void persistent_kernel_ptr(void (**k)(DevMesh, DevState, FluxParams, BcParams, int, int, int, int, int, int, int,
                                      unsigned int),
                           int minb) {
  if (minb == 0) minb = std::is_same<T, float>::value ? 8 : 6;  // the faster budget of each form on B200
  *k = minb == 8 ? k_persistent_stage<T, DISS, 8>
                  : minb == 6 ? k_persistent_stage<T, DISS, 6> : k_persistent_stage<T, DISS, 4>;
}

// Largest co-resident grid of the persistent stage kernel on this device (0: not available).
int persistent_grid(const FluxParams &fp) {
  void (*k)(DevMesh, DevState, FluxParams, BcParams, int, int, int, int, int, int, int, unsigned int) = nullptr;
  const bool f32 = fp.precision == 1;
  switch (face_scheme(fp)) {
    case 103: f32 ? persistent_kernel_ptr<float, 103>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 103>(&k, fp.persist_minb); break;
    case 6: f32 ? persistent_kernel_ptr<float, 6>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 6>(&k, fp.persist_minb); break;
    case 7: f32 ? persistent_kernel_ptr<float, 7>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 7>(&k, fp.persist_minb); break;
    case 8: f32 ? persistent_kernel_ptr<float, 8>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 8>(&k, fp.persist_minb); break;
    default: f32 ? persistent_kernel_ptr<float, 3>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 3>(&k, fp.persist_minb); break;
  }
  int dev = 0, sms = 0, per_sm = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kPersistBlock, 0) != cudaSuccess) return 0;
  return sms * per_sm;
}

int launch_persistent_stage(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp,
                            const BcParams &bp, int kind, int lts, int fuse_final, int keep_delu, int flags,
                            int with_dt, int with_bc, int grid, unsigned int test_arrivals) {
  void (*k)(DevMesh, DevState, FluxParams, BcParams, int, int, int, int, int, int, int, unsigned int) = nullptr;
  const bool f32 = fp.precision == 1;
  switch (face_scheme(fp)) {
    case 103: f32 ? persistent_kernel_ptr<float, 103>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 103>(&k, fp.persist_minb); break;
    case 6: f32 ? persistent_kernel_ptr<float, 6>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 6>(&k, fp.persist_minb); break;
    case 7: f32 ? persistent_kernel_ptr<float, 7>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 7>(&k, fp.persist_minb); break;
    case 8: f32 ? persistent_kernel_ptr<float, 8>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 8>(&k, fp.persist_minb); break;
    default: f32 ? persistent_kernel_ptr<float, 3>(&k, fp.persist_minb) : persistent_kernel_ptr<double, 3>(&k, fp.persist_minb); break;
  }
  DevMesh mm = m;
  DevState ss = st;
  FluxParams ff = fp;
  BcParams bb = bp;
  void *args[] = {&mm, &ss, &ff, &bb, &kind, &lts, &fuse_final, &keep_delu, &flags, &with_dt, &with_bc, &test_arrivals};
  cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k), dim3(grid), dim3(kPersistBlock), args, 0, s);
  return 1;
}

template <typename T>
void *steps_kernel_t(const FluxParams &fp) {
  switch (face_scheme(fp)) {
    case 103: return reinterpret_cast<void *>(k_steps<T, 103>);
    case 6: return reinterpret_cast<void *>(k_steps<T, 6>);
    case 7: return reinterpret_cast<void *>(k_steps<T, 7>);
    case 8: return reinterpret_cast<void *>(k_steps<T, 8>);
    default: return reinterpret_cast<void *>(k_steps<T, 3>);
  }
}
void *steps_kernel(const FluxParams &fp) { return fp.precision == 1 ? steps_kernel_t<float>(fp) : steps_kernel_t<double>(fp); }

int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return sms;
}

// Threads per cell of the per-cell flux kernel: four while they fit five blocks of 128 per SM, so that a
// small mesh still fills the chip and the four faces' chains run side by side.  Per pseudo-step of three
// stages (four lanes against one, LLF / ROE / ROE_2O / HLLC, B200): 27 / 29 / 29 / 30 us against
// 34 / 40 / 46 / 36 at 3,200 cells, 33 / 36 / 44 / 38 against 36 / 42 / 48 / 38 at 20,000,
// 47 / 52 / 62 / 52 against 37 / 48 / 56 / 44 at 45,451.
int flux_lanes_for(int cells) { return 4LL * cells <= 640LL * device_sms() ? 4 : 1; }

bool two_waves(int cells) { return cells >= 2LL * 6 * kFluxBlock * device_sms(); }

// Whether k_stage writes the next evaluation's ghosts or k_bc forms them in its own launch.  Per pseudo-step
// (k_stage / k_bc, B200): ROE_2O 54 / 58 us at 24,200 cells, 89 / 92 at 109,200, 136 / 136.5 at 180,000,
// 241 / 227 at 320,000, 381 / 354 at 524,288, ROE 270 / 244 there: with more than two waves the kernel's
// lower occupancy costs more than the launch.
bool stage_ghosts_for(int cells) { return !two_waves(cells); }

// Programmatic dependent launch pays from two waves of the six-blocks-per-SM kernels on: per pseudo-step at
// 524,288 cells 252 -> 249 us (gradient MUSCL), 225 -> 220 (FP32-flux), 358 -> 355 (ROE_2O), 239 -> 235
// (LLF).  Below, blocks that start while the previous kernel still holds part of the chip are spread unevenly
// over the SMs: ROE_2O at 45,451 cells 57 -> 64 us, at 11,250 35.4 -> 35.4 (B200).
int pdl_for(int cells) { return two_waves(cells) ? 1 : 0; }
int grad_ahead_for(int cells) { return two_waves(cells) ? device_sms() : 0; }

// Threads of a block whose widest phase has n items, in whole warps; at least four (reduce_rows takes
// three of the nine reduced quantities per warp).
int steps_threads(int n) {
  const int t = (n + 31) & ~31;
  return t < 128 ? 128 : (t > kStepsThreads ? kStepsThreads : t);
}

// This block's share of the items [begin, end): equal ranges of whole warps.
static int2 block_share(int begin, int end, int rank, int blocks) {
  const int per = (((end - begin + blocks - 1) / blocks) + 31) & ~31;
  const int lo = std::min(begin + rank * per, end);
  return make_int2(lo, std::min(lo + per, end));
}

// The line is the capacity: one block per SM, every share in its shared memory (about 101,000 cells of a
// structured block).  Up to there the launch is the faster or an equal form.  Per pseudo-step in one launch
// against the separate kernels (B200): FP64 58.9 / 67.6 us at 98,304 cells, 61.5 / 67.6 at 101,120, a batch of
// 49 channels (100,352) 60.7 / 69.9; FP32-flux 57.6 / 57.7, 60.3 / 59.7 and 59.3 / 63.4.
StepsShape steps_shape(const FluxParams &fp, const int *bptr, const int4 *inst, int instances,
                       std::vector<StepsBlock> &blocks) {
  StepsShape sh{};
  blocks.clear();
  const int sms = device_sms();
  int dev = 0, optin = 0, coop = 0;
  if (sms <= 0 || instances < 1 || instances > sms || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return sh;
  long long total = 0;
  for (int i = 0; i < instances; i++) total += inst[i].y - inst[i].x;
  if (total <= 0) return sh;
  // Blocks in proportion to the cells, at least one each and no more than hold a warp of cells.
  for (int i = 0; i < instances; i++) {
    const int n = inst[i].y - inst[i].x;
    int nb = static_cast<int>((long long)(sms - instances) * n / total) + 1;
    nb = std::min(nb, (n + 31) / 32);
    for (int r = 0; r < nb; r++) {
      const int2 c = block_share(inst[i].x, inst[i].y, r, nb), f = block_share(inst[i].z, inst[i].w, r, nb);
      blocks.push_back(StepsBlock{c.x, c.y, f.x, f.y, i, nb});
      sh.cells = std::max(sh.cells, c.y - c.x);
      sh.faces = std::max(sh.faces, f.y - f.x);
      sh.entries = std::max(sh.entries, c.y > c.x ? bptr[c.y] - bptr[c.x] : 0);
    }
  }
  sh.cells = (sh.cells + 3) & ~3;  // keeps the int4 tables behind the doubles aligned
  sh.faces = (sh.faces + 3) & ~3;
  const size_t sm = steps_smem(sh.cells, sh.faces, sh.entries);
  const int room = optin - 4096;  // static shared memory of the reductions
  const int threads = steps_threads(sh.faces);
  int per_sm = 0;
  void *k = steps_kernel(fp);
  if (sm <= (size_t)room &&
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, room) == cudaSuccess &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, sm) == cudaSuccess && per_sm >= 1 &&
      (int)blocks.size() <= sms) {
    sh.blocks = static_cast<int>(blocks.size());
    sh.threads = threads;
    sh.groups = instances;
  }
  cudaGetLastError();
  return sh;
}

const void *cell_steps_kernel(const FluxParams &fp) {
  const bool two = fp.second_order;
  switch (fp.dissipation) {
    case 1: return (const void *)k_cell_steps<1, 1>;
    case 2: return two ? (const void *)k_cell_steps<2, 2> : (const void *)k_cell_steps<2, 1>;
    case 3: return two ? (const void *)k_cell_steps<3, 2> : (const void *)k_cell_steps<3, 1>;
    case 4: return two ? (const void *)k_cell_steps<4, 2> : (const void *)k_cell_steps<4, 1>;
    case 5: return two ? (const void *)k_cell_steps<5, 2> : (const void *)k_cell_steps<5, 1>;
    case 6: return (const void *)k_cell_steps<6, 1>;
    case 7: return (const void *)k_cell_steps<7, 1>;
  }
  return nullptr;
}

bool cell_steps_available(const FluxParams &fp, int cells) {
  const void *k = cell_steps_kernel(fp);
  int dev = 0, coop = 0, per_sm = 0;
  if (!k || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kFlux4Block, 0) != cudaSuccess)
    return false;
  return nblk(4 * cells, kFlux4Block) <= per_sm * device_sms();
}

int launch_cell_steps(cudaStream_t s, const DevMesh &m, const DevState &st, const FluxParams &fp, const BcParams &bp,
                      unsigned int *sync, int n_steps, int n_stages, int kind0, int lts0, int lts1, int src_S,
                      unsigned int test_arrivals) {
  DevMesh mm = m;
  DevState ss = st;
  FluxParams ff = fp;
  BcParams bb = bp;
  CellStepsArgs a{};
  a.s.n_steps = n_steps;
  a.s.n_stages = n_stages;
  a.s.kind0 = kind0;
  a.s.arrivals = sync;
  a.s.gave_up = sync + kStepsBarrierStride;
  a.s.test_arrivals = test_arrivals;
  a.lts0 = lts0;
  a.lts1 = lts1;
  a.src_S = src_S;
  a.dt_min = reinterpret_cast<unsigned long long *>(sync + 2 * kStepsBarrierStride);
  void *args[] = {&mm, &ss, &ff, &bb, &a};
  cudaMemsetAsync(sync, 0, sizeof(unsigned int), s);
  cudaMemsetAsync(a.dt_min, 0xff, 3 * sizeof(unsigned long long), s);
  cudaLaunchCooperativeKernel(cell_steps_kernel(fp), dim3(nblk(4 * m.NP, kFlux4Block)), dim3(kFlux4Block), args, 0, s);
  return 1;
}

int launch_steps(cudaStream_t s, const DevMesh &m, const DevState &st, const FluxParams &fp, const BcParams &bp,
                 const StepsShape &sh, const StepsBlock *blocks, unsigned int *arrivals, unsigned int *gave_up, int n_steps,
                 int n_stages, int kind0, int keep_delu, int reduce, int may_stop, unsigned int test_arrivals) {
  DevMesh mm = m;
  DevState ss = st;
  FluxParams ff = fp;
  BcParams bb = bp;
  StepsArgs a{n_steps, n_stages, kind0,    keep_delu, sh.cells, sh.faces, sh.entries,
              reduce,  may_stop, blocks,   arrivals,  gave_up,  test_arrivals};
  void *args[] = {&mm, &ss, &ff, &bb, &a};
  cudaMemsetAsync(arrivals, 0, sizeof(unsigned int) * (size_t)sh.groups * kStepsBarrierStride, s);
  cudaLaunchCooperativeKernel(steps_kernel(fp), dim3(sh.blocks), dim3(sh.threads), args,
                              steps_smem(sh.cells, sh.faces, sh.entries), s);
  return 1;
}

int launch_muscl_gradients(cudaStream_t s, const DevMesh &m, DevState &st, const FluxParams &fp, int with_dt,
                           const BcParams *bc) {
  const int g = m.rblk ? m.n_rblk : nblk(m.NT, kBlock);
  if (m.rblk && g == 0) return 0;
  const BcParams bp = bc ? *bc : BcParams{};
  const int with_bc = bc ? 1 : 0;
  if (with_dt) launch_k(m, k_muscl_gradients<true>, g, kBlock, s, m, st, fp, bp, with_bc);
  else launch_k(m, k_muscl_gradients<false>, g, kBlock, s, m, st, fp, bp, with_bc);
  return 1;
}

int launch_amr_indicator(cudaStream_t s, const DevMesh &m, DevState &st, double *ind) {
  k_amr_indicator<<<nblk(m.NP, kBlock), kBlock, 0, s>>>(m, st, ind);
  return 1;
}

int launch_import_aos(cudaStream_t s, const double *aos, const int *perm, int NP, int NT, double *U) {
  k_import_aos<<<nblk(NT, kBlock), kBlock, 0, s>>>(aos, perm, NP, NT, U);
  return 1;
}

int launch_export_aos(cudaStream_t s, const double *U, const int *perm, int NP, int NT, int ld, double *aos) {
  k_export_aos<<<nblk(NT, kBlock), kBlock, 0, s>>>(U, perm, NP, NT, ld, aos);
  return 1;
}

int launch_amr_tags(cudaStream_t s, const double *ind, const int *ref, int NP, double threshold, double max_fraction,
                    void *scratch, uint8_t *tags) {
  // scratch: two SelectState + 256 histogram counters
  SelectState *sel = reinterpret_cast<SelectState *>(scratch);
  SelectState *sel_ref = sel + 1;
  unsigned int *hist = reinterpret_cast<unsigned int *>(sel + 2);
  const bool top = max_fraction > 0.0 && max_fraction < 1.0;
  int n = 0;
  if (top) {
    long long nRefine = static_cast<long long>(max_fraction * NP);
    if (nRefine < 1) nRefine = 1;
    SelectState init[2] = {{0ull, 0ull, nRefine, 0}, {0ull, 0ull, 0, 0}};
    cudaMemcpyAsync(sel, init, sizeof(init), cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(hist, 0, 256 * sizeof(unsigned int), s);
    const int g = nblk(NP, kBlock) < 1184 ? nblk(NP, kBlock) : 1184;
    for (int shift = 56; shift >= 0; shift -= 8) {
      k_amr_hist<<<g, kBlock, 0, s>>>(ind, ref, NP, sel, shift, 0, 0ull, hist);
      k_amr_pick<<<1, 32, 0, s>>>(sel, shift, 0, hist);
      n += 2;
    }
    // Among the cells whose key equals the cut value, the `remaining` lowest reference ids.
    // The key to match is read on the device inside k_amr_hist via sel_ref->... so copy it.
    SelectState host_sel;
    cudaMemcpyAsync(&host_sel, sel, sizeof(host_sel), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    SelectState init_ref = {0ull, 0xffffffff00000000ull, host_sel.remaining, 0};
    cudaMemcpyAsync(sel_ref, &init_ref, sizeof(init_ref), cudaMemcpyHostToDevice, s);
    for (int shift = 24; shift >= 0; shift -= 8) {
      k_amr_hist<<<g, kBlock, 0, s>>>(ind, ref, NP, sel_ref, shift, 1, host_sel.prefix, hist);
      k_amr_pick<<<1, 32, 0, s>>>(sel_ref, shift, 1, hist);
      n += 2;
    }
  }
  k_amr_tag<<<nblk(NP, kBlock), kBlock, 0, s>>>(ind, ref, NP, threshold, top ? 1 : 0, sel, sel_ref, tags);
  return n + 1;
}

int launch_set_ctl(cudaStream_t s, DevState &st, int idx, double v) {
  k_set_ctl<<<1, 1, 0, s>>>(st.ctl, idx, v);
  return 1;
}

}  // namespace cfdb
