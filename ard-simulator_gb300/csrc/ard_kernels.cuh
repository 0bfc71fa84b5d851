// sm_103a kernels of the ARD time step.  Templated on the working type T
// (float: the product path; double: the FP64 GPU oracle).
//
// Per step (t, parity par = t & 1), in launch order:
//   pml_kernel          Grote-Sim PML update of every slab (own stream)
//   face_kernel         (ard_face.cuh) forward 2D DCT-II of the 18 force face
//                       layers of every air partition, fused per layer pair in
//                       shared memory
//                       (face_gemm_kernel: the same as two GEMM passes where
//                       a layer pair does not fit)
//   modal_kernel        (ard_modal.cuh) F = expansion of the face transforms
//                       (+ point sources); M(t) = a (2 cos M(t-1) - M(t-2) + psi F);
//                       contraction of M(t) onto the face rows and the
//                       recorder cells
//   post_modal_kernel   recorder samples of step t + sums of the contraction
//                       partials
//   face_kernel         inverse 2D transforms -> pressure face layers
//                       (face_gemm_kernel: two GEMM passes)
//   iface_kernel        6th-order interface forcing into the force face
//                       layers / PML strips (owner masks resolve overlapping
//                       strips in the reference's list order)
// The air partitions' kernels (face, modal, sums) launch once per air group
// (up to two groups on two streams).  The host launches the step kernels with
// programmatic stream serialization; each loads its constants and then waits
// (grid_dependency_wait) before it touches what earlier kernels write.
// xform_gemm_kernel (register-staged GEMM) serves the dense
// whole-field transforms of the readouts and the initial pressure.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>
#include <utility>

#include "ard_async.cuh"
#include "ard_device.cuh"

namespace ard {

// Face layer (0..5) of coordinate c in an extent-n axis, -1 if not on the shell.
__host__ __device__ inline int face_layer(int c, int n) {
  return c < 3 ? c : (c >= n - 3 ? c - (n - 6) : -1);
}

// Offset of the force value of local cell (x, y, z) in the shell layers of D
// (X layers own x on the shell, then Y layers, then Z layers); -1 inside.
__host__ __device__ inline long long shell_index(const DctDev& D, int x, int y, int z) {
  int l = face_layer(x, D.w);
  if (l >= 0) return D.fX + ((long long)l * D.d + z) * D.h + y;
  l = face_layer(y, D.h);
  if (l >= 0) return D.fY + ((long long)l * D.d + z) * D.wp + x;
  l = face_layer(z, D.d);
  if (l >= 0) return D.fZ + ((long long)l * D.h + y) * D.wp + x;
  return -1;
}

// ---- 4-wide vector access (128-bit for float, 2 x 128-bit for double) ----
__device__ __forceinline__ void load4(const float* p, float (&r)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
}
__device__ __forceinline__ void load4(const double* p, double (&r)[4]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  r[0] = a.x; r[1] = a.y; r[2] = b.x; r[3] = b.y;
}
__device__ __forceinline__ void store4(float* p, const float (&r)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(r[0], r[1], r[2], r[3]);
}
__device__ __forceinline__ void store4(double* p, const double (&r)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(r[0], r[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(r[2], r[3]);
}

// ---- pairs of elements: packed FP32 arithmetic (one instruction for two
// IEEE-rounded results, sm_100 and later), two scalar operations for FP64 ----
template <typename T>
struct alignas(2 * sizeof(T)) Pair {
  T x, y;
};
__device__ __forceinline__ unsigned long long& pair_bits(Pair<float>& p) { return reinterpret_cast<unsigned long long&>(p); }
__device__ __forceinline__ Pair<float> fma2(Pair<float> a, Pair<float> b, Pair<float> c) {
  Pair<float> r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(pair_bits(r)) : "l"(pair_bits(a)), "l"(pair_bits(b)), "l"(pair_bits(c)));
  return r;
}
__device__ __forceinline__ Pair<float> mul2(Pair<float> a, Pair<float> b) {
  Pair<float> r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(pair_bits(r)) : "l"(pair_bits(a)), "l"(pair_bits(b)));
  return r;
}
__device__ __forceinline__ Pair<float> add2(Pair<float> a, Pair<float> b) {
  Pair<float> r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(pair_bits(r)) : "l"(pair_bits(a)), "l"(pair_bits(b)));
  return r;
}
__device__ __forceinline__ Pair<double> fma2(Pair<double> a, Pair<double> b, Pair<double> c) {
  return {fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)};
}
__device__ __forceinline__ Pair<double> mul2(Pair<double> a, Pair<double> b) { return {a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ Pair<double> add2(Pair<double> a, Pair<double> b) { return {a.x + b.x, a.y + b.y}; }
template <typename T>
__device__ __forceinline__ Pair<T> dup2(T v) { return {v, v}; }
// four consecutive elements as two pairs
template <typename T>
__device__ __forceinline__ void load4(const T* p, Pair<T> (&r)[2]) {
  T v[4];
  load4(p, v);
  r[0] = {v[0], v[1]};
  r[1] = {v[2], v[3]};
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const Pair<T> (&r)[2]) {
  const T v[4] = {r[0].x, r[0].y, r[1].x, r[1].y};
  store4(p, v);
}

// ---- asynchronous global -> shared copies (cp.async, L2-cached) ----
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;  // 0: zero-fill, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_scalar(float* smem, const float* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_scalar(double* smem, const double* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(n) : "memory");
}
// 4 consecutive elements (16 B for float, 2 x 16 B for double)
__device__ __forceinline__ void cp_async4(float* smem, const float* gmem, bool valid) { cp_async16(smem, gmem, valid); }
__device__ __forceinline__ void cp_async4(double* smem, const double* gmem, bool valid) {
  cp_async16(smem, gmem, valid);
  cp_async16(smem + 2, gmem + 2, valid);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Programmatic dependent launch: a step kernel launched with programmatic
// stream serialization may start while its predecessor in the stream is
// finishing; griddepcontrol.wait returns once the predecessor has completed
// and its writes are visible (at once for an ordinary launch).  Every block of
// every step kernel waits, before its first access to what a step kernel
// writes (constants - descriptors, job lists, tables - may be read before):
// since each kernel waits for its predecessor and that one for its own, all
// earlier writes are visible after it.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Lets the successor's blocks be scheduled once every block of this grid has
// got here (or ended).  Called where a block has little left to do: the
// successor's launch and constant loads then lie under this grid's last part
// (2-3 % of a step of a single room).  Earlier, its waiting blocks would hold
// the slots of the streams beside it (at kernel entry: L-shaped room 75 -> 96
// us per step).
__device__ __forceinline__ void grid_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---------------------------------------------------------------------------
// Batched 1D transforms as small GEMMs (see XformJob); one 64 x 64 output
// tile per block iteration, K staged through registers and shared memory in
// chunks of 16, 4 x 4 outputs per thread.  Used for the dense whole-field
// transforms (readouts, initial pressure); the step's face passes use
// face_gemm_kernel below.
// ---------------------------------------------------------------------------

__device__ __forceinline__ int find_job(const XformJob* __restrict__ jobs, int njobs, int unit) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].first <= unit) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T>
__device__ __forceinline__ T job_input(const T* __restrict__ buf, const XformJob& J, long long off) {
  const T a = buf[J.in0 + off];
  return J.in1 >= 0 ? a + (T)J.sgn * buf[J.in1 + off] : a;
}

template <typename T>
__global__ void __launch_bounds__(256) xform_gemm_kernel(T* __restrict__ buf, const XformJob* __restrict__ jobs,
                                                          int njobs, int total) {
  grid_dependency_wait();
  // two K-chunk buffers: chunk k+1 is fetched into registers while chunk k is
  // multiplied; chunks of 16 k (32 measured slower)
  constexpr int BK = 16;
  constexpr int NR = BK / 4;                     // elements of each operand a thread stages per chunk
  __shared__ __align__(16) T Ps[2][BK][64 + 4];  // P(m0 + mm, k0 + kk) at [kk][mm]
  __shared__ __align__(16) T Qs[2][BK][64 + 4];  // Q(k0 + kk, n0 + nn) at [kk][nn]
  // first unit of every job, cached in shared memory for the per-unit job search
  constexpr int kMaxCachedJobs = 1024;
  __shared__ int sfirst[kMaxCachedJobs];
  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
  const bool cached = njobs <= kMaxCachedJobs;
  if (cached)
    for (int i = tid; i < njobs; i += 256) sfirst[i] = jobs[i].first;
  __syncthreads();
  for (int unit = blockIdx.x; unit < total; unit += gridDim.x) {
    int ji;
    if (cached) {
      int lo = 0, hi = njobs - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sfirst[mid] <= unit) lo = mid; else hi = mid - 1;
      }
      ji = lo;
    } else {
      ji = find_job(jobs, njobs, unit);
    }
    const XformJob J = jobs[ji];
    const int t = unit - J.first;
    const int m0 = (t / J.tn) * 64, n0 = (t % J.tn) * 64;
    const int Md = J.rows ? J.batch : J.n;
    const int Nd = J.rows ? J.n : J.batch;
    const int K = J.n;
    const T* A = buf + J.ctab;
    T pr[NR], qr[NR];
    // global -> registers for the chunk at k0
    auto fetch = [&](int k0) {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int e = tid + 256 * r;
        if (!J.rows) {
          // P = A (m = output o, k = j); Q = X (k = j, n = column)
          const int mm = J.inverse ? (e & 63) : (e / BK), kk = J.inverse ? (e >> 6) : (e % BK);
          const int m = m0 + mm, k = k0 + kk;
          T pv = 0;
          if (m < Md && k < K) pv = J.inverse ? A[(long long)k * K + m] : A[(long long)m * K + k];
          pr[r] = pv;
          const int nn = e & 63, kq = e >> 6;
          const int n = n0 + nn, kk2 = k0 + kq;
          qr[r] = (n < Nd && kk2 < K) ? job_input(buf, J, (long long)kk2 * J.ld + n) : (T)0;
        } else {
          // P = X (m = line, k = j); Q(k, n) = A(n, k)
          const int mm = e / BK, kk = e % BK;
          const int m = m0 + mm, k = k0 + kk;
          pr[r] = (m < Md && k < K) ? job_input(buf, J, (long long)m * J.ld + k) : (T)0;
          const int nn = J.inverse ? (e & 63) : (e / BK), kq = J.inverse ? (e >> 6) : (e % BK);
          const int n = n0 + nn, kk2 = k0 + kq;
          T qv = 0;
          if (n < Nd && kk2 < K) qv = J.inverse ? A[(long long)kk2 * K + n] : A[(long long)n * K + kk2];
          qr[r] = qv;
        }
      }
    };
    auto commit = [&](int sb) {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int e = tid + 256 * r;
        if (!J.rows) {
          const int mm = J.inverse ? (e & 63) : (e / BK), kk = J.inverse ? (e >> 6) : (e % BK);
          Ps[sb][kk][mm] = pr[r];
          Qs[sb][e >> 6][e & 63] = qr[r];
        } else {
          Ps[sb][e % BK][e / BK] = pr[r];
          const int nn = J.inverse ? (e & 63) : (e / BK), kq = J.inverse ? (e >> 6) : (e % BK);
          Qs[sb][kq][nn] = qr[r];
        }
      }
    };
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    __syncthreads();  // the previous unit is done with both buffers
    fetch(0);
    commit(0);
    __syncthreads();
    int sb = 0;
    for (int k0 = 0; k0 < K; k0 += BK) {
      const bool more = k0 + BK < K;
      if (more) fetch(k0 + BK);
#pragma unroll
      for (int kk = 0; kk < BK; ++kk) {
        T pa[4], qb[4];
        load4(&Ps[sb][kk][ty * 4], pa);
        load4(&Qs[sb][kk][tx * 4], qb);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] += pa[i] * qb[j];
      }
      if (more) commit(sb ^ 1);
      __syncthreads();
      sb ^= 1;
    }
    const T scale = (T)J.scale;
    const int nb = n0 + tx * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + ty * 4 + i;
      if (m >= Md) continue;
      const long long o = J.out + (long long)m * J.ld + nb;
      if (nb + 3 < Nd && (o & 3) == 0) {
        T v[4] = {acc[i][0] * scale, acc[i][1] * scale, acc[i][2] * scale, acc[i][3] * scale};
        store4(buf + o, v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (nb + j < Nd) buf[o + j] = acc[i][j] * scale;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Face transforms of the step as GEMM passes (faces too large for the fused
// kernel): the same jobs as xform_gemm_kernel, with both operands staged by
// cp.async into a three-deep ring of 32-wide K chunks (no register staging,
// one barrier per chunk).  An operand whose source is contiguous along K
// ("k-contiguous": the X lines of a row pass, the forward tables) is kept
// [m or n][32 k] with its 16-byte chunks XOR-swizzled by (row / 4) % 8; an
// operand contiguous along m or n is kept [32 k][64 + 4].  The pass's input
// combination X = in0 + sgn in1 is formed when the X operand is read.
// Instances (one per job list, all jobs of a list alike):
//   PK, QK = 1, 1, CP: row pass, forward  (P = X lines, Q(k, n) = A[n K + k])
//   PK, QK = 1, 0:     column pass, forward (P = A[m K + k], Q = X rows) and
//                      row pass, inverse (P = X lines, Q(k, n) = A[k K + n])
//   PK, QK = 0, 0, CQ: column pass, inverse (P(m, k) = A[k K + m], Q = X rows)
// ---------------------------------------------------------------------------

constexpr int kGemmBK = 32;
constexpr int kGemmStages = 3;
constexpr int kGemmTile = kGemmBK * 68;   // elements of one staged operand tile (either layout)
__host__ __device__ constexpr int face_gemm_smem_elems(bool comb) { return kGemmStages * (comb ? 3 : 2) * kGemmTile; }

// k-contiguous tile: element (r, k) of the [64][32] tile
__device__ __forceinline__ int kc_index(int r, int k) { return r * kGemmBK + ((((k >> 2) ^ (r >> 2)) & 7) << 2) + (k & 3); }

template <typename T, bool PK, bool QK, bool CP, bool CQ>
__global__ void __launch_bounds__(256, 2) face_gemm_kernel(T* __restrict__ buf, const XformJob* __restrict__ jobs,
                                                            int njobs, int total) {
  grid_dependency_wait();
  constexpr bool COMB = CP || CQ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* sm = reinterpret_cast<T*>(smem_raw);
  constexpr int kMaxCachedJobs = 1024;
  __shared__ int sfirst[kMaxCachedJobs];
  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
  const bool cached = njobs <= kMaxCachedJobs;
  if (cached)
    for (int i = tid; i < njobs; i += 256) sfirst[i] = jobs[i].first;
  __syncthreads();
  for (int unit = blockIdx.x; unit < total; unit += gridDim.x) {
    int ji;
    if (cached) {
      int lo = 0, hi = njobs - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sfirst[mid] <= unit) lo = mid; else hi = mid - 1;
      }
      ji = lo;
    } else {
      ji = find_job(jobs, njobs, unit);
    }
    const XformJob J = jobs[ji];
    const int t = unit - J.first;
    const int m0 = (t / J.tn) * 64, n0 = (t % J.tn) * 64;
    const int Md = J.rows ? J.batch : J.n;
    const int Nd = J.rows ? J.n : J.batch;
    const int K = J.n;
    // operand sources: P (m, k) and Q (k, n); the X operand may have a second input
    long long p0, p1 = 0, q0, q1 = 0;
    int sp, sq;
    if (J.rows) { p0 = J.in0; p1 = J.in1; sp = J.ld; q0 = J.ctab; sq = K; }
    else { p0 = J.ctab; sp = K; q0 = J.in0; q1 = J.in1; sq = J.ld; }
    const T sgn = (T)J.sgn;
    // stage one operand tile: rows of the k-contiguous layout are m (or n),
    // rows of the other layout are k; lim = extent of m (or n)
    auto stage_kc = [&](T* dst, long long base, int stride, int r0, int lim, int k0) {
      const bool vec = ((stride | K) & 3) == 0 && (base & 3) == 0;
      if (vec) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int e = tid + 256 * v;          // 512 vectors: row e / 8, chunk e % 8
          const int r = e >> 3, c = e & 7;
          const bool ok = r0 + r < lim && k0 + 4 * c < K;
          cp_async4(dst + kc_index(r, 4 * c), buf + (ok ? base + (long long)(r0 + r) * stride + k0 + 4 * c : 0), ok);
        }
      } else {
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const int e = tid + 256 * v;          // 2048 elements: row e / 32, k e % 32
          const int r = e >> 5, k = e & 31;
          const bool ok = r0 + r < lim && k0 + k < K;
          cp_async_scalar(dst + kc_index(r, k), buf + (ok ? base + (long long)(r0 + r) * stride + k0 + k : 0), ok);
        }
      }
    };
    auto stage_mn = [&](T* dst, long long base, int stride, int c0, int lim, int k0) {
      const bool vec = ((stride | lim) & 3) == 0 && (base & 3) == 0;
      if (vec) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const int e = tid + 256 * v;          // 512 vectors: k e / 16, columns 4 (e % 16)
          const int k = e >> 4, c = (e & 15) * 4;
          const bool ok = k0 + k < K && c0 + c < lim;
          cp_async4(dst + k * 68 + c, buf + (ok ? base + (long long)(k0 + k) * stride + c0 + c : 0), ok);
        }
      } else {
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const int e = tid + 256 * v;          // 2048 elements: k e / 64, column e % 64
          const int k = e >> 6, c = e & 63;
          const bool ok = k0 + k < K && c0 + c < lim;
          cp_async_scalar(dst + k * 68 + c, buf + (ok ? base + (long long)(k0 + k) * stride + c0 + c : 0), ok);
        }
      }
    };
    constexpr int NT = COMB ? 3 : 2;
    auto issue = [&](int k0, int sb) {
      T* st = sm + sb * NT * kGemmTile;
      if constexpr (PK) stage_kc(st, p0, sp, m0, Md, k0); else stage_mn(st, p0, sp, m0, Md, k0);
      if constexpr (QK) stage_kc(st + kGemmTile, q0, sq, n0, Nd, k0); else stage_mn(st + kGemmTile, q0, sq, n0, Nd, k0);
      if constexpr (CP) stage_kc(st + 2 * kGemmTile, p1, sp, m0, Md, k0);
      if constexpr (CQ) stage_mn(st + 2 * kGemmTile, q1, sq, n0, Nd, k0);
    };
    T acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    const int nch = (K + kGemmBK - 1) / kGemmBK;
    __syncthreads();   // the previous unit is done with the ring
#pragma unroll
    for (int p = 0; p < kGemmStages - 1; ++p) {
      if (p < nch) issue(p * kGemmBK, p);
      cp_async_commit();
    }
    for (int c = 0; c < nch; ++c) {
      cp_async_wait<kGemmStages - 2>();
      __syncthreads();   // chunk c visible; chunk c - 1's slot free
      if (c + kGemmStages - 1 < nch) issue((c + kGemmStages - 1) * kGemmBK, (c + kGemmStages - 1) % kGemmStages);
      cp_async_commit();
      const T* st = sm + (c % kGemmStages) * NT * kGemmTile;
      const T* Pt = st;
      const T* Qt = st + kGemmTile;
      const T* Xt = st + 2 * kGemmTile;
#pragma unroll 2
      for (int kq = 0; kq < kGemmBK; kq += 4) {
        T pa[4][4], qb[4][4];   // [row i or column j][k of the quad]
        if constexpr (PK) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            load4(Pt + kc_index(ty * 4 + i, kq), pa[i]);
            if constexpr (CP) {
              T x[4];
              load4(Xt + kc_index(ty * 4 + i, kq), x);
#pragma unroll
              for (int k = 0; k < 4; ++k) pa[i][k] += sgn * x[k];
            }
          }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            T v[4];
            load4(Pt + (kq + k) * 68 + ty * 4, v);
#pragma unroll
            for (int i = 0; i < 4; ++i) pa[i][k] = v[i];
          }
        }
        if constexpr (QK) {
#pragma unroll
          for (int j = 0; j < 4; ++j) load4(Qt + kc_index(tx * 4 + j, kq), qb[j]);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            T v[4];
            load4(Qt + (kq + k) * 68 + tx * 4, v);
            if constexpr (CQ) {
              T x[4];
              load4(Xt + (kq + k) * 68 + tx * 4, x);
#pragma unroll
              for (int j = 0; j < 4; ++j) v[j] += sgn * x[j];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) qb[j][k] = v[j];
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += pa[i][k] * qb[j][k];
      }
    }
    cp_async_wait<0>();
    const T scale = (T)J.scale;
    const int nb = n0 + tx * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + ty * 4 + i;
      if (m >= Md) continue;
      const long long o = J.out + (long long)m * J.ld + nb;
      if (nb + 3 < Nd && (o & 3) == 0) {
        T v[4] = {acc[i][0] * scale, acc[i][1] * scale, acc[i][2] * scale, acc[i][3] * scale};
        store4(buf + o, v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (nb + j < Nd) buf[o + j] = acc[i][j] * scale;
      }
    }
  }
}

// Host: a step kernel launched with programmatic stream serialization: the
// grid is scheduled while its predecessor in the stream drains and waits for
// it on the device (grid_dependency_wait), which hides the launch gap between
// the dependent kernels of a step (also inside the captured graphs).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(void (*kernel)(KArgs...), long long grid, int block, size_t smem, cudaStream_t s,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Host: the face_gemm_kernel instance for a job list (all jobs of a list share
// rows, inverse and whether the X operand has a second input), `grid` blocks.
template <typename T>
inline cudaError_t launch_face_gemm(T* buf, const XformJob& j0, const XformJob* d_jobs, int njobs, int units, int grid,
                                    cudaStream_t s) {
  if (njobs == 0) return cudaSuccess;
  const bool comb = j0.in1 >= 0;
  const size_t s2 = (size_t)face_gemm_smem_elems(false) * sizeof(T), s3 = (size_t)face_gemm_smem_elems(true) * sizeof(T);
  if (j0.rows && !j0.inverse && comb)
    return launch_dep(face_gemm_kernel<T, true, true, true, false>, grid, 256, s3, s, buf, d_jobs, njobs, units);
  if (!comb && (j0.rows != 0) == (j0.inverse != 0))
    return launch_dep(face_gemm_kernel<T, true, false, false, false>, grid, 256, s2, s, buf, d_jobs, njobs, units);
  if (!j0.rows && j0.inverse && comb)
    return launch_dep(face_gemm_kernel<T, false, false, false, true>, grid, 256, s3, s, buf, d_jobs, njobs, units);
  return cudaErrorInvalidValue;
}

// Host: dynamic shared memory of the face_gemm_kernel instances (set in every
// translation unit that launches them).
template <typename T>
inline cudaError_t configure_face_gemm() {
  const int s2 = (int)(face_gemm_smem_elems(false) * sizeof(T)), s3 = (int)(face_gemm_smem_elems(true) * sizeof(T));
  cudaError_t e = cudaFuncSetAttribute(face_gemm_kernel<T, true, true, true, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, s3);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(face_gemm_kernel<T, true, false, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(face_gemm_kernel<T, false, false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3);
  return e;
}

// ---------------------------------------------------------------------------
// Recorder samples and sums of the contraction partials
// ---------------------------------------------------------------------------

// In-place sum of the per-tile partial slabs of the modal contraction:
// slab 0 of each job receives the sum of its nb slabs (fixed order).  A
// job's elements occupy [first, first + count) of the launch's index space,
// first a multiple of kSumChunk.
constexpr int kSumChunk = 2048;
constexpr int kSumBlocksPerSM = 5;   // resident blocks of the sums (8: 83 us, 5: 78 us, 4: 79 us for 15 M sums)
struct SumJob {
  long long base;     // slab 0
  long long count;    // elements per slab
  long long stride;   // slab stride
  long long first;    // first element of this job in the launch's index space
  int nb;
};

// After the modal update: the recorder samples of the step (blocks
// [0, rec_blocks): one warp per recorder, the sum of the tiles' partials
// times s_i into the double history) and the in-place partial sums (the
// other blocks: launches of at least a wave of chunks grid-stride over
// chunks of kSumChunk elements, 8 per thread; smaller ones take one element
// per thread with all its slabs in flight).  One launch for both.
template <typename T>
struct PostModalArgs {
  T* buf;
  const DctDev* dct;
  // points read out: the recorders [rec_first, rec_first + nrec) into the
  // history row of the step, or (adjoint) the sources into the row of the
  // source-series gradient
  bool adjoint;
  const PointDev* recs;
  int rec_first, nrec;
  int nrec_total;         // row width of the history (gradient)
  double* hist;
  const long long* tcount;
  int tstep;
  long long max_steps;
  int rec_blocks;
  const SumJob* jobs;     // this launch's sum jobs; their elements start at `first`
  int njobs;
  long long first;
  long long total;        // a multiple of kSumChunk
  int per;                // elements per thread: 8 (chunked), 0: one element per thread.  The chunked loop
                          // takes 1, 2, 4 or 8 as it comes: with 8 fixed in the code the compiler's
                          // registers cost the 15 M sums of 187.5 M cells 84 instead of 79 us
};

template <typename T>
__global__ void __launch_bounds__(256, kSumBlocksPerSM) post_modal_kernel(PostModalArgs<T> a) {
  if ((int)blockIdx.x < a.rec_blocks) {
    const int lane = threadIdx.x & 31;
    const int rl = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int r = a.rec_first + min(rl, a.nrec - 1);
    const PointDev q = a.recs[r];
    const DctDev& D = a.dct[q.part];
    const int local = r - (a.adjoint ? D.src0 : D.rec0), n = a.adjoint ? D.nsrc : D.nrec;
    const T* part = a.buf + (a.adjoint ? D.srcpart : D.recpart) + local;
    const int ntiles = D.ntiles;
    const double scale = a.adjoint ? D.sf : D.si;
    grid_dependency_wait();
    if (rl >= a.nrec) return;
    T s[4] = {0, 0, 0, 0};   // four loads in flight
    for (int i = lane; i < ntiles; i += 128)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + 32 * k < ntiles) s[k] += part[(long long)(i + 32 * k) * n];
    const T sum = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
    if (lane != 0) return;
    if (a.adjoint) {
      a.hist[(*a.tcount - a.tstep) * a.nrec_total + q.slot] = (double)sum * scale;
    } else {
      const long long t = *a.tcount + a.tstep;
      if (t < a.max_steps) a.hist[t * a.nrec_total + q.slot] = (double)(sum * (T)scale);
    }
    return;
  }
  T* __restrict__ buf = a.buf;
  // first elements of the jobs, cached for the per-chunk job search
  constexpr int kMaxCachedJobs = 1024;
  __shared__ long long sfirst[kMaxCachedJobs];
  const bool cached = a.njobs <= kMaxCachedJobs;
  if (cached)
    for (int i = threadIdx.x; i < a.njobs; i += blockDim.x) sfirst[i] = a.jobs[i].first;
  __syncthreads();
  grid_dependency_wait();   // the jobs are constants
  // chunks of kSumChunk elements: a job's elements start on a chunk boundary
  // of the index space, so a chunk lies in one job; a thread sums 8 elements
  // (256 apart) over the job's slabs, slab by slab in order
  const long long nb = (long long)gridDim.x - a.rec_blocks;
  if (a.per == 0) {
    // small launches: one element per thread, all its slabs in flight at once
    for (long long g = ((long long)blockIdx.x - a.rec_blocks) * blockDim.x + threadIdx.x; g < a.total;
         g += nb * blockDim.x) {
      const long long gg = g + a.first;
      int lo = 0, hi = a.njobs - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((cached ? sfirst[mid] : a.jobs[mid].first) <= gg) lo = mid; else hi = mid - 1;
      }
      const SumJob J = a.jobs[lo];
      const long long e = gg - J.first;
      if (e >= J.count) continue;   // the chunk padding of the index space
      const T* p = buf + J.base + e;
      T v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      int b = 0;
      for (; b + 8 <= J.nb; b += 8) {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] += p[(long long)(b + k) * J.stride];
      }
#pragma unroll
      for (int k = 0; k < 7; ++k)
        if (b + k < J.nb) v[k] += p[(long long)(b + k) * J.stride];
      buf[J.base + e] = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
    }
    return;
  }
  // work items: a chunk in kSumChunk / (256 per) parts of 256 per elements,
  // `per` (1, 2, 4 or 8) elements per thread, 256 apart
  const int per = a.per;
  const int parts = kSumChunk / (256 * per);
  const long long nitems = a.total / kSumChunk * parts;
  for (long long item = (long long)blockIdx.x - a.rec_blocks; item < nitems; item += nb) {
    const long long ch = item / parts;
    const int part = (int)(item - ch * parts);
    const long long gg = a.first + ch * kSumChunk;   // first element of the chunk among all sum jobs
    int lo = 0, hi = a.njobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((cached ? sfirst[mid] : a.jobs[mid].first) <= gg) lo = mid; else hi = mid - 1;
    }
    const SumJob J = a.jobs[lo];
    const long long e0 = gg - J.first + (long long)part * 256 * per;
    T* p = buf + J.base + e0;
    constexpr int kPer = kSumChunk / 256;
    bool ok[kPer];
    T v[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const int idx = (int)threadIdx.x + 256 * i;
      ok[i] = i < per && e0 + idx < J.count;
      v[i] = ok[i] ? p[idx] : (T)0;
    }
#pragma unroll 2
    for (int b = 1; b < J.nb; ++b) {
      const T* q = p + (long long)b * J.stride;
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (ok[i]) v[i] += q[threadIdx.x + 256 * i];
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i)
      if (ok[i]) p[threadIdx.x + 256 * i] = v[i];
  }
}

// ---------------------------------------------------------------------------
// PML
// ---------------------------------------------------------------------------

// Forward PML history kept for the adjoint's damping gradient: for steps
// t0 <= t < t1 the PML kernel also writes p(t) to p[(t - t0 + 1) hlen + ...]
// and phi_n(t) to phn[(t - t0) hlen + ...] (all-slab region layout, slab at
// PmlDev::hoff).  p == null: nothing is kept.
// Strip forces: for steps ft0 <= t < ft1 the kernel also writes the strip
// force it reads (the interfaces' forcing of step t-1) to f[(t - ft0) flen +
// PmlDev::foff + ...]; with fsrc set it reads the strip force of step t from
// fsrc[(t - fs0) flen + ...] instead of the context's strips (the PML runs
// again on its own, replaying the recorded forcing).
template <typename T>
struct PmlHist {
  T* p;
  T* phn;
  long long hlen;
  long long t0, t1;
  T* f;
  long long flen;
  long long ft0, ft1;
  const T* fsrc;
  long long fs0;
};

template <typename T>
struct PmlArgs {
  T* buf;
  const PmlDev* pml;
  const int4* blocks;   // {slab, a0, b0}: plane tiles (pml_shape)
  int nblocks;
  int par;
  T dt, dt2;
  T klap, r12;          // c0^2 dt^2 / (180 dh^2), 1 / (12 dh)
  const PmlHist<T>* hist;   // null without the adjoint
  const long long* tcount;
  int tstep;
  const CUtensorMap* maps;  // per slab: p[0], p[1], pha[0], pha[1], phb[0], phb[1] as [L][A][B] tensors
  int* err;                 // set to 1 when a bounded wait runs out
};

// Plane tile of a slab: a block of kPmlThreads threads, four consecutive b
// each, 2^q of them along b: 32 x 16, 16 x 32 or 8 x 64 cells (a x b),
// whichever covers the slab's plane with the fewest tiles.
constexpr int kPmlThreads = 128;
constexpr int kPmlStages = 2;   // a third stage measured no faster
struct PmlShape {
  int q;        // log2 of the threads along b
  int TA, TB;   // tile extents
  int PW;       // row pitch of the p and phi_b boxes
};
__host__ __device__ inline PmlShape pml_shape(int q) { return {q, kPmlThreads >> q, 4 << q, (4 << q) + 8}; }
__host__ __device__ inline int pml_tiles(int q, int A, int B) {
  const PmlShape s = pml_shape(q);
  return ((A + s.TA - 1) / s.TA) * ((B + s.TB - 1) / s.TB);
}
inline int pml_pick_shape(int A, int B) {
  int best = 3;
  for (int q : {2, 4})
    if (pml_tiles(q, A, B) < pml_tiles(best, A, B)) best = q;
  return best;
}

// The boxes that the TMA unit loads per layer: p with a halo of 3 along a and
// of 4 / 4 along b (x starts at b0 - 4, on a 16-byte boundary), phi_a with a
// halo of 2 along a, phi_b with a halo of 4 / 4 along b; each box 128-byte
// aligned in the stage.
template <typename T>
struct PmlBoxes {
  int p, fa, fb;      // bytes
  int off_fa, off_fb; // offsets in the stage
  __host__ __device__ explicit PmlBoxes(const PmlShape& s) {
    p = (s.TA + 6) * s.PW * (int)sizeof(T);
    fa = (s.TA + 4) * s.TB * (int)sizeof(T);
    fb = s.TA * s.PW * (int)sizeof(T);
    off_fa = (p + 127) & ~127;
    off_fb = off_fa + fa;   // fa is a multiple of 128
  }
};
// bytes of a stage: the largest shape (8 x 64)
template <typename T>
__host__ __device__ constexpr int pml_stage_bytes() {
  return ((14 * 72 * (int)sizeof(T) + 127) & ~127) + 12 * 64 * (int)sizeof(T) + 8 * 72 * (int)sizeof(T) + 128;
}
template <typename T>
constexpr size_t pml_smem_bytes() { return (size_t)kPmlStages * pml_stage_bytes<T>() + 128; }
template <typename T>
constexpr int pml_blocks_per_sm() { return sizeof(T) == 4 ? 4 : 2; }

// Grote-Sim PML (pml_partition.cpp:113-200) in slab coordinates: layer l
// along the normal, (a, b) in the plane; outside the slab every field reads
// zero (the reference's sentinel cell).  Only the normal damping zeta_n is
// non-zero in a slab (zeta_a = zeta_b = 0 in the reference's formulas).
// A block owns a plane tile (pml_shape) and walks the layers; a thread owns
// four consecutive b.  The in-plane stencils read tiles of p(t-1) (halo 3),
// phi_a and phi_b (halo 2 along their own axis) that the TMA unit brings into
// a ring of shared memory, ahead of the computation and across the block's
// tiles; the tensor maps' zero fill outside the slab is the sentinel.  The
// normal-axis stencils run from register windows; p(t-2) and the strip force
// of the next layer are fetched into registers while the current one computes.
// In FP32 the Laplacian sums taps minus the centre before it weights them
// (rounding, for smooth fields, a fifth of the tap-by-tap chain's).  Large slabs are bound by HBM and by the chain of
// a layer at 16 warps per SM (the windows take the registers): GB300, 22.3 M
// cells 249 -> 185 us (4.3 TB/s of 36 bytes per cell), 20.8 M cells in the
// slabs of 128 scenes 342 -> 213 us, against one cell per thread and 8 x 32
// tiles; three blocks per SM were 16 % slower, five spill (half as fast).  FP64 is
// bound by its arithmetic (0.22 M cells 98 -> 80 us).  Every wait is bounded:
// one that runs out sets the kernel's error word and the block leaves its
// loops.
template <typename T>
__global__ void __launch_bounds__(kPmlThreads, pml_blocks_per_sm<T>()) pml_kernel(PmlArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* const stage =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
  constexpr int kStage = pml_stage_bytes<T>();
  __shared__ uint64_t bar[kPmlStages];
  __shared__ volatile int s_abort;
  if (threadIdx.x == 0) {
    for (int k = 0; k < kPmlStages; ++k) mbar_init(&bar[k], 1);
    mbar_init_fence();
    s_abort = 0;
  }
  grid_dependency_wait();
  __syncthreads();
  T* hp = nullptr;
  T* hfn = nullptr;
  T* hf = nullptr;
  const T* fsrc = nullptr;
  if (a.hist) {
    const PmlHist<T> h = *a.hist;
    const long long t = *a.tcount + a.tstep;
    if (h.p && t >= h.t0 && t < h.t1) {
      hp = h.p + (t - h.t0 + 1) * h.hlen;
      hfn = h.phn + (t - h.t0) * h.hlen;
    }
    if (h.f && t >= h.ft0 && t < h.ft1) hf = h.f + (t - h.ft0) * h.flen;
    if (h.fsrc) fsrc = h.fsrc + (t - h.fs0) * h.flen;
  }
  // thread 0's issue cursor over the block's (tile, layer) sequence
  int ibi = blockIdx.x, il = 0, iL = 0, iq = 0, ist = 0;
  const int lev = a.par ^ 1;   // time level t-1 of p, phi_a, phi_b
  auto issue_next = [&]() {
    if (ibi >= a.nblocks) return;
    const int4 blk = a.blocks[ibi];
    if (il == 0) {
      iL = a.pml[blk.x].L;
      iq = a.pml[blk.x].q;
    }
    const PmlShape S = pml_shape(iq);
    const PmlBoxes<T> X(S);
    const CUtensorMap* mp = a.maps + 6LL * blk.x;
    unsigned char* sb = stage + ist * kStage;
    uint64_t* br = &bar[ist];
    mbar_arrive_expect_tx(br, (uint32_t)(X.p + X.fa + X.fb));
    tma_load_3d(sb, mp + lev, blk.z - 4, blk.y - 3, il, br);
    tma_load_3d(sb + X.off_fa, mp + 2 + lev, blk.z, blk.y - 2, il, br);
    tma_load_3d(sb + X.off_fb, mp + 4 + lev, blk.z - 4, blk.y, il, br);
    ist = ist + 1 == kPmlStages ? 0 : ist + 1;
    if (++il == iL) {
      il = 0;
      ibi += gridDim.x;
    }
  };
  if (threadIdx.x == 0)
    for (int k = 0; k < kPmlStages; ++k) issue_next();
  int sg = 0;           // stage and phase of the layer being computed (uniform)
  uint32_t phase = 0;
  bool stop = false;
  for (int bi = blockIdx.x; bi < a.nblocks && !stop; bi += gridDim.x) {
    const int4 blk = a.blocks[bi];
    const PmlDev& P = a.pml[blk.x];
    const int L = P.L, A = P.A, B = P.B, Bp = P.Bp;
    const PmlShape S = pml_shape(P.q);
    const PmlBoxes<T> X(S);
    const int PW = S.PW, TB = S.TB;
    const int tb = 4 * ((int)threadIdx.x & ((1 << S.q) - 1)), ta = (int)threadIdx.x >> S.q;
    const int strip0 = P.strip0;       // held in registers: the layer loop stores through the pool pointer
    const long long hoff = P.hoff;
    const int ia = blk.y + ta, ib = blk.z + tb;
    const bool inside = ia < A && ib < B;
    const int nb = B - ib;             // cells of the thread's four that lie in the slab
    const long long lstride = (long long)A * Bp;
    const long long col = inside ? (long long)ia * Bp + ib : 0;
    const T* p = a.buf + P.p[a.par ^ 1] + col;   // p(t-1)
    T* pn = a.buf + P.p[a.par] + col;            // p(t-2) -> p(t)
    const T* fn = a.buf + P.phn[a.par ^ 1] + col;
    T* fn_o = a.buf + P.phn[a.par] + col;
    T* fa_o = a.buf + P.pha[a.par] + col;
    T* fb_o = a.buf + P.phb[a.par] + col;
    const T* zeta = a.buf + P.zeta;
    const T* force = (fsrc ? fsrc + P.foff : a.buf + P.force) + col;
    T* force_rec = hf ? hf + P.foff + col : nullptr;
    auto quad = [&](const T* q, bool ok, T (&v)[4]) {
      if (ok) {
        load4(q, v);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = 0;
      }
    };
    // register windows along the normal: p(l-3 .. l+3), phi_n(l-2 .. l+2)
    T pw[7][4], fw[5][4];
#pragma unroll
    for (int m = 0; m < 7; ++m) quad(p + (m - 3) * lstride, inside && m >= 3 && m - 3 < L, pw[m]);
#pragma unroll
    for (int m = 0; m < 5; ++m) quad(fn + (m - 2) * lstride, inside && m >= 2 && m - 2 < L, fw[m]);
    T nold[4], nforce[4];
    auto fetch = [&](int l) {
      const int sl = l - strip0;
      quad(pn + l * lstride, inside, nold);
      quad(force + sl * lstride, inside && sl >= 0 && sl < 3, nforce);
    };
    fetch(0);
    for (int l = 0; l < L; ++l) {
      T pold[4], f[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        pold[e] = nold[e];
        f[e] = nforce[e];
      }
      if (l + 1 < L) fetch(l + 1);
      if (force_rec && inside) {
        const int sl = l - strip0;
        if (sl >= 0 && sl < 3) store4(force_rec + sl * lstride, f);
      }
      const T zn = zeta[l];
      mbar_wait_bounded(&bar[sg], phase, &s_abort);
      if (inside && !s_abort) {
        const unsigned char* sb = stage + sg * kStage;
        const T* Ps = reinterpret_cast<const T*>(sb) + ta * PW + tb + 4;                  // rows ia - 3 .., columns ib ..
        const T* FA = reinterpret_cast<const T*>(sb + X.off_fa) + ta * TB + tb;           // rows ia - 2 ..
        const T* FB = reinterpret_cast<const T*>(sb + X.off_fb) + ta * PW + tb + 4;
        T lap[4], g1[4], g2[4], ua[4], ub[4], v[4], u[4], w[12];   // w: p along b from ib - 4
        load4(Ps + 3 * PW - 4, v); load4(Ps + 3 * PW + 4, u);
#pragma unroll
        for (int e = 0; e < 4; ++e) { w[e] = v[e]; w[4 + e] = pw[3][e]; w[8 + e] = u[e]; }
#pragma unroll
        for (int e = 0; e < 4; ++e) ub[e] = (w[e + 2] - w[e + 6]) + (T)8 * (w[e + 5] - w[e + 3]);
        if constexpr (sizeof(T) == 4) {
          // 2 t3 - 27 t2 + 270 t1, t_m the axes' sums of p(+m) + p(-m) - 2 p:
          // taps minus the centre cancel before they are weighted (t1 by
          // differences, which are exact for neighbours within a factor of two)
          T t1[4], t2[4], t3[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const T pc = pw[3][e], m2 = (T)-2 * pc;
            t1[e] = ((pw[2][e] - pc) + (pw[4][e] - pc)) + ((w[e + 3] - pc) + (w[e + 5] - pc));
            t2[e] = ((pw[1][e] + pw[5][e]) + m2) + ((w[e + 2] + w[e + 6]) + m2);
            t3[e] = ((pw[0][e] + pw[6][e]) + m2) + ((w[e + 1] + w[e + 7]) + m2);
          }
          load4(Ps, v); load4(Ps + 6 * PW, u);
#pragma unroll
          for (int e = 0; e < 4; ++e) t3[e] += (v[e] + u[e]) - (T)2 * pw[3][e];
          load4(Ps + PW, v); load4(Ps + 5 * PW, u);
#pragma unroll
          for (int e = 0; e < 4; ++e) { t2[e] += (v[e] + u[e]) - (T)2 * pw[3][e]; ua[e] = v[e] - u[e]; }
          load4(Ps + 2 * PW, v); load4(Ps + 4 * PW, u);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            t1[e] += (v[e] - pw[3][e]) + (u[e] - pw[3][e]);
            ua[e] += (T)8 * (u[e] - v[e]);
            lap[e] = (T)270 * t1[e] - (T)27 * t2[e] + (T)2 * t3[e];
          }
        } else {
          // FP64 is bound by its operations: three weighted chains
          const T c7[7] = {2, -27, 270, -490, 270, -27, 2};
          T la[4] = {0, 0, 0, 0}, lb[4] = {0, 0, 0, 0}, ln[4] = {0, 0, 0, 0};
#pragma unroll
          for (int m = 0; m < 7; ++m) {
            load4(Ps + m * PW, v);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              la[e] += c7[m] * v[e];
              lb[e] += c7[m] * w[e + 1 + m];
              ln[e] += c7[m] * pw[m][e];
              if (m == 1) ua[e] = v[e];
              if (m == 2) ua[e] -= (T)8 * v[e];
              if (m == 4) ua[e] += (T)8 * v[e];
              if (m == 5) ua[e] -= v[e];
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) lap[e] = ln[e] + la[e] + lb[e];
        }
        // divergence of phi: taps -2, +2 in g2, +1, -1 in g1
#pragma unroll
        for (int e = 0; e < 4; ++e) { g2[e] = fw[0][e] - fw[4][e]; g1[e] = fw[3][e] - fw[1][e]; }
        load4(FA, v); load4(FA + 4 * TB, u);
#pragma unroll
        for (int e = 0; e < 4; ++e) g2[e] += v[e] - u[e];
        load4(FA + TB, v); load4(FA + 3 * TB, u);
#pragma unroll
        for (int e = 0; e < 4; ++e) g1[e] += u[e] - v[e];
        T fb0[4], fa0[4];
        load4(FA + 2 * TB, fa0);
        {
          load4(FB - 4, v); load4(FB, fb0); load4(FB + 4, u);
#pragma unroll
          for (int e = 0; e < 4; ++e) { w[e] = v[e]; w[4 + e] = fb0[e]; w[8 + e] = u[e]; }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            g2[e] += w[e + 2] - w[e + 6];
            g1[e] += w[e + 5] - w[e + 3];
          }
        }
        const T dz = a.dt * zn, dzr = dz * a.r12, kdiv = a.dt2 * a.r12;
        T pnew[4], fnew[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const T pc = pw[3][e];
          const T div = g2[e] + (T)8 * g1[e];
          const T un = (pw[1][e] - pw[5][e]) + (T)8 * (pw[4][e] - pw[2][e]);
          pnew[e] = ((T)2 * pc - pold[e]) + (a.klap * lap[e] - dz * (pc - pold[e]) + kdiv * div + a.dt2 * f[e]);
          const T fc = fw[2][e];
          fnew[e] = fc - dz * fc - dzr * un;
          fa0[e] += dzr * ua[e];
          fb0[e] += dzr * ub[e];
        }
        if (nb < 4) {   // the row pitch's padding columns stay zero
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (e >= nb) pnew[e] = fnew[e] = fa0[e] = fb0[e] = 0;
        }
        const long long I = l * lstride;
        store4(pn + I, pnew);
        store4(fn_o + I, fnew);
        store4(fa_o + I, fa0);
        store4(fb_o + I, fb0);
        if (hp) {
          store4(hp + hoff + col + I, pnew);
          store4(hfn + hoff + col + I, fnew);
        }
      }
      // slide the windows one layer
#pragma unroll
      for (int m = 0; m < 6; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) pw[m][e] = pw[m + 1][e];
      quad(p + (l + 4) * lstride, inside && l + 4 < L, pw[6]);
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) fw[m][e] = fw[m + 1][e];
      quad(fn + (l + 3) * lstride, inside && l + 3 < L, fw[4]);
      __syncthreads();   // every thread is done with stage sg
      if (s_abort) {
        stop = true;
        break;
      }
      if (threadIdx.x == 0) issue_next();
      if (++sg == kPmlStages) {
        sg = 0;
        phase ^= 1;
      }
    }
  }
  if (s_abort) {
    // a wait ran out: report it, and give loads still in flight time to land
    // (bounded) before the block's shared memory is released
    if (threadIdx.x == 0) {
      atomicExch(a.err, 1);
      const long long t0 = clock64();
      while (clock64() - t0 < 20000000LL) {
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Interfaces
// ---------------------------------------------------------------------------

template <typename T>
struct IfaceArgs {
  T* buf;
  const IfaceDev* ifs;
  const IfaceItem* items;
  int nitems;
  const unsigned char* masks;
  int par;
  T k0;   // c0^2 / (180 dh^2)
};
constexpr int kIfaceThreads = 128;

// A lane's addresses on one side of an interface: the pressure of stencil
// layer k = 0 .. 2 (crossing coordinate ext - 3 + k on the lo side, k on the
// hi side) in row r is p + k ps + r pv, its force f + k fk + r fv.
struct SideRow {
  long long p, ps, f, fk;
  int pv, fv;
};
__device__ __forceinline__ SideRow side_row(const SideDev& S, int type, bool lo, int u, int v, int par) {
  SideRow r;
  r.pv = S.psv;
  r.p = S.pb[0][par] + (long long)v * S.psv + u;
  r.ps = S.pb[1][par] - S.pb[0][par];
  const int c0 = lo ? S.ext - 3 : 0, l0 = lo ? 3 : 0;   // crossing coordinate and face layer of k = 0
  int l;
  if (S.kind == 1) {                                         // PML strip
    r.f = S.fb + (long long)c0 * S.fls + (long long)v * S.fsv + u;
    r.fk = S.fls;
    r.fv = S.fsv;
  } else if (type == 0) {                                    // X layers own what they touch
    r.f = S.fx + ((long long)l0 * S.d + v) * S.h + u;
    r.fk = (long long)S.d * S.h;
    r.fv = S.h;
  } else if ((l = face_layer(u, S.w)) >= 0) {                // u = x on the shell
    r.f = type == 1 ? S.fx + ((long long)l * S.d + v) * S.h + c0 : S.fx + ((long long)l * S.d + c0) * S.h + v;
    r.fk = type == 1 ? 1 : S.h;
    r.fv = type == 1 ? S.h : 1;
  } else if (type == 1) {                                    // Y layers own the rest of theirs
    r.f = S.fy + ((long long)l0 * S.d + v) * S.wp + u;
    r.fk = (long long)S.d * S.wp;
    r.fv = S.wp;
  } else if ((l = face_layer(v, S.h)) >= 0) {                // v = y on the shell (one row to an item)
    r.f = S.fy + ((long long)l * S.d + c0) * S.wp + u;
    r.fk = S.wp;
    r.fv = 0;
  } else {
    r.f = S.fz + ((long long)l0 * S.h + v) * S.wp + u;
    r.fk = (long long)S.h * S.wp;
    r.fv = S.wp;
  }
  return r;
}

// The interface stencil (boundary.cpp:23-29): force of layer m - 3 from the
// three pressures on each side.
__device__ constexpr int kIfaceC[6][6] = {{0, 0, -2, 2, 0, 0},         {0, -2, 27, -27, 2, 0},   {-2, 27, -270, 270, -27, 2},
                                          {2, -27, 270, -270, 27, -2}, {0, 2, -27, 27, -2, 0},   {0, 0, 2, -2, 0, 0}};

// Boundary::ComputeForcingTerms (boundary.cpp:21-173) for every face cell of
// every interface; the per-cell mask keeps only the writes that survive the
// reference's list-order overwrites.  A warp takes 32 cells along u of a few
// rows of one interface: the descriptors are read and the addresses formed
// once, and both are linear over the rows.  GB300, against one thread per cell
// with its own descriptor reads, a division and the owner's search (540
// instructions per cell): 4.1 M cells 89 -> 56 us, 5.9 M cells of 128 scenes
// 131 -> 101, one 100^3 room 8.4 -> 7.7.
template <typename T>
__global__ void __launch_bounds__(kIfaceThreads) iface_kernel(IfaceArgs<T> a) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (kIfaceThreads / 32);
  bool waited = false;
  for (int i = blockIdx.x * (kIfaceThreads / 32) + (threadIdx.x >> 5); i < a.nitems; i += warps) {
    const IfaceItem it = a.items[i];
    const IfaceDev& I = a.ifs[it.iface];
    const int type = I.type, nu = I.u1 - I.u0, u = it.u0 + lane;
    const bool ok = u < nu;
    SideRow L = side_row(I.lo, type, true, I.u0 + u - I.lo.ou, I.v0 + it.v0 - I.lo.ov, a.par);
    SideRow H = side_row(I.hi, type, false, I.u0 + u - I.hi.ou, I.v0 + it.v0 - I.hi.ov, a.par);
    const bool lself = I.lo.self != 0, hself = I.hi.self != 0;
    const T k = (T)I.absorption * a.k0;
    const unsigned char* mk = a.masks + I.mask + (long long)it.v0 * nu + u;
    if (!waited) {
      grid_dependency_wait();   // items, descriptors and masks are constants
      waited = true;
    }
    for (int r = 0; r < it.n; ++r) {
      const unsigned mask = ok ? *mk : 0u;
      T p[6];
#pragma unroll
      for (int n = 0; n < 3; ++n) {
        p[n] = ok ? a.buf[L.p + n * L.ps] : (T)0;
        p[3 + n] = ok ? a.buf[H.p + n * H.ps] : (T)0;
      }
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        T s1 = 0, s2 = 0;
#pragma unroll
        for (int n = 0; n < 3; ++n) {
          s1 += (T)kIfaceC[m][n] * p[n];
          s2 += (T)kIfaceC[m][3 + n] * p[3 + n];
        }
        const T s = (m < 3 ? (lself ? s1 + s2 : s2) : (hself ? s1 + s2 : s1)) * k;
        if (mask >> m & 1) a.buf[m < 3 ? L.f + m * L.fk : H.f + (m - 3) * H.fk] = s;
      }
      mk += nu;
      L.p += L.pv;
      L.f += L.fv;
      H.p += H.pv;
      H.f += H.fv;
    }
  }
  if (!waited) grid_dependency_wait();   // no item: still not done before the predecessor
}

static __global__ void advance_time_kernel(long long* tcount, int n) {
  if (threadIdx.x == 0 && blockIdx.x == 0) *tcount += n;
}

// ---- setup kernels (FP64 arithmetic) ----

// Per extent n, three n*n tables: C[k][j] = 2 cos(pi (j + 1/2) k / n) (the
// REDFT10 matrix), the REDFT01 matrix Ci[k][j] = C[k][j] with row k = 0
// halved (REDFT01 weights X_0 by 1, the others by 2), and the transpose of Ci
// (contiguous along k, as the neighbourhood sums read it).
template <typename T>
__global__ void cos_table_kernel(T* buf, long long off, int n) {
  const long long nn = (long long)n * n;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i / n), j = (int)(i - (long long)k * n);
    const long long q = ((long long)(2 * j + 1) * k) % (4LL * n);  // argument reduced exactly in integers
    const double v = 2.0 * cospi((double)q / (2.0 * n));
    const double vi = k == 0 ? 0.5 * v : v;
    buf[off + i] = (T)v;
    buf[off + nn + i] = (T)vi;
    buf[off + 2 * nn + (long long)j * n + k] = (T)vi;
  }
}

// Accurate-arithmetic tables: tabA = 1 - cos(w dt) = 2 sin^2(w dt / 2),
// tabB = 2 (1 - cos(w dt)) / w^2, in FP64 then rounded to T; [d][h][wp],
// padding columns zero.
template <typename T>
__global__ void modal_table_kernel(T* buf, long long tabA, long long tabB, int w, int wp, int h, int d, double dh,
                                   double dt, double c0) {
  const long long N = (long long)wp * h * d;
  const double lx = w * dh, ly = h * dh, lz = d * dh;
  const double pi = 3.14159265358979323846;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const int kx = (int)(i % wp);
    const int ky = (int)((i / wp) % h);
    const int kz = (int)(i / ((long long)wp * h));
    if (kx >= w) { buf[tabA + i] = 0; buf[tabB + i] = 0; continue; }
    // 1-based mode numbers, as dct_partition.cpp:24-36
    const double ax = (kx + 1) / lx, ay = (ky + 1) / ly, az = (kz + 1) / lz;
    const double omega = c0 * pi * sqrt(az * az + ay * ay + ax * ax);
    const double th = omega * dt;
    const double s = sin(0.5 * th);
    const double vers = 2.0 * s * s;
    buf[tabA + i] = (T)vers;
    buf[tabB + i] = (T)(2.0 * vers / (omega * omega));
  }
}

}  // namespace ard
